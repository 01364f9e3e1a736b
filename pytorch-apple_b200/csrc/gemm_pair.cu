// Linear layers on CTA pairs (cta_group::2), weights on the 256-row side of the MMA, tokens on its N side.
//
// A 128 x 256 tile per CTA needs 48 KB of operands per 4.2 MFLOP; at the rate the L2 feeds the SMs (measured ~11 TB/s over
// all SMs) that bounds the persistent kernel at ~1 PFLOP/s.  Here the two CTAs of a cluster share one tile of 256 weight rows x NT tokens:
// each loads its own 128 weight rows and its own half of the token rows by plain TMA copies whose bytes are counted on a barrier of rank 0 (no
// multicast), rank 0 issues M = 256 MMAs that read both CTAs' shared memory and write both CTAs' tensor memory.
//
// NT is any multiple of 16 up to 256, so that a prompt is cut into equal tiles instead of leaving the last one mostly empty: 777 rows are four
// tiles of 208 (256-row tiles: 1024 rows), 128 rows one of 128.  Accumulator rows are output columns and accumulator columns tokens: the epilogue
// turns 32 tokens at a time round in shared memory and writes (and reads residuals of) whole 16-byte words of a token's row.
// Few tiles but a long reduction: the pairs split K (units of (tile, split)) and leave fp32 partial sums in p.partial, which a
// second kernel adds up.
//
// Bound by what an SM can take in (32 KB per k-block and CTA at 256 tokens: ~78 KB per us) and, before a ring stage held two k-blocks, by
// the issuing thread (a barrier probe and a commit per k-block: 0.41 us whatever NT).  us, 256 x 256 tiles with tokens on the 256-row side and a k-block
// per stage -> this (gate/up 17920 x 1536, down 1536 x 8960 with its reduce kernel, vocabulary 151936 x 1536):
//    128 rows  gate/up 16.1 -> 13.9 (one-tile kernel there), vocabulary 96 -> 91;   256 rows 15.8 -> 16.6, 109 -> 106
//    512 rows  25.0 -> 24.6   down 22.2 -> 21.9   192 -> 185;    777 rows 43.2 -> 38.4   31.0 -> 25.4   339 -> 303
//   2048 rows  86.5 -> 79.7        72.8 -> 66.4   679 -> 637 (1.50 PFLOP/s, 0.90 of the cuBLAS burst)
// Measured and not used: two producer threads per operand (the epilogue then has 128 registers; with 168 it requests the next 32 tokens
// while it finishes 32: 2048 rows gate/up 88.3 -> 79.7), partial sums without that (down of 512 rows 24.9).
#include "gemm_epilogue.cuh"
#include "tc5.cuh"

namespace b200 {

// time-out code of the last failed wait of this kernel (reported through b200_debug_device_error)
__device__ int g_pair_error = 0;

namespace {

// warps: 0 token producer, 6 weight producer, 1 MMA (rank 0) and tensor memory, 2-5 and 7-10 two epilogue groups (every second 32 tokens)
constexpr int PR_ST = 3, PR_KPS = 2, PR_THREADS = 352;          // ring stages of two k-blocks
constexpr int PR_W = 128 * 128, PR_KB = 2 * PR_W, PR_STAGE = PR_KPS * PR_KB;   // a k-block: 128 weight rows, up to 128 token rows
constexpr int PR_CHUNK = 32, PR_BUF = PR_CHUNK * 128 * 2;        // 32 tokens x 128 output columns, 16-bit
constexpr int PR_SMEM = PR_ST * PR_STAGE + 4 * PR_BUF + 1024;

template <typename T>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(PR_THREADS, 1)
    gemm_pair_kernel(const __grid_constant__ CUtensorMap map_x, const __grid_constant__ CUtensorMap map_w, const __grid_constant__ Tc5Params p, const int nt,
                     const int tiles_t, const int n_tiles) {
  constexpr int ST = PR_ST;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  // full_bar / acc_empty are used in rank 0 only (its MMA thread waits on them); empty_bar / acc_full in both
  __shared__ __align__(8) uint64_t full_bar[ST], empty_bar[ST], acc_full[2], acc_empty[2];
  __shared__ uint32_t tmem_holder;
  __shared__ int failed;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = tc5::cluster_ctarank();
  const int pair = blockIdx.x >> 1, n_pairs = gridDim.x >> 1;
  const int KB = static_cast<int>((p.K + 63) / 64);
  const int n_units = n_tiles * p.splits;
  auto unit_kb0 = [&](int unit) { return (unit / n_tiles) * p.kb_per_split; };
  auto unit_nkb = [&](int unit) { const int k0 = unit_kb0(unit); return KB - k0 < p.kb_per_split ? KB - k0 : p.kb_per_split; };
  if (threadIdx.x == 0) {
    failed = 0;
    for (int s = 0; s < ST; ++s) { tc5::mbar_init(&full_bar[s], 2); tc5::mbar_init(&empty_bar[s], 1); }   // full: rank 0's two producers of the stage
    for (int b = 0; b < 2; ++b) { tc5::mbar_init(&acc_full[b], 1); tc5::mbar_init(&acc_empty[b], 16); }    // empty: eight epilogue warps of each CTA
    tc5::fence_barrier_init();
    tc5::prefetch_tensormap(&map_x);
    tc5::prefetch_tensormap(&map_w);
  }
  if (warp == 1) { tc5::tmem_alloc_pair(&tmem_holder, 512); tc5::tmem_relinquish_pair(); }
  tc5::tc_fence_before();
  __syncthreads();
  tc5::cluster_sync();   // the peer's barriers exist before anything arrives on them
  tc5::tc_fence_after();
  const uint32_t tmem_base = tmem_holder;
  pdl_trigger();
  auto dead = [&]() { return *reinterpret_cast<volatile int*>(&failed) != 0; };
  auto fail = [&](int code) { failed = 1; atomicExch(&g_pair_error, code); };
  const uint32_t ring_addr = tc5::smem_addr(smem), full0 = tc5::smem_addr(&full_bar[0]), empty0 = tc5::smem_addr(&empty_bar[0]);

  if (warp == 0 || warp == 6) {
    // ---- producers, one thread per operand (two each, in turn, where a stage was one k-block: a barrier wait behind a copy costs ~0.3 us) ----
    if (lane == 0) {
      const bool is_x = warp == 0;
      if (is_x || !(p.epilogue & B200_EPI_W_STATIC)) pdl_wait();
      const CUtensorMap* map = is_x ? &map_x : &map_w;
      const int rows = is_x ? nt >> 1 : 128;   // of this CTA
      const uint32_t lead_full0 = tc5::map_to_rank(full0, 0);
      int s = 0;
      uint32_t ph = 0, dst = ring_addr + (is_x ? PR_W : 0);
      const uint32_t dst0 = dst;
      bool alive = true;
      for (int unit = pair; unit < n_units && alive && !dead(); unit += n_pairs) {
        const int tile = unit % n_tiles;
        const int row0 = (is_x ? (tile % tiles_t) * nt : (tile / tiles_t) * 256) + static_cast<int>(rank) * rows;
        const int kb0 = unit_kb0(unit), kb1 = kb0 + unit_nkb(unit);
        for (int kb = kb0; kb < kb1; kb += PR_KPS) {
          {
            const int cnt = kb1 - kb < PR_KPS ? kb1 - kb : PR_KPS;
            if (!tc5::mbar_wait_a(empty0 + 8u * s, ph ^ 1u)) { fail(40); alive = false; break; }
            if (rank == 0) tc5::mbar_arrive_expect_tx_a(full0 + 8u * s, cnt * 2 * rows * 128);   // both CTAs' halves of this operand
#pragma unroll
            for (int j = 0; j < PR_KPS; ++j)
              if (j < cnt) tc5::tma_load_2d_pair(dst + j * PR_KB, map, lead_full0 + 8u * s, (kb + j) * 64, row0);
          }
          dst += PR_STAGE;
          if (++s == ST) { s = 0; ph ^= 1u; dst = dst0; }
        }
      }
    }
  } else if (warp == 1) {
    if (lane == 0 && rank == 0) {
      // ---- MMA issuer (rank 0 only) ----
      const uint32_t idesc = tc5::umma_idesc(256, nt, AbFormat<T>::value);
      const uint32_t ring_lo = tc5::desc_sw128_lo(ring_addr);
      const uint32_t acc_full0 = tc5::smem_addr(&acc_full[0]), acc_empty0 = tc5::smem_addr(&acc_empty[0]);
      int ti = 0, s = 0;
      uint32_t ph = 0, a_lo = ring_lo;
      bool alive = true;
      for (int unit = pair; unit < n_units && alive && !dead(); unit += n_pairs, ++ti) {
        const int b = ti & 1;
        if (!tc5::mbar_wait_a(acc_empty0 + 8u * b, ((ti >> 1) & 1) ^ 1)) { fail(41); break; }
        tc5::tc_fence_after();
        const uint32_t acc = tmem_base + b * 256;
        const int nkb = unit_nkb(unit);
        for (int kb = 0; kb < nkb; kb += PR_KPS) {
          if (!tc5::mbar_wait_a(full0 + 8u * s, ph)) { fail(42); alive = false; break; }
#pragma unroll
          for (int j = 0; j < PR_KPS; ++j)
            if (kb + j < nkb) tc5::umma_f16_kblock_pair(acc, a_lo + j * (PR_KB >> 4), a_lo + ((j * PR_KB + PR_W) >> 4), idesc, kb + j);
          tc5::umma_commit_pair(empty0 + 8u * s);   // frees the stage in both CTAs
          a_lo += PR_STAGE >> 4;
          if (++s == ST) { s = 0; ph ^= 1u; a_lo = ring_lo; }
        }
        if (!alive) break;
        tc5::umma_commit_pair(acc_full0 + 8u * b);
      }
    }
  } else {
    // ---- epilogue: this CTA's 128 output columns, two groups of four warps that take 32 tokens in turn ----
    const int q = warp & 3, g = warp >= 7 ? 1 : 0, t = q * 32 + lane;   // t: accumulator row, output column of the block
    uint8_t* const buf = smem + PR_ST * PR_STAGE + g * 2 * PR_BUF;
    pdl_wait();
    const bool glu = (p.epilogue & B200_EPI_GLU) != 0, silu = (p.epilogue & B200_EPI_SILU_MUL) != 0, relu = (p.epilogue & B200_EPI_RELU) != 0;
    const T* const res = static_cast<const T*>(p.residual);
    const bool res_vec = res && p.ldr % 8 == 0 && p.N % 8 == 0 && (reinterpret_cast<uintptr_t>(res) & 15u) == 0;
    const uint32_t lead_acc_empty0 = tc5::map_to_rank(tc5::smem_addr(&acc_empty[0]), 0);
    // the group's four warps leave together: they meet at a barrier of their own
    auto any = [&](bool v) {
      uint32_t x = v;
      asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.u32 q, %0, 0;\n\tbar.red.or.pred p, %1, 128, q;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "+r"(x) : "r"(1 + g) : "memory");
      return x != 0;
    };
    int ti = 0, round = 0;
    for (int unit = pair; unit < n_units; unit += n_pairs, ++ti) {
      const int b = ti & 1, tile = unit % n_tiles;
      const int64_t n0 = static_cast<int64_t>(tile / tiles_t) * 256 + rank * 128, m0 = static_cast<int64_t>(tile % tiles_t) * nt;   // of this CTA
      const float bias = p.bias && p.splits == 1 && n0 + t < p.N ? load_as_f32(p.bias, n0 + t, p.bias_dtype) : 0.f;
      const bool ok = tc5::mbar_wait(&acc_full[b], (ti >> 1) & 1);
      if (any(!ok || dead())) { if (!ok) fail(43); break; }
      tc5::tc_fence_after();
      const uint32_t t_row = tmem_base + b * 256 + (static_cast<uint32_t>(q * 32) << 16);
      if (p.splits > 1) {
        // raw partial sums of this unit's k-range, 32 tokens in flight while 32 are stored: a warp writes 128 consecutive bytes per token
        float* dst = p.partial + (static_cast<int64_t>(unit / n_tiles) * p.M + m0 + PR_CHUNK * g) * p.N + n0 + t;
        const int tokens = n0 + t < p.N ? static_cast<int>(p.M - m0 < nt ? p.M - m0 : nt) : 0;
        auto put = [&](const float (&v)[PR_CHUNK], int c) {
          float* d = dst;
#pragma unroll
          for (int j = 0; j < PR_CHUNK; ++j, d += p.N)
            if (c + j < tokens) *d = v[j];
          dst += 2 * PR_CHUNK * p.N;
        };
        float va[PR_CHUNK], vb[PR_CHUNK];
        __syncwarp();
        tc5::tmem_ld_32x32_async(t_row + PR_CHUNK * g, va);
#pragma unroll 1
        for (int c = PR_CHUNK * g; c < nt; c += 4 * PR_CHUNK) {
          tc5::tmem_ld_wait();
          if (c + 2 * PR_CHUNK < nt) tc5::tmem_ld_32x32_async(t_row + c + 2 * PR_CHUNK, vb);
          put(va, c);
          __syncwarp();
          tc5::tmem_ld_wait();
          if (c + 4 * PR_CHUNK < nt) tc5::tmem_ld_32x32_async(t_row + c + 4 * PR_CHUNK, va);
          if (c + 2 * PR_CHUNK < nt) put(vb, c + 2 * PR_CHUNK);
          __syncwarp();
        }
      } else {
        float v[PR_CHUNK];
        __syncwarp();
        tc5::tmem_ld_32x32_async(t_row + PR_CHUNK * g, v);
#pragma unroll 1
        for (int c = PR_CHUNK * g; c < nt; c += 2 * PR_CHUNK) {
          const int cnt = nt - c < PR_CHUNK ? nt - c : PR_CHUNK;
          const int tokens = static_cast<int>(p.M - m0 - c < cnt ? (p.M - m0 - c < 0 ? 0 : p.M - m0 - c) : cnt);   // that exist
          // 16-byte words of the result that this thread finishes: token i / 16, columns 8 (i % 16) .. (gated: i / 8, i % 8); residual requested now
          uint4 r[4];
          if (res_vec) {
#pragma unroll
            for (int k = 0; k < 4; ++k) {
              const int i = t + 128 * k, j = i >> 4;
              const int64_t n = n0 + 8 * (i & 15);
              r[k] = j < tokens && n < p.N ? __ldg(reinterpret_cast<const uint4*>(res + (m0 + c + j) * p.ldr + n)) : make_uint4(0u, 0u, 0u, 0u);
            }
          }
          T* const turn = reinterpret_cast<T*>(buf + (round & 1) * PR_BUF);
          ++round;
          tc5::tmem_ld_wait();
#pragma unroll
          for (int j = 0; j < PR_CHUNK; ++j) turn[j * 128 + t] = from_f32<T>(v[j] + bias);
          if (c + 2 * PR_CHUNK < nt) tc5::tmem_ld_32x32_async(t_row + c + 2 * PR_CHUNK, v);   // the next 32 tokens, while these are finished
          // (two buffers: whoever writes one again has passed the barrier behind which everybody had read it)
          asm volatile("bar.sync %0, 128;" ::"r"(1 + g) : "memory");
          if (glu) {
#pragma unroll
            for (int k = 0; k < 2; ++k) {
              const int i = t + 128 * k, j = i >> 3, cc = 8 * (i & 7);
              if (j < tokens && n0 < p.N) {   // (N is a multiple of 128: the block is whole)
                float gt[8], up[8];
                unpack8<T>(*reinterpret_cast<const uint4*>(turn + j * 128 + cc), gt);
                unpack8<T>(*reinterpret_cast<const uint4*>(turn + j * 128 + 64 + cc), up);
#pragma unroll
                for (int e = 0; e < 8; e += 2) {
                  float a = silu_f32(gt[e]), d = silu_f32(gt[e + 1]);
                  round2<T>(a, d);
                  gt[e] = a * up[e]; gt[e + 1] = d * up[e + 1];
                }
                store_cols<T, 8>(static_cast<T*>(p.out) + (m0 + c + j) * p.ldo + n0 / 2 + cc, gt, 8);
              }
            }
          } else {
#pragma unroll
            for (int k = 0; k < 4; ++k) {
              const int i = t + 128 * k, j = i >> 4;
              const int64_t n = n0 + 8 * (i & 15), m = m0 + c + j;
              if (j >= tokens || n >= p.N) continue;
              const int left = static_cast<int>(p.N - n < 8 ? p.N - n : 8);
              float f[8];
              unpack8<T>(*reinterpret_cast<const uint4*>(turn + j * 128 + 8 * (i & 15)), f);
              if (res) {
                float rf[8];
                if (res_vec) unpack8<T>(r[k], rf);
                else load_cols<T, 8>(res, p.ldr, m, n, left, rf);
#pragma unroll
                for (int e = 0; e < 8; ++e) f[e] += rf[e];
              }
              if (relu) {
#pragma unroll
                for (int e = 0; e < 8; ++e) f[e] = fmaxf(f[e], 0.f);
              }
              if (silu) {
                float x[8];
                load_cols<T, 8>(static_cast<const T*>(p.aux), p.ldaux, m, n, left, x);
#pragma unroll
                for (int e = 0; e < 8; ++e) f[e] = round_as<T>(silu_f32(round_as<T>(f[e]))) * x[e];
              }
              store_cols<T, 8>(static_cast<T*>(p.out) + m * p.ldo + n, f, left);
            }
          }
          __syncwarp();
        }
      }
      tc5::tc_fence_before();
      __syncwarp();
      if (lane == 0) tc5::mbar_arrive_cluster(lead_acc_empty0 + 8u * b);   // this warp has drained its share of the accumulator
    }
  }
  tc5::tc_fence_before();
  __syncthreads();
  tc5::cluster_sync();   // neither CTA leaves while the other may still signal its barriers or read its shared memory
  if (warp == 1) { tc5::tc_fence_after(); tc5::tmem_dealloc_pair(tmem_base, 512); }
}

template <typename T> int launch_pair_t(const Tc5Args& a, Tc5Params p, cudaStream_t st) {
  static PerDevice<bool> configured_on;
  bool* configured = configured_on.slot();
  if (!configured) return B200_ENOTSUP;
  if (!*configured) {
    if (cudaFuncSetAttribute(gemm_pair_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, PR_SMEM) != cudaSuccess) {
      cudaGetLastError();
      return B200_ENOTSUP;
    }
    *configured = true;
  }
  const int64_t tiles_t = ceil_div(a.M, 256);
  const int nt = static_cast<int>(ceil_div(ceil_div(a.M, tiles_t), 16) * 16);
  const int64_t tiles = ceil_div(a.M, nt) * ceil_div(a.N, 256), units = tiles * p.splits;
  if (units >= (1ll << 30)) return B200_ENOTSUP;
  auto map = [&](CUtensorMap* m, const void* base, int64_t rows, int64_t ld, int box_rows) {
    const uint64_t dims[2] = {static_cast<uint64_t>(a.K), static_cast<uint64_t>(rows)}, str[1] = {static_cast<uint64_t>(ld) * 2};
    const uint32_t box[2] = {64, static_cast<uint32_t>(box_rows)};
    return tma_encode_sw128(m, a.dtype, 2, base, dims, str, box);
  };
  CUtensorMap mx, mw;
  if (!map(&mx, a.A, a.M, a.lda, nt / 2) || !map(&mw, a.W, a.N, a.ldw, 128)) return B200_ENOTSUP;
  const int pairs = static_cast<int>(units < sm_count() / 2 ? units : sm_count() / 2);
  launch_pdl(gemm_pair_kernel<T>, dim3(2 * pairs), dim3(PR_THREADS), PR_SMEM, st, mx, mw, p, nt, static_cast<int>(ceil_div(a.M, nt)), static_cast<int>(tiles));
  B200_CHECK_LAUNCH("gemm_pair_kernel");
  return B200_OK;
}

}  // namespace

int gemm_pair(const Tc5Args& a, const Tc5Params& p, cudaStream_t st) {
  return a.dtype == B200_BF16 ? launch_pair_t<__nv_bfloat16>(a, p, st) : launch_pair_t<__half>(a, p, st);
}

int gemm_pair_error(bool clear) {
  int v = 0;
  if (cudaMemcpyFromSymbol(&v, g_pair_error, sizeof(int)) != cudaSuccess) return -1;
  if (clear && v) {
    const int zero = 0;
    cudaMemcpyToSymbol(g_pair_error, &zero, sizeof(int));
  }
  return v;
}

}  // namespace b200

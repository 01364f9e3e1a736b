// Linear layers on CTA pairs (cta_group::2), weights on the 256-row side of the MMA, tokens on its N side.
//
// A 128 x 256 tile per CTA needs 48 KB of operands per 4.2 MFLOP; at the rate the L2 feeds the SMs (measured ~11 TB/s over
// all SMs) that bounds the persistent kernel at ~1 PFLOP/s.  Here the two CTAs of a cluster share one tile of 256 weight rows x NT tokens:
// each loads its own 128 weight rows and its own half of the token rows by plain TMA copies whose bytes are counted on a barrier of rank 0 (no
// multicast), rank 0 issues M = 256 MMAs that read both CTAs' shared memory and write both CTAs' tensor memory.
//
// NT is any multiple of 16 up to 256, so that a prompt is cut into equal tiles instead of leaving the last one mostly empty: 777 rows are four
// tiles of 208 (256-row tiles: 1024 rows), 128 rows one of 128.  Accumulator rows are output columns and accumulator columns tokens: the epilogue
// turns 32 tokens at a time round in shared memory, a word for two tokens of a column, and writes (and reads residuals of) whole 16-byte words of a
// token's row; where rows are no such words a warp writes 32 columns of a token straight from its registers.
// Few tiles but a long reduction: the pairs split K (units of (tile, split)) and leave fp32 partial sums in p.partial, which a
// second kernel adds up.
//
// Bound by what an SM can take in (32 KB per k-block and CTA at 256 tokens: ~78 KB per us) and, before a ring stage held two k-blocks, by
// the issuing thread (a barrier probe and a commit per k-block: 0.41 us whatever NT).  us, 256 x 256 tiles with tokens on the 256-row side and a k-block
// per stage -> this, weights from memory (gate/up 17920 x 1536, down 1536 x 8960 with its reduce kernel, vocabulary 151936 x 1536):
//     65 rows  gate/up 15.1 -> 12.8, 128 rows 16.1 -> 13.4 (one-tile kernel there), vocabulary 96 -> 91;   256 rows 16.3 -> 16.1, 134 -> 128
//    512 rows  26.2 -> 24.8   down 22.2 -> 21.9   192 -> 185;    777 rows 45.1 -> 38.6   29.4 -> 25.1   339 -> 303
//   2048 rows  86.5 -> 79.7        60.0 -> 53.2   679 -> 637 (1.50 PFLOP/s, 0.90 of the cuBLAS burst)
//   256 x 12288 x 1536 plain 17.3 -> 15.4, with a residual 18.8 -> 15.9; 2048 x 12288 69.6 -> 61.6, 88 -> 68; 512 x 9999 81 -> 25, 91 -> 38
// By single tokens and through fp32 the epilogue cost more than it saved in one wave of 256-token tiles (gate/up of 256 rows 16.9, 256 x 9352 x 1536
// with a residual 15.7 -> 17.8, here 14.9).  Measured and not used: two producer threads per operand (the epilogue then has 128 registers; with
// 168 it requests the next 32 tokens while it finishes 32: 2048 rows gate/up 88.3 -> 79.7), partial sums without that (down of 512 rows 24.9), staging
// the next 32 tokens before the 32 in shared memory are finished (plain epilogues 1 to 2 % slower, gated ones level).
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

// What a tile's results become: one kernel each, since a launch is a few tiles long and fetches its epilogue's code while it runs (gate/up of 65
// rows: 13.0 us, with the code of the other forms between 13.5)
enum class PairForm {
  SPLIT,   // fp32 partial sums
  GATED,   // silu(gate) * up
  WORDS,   // bias, residual, ReLU, silu(.) * aux; rows of whole 16-byte words
  ANY      // the same, any rows
};

template <typename T, PairForm FORM>
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
    const bool silu = (p.epilogue & B200_EPI_SILU_MUL) != 0, relu = (p.epilogue & B200_EPI_RELU) != 0;
    const T* const res = static_cast<const T*>(p.residual);
    const T* const early = res ? res : silu ? static_cast<const T*>(p.aux) : nullptr;
    const int64_t early_ld = res ? p.ldr : p.ldaux;
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
      const float bias = FORM != PairForm::SPLIT && p.bias && n0 + t < p.N ? load_as_f32(p.bias, n0 + t, p.bias_dtype) : 0.f;
      const bool ok = tc5::mbar_wait(&acc_full[b], (ti >> 1) & 1);
      if (any(!ok || dead())) { if (!ok) fail(43); break; }
      tc5::tc_fence_after();
      const uint32_t t_row = tmem_base + b * 256 + (static_cast<uint32_t>(q * 32) << 16);
      if constexpr (FORM == PairForm::SPLIT) {
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
          if constexpr (FORM == PairForm::ANY) {   // a warp writes (and reads) 32 consecutive columns of a token, the reads of a chunk in flight together
            const int64_t n = n0 + t;
            auto there = [&](int j) { return j < tokens && n < p.N; };
            auto column = [&](const void* base, int64_t ld, T (&x)[PR_CHUNK]) {
#pragma unroll
              for (int j = 0; j < PR_CHUNK; ++j) x[j] = there(j) ? static_cast<const T*>(base)[(m0 + c + j) * ld + n] : from_f32<T>(0.f);
            };
            T x[PR_CHUNK];
            if (res) column(res, p.ldr, x);
            tc5::tmem_ld_wait();
#pragma unroll
            for (int j = 0; j < PR_CHUNK; ++j) v[j] += bias;
            if (res) {
#pragma unroll
              for (int j = 0; j < PR_CHUNK; ++j) v[j] = round_as<T>(v[j]) + to_f32<T>(x[j]);
            }
            if (relu) {
#pragma unroll
              for (int j = 0; j < PR_CHUNK; ++j) v[j] = fmaxf(v[j], 0.f);
            }
            if (silu) {
              column(p.aux, p.ldaux, x);
#pragma unroll
              for (int j = 0; j < PR_CHUNK; ++j) v[j] = round_as<T>(silu_f32(round_as<T>(v[j]))) * to_f32<T>(x[j]);
            }
#pragma unroll
            for (int j = 0; j < PR_CHUNK; ++j)
              if (there(j)) static_cast<T*>(p.out)[(m0 + c + j) * p.ldo + n] = from_f32<T>(v[j]);
            __syncwarp();
            if (c + 2 * PR_CHUNK < nt) tc5::tmem_ld_32x32_async(t_row + c + 2 * PR_CHUNK, v);
            continue;
          }
          // 16-byte words of the result that this thread finishes: two items of two tokens 2 (i / 16) .. and columns 8 (i % 16) ..; what is read with
          // them (residual, else the other factor) is requested now
          uint4 r[4];
          if (FORM == PairForm::WORDS && early) {
#pragma unroll
            for (int k = 0; k < 4; ++k) {
              const int i = t + 128 * (k >> 1), j = 2 * (i >> 4) + (k & 1);
              const int64_t n = n0 + 8 * (i & 15);
              r[k] = j < tokens && n < p.N ? __ldg(reinterpret_cast<const uint4*>(early + (m0 + c + j) * early_ld + n)) : make_uint4(0u, 0u, 0u, 0u);
            }
          }
          // [pair of tokens][column], a word each: half the stores of single values, and no two of a warp in one bank
          uint32_t* const pairs = reinterpret_cast<uint32_t*>(buf + (round & 1) * PR_BUF);
          ++round;
          tc5::tmem_ld_wait();
#pragma unroll
          for (int j = 0; j < PR_CHUNK; j += 2) pairs[(j >> 1) * 128 + t] = pack2<T>(v[j] + bias, v[j + 1] + bias);
          if (c + 2 * PR_CHUNK < nt) tc5::tmem_ld_32x32_async(t_row + c + 2 * PR_CHUNK, v);   // the next 32 tokens, while these are finished
          // (two buffers: whoever writes one again has passed the barrier behind which everybody had read it)
          asm volatile("bar.sync %0, 128;" ::"r"(1 + g) : "memory");
          const int turned = (t >> 2) & 1;   // half of the threads take their words in the other order: no bank twice
          if constexpr (FORM == PairForm::GATED) {
            const int j = 2 * (t >> 3), cc = 8 * (t & 7);
            if (j < tokens && n0 < p.N) {   // (N is a multiple of 128: the block is whole)
              uint32_t lo[2][2], hi[2][2];   // of the first and the second token: four columns at a time
#pragma unroll
              for (int k = 0; k < 2; ++k) {
                const uint32_t* src = pairs + (j >> 1) * 128 + cc + 4 * (k ^ turned);
                const uint4 gw = *reinterpret_cast<const uint4*>(src), uw = *reinterpret_cast<const uint4*>(src + 64);
                const uint32_t gv[4] = {gw.x, gw.y, gw.z, gw.w}, uv[4] = {uw.x, uw.y, uw.z, uw.w};
                float f0[4], f1[4];
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                  float a, d, x, y;
                  unpack2<T>(gv[e], a, d);
                  unpack2<T>(uv[e], x, y);
                  a = silu_f32(a); d = silu_f32(d);
                  round2<T>(a, d);
                  f0[e] = a * x; f1[e] = d * y;
                }
                lo[k][0] = pack2<T>(f0[0], f0[1]); lo[k][1] = pack2<T>(f0[2], f0[3]);
                hi[k][0] = pack2<T>(f1[0], f1[1]); hi[k][1] = pack2<T>(f1[2], f1[3]);
              }
              T* const dst = static_cast<T*>(p.out) + (m0 + c + j) * p.ldo + n0 / 2 + cc;
              auto put = [&](T* d, const uint32_t (&w)[2][2]) {
                const uint4 o = turned ? make_uint4(w[1][0], w[1][1], w[0][0], w[0][1]) : make_uint4(w[0][0], w[0][1], w[1][0], w[1][1]);
                float f[8];
                if (p.ldo % 8 == 0 && (reinterpret_cast<uintptr_t>(p.out) & 15u) == 0) { *reinterpret_cast<uint4*>(d) = o; return; }
                unpack8<T>(o, f);
                store_cols<T, 8>(d, f, 8);
              };
              put(dst, lo);
              if (j + 1 < tokens) put(dst + p.ldo, hi);
            }
          } else {
#pragma unroll
            for (int k = 0; k < 2; ++k) {
              const int i = t + 128 * k, j = 2 * (i >> 4);
              const int64_t n = n0 + 8 * (i & 15);
              if (j >= tokens || n >= p.N) continue;
              const uint32_t* src = pairs + (j >> 1) * 128 + 8 * (i & 15);
              const uint4 w0 = *reinterpret_cast<const uint4*>(src + 4 * turned), w1 = *reinterpret_cast<const uint4*>(src + 4 * (turned ^ 1));
              const uint4 a = turned ? w1 : w0, d = turned ? w0 : w1;
#pragma unroll
              for (int e = 0; e < 2; ++e) {   // the first and the second token
                if (j + e >= tokens) continue;
                const int64_t m = m0 + c + j + e;
                const uint32_t half = e ? 0x7632u : 0x5410u;
                uint32_t o[4] = {__byte_perm(a.x, a.y, half), __byte_perm(a.z, a.w, half), __byte_perm(d.x, d.y, half), __byte_perm(d.z, d.w, half)};
                T* const dst = static_cast<T*>(p.out) + m * p.ldo + n;
                const uint32_t rv[4] = {r[2 * k + e].x, r[2 * k + e].y, r[2 * k + e].z, r[2 * k + e].w};
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                  if (res) o[q] = add2<T>(o[q], rv[q]);   // (the exact sum of two 16-bit numbers rounded once: what an fp32 addition and its rounding give)
                  if (relu) o[q] = relu2<T>(o[q]);
                }
                if (silu) {
                  float f[8], x[8];
                  unpack8<T>(make_uint4(o[0], o[1], o[2], o[3]), f);
                  unpack8<T>(res ? __ldg(reinterpret_cast<const uint4*>(static_cast<const T*>(p.aux) + m * p.ldaux + n)) : r[2 * k + e], x);
#pragma unroll
                  for (int q = 0; q < 8; q += 2) {
                    float y0 = silu_f32(f[q]), y1 = silu_f32(f[q + 1]);
                    round2<T>(y0, y1);
                    o[q >> 1] = pack2<T>(y0 * x[q], y1 * x[q + 1]);
                  }
                }
                *reinterpret_cast<uint4*>(dst) = make_uint4(o[0], o[1], o[2], o[3]);
              }
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

template <typename T, PairForm FORM> int launch_pair_t(const Tc5Args& a, Tc5Params p, cudaStream_t st) {
  static PerDevice<bool> configured_on;
  bool* configured = configured_on.slot();
  if (!configured) return B200_ENOTSUP;
  if (!*configured) {
    if (cudaFuncSetAttribute(gemm_pair_kernel<T, FORM>, cudaFuncAttributeMaxDynamicSharedMemorySize, PR_SMEM) != cudaSuccess) {
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
  launch_pdl(gemm_pair_kernel<T, FORM>, dim3(2 * pairs), dim3(PR_THREADS), PR_SMEM, st, mx, mw, p, nt, static_cast<int>(ceil_div(a.M, nt)), static_cast<int>(tiles));
  B200_CHECK_LAUNCH("gemm_pair_kernel");
  return B200_OK;
}

template <typename T> int launch_pair_form(const Tc5Args& a, const Tc5Params& p, cudaStream_t st) {
  if (p.splits > 1) return launch_pair_t<T, PairForm::SPLIT>(a, p, st);
  if (p.epilogue & B200_EPI_GLU) return launch_pair_t<T, PairForm::GATED>(a, p, st);
  const bool words = p.N % 8 == 0 && p.ldo % 8 == 0 && aligned16(p.out) && (!p.residual || (p.ldr % 8 == 0 && aligned16(p.residual))) &&
                     (!(p.epilogue & B200_EPI_SILU_MUL) || (p.ldaux % 8 == 0 && aligned16(p.aux)));
  return words ? launch_pair_t<T, PairForm::WORDS>(a, p, st) : launch_pair_t<T, PairForm::ANY>(a, p, st);
}

}  // namespace

int gemm_pair(const Tc5Args& a, const Tc5Params& p, cudaStream_t st) {
  return a.dtype == B200_BF16 ? launch_pair_form<__nv_bfloat16>(a, p, st) : launch_pair_form<__half>(a, p, st);
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

// 3x3 / stride-1 / padding-1 convolutions over channels-last images whose rows stay in shared memory.
//
// As an implicit GEMM with an im2col box per filter tap, every input pixel enters an SM nine times: 144 KB of boxes per 128
// outputs and 64 channels, and the rate at which L2 feeds the SMs (~70 KB per us and SM) is what such a layer takes.  Here a tile is TR
// output rows of one image, and the TR + 2 input rows that it needs arrive once per 64 channels, by one TMA box that starts one
// pixel left of the image: pixels outside arrive as zeros, so that the box is the zero-padded image with a row pitch of
// W + 1 (the pixel behind a row's end is the one before the next row's start).  In that flat order tap (r, s) of every output
// position is its own position + r (W + 1) + s: a pixel's 64 channels are one 128-byte row of a K-major operand with the 128-byte
// swizzle - which is a function of the address - and the MMA of a tap reads the same rows from r (W + 1) + s rows further on.
// One position per row and image row is padding and is computed for nothing (W of W + 1), as are the accumulator rows
// beyond TR (W + 1) <= 128: 112 of 128 rows count for 56 and 28 wide images, 98 on average for 14.
// - A = input rows per 64 channels, in a ring.  Weights: resident where they fit (64 channels to 64), else a filter row
//   (three taps) per stage of a second ring; a unit of MT tiles shares each weight stage.
// - Accumulators are double-buffered in tensor memory; eight epilogue warps (two per lane quarter, half the columns each) add bias and
//   residual, apply ReLU and write the valid positions, closed up, to a C buffer that one thread stores by TMA (residual
//   tiles come into the same buffers beforehand).
// - With resident weights two threads issue the MMAs of the tiles in turn: probes and commits of one (~0.4 us per tile) run
//   beside the other's MMAs.
// Busiest unit, 256 images: the shared-memory pipe with the MMAs' operand reads, 64 % of the active cycles for 64 channels (tensor pipe 43 %) and
// 62 % (62 %) for 128, where the last wave leaves a fifth of the time empty besides; L2 14 %, DRAM 23 % and below.  What fills the
// rest is not measured.  us per layer, im2col boxes -> this: 64 channels, 56 x 56, 256 / 32 / 16 images 144 -> 73, 24 -> 14, 15 -> 10;
// 128 channels, 28 x 28 86 -> 63, 17.7 -> 13.8, 15.0 -> 9.2; 256 channels, 14 x 14, 32 images 24 -> 13.
#include "gemm_epilogue.cuh"
#include "tc5.cuh"

namespace b200 {

// time-out code of the last failed wait of this kernel (reported through b200_debug_device_error)
__device__ int g_rows_error = 0;

namespace {

constexpr int CR_THREADS = 13 * 32;   // warps: 0 input rows, 1-2 MMA, 3 weights, 4-11 epilogue, 12 store and residual
constexpr int CR_LIMIT = 227 * 1024 - 1024;
template <int MT> constexpr int CR_BUFS = MT == 1 ? 2 : 1;   // C buffers: with two tiles per unit the rings need the room, and the products outlast two epilogues

struct ConvRowsParams {
  const void* bias; int bias_dtype, relu, has_res;
  int H, W, O, TR, pitch, NKB;
  int tiles_img, n_tiles, n_mu, n_units;      // tiles per image, tiles, units of MT tiles, units over all column tiles
  int a_st, a_sub, a_stage, w_st, w_off, c_off;
};

__device__ __forceinline__ void cr_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(tc5::smem_addr(bar)) : "memory");
}

template <typename T, int BN, int MT, bool WRES>
__global__ void __launch_bounds__(CR_THREADS, 1)
    conv_rows_kernel(const __grid_constant__ CUtensorMap map_x, const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_r,
                     const __grid_constant__ CUtensorMap map_o, const __grid_constant__ ConvRowsParams p) {
  constexpr int W_TAP = BN * 128, W_STAGE = 3 * W_TAP;   // weights of one tap / filter row and 64 channels
  constexpr int CB = 128 * BN * 2, NCB = CR_BUFS<MT>, MAX_A = 8, MAX_W = 8, ISSUERS = WRES ? 2 : 1;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  uint8_t* const w_s = smem + p.w_off;
  uint8_t* const cbuf = smem + p.c_off;
  __shared__ __align__(8) uint64_t a_full[MAX_A], a_empty[MAX_A], w_full[MAX_W], w_empty[MAX_W], acc_full[2], acc_empty[2], c_full[NCB], c_ready[NCB], c_free[NCB];
  __shared__ uint32_t tmem_holder;
  __shared__ int failed;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    failed = 0;
    for (int s = 0; s < MAX_A; ++s) { tc5::mbar_init(&a_full[s], 1); tc5::mbar_init(&a_empty[s], 1); }
    for (int s = 0; s < MAX_W; ++s) { tc5::mbar_init(&w_full[s], 1); tc5::mbar_init(&w_empty[s], 1); }
    for (int s = 0; s < 2; ++s) { tc5::mbar_init(&acc_full[s], 1); tc5::mbar_init(&acc_empty[s], 8); }
    for (int s = 0; s < NCB; ++s) { tc5::mbar_init(&c_full[s], 1); tc5::mbar_init(&c_ready[s], 8); tc5::mbar_init(&c_free[s], 1); }
    tc5::fence_barrier_init();
    tc5::prefetch_tensormap(&map_x);
    tc5::prefetch_tensormap(&map_w);
    tc5::prefetch_tensormap(&map_o);
    if (p.has_res) tc5::prefetch_tensormap(&map_r);
  }
  if (warp == 1) { tc5::tmem_alloc(&tmem_holder, 2 * MT * BN); tc5::tmem_relinquish(); }
  // the pixel behind the last row of a window, which no box writes, is padding like those between the rows
  for (int i = threadIdx.x; i < p.a_st * MT * 8; i += CR_THREADS)
    *reinterpret_cast<uint4*>(smem + (i >> 3) / MT * p.a_stage + (i >> 3) % MT * p.a_sub + (p.TR + 2) * p.pitch * 128 + (i & 7) * 16) = make_uint4(0u, 0u, 0u, 0u);
  tc5::fence_proxy_async();
  tc5::tc_fence_before();
  __syncthreads();
  tc5::tc_fence_after();
  const uint32_t tmem_base = tmem_holder;
  pdl_trigger();
  auto dead = [&]() { return *reinterpret_cast<volatile int*>(&failed) != 0; };
  auto fail = [&](int code) { failed = 1; atomicExch(&g_rows_error, code); };
  const int units = static_cast<int>(blockIdx.x) < p.n_units ? (p.n_units - static_cast<int>(blockIdx.x) + static_cast<int>(gridDim.x) - 1) / static_cast<int>(gridDim.x) : 0;   // of this CTA
  // tile t of unit i: image and first output row; false past the last tile
  auto tile_of = [&](int i, int t, int& n, int& h0, int& n0) {
    const int unit = blockIdx.x + i * gridDim.x, col = unit / p.n_mu, tile = (unit - col * p.n_mu) * MT + t;
    n = tile / p.tiles_img;
    h0 = (tile - n * p.tiles_img) * p.TR;
    n0 = col * BN;
    return tile < p.n_tiles;
  };

  if (warp == 0) {
    if (lane == 0) {   // ---- input rows ----
      pdl_wait();
      int s = 0, it = 0;
      uint32_t ph = 1;
      const uint32_t bytes = static_cast<uint32_t>((p.TR + 2) * p.pitch * 128);
      bool alive = true;
      for (int i = 0; i < units && alive; ++i) {
        int n[MT], h0[MT], n0, cnt = 0;
#pragma unroll
        for (int t = 0; t < MT; ++t) cnt += tile_of(i, t, n[t], h0[t], n0);
        for (int kb = 0; kb < p.NKB; ++kb, ++it) {
          if (!tc5::mbar_wait(&a_empty[s], ph)) { fail(60); alive = false; break; }
          if (dead()) { alive = false; break; }
          tc5::mbar_arrive_expect_tx(&a_full[s], bytes * cnt);
#pragma unroll
          for (int t = 0; t < MT; ++t)
            if (t < cnt) tc5::tma_load_4d(smem + s * p.a_stage + t * p.a_sub, &map_x, &a_full[s], kb * 64, -1, h0[t] - 1, n[t]);
          if (++s == p.a_st) { s = 0; ph ^= 1u; }
        }
      }
      if (dead())
        for (int i = it > p.a_st ? it - p.a_st : 0; i < it; ++i) tc5::mbar_wait(&a_full[i % p.a_st], (i / p.a_st) & 1, 1u << 16);
    }
  } else if (warp == 3) {
    if (lane == 0) {   // ---- weights: column block tap * C + 64 kb of [O][9 C] ----
      pdl_wait();
      const int C = p.NKB * 64;
      if (WRES) {
        if (units > 0) {
          tc5::mbar_arrive_expect_tx(&w_full[0], 9 * W_TAP);
          for (int tap = 0; tap < 9; ++tap) tc5::tma_load_2d(w_s + tap * W_TAP, &map_w, &w_full[0], tap * C, 0);
          if (dead()) tc5::mbar_wait(&w_full[0], 0, 1u << 16);
        }
      } else {
        int s = 0, it = 0;
        uint32_t ph = 1;
        bool alive = true;
        for (int i = 0; i < units && alive; ++i) {
          int n, h0, n0;
          tile_of(i, 0, n, h0, n0);
          for (int kr = 0; kr < 3 * p.NKB; ++kr, ++it) {
            const int kb = kr / 3, r = kr - 3 * kb;
            if (!tc5::mbar_wait(&w_empty[s], ph)) { fail(61); alive = false; break; }
            if (dead()) { alive = false; break; }
            tc5::mbar_arrive_expect_tx(&w_full[s], W_STAGE);
#pragma unroll
            for (int c = 0; c < 3; ++c) tc5::tma_load_2d(w_s + s * W_STAGE + c * W_TAP, &map_w, &w_full[s], (3 * r + c) * C + kb * 64, n0);
            if (++s == p.w_st) { s = 0; ph ^= 1u; }
          }
        }
        if (dead())
          for (int i = it > p.w_st ? it - p.w_st : 0; i < it; ++i) tc5::mbar_wait(&w_full[i % p.w_st], (i / p.w_st) & 1, 1u << 16);
      }
    }
  } else if (warp < 3) {
    const int id = warp - 1;
    if (lane == 0 && id < ISSUERS) {   // ---- MMA issuers ----
      constexpr uint32_t idesc = tc5::umma_idesc(128, BN, AbFormat<T>::value);
      const uint32_t a_lo0 = tc5::desc_sw128_lo(tc5::smem_addr(smem)), w_lo0 = tc5::desc_sw128_lo(tc5::smem_addr(w_s));
      const uint32_t row = static_cast<uint32_t>(p.pitch) * 8u;   // a filter row further: pitch rows of 128 bytes
      int s = id, ws = 0;            // (the ring has an even number of stages where two threads take turns: each stage is one thread's)
      uint32_t ph = 0, wph = 0;
      bool alive = true;
      if (WRES && units > 0 && !tc5::mbar_wait(&w_full[0], 0)) { fail(62); alive = false; }
      for (int i = id; i < units && alive && !dead(); i += ISSUERS) {
        const int b = i & 1;
        if (!tc5::mbar_wait(&acc_empty[b], ((i >> 1) & 1) ^ 1)) { fail(63); break; }
        const uint32_t acc = tmem_base + b * MT * BN;
        for (int kb = 0; kb < p.NKB && alive; ++kb) {
          if (!tc5::mbar_wait(&a_full[s], ph)) { fail(64); alive = false; break; }
          tc5::tc_fence_after();
          const uint32_t a_lo = a_lo0 + s * (p.a_stage >> 4);
#pragma unroll 1
          for (int r = 0; r < 3; ++r) {
            uint32_t w_lo = w_lo0 + r * (W_STAGE >> 4);
            if (!WRES) {
              if (!tc5::mbar_wait(&w_full[ws], wph)) { fail(65); alive = false; break; }
              tc5::tc_fence_after();
              w_lo = w_lo0 + ws * (W_STAGE >> 4);
            }
#pragma unroll
            for (int c = 0; c < 3; ++c)
#pragma unroll
              for (int t = 0; t < MT; ++t)
                tc5::umma_f16_kblock(acc + t * BN, a_lo + t * (p.a_sub >> 4) + r * row + c * 8, w_lo + c * (W_TAP >> 4), idesc, (kb | r | c) != 0);
            if (!WRES) {
              tc5::umma_commit(&w_empty[ws]);
              if (++ws == p.w_st) { ws = 0; wph ^= 1u; }
            }
          }
          if (!alive) break;
          tc5::umma_commit(&a_empty[s]);
          s += ISSUERS;
          if (s >= p.a_st) { s -= p.a_st; ph ^= 1u; }
        }
        if (!alive) break;
        tc5::umma_commit(&acc_full[b]);
      }
    }
  } else if (warp < 12) {
    // ---- epilogue: two warps per lane quarter, half the columns each ----
    const int q = warp & 3, c_begin = warp >= 8 ? BN / 2 : 0;
    const int pos = q * 32 + lane, prow = pos / p.pitch, pcol = pos - prow * p.pitch;
    const bool inside = prow < p.TR && pcol < p.W;   // (rows past the image's end are clipped by the store)
    const int cr = prow * p.W + pcol;                // row of the C buffer
    pdl_wait();
    const bool bias_f32_vec = p.bias && p.bias_dtype == B200_F32 && (reinterpret_cast<uintptr_t>(p.bias) & 15u) == 0;
    Tc5Params bp{};
    bp.bias = p.bias; bp.bias_dtype = p.bias_dtype; bp.N = p.O;
    int ct = 0;   // tiles so far: C buffer ct % NCB
    for (int i = 0; i < units; ++i) {
      const int b = i & 1;
      bool ok = __all_sync(0xffffffffu, tc5::mbar_wait(&acc_full[b], (i >> 1) & 1) && !dead());
      if (!ok) { if (lane == 0) fail(66); break; }
      tc5::tc_fence_after();
#pragma unroll 1
      for (int t = 0; t < MT; ++t) {
        int n, h0, n0;
        if (!tile_of(i, t, n, h0, n0)) break;
        const int cb = ct % NCB, u = ct / NCB;
        ++ct;
        ok = __all_sync(0xffffffffu, p.has_res ? tc5::mbar_wait(&c_full[cb], u & 1) : tc5::mbar_wait(&c_free[cb], (u & 1) ^ 1));
        if (!ok) { if (lane == 0) fail(67); break; }
        const uint32_t crow = tc5::smem_addr(cbuf + cb * CB) + cr * 128;
        const uint32_t t_row = tmem_base + (b * MT + t) * BN + (static_cast<uint32_t>(q * 32) << 16);
        auto unit = [&](float (&v)[16], int c) {
          const int o0 = n0 + c;
          if (bias_f32_vec && o0 + 16 <= p.O) {
            const float4* bv = reinterpret_cast<const float4*>(static_cast<const float*>(p.bias) + o0);
#pragma unroll
            for (int k = 0; k < 4; ++k) {
              const float4 f = __ldg(bv + k);
              v[4 * k] += f.x; v[4 * k + 1] += f.y; v[4 * k + 2] += f.z; v[4 * k + 3] += f.w;
            }
          } else {
            add_bias<16>(bp, v, o0, p.O - o0 < 16 ? (p.O - o0 < 0 ? 0 : p.O - o0) : 16);
          }
          const int k = (c & 63) >> 3;
          const uint32_t a0 = crow + (c >> 6) * (128 * 128) + ((k ^ (cr & 7)) << 4), a1 = crow + (c >> 6) * (128 * 128) + (((k + 1) ^ (cr & 7)) << 4);
          uint32_t o[8];
#pragma unroll
          for (int e = 0; e < 8; ++e) o[e] = pack2<T>(v[2 * e], v[2 * e + 1]);
          if (!inside) return;
          if (p.has_res) {
            uint32_t r[8];
            asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(a0));
            asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]) : "r"(a1));
#pragma unroll
            for (int e = 0; e < 8; ++e) o[e] = add2<T>(o[e], r[e]);
          }
          if (p.relu) {
#pragma unroll
            for (int e = 0; e < 8; ++e) o[e] = relu2<T>(o[e]);
          }
          asm volatile("st.shared.v4.u32 [%0], {%1,%2,%3,%4};" ::"r"(a0), "r"(o[0]), "r"(o[1]), "r"(o[2]), "r"(o[3]) : "memory");
          asm volatile("st.shared.v4.u32 [%0], {%1,%2,%3,%4};" ::"r"(a1), "r"(o[4]), "r"(o[5]), "r"(o[6]), "r"(o[7]) : "memory");
        };
        float va[16], vb[16];   // two units in flight: the next tcgen05.ld runs under the current unit's math
        __syncwarp();
        tc5::tmem_ld_32x16(t_row + c_begin, va);
#pragma unroll 1
        for (int c = c_begin; c < c_begin + BN / 2; c += 32) {
          tc5::tmem_ld_wait();
          tc5::tmem_ld_32x16(t_row + c + 16, vb);
          unit(va, c);
          __syncwarp();
          tc5::tmem_ld_wait();
          if (c + 32 < c_begin + BN / 2) tc5::tmem_ld_32x16(t_row + c + 32, va);
          unit(vb, c + 16);
          __syncwarp();
        }
        tc5::fence_proxy_async();   // the TMA store reads these generic-proxy writes
        __syncwarp();
        if (lane == 0) cr_arrive(&c_ready[cb]);
      }
      if (!ok) break;
      tc5::tc_fence_before();
      __syncwarp();
      if (lane == 0) cr_arrive(&acc_empty[b]);
    }
  } else if (lane == 0) {
    // ---- C-buffer store and residual prefetch ----
    pdl_wait();   // the output buffer may still be read by the kernel before this one
    const uint32_t res_bytes = static_cast<uint32_t>(p.TR * p.W * 128 * (BN / 64));
    int ri = 0, rt = 0, loaded = 0;   // next residual tile: unit, tile of the unit; tiles requested
    auto load_residual = [&]() {
      int n, h0, n0;
      if (ri >= units) return;
      if (!tile_of(ri, rt, n, h0, n0)) { ri = units; return; }   // (only the last tiles of a column are missing; see `next`)
      const int cb = loaded % NCB;
      tc5::mbar_arrive_expect_tx(&c_full[cb], res_bytes);
      for (int j = 0; j < BN / 64; ++j) tc5::tma_load_3d(cbuf + cb * CB + j * (128 * 128), &map_r, &c_full[cb], n0 + 64 * j, h0 * p.W, n);
      ++loaded;
      do {
        if (++rt == MT) { rt = 0; ++ri; }
      } while (ri < units && !tile_of(ri, rt, n, h0, n0));
    };
    if (p.has_res)
      for (int k = 0; k < NCB; ++k) load_residual();
    int ct = 0;
    for (int i = 0; i < units && !dead(); ++i)
      for (int t = 0; t < MT; ++t) {
        int n, h0, n0;
        if (!tile_of(i, t, n, h0, n0)) break;
        const int cb = ct % NCB;
        if (!tc5::mbar_wait(&c_ready[cb], (ct / NCB) & 1)) { fail(68); break; }
        ++ct;
        for (int j = 0; j < BN / 64; ++j)
          if (n0 + 64 * j < p.O) tc5::tma_store_3d(&map_o, cbuf + cb * CB + j * (128 * 128), n0 + 64 * j, h0 * p.W, n);
        tc5::tma_store_commit();
        tc5::tma_store_wait_read();
        if (p.has_res) load_residual();
        else cr_arrive(&c_free[cb]);
      }
    if (dead() && p.has_res)
      for (int k = loaded > NCB ? loaded - NCB : 0; k < loaded; ++k) tc5::mbar_wait(&c_full[k % NCB], (k / NCB) & 1, 1u << 16);
    tc5::tma_store_wait_all();
  }
  tc5::tc_fence_before();
  __syncthreads();
  if (warp == 1) { tc5::tc_fence_after(); tc5::tmem_dealloc(tmem_base, 2 * MT * BN); }
}

template <typename T, int BN, int MT, bool WRES>
int launch_conv_rows(const Tc5Args& a, const Tc5Conv& g, ConvRowsParams p, cudaStream_t st) {
  constexpr int CB = 128 * BN * 2, W_STAGE = 3 * BN * 128, NCB = CR_BUFS<MT>;
  // shared memory: input ring, weights, C buffers; the last MMA of a tile reads up to 127 rows from its last tap on, of
  // which those past the window belong to positions that do not count - they only have to lie inside the allocation
  p.a_sub = static_cast<int>(ceil_div(((p.TR + 2) * p.pitch + 1) * 128, 1024) * 1024);   // and the pixel behind the last row
  p.a_stage = MT * p.a_sub;
  const int reach = (2 * p.pitch + 2 + 128) * 128 - p.a_sub;
  const int slack = reach > 0 ? static_cast<int>(ceil_div(reach, 1024) * 1024) : 0;
  const int fixed = NCB * CB + slack + 1024;
  if (WRES) {
    p.w_st = 1;
    const int left = CR_LIMIT - fixed - 9 * BN * 128;
    p.a_st = left / p.a_stage >= 4 ? 4 : left / p.a_stage >= 2 ? 2 : 0;   // even: see the MMA issuers
  } else {
    p.w_st = 2;
    p.a_st = (CR_LIMIT - fixed - 2 * W_STAGE) / p.a_stage;
    if (p.a_st > 4) p.a_st = 4;
    while (p.w_st < 4 && p.a_st >= 2 && fixed + p.a_st * p.a_stage + (p.w_st + 1) * W_STAGE <= CR_LIMIT) ++p.w_st;
  }
  if (p.a_st < 2) return B200_ENOTSUP;
  p.w_off = p.a_st * p.a_stage + slack;
  p.c_off = p.w_off + (WRES ? 9 * BN * 128 : p.w_st * W_STAGE);
  const int smem = p.c_off + NCB * CB + 1024;
  p.n_mu = static_cast<int>(ceil_div(p.n_tiles, MT));
  const int64_t units = static_cast<int64_t>(p.n_mu) * ceil_div(p.O, BN);
  if (units >= (1ll << 30)) return B200_ENOTSUP;
  p.n_units = static_cast<int>(units);
  static PerDevice<bool> configured_on;
  bool* configured = configured_on.slot();
  if (!configured) return B200_ENOTSUP;
  if (!*configured) {
    if (cudaFuncSetAttribute(conv_rows_kernel<T, BN, MT, WRES>, cudaFuncAttributeMaxDynamicSharedMemorySize, CR_LIMIT) != cudaSuccess) {
      cudaGetLastError();
      return B200_ENOTSUP;
    }
    *configured = true;
  }
  CUtensorMap mx, mw, mr, mo;
  const uint64_t C = g.C, W = g.W, H = g.H, N = g.batch, O = a.N;
  {
    const uint64_t dims[4] = {C, W, H, N}, str[3] = {2 * C, 2 * C * W, 2 * C * W * H};
    const uint32_t box[4] = {64, static_cast<uint32_t>(p.pitch), static_cast<uint32_t>(p.TR + 2), 1};
    if (!tma_encode_sw128(&mx, a.dtype, 4, a.A, dims, str, box)) return B200_ENOTSUP;
  }
  {
    const uint64_t dims[2] = {9 * C, O}, str[1] = {2 * static_cast<uint64_t>(a.ldw)};
    const uint32_t box[2] = {64, BN};
    if (!tma_encode_sw128(&mw, a.dtype, 2, a.W, dims, str, box)) return B200_ENOTSUP;
  }
  auto map_out = [&](CUtensorMap* m, const void* base, int64_t ld) {
    const uint64_t dims[3] = {O, W * H, N}, str[2] = {2 * static_cast<uint64_t>(ld), 2 * static_cast<uint64_t>(ld) * W * H};
    const uint32_t box[3] = {64, static_cast<uint32_t>(p.TR * g.W), 1};
    return tma_encode_sw128(m, a.dtype, 3, base, dims, str, box);
  };
  if (!map_out(&mo, a.out, a.ldo)) return B200_ENOTSUP;
  mr = mo;
  if (a.residual && !map_out(&mr, a.residual, a.ldr)) return B200_ENOTSUP;
  const int grid = p.n_units < sm_count() ? p.n_units : sm_count();
  launch_pdl(conv_rows_kernel<T, BN, MT, WRES>, dim3(grid), dim3(CR_THREADS), smem, st, mx, mw, mr, mo, p);
  B200_CHECK_LAUNCH("conv_rows_kernel");
  return B200_OK;
}

template <typename T> int dispatch_conv_rows(const Tc5Args& a, const Tc5Conv& g, const ConvRowsParams& p, int im2col_bn, cudaStream_t st) {
  if (g.C == 64 && a.N <= 64) return launch_conv_rows<T, 64, 1, true>(a, g, p, st);
  // Streamed weights.  The im2col route keeps 256-wide tiles (a weight stage of theirs serves as many rows and twice the columns: 512
  // channels, 14 x 14, 128 images 94 us, 115 here) and results of 64 channels and fewer, for which half of each tile here is padding.
  // Else the waves decide, a wave there counted as one and a half here, a wave of units of two tiles as 1.75 of single ones:
  // they take 4.7 to 5.2 and 8.0 to 9.9 us (128 channels, 28 x 28), 8.6 to 10 and 14.4 to 19 (256 channels, 14 x 14).  256 channels,
  // 14 x 14, 48 images: one wave there 18.5, two here 21.3; 128 channels, 28 x 28, 20 images: two there 15.8, one here 9.8.
  // Units of two leave SMs idle where they are few (128 channels, 32 images, 112 units: 13.7 us, single ones 13.3).
  if (im2col_bn > 128 || a.N <= 64) return B200_ENOTSUP;
  const int64_t cols = ceil_div(a.N, 128), sms = sm_count(), two = ceil_div(p.n_tiles, 2) * cols;
  const int64_t w1 = 4 * ceil_div(p.n_tiles * cols, sms), w2 = 5 * two >= 4 * sms ? 7 * ceil_div(two, sms) : w1;   // quarters of a wave
  const int64_t w0 = 4 * ceil_div(ceil_div(a.M, 128) * ceil_div(a.N, im2col_bn), sms);
  if (2 * (w1 < w2 ? w1 : w2) >= 3 * w0) return B200_ENOTSUP;
  if (w2 < w1)
    if (const int rc = launch_conv_rows<T, 128, 2, false>(a, g, p, st); rc != B200_ENOTSUP) return rc;
  return launch_conv_rows<T, 128, 1, false>(a, g, p, st);
}

}  // namespace

int conv_rows(const Tc5Args& a, const Tc5Conv& g, int im2col_bn, cudaStream_t st) {
  // 16-byte words in every row of the operands, bias / residual / ReLU only
  if (g.KH != 3 || g.KW != 3 || g.sh != 1 || g.sw != 1 || g.ph != 1 || g.pw != 1 || g.C % 64 || g.batch <= 0 || g.Ho != g.H || g.Wo != g.W) return B200_ENOTSUP;
  if (a.N % 8 || a.ldo % 8 || !aligned16(a.out) || (a.residual && (a.ldr % 8 || !aligned16(a.residual)))) return B200_ENOTSUP;
  if (g.W > 127 || static_cast<int64_t>(g.batch) * g.H >= (1ll << 30)) return B200_ENOTSUP;
  ConvRowsParams p = {};
  p.bias = a.bias; p.bias_dtype = a.bias_dtype; p.relu = (a.epilogue & B200_EPI_RELU) ? 1 : 0; p.has_res = a.residual ? 1 : 0;
  p.H = g.H; p.W = g.W; p.O = static_cast<int>(a.N); p.NKB = g.C / 64;
  p.pitch = g.W + 1;
  p.TR = 128 / p.pitch < g.H ? 128 / p.pitch : g.H;
  p.tiles_img = static_cast<int>(ceil_div(g.H, p.TR));
  p.n_tiles = g.batch * p.tiles_img;
  // at least 70 of 100 accumulator rows count
  if (static_cast<int64_t>(g.H) * g.W * 100 < static_cast<int64_t>(p.tiles_img) * 128 * 70) return B200_ENOTSUP;
  return a.dtype == B200_BF16 ? dispatch_conv_rows<__nv_bfloat16>(a, g, p, im2col_bn, st) : dispatch_conv_rows<__half>(a, g, p, im2col_bn, st);
}

int conv_rows_error(bool clear) {
  int v = 0;
  if (cudaMemcpyFromSymbol(&v, g_rows_error, sizeof(int)) != cudaSuccess) return -1;
  if (clear && v) {
    const int zero = 0;
    cudaMemcpyToSymbol(g_rows_error, &zero, sizeof(int));
  }
  return v;
}

}  // namespace b200

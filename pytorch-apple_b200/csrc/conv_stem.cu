// The head of a convolution network in one kernel: 7-wide / stride-2 convolution over at most four planar input channels,
// bias, ReLU, and the 3x3 / stride-2 max-pooling behind it.  Replaces three kernels - the repack of the image to eight
// interleaved channels, the convolution, the pooling - of which the first two wrote, and the last two read, tensors
// many times the size of the input and of the result (256 images: 77 MB in, 103 MB out, 1.2 GB in between).
//
// A persistent CTA owns consecutive pooled rows and walks the convolution rows that they need (two per pooled row, three
// for the first one of a CTA or an image); nothing between the image and the pooled row leaves the SM:
// - a producer thread brings new input rows in pairs, planar as they are, by TMA (rows and pixels outside the image
//   arrive as zeros) into a ring; images whose rows are no whole 16-byte words, or wider than one box, are copied there by the loaders
//   themselves, element by element, which is slower than the three kernels (256 wide, 128 images: 798 us against 360): the executor
//   keeps those for such images;
// - loaders (128 threads, one per column) write them to a window of 16 row slots as sliding windows: per plane, 16 bytes for
//   output column p hold its pixels 2p - 4 .. 2p + 3 - the eight taps of a filter row, the first of which is no tap and zero.  That
//   is the unswizzled K-major core-matrix layout (8 columns x 16 bytes, every core matrix a 128-byte line), and the MMA reads its A
//   operand in place: two instructions (K = 16: the taps of two planes) per filter row.  (Windows that overlap in memory instead of
//   being written out need no copies, but core matrices that straddle two lines: 143 cycles per MMA instead of 85.);
// - two threads issue the MMAs of the rows (128 columns x 64 channels into one of four accumulators) in turn: what one of them
//   spends between two rows (barrier probe, commits: 700 cycles) the tensor core works for the other;
// - epilogue (128 threads, one per column): the maximum over the three rows in registers (the last row of a pooled row is the first
//   one of the next), then bias and rounding to the activation type, which change no order; the column maxima go to shared memory;
// - poolers (128 threads): the maximum over three columns, ReLU, 16 bytes per thread and step, to global memory.
// Bounds: the tensor core, 14 MMAs of N = 64 per row at ~80 cycles (45 with swizzled operands, which sliding windows cannot be): 110
// us for 256 images; the memory 28 us.  us, repack + convolution + pooling -> this, images from memory: 256 images 584 -> 172,
// 32 images 87 -> 29, one image 15 -> 8.  On the way there: a window of one entry per two pixels x four channels, read in place at
// shifted addresses 205 (MMAs of 143 cycles); the same written four times 312 (the loaders); one MMA thread for all rows 205; a
// division per pooled row in each role 216.
#include "gemm_tc5.cuh"
#include "mma.cuh"
#include "tc5.cuh"

namespace b200 {

// time-out code of the last failed wait of this kernel (reported through b200_debug_device_error)
__device__ int g_stem_error = 0;

namespace {

constexpr int SP_BN = 64, SP_ROWS = 4;   // output channels; rows (input rows, accumulators) under way
constexpr int SP_PLANE = 128 * 16, SP_SLOT = 4 * SP_PLANE, SP_SLOTS = 16;   // an input row: [plane][128 columns][16 bytes]
constexpr int SP_W_PANEL = SP_BN * 128;   // weights of two filter rows (each four planes x eight taps): [64][128 bytes], swizzled
constexpr int SP_V = 128 * SP_BN * 2;                              // a row of column maxima, [128 columns][128 bytes], chunks swizzled
constexpr int SP_KH = 8;
constexpr int SP_RAW = 5, SP_RAW_PITCH = 544, SP_RAW_STAGE = 2 * 4 * SP_RAW_PITCH, SP_TMA_WIDTH = 240;   // ring of planar row pairs: [plane][2 rows][8 pixels of margin, image, margin]
constexpr int SP_SMEM = 2 * SP_V + SP_KH / 2 * SP_W_PANEL + SP_SLOTS * SP_SLOT + SP_RAW * SP_RAW_STAGE + 1024 + 64;
constexpr int SP_THREADS = 15 * 32;                                // warps: 0 and 14 MMA, 1-4 epilogue, 5-8 loaders, 9-12 poolers, 13 TMA producer

struct StemPoolParams {
  const void* x; const void* w; const float* bias; void* y;
  int N, C, H, W, Ho, Wo, PH, PW, O, KH, ph, relu, tma;
  int rows, rows_per_cta;   // pooled rows over all images
};

template <typename T> struct Ab;
template <> struct Ab<__half> { static constexpr int value = 0; using Pair = __half2; };
template <> struct Ab<__nv_bfloat16> { static constexpr int value = 1; using Pair = __nv_bfloat162; };
// Maxima.  With ReLU behind them a NaN counts as absent (fmaxf(NaN, 0) is 0), without it wins, as in the pooling kernel.
template <typename T, bool RELU> __device__ __forceinline__ uint32_t max2(uint32_t a, uint32_t b) {
  using P = typename Ab<T>::Pair;
  const P m = RELU ? __hmax2(reinterpret_cast<const P&>(a), reinterpret_cast<const P&>(b)) : __hmax2_nan(reinterpret_cast<const P&>(a), reinterpret_cast<const P&>(b));
  return reinterpret_cast<const uint32_t&>(m);
}
template <bool RELU> __device__ __forceinline__ float max1(float a, float b) {
  if (RELU) return fmaxf(a, b);
  float m;
  asm("max.NaN.f32 %0, %1, %2;" : "=f"(m) : "f"(a), "f"(b));
  return m;
}
__device__ __forceinline__ void arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(tc5::smem_addr(bar)) : "memory");
}

// The convolution rows of a CTA's pooled rows, in order: f(i, image, row, pooled row, first row of a window, last row of the
// pooled row).  Every role walks the same list.
template <typename F> __device__ __forceinline__ void walk(const StemPoolParams& p, int first, int count, F&& f) {
  int i = 0, n = first / p.PH, ph = first - n * p.PH - 1;
  for (int k = 0; k < count; ++k) {
    if (++ph == p.PH) { ph = 0; ++n; }   // (a division here is 250 cycles of a role's row)
    const bool fresh = k == 0 || ph == 0;
    const int lo = fresh && ph > 0 ? 2 * ph - 1 : 2 * ph, hi = 2 * ph + 1 < p.Ho ? 2 * ph + 1 : p.Ho - 1;
    for (int oh = lo; oh <= hi; ++oh, ++i)
      if (!f(i, n, oh, k, fresh && oh == lo, oh == hi)) return;
  }
}

template <typename T, bool RELU>
__global__ void __launch_bounds__(SP_THREADS, 1) conv_stem_pool_kernel(const __grid_constant__ CUtensorMap map_x, const __grid_constant__ StemPoolParams p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  uint8_t* const v_s = smem;                       // two rows of column maxima
  uint8_t* const w_s = smem + 2 * SP_V;
  uint8_t* const window = w_s + SP_KH / 2 * SP_W_PANEL;
  uint8_t* const raw = window + SP_SLOTS * SP_SLOT;
  __shared__ __align__(8) uint64_t row_go[SP_ROWS], row_done[SP_ROWS], acc_full[SP_ROWS], v_ready[2], v_free[2], raw_full[SP_RAW], raw_empty[SP_RAW], w_ready;
  __shared__ __align__(16) float s_bias[SP_BN];
  __shared__ uint32_t tmem_holder;
  __shared__ int failed;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int first = blockIdx.x * p.rows_per_cta;
  const int count = p.rows - first < p.rows_per_cta ? p.rows - first : p.rows_per_cta;

  if (threadIdx.x == 0) {
    failed = 0;
    for (int s = 0; s < SP_ROWS; ++s) {
      tc5::mbar_init(&row_go[s], 256);   // the loaders' input rows are there, the epilogue has read the row that had this accumulator
      tc5::mbar_init(&row_done[s], 1);
      tc5::mbar_init(&acc_full[s], 1);
    }
    for (int s = 0; s < 2; ++s) { tc5::mbar_init(&v_ready[s], 128); tc5::mbar_init(&v_free[s], 128); }
    for (int s = 0; s < SP_RAW; ++s) { tc5::mbar_init(&raw_full[s], 1); tc5::mbar_init(&raw_empty[s], 128); }
    tc5::mbar_init(&w_ready, 256);
    tc5::fence_barrier_init();
    if (p.tma) tc5::prefetch_tensormap(&map_x);
  }
  if (warp == 0) { tc5::tmem_alloc(&tmem_holder, SP_ROWS * SP_BN); tc5::tmem_relinquish(); }
  tc5::tc_fence_before();
  __syncthreads();
  tc5::tc_fence_after();
  const uint32_t tmem_base = tmem_holder;
  pdl_trigger();
  auto dead = [&]() { return *reinterpret_cast<volatile int*>(&failed) != 0; };
  auto fail = [&](int code) { failed = 1; atomicExch(&g_stem_error, code); };

  // Epilogue and pooler warps prepare what stays, while the first input rows are on their way
  if ((warp >= 1 && warp < 5) || (warp >= 9 && warp < 13)) {
    pdl_wait();   // (the kernel before this one may be the one that prepares the weights)
    const int t = threadIdx.x - (warp < 5 ? 32 : 5 * 32);
    // weights [O][KH][7][8] -> [two filter rows][O][row, plane, tap + 1] with the 128-byte swizzle; tap 0 and absent output channels are zero
    for (int i = t; i < p.KH * 4 * SP_BN; i += 256) {
      const int ch = i & 3, oc = (i >> 2) & (SP_BN - 1), r = i >> 8;
      const uint16_t* src = static_cast<const uint16_t*>(p.w) + (static_cast<int64_t>(oc) * p.KH + r) * 7 * 8 + ch;
      uint32_t v[8] = {0u, 0u, 0u, 0u, 0u, 0u, 0u, 0u};
      if (oc < p.O && ch < p.C) {
#pragma unroll
        for (int tap = 0; tap < 7; ++tap) v[tap + 1] = src[tap * 8];
      }
      *reinterpret_cast<uint4*>(w_s + (r >> 1) * SP_W_PANEL + oc * 128 + (((4 * (r & 1) + ch) ^ (oc & 7)) << 4)) =
          make_uint4(v[0] | (v[1] << 16), v[2] | (v[3] << 16), v[4] | (v[5] << 16), v[6] | (v[7] << 16));
    }
    // planes that the image has not got
    for (int i = t; i < (4 - p.C) * SP_SLOTS * 128; i += 256) {
      const int slot = i >> 7 & (SP_SLOTS - 1), ch = p.C + i / (SP_SLOTS * 128);
      *reinterpret_cast<uint4*>(window + slot * SP_SLOT + ch * SP_PLANE + (i & 127) * 16) = make_uint4(0u, 0u, 0u, 0u);
    }
    if (t < SP_BN) s_bias[t] = p.bias && t < p.O ? p.bias[t] : 0.f;
    tc5::fence_proxy_async();
    arrive(&w_ready);
  }

  if (warp == 0 || warp == 14) {
    if (lane == 0) {   // ---- MMA issuers: even and odd rows ----
      constexpr uint32_t idesc = tc5::umma_idesc(128, SP_BN, Ab<T>::value);
      constexpr uint32_t A_HI = (128u >> 4) | (1u << 14);   // descriptor words as in umma_desc_nosw: 128 bytes between groups of eight columns,
      const uint32_t win = ((tc5::smem_addr(window) & 0x3FFFFu) >> 4) | ((SP_PLANE >> 4) << 16);   // a plane to the next eight taps
      const uint32_t wts = tc5::desc_sw128_lo(tc5::smem_addr(w_s));
      const int run = (p.KH + 1) / 2 * 2;   // input rows of a new window: whole pairs
      if (!tc5::mbar_wait(&w_ready, 0)) fail(56);
      int v0 = 0;   // window position of the row's first input row (rows are numbered as they are loaded)
      walk(p, first, count, [&](int i, int, int, int, bool fresh, bool) {
        if (i > 0) v0 += fresh ? run : 2;
        const int b = i % SP_ROWS;
        if ((i & 1) != (warp == 14)) return true;
        // (one probe per row: a probe behind asynchronous instructions costs this thread ~0.3 us)
        if (!tc5::mbar_wait(&row_go[b], (i / SP_ROWS) & 1)) { fail(50); return false; }
        tc5::tc_fence_after();
#pragma unroll
        for (int r = 0; r < SP_KH; ++r)
          if (r < p.KH)
          asm volatile(
              "{\n\t.reg .pred p, q;\n\t.reg .b64 da, db;\n\t.reg .b32 al, bl;\n\t"
              "setp.ne.u32 p, %4, 0;\n\tsetp.eq.u32 q, 0, 0;\n\t"
              "mov.b64 da, {%1, %5};\n\tmov.b64 db, {%2, %6};\n\t"
              "tcgen05.mma.cta_group::1.kind::f16 [%0], da, db, %3, p;\n\t"
              "add.u32 al, %1, %7;\n\tadd.u32 bl, %2, 2;\n\tmov.b64 da, {al, %5};\n\tmov.b64 db, {bl, %6};\n\t"
              "tcgen05.mma.cta_group::1.kind::f16 [%0], da, db, %3, q;\n\t}"
              ::"r"(tmem_base + b * SP_BN), "r"(win + ((v0 + r) & (SP_SLOTS - 1)) * (SP_SLOT >> 4)), "r"(wts + (r >> 1) * (SP_W_PANEL >> 4) + 4 * (r & 1)),
                "r"(idesc), "r"(r), "r"(A_HI), "r"(tc5::DESC_SW128_HI), "n"(2 * SP_PLANE >> 4) : "memory");
        tc5::umma_commit(&acc_full[b]);
        tc5::umma_commit(&row_done[b]);
        return !dead();
      });
    }
  } else if (warp < 5) {
    // ---- epilogue: column r of the row ----
    const int q = warp & 3, r = q * 32 + lane;
    float vm[SP_BN];   // maximum over the rows of the pooled row so far
    for (int s = 0; s < SP_ROWS; ++s) arrive(&row_go[s]);   // all accumulators are free
    if (!__all_sync(0xffffffffu, tc5::mbar_wait(&w_ready, 0)) && lane == 0) fail(56);   // (the bias is another thread's)
    walk(p, first, count, [&](int i, int, int, int k, bool fresh, bool last) {
      const int b = i % SP_ROWS;
      bool ok = tc5::mbar_wait(&acc_full[b], (i / SP_ROWS) & 1);
      if (last) ok = ok && tc5::mbar_wait(&v_free[k & 1], ((k >> 1) & 1) ^ 1);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) { if (lane == 0) fail(52); return false; }
      tc5::tc_fence_after();
      if (fresh) {
#pragma unroll
        for (int c = 0; c < SP_BN; ++c) vm[c] = -INFINITY;
      }
      uint8_t* const v_row = v_s + (k & 1) * SP_V + r * 128;
#pragma unroll
      for (int c0 = 0; c0 < SP_BN; c0 += 32) {
        float v[32];
        tc5::tmem_ld_32x32_async(tmem_base + b * SP_BN + (static_cast<uint32_t>(q * 32) << 16) + c0, v);
        tc5::tmem_ld_wait();
        if (c0 + 32 == SP_BN) {
          tc5::tc_fence_before();
          arrive(&row_go[b]);   // row i + SP_ROWS may have this accumulator
        }
        if (!last) {
#pragma unroll
          for (int c = 0; c < 32; ++c) vm[c0 + c] = max1<RELU>(vm[c0 + c], v[c]);
        } else {
#pragma unroll
          for (int c = 0; c < 32; c += 8) {
            uint32_t m[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              const float2 bias = *reinterpret_cast<const float2*>(&s_bias[c0 + c + 2 * e]);
              float &m0 = vm[c0 + c + 2 * e], &m1 = vm[c0 + c + 2 * e + 1];
              m[e] = pack2<T>(max1<RELU>(m0, v[c + 2 * e]) + bias.x, max1<RELU>(m1, v[c + 2 * e + 1]) + bias.y);
              m0 = v[c + 2 * e];   // the last row of a pooled row is the first one of the next
              m1 = v[c + 2 * e + 1];
            }
            *reinterpret_cast<uint4*>(v_row + ((((c0 + c) >> 3) ^ (r & 7)) << 4)) = make_uint4(m[0], m[1], m[2], m[3]);
          }
        }
      }
      if (last) arrive(&v_ready[k & 1]);
      return true;
    });
  } else if (warp < 9) {
    // ---- loaders: thread t writes column t of every new input row ----
    const int t = threadIdx.x - 5 * 32;
    const int64_t plane = static_cast<int64_t>(p.H) * p.W;
    const int pitch = p.tma ? 512 : SP_RAW_PITCH;
    if (!p.tma) pdl_wait();
    // Row i may be written once nobody reads the slots that it overwrites: 16 slots, a window is up to eight rows and moves by two, or
    // by all its rows where a new one starts.  Within a run of windows that move by two row i - 5 is the last one to read them, so that
    // the accumulators set the pace (row i - 4); the rows before a new window are further back: `run` rows into it, row
    // i - run - 1 has to be done (at its start i - 2).  Rows are seen done one after the other: a parity wait must not skip a phase.
    static_assert(SP_KH + 2 * 5 > SP_SLOTS && SP_KH + 2 * 4 <= SP_SLOTS && SP_ROWS == 4, "window");
    int seen = 0, start = 0, u = 0;   // rows seen done; row with which the current window started; pair of input rows
    walk(p, first, count, [&](int i, int n, int oh, int, bool fresh, bool) {
      if (fresh) start = i;
      const int need = max(i - SP_ROWS, i - max(i - start + 1, 2));
      bool ok = true;
      for (; seen <= need; ++seen) ok = ok && tc5::mbar_wait(&row_done[seen % SP_ROWS], (seen / SP_ROWS) & 1);
      const int pairs = fresh ? (p.KH + 1) / 2 : 1;
      const int ih0 = 2 * oh - p.ph + (fresh ? 0 : (p.KH + 1) / 2 * 2 - 2);   // first new input row
      for (int k = 0; k < pairs; ++k, ++u) {
        const int s = u % SP_RAW;
        uint8_t* const src = raw + s * SP_RAW_STAGE;
        if (p.tma) {
          ok = ok && tc5::mbar_wait(&raw_full[s], (u / SP_RAW) & 1);
        } else {   // the pixels -8 .. 263 of the two rows, plane by plane; the loaders meet before and after, and leave together after a failure
          uint32_t stop = !ok || dead();
          asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.u32 q, %0, 0;\n\tbar.red.or.pred p, 1, 128, q;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "+r"(stop) : : "memory");
          if (stop) { if (!ok) fail(53); return false; }
          for (int e = t; e < SP_RAW_PITCH / 2; e += 128)
#pragma unroll
            for (int j = 0; j < 2; ++j)
#pragma unroll
              for (int ch = 0; ch < 4; ++ch) {
                const int ih = ih0 + 2 * k + j, px = e - 8;
                if (ch < p.C)
                  reinterpret_cast<uint16_t*>(src + (ch * 2 + j) * SP_RAW_PITCH)[e] =
                      ih >= 0 && ih < p.H && px >= 0 && px < p.W ? __ldg(static_cast<const uint16_t*>(p.x) + (n * p.C + ch) * plane + static_cast<int64_t>(ih) * p.W + px) : uint16_t(0);
              }
          asm volatile("bar.sync 1, 128;" ::: "memory");
        }
        if (!ok) { fail(53); return false; }
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          uint8_t* const slot = window + ((2 * u + j) & (SP_SLOTS - 1)) * SP_SLOT + t * 16;
#pragma unroll
          for (int ch = 0; ch < 4; ++ch)
            if (ch < p.C) {
              const uint32_t* px = reinterpret_cast<const uint32_t*>(src + (ch * 2 + j) * pitch + 4 * t + 8);   // pixel 2t - 4
              // (pixel 2t - 4 belongs to no tap: an infinity there times the zero weight would be a NaN)
              *reinterpret_cast<uint4*>(slot + ch * SP_PLANE) = make_uint4(px[0] & 0xffff0000u, px[1], px[2], px[3]);
            }
        }
        if (p.tma) arrive(&raw_empty[s]);
      }
      tc5::fence_proxy_async();     // read by the tensor core (async proxy)
      arrive(&row_go[i % SP_ROWS]);
      return true;
    });
  } else if (warp < 13) {
    // ---- poolers: pixel pw, eight channels per thread and step ----
    const int t = threadIdx.x - 9 * 32, k8 = t & 7;
    for (int k = 0; k < count; ++k) {
      const int row = first + k;
      const bool ok = __all_sync(0xffffffffu, tc5::mbar_wait(&v_ready[k & 1], (k >> 1) & 1));
      if (!ok) { if (lane == 0) fail(55); break; }
      const uint8_t* v_row = v_s + (k & 1) * SP_V;
      auto at = [&](int px) { return *reinterpret_cast<const uint4*>(v_row + px * 128 + ((k8 ^ (px & 7)) << 4)); };
      if (8 * k8 < p.O)
        for (int pw = t >> 3; pw < p.PW; pw += 16) {
          uint4 m = at(2 * pw);
          auto take = [&](const uint4& o) { m.x = max2<T, RELU>(m.x, o.x); m.y = max2<T, RELU>(m.y, o.y); m.z = max2<T, RELU>(m.z, o.z); m.w = max2<T, RELU>(m.w, o.w); };
          if (pw > 0) take(at(2 * pw - 1));
          if (2 * pw + 1 < p.Wo) take(at(2 * pw + 1));
          if (RELU) m = make_uint4(relu2<T>(m.x), relu2<T>(m.y), relu2<T>(m.z), relu2<T>(m.w));
          *reinterpret_cast<uint4*>(static_cast<T*>(p.y) + (static_cast<int64_t>(row) * p.PW + pw) * p.O + 8 * k8) = m;
        }
      arrive(&v_free[k & 1]);
    }
  } else if (p.tma && lane == 0) {
    // ---- TMA producer: pairs of input rows, all planes, pixels -8 .. 247 ----
    pdl_wait();
    int u = 0;
    walk(p, first, count, [&](int, int n, int oh, int, bool fresh, bool) {
      const int pairs = fresh ? (p.KH + 1) / 2 : 1;
      const int ih0 = 2 * oh - p.ph + (fresh ? 0 : (p.KH + 1) / 2 * 2 - 2);
      for (int k = 0; k < pairs; ++k, ++u) {
        const int s = u % SP_RAW;
        if (u >= SP_RAW && !tc5::mbar_wait(&raw_empty[s], ((u / SP_RAW) & 1) ^ 1)) { fail(54); return false; }
        if (dead()) return false;
        tc5::mbar_arrive_expect_tx(&raw_full[s], p.C * 2 * 512);
        tc5::tma_load_4d(raw + s * SP_RAW_STAGE, &map_x, &raw_full[s], -8, ih0 + 2 * k, 0, n);
      }
      return true;
    });
    if (dead())   // after a failure: the copies in flight land before the CTA leaves
      for (int i = u > SP_RAW ? u - SP_RAW : 0; i < u; ++i) tc5::mbar_wait(&raw_full[i % SP_RAW], (i / SP_RAW) & 1, 1u << 16);
  }
  tc5::tc_fence_before();
  __syncthreads();
  if (warp == 0) { tc5::tc_fence_after(); tc5::tmem_dealloc(tmem_base, SP_ROWS * SP_BN); }
}

bool stem_pool_shape(int C, int H, int W, int c_pad, int O, int KH, int KW, int sh, int sw, int ph, int pw, int dtype) {
  return (dtype == B200_F16 || dtype == B200_BF16) && C >= 1 && C <= 4 && c_pad == 8 && O >= 8 && O <= SP_BN && O % 8 == 0 && KH >= 2 && KH <= SP_KH && KW == 7 &&
         sh == 2 && sw == 2 && pw == 3 && ph >= 0 && ph < KH && H >= 1 && W >= 1 && (W + 2 * pw - KW) / 2 + 1 <= 128 && H + 2 * ph >= KH;
}

template <typename T, bool RELU> int launch_stem_pool(StemPoolParams p, int dtype, cudaStream_t st) {
  static PerDevice<bool> configured_on;
  bool* configured = configured_on.slot();
  if (!configured) B200_FAIL(B200_ELAUNCH, "conv_stem_pool_kernel: no current device");
  if (!*configured) {
    const cudaError_t e = cudaFuncSetAttribute(conv_stem_pool_kernel<T, RELU>, cudaFuncAttributeMaxDynamicSharedMemorySize, SP_SMEM);
    if (e != cudaSuccess) { cudaGetLastError(); B200_FAIL(B200_ELAUNCH, "conv_stem_pool_kernel attribute: %s", cudaGetErrorString(e)); }
    *configured = true;
  }
  // Planar rows by TMA: whole 16-byte words per row, and a box of 256 pixels that holds the image with eight on each side
  CUtensorMap mx = {};
  p.tma = 0;
  if (p.W % 8 == 0 && p.W <= SP_TMA_WIDTH && aligned16(p.x)) {
    const uint64_t w = static_cast<uint64_t>(p.W), dims[4] = {w, static_cast<uint64_t>(p.H), static_cast<uint64_t>(p.C), static_cast<uint64_t>(p.N)};
    const uint64_t str[3] = {2 * w, 2 * w * p.H, 2 * w * p.H * p.C};
    const uint32_t box[4] = {256, 2, static_cast<uint32_t>(p.C), 1};
    p.tma = tma_encode_plain(&mx, dtype, 4, p.x, dims, str, box) ? 1 : 0;
  }
  launch_pdl(conv_stem_pool_kernel<T, RELU>, dim3(static_cast<unsigned>(ceil_div(p.rows, p.rows_per_cta))), dim3(SP_THREADS), SP_SMEM, st, mx, p);
  B200_CHECK_LAUNCH("conv_stem_pool_kernel");
  return B200_OK;
}

}  // namespace

int conv_stem_error(bool clear) {
  int v = 0;
  if (cudaMemcpyFromSymbol(&v, g_stem_error, sizeof(int)) != cudaSuccess) return -1;
  if (clear && v) {
    const int zero = 0;
    cudaMemcpyToSymbol(g_stem_error, &zero, sizeof(int));
  }
  return v;
}

}  // namespace b200

using namespace b200;

extern "C" int b200_conv_stem_pool_supported(int C, int H, int W, int C_pad, int O, int KH, int KW, int sh, int sw, int ph, int pw, int dtype) {
  return tc5_enabled() && stem_pool_shape(C, H, W, C_pad, O, KH, KW, sh, sw, ph, pw, dtype) ? 1 : 0;
}

extern "C" int b200_conv_stem_pool(const void* x, const void* w, const float* bias, void* y, int N, int C, int H, int W, int C_pad, int O, int KH,
                                   int KW, int sh, int sw, int ph, int pw, int dtype, int epilogue, void* stream) {
  B200_CHECK_ARG(x && w && y && N >= 0 && !(epilogue & ~B200_EPI_RELU), "b200_conv_stem_pool: bad arguments");
  if (!b200_conv_stem_pool_supported(C, H, W, C_pad, O, KH, KW, sh, sw, ph, pw, dtype))
    B200_FAIL(B200_ENOTSUP, "b200_conv_stem_pool: %dx%d filter, %d -> %d channels, %d columns is not implemented", KH, KW, C, O, W);
  if (!aligned16(y) || (reinterpret_cast<uintptr_t>(w) & 7u) || (reinterpret_cast<uintptr_t>(x) & 1u)) B200_FAIL(B200_EALIGN, "b200_conv_stem_pool: misaligned operands");
  if (N == 0) return B200_OK;
  StemPoolParams p;
  p.x = x; p.w = w; p.bias = bias; p.y = y;
  p.N = N; p.C = C; p.H = H; p.W = W; p.O = O; p.KH = KH; p.ph = ph; p.relu = epilogue & B200_EPI_RELU;
  p.Ho = (H + 2 * ph - KH) / 2 + 1; p.Wo = (W + 2 * pw - KW) / 2 + 1;
  p.PH = (p.Ho - 1) / 2 + 1; p.PW = (p.Wo - 1) / 2 + 1;
  const int64_t rows = static_cast<int64_t>(N) * p.PH;
  if (rows >= (1ll << 31)) B200_FAIL(B200_ELIMIT, "b200_conv_stem_pool: too many rows");
  p.rows = static_cast<int>(rows);
  p.rows_per_cta = static_cast<int>(ceil_div(rows, sm_count()));
  const cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (dtype == B200_BF16) return p.relu ? launch_stem_pool<__nv_bfloat16, true>(p, dtype, st) : launch_stem_pool<__nv_bfloat16, false>(p, dtype, st);
  return p.relu ? launch_stem_pool<__half, true>(p, dtype, st) : launch_stem_pool<__half, false>(p, dtype, st);
}

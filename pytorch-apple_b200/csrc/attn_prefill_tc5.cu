// Prefill attention on the 5th-generation tensor cores (tcgen05.mma, accumulators in tensor
// memory, operands staged by TMA), head_dim 128.
//
// One CTA = 128 query rows of one head.  Q sits in shared memory for the CTA's life; K and V arrive by TMA in 128-key
// tiles through rings of two stages each (128-byte swizzle).  Two groups of four softmax warps share a tile: group g works
// on its keys 64 g .. 64 g + 63 with its own running maxima and output accumulator, one thread per query row, so that no
// thread waits for another within a tile and the groups need not keep in step.  Per tile:
//   S[128 x 128]    = Q K^T     tcgen05.mma, K tile as the K-major B operand, S in tensor memory (two buffers: the
//                   scores of the next tile are there when a group has finished this one)
//   softmax         one thread per query row and group reads its half row of S with tcgen05.ld, adds the mask where the tile
//                   needs it, keeps the running max / sum (log2 domain) and writes the probabilities, rounded to the
//                   activation type as the unfused graph rounds them, into shared memory in the
//                   K-major swizzled layout of an A operand (two buffers)
//   O_g[128 x 128] += P_g V_g   tcgen05.mma, V tile as the MN-major B operand (V rows are keys, the
//                   head dimension is the contiguous one)
//   correction      the stored maximum of a row follows the true one only when that has grown by more than RESCALE_STEP
//                   (probabilities then stay below 2^RESCALE_STEP, which changes no relative rounding); only then are the
//                   row's sums rescaled in tensor memory (tcgen05.ld / tcgen05.st)
// At the end each group takes half of the head dimension of both accumulators and writes it.
//
// The mask is the only statement of what is attended; nothing assumes that it is causal.  Each (128 rows x 128 keys) tile
// of it has a state: nothing unmasked (the tile is neither fetched nor multiplied), all zero (nothing to add), or mixed.  The
// states come from b200_mask_tiles, which looks at a mask once for all heads and layers that share it (read per head
// and layer, a mask of 2048 x 2048 is 100 MB of L2 traffic per layer, as much as all K and V tiles), or, where the caller
// has none, from a scan of the CTA's own rows at its start.  A mixed tile travels by TMA into the probability buffer of
// its tile, which has the same layout and is free until then: each thread reads its row's mask where it then writes its
// row's probabilities.  (Read by the threads themselves, one such tile cost 11 us of L2 round trips.)
//
// Bounds: per tile 1024 tensor cycles (16 MMAs of N = 128), 1024 cycles of ex2 per scheduler and 64 KB of K and V into
// the SM, which are level; short prompts are bound by the chain Q, K -> S -> softmax -> O of their longest row block.
// us per launch (12 heads over 2 KV heads, causal mask), the 64-key kernel with two threads per
// row that this one replaced -> this one, in chains of launches: 128 tokens 8.8 -> 6.7, 512 18.3 -> 10.2,
// 777 24.0 -> 13.0, 1024 30.5 -> 15.4, 2048 59.9 -> 26.0 (whole prompts of 512 and 2048 tokens 2930 -> 2680, 8300 -> 7250).
// Of the 2600 cycles that a tile of a long row block takes, exponentials are 1150 (both groups at once), the scores' way
// from tensor memory to their maximum 450, barrier waits that find their phase complete 100 to 250 each.
// Measured and not used: all 128 keys of a row in the registers of one thread (12 us for a single tile: fetching that much
// straight-line code), two passes over scores that stay in tensor memory (32.1 us for 2048 tokens), groups that take
// whole tiles in turn (27.6: their scores are then computed while they wait), a second producer thread (28.1).
//
// Warp roles: warps 0-3 and 4-7 the softmax groups (warp w reads the 32 tensor-memory lanes of quarter w % 4), warp 8 MMA
// issuer and owner of the tensor-memory allocation, warp 9 TMA producer.  Every
// barrier wait is bounded; on a time-out the CTA records a code in the library's device error
// word, stops issuing, frees its tensor memory and returns.
#include "attention.cuh"
#include "gemm_tc5.cuh"
#include "tc5.cuh"

namespace b200 {

// time-out code of the last failed wait in this file's kernel (reported through b200_debug_device_error)
__device__ int g_attn5_error = 0;
#define g_tc5_error g_attn5_error

namespace {

constexpr int PD = 128;                        // head dim
constexpr int BQ = 128, BKV = MASK_TILE;
constexpr int PANEL = 128 * 128;               // [128 rows][128 bytes]: 64 columns of an operand tile
constexpr int TILE_BYTES = 2 * PANEL;          // a 128 x 128 operand tile: two panels
constexpr int PF5_THREADS = 320;
constexpr int PF5_SMEM = TILE_BYTES * 7 + 1024;   // Q, K x 2, V x 2, P x 2, alignment
constexpr int MAX_TILES = 256;                 // key tiles per launch (S <= 32768)
constexpr uint32_t MIXED = 1u << 15;
constexpr float MASKED_F = -1e30f;
constexpr float LOG2E_F = 1.4426950408889634f;
constexpr float RESCALE_STEP = 8.f;
constexpr int TMEM_COLS = 512;                 // two buffers of S, O of both groups: 128 columns each

template <typename T> struct Fmt;
template <> struct Fmt<__half> { static constexpr int value = 0; };
template <> struct Fmt<__nv_bfloat16> { static constexpr int value = 1; };

__device__ __forceinline__ float ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ void mbar_arrive1(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(tc5::smem_addr(bar)) : "memory");
}

// What a tile of the mask holds, gathered word by word: the largest element (NaN ignored) and the bits of all of them
// without their signs.
template <typename T> struct Pair;
template <> struct Pair<__half> { using type = __half2; };
template <> struct Pair<__nv_bfloat16> { using type = __nv_bfloat162; };
template <typename T> struct TileScan {
  typename Pair<T>::type top;
  uint32_t bits = 0;
  __device__ __forceinline__ TileScan() {
    const uint32_t lowest = Fmt<T>::value ? 0xff80ff80u : 0xfc00fc00u;   // -infinity, twice
    top = reinterpret_cast<const typename Pair<T>::type&>(lowest);
  }
  __device__ __forceinline__ void word(uint32_t w) {
    top = __hmax2(top, reinterpret_cast<const typename Pair<T>::type&>(w));
    bits |= w & 0x7fff7fffu;
  }
  __device__ __forceinline__ void take(const uint4& v) { word(v.x); word(v.y); word(v.z); word(v.w); }
  // bit 0: an unmasked element, bit 1: an element that is not zero
  __device__ __forceinline__ uint32_t verdict() const {
    const uint32_t w = reinterpret_cast<const uint32_t&>(top);
    const uint16_t a = static_cast<uint16_t>(w), b = static_cast<uint16_t>(w >> 16);
    const float m = fmaxf(to_f32<T>(reinterpret_cast<const T&>(a)), to_f32<T>(reinterpret_cast<const T&>(b)));
    return (m > MASKED_F ? 1u : 0u) | (bits ? 2u : 0u);
  }
};
// Verdict of this thread's share (thread i of n, n a multiple of 16) of the tile rows [q0, q0 + rows) x keys [key0, key0 + BKV):
// eight keys of every (n / 16)th row, as a vector where `vec` allows it.
template <typename T>
__device__ __forceinline__ uint32_t scan_tile(const T* m0, int64_t mask_t, int rows, int64_t key0, int64_t S, bool vec, int i, int n) {
  TileScan<T> t;
  const T* src = m0 + key0 + 8 * (i & 15);
  const int64_t keys = S - key0 - 8 * (i & 15);
  if (vec && keys >= 8) {
#pragma unroll 8
    for (int r = i >> 4; r < rows; r += n >> 4) t.take(__ldg(reinterpret_cast<const uint4*>(src + r * mask_t)));
  } else if (keys > 0) {
    for (int r = i >> 4; r < rows; r += n >> 4) {
      const uint16_t* e = reinterpret_cast<const uint16_t*>(src + r * mask_t);
      uint32_t w[8];
#pragma unroll
      for (int k = 0; k < 8; ++k) w[k] = e[k < keys ? k : 0];   // an absent key repeats the first one, which changes nothing
#pragma unroll
      for (int k = 0; k < 8; k += 2) t.word(w[k] | (w[k + 1] << 16));
    }
  }
  return t.verdict();
}

// One block per tile of the mask
template <typename T>
__global__ void __launch_bounds__(256) mask_tiles_kernel(const T* mask, int64_t rows, int64_t S, int64_t mask_b, int64_t mask_t, uint8_t* out) {
  const int64_t q0 = static_cast<int64_t>(blockIdx.y) * BQ, key0 = static_cast<int64_t>(blockIdx.x) * BKV;
  const T* m0 = mask + blockIdx.z * mask_b + q0 * mask_t;
  const bool vec = (reinterpret_cast<uintptr_t>(mask) & 15u) == 0 && mask_b % 8 == 0 && mask_t % 8 == 0;
  pdl_trigger();
  pdl_wait();
  const uint32_t v = scan_tile<T>(m0, mask_t, static_cast<int>(rows - q0 < BQ ? rows - q0 : BQ), key0, S, vec, threadIdx.x, 256);
  const int any = __syncthreads_or(v & 1u), mixed = __syncthreads_or(v & 2u);
  if (threadIdx.x == 0)
    out[(static_cast<int64_t>(blockIdx.z) * gridDim.y + blockIdx.y) * gridDim.x + blockIdx.x] = !any ? MASK_TILE_NONE : mixed ? MASK_TILE_MIXED : MASK_TILE_ZERO;
}

template <typename T>
__global__ void __launch_bounds__(PF5_THREADS, 1)
    attn_prefill_tc5_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
                            const __grid_constant__ CUtensorMap map_v, const __grid_constant__ CUtensorMap map_m, const PrefillParams p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  uint8_t* q_s = smem;
  uint8_t* k_s = smem + TILE_BYTES;
  uint8_t* v_s = smem + 3 * TILE_BYTES;
  uint8_t* p_s = smem + 5 * TILE_BYTES;
  // tile n lives in stage / buffer n & 1
  __shared__ __align__(8) uint64_t q_full, k_full[2], k_empty[2], v_full[2], v_empty[2], m_full[2], s_full[2], p_ready[2], o_full[2];
  __shared__ uint32_t tmem_holder;
  __shared__ uint8_t s_state[MAX_TILES];
  __shared__ uint16_t s_tile[MAX_TILES];   // the tiles to be processed: key tile, MIXED where the mask has to be added
  __shared__ int s_count;
  __shared__ int failed;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // heads fastest (the CTAs that share K, V and mask rows run together and find them in L2), late row blocks -
  // the ones with the most key tiles under a causal mask - first
  const int h = blockIdx.x, b = blockIdx.z;
  const int q0 = static_cast<int>(gridDim.y - 1 - blockIdx.y) * BQ;
  const int hk = h / (p.Hq / p.Hkv);
  const int b_m = p.mask_b == 0 ? 0 : b;   // a mask without a batch stride is shared by all sequences
  const int n_tiles = static_cast<int>((p.S + BKV - 1) / BKV);
  const int rows_valid = static_cast<int>(p.T - q0 < BQ ? p.T - q0 : BQ);
  const bool has_mask = p.mask != nullptr;
  const T* const mask0 = static_cast<const T*>(p.mask) + static_cast<int64_t>(b_m) * p.mask_b + static_cast<int64_t>(q0) * p.mask_t;

  if (warp == 9 && lane == 0) {
    failed = 0;
    tc5::mbar_init(&q_full, 1);
    for (int s = 0; s < 2; ++s) {
      tc5::mbar_init(&k_full[s], 1);
      tc5::mbar_init(&k_empty[s], 1);
      tc5::mbar_init(&v_full[s], 1);
      tc5::mbar_init(&v_empty[s], 1);
      tc5::mbar_init(&m_full[s], 1);
      tc5::mbar_init(&s_full[s], 1);
      tc5::mbar_init(&p_ready[s], 256);
      tc5::mbar_init(&o_full[s], 1);
    }
    tc5::fence_barrier_init();
    tc5::prefetch_tensormap(&map_q);
    tc5::prefetch_tensormap(&map_k);
    tc5::prefetch_tensormap(&map_v);
    if (has_mask) tc5::prefetch_tensormap(&map_m);
  }
  if (warp == 8) { tc5::tmem_alloc(&tmem_holder, TMEM_COLS); tc5::tmem_relinquish(); }
  pdl_trigger();
  pdl_wait();   // q, k, v and the mask come from earlier kernels
  if (warp == 9 && lane == 0) {
    tc5::mbar_arrive_expect_tx(&q_full, TILE_BYTES);
    tc5::tma_load_5d(q_s, &map_q, &q_full, 0, q0, 0, h, b);
    // the first key tile as well, before it is known whether it is wanted: it nearly always is
    tc5::mbar_arrive_expect_tx(&k_full[0], TILE_BYTES);
    tc5::tma_load_5d(k_s, &map_k, &k_full[0], 0, 0, 0, hk, b);
    tc5::mbar_arrive_expect_tx(&v_full[0], TILE_BYTES);
    tc5::tma_load_5d(v_s, &map_v, &v_full[0], 0, 0, 0, hk, b);
  }
  const bool scan = has_mask && !p.tiles;
  if (scan && warp < 8) {   // a warp per tile
    const bool vec = (reinterpret_cast<uintptr_t>(p.mask) & 15u) == 0 && p.mask_b % 8 == 0 && p.mask_t % 8 == 0;
    for (int j = warp; j < n_tiles; j += 8) {
      const uint32_t v = __reduce_or_sync(0xffffffffu, scan_tile<T>(mask0, p.mask_t, rows_valid, static_cast<int64_t>(j) * BKV, p.S, vec, lane, 32));
      if (lane == 0) s_state[j] = !(v & 1u) ? MASK_TILE_NONE : v & 2u ? MASK_TILE_MIXED : MASK_TILE_ZERO;
    }
  }
  if (scan) __syncthreads();
  if (warp == 0) {   // the list of the tiles to be processed
    const uint8_t* states = has_mask && p.tiles ? p.tiles + (static_cast<int64_t>(b_m) * gridDim.y + q0 / BQ) * n_tiles : nullptr;
    int count = 0;
    for (int j = lane; j - lane < n_tiles; j += 32) {
      uint32_t state = MASK_TILE_NONE;
      if (j < n_tiles) state = states ? __ldg(states + j) : scan ? s_state[j] : MASK_TILE_ZERO;
      const uint32_t valid = __ballot_sync(0xffffffffu, state != MASK_TILE_NONE);
      if (state != MASK_TILE_NONE) s_tile[count + __popc(valid & ((1u << lane) - 1u))] = static_cast<uint16_t>(j | (state == MASK_TILE_MIXED ? MIXED : 0u));
      count += __popc(valid);
    }
    if (lane == 0) s_count = count;
  }
  tc5::tc_fence_before();
  __syncthreads();
  tc5::tc_fence_after();
  const uint32_t tmem_base = tmem_holder;
  const int N = s_count;
  // Tile 0 is not the first one: its copies count as a phase of stage 0 that nobody works on.  Nobody may look at these barriers
  // before that phase is complete: a wait for the phase behind it would take the parity of the one before it for done, run a phase
  // ahead of its operands from then on, and leave with copies in flight.  (With no tile at all nobody else looks for Q either:
  // every copy has landed before the CTA leaves.)
  const uint32_t missed = N == 0 || (s_tile[0] & (MIXED - 1)) != 0;
  if (missed) {
    if (warp == 9 && lane == 0 && !(tc5::mbar_wait(&k_full[0], 0) & tc5::mbar_wait(&v_full[0], 0) & tc5::mbar_wait(&q_full, 0))) {
      failed = 1;
      atomicExch(&g_tc5_error, 29);
    }
    __syncthreads();
  }
  auto full_parity = [&](int n) { return ((n >> 1) + (n & 1 ? 0 : missed)) & 1; };   // of k_full and v_full

  if (warp == 9) {
    if (lane == 0) {   // ---- TMA producer: one instruction per tile (the maps split the head dimension into (64, 2): two panels) ----
      int n = 0;
      uint32_t masks = 0;   // mixed tiles so far of each buffer, 16 bits each
      for (; n < N; ++n) {
        const int st = n & 1, j = s_tile[n] & (MIXED - 1);
        // A stage's first tile waits for nothing (nor could it ask: with the copies of tile 0 on their way since the start, its
        // scores may be done, and the barrier a phase further, before this thread gets here).
        const uint32_t parity = ((n >> 1) & 1) ^ 1;
        if (n >= 2 && !tc5::mbar_wait(&k_empty[st], parity)) { failed = 1; atomicExch(&g_tc5_error, 30); break; }
        if (*reinterpret_cast<volatile int*>(&failed)) break;
        const bool there = n == 0 && !missed;   // its copies are on their way
        if (!there) {
          tc5::mbar_arrive_expect_tx(&k_full[st], TILE_BYTES);
          tc5::tma_load_5d(k_s + st * TILE_BYTES, &map_k, &k_full[st], 0, j * BKV, 0, hk, b);
        }
        if (n >= 2 && !tc5::mbar_wait(&v_empty[st], parity)) {
          failed = 1;
          atomicExch(&g_tc5_error, 31);
          tc5::mbar_wait(&k_full[st], full_parity(n), 1u << 16);   // the copy just issued
          break;
        }
        if (s_tile[n] & MIXED) {   // the stage's last product is complete: nothing reads its probabilities any more
          tc5::mbar_arrive_expect_tx(&m_full[st], TILE_BYTES);
          tc5::tma_load_3d(p_s + st * TILE_BYTES, &map_m, &m_full[st], j * BKV, q0, b_m);
          tc5::tma_load_3d(p_s + st * TILE_BYTES + PANEL, &map_m, &m_full[st], j * BKV + 64, q0, b_m);
          masks += 1u << (16 * st);
        }
        if (!there) {
          tc5::mbar_arrive_expect_tx(&v_full[st], TILE_BYTES);
          tc5::tma_load_5d(v_s + st * TILE_BYTES, &map_v, &v_full[st], 0, j * BKV, 0, hk, b);
        }
      }
      // on a failure elsewhere the copies in flight must land before the CTA leaves
      if (*reinterpret_cast<volatile int*>(&failed)) {
        tc5::mbar_wait(&q_full, 0, 1u << 16);
        for (int i = n > 2 ? n - 2 : 0; i < n; ++i) {
          tc5::mbar_wait(&k_full[i & 1], full_parity(i), 1u << 16);
          tc5::mbar_wait(&v_full[i & 1], full_parity(i), 1u << 16);
        }
        for (int g = 0; g < 2; ++g)
          if (const uint32_t m = (masks >> (16 * g)) & 0xffffu) tc5::mbar_wait(&m_full[g], (m - 1) & 1, 1u << 16);
      }
    }
  } else if (warp == 8) {
    if (lane == 0) {   // ---- MMA issuer ----
      constexpr uint32_t idesc_s = tc5::umma_idesc(BQ, BKV, Fmt<T>::value);
      constexpr uint32_t idesc_o = tc5::umma_idesc(BQ, PD, Fmt<T>::value) | (1u << 16);   // B operand MN-major
      const uint32_t q_lo = tc5::desc_sw128_lo(tc5::smem_addr(q_s));
      auto issue_s = [&](int st) {   // S = Q K^T of the tile in stage st
        const uint32_t k_lo = tc5::desc_sw128_lo(tc5::smem_addr(k_s + st * TILE_BYTES));
        tc5::umma_f16_kblock(tmem_base + 128 * st, q_lo, k_lo, idesc_s, 0);
        tc5::umma_f16_kblock(tmem_base + 128 * st, q_lo + (PANEL >> 4), k_lo + (PANEL >> 4), idesc_s, 1);
        tc5::umma_commit(&s_full[st]);
        tc5::umma_commit(&k_empty[st]);
      };
      bool ok = N == 0 || tc5::mbar_wait(&q_full, 0);
      for (int n = 0; ok && n < 2 && n < N; ++n) {
        ok = tc5::mbar_wait(&k_full[n], full_parity(n));
        tc5::tc_fence_after();
        if (ok) issue_s(n);
      }
      if (!ok) { failed = 1; atomicExch(&g_tc5_error, 33); }
      // One probe per tile (a probe behind asynchronous instructions costs this thread ~0.3 us): the softmax threads look
      // for the copies that the next products read before they arrive on p_ready.
      for (int n = 0; ok && n < N; ++n) {
        const int st = n & 1;
        const uint32_t v_addr = tc5::smem_addr(v_s + st * TILE_BYTES), p_addr = tc5::smem_addr(p_s + st * TILE_BYTES);
        if (!tc5::mbar_wait(&p_ready[st], (n >> 1) & 1)) { failed = 1; atomicExch(&g_tc5_error, 34); break; }
        tc5::tc_fence_after();
#pragma unroll
        for (int k = 0; k < 8; ++k) {     // 16 keys per instruction = two 8-key groups of the V panels
          const uint64_t da = tc5::umma_desc_sw128(p_addr + (k >> 2) * PANEL) + 2 * (k & 3);
          const uint64_t db = tc5::umma_desc_sw128_mn(v_addr + k * 2048, PANEL, 1024);
          tc5::umma_f16(tmem_base + 256 + 128 * (k >> 2), da, db, idesc_o, n > 0 || (k & 3) != 0);
        }
        tc5::umma_commit(&o_full[st]);
        tc5::umma_commit(&v_empty[st]);
        if (n + 2 < N) issue_s(st);
      }
    }
  } else {
    // ---- softmax: one thread per query row and group, group g on keys 64 g .. of a tile ----
    const int g = warp >> 2, quarter = warp & 3;
    const int r = 32 * quarter + lane;   // the tensor-memory lane this thread may read
    const uint32_t t_lane = tmem_base + (static_cast<uint32_t>(32 * quarter) << 16);
    const uint32_t t_o = t_lane + 256 + 128 * g;
    const float c = p.scale * LOG2E_F;   // scores in the log2 domain
    float m_run = -INFINITY, l_run = 0.f;   // maximum that the row's sums are relative to, sum of the probabilities
    bool alive = true;
    // Every lane polls and the warp leaves together (one lane polling for the others, and one arriving for them, is slower:
    // 31.2 us against 27.5 for 2048 tokens).
    auto wait_all = [&](uint64_t* bar, uint32_t parity, int code) {
      bool got = tc5::mbar_try_wait(bar, parity);
      if (!__all_sync(0xffffffffu, got)) got = __all_sync(0xffffffffu, tc5::mbar_wait(bar, parity));
      if (!got && lane == 0) { failed = 1; atomicExch(&g_tc5_error, code); }
      return got;
    };
    int n = 0;
    uint32_t m_parity = 0;   // phase of m_full, a bit per buffer
#pragma unroll 1
    for (; n < N; ++n) {
      const int st = n & 1;
      const uint32_t tile = s_tile[n];
      const int left = static_cast<int>(p.S) - static_cast<int>(tile & (MIXED - 1)) * BKV - 64 * g;   // keys of this half (64 or more: all)
      uint8_t* const p_own = p_s + st * TILE_BYTES + g * PANEL + r * 128;
      if (!wait_all(&s_full[st], (n >> 1) & 1, 35)) { alive = false; break; }
      tc5::tc_fence_after();
      float u[64];
      tc5::tmem_ld_32x32_async(t_lane + 128 * st + 64 * g, *reinterpret_cast<float(*)[32]>(&u[0]));
      tc5::tmem_ld_32x32_async(t_lane + 128 * st + 64 * g + 32, *reinterpret_cast<float(*)[32]>(&u[32]));
      tc5::tmem_ld_wait();
      float to_log2 = c;
      if (tile & MIXED) {
        if (!wait_all(&m_full[st], (m_parity >> st) & 1, 38)) { alive = false; break; }
        m_parity ^= 1u << st;
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          float f[8];
          unpack8<T>(*reinterpret_cast<const uint4*>(p_own + ((k ^ (r & 7)) << 4)), f);
#pragma unroll
          for (int e = 0; e < 8; e += 2) {
            tc5::fma2(u[8 * k + e], u[8 * k + e + 1], p.scale, f[e], f[e + 1]);
            tc5::mul2(u[8 * k + e], u[8 * k + e + 1], LOG2E_F);
          }
        }
        to_log2 = 1.f;
      } else if (c <= 0.f) {   // (with the factor left for later the maximum would be the minimum, and 0 times an absent key's -infinity no number)
#pragma unroll
        for (int e = 0; e < 64; e += 2) tc5::mul2(u[e], u[e + 1], c);
        to_log2 = 1.f;
      }
      if (left < 64) {   // keys past the end
#pragma unroll
        for (int e = 0; e < 64; ++e)
          if (e >= left) u[e] = -INFINITY;
      }
      float mx[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
      for (int e = 0; e < 64; e += 8)
#pragma unroll
        for (int k = 0; k < 4; ++k) mx[k] = fmaxf(mx[k], fmaxf(u[e + 2 * k], u[e + 2 * k + 1]));
      const float top = fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3])) * to_log2;
      const bool moved = top > m_run + RESCALE_STEP || (m_run == -INFINITY && top > m_run);
      const float m_new = moved ? top : m_run;
      const float m_use = m_new == -INFINITY ? 0.f : m_new;
      if (n > 0 && __any_sync(0xffffffffu, moved)) {   // rescale this warp's rows, once the product before has finished
        if (!wait_all(&o_full[st ^ 1], ((n - 1) >> 1) & 1, 36)) { alive = false; break; }
        const float alpha = moved ? ex2(m_run - m_use) : 1.f;   // 0 for the first maximum of a row
        tc5::tc_fence_after();
#pragma unroll 1
        for (int q = 0; q < PD; q += 16) {
          float t[16];
          tc5::tmem_ld_32x16(t_o + q, t);
          tc5::tmem_ld_wait();
#pragma unroll
          for (int e = 0; e < 16; e += 2) tc5::mul2(t[e], t[e + 1], alpha);
          tc5::tmem_st_32x16(t_o + q, t);
        }
        tc5::tmem_st_wait();
        l_run *= alpha;
      }
      m_run = m_new;
      // the product that read this buffer's last probabilities (every phase of the barrier is seen here, one after the other)
      if (n > 1 && !wait_all(&o_full[st], ((n - 2) >> 1) & 1, 37)) { alive = false; break; }
      float sum[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        float pr[8];
#pragma unroll
        for (int e = 0; e < 8; e += 2) {
          float a = u[8 * k + e], d = u[8 * k + e + 1];
          tc5::fma2(a, d, to_log2, -m_use, -m_use);
          pr[e] = ex2(a);
          pr[e + 1] = ex2(d);
          tc5::add2(sum[e & 2], sum[(e & 2) + 1], pr[e], pr[e + 1]);
        }
        *reinterpret_cast<uint4*>(p_own + ((k ^ (r & 7)) << 4)) = pack8<T>(pr);
      }
      l_run += (sum[0] + sum[1]) + (sum[2] + sum[3]);
      tc5::fence_proxy_async();   // the probabilities are read by the tensor core (async proxy)
      tc5::tc_fence_before();     // this thread's tcgen05.ld / st are complete before S and O are touched again
      // what the products of this tile and the scores of the one after next read has landed: looked for by one warp per group
      if (quarter == 0) {
        if (g == 0 ? !wait_all(&v_full[st], full_parity(n), 32) : n + 2 < N && !wait_all(&k_full[st], full_parity(n + 2), 32)) { alive = false; break; }
      }
      mbar_arrive1(&p_ready[st]);
    }
    // ---- both groups' sums: the half of the head dimension that this group writes, from both accumulators ----
    if (n > 0 && alive) alive = wait_all(&o_full[(n - 1) & 1], ((n - 1) >> 1) & 1, 39);
    float* const ml = reinterpret_cast<float*>(p_s + g * PANEL);
    ml[r] = m_run;
    ml[BQ + r] = l_run;
    tc5::tc_fence_before();
    asm volatile("bar.sync 1, 256;" ::: "memory");
    tc5::tc_fence_after();
    if (alive) {
      const float *ml_0 = reinterpret_cast<const float*>(p_s) + r, *ml_1 = reinterpret_cast<const float*>(p_s + PANEL) + r;
      const float m_0 = ml_0[0], m_1 = ml_1[0];
      const float m_all = fmaxf(m_0, m_1), m_ref = m_all == -INFINITY ? 0.f : m_all;
      float w_0 = ex2(m_0 - m_ref), w_1 = ex2(m_1 - m_ref);
      const float l_all = ml_0[BQ] * w_0 + ml_1[BQ] * w_1;
      const float inv = l_all > 0.f ? 1.f / l_all : 0.f;   // a row whose mask admits no key gives zeros
      w_0 *= inv;
      w_1 *= inv;
      T* orow = static_cast<T*>(p.out) + ((static_cast<int64_t>(b) * p.T + q0 + r) * p.Hq + h) * PD + g * 64;
#pragma unroll 1
      for (int q = 0; q < 64; q += 16) {
        float t0[16], t1[16];
        if (n > 0) {
          tc5::tmem_ld_32x16(t_lane + 256 + g * 64 + q, t0);
          tc5::tmem_ld_32x16(t_lane + 384 + g * 64 + q, t1);
          tc5::tmem_ld_wait();
        } else {
#pragma unroll
          for (int e = 0; e < 16; ++e) t0[e] = t1[e] = 0.f;
        }
        if (r < rows_valid) {
#pragma unroll
          for (int k = 0; k < 2; ++k) {
            float f[8];
#pragma unroll
            for (int e = 0; e < 8; ++e) f[e] = fmaf(t1[8 * k + e], w_1, t0[8 * k + e] * w_0);
            reinterpret_cast<uint4*>(orow + q)[k] = pack8<T>(f);
          }
        }
      }
    }
  }
  tc5::tc_fence_before();
  __syncthreads();
  if (warp == 8) { tc5::tc_fence_after(); tc5::tmem_dealloc(tmem_base, TMEM_COLS); }
}

template <typename T>
int launch_prefill_tc5(const PrefillParams& p, int dtype, cudaStream_t st) {
  static PerDevice<bool> configured_on;
  bool* configured = configured_on.slot();
  if (!configured) return B200_ENOTSUP;
  if (!*configured) {
    if (cudaFuncSetAttribute(attn_prefill_tc5_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, PF5_SMEM) != cudaSuccess) {
      cudaGetLastError();
      return B200_ENOTSUP;
    }
    *configured = true;
  }
  CUtensorMap mq, mk, mv, mm;
  auto st_of = [](int64_t elems, uint64_t fallback) { return elems > 0 ? static_cast<uint64_t>(elems) * 2 : fallback; };
  // [batch, head, row, 128] as (64, rows, 2, heads, batch): a box of (64, 128, 2) lands as two panels of [128 rows][128 bytes]
  auto map5 = [&](CUtensorMap* m, const void* base, int64_t rows, int heads, const int64_t* strides) {
    const uint64_t dims[5] = {64, static_cast<uint64_t>(rows), 2, static_cast<uint64_t>(heads), static_cast<uint64_t>(p.B)};
    const uint64_t str[4] = {st_of(strides[2], PD * 2), 128, st_of(strides[1], PD * 2), st_of(strides[0], PD * 2)};
    const uint32_t box[5] = {64, 128, 2, 1, 1};
    return tma_encode_sw128(m, dtype, 5, base, dims, str, box);
  };
  if (!map5(&mq, p.q, p.T, p.Hq, p.qs) || !map5(&mk, p.k, p.S, p.Hkv, p.ks) || !map5(&mv, p.v, p.S, p.Hkv, p.vs)) return B200_ENOTSUP;
  mm = mq;
  if (p.mask) {
    const uint64_t dims[3] = {static_cast<uint64_t>(p.S), static_cast<uint64_t>(p.T), static_cast<uint64_t>(p.mask_b == 0 ? 1 : p.B)};
    const uint64_t str[2] = {static_cast<uint64_t>(p.mask_t) * 2, st_of(p.mask_b, static_cast<uint64_t>(p.mask_t) * 2)};
    const uint32_t box[3] = {64, BQ, 1};
    if (!tma_encode_sw128(&mm, dtype, 3, p.mask, dims, str, box)) return B200_ENOTSUP;
  }
  dim3 grid(static_cast<unsigned>(p.Hq), static_cast<unsigned>((p.T + BQ - 1) / BQ), static_cast<unsigned>(p.B));
  launch_pdl(attn_prefill_tc5_kernel<T>, grid, dim3(PF5_THREADS), PF5_SMEM, st, mq, mk, mv, mm, p);
  return cudaGetLastError() == cudaSuccess ? B200_OK : B200_ELAUNCH;
}

}  // namespace

#undef g_tc5_error
int attn_prefill_tc5_error(bool clear) {
  int v = 0;
  if (cudaMemcpyFromSymbol(&v, g_attn5_error, sizeof(int)) != cudaSuccess) return -1;
  if (clear && v) {
    const int zero = 0;
    cudaMemcpyToSymbol(g_attn5_error, &zero, sizeof(int));
  }
  return v;
}

// Keys and masks that this kernel takes.
// One 64-key tile of the mma.sync kernel: no barriers, tensor memory or 128-key tile to set up for it.  us, 12 heads, here -> there: 16 x 16
// 5.5 -> 3.8 (64-key tiles on this path had taken 5.1), 63 x 63 6.1 -> 4.6, 64 x 64 5.8 -> 4.7, 16 sequences of 64 11.2 -> 6.9, 128 x 64 6.5 -> 4.8;
// 65 keys, 16 sequences 12.6 -> 12.3, two queries 4.8 -> 5.6; 128 x 128 7.1 -> 6.2, 16 sequences 13.4 -> 14.6.
static bool keys_fit(int64_t S) { return S > 64 && S <= static_cast<int64_t>(BKV) * MAX_TILES; }
// The mask's mixed tiles travel by TMA: aligned rows, of any length.
static bool mask_fits(const void* mask, int mask_dtype, int64_t S, int64_t mask_b, int64_t mask_t, int dtype) {
  return mask_dtype == dtype && aligned16(mask) && mask_b % 8 == 0 && mask_b >= 0 && mask_t >= S && mask_t % 8 == 0;
}

int attn_prefill_tc5(const PrefillParams& p, int dtype, cudaStream_t stream) {
  if (dtype != B200_BF16 && dtype != B200_F16) return B200_ENOTSUP;
  if (!keys_fit(p.S) || (p.T + BQ - 1) / BQ > 65535 || p.Hq % p.Hkv) return B200_ENOTSUP;
  if (p.mask && !mask_fits(p.mask, p.mask_dtype, p.S, p.mask_b, p.mask_t, dtype)) return B200_ENOTSUP;
  // TMA: 16-byte aligned bases (checked by the caller) and strides that are multiples of 16 bytes
  for (int i = 0; i < 3; ++i)
    if (p.qs[i] % 8 || p.ks[i] % 8 || p.vs[i] % 8 || p.qs[i] < 0 || p.ks[i] < 0 || p.vs[i] < 0) return B200_ENOTSUP;
  return dtype == B200_BF16 ? launch_prefill_tc5<__nv_bfloat16>(p, dtype, stream) : launch_prefill_tc5<__half>(p, dtype, stream);
}

}  // namespace b200

using namespace b200;

extern "C" int b200_mask_tiles(const void* mask, int64_t B, int64_t T, int64_t S, int64_t mask_b, int64_t mask_t, int dtype, void* tiles, void* stream) {
  B200_CHECK_ARG(mask && tiles && B >= 0 && T >= 0 && S >= 0, "b200_mask_tiles: bad arguments");
  const int64_t rows = ceil_div(T, BQ), cols = ceil_div(S, BKV);
  if (B == 0 || rows == 0 || cols == 0) return B200_OK;
  B200_CHECK_ARG(B <= 65535 && rows <= 65535 && cols < (1ll << 31), "b200_mask_tiles: mask too large");
  const dim3 grid(static_cast<unsigned>(cols), static_cast<unsigned>(rows), static_cast<unsigned>(B));
  B200_DISPATCH_HALF(dtype, T_, {
    launch_pdl(mask_tiles_kernel<T_>, grid, dim3(256), 0, static_cast<cudaStream_t>(stream), static_cast<const T_*>(mask), T, S, mask_b, mask_t,
               static_cast<uint8_t*>(tiles));
  });
  B200_CHECK_LAUNCH("mask_tiles_kernel");
  return B200_OK;
}

extern "C" int b200_attn_prefill_reads_tiles(const void* mask, int64_t S, int64_t mask_b, int64_t mask_t, int dtype) {
  return tc5_enabled() && mask && (dtype == B200_BF16 || dtype == B200_F16) && keys_fit(S) && mask_fits(mask, dtype, S, mask_b, mask_t, dtype) ? 1 : 0;
}

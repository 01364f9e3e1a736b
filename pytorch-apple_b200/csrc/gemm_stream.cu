// Weight-streaming GEMM for a few rows (decode):  out[M,N] = epi(A[M,K] * W[N,K]^T + bias + residual), M <= 24.
//
// With a handful of rows the weights are the work: every byte of W is read once and nothing else matters as long
// as enough of them are in flight, from before the predecessor has finished until the last one has arrived.
// - The problem is transposed: 16 weight rows are the M side of mma.sync m16n8k16, 8 sequences its N side (8 flop/B
//   at 8 rows: the legacy tensor path is far from its limit, and a warp needs no barrier to feed it).
// - Weights go from memory straight into the registers that are the MMA operands: k is permuted alike in both operands,
//   so that thread t of a quad owns k = 16t..16t+15 of a 64-wide chunk - one 256-bit load per row, a full 128-byte line
//   per quad.  Two chunks per warp (128 registers) are in flight; the registers of a 16-row tile are reloaded as soon
//   as its MMAs have been issued.  No shared-memory ring, no barrier, no copy-and-read-back per byte.
// - A CTA is 64 output columns x one K range, four warps interleaved over the 64-wide chunks; two CTAs fit an SM, so
//   the next kernel's first chunks (B200_EPI_W_STATIC, programmatic launch) load next to this one's tail.
// - Too few column blocks for the chip: the K ranges of one block form a thread-block cluster; after a sum over the
//   warps each row's partial sums go to the CTA that owns the row (distributed shared memory, one cluster barrier,
//   added in rank order: deterministic).
// - Gated pairs and rotary halves (columns c and c + 64) are the two row halves of one MMA tile, so they meet in
//   one thread of the final pass.
// Bound by HBM for the wide layers and by the chain release -> activations from L2 -> exchange -> final pass for the
// narrow ones.  us per GEMM in a chain of 28 layers of the 1.5B model, gemm_tc5_kernel -> this kernel (q/k/v, output,
// gate/up, down projection; 6.3, 4.7, 55 and 27.5 MB of weights, so 1.0, 0.7, 8.4 and 4.2 us at the copy rate):
//    1 row    6.3 ->  4.0    5.0 ->  3.1   13.3 ->  9.6    9.3 ->  7.2   vocabulary (467 MB) 105 -> 74 (6.3 TB/s)
//    8 rows   6.6 ->  4.7    5.4 ->  3.5   12.8 -> 10.5    9.8 ->  7.7                       100 -> 76
//   16 rows   7.7 ->  6.0    5.4 ->  4.0   13.4 -> 13.5    9.8 ->  9.3                        99 -> 84
// The activations of a CTA's K range stay in shared memory, which bounds the rows that two CTAs per SM can take: 16 for
// a 1536-wide unsplit row and for an eighth of 8960, 24 for a sixth of 1536 (q/k/v and output projection at 19 rows 7.4 ->
// 6.1 and 5.4 -> 4.1 us); other rows stay with the tensor-map kernel (gate/up at 19 rows: 13.1 there, 22 here).
// The eviction hint on the weights does not cost those that fit L2 and come again: 1536 x 8960, one row, in L2 4.7 us,
// from memory 7.2 (tensor-map kernel 8.2 and 9.3).
// Measured and not used: the same loop on a cp.async ring (paced by shared-memory traffic and waits: 28.9 against 24.6 us
// per layer), prefetching a later part of the weights into L2 (every form slower, by up to 13 us per layer).
#include "gemm_epilogue.cuh"
#include "tc5.cuh"

namespace b200 {
namespace {

constexpr int SW_COLS = 64, SW_WARPS = 4, SW_THREADS = SW_WARPS * 32, SW_CHUNK = 64, SW_PITCH = SW_COLS + 4;
constexpr int SW_STRIDE = SW_WARPS * SW_CHUNK;   // k from one chunk of a warp to its next
constexpr int SW_DEPTH = 2;                      // weight chunks in flight per warp
constexpr int SW_CARVEOUT = 60;                  // percent of the 228 KB, see launch_stream
constexpr int SW_SMEM_MAX = 66 * 1024;           // two CTAs in that share (1 KB each is the system's)

template <int NT> struct SwCfg {   // NT = groups of 8 rows
  static constexpr int ROWS = NT * 8;
  static constexpr int X_CHUNK = NT * 1024;                          // activations of one chunk: a warp's words in operand order
  static constexpr int PART = SW_WARPS * ROWS * SW_PITCH * 4;        // fp32 sums of the four warps
  static constexpr int RECV = (ROWS + 8) * SW_PITCH * 4;             // split-K: slots of the rows this CTA owns
};

struct SwParams {
  Tc5Params e;                   // epilogue fields
  const void* A; const void* W;
  int64_t lda, ldw;
  int units, chunks;             // 64-column blocks, 64-wide chunks of K
  int chunks_per_split, splits;
  int x_chunks;                  // chunks of a warp, at most
  int rpo, rpo_inv;              // rows per owner, ceil(2^16 / rpo)
};

struct W8 { uint32_t r[8]; };    // 16 consecutive k of one weight row
__device__ __forceinline__ void ld_stream(W8& v, const void* p) {
  asm volatile("ld.global.L1::evict_first.L2::evict_first.v8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
               : "=r"(v.r[0]), "=r"(v.r[1]), "=r"(v.r[2]), "=r"(v.r[3]), "=r"(v.r[4]), "=r"(v.r[5]), "=r"(v.r[6]), "=r"(v.r[7]) : "l"(p));
}

// What the final pass needs besides the sums, for row m and this lane's column pair; requested before the main loop.
template <typename T> struct Tail { T res_a, res_b, cl, ch, sl, sh; float rinv; };

template <typename T, int NT>
__global__ void __launch_bounds__(SW_THREADS, 2) gemm_stream_kernel(const __grid_constant__ SwParams p) {
  using C = SwCfg<NT>;
  extern __shared__ __align__(16) uint8_t smem_raw[];
  __shared__ float s_rinv[C::ROWS];
  float* const part = reinterpret_cast<float*>(smem_raw);
  float* const recv = part + C::PART / 4;
  uint4* const x_sm = reinterpret_cast<uint4*>(smem_raw + C::PART + (p.splits > 1 ? C::RECV : 0));
  const Tc5Params& e = p.e;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int M = static_cast<int>(e.M);
  const int nsp = p.splits, rank = blockIdx.y;
  const bool glu = (e.epilogue & B200_EPI_GLU) != 0, rope = e.rope.cos != nullptr, paired = glu || rope;
  const int c0 = rank * p.chunks_per_split + warp, c1 = min(p.chunks, rank * p.chunks_per_split + p.chunks_per_split);   // this warp: c0, c0 + 4, ..
  const int nmy = c1 > c0 ? (c1 - c0 + SW_WARPS - 1) / SW_WARPS : 0;

  if (nsp > 1) tc5::cluster_arrive();   // peers must be running before anyone writes into their memory (waited for below)

  // ---- weights: w[slot][2j + h] = row half h of MMA tile j
  const int64_t sj = (paired ? 8 : 16) * p.ldw, sh = (paired ? 64 : 8) * p.ldw;   // elements between tiles / row halves
  auto unit_row = [&](int u) { return static_cast<int64_t>(paired ? (u >> 1) * 128 + (u & 1) * 32 : u * SW_COLS); };
  auto w_src = [&](int u) { return static_cast<const T*>(p.W) + (unit_row(u) + g) * p.ldw + c0 * SW_CHUNK + t * 16; };
  W8 w[SW_DEPTH][8];
  const T* wp = w_src(blockIdx.x);
  // weights that no kernel of this stream writes are requested before the predecessor has finished
  if (!(e.epilogue & B200_EPI_W_STATIC)) pdl_wait();
#pragma unroll
  for (int d = 0; d < SW_DEPTH; ++d)
    if (d < nmy) {
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        ld_stream(w[d][2 * j], wp + d * SW_STRIDE + j * sj);
        ld_stream(w[d][2 * j + 1], wp + d * SW_STRIDE + j * sj + sh);
      }
    }
  pdl_wait();
  // The successor may start from here on, not before: it would let kernels two steps ahead take the registers that
  // this kernel's and the attention's blocks still need (a layer of one sequence: 38.8 us triggered at the start, 34.1 here).
  pdl_trigger();

  // ---- activations, in operand order (a lane reads back its own words); rows that do not exist read as zero
  uint4* const x_own = x_sm + warp * p.x_chunks * (C::X_CHUNK / 16) + lane;
  {
    constexpr int XB = 6 / NT;   // chunks requested together
    const T* const src = static_cast<const T*>(p.A) + g * p.lda + c0 * SW_CHUNK + t * 16;
#pragma unroll 1
    for (int b = 0; b < nmy; b += XB) {
      uint4 v[XB][NT][2];
#pragma unroll
      for (int j = 0; j < XB; ++j)
#pragma unroll
        for (int i = 0; i < NT; ++i) {
          const bool ok = b + j < nmy && 8 * i + g < M;
          const uint4* s = reinterpret_cast<const uint4*>(src + i * 8 * p.lda + (b + j) * SW_STRIDE);
          v[j][i][0] = ok ? __ldcg(s) : make_uint4(0u, 0u, 0u, 0u);
          v[j][i][1] = ok ? __ldcg(s + 1) : make_uint4(0u, 0u, 0u, 0u);
        }
#pragma unroll
      for (int j = 0; j < XB; ++j)
#pragma unroll
        for (int i = 0; i < NT; ++i)
          if (b + j < nmy) {
            x_own[((b + j) * NT + i) * 64] = v[j][i][0];
            x_own[((b + j) * NT + i) * 64 + 32] = v[j][i][1];
          }
    }
  }

  // RMSNorm factor of the input rows, needed in the final pass only: the four lanes of a quad request the partials of a row
  // together, then add them up in index order, as the tensor-map kernel does.  (Decode step of eight sequences, us: 1128;
  // a sum per lane and two exchanges, in another order, 1137; a thread per row with all loads of its own 1371.)
  static_assert(STREAM_MAX_ROWS <= SW_THREADS / 4 && NORM_MAX_PARTS % 4 == 0, "a quad per row");
  if (const int m = threadIdx.x >> 2; e.sumsq_in && m < M) {
    const float* sp = e.sumsq_in + static_cast<int64_t>(m) * e.sumsq_in_cols + t;
    float v[NORM_MAX_PARTS / 4];
#pragma unroll
    for (int j = 0; j < NORM_MAX_PARTS / 4; ++j) v[j] = 4 * j + t < e.sumsq_in_cols ? __ldcg(sp + 4 * j) : 0.f;
    const unsigned quad = 0xfu << (lane & 28);
    float ss = 0.f;
#pragma unroll
    for (int j = 0; j < NORM_MAX_PARTS; ++j) ss += __shfl_sync(quad, v[j >> 2], (lane & 28) + (j & 3));
    if (t == 0) s_rinv[m] = 1.0f / sqrtf(ss / static_cast<float>(e.K) + e.norm_eps);
  }
  // The final pass: a warp per row, a lane two of its 64 columns (2 lane, 2 lane + 1; gated / rotary: lane and its other
  // half).  It runs once per CTA, so what it costs is instructions fetched: one pair per lane is the shortest code.
  const int own0 = rank * p.rpo, own_rows = min(p.rpo, M - own0);   // (may be negative; one split: all rows)
  const int ca = paired ? lane : 2 * lane, cb = paired ? lane + 32 : 2 * lane + 1;   // in the block
  T* const outp = static_cast<T*>(e.out);
  const T* const resp = static_cast<const T*>(e.residual);
  auto fetch_tail = [&](Tail<T>& tl, int lr, int64_t na, int64_t nb) {
    const int64_t m = own0 + lr;
    if (resp) { tl.res_a = resp[m * e.ldr + na]; tl.res_b = resp[m * e.ldr + nb]; }
    if (rope) {
      const int64_t i = m * 128 + (na & 127);
      tl.cl = static_cast<const T*>(e.rope.cos)[i]; tl.ch = static_cast<const T*>(e.rope.cos)[i + 64];
      tl.sl = static_cast<const T*>(e.rope.sin)[i]; tl.sh = static_cast<const T*>(e.rope.sin)[i + 64];
    }
  };
  int64_t pos = 0;
  if (rope) pos = load_index(e.rope.cache_pos, 0, e.rope.pos_dtype);

  __syncwarp();
  if (nsp > 1) tc5::cluster_wait();
#pragma unroll 1
  for (int u = blockIdx.x; u < p.units; u += gridDim.x) {
    const int64_t na = unit_row(u) + ca, nb = paired ? na + 64 : na + 1;   // this lane's columns in the final pass
    float bias_a = 0.f, bias_b = 0.f;
    if (e.bias) { bias_a = load_as_f32(e.bias, na, e.bias_dtype); bias_b = load_as_f32(e.bias, nb, e.bias_dtype); }
    Tail<T> tail;
    if (warp < own_rows) fetch_tail(tail, warp, na, nb);
    const int un = u + gridDim.x;
    const T* const wn = un < p.units ? w_src(un) : nullptr;   // the next unit's weights

    float acc[4][NT][4];
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int i = 0; i < NT; ++i)
#pragma unroll
        for (int k = 0; k < 4; ++k) acc[j][i][k] = 0.f;
#pragma unroll 1
    for (int c = 0; c < nmy; c += SW_DEPTH) {
#pragma unroll
      for (int d = 0; d < SW_DEPTH; ++d) {
        if (c + d < nmy) {
          uint32_t x[NT][8];
#pragma unroll
          for (int i = 0; i < NT; ++i) {
            const uint4 x0 = x_own[((c + d) * NT + i) * 64], x1 = x_own[((c + d) * NT + i) * 64 + 32];
            x[i][0] = x0.x; x[i][1] = x0.y; x[i][2] = x0.z; x[i][3] = x0.w;
            x[i][4] = x1.x; x[i][5] = x1.y; x[i][6] = x1.z; x[i][7] = x1.w;
          }
          // the chunk that takes this slot next: of this unit, else of the next one
          const T* const next = c + d + SW_DEPTH < nmy ? wp + (c + d + SW_DEPTH) * SW_STRIDE : wn ? wn + d * SW_STRIDE : nullptr;
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const W8 &lo = w[d][2 * j], &hi = w[d][2 * j + 1];
#pragma unroll
            for (int s = 0; s < 4; ++s) {
              const uint32_t a[4] = {lo.r[2 * s], hi.r[2 * s], lo.r[2 * s + 1], hi.r[2 * s + 1]};
#pragma unroll
              for (int i = 0; i < NT; ++i) {
                const uint32_t b[2] = {x[i][2 * s], x[i][2 * s + 1]};
                MmaType<T>::mma(acc[j][i], a, b);
              }
            }
            if (next) {
              ld_stream(w[d][2 * j], next + j * sj);
              ld_stream(w[d][2 * j + 1], next + j * sj + sh);
            }
          }
        }
      }
    }
    wp = wn;

    // ---- sums of the four warps: acc[j][i] holds columns (tile j, row g / g + 8) of rows 8i + 2t, 8i + 2t + 1
    if (u != static_cast<int>(blockIdx.x)) __syncthreads();   // the previous unit's sums have been read
    {
      const int cl = paired ? 8 : 16, ch = paired ? 32 : 8;
#pragma unroll
      for (int i = 0; i < NT; ++i) {
        const int m = 8 * i + 2 * t;
        float* d = part + (warp * C::ROWS + m) * SW_PITCH + g;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          if (m < M) { d[j * cl] = acc[j][i][0]; d[j * cl + ch] = acc[j][i][2]; }
          if (m + 1 < M) { d[SW_PITCH + j * cl] = acc[j][i][1]; d[SW_PITCH + j * cl + ch] = acc[j][i][3]; }
        }
      }
    }
    __syncthreads();
    const float* fsrc = part;             // where the final pass finds its slots
    int fslots = SW_WARPS, fstride = C::ROWS * SW_PITCH;
    if (nsp > 1) {
#pragma unroll 1
      for (int idx = threadIdx.x; idx < M << 4; idx += SW_THREADS) {
        const int m = idx >> 4, c = (idx & 15) << 2;
        const float* s = part + m * SW_PITCH + c;
        float4 v = *reinterpret_cast<const float4*>(s);
#pragma unroll
        for (int k = 1; k < SW_WARPS; ++k) {
          const float4 a = *reinterpret_cast<const float4*>(s + k * C::ROWS * SW_PITCH);
          v.x += a.x; v.y += a.y; v.z += a.z; v.w += a.w;
        }
        const int owner = (m * p.rpo_inv) >> 16;
        tc5::st_cluster_f4(tc5::map_to_rank(smem_u32(recv + (rank * p.rpo + m - owner * p.rpo) * SW_PITCH + c), owner), v.x, v.y, v.z, v.w);
      }
      __syncwarp();
      tc5::cluster_sync();                // after this nobody touches a peer's memory
      fsrc = recv; fslots = nsp; fstride = p.rpo * SW_PITCH;
    }
#pragma unroll 1
    for (int lr = warp; lr < own_rows; lr += SW_WARPS) {
      const int64_t m = own0 + lr;
      const float* s = fsrc + lr * SW_PITCH;
      float a = 0.f, b = 0.f;
#pragma unroll 4
      for (int k = 0; k < fslots; ++k, s += fstride) { a += s[ca]; b += s[cb]; }
      if (e.sumsq_in) { a *= s_rinv[m]; b *= s_rinv[m]; }
      a += bias_a; b += bias_b;
      if (glu) {
        round2<T>(a, b);
        outp[m * e.ldo + (u >> 1) * 64 + (u & 1) * 32 + lane] = from_f32<T>(round_as<T>(silu_f32(a)) * b);
      } else if (rope) {
        // rounded as the linear layer's output; x*cos + rotate_half(x)*sin with the roundings of the unfused operators
        // (both products, then the sum) for query and key heads, to rope(q) / the cache rows
        const Tc5Args::Rope& r = e.rope;
        const int head = u >> 1, hk = head - r.Hq, c = (u & 1) * 32 + lane;
        round2<T>(a, b);
        if (hk < r.Hkv) {
          const float lo = a, hi = b;
          a = round_as<T>(lo * to_f32<T>(tail.cl)) + round_as<T>(-hi * to_f32<T>(tail.sl));
          b = round_as<T>(hi * to_f32<T>(tail.ch)) + round_as<T>(lo * to_f32<T>(tail.sh));
        }
        T* dst = static_cast<T*>(r.q_out) + (m * r.Hq + head) * 128 + c;
        const int64_t row = pos < 0 ? pos + r.cache_len : pos;
        if (hk >= 0) dst = static_cast<T*>(hk < r.Hkv ? r.k_cache : r.v_cache) + ((m * r.Hkv + hk - (hk < r.Hkv ? 0 : r.Hkv)) * r.cache_len + row) * 128 + c;
        if (hk < 0 || (row >= 0 && row < r.cache_len)) { dst[0] = from_f32<T>(a); dst[64] = from_f32<T>(b); }
      } else {
        if (resp) {
          round2<T>(a, b);
          a += to_f32<T>(tail.res_a); b += to_f32<T>(tail.res_b);
        }
        if (e.epilogue & B200_EPI_RELU) { a = fmaxf(a, 0.f); b = fmaxf(b, 0.f); }
        if (e.epilogue & B200_EPI_SILU_MUL) {
          const T* aux = static_cast<const T*>(e.aux) + m * e.ldaux + na;
          round2<T>(a, b);
          a = round_as<T>(silu_f32(a)) * to_f32<T>(aux[0]);
          b = round_as<T>(silu_f32(b)) * to_f32<T>(aux[1]);
        }
        T* o = outp + m * e.ldo + na;
        if ((reinterpret_cast<uintptr_t>(o) & 3u) == 0) {
          *reinterpret_cast<uint32_t*>(o) = pack2<T>(a, b);
        } else {
          o[0] = from_f32<T>(a);
          o[1] = from_f32<T>(b);
        }
        if (e.sumsq_out) {   // one partial per row and 64-column block: the warp holds it
          round2<T>(a, b);
          const float sq = warp_sum(a * a + b * b);
          if (lane == 0) e.sumsq_out[m * (e.N >> 6) + u] = sq;
        }
      }
      if (lr + SW_WARPS < own_rows) fetch_tail(tail, lr + SW_WARPS, na, nb);
    }
  }
}

struct SwPlan { int units, chunks, splits, chunks_per_split; };

// Column blocks are split along K (clusters of up to eight) until about every SM has a CTA or two: the down projection
// of one row takes 7.2 us with eight splits (192 CTAs), 8.2 with six, 10.5 with four; the short reductions are level
// from four splits on.  Larger (non-portable) clusters lose: ten 7.9, twelve 9.9 us.  Besides:
// - One block per SM, no split: four warps do not keep enough loads in flight, and from 9 rows on the tensor-map kernel
//   was faster; two splits where a half still fills the loads in flight of its warps (us: N 8960, K 1536: 1 row 7.6 -> 5.8,
//   16 rows 10.0 -> 7.5, tensor-map kernel 9.5; N 9472, K 3584, 8 rows 17.7 -> 12.5, 14.5; with K 512 two splits lose: 2.6 -> 3.3).
// - Four splits for three where that leaves a warp fewer chunks (K = N = 3584: 1 row 7.1 -> 6.1, 16 rows 9.2 -> 8.0, tensor-map
//   kernel 8.7; N 3840, K 1536, two chunks per warp either way, loses: 9 rows 4.5 -> 4.9).
SwPlan plan_stream(int64_t N, int64_t K) {
  SwPlan pl;
  pl.units = static_cast<int>(N / SW_COLS);
  pl.chunks = static_cast<int>(K / SW_CHUNK);
  const auto per_warp = [&](int splits) { return ceil_div(ceil_div(pl.chunks, splits), SW_WARPS); };
  int s = 192 / pl.units;
  if (s > pl.chunks / SW_WARPS) s = pl.chunks / SW_WARPS;
  if (s > 8) s = 8;
  if (s < 1) s = 1;
  if (s == 1 && pl.units <= 148 && pl.chunks >= 2 * SW_WARPS * SW_DEPTH) s = 2;
  if (s == 3 && per_warp(4) < per_warp(3)) s = 4;
  pl.chunks_per_split = static_cast<int>(ceil_div(pl.chunks, s));
  pl.splits = static_cast<int>(ceil_div(pl.chunks, pl.chunks_per_split));
  return pl;
}

template <typename T, int NT> int launch_stream(const Tc5Args& a, cudaStream_t st) {
  using C = SwCfg<NT>;
  const SwPlan pl = plan_stream(a.N, a.K);
  SwParams p;
  p.x_chunks = static_cast<int>(ceil_div(pl.chunks_per_split, SW_WARPS));
  const int64_t smem = C::PART + (pl.splits > 1 ? C::RECV : 0) + static_cast<int64_t>(SW_WARPS) * p.x_chunks * C::X_CHUNK;
  if (smem > SW_SMEM_MAX) return B200_ENOTSUP;
  static PerDevice<bool> configured_on;
  bool* configured = configured_on.slot();
  if (!configured) return B200_ENOTSUP;
  if (!*configured) {
    // The loads in flight land in L1, so shared memory must not take all of an SM (layer of one row 24.6 us at 60 %, 25.5 at
    // 80, 32.9 at 100); left to itself the driver takes the least that fits, and then every SM is reconfigured between
    // this kernel and the attention (layer of eight rows with its attention 44.1 us by default, 36.6 at 60 %).
    if (cudaFuncSetAttribute(gemm_stream_kernel<T, NT>, cudaFuncAttributeMaxDynamicSharedMemorySize, SW_SMEM_MAX) != cudaSuccess ||
        cudaFuncSetAttribute(gemm_stream_kernel<T, NT>, cudaFuncAttributePreferredSharedMemoryCarveout, SW_CARVEOUT) != cudaSuccess) {
      cudaGetLastError();
      return B200_ENOTSUP;
    }
    *configured = true;
  }
  p.e = Tc5Params{};
  p.e.bias = a.bias; p.e.residual = a.residual; p.e.aux = a.aux; p.e.out = a.out;
  p.e.M = a.M; p.e.N = a.N; p.e.K = a.K; p.e.ldo = a.ldo; p.e.ldr = a.ldr; p.e.ldaux = a.ldaux;
  p.e.bias_dtype = a.bias_dtype; p.e.epilogue = a.epilogue;
  p.e.norm_eps = a.norm_eps; p.e.sumsq_in = a.sumsq_in; p.e.sumsq_in_cols = a.sumsq_in_cols; p.e.sumsq_out = a.sumsq_out;
  p.e.rope = a.rope;
  p.A = a.A; p.W = a.W; p.lda = a.lda; p.ldw = a.ldw;
  p.units = pl.units; p.chunks = pl.chunks; p.splits = pl.splits; p.chunks_per_split = pl.chunks_per_split;
  p.rpo = static_cast<int>(ceil_div(a.M, pl.splits));
  p.rpo_inv = (65536 + p.rpo - 1) / p.rpo;
  const int slots = 2 * sm_count();
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(static_cast<unsigned>(pl.splits > 1 || pl.units < slots ? pl.units : slots), static_cast<unsigned>(pl.splits));
  cfg.blockDim = dim3(SW_THREADS);
  cfg.dynamicSmemBytes = static_cast<size_t>(smem);
  cfg.stream = st;
  cudaLaunchAttribute attrs[2];
  int n_attrs = 0;
  if (pdl_enabled()) {
    attrs[n_attrs].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attrs[n_attrs].val.programmaticStreamSerializationAllowed = 1;
    ++n_attrs;
  }
  if (pl.splits > 1) {
    attrs[n_attrs].id = cudaLaunchAttributeClusterDimension;
    attrs[n_attrs].val.clusterDim.x = 1;
    attrs[n_attrs].val.clusterDim.y = static_cast<unsigned>(pl.splits);
    attrs[n_attrs].val.clusterDim.z = 1;
    ++n_attrs;
  }
  cfg.attrs = attrs;
  cfg.numAttrs = n_attrs;
  cudaLaunchKernelEx(&cfg, gemm_stream_kernel<T, NT>, p);
  B200_CHECK_LAUNCH("gemm_stream_kernel");
  return B200_OK;
}

template <typename T> int dispatch_stream(const Tc5Args& a, cudaStream_t st) {
  return a.M <= 8 ? launch_stream<T, 1>(a, st) : a.M <= 16 ? launch_stream<T, 2>(a, st) : launch_stream<T, 3>(a, st);
}

}  // namespace

int linear_stream(const Tc5Args& a, cudaStream_t st) {
  // whole column blocks and chunks, 32-byte aligned weight rows; other shapes stay with the tensor-map kernels
  if (a.M > STREAM_MAX_ROWS || a.N % SW_COLS || a.K % SW_CHUNK || a.ldw % 16 || (reinterpret_cast<uintptr_t>(a.W) & 31u)) return B200_ENOTSUP;
  return a.dtype == B200_BF16 ? dispatch_stream<__nv_bfloat16>(a, st) : dispatch_stream<__half>(a, st);
}

}  // namespace b200

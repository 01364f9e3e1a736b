// Kernel parameters and fp32 epilogues shared by the 16-bit GEMM kernels (gemm_tc5.cu, gemm_stream.cu): bias, residual,
// ReLU, silu * mul, the gated pair, and the rotary embedding with its q / KV-cache destinations.
#pragma once
#include "gemm_tc5.cuh"
#include "mma.cuh"

namespace b200 {

struct Tc5Params {
  const void* bias; const void* residual; const void* aux; void* out;
  int64_t M, N, K, ldo, ldr, ldaux;
  int bias_dtype, epilogue, splits, kb_per_split;
  const void* x;   // convolution input (implicit-GEMM mode only)
  Tc5Conv g;
  // persistent kernel: shared-memory plan chosen by the host (bytes from the aligned base)
  int pst, pstage;      // ring stages and bytes per stage
  int wr, w_off;        // weights resident: all k-blocks of the CTA's weight tile stay in shared memory at w_off
  int pncb, c_off;      // C buffers (bulk-copy epilogue) and where they start
  int npa;              // persistent kernel: activation producer threads (1 or 2), ring stages dealt round-robin
  int kps;              // persistent kernel: k-blocks per ring stage (1 or 2): one barrier hand-off covers that many
  int nfast;            // persistent kernel: column tiles fastest in the tile order
  // one-tile kernel, M <= 64: scale the output rows by the RMSNorm factor of the input rows / write
  // sum-of-squares partials of the output rows
  const float* sumsq_in; float* sumsq_out;
  float norm_eps;
  int sumsq_in_cols;
  // CTA-pair kernel with split-K (p.splits > 1): fp32 partial sums [split][M][N] instead of outputs
  float* partial;
  // one-tile kernel, M <= 64, 128-wide tiles: rotary embedding + q / KV-cache destinations in the final pass
  Tc5Args::Rope rope;
};

// The CTA-pair kernel (gemm_pair.cu): tiles of 256 weight rows x up to 256 tokens; p.splits > 1: partial sums to p.partial.
int gemm_pair(const Tc5Args& a, const Tc5Params& p, cudaStream_t st);
int gemm_pair_error(bool clear);

template <typename T> struct AbFormat;
template <> struct AbFormat<__half> { static constexpr int value = 0; };
template <> struct AbFormat<__nv_bfloat16> { static constexpr int value = 1; };


// The epilogue code runs once or a few times per CTA, so it is written as short rolled loops
// over 16-column units: straight-line code unrolled over a whole tile row costs more in
// instruction fetch (cold instruction cache on every SM) than in execution.

// v[i] += bias[n + i]
template <int CNT>
__device__ __forceinline__ void add_bias(const Tc5Params& p, float (&v)[CNT], int64_t n, int cnt) {
  if (!p.bias) return;
  if (p.bias_dtype == B200_F32) {
    const float* __restrict__ bp = static_cast<const float*>(p.bias) + n;
#pragma unroll
    for (int i = 0; i < CNT; ++i) if (i < cnt) v[i] += bp[i];
  } else if (p.bias_dtype == B200_BF16) {
    const __nv_bfloat16* __restrict__ bp = static_cast<const __nv_bfloat16*>(p.bias) + n;
#pragma unroll
    for (int i = 0; i < CNT; ++i) if (i < cnt) v[i] += __bfloat162float(bp[i]);
  } else if (p.bias_dtype == B200_F16) {
    const __half* __restrict__ bp = static_cast<const __half*>(p.bias) + n;
#pragma unroll
    for (int i = 0; i < CNT; ++i) if (i < cnt) v[i] += __half2float(bp[i]);
  } else {
#pragma unroll
    for (int i = 0; i < CNT; ++i) if (i < cnt) v[i] += load_as_f32(p.bias, n + i, p.bias_dtype);   // (static indices keep v in registers)
  }
}

// CNT (8 or 16) consecutive values of row `row` of a [*, ld] matrix of T starting at column n
template <typename T, int CNT>
__device__ __forceinline__ void load_cols(const T* __restrict__ base, int64_t ld, int64_t row, int64_t n, int cnt, float (&f)[CNT]) {
  const T* src = base + row * ld + n;
  if (cnt == CNT && (reinterpret_cast<uintptr_t>(src) & 15u) == 0) {
#pragma unroll
    for (int j = 0; j < CNT / 8; ++j) {
      float t[8];
      unpack8<T>(reinterpret_cast<const uint4*>(src)[j], t);
#pragma unroll
      for (int i = 0; i < 8; ++i) f[8 * j + i] = t[i];
    }
  } else {
#pragma unroll
    for (int i = 0; i < CNT; ++i) f[i] = i < cnt ? to_f32<T>(src[i]) : 0.f;
  }
}

template <typename T, int CNT>
__device__ __forceinline__ void store_cols(T* __restrict__ dst, const float (&v)[CNT], int cnt) {
  if (cnt == CNT && (reinterpret_cast<uintptr_t>(dst) & 15u) == 0) {
#pragma unroll
    for (int j = 0; j < CNT / 8; ++j) {
      float f[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) f[i] = v[8 * j + i];
      reinterpret_cast<uint4*>(dst)[j] = pack8<T>(f);
    }
  } else {
#pragma unroll
    for (int i = 0; i < CNT; ++i) if (i < cnt) dst[i] = from_f32<T>(v[i]);
  }
}

// bias / residual / activation on CNT consecutive outputs of row m starting at column n, then store
template <typename T, int CNT>
__device__ __forceinline__ void finish_cols(const Tc5Params& p, float (&v)[CNT], int64_t m, int64_t n) {
  const int cnt = static_cast<int>(p.N - n < CNT ? p.N - n : CNT);
  add_bias<CNT>(p, v, n, cnt);
  if (p.residual) {
    float r[CNT];
    load_cols<T, CNT>(static_cast<const T*>(p.residual), p.ldr, m, n, cnt, r);
#pragma unroll
    for (int i = 0; i < CNT; i += 2) {
      round2<T>(v[i], v[i + 1]);
      v[i] += r[i]; v[i + 1] += r[i + 1];
    }
  }
  if (p.epilogue & B200_EPI_RELU) {
#pragma unroll
    for (int i = 0; i < CNT; ++i) v[i] = fmaxf(v[i], 0.f);
  }
  if (p.epilogue & B200_EPI_SILU_MUL) {
    float x[CNT];
    load_cols<T, CNT>(static_cast<const T*>(p.aux), p.ldaux, m, n, cnt, x);
#pragma unroll
    for (int i = 0; i < CNT; ++i) v[i] = round_as<T>(silu_f32(round_as<T>(v[i]))) * x[i];
  }
  store_cols<T, CNT>(static_cast<T*>(p.out) + m * p.ldo + n, v, cnt);
}

// gated-MLP epilogue: CNT gate accumulators (merged columns n_merged..) and the matching up
// accumulators (merged columns n_merged + 64 ..) of row m -> CNT outputs starting at column n_out
template <typename T, int CNT>
__device__ __forceinline__ void finish_glu_cols(const Tc5Params& p, float (&g)[CNT], float (&u)[CNT], int64_t m, int64_t n_merged, int64_t n_out) {
  add_bias<CNT>(p, g, n_merged, CNT);
  add_bias<CNT>(p, u, n_merged + 64, CNT);
#pragma unroll
  for (int i = 0; i < CNT; i += 2) {   // pairs: the three roundings to T go through packed conversions
    float g0 = g[i], g1 = g[i + 1], u0 = u[i], u1 = u[i + 1];
    round2<T>(g0, g1);
    g0 = silu_f32(g0); g1 = silu_f32(g1);
    round2<T>(g0, g1);
    round2<T>(u0, u1);
    g[i] = g0 * u0; g[i + 1] = g1 * u1;
  }
  store_cols<T, CNT>(static_cast<T*>(p.out) + m * p.ldo + n_out, g, CNT);
}

// Final pass of the merged q/k/v projection of a decode step: `lo` / `hi` are columns col..col+3 and
// col+64..col+67 of head `head` (a 128-wide tile) for sequence b.  Adds the bias, rounds to T as the linear
// layer's output is rounded, applies x*cos + rotate_half(x)*sin with the roundings of the unfused
// operators (both products, then the sum) to query and key heads, and stores to rope(q) / the cache rows.
template <typename T>
__device__ __forceinline__ void finish_rope4(const Tc5Params& p, const float4& lo4, const float4& hi4, int64_t b, int head, int col) {
  float lo[4] = {lo4.x, lo4.y, lo4.z, lo4.w}, hi[4] = {hi4.x, hi4.y, hi4.z, hi4.w};
  const int64_t n = static_cast<int64_t>(head) * 128 + col;
  add_bias<4>(p, lo, n, 4);
  add_bias<4>(p, hi, n + 64, 4);
#pragma unroll
  for (int i = 0; i < 4; ++i) { lo[i] = round_as<T>(lo[i]); hi[i] = round_as<T>(hi[i]); }
  const Tc5Args::Rope& r = p.rope;
  const int which = head < r.Hq ? 0 : (head < r.Hq + r.Hkv ? 1 : 2);
  if (which != 2) {
    const T* cs = static_cast<const T*>(r.cos) + b * 128 + col;
    const T* sn = static_cast<const T*>(r.sin) + b * 128 + col;
    float c0, c1, c2, c3, s0, s1, s2, s3, d0, d1, d2, d3, t0, t1, t2, t3;
    const uint2 cl = *reinterpret_cast<const uint2*>(cs), ch = *reinterpret_cast<const uint2*>(cs + 64);
    const uint2 sl = *reinterpret_cast<const uint2*>(sn), sh = *reinterpret_cast<const uint2*>(sn + 64);
    unpack2<T>(cl.x, c0, c1); unpack2<T>(cl.y, c2, c3); unpack2<T>(sl.x, s0, s1); unpack2<T>(sl.y, s2, s3);
    unpack2<T>(ch.x, d0, d1); unpack2<T>(ch.y, d2, d3); unpack2<T>(sh.x, t0, t1); unpack2<T>(sh.y, t2, t3);
    const float cl4[4] = {c0, c1, c2, c3}, sl4[4] = {s0, s1, s2, s3}, ch4[4] = {d0, d1, d2, d3}, sh4[4] = {t0, t1, t2, t3};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float a = lo[i], h = hi[i];
      lo[i] = round_as<T>(a * cl4[i]) + round_as<T>(-h * sl4[i]);
      hi[i] = round_as<T>(h * ch4[i]) + round_as<T>(a * sh4[i]);
    }
  }
  T* dst;
  if (which == 0) {
    dst = static_cast<T*>(r.q_out) + (b * r.Hq + head) * 128;
  } else {
    int64_t pos = load_index(r.cache_pos, 0, r.pos_dtype);
    if (pos < 0) pos += r.cache_len;
    if (pos < 0 || pos >= r.cache_len) return;
    const int hk = head - r.Hq - (which == 2 ? r.Hkv : 0);
    dst = static_cast<T*>(which == 1 ? r.k_cache : r.v_cache) + ((b * r.Hkv + hk) * r.cache_len + pos) * 128;
  }
  *reinterpret_cast<uint2*>(dst + col) = make_uint2(pack2<T>(lo[0], lo[1]), pack2<T>(lo[2], lo[3]));
  *reinterpret_cast<uint2*>(dst + col + 64) = make_uint2(pack2<T>(hi[0], hi[1]), pack2<T>(hi[2], hi[3]));
}

// four consecutive outputs of row m starting at column n (split-K final pass)
template <typename T>
__device__ __forceinline__ void finish4(const Tc5Params& p, const float4& acc, int64_t m, int64_t n) {
  float v[4] = {acc.x, acc.y, acc.z, acc.w};
  const int cnt = static_cast<int>(p.N - n < 4 ? p.N - n : 4);
  add_bias<4>(p, v, n, cnt);
  const T* __restrict__ res = static_cast<const T*>(p.residual);
  const T* __restrict__ aux = static_cast<const T*>(p.aux);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    if (i < cnt) {
      if (res) v[i] = round_as<T>(v[i]) + to_f32<T>(res[m * p.ldr + n + i]);
      if (p.epilogue & B200_EPI_RELU) v[i] = fmaxf(v[i], 0.f);
      if (p.epilogue & B200_EPI_SILU_MUL) v[i] = round_as<T>(silu_f32(round_as<T>(v[i]))) * to_f32<T>(aux[m * p.ldaux + n + i]);
    }
  }
  T* o = static_cast<T*>(p.out) + m * p.ldo + n;
  if (cnt == 4 && (reinterpret_cast<uintptr_t>(o) & 7u) == 0) {
    *reinterpret_cast<uint2*>(o) = make_uint2(pack2<T>(v[0], v[1]), pack2<T>(v[2], v[3]));
  } else {
#pragma unroll
    for (int i = 0; i < 4; ++i) if (i < cnt) o[i] = from_f32<T>(v[i]);
  }
}

// four gate accumulators and the matching up accumulators of row m (split-K final pass)
template <typename T>
__device__ __forceinline__ void finish_glu4(const Tc5Params& p, const float4& gate, const float4& up, int64_t m, int64_t n_merged, int64_t n_out) {
  float g[4] = {gate.x, gate.y, gate.z, gate.w}, u[4] = {up.x, up.y, up.z, up.w};
  add_bias<4>(p, g, n_merged, 4);
  add_bias<4>(p, u, n_merged + 64, 4);
#pragma unroll
  for (int i = 0; i < 4; i += 2) {
    float g0 = g[i], g1 = g[i + 1], u0 = u[i], u1 = u[i + 1];
    round2<T>(g0, g1);
    g0 = silu_f32(g0); g1 = silu_f32(g1);
    round2<T>(g0, g1);
    round2<T>(u0, u1);
    g[i] = g0 * u0; g[i + 1] = g1 * u1;
  }
  T* o = static_cast<T*>(p.out) + m * p.ldo + n_out;
  if ((reinterpret_cast<uintptr_t>(o) & 7u) == 0) {
    *reinterpret_cast<uint2*>(o) = make_uint2(pack2<T>(g[0], g[1]), pack2<T>(g[2], g[3]));
  } else {
#pragma unroll
    for (int i = 0; i < 4; ++i) o[i] = from_f32<T>(g[i]);
  }
}

}  // namespace b200

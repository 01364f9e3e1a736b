// Shared between the two prefill attention kernels (attention.cu: mma.sync; attn_prefill_tc5.cu: tcgen05).
#pragma once
#include "common.cuh"

namespace b200 {

// States of the tiles of an additive mask (b200_mask_tiles): nothing unmasked, all zero, anything else
constexpr int MASK_TILE = 128;
enum : uint8_t { MASK_TILE_NONE = 0, MASK_TILE_ZERO = 1, MASK_TILE_MIXED = 2 };

struct PrefillParams {
  const void* q; const void* k; const void* v; const void* mask; void* out;
  int64_t B, T, S;
  int Hq, Hkv;
  int64_t qs[3], ks[3], vs[3];
  int64_t mask_b, mask_t;
  const uint8_t* tiles;   // states of the mask's tiles, or nullptr: the kernel looks for itself
  float scale;
  int mask_dtype;
  int mask_staged;   // the mask can travel through shared memory (activation dtype, 16-byte-aligned rows)
};

// Prefill attention on the tcgen05 path (head_dim 128, 16-bit types, 16-byte aligned strides, 65 to 32768 keys, mask
// absent or in the activation type).  Returns B200_ENOTSUP for anything else; the caller then uses the mma.sync kernel.
int attn_prefill_tc5(const PrefillParams& p, int dtype, cudaStream_t stream);
// code left by a bounded wait of that kernel that ran out (0 = none); optionally cleared
int attn_prefill_tc5_error(bool clear);

}  // namespace b200

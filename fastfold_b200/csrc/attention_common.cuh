// Helpers shared by the attention kernels (attention_infer.cu, attention_tcgen05.cu).
#pragma once
#include "common.cuh"

namespace ffb {

constexpr float LOG2E = 1.4426950408889634f;

// descriptor with explicit layout code: 2 = 128B swizzle, 4 = 64B swizzle
__device__ __forceinline__ uint64_t make_desc(uint32_t saddr, uint32_t lbo_bytes, uint32_t sbo_bytes, uint32_t layout) {
  uint64_t d = 0;
  d |= static_cast<uint64_t>((saddr & 0x3FFFF) >> 4);
  d |= static_cast<uint64_t>((lbo_bytes >> 4) & 0x3FFF) << 16;
  d |= static_cast<uint64_t>((sbo_bytes >> 4) & 0x3FFF) << 32;
  d |= static_cast<uint64_t>(1) << 46;
  d |= static_cast<uint64_t>(layout) << 61;
  return d;
}

__device__ __forceinline__ float ex2f(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// two bf16 packed in a word -> two floats (low half first)
__device__ __forceinline__ float bf_lo(uint32_t w) { return __uint_as_float(w << 16); }
__device__ __forceinline__ float bf_hi(uint32_t w) { return __uint_as_float(w & 0xffff0000u); }

// Keep-bits of 64 consecutive keys starting at kbase: bit c of (lo | hi << 32) is set when key kbase + c is inside the
// sequence and its mask entry is non-zero.  `valid` gets the in-sequence bits alone.  One warp-wide call.
__device__ __forceinline__ void key_bits(const bf16* mrow, int kbase, int n_k, int lane, uint32_t& keep_lo, uint32_t& keep_hi,
                                         uint32_t& valid_lo, uint32_t& valid_hi) {
  const int k_a = kbase + lane, k_b = kbase + 32 + lane;
  const bool in_a = k_a < n_k, in_b = k_b < n_k;
  bool on_a = in_a, on_b = in_b;
  if (mrow) {
    if (in_a) on_a = __bfloat162float(mrow[k_a]) != 0.f;
    if (in_b) on_b = __bfloat162float(mrow[k_b]) != 0.f;
  }
  valid_lo = __ballot_sync(0xffffffffu, in_a);
  valid_hi = __ballot_sync(0xffffffffu, in_b);
  keep_lo = __ballot_sync(0xffffffffu, on_a);
  keep_hi = __ballot_sync(0xffffffffu, on_b);
}

// The same in two steps, for entries that are loaded ahead of their use.
struct KeyMask {
  uint16_t a, b;                  // non-zero (but for the sign): key kbase + lane, key kbase + 32 + lane counts
};
__device__ __forceinline__ KeyMask load_keys(const bf16* mrow, int kbase, int n_k, int lane) {
  KeyMask m = {0, 0};
  const uint16_t* p = reinterpret_cast<const uint16_t*>(mrow) + kbase + lane;
  if (kbase + lane < n_k) m.a = mrow ? p[0] : 1;
  if (kbase + 32 + lane < n_k) m.b = mrow ? p[32] : 1;
  return m;
}
struct alignas(8) Keys {
  uint32_t lo, hi;
};
__device__ __forceinline__ Keys key_bits(KeyMask m) {
  return Keys{__ballot_sync(0xffffffffu, m.a & 0x7fffu), __ballot_sync(0xffffffffu, m.b & 0x7fffu)};
}

// Masked keys take this logit (replaced, not added).  -2^30 instead of the reference's -1e9: its product with log2(e) is
// exact in fp32, so a fully masked row still comes out as exactly uniform weights from the fused multiply-add form
// exp2(v * log2e - m * log2e); any finite logit next to it underflows to weight 0 either way.
constexpr float MASKED_LOGIT = -1073741824.f;

}  // namespace ffb

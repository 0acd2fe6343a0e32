// Fused attention core for the Evoformer's axial attentions, forward without gradients:
//
//   O[b,i,h,:] = softmax_j( scale * <Q[b,i,h,:], K[b,j,h,:]> + bias[h,i,j]  |  key mask[b,j] ) V[b,j,h,:]
//
// in one kernel, flash style: logits never reach global memory.  The pair bias
// is shared by every batch row b (MSA row attention: all N_seq rows; triangle
// attention: all N_res rows), so a CTA works on FOUR batch rows of one (head,
// 128-query tile) at a time and all four read the same bias tile in shared memory.
//
// Per CTA (640 threads):
//   warp 0      TMA producer: per group a Q tile (2 stages) and K / V blocks of 64 keys (2 stages; swizzled, straight out
//               of the fused QKV projection output), bias tiles of 128 x 64 (4 slots, resident for up to 256 keys)
//   warps 1-2   MMA issuers, two groups each: S = Q K^T (128 x 64) and O += P V (128 x D x 64, P read from tensor memory);
//               the S product of a group's next block goes out as soon as the group has read the last one
//   warps 4-19  softmax, four groups of four warps, one batch row each, one thread per query row.  A thread streams its
//               row's 64 logits once: p = exp2(logit * log2e - M), row sum, P packed to bf16 into tensor memory.
//
// What should bound it are the exponentials, 16 per clock and SM; what does is instruction issue and the latency around a
// block.  So the loop around the exponentials is kept short: two-wide FMA / add (fma.rn.f32x2), no running maximum and no
// rescaling of the output.  The reference point M of a row only has to keep the row sum inside the exponent range, so it
// starts at 0 and is moved (exact block maximum, output and sum rescaled) only when the sum leaves [2^-60, 2^60] - a
// warp-uniform side path; bf16 and fp32 have the same exponent range, so P, the sums and the output lose no precision at
// any M in between, as long as P V has room too: a row whose sum is near 2^60 takes values up to 2^68, one near 2^-60 down
// to 2^-56.  A narrower window would give them more, but the side path nearly doubles a block's time (q 4x as large,
// n 256, B 256: 40 us with this window, 43 with 2^+-32, 69 with 2^+-24).  Rows whose logits are themselves masks (biases of
// -1e9, the lowest bf16 value, -inf) take a general step, see FAR_LOGIT.
// Four groups, because a group waits for its S product once per block and the others fill that time.
// Two issuer warps with descriptors that are only added to: with one issuer that built each descriptor where it was used,
// its instructions were the longest chain of a block and the kernel took 1.8x as long.
//   Measured (B200 at 1965 MHz, alternating with the kernel that also serves training, which keeps a running maximum and P
//   in shared memory): B 128, H 4, n 1024 with bias 451 -> 246 us, with a random mask 516 -> 267 us; B 256, H 4, n 256
//   67 -> 40 us; B 256, H 8, n 128 without bias 46 -> 21 us; B 32, H 8, n 64 8.6 -> 5.8 us.
// Masked keys get a huge negative logit (replaced, not added; -2^30 here, -1e9 in the reference's
// softmax kernels, softmax_cuda_kernel.cu:338-423,618-706 - same weights), which is weight 0 next to any ordinary
// key: there they are left out; keys beyond the sequence end get -inf.
// The forward pass of training stays on the kernel of attention_tcgen05.cu, which also leaves the row statistic for the
// backward pass: the logits' gradients are differences of nearly equal numbers (dP - rowsum(dO o O)), so rounding P at
// another reference point moves weight gradients by up to 4% of their norm, with neither kernel closer to 64 bits (0.057
// against 0.058) - and a training step is not bound there.
//
// Replaces logits matmul + fused_softmax + weights*v of the reference
// (fastfold/model/fastnn/ops.py:304-319) and its unused Triton forward-only
// attention core (kernel/triton/attention_core.py:12-121).
#include "attention_common.cuh"
#include "tmap.h"

namespace ffb {

constexpr int AF_BQ = 128;      // queries per tile
constexpr int AF_GROUPS = 4;    // batch rows in flight per CTA
constexpr int AF_BK = 64;       // keys per block
constexpr int AF_THREADS = 128 + AF_GROUPS * 128;
constexpr int AF_BSLOTS = 4;    // bias tiles in shared memory
constexpr int AF_ISSUERS = 2;   // MMA issuer warps
// tensor memory of group g: columns g * 128 + [0, 64) S, [64, 96) P (bf16 pairs), [96, 128) O
constexpr uint32_t AF_TM_P = 64, AF_TM_O = 96;

struct AttnInferArgs {
  int B, H, n_q, n_k;            // batch rows, heads, query / key lengths
  int n_qt, n_kb;                // query tiles (128), key blocks (64)
  int units;                     // H * n_qt * B (head, query tile, batch row) units
  int bias_resident;             // 1: n_kb <= AF_BSLOTS, bias tiles stay in shared memory across batch rows
  float scale, scale_log2e;      // logit scale, and times log2(e)
  const bf16* mask;              // [B][n_k] or null
  long long mask_bstride;
  bf16* out;                     // [B][n_q][H*D]
  long long out_bstride, out_rstride;
};

// Forward: per-warp table of the 64 keys of a block, 0 for a key that counts and -inf for any other.
__device__ __forceinline__ void write_penalties(float* pen, int lane, uint32_t keep_lo, uint32_t keep_hi) {
  __syncwarp();                                   // the previous block's reads of the table are done
  pen[lane] = (keep_lo >> lane) & 1u ? 0.f : -INFINITY;
  pen[lane + 32] = (keep_hi >> lane) & 1u ? 0.f : -INFINITY;
  __syncwarp();
}

struct AttnInferSmem {
  // offsets (bytes) from the 1024-aligned base
  static constexpr int Q = 0;                                          // [group][2] x [128][64 B]          64 KB
  static constexpr int KV = Q + AF_GROUPS * 2 * 8192;                  // [group][2] x (K 4 KB + V 4 KB)    64 KB
  static constexpr int BIAS = KV + AF_GROUPS * 2 * 8192;               // [slot] x [128][128 B]             64 KB
  static constexpr int KP = BIAS + AF_BSLOTS * 16384;                  // [16 warps][64] penalties            4 KB
  static constexpr int BARS = KP + AF_GROUPS * 4 * 64 * 4;
  static constexpr int TOTAL = BARS + 512 + 1024;
};

// two floats in one 64-bit register pair: the FMA pipe does both in one instruction
__device__ __forceinline__ uint64_t pk2(float lo, float hi) {
  uint64_t d;
  asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(lo), "f"(hi));
  return d;
}
__device__ __forceinline__ void up2(uint64_t v, float& lo, float& hi) { asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v)); }
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b) {
  uint64_t d;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}

// 32 logits (columns c0 .. c0+31 of the block) of one row in the log2 domain, relative to the row's reference point:
// s * scale * log2e + (bias * log2e + add), plus the penalty of keys that do not count unless all of the block's do.
template <bool PLAIN, bool BIAS>
__device__ __forceinline__ void logits32(uint64_t (&t)[16], const float (&s)[32], const uint8_t* brow, int r, int c0, const float* pen,
                                         float scale_log2e, float add) {
  const uint64_t sc = pk2(scale_log2e, scale_log2e), ad = pk2(add, add), l2e = pk2(LOG2E, LOG2E);
#pragma unroll
  for (int u = 0; u < 4; ++u) {
    uint64_t b[4];
    if (BIAS) {
      const uint4 raw = *reinterpret_cast<const uint4*>(brow + ((((c0 >> 3) + u) ^ (r & 7)) << 4));
      b[0] = fma2(pk2(bf_lo(raw.x), bf_hi(raw.x)), l2e, ad);
      b[1] = fma2(pk2(bf_lo(raw.y), bf_hi(raw.y)), l2e, ad);
      b[2] = fma2(pk2(bf_lo(raw.z), bf_hi(raw.z)), l2e, ad);
      b[3] = fma2(pk2(bf_lo(raw.w), bf_hi(raw.w)), l2e, ad);
    } else {
#pragma unroll
      for (int e = 0; e < 4; ++e) b[e] = ad;
    }
#pragma unroll
    for (int e = 0; e < 4; ++e) t[u * 4 + e] = fma2(pk2(s[u * 8 + 2 * e], s[u * 8 + 2 * e + 1]), sc, b[e]);
    if (!PLAIN) {
      const float4 k0 = *reinterpret_cast<const float4*>(pen + c0 + u * 8);         // same address in every lane: broadcast
      const float4 k1 = *reinterpret_cast<const float4*>(pen + c0 + u * 8 + 4);
      t[u * 4] = add2(t[u * 4], pk2(k0.x, k0.y));
      t[u * 4 + 1] = add2(t[u * 4 + 1], pk2(k0.z, k0.w));
      t[u * 4 + 2] = add2(t[u * 4 + 2], pk2(k1.x, k1.y));
      t[u * 4 + 3] = add2(t[u * 4 + 3], pk2(k1.z, k1.w));
    }
  }
}

// p = exp2(t) of 32 logits, packed to bf16 pairs, and the two-wide running sum of p as rounded to bf16 - that is what the
// tensor core multiplies V with, so in a row that one key dominates the rounding of its p cancels.
__device__ __forceinline__ void exp32(const uint64_t (&t)[16], uint32_t (&p)[16], uint64_t& sum) {
#pragma unroll
  for (int i = 0; i < 16; ++i) {
    float a, b;
    up2(t[i], a, b);
    a = ex2f(a);
    b = ex2f(b);
    const bf162 h = __floats2bfloat162_rn(a, b);
    p[i] = *reinterpret_cast<const uint32_t*>(&h);
    sum = add2(sum, pk2(bf_lo(p[i]), bf_hi(p[i])));
  }
}

__device__ __forceinline__ void tmem_st_32x16(uint32_t taddr, const uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%16], {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15};"
      ::"r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]),
        "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(taddr)
      : "memory");
}

// One pass over the 64 logits of a row's block: probabilities into tensor memory, their sum.
template <bool PLAIN, bool BIAS>
__device__ __forceinline__ void softmax_block(uint32_t tm_s, uint32_t tm_p, const uint8_t* brow, int r, const float* pen, float scale_log2e,
                                              float add, uint64_t& sum) {
#pragma unroll 1
  for (int c = 0; c < 2; ++c) {
    float s[32];
    uint64_t t[16];
    uint32_t p[16];
    tmem_ld_32x32(tm_s + c * 32, s);
    tmem_ld_wait();
    logits32<PLAIN, BIAS>(t, s, brow, r, c * 32, pen, scale_log2e, add);
    exp32(t, p, sum);
    tmem_st_32x16(tm_p + c * 16, p);
  }
}

// D[tmem] (+)= A[tmem] * B[smem]: bf16 A, two elements per column
__device__ __forceinline__ void umma_bf16_ts(uint32_t d_tmem, uint32_t a_tmem, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
      ::"r"(d_tmem), "r"(a_tmem), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}

constexpr float ROW_SUM_LO = 8.673617379884035e-19f, ROW_SUM_HI = 1.152921504606847e18f;   // 2^-60, 2^60

// Rows whose largest logit is this far out (log2 domain) are `far` rows.  There the two formulas of the ordinary path end:
// masked keys no longer have weight 0 next to such a row's keys (a pair bias of -1e9, of the type's lowest value or -inf is
// itself a mask), the log2 domain overflows for the lowest and largest bf16 values, and one ulp of a reference point is no
// longer small against 1.  A far row's reference point is its running maximum in natural units, masked keys take part in it
// with MASKED_LOGIT, and its logits are rounded as the kernel with gradients rounds them.
constexpr float FAR_LOGIT = 1048576.f;

struct RowState {
  float M, l;                     // reference point (log2 domain; natural units in a far row), row sum relative to it
  int far;                        // int: as a bool it takes a predicate and the ordinary path a spilled register more
};

__device__ __forceinline__ void tmem_ld_32x8(uint32_t taddr, float (&v)[8]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]), "=f"(v[7])
               : "r"(taddr));
}

__device__ __forceinline__ void tmem_st_32x8(uint32_t taddr, const float (&v)[8]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%8], {%0, %1, %2, %3, %4, %5, %6, %7};"
               ::"f"(v[0]), "f"(v[1]), "f"(v[2]), "f"(v[3]), "f"(v[4]), "f"(v[5]), "f"(v[6]), "f"(v[7]), "r"(taddr)
               : "memory");
}

__device__ __forceinline__ void tmem_st_32x4(uint32_t taddr, const uint32_t (&v)[4]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%4], {%0, %1, %2, %3};" ::"r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(taddr) : "memory");
}

// A block of keys for a warp that holds a far row: the general softmax step.  Rows with `move` get a new reference point (the
// output and the sum so far are rescaled to it), the others keep theirs.  Eight columns at a time and inlined: no row of a
// model's own biases gets here, but the ordinary path uses all registers that five warps per scheduler leave, and a call or
// wider pieces cost it 2 - 8 % (n 389, B 389, H 4 with bias: 192 us without this path, 193 us as it is, 205 us as a call).
template <bool BIAS>
__device__ __forceinline__ RowState far_block(RowState st, bool move, uint32_t tm, bool has_o, const uint8_t* brow, int r, uint32_t keep_lo,
                                           uint32_t keep_hi, int keys, float scale, float scale_log2e) {
  constexpr float LN2 = 0.6931471805599453f;
  const uint64_t keep = keep_lo | (uint64_t)keep_hi << 32;        // `keys` of the 64 are in the sequence
  auto load = [&](int c, float (&s)[8], float (&b)[8]) {
    tmem_ld_32x8(tm + c * 8, s);
    tmem_ld_wait();
    if (BIAS) {
      const uint4 raw = *reinterpret_cast<const uint4*>(brow + ((c ^ (r & 7)) << 4));
      b[0] = bf_lo(raw.x), b[1] = bf_hi(raw.x), b[2] = bf_lo(raw.y), b[3] = bf_hi(raw.y);
      b[4] = bf_lo(raw.z), b[5] = bf_hi(raw.z), b[6] = bf_lo(raw.w), b[7] = bf_hi(raw.w);
    } else {
#pragma unroll
      for (int e = 0; e < 8; ++e) b[e] = 0.f;
    }
  };
  auto logit = [&](int key, float s, float b) -> float {          // natural units
    return (keep >> key) & 1u ? fmaf(s, scale, b) : (key < keys ? MASKED_LOGIT : -INFINITY);
  };
  tmem_st_wait();                          // what the ordinary path stored for this block is about to be replaced
  float mx = -INFINITY, alpha = 1.f;
#pragma unroll 1
  for (int c = 0; c < 8; ++c) {
    float s[8], b[8];
    load(c, s, b);
#pragma unroll
    for (int e = 0; e < 8; ++e) mx = fmaxf(mx, logit(c * 8 + e, s[e], b[e]));
  }
  if (move) {
    const float top = st.l > 0.f ? fmaxf(mx, st.far ? st.M : (st.M + log2f(st.l)) * LN2) : mx;
    if (top != -INFINITY) {                // a row without any key yet keeps its reference point
      const bool far = !(fabsf(top * LOG2E) < FAR_LOGIT);
      const float m2 = far ? top : top * LOG2E;
      if (st.l > 0.f) alpha = ex2f(far ? ((st.far ? st.M : st.M * LN2) - top) * LOG2E : (st.far ? st.M * LOG2E : st.M) - m2);
      st.M = m2;
      st.far = far;
    }
  }
  if (has_o) {
#pragma unroll 1
    for (int c = 0; c < 4; ++c) {          // heads of 16 channels: the upper columns are nobody's
      float o[8];
      tmem_ld_32x8(tm + AF_TM_O + c * 8, o);
      tmem_ld_wait();
#pragma unroll
      for (int e = 0; e < 8; ++e) o[e] *= alpha;
      tmem_st_32x8(tm + AF_TM_O + c * 8, o);
    }
  }
  float sum = 0.f;
#pragma unroll 1
  for (int c = 0; c < 8; ++c) {
    float s[8], b[8];
    uint32_t p[4];
    load(c, s, b);
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      if (st.far) s[e] = ex2f((logit(c * 8 + e, s[e], b[e]) - st.M) * LOG2E);
      else s[e] = (keep >> (c * 8 + e)) & 1u ? ex2f(fmaf(s[e], scale_log2e, fmaf(b[e], LOG2E, -st.M))) : 0.f;
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const bf162 h = __floats2bfloat162_rn(s[2 * i], s[2 * i + 1]);
      p[i] = *reinterpret_cast<const uint32_t*>(&h);
      sum += bf_lo(p[i]) + bf_hi(p[i]);
    }
    tmem_st_32x4(tm + AF_TM_P + c * 4, p);
  }
  st.l = st.l * alpha + sum;
  return st;
}

template <int D, bool BIAS>   // head dim: 32 (64-byte rows, 64-byte swizzle) or 16 (32-byte)
__global__ void __launch_bounds__(AF_THREADS, 1) attn_infer_kernel(const __grid_constant__ CUtensorMap tmQ,
                                                                 const __grid_constant__ CUtensorMap tmK,
                                                                 const __grid_constant__ CUtensorMap tmV,
                                                                 const __grid_constant__ CUtensorMap tmBias, const AttnInferArgs a) {
  pdl_launch_dependents();
  static_assert(D == 32 || D == 16, "head dim");
  constexpr uint32_t Q_BYTES = AF_BQ * D * 2, KV_BYTES = AF_BK * D * 2;       // one Q tile, one K or V block
  constexpr uint32_t LAYOUT = D == 32 ? 4 : 6, GROUP = 8 * D * 2;             // descriptor layout code, bytes of 8 rows
  extern __shared__ uint8_t smem_raw[];
  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* sm = smem_raw + (base - smem_u32(smem_raw));
  const uint32_t b0 = base + AttnInferSmem::BARS;
  // barrier map (8 bytes each): [group][2 stages] for Q and K / V, [slot] for the bias, [group] for the rest
  const uint32_t q_full = b0, q_empty = b0 + 64, kv_full = b0 + 128, kv_empty = b0 + 192;
  const uint32_t bias_full = b0 + 256, bias_empty = b0 + 288, s_full = b0 + 320, p_full = b0 + 352, o_done = b0 + 384;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(sm + AttnInferSmem::BARS + 448);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    for (int i = 0; i < 2 * AF_GROUPS; ++i) {
      mbar_init(q_full + 8 * i, 1);
      mbar_init(q_empty + 8 * i, 1);
      mbar_init(kv_full + 8 * i, 1);
      mbar_init(kv_empty + 8 * i, 1);
    }
    for (int i = 0; i < AF_BSLOTS; ++i) {
      mbar_init(bias_full + 8 * i, 1);
      mbar_init(bias_empty + 8 * i, AF_GROUPS * 4);
    }
    for (int i = 0; i < AF_GROUPS; ++i) {
      mbar_init(s_full + 8 * i, 1);
      mbar_init(p_full + 8 * i, 4);
      mbar_init(o_done + 8 * i, 1);
    }
    *abort_flag = 0;
    fence_mbar_init();
    prefetch_tmap(&tmQ);
    prefetch_tmap(&tmK);
    prefetch_tmap(&tmV);
    if (BIAS) prefetch_tmap(&tmBias);
  }
  if (warp == 0) {
    __syncwarp();
    tmem_alloc(smem_u32(tmem_slot), 512);
    tmem_relinquish();
  }
  pdl_wait();          // the prologue above touched no global memory; everything below may
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;

  // Contiguous range of units for this CTA; unit = (h * n_qt + qt) * B + b.  A round takes up to AF_GROUPS consecutive
  // batch rows of one (head, query tile); every role walks the same rounds.
  const int per = (a.units + gridDim.x - 1) / gridDim.x;
  const int u_begin = blockIdx.x * per;
  int u_end = u_begin + per;
  if (u_end > a.units) u_end = a.units;
  auto round_count = [&](int u) -> int {        // batch rows in the round that starts at unit u (0 past the end)
    if (u >= u_end) return 0;
    int c = a.B - u % a.B;
    if (c > u_end - u) c = u_end - u;
    return c < AF_GROUPS ? c : AF_GROUPS;
  };

  if (warp == 0) {
    if (lane == 0) {
      // ---------------- TMA producer ----------------
      uint32_t qi[AF_GROUPS], jt[AF_GROUPS];     // items and key blocks loaded per group
#pragma unroll
      for (int g = 0; g < AF_GROUPS; ++g) qi[g] = jt[g] = 0;
      uint32_t fill = 0;                         // bias: streamed tiles so far, or resident (head, tile) sets so far
      int prev = -1;
      bool ok = true;
      for (int u = u_begin; u < u_end && ok;) {
        const int cnt = round_count(u);
        const int grp = u / a.B, bb = u % a.B;
        const int qt = grp % a.n_qt, h = grp / a.n_qt;
        const bool load_bias = BIAS && (!a.bias_resident || grp != prev);
        const uint32_t set = fill;               // resident: index of the set loaded in this round
        if (load_bias && a.bias_resident) ++fill;
        prev = grp;
        for (int j = 0; j < a.n_kb && ok; ++j) {
          if (load_bias) {
            const uint32_t slot = a.bias_resident ? (uint32_t)j : fill % AF_BSLOTS;
            const uint32_t nth = a.bias_resident ? set : fill / AF_BSLOTS;       // fill index of this slot
            if (!mbar_wait(bias_empty + 8 * slot, (nth & 1) ^ 1)) { report(ST_TIMEOUT_EPI, 11); ok = false; break; }
            mbar_expect_tx(bias_full + 8 * slot, 16384);
            tma_load_3d(base + AttnInferSmem::BIAS + slot * 16384, &tmBias, bias_full + 8 * slot, j * AF_BK, qt * AF_BQ, h);
            if (!a.bias_resident) ++fill;
          }
#pragma unroll
          for (int g = 0; g < AF_GROUPS; ++g) {
            if (g >= cnt || !ok) continue;
            if (j == 0) {
              const uint32_t qs = g * 2 + (qi[g] & 1);
              if (!mbar_wait(q_empty + 8 * qs, ((qi[g] >> 1) & 1) ^ 1)) { report(ST_TIMEOUT_MMA, 10); ok = false; continue; }
              mbar_expect_tx(q_full + 8 * qs, Q_BYTES);
              tma_load_3d(base + AttnInferSmem::Q + qs * 8192, &tmQ, q_full + 8 * qs, h * D, qt * AF_BQ, bb + g);
              ++qi[g];
            }
            const uint32_t ks = g * 2 + (jt[g] & 1);
            if (!mbar_wait(kv_empty + 8 * ks, ((jt[g] >> 1) & 1) ^ 1)) { report(ST_TIMEOUT_MMA, 12); ok = false; continue; }
            mbar_expect_tx(kv_full + 8 * ks, 2 * KV_BYTES);
            tma_load_3d(base + AttnInferSmem::KV + ks * 8192, &tmK, kv_full + 8 * ks, h * D, j * AF_BK, bb + g);
            tma_load_3d(base + AttnInferSmem::KV + ks * 8192 + 4096, &tmV, kv_full + 8 * ks, h * D, j * AF_BK, bb + g);
            ++jt[g];
          }
        }
        u += cnt;
      }
      if (!ok) *abort_flag = 1;
    }
    __syncwarp();
  } else if (warp <= AF_ISSUERS) {
    if (lane == 0) {
      // ---------------- MMA issuers: GPI groups each ----------------
      constexpr uint32_t idesc_s = make_idesc_bf16(128, AF_BK, 0, 0);     // Q (K-major) x K (K-major)
      constexpr uint32_t idesc_o = make_idesc_bf16(128, D, 0, 1);         // P (tensor memory) x V (MN-major)
      constexpr int GPI = AF_GROUPS / AF_ISSUERS;
      const int gb = (warp - 1) * GPI;
      // descriptors of stage 0 of group gb; the address field counts 16 bytes, so stages and groups are additions
      const uint64_t dq = make_desc(base + AttnInferSmem::Q + gb * 16384, 16, GROUP, LAYOUT), dk = make_desc(base + AttnInferSmem::KV + gb * 16384, 16, GROUP, LAYOUT),
                     dv = make_desc(base + AttnInferSmem::KV + gb * 16384 + 4096, 16, GROUP, LAYOUT);
      uint32_t si[GPI], qi[GPI], pi[GPI];                                 // per group: S products, items, PV products issued
      bool ahead[GPI];                                                    // S of the group's next block already issued
#pragma unroll
      for (int e = 0; e < GPI; ++e) {
        si[e] = qi[e] = pi[e] = 0;
        ahead[e] = false;
      }
      bool ok = true;
      // S product of a group's next block; `first` / `last`: position of that block in its item
      auto issue_s = [&](int e, uint32_t& sg, uint32_t& qg, bool first, bool last) -> bool {
        const uint32_t qs = (gb + e) * 2 + (qg & 1), ks = (gb + e) * 2 + (sg & 1);
        if (first && !mbar_wait(q_full + 8 * qs, (qg >> 1) & 1)) { report(ST_TIMEOUT_TMA, 22); return false; }
        if (!mbar_wait(kv_full + 8 * ks, (sg >> 1) & 1)) { report(ST_TIMEOUT_TMA, 20); return false; }
        tc_fence_after();
        const uint64_t q = dq + (e * 2 + (qg & 1)) * (8192 >> 4), k = dk + (e * 2 + (sg & 1)) * (8192 >> 4);
#pragma unroll
        for (int i = 0; i < D / 16; ++i) umma_bf16(tmem + (gb + e) * 128, q + i * (32 >> 4), k + i * (32 >> 4), idesc_s, i > 0 ? 1u : 0u);
        umma_commit(s_full + 8 * (gb + e));
        ++sg;
        if (last) {
          umma_commit(q_empty + 8 * qs);        // all S products of this item issued: the Q slot drains with them
          ++qg;
        }
        return true;
      };
      for (int u = u_begin; u < u_end && ok;) {
        const int cnt = round_count(u);
        const int cnt_next = round_count(u + cnt);
#pragma unroll
        for (int e = 0; e < GPI; ++e) {
          if (gb + e < cnt && !ahead[e] && ok) ok = issue_s(e, si[e], qi[e], true, a.n_kb == 1);
          ahead[e] = false;
        }
        for (int j = 0; j < a.n_kb && ok; ++j) {
          const bool last = j + 1 == a.n_kb;
#pragma unroll
          for (int e = 0; e < GPI; ++e) {
            if (gb + e >= cnt || !ok) continue;
            const int g = gb + e;
            // the group has read S of block j and written P
            if (!mbar_wait(p_full + 8 * g, pi[e] & 1)) { if (*abort_flag == 0) report(ST_TIMEOUT_EPI, 23); ok = false; continue; }
            tc_fence_after();
            const uint32_t st = pi[e] & 1;
            if (!last) {
              ok = issue_s(e, si[e], qi[e], false, j + 2 == a.n_kb);
            } else if (g < cnt_next) {
              ok = issue_s(e, si[e], qi[e], true, a.n_kb == 1);
              ahead[e] = true;
            }
            if (!ok) continue;
            const uint64_t v = dv + (e * 2 + st) * (8192 >> 4);
#pragma unroll
            for (int k = 0; k < AF_BK / 16; ++k)
              umma_bf16_ts(tmem + g * 128 + AF_TM_O, tmem + g * 128 + AF_TM_P + k * 8, v + ((k * 2 * GROUP) >> 4), idesc_o, (j > 0 || k > 0) ? 1u : 0u);
            umma_commit(o_done + 8 * g);
            umma_commit(kv_empty + 8 * (g * 2 + st));
            ++pi[e];
          }
        }
        u += cnt;
      }
      if (!ok) *abort_flag = 1;
    }
    __syncwarp();
  } else if (warp >= 4) {
    // ---------------- softmax / output (warps 4..19): group = batch row of the round, thread = query row ----------------
    const int quad = warp & 3;                      // TMEM lane quadrant this warp may read
    const int g = (warp - 4) >> 2;
    const int r = quad * 32 + lane;                 // row within the query tile
    const uint32_t tm = tmem + ((uint32_t)(quad * 32) << 16) + (uint32_t)g * 128;
    float* pen = reinterpret_cast<float*>(sm + AttnInferSmem::KP) + (warp - 4) * 64;
    uint32_t jt = 0;                                // blocks of this group so far
    uint32_t fill = 0;                              // bias tiles (streamed) or sets (resident) this warp has waited for
    int prev = -1;
    bool ok = true;
    for (int u = u_begin; u < u_end && ok;) {
      const int cnt = round_count(u);
      const int grp = u / a.B, b = u % a.B + g;
      const int qt = grp % a.n_qt, h = grp / a.n_qt;
      const bool active = g < cnt;
      u += cnt;
      const bool new_set = BIAS && grp != prev;
      if (new_set && a.bias_resident) ++fill;
      prev = grp;
      // resident tiles are released in the last round that reads them, streamed ones at once
      const bool release = BIAS && (!a.bias_resident || u >= u_end || u / a.B != grp);
      RowState row = {0.f, 0.f, false};
      const bf16* mrow = (a.mask && active) ? a.mask + (long long)b * a.mask_bstride : nullptr;
      for (int j = 0; j < a.n_kb; ++j) {
        uint32_t slot = 0, bpar = 0;
        if (BIAS) {
          slot = a.bias_resident ? (uint32_t)j : fill % AF_BSLOTS;
          bpar = a.bias_resident ? (fill - 1) & 1 : (fill / AF_BSLOTS) & 1;
          if (!a.bias_resident) ++fill;
        }
        if (!active) {                              // keeps the tile accounting: one release per warp and fill
          if (release) {
            bool w = mbar_wait(bias_full + 8 * slot, bpar);
            ok = __all_sync(0xffffffffu, w);
            if (!ok) break;
            if (lane == 0) mbar_arrive(bias_empty + 8 * slot);
          }
          continue;
        }
        // key bits first: their global loads overlap the wait for S
        uint32_t keep_lo, keep_hi, valid_lo, valid_hi;
        key_bits(mrow, j * AF_BK, a.n_k, lane, keep_lo, keep_hi, valid_lo, valid_hi);
        const bool plain = (keep_lo & keep_hi) == 0xffffffffu;         // every key of this block in range and unmasked
        const bool none = (keep_lo | keep_hi) == 0u;                   // no key of this block counts
        if (!plain && !none) write_penalties(pen, lane, keep_lo, keep_hi);
        bool w = true;
        if (BIAS && !mbar_wait(bias_full + 8 * slot, bpar)) { if (lane == 0 && *abort_flag == 0) report(ST_TIMEOUT_TMA, 30); w = false; }
        if (w && !mbar_wait(s_full + 8 * g, jt & 1)) { if (lane == 0 && *abort_flag == 0) report(ST_TIMEOUT_MMA, 31); w = false; }
        ok = __all_sync(0xffffffffu, w);
        if (!ok) break;
        tc_fence_after();
        const uint8_t* brow = BIAS ? sm + AttnInferSmem::BIAS + slot * 16384 + r * 128 : nullptr;
        // P of the previous block has been read and O holds its product
        if (j > 0) {
          w = mbar_wait(o_done + 8 * g, (jt - 1) & 1);
          if (!w && lane == 0 && *abort_flag == 0) report(ST_TIMEOUT_MMA, 32);
          ok = __all_sync(0xffffffffu, w);
          if (!ok) break;
          tc_fence_after();
        }
        uint64_t sum = pk2(0.f, 0.f);
        if (none) {
          // masked keys next to a real one have weight 0; where there has been no other key they all have the same logit
          const bool alone = row.l == 0.f || (row.far && row.M == MASKED_LOGIT);
          if (__any_sync(0xffffffffu, row.far && !alone)) {
            row = far_block<BIAS>(row, alone || row.far, tm, j > 0, brow, r, 0u, 0u, a.n_k - j * AF_BK, a.scale, a.scale_log2e);
          } else {
            if (alone) {
              row.M = MASKED_LOGIT;
              row.far = 1;
              row.l += (float)(__popc(valid_lo) + __popc(valid_hi));
            }
#pragma unroll
            for (int c = 0; c < 2; ++c) {
              uint32_t p[16];
#pragma unroll
              for (int i = 0; i < 16; ++i) {
                const uint32_t bits = ((c ? valid_hi : valid_lo) >> (2 * i)) & 3u;
                p[i] = alone ? (bits & 1u) * 0x3f80u + (bits >> 1) * 0x3f800000u : 0u;
              }
              tmem_st_32x16(tm + AF_TM_P + c * 16, p);
            }
          }
        } else {
          if (plain) softmax_block<true, BIAS>(tm, tm + AF_TM_P, brow, r, pen, a.scale_log2e, -row.M, sum);
          else softmax_block<false, BIAS>(tm, tm + AF_TM_P, brow, r, pen, a.scale_log2e, -row.M, sum);
          float sx, sy;
          up2(sum, sx, sy);
          float ln = row.l + (sx + sy);
          const bool bad = row.far || !(ln > ROW_SUM_LO && ln < ROW_SUM_HI);
          if (__any_sync(0xffffffffu, bad)) {
            // some row's sum has left the safe range (first block of a row with large logits, only masked keys before this
            // block, or a much larger logit in it): move that row's reference point and redo the block
            if (plain) write_penalties(pen, lane, 0xffffffffu, 0xffffffffu);
            float mx = -INFINITY, alpha = 1.f;
            tmem_st_wait();                         // the first attempt's P is about to be replaced
#pragma unroll 1
            for (int c = 0; c < 2; ++c) {
              float s[32];
              uint64_t t[16];
              tmem_ld_32x32(tm + c * 32, s);
              tmem_ld_wait();
              logits32<false, BIAS>(t, s, brow, r, c * 32, pen, a.scale_log2e, 0.f);
#pragma unroll
              for (int i = 0; i < 16; ++i) {
                float x, y;
                up2(t[i], x, y);
                mx = fmaxf(mx, fmaxf(x, y));
              }
            }
            const float m2 = (row.l > 0.f && !row.far) ? fmaxf(mx, row.M + log2f(row.l)) : mx;
            // a row that leaves the domain of the ordinary path, or that has not re-entered it from above
            const bool out = bad && (!(fabsf(m2) < FAR_LOGIT) || (row.far && row.M > 0.f));
            if (__any_sync(0xffffffffu, out)) {
              // the keys from the table: bits kept until here would be spilled
              row = far_block<BIAS>(row, bad, tm, j > 0, brow, r, __ballot_sync(0xffffffffu, pen[lane] == 0.f),
                                    __ballot_sync(0xffffffffu, pen[lane + 32] == 0.f), a.n_k - j * AF_BK, a.scale, a.scale_log2e);
            } else {
              if (bad) {
                if (row.l > 0.f) alpha = ex2f((row.far ? row.M * LOG2E : row.M) - m2);
                row.M = m2;
                row.far = 0;
              }
              if (j > 0) {
                float o[32];                        // D = 16: the upper columns are nobody's
                tmem_ld_32x32(tm + AF_TM_O, o);
                tmem_ld_wait();
#pragma unroll
                for (int c = 0; c < 32; ++c) o[c] *= alpha;
                tmem_st_32x32(tm + AF_TM_O, o);
              }
              sum = pk2(0.f, 0.f);
              softmax_block<false, BIAS>(tm, tm + AF_TM_P, brow, r, pen, a.scale_log2e, -row.M, sum);
              up2(sum, sx, sy);
              row.l = row.l * alpha + (sx + sy);
            }
          } else {
            row.l = ln;
          }
        }
        tmem_st_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) {
          mbar_arrive(p_full + 8 * g);              // S may be overwritten, P is complete
          if (release) mbar_arrive(bias_empty + 8 * slot);
        }
        ++jt;
      }
      if (!ok || !active) continue;
      // ---- the item's output row ----
      {
        bool w = mbar_wait(o_done + 8 * g, (jt - 1) & 1);
        if (!w && lane == 0 && *abort_flag == 0) report(ST_TIMEOUT_MMA, 33);
        ok = __all_sync(0xffffffffu, w);
        if (!ok) break;
      }
      tc_fence_after();
      float o[32];
      tmem_ld_32x32(tm + AF_TM_O, o);
      tmem_ld_wait();
      const int qrow = qt * AF_BQ + r;
      if (qrow < a.n_q) {
        const float inv = 1.f / row.l;
        bf16* dst = a.out + (long long)b * a.out_bstride + (long long)qrow * a.out_rstride + h * D;
#pragma unroll
        for (int c = 0; c < D; c += 8) {
          uint4 pk;
          bf162* hp = reinterpret_cast<bf162*>(&pk);
#pragma unroll
          for (int e = 0; e < 4; ++e) hp[e] = __floats2bfloat162_rn(o[c + 2 * e] * inv, o[c + 2 * e + 1] * inv);
          *reinterpret_cast<uint4*>(dst + c) = pk;
        }
      }
      tc_fence_before();
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 0) {
    tc_fence_after();
    tmem_dealloc(tmem, 512);
  }
}

}  // namespace ffb

using namespace ffb;

extern "C" {

// q, k, v: bf16, element (b, i, h, c) at ptr[b * bstride + i * rstride + h * D + c]; D = 32 or 16.
// bias: bf16, element (h, i, j) at bias[(h * n_q + i) * bias_rstride + j], or null; mask: bf16 [B][n_k] or null (0 = masked key).
// out: bf16 (b, i, h, c) at out[b * out_bstride + i * out_rstride + h * D + c].
// n_q and n_k are free; TMA wants 16-byte strides, so bias rows are padded to a multiple of 8 where n_k is not one.
int ffb_attention_infer(const void* q, const void* k, const void* v, long long q_bstride, long long q_rstride, long long kv_bstride,
                      long long kv_rstride, const void* bias, long long bias_rstride, const void* mask, long long mask_bstride, void* out,
                      long long out_bstride, long long out_rstride, int B, int H, int n_q, int n_k, int D, float scale,
                      void* stream) {
  if (D != 32 && D != 16) return -2;
  if ((q_rstride % 8) || (kv_rstride % 8) || (q_bstride % 8) || (kv_bstride % 8) || (out_rstride % 8) || (out_bstride % 8)) return -3;
  if (bias && (bias_rstride % 8 || bias_rstride < n_k)) return -4;
  AttnInferArgs a;
  a.B = B; a.H = H; a.n_q = n_q; a.n_k = n_k;
  a.n_qt = (n_q + AF_BQ - 1) / AF_BQ;
  a.n_kb = (n_k + AF_BK - 1) / AF_BK;
  const long long units = (long long)H * a.n_qt * B;
  if (units <= 0 || units > 0x7fffffffLL || a.n_kb <= 0) return -6;
  a.units = (int)units;
  a.bias_resident = (bias && a.n_kb <= AF_BSLOTS) ? 1 : 0;
  a.scale = scale;
  a.scale_log2e = scale * LOG2E;
  a.mask = (const bf16*)mask;
  a.mask_bstride = mask_bstride;
  a.out = (bf16*)out;
  a.out_bstride = out_bstride;
  a.out_rstride = out_rstride;
  CUtensorMap tq, tk, tv, tb;
  // the q/k/v views are addressed as [B][n][H*D] slabs of a possibly wider row (fused qkv projection output)
  if (encode_tmap3_bf16(&tq, q, (long long)H * D, n_q, B, q_rstride, q_bstride, D, AF_BQ, 2 * D)) return -10;
  if (encode_tmap3_bf16(&tk, k, (long long)H * D, n_k, B, kv_rstride, kv_bstride, D, AF_BK, 2 * D)) return -11;
  if (encode_tmap3_bf16(&tv, v, (long long)H * D, n_k, B, kv_rstride, kv_bstride, D, AF_BK, 2 * D)) return -12;
  if (bias) {
    if (encode_tmap3_bf16(&tb, bias, n_k, n_q, H, bias_rstride, (long long)n_q * bias_rstride, AF_BK, AF_BQ, 128)) return -13;
  } else {
    tb = tq;
  }
  auto kern = D == 32 ? (bias ? attn_infer_kernel<32, true> : attn_infer_kernel<32, false>)
                      : (bias ? attn_infer_kernel<16, true> : attn_infer_kernel<16, false>);
  static SmemLimit limit[4];
  if (!limit[(D == 32 ? 0 : 2) + (bias ? 1 : 0)].raise(kern, AttnInferSmem::TOTAL)) return -14;
  static int sm_count = 0;
  if (!sm_count) {
    int dev = 0;
    cudaGetDevice(&dev);
    if (cudaDeviceGetAttribute(&sm_count, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sm_count <= 0) sm_count = 148;
  }
  const int grid = units < sm_count ? (int)units : sm_count;
  launch_k(kern, grid, AF_THREADS, AttnInferSmem::TOTAL,
           reinterpret_cast<cudaStream_t>(stream), tq, tk, tv, tb, a);
  return cudaGetLastError() == cudaSuccess ? 0 : -15;
}

}  // extern "C"

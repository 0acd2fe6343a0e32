// Fused attention core for the Evoformer's axial attentions, forward without gradients:
//
//   O[b,i,h,:] = softmax_j( scale * <Q[b,i,h,:], K[b,j,h,:]> + bias[h,i,j]  |  key mask[b,j] ) V[b,j,h,:]
//
// in one kernel, flash style: logits never reach global memory.  The pair bias
// is shared by every batch row b (MSA row attention: all N_seq rows; triangle
// attention: all N_res rows), so a CTA works on THREE batch rows of one (head,
// 128-query tile) at a time and all three read the same bias tile in shared memory.
//
// Per CTA (512 threads):
//   warp 0      TMA producer: per group a Q tile (2 stages) and K / V blocks of 64 keys (4 stages; swizzled, straight out
//               of the fused QKV projection output), bias tiles of 128 x 64 (4 slots, resident for up to 256 keys)
//   warps 1-3   MMA issuer of a group each: S = Q K^T (128 x 64, two blocks ahead, into two buffers) and O += P V (128 x D x 64,
//               P read from tensor memory); these warps also work out which keys of a block count and release the bias tiles
//   warps 4-15  softmax, three groups of four warps, one batch row each, one thread per query row.  A thread streams its
//               row's 64 logits once: p = exp2(logit * log2e - M), row sum, P packed to bf16 into tensor memory.
//
// What should bound it are the exponentials, 16 per clock and SM: 512 cycles a block of 128 x 64.  The arithmetic around them
// (unpacking the bias, packing P, the sum) brings three softmax warps on a scheduler to 640; the rest is what happens between two
// blocks.  So everything that another warp can do is done there, the loop around the exponentials is kept short: two-wide
// FMA (fma.rn.f32x2), sums of bf16 without unpacking (add.f32.bf16), no running maximum and no rescaling of the output; and the
// warps of a scheduler are kept out of step (take_turn).  The reference point M of a row only has to keep the row sum inside the
// exponent range, so it starts at 0 and is moved (exact block maximum, output and sum rescaled) only when the sum leaves
// [2^-60, 2^60] - a warp-uniform side path; bf16 and fp32 have the same exponent range, so P, the sums and the output lose no precision at
// any M in between, as long as P V has room too: a row whose sum is near 2^60 takes values up to 2^68, one near 2^-60 down
// to 2^-56.  A narrower window would give them more, but the side path nearly doubles a block's time (q 4x as large,
// n 256, B 256: 40 us with this window, 43 with 2^+-32, 69 with 2^+-24).  Rows whose logits are themselves masks (biases of
// -1e9, the lowest bf16 value, -inf) take a general step, see FAR_LOGIT.
// Three groups with two S buffers each (480 of the 512 columns; P takes the place of the S it was made from), not four with one:
// a group never waits for its S product.  With four of them the products' latency, 1500 - 1900 cycles of 4400 a block, was
// bare, since all four were in step.
//   Measured (B200, graph replay, us; four groups with one S buffer -> this): B 384, H 4, n 1536 with bias and mask 1685 -> 1397;
//   B 64, H 4, n 1024 132 -> 113; B 389, H 4, n 389 192 -> 142; B 256, H 4, n 256 41.6 -> 36.2; B 1024, H 8, D 16, n 256 310 -> 214;
//   B 300, H 2, n 700 without bias 139 -> 119; B 256, H 8, n 128 without bias 23.2 -> 21.7; B 32, H 8, n 64 5.7 -> 5.0.  Random masks:
//   1854 -> 1595, 147 -> 136, 205 -> 157, 45.3 -> 41.6, 328 -> 256, 148 -> 132, 24.5 -> 23.9, 6.0 -> 5.3.  The wait between a P V product
//   and the S product over its P (issue_s) is in these times; it costs 1 - 2 %.
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
constexpr int AF_GROUPS = 3;    // batch rows in flight per CTA
constexpr int AF_BK = 64;       // keys per block
constexpr int AF_THREADS = 128 + AF_GROUPS * 128;
constexpr int AF_BSLOTS = 4;    // bias tiles in shared memory
constexpr int AF_KVST = 4;      // K / V stages per group
constexpr int AF_COST = 16;     // cost of a round of a full query tile
// tensor memory of group g: columns g * 160 + [0, 64) and [64, 128) two S buffers, each with its P (bf16 pairs) over the first 32
// columns once it has been read, [128, 160) O
constexpr uint32_t AF_TM_GROUP = 160, AF_TM_O = 128;

struct AttnInferArgs {
  int B, H, n_q, n_k;            // batch rows, heads, query / key lengths
  int n_qt, n_kb;                // query tiles (128), key blocks (64)
  int rounds, few, rest;         // rounds of a (head, query tile): `few` batch rows each, one more in the first `rest`
  int cost_last;                 // cost of a round of the last query tile, where others cost AF_COST
  long long share;               // cost of a CTA's rounds; the first `extra` CTAs take one more
  int extra;
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
  static constexpr int Q = 0;                                          // [group][2] x [128][64 B]          48 KB
  static constexpr int KV = Q + AF_GROUPS * 2 * 8192;                  // [group][stage] x (K 4 KB + V 4 KB) 96 KB
  static constexpr int BIAS = KV + AF_GROUPS * AF_KVST * 8192;         // [slot] x [128][128 B]             64 KB
  static constexpr int KP = BIAS + AF_BSLOTS * 16384;                  // [12 warps][64] penalties            3 KB
  static constexpr int KEYS = KP + AF_GROUPS * 4 * 64 * 4;             // [group][2] key bits of the blocks in the S buffers
  static constexpr int TURN = KEYS + 48;                               // [scheduler] whose turn it is
  static constexpr int BARS = TURN + 16;
  static constexpr int TOTAL = BARS + 576 + 1024;
};

// a + the lower / upper bf16 of w
__device__ __forceinline__ float add_lo(float a, uint32_t w) {
  float d;
  asm("{\n\t.reg .b16 l, h;\n\tmov.b32 {l, h}, %2;\n\tadd.rn.f32.bf16 %0, l, %1;\n\t}" : "=f"(d) : "f"(a), "r"(w));
  return d;
}
__device__ __forceinline__ float add_hi(float a, uint32_t w) {
  float d;
  asm("{\n\t.reg .b16 l, h;\n\tmov.b32 {l, h}, %2;\n\tadd.rn.f32.bf16 %0, h, %1;\n\t}" : "=f"(d) : "f"(a), "r"(w));
  return d;
}

// 16 logits (columns c0 .. c0+15 of the block) of one row in the log2 domain, relative to the row's reference point:
// s * scale * log2e + (bias * log2e + add), plus the penalty of keys that do not count unless all of the block's do.
template <bool PLAIN, bool BIAS>
__device__ __forceinline__ void logits16(uint64_t (&t)[8], const float (&s)[16], const uint8_t* brow, int r, int c0, const float* pen,
                                         float scale_log2e, float add) {
  const uint64_t sc = pair2(scale_log2e, scale_log2e), ad = pair2(add, add), l2e = pair2(LOG2E, LOG2E);
#pragma unroll
  for (int u = 0; u < 2; ++u) {
    uint64_t b[4];
    if (BIAS) {
      const uint4 raw = *reinterpret_cast<const uint4*>(brow + ((((c0 >> 3) + u) ^ (r & 7)) << 4));
      b[0] = fma2(pair2(bf_lo(raw.x), bf_hi(raw.x)), l2e, ad);
      b[1] = fma2(pair2(bf_lo(raw.y), bf_hi(raw.y)), l2e, ad);
      b[2] = fma2(pair2(bf_lo(raw.z), bf_hi(raw.z)), l2e, ad);
      b[3] = fma2(pair2(bf_lo(raw.w), bf_hi(raw.w)), l2e, ad);
    } else {
#pragma unroll
      for (int e = 0; e < 4; ++e) b[e] = ad;
    }
#pragma unroll
    for (int e = 0; e < 4; ++e) t[u * 4 + e] = fma2(pair2(s[u * 8 + 2 * e], s[u * 8 + 2 * e + 1]), sc, b[e]);
    if (!PLAIN) {
      const float4 k0 = *reinterpret_cast<const float4*>(pen + c0 + u * 8);         // same address in every lane: broadcast
      const float4 k1 = *reinterpret_cast<const float4*>(pen + c0 + u * 8 + 4);
      t[u * 4] = add2(t[u * 4], pair2(k0.x, k0.y));
      t[u * 4 + 1] = add2(t[u * 4 + 1], pair2(k0.z, k0.w));
      t[u * 4 + 2] = add2(t[u * 4 + 2], pair2(k1.x, k1.y));
      t[u * 4 + 3] = add2(t[u * 4 + 3], pair2(k1.z, k1.w));
    }
  }
}

// 16 columns of a row
__device__ __forceinline__ void tmem_ld_32x16(uint32_t taddr, float (&v)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]), "=f"(v[7]), "=f"(v[8]), "=f"(v[9]), "=f"(v[10]),
        "=f"(v[11]), "=f"(v[12]), "=f"(v[13]), "=f"(v[14]), "=f"(v[15])
      : "r"(taddr));
}

// tmem_ld_wait that the loaded registers pass through: nothing that reads them moves ahead of it
template <int N>
__device__ __forceinline__ void tmem_ld_wait_for(float (&v)[N]) {
  tmem_ld_wait();
#pragma unroll
  for (int i = 0; i < N; i += 8)
    asm volatile("" : "+f"(v[i]), "+f"(v[i + 1]), "+f"(v[i + 2]), "+f"(v[i + 3]), "+f"(v[i + 4]), "+f"(v[i + 5]), "+f"(v[i + 6]), "+f"(v[i + 7]));
}

// The 64 logits of a row's block, 16 at a time with the next 16 on their way: p = exp2(t), packed to bf16 pairs, and the two-wide
// running sum of p as rounded to bf16 - that is what the tensor core multiplies V with, so in a row that one key dominates the
// rounding of its p cancels.  Not PLAIN: where none of 16 keys counts the weights are 0.
// `after_first` is called once a quarter is done.
template <bool PLAIN, bool BIAS, typename F>
__device__ __forceinline__ void softmax_block(uint32_t tm_s, const uint8_t* brow, int r, const float* pen, float scale_log2e, float add,
                                              Keys keys, uint32_t (&p)[32], float2& sum, F&& after_first) {
  float s[2][16];
  tmem_ld_32x16(tm_s, s[0]);
  tmem_ld_wait_for(s[0]);
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    if (q < 3) tmem_ld_32x16(tm_s + (q + 1) * 16, s[(q + 1) & 1]);
    if (q == 1) after_first();
    if (PLAIN || ((q < 2 ? keys.lo : keys.hi) & (q & 1 ? 0xffff0000u : 0xffffu))) {
      uint64_t t[8];
      logits16<PLAIN, BIAS>(t, s[q & 1], brow, r, q * 16, pen, scale_log2e, add);
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const float2 f = split2(t[i]);
        const bf162 h = __floats2bfloat162_rn(ex2f(f.x), ex2f(f.y));
        const uint32_t w = *reinterpret_cast<const uint32_t*>(&h);
        p[q * 8 + i] = w;
        sum.x = add_lo(sum.x, w);
        sum.y = add_hi(sum.y, w);
      }
    } else {
#pragma unroll
      for (int i = 0; i < 8; ++i) p[q * 8 + i] = 0u;
    }
    if (q < 3) tmem_ld_wait_for(s[(q + 1) & 1]);
  }
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
// model's own biases gets here, and the ordinary path uses all registers that four warps per scheduler leave: a call or wider
// pieces cost it.
template <bool BIAS>
__device__ __forceinline__ RowState far_block(RowState st, bool move, uint32_t tm_s, uint32_t tm_o, bool has_o, const uint8_t* brow, int r,
                                           Keys kb, int keys, float scale, float scale_log2e) {
  constexpr float LN2 = 0.6931471805599453f;
  const uint64_t keep = kb.lo | (uint64_t)kb.hi << 32;        // `keys` of the 64 are in the sequence
  auto load = [&](int c, float (&s)[8], float (&b)[8]) {
    tmem_ld_32x8(tm_s + c * 8, s);
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
      tmem_ld_32x8(tm_o + c * 8, o);
      tmem_ld_wait();
#pragma unroll
      for (int e = 0; e < 8; ++e) o[e] *= alpha;
      tmem_st_32x8(tm_o + c * 8, o);
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
    tmem_st_32x4(tm_s + c * 4, p);         // over columns that have been read: 4c + 3 < 8 (c + 1)
  }
  st.l = st.l * alpha + sum;
  return st;
}

// Where the rows of a (query tile, batch row) lie in the tile's 128 lanes.  The last tile of a sequence may fill only some of the
// four warps; such a tile is loaded so that it starts at another warp's lanes from batch row to batch row, because warp q of a
// group runs on scheduler q: the warps without a row have nothing to do, and the work stays spread over the schedulers.
struct TileRows {
  int first, warps;               // first warp with rows, number of warps with rows
};
__device__ __forceinline__ TileRows tile_rows(int n_q, int qt, int b) {
  const int rows = n_q - qt * AF_BQ;
  TileRows t;
  t.warps = rows >= AF_BQ ? 4 : (rows + 31) >> 5;
  t.first = t.warps == 1 ? (b & 3) : t.warps == 2 ? (b & 1) * 2 : t.warps == 3 ? (b & 1) : 0;
  return t;
}

// A round is up to AF_GROUPS batch rows of one (head, query tile), spread evenly over the tile's rounds; rounds are numbered tile by
// tile, and every role of a CTA walks the same ones.
struct Round {
  int i, b, cnt;                  // number, first batch row, batch rows
  int k, qt, h;                   // number within the tile, query tile, head
  __device__ __forceinline__ Round(const AttnInferArgs& a, int round) : i(round) {
    const int tile = round / a.rounds;
    k = round - tile * a.rounds;
    h = tile / a.n_qt;
    qt = tile - h * a.n_qt;
    rows(a);
  }
  __device__ __forceinline__ void rows(const AttnInferArgs& a) {       // the first `rest` rounds have a row more than the others
    b = k * a.few + min(k, a.rest);
    cnt = a.few + (k < a.rest);
  }
  __device__ __forceinline__ void next(const AttnInferArgs& a) {
    ++i;
    if (++k == a.rounds) {
      k = 0;
      if (++qt == a.n_qt) {
        qt = 0;
        ++h;
      }
    }
    rows(a);
  }
  __device__ __forceinline__ bool fresh() const { return k == 0; }     // first round of a tile
  __device__ __forceinline__ bool last(const AttnInferArgs& a) const { return k + 1 == a.rounds; }
};

// Rounds are shared out by their cost: first round at or after position `x` of the work.
template <typename T>
__device__ __forceinline__ int round_at(const AttnInferArgs& a, T x) {
  if (a.n_qt == 1) return (int)((x + a.cost_last - 1) / a.cost_last);
  const T full = (T)AF_COST * (a.n_qt - 1) * a.rounds, head = full + (T)a.cost_last * a.rounds;
  const int h = (int)(x / head);
  const T rem = x - h * head;
  const int in_head = rem <= full ? (int)((rem + AF_COST - 1) / AF_COST) : (a.n_qt - 1) * a.rounds + (int)((rem - full + a.cost_last - 1) / a.cost_last);
  return h * a.n_qt * a.rounds + in_head;
}
// where the rounds of CTA `i` begin
__device__ __forceinline__ int cta_begin(const AttnInferArgs& a, int i) {
  const long long x = a.share * i + min(i, a.extra);
  return a.share * gridDim.x < 0x70000000LL ? round_at<uint32_t>(a, (uint32_t)x) : round_at<long long>(a, x);
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
  // barrier map (8 bytes each): [group][2] Q stages, [group][AF_KVST] K / V stages, [slot] bias, [group][2] S buffers
  const uint32_t q_full = b0, q_empty = b0 + 48, kv_full = b0 + 96, kv_empty = b0 + 192, bias_full = b0 + 288, bias_empty = b0 + 320;
  const uint32_t s_full = b0 + 352, p_full = b0 + 400, o_done = b0 + 448;
  static_assert(AF_GROUPS == 3 && AF_KVST == 4 && AF_BSLOTS == 4, "barrier map");
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(sm + AttnInferSmem::BARS + 512);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    for (int i = 0; i < 2 * AF_GROUPS; ++i) {
      mbar_init(q_full + 8 * i, 1);
      mbar_init(q_empty + 8 * i, 1);
      mbar_init(s_full + 8 * i, 2);               // the S product, and the block's key bits
      mbar_init(p_full + 8 * i, 4);
      mbar_init(o_done + 8 * i, 1);
    }
    for (int i = 0; i < AF_KVST * AF_GROUPS; ++i) {
      mbar_init(kv_full + 8 * i, 1);
      mbar_init(kv_empty + 8 * i, 1);
    }
    for (int i = 0; i < AF_BSLOTS; ++i) {
      mbar_init(bias_full + 8 * i, 1);
      mbar_init(bias_empty + 8 * i, AF_GROUPS);
    }
    *abort_flag = 0;
    for (int i = 0; i < 4; ++i) reinterpret_cast<int*>(sm + AttnInferSmem::TURN)[i] = 0;
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
  // contiguous range of rounds of this CTA
  const int r_begin = cta_begin(a, blockIdx.x), r_end = cta_begin(a, blockIdx.x + 1);
  const Round rd0(a, r_begin);
  pdl_wait();          // the prologue above touched no global memory; everything below may
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;

  // A wait of this CTA's pipeline.  The first one that runs out reports and sets the flag, at which all others end: the kernel
  // then runs to its end on whatever the buffers hold, and the caller sees the status.  A try lasts 4 us; the flag is looked at after a few
  // of them, since a wait may still follow for every block that this CTA has left.
  auto wait = [&](uint32_t bar, uint32_t parity, int code, int detail) -> bool {
    if (mbar_try_wait(bar, parity)) return true;
    const uint64_t t0 = globaltimer_ns();
    for (;;) {
#pragma unroll 1
      for (int i = 0; i < 8; ++i)
        if (mbar_try_wait(bar, parity)) return true;
      if (*abort_flag) return false;
      if (globaltimer_ns() - t0 > FFB_LOCAL_WAIT_NS) {
        report(code, detail);
        *abort_flag = 1;
        return false;
      }
    }
  };


  // The producer and the issuers run as whole warps (see umma_bf16_by).
  if (warp == 0) {
    // ---------------- TMA producer ----------------
    const uint32_t lead = elect_one();
    uint32_t qi[AF_GROUPS], jt[AF_GROUPS];     // items and key blocks loaded per group
#pragma unroll
    for (int g = 0; g < AF_GROUPS; ++g) qi[g] = jt[g] = 0;
    uint32_t fill = 0;                         // bias: streamed tiles so far, or resident (head, tile) sets so far
    bool ok = true;
    for (Round rd = rd0; rd.i < r_end && ok; rd.next(a)) {
      const int cnt = rd.cnt, bb = rd.b, qt = rd.qt, h = rd.h;
      const bool load_bias = BIAS && (!a.bias_resident || rd.i == r_begin || rd.fresh());
      const uint32_t set = fill;               // resident: index of the set loaded in this round
      if (load_bias && a.bias_resident) ++fill;
      for (int j = 0; j < a.n_kb && ok; ++j) {
#pragma unroll
        for (int g = 0; g < AF_GROUPS; ++g) {
          if (g >= cnt || !ok) continue;
          if (j == 0) {
            const uint32_t qs = g * 2 + (qi[g] & 1);
            if (!(ok = wait(q_empty + 8 * qs, ((qi[g] >> 1) & 1) ^ 1, ST_TIMEOUT_MMA, 10))) continue;
            mbar_expect_tx_by(lead, q_full + 8 * qs, Q_BYTES);
            tma_load_3d_by(lead, base + AttnInferSmem::Q + qs * 8192, &tmQ, q_full + 8 * qs, h * D, qt * AF_BQ - 32 * tile_rows(a.n_q, qt, bb + g).first, bb + g);
            ++qi[g];
          }
          const uint32_t ks = g * AF_KVST + (jt[g] % AF_KVST);
          if (!(ok = wait(kv_empty + 8 * ks, ((jt[g] / AF_KVST) & 1) ^ 1, ST_TIMEOUT_MMA, 12))) continue;
          mbar_expect_tx_by(lead, kv_full + 8 * ks, 2 * KV_BYTES);
          tma_load_3d_by(lead, base + AttnInferSmem::KV + ks * 8192, &tmK, kv_full + 8 * ks, h * D, j * AF_BK, bb + g);
          tma_load_3d_by(lead, base + AttnInferSmem::KV + ks * 8192 + 4096, &tmV, kv_full + 8 * ks, h * D, j * AF_BK, bb + g);
          ++jt[g];
        }
        if (load_bias && ok) {
          const uint32_t slot = a.bias_resident ? (uint32_t)j : fill % AF_BSLOTS;
          const uint32_t nth = a.bias_resident ? set : fill / AF_BSLOTS;       // fill index of this slot
          if (!(ok = wait(bias_empty + 8 * slot, (nth & 1) ^ 1, ST_TIMEOUT_EPI, 11))) break;
          mbar_expect_tx_by(lead, bias_full + 8 * slot, 16384);
          tma_load_3d_by(lead, base + AttnInferSmem::BIAS + slot * 16384, &tmBias, bias_full + 8 * slot, j * AF_BK, qt * AF_BQ, h);
          if (!a.bias_resident) ++fill;
        }
      }
    }
    if (!ok) {                                 // copies that nobody will wait for any more: they land long before this ends
      const uint64_t t0 = globaltimer_ns();
      while (globaltimer_ns() - t0 < 1000000ull) {
      }
    }
  } else if (warp <= AF_GROUPS) {
    // ---------------- MMA issuer of one group ----------------
    const uint32_t lead = elect_one();
    constexpr uint32_t idesc_s = make_idesc_bf16(128, AF_BK, 0, 0);     // Q (K-major) x K (K-major)
    constexpr uint32_t idesc_o = make_idesc_bf16(128, D, 0, 1);         // P (tensor memory) x V (MN-major)
    const int g = warp - 1;
    const uint32_t tg = tmem + (uint32_t)g * AF_TM_GROUP;
    // descriptors of stage 0; the address field counts 16 bytes, so stages are additions
    const uint64_t dq = make_desc(base + AttnInferSmem::Q + g * 16384, 16, GROUP, LAYOUT),
                   dk = make_desc(base + AttnInferSmem::KV + g * AF_KVST * 8192, 16, GROUP, LAYOUT),
                   dv = make_desc(base + AttnInferSmem::KV + g * AF_KVST * 8192 + 4096, 16, GROUP, LAYOUT);
    uint32_t si = 0, qi = 0, pi = 0;                                    // S products, items, PV products issued
    Round rs = rd0;                                               // block of the next S product
    int sj = 0;
    auto next_s = [&]() {                                               // rounds without a row for this group have none
      while (rs.i < r_end && g >= rs.cnt) rs.next(a);
    };
    next_s();
    // Two S products ahead, but not past the round after the one whose P V products are being issued: in a round without a row
    // for this group there are still bias tiles to release.
    int reach = r_begin;
    uint32_t slot = 0, bpar = a.bias_resident ? 1u : 0u;                // bias tile of the block, phase of its barrier
    // This warp has time to spare: it also works out which keys of a block count, from entries loaded a block ahead.
    Keys* key_ring = reinterpret_cast<Keys*>(sm + AttnInferSmem::KEYS) + g * 2;
    const bf16* mrow = nullptr;
    KeyMask km = {0, 0};
    auto look_ahead = [&]() {
      if (rs.i >= r_end) return;
      if (sj == 0) mrow = a.mask ? a.mask + (long long)(rs.b + g) * a.mask_bstride : nullptr;
      km = load_keys(mrow, sj * AF_BK, a.n_k, lane);
    };
    look_ahead();
    // S product of the next block, into the buffer whose last P V product is over.  That one has been issued by then, but products with
    // different accumulators and shapes have no order among themselves.  The wait is short and nobody needs this S for a block yet
    auto issue_s = [&]() {
      const uint32_t qs = g * 2 + (qi & 1), ks = g * AF_KVST + si % AF_KVST;
      const Keys keys = key_bits(km);
      if (sj == 0) wait(q_full + 8 * qs, (qi >> 1) & 1, ST_TIMEOUT_TMA, 22);
      wait(kv_full + 8 * ks, (si / AF_KVST) & 1, ST_TIMEOUT_TMA, 20);
      wait(o_done + 8 * (g * 2 + (si & 1)), ((si >> 1) & 1) ^ 1, ST_TIMEOUT_MMA, 24);
      tc_fence_after();
      const uint64_t q = dq + (qi & 1) * (8192 >> 4), k = dk + (si % AF_KVST) * (8192 >> 4);
#pragma unroll
      for (int i = 0; i < D / 16; ++i) umma_bf16_by(lead, tg + (si & 1) * AF_BK, q + i * (32 >> 4), k + i * (32 >> 4), idesc_s, i > 0 ? 1u : 0u);
      umma_commit_by(lead, s_full + 8 * (g * 2 + (si & 1)));
      if (lead) {
        key_ring[si & 1] = keys;
        mbar_arrive(s_full + 8 * (g * 2 + (si & 1)));
      }
      ++si;
      if (++sj == a.n_kb) {
        umma_commit_by(lead, q_empty + 8 * qs);       // all S products of this item issued: the Q slot drains with them
        ++qi;
        sj = 0;
        rs.next(a);
        next_s();
      }
      look_ahead();
    };
    for (Round rd = rd0; rd.i < r_end; rd.next(a)) {
      if (BIAS && a.bias_resident) {
        slot = 0;
        bpar ^= rd.i == r_begin || rd.fresh();
      }
      // resident tiles are released in the last round that reads them, streamed ones at once
      const bool release = BIAS && (!a.bias_resident || rd.i + 1 == r_end || rd.last(a));
      const bool active = g < rd.cnt;
      reach = rd.i + 1;
      while (active && si < pi + 2 && rs.i < r_end && rs.i <= reach) issue_s();
      for (int j = 0; j < a.n_kb; ++j) {
        if (active) {
          const uint32_t buf = pi & 1, st = pi % AF_KVST;
          // the group has read S of this block and written P
          wait(p_full + 8 * (g * 2 + buf), (pi >> 1) & 1, ST_TIMEOUT_EPI, 23);
          tc_fence_after();
          const uint64_t v = dv + st * (8192 >> 4);
#pragma unroll
          for (int k = 0; k < AF_BK / 16; ++k)
            umma_bf16_ts_by(lead, tg + AF_TM_O, tg + buf * AF_BK + k * 8, v + ((k * 2 * GROUP) >> 4), idesc_o, (j > 0 || k > 0) ? 1u : 0u);
          umma_commit_by(lead, o_done + 8 * (g * 2 + buf));
          umma_commit_by(lead, kv_empty + 8 * (g * AF_KVST + st));
          ++pi;
        } else if (release) {
          wait(bias_full + 8 * slot, bpar, ST_TIMEOUT_TMA, 30);
        }
        if (release) {
          if (lead) mbar_arrive(bias_empty + 8 * slot);
          if (++slot == AF_BSLOTS && !a.bias_resident) {
            slot = 0;
            bpar ^= 1;
          }
        }
        if (active && rs.i < r_end && rs.i <= reach) issue_s();
      }
    }
    if (*abort_flag) {                         // products that nobody will wait for any more: they are over long before this ends
      const uint64_t t0 = globaltimer_ns();
      while (globaltimer_ns() - t0 < 1000000ull) {
      }
    }
  } else {
    // ---------------- softmax / output (warps 4..15): group = batch row of the round, thread = query row ----------------
    const int quad = warp & 3;                      // TMEM lane quadrant this warp may read
    const int g = (warp - 4) >> 2;
    const uint32_t tg = tmem + ((uint32_t)(quad * 32) << 16) + (uint32_t)g * AF_TM_GROUP;
    float* pen = reinterpret_cast<float*>(sm + AttnInferSmem::KP) + (warp - 4) * 64;
    uint32_t jt = 0;                                // blocks of this group so far
    // Warps that share a scheduler (one of each group) begin a block one after the other: a warp takes the turn for the first
    // quarter of its logits.  Left alone they fall into step - whoever is ahead finds fewer others and is slowed down when they
    // come - and then all are in their exponentials at once and all between blocks at once (n 1024: 2700 cycles a block, of which
    // 450 between blocks; n 1536, B 384: 1440 us, 1380 with turns).  Only a hint: the tries are few, and it is harmless to go on
    // without the turn.
    int* turn = reinterpret_cast<int*>(sm + AttnInferSmem::TURN) + quad;
    auto take_turn = [&]() {
      if (lane == 0)
        for (int i = 0; i < 32 && atomicExch(turn, 1) != 0; ++i) {
        }
      __syncwarp();
    };
    auto pass_turn = [&]() {
      if (lane == 0) *reinterpret_cast<volatile int*>(turn) = 0;
    };
    // P V product of block `t` of this group: O holds it
    auto wait_o = [&](uint32_t t, int detail) {
      wait(o_done + 8 * (g * 2 + (t & 1)), (t >> 1) & 1, ST_TIMEOUT_MMA, detail);
      __syncwarp();
      tc_fence_after();
    };
    const Keys* key_ring = reinterpret_cast<const Keys*>(sm + AttnInferSmem::KEYS) + g * 2;
    uint32_t slot = 0, bpar = a.bias_resident ? 1u : 0u;      // bias tile of the block, phase of its barrier
    for (Round rd = rd0; rd.i < r_end; rd.next(a)) {
      const bool first = rd.i == r_begin || rd.fresh();
      if (BIAS && a.bias_resident) {
        slot = 0;
        bpar ^= first;
      }
      if (g >= rd.cnt) {
        if (BIAS && !a.bias_resident) {             // tiles of a round without a row for this group
          slot += a.n_kb;
          bpar ^= (slot / AF_BSLOTS) & 1;
          slot %= AF_BSLOTS;
        }
        continue;
      }
      const int qt = rd.qt, h = rd.h, b = rd.b + g;
      const bool look = BIAS && (!a.bias_resident || first);                        // tiles that this warp has not waited for yet
      const TileRows rows = tile_rows(a.n_q, qt, b);
      const bool mine = quad >= rows.first && quad < rows.first + rows.warps;       // this warp has query rows
      const int r = (quad - rows.first) * 32 + lane;                                // row within the query tile
      RowState row = {0.f, 0.f, false};
      for (int j = 0; j < a.n_kb; ++j) {
        // S first: the phase of the bias tile's barrier means something only once S is there, until then tiles of a round without a
        // row for this group may still be on their way.  Not side by side either: the first may be suspended and end well while
        // the second has long been answered.
        wait(s_full + 8 * (g * 2 + (jt & 1)), (jt >> 1) & 1, ST_TIMEOUT_MMA, 31);
        if (look) wait(bias_full + 8 * slot, bpar, ST_TIMEOUT_TMA, 32);
        __syncwarp();
        tc_fence_after();
        const uint8_t* brow = BIAS ? sm + AttnInferSmem::BIAS + slot * 16384 + r * 128 : nullptr;
        const uint32_t tm_s = tg + (jt & 1) * AF_BK;
        if (mine) {
          const Keys kb = key_ring[jt & 1];
          const bool plain = (kb.lo & kb.hi) == 0xffffffffu;           // every key of this block in range and unmasked
          if (kb.lo | kb.hi) {
            float2 sum = {0.f, 0.f};
            uint32_t p[32];                         // stored once the sum is known to be in range: P takes the place of S
            bool store = true;
            if (plain) {
              take_turn();
              softmax_block<true, BIAS>(tm_s, brow, r, pen, a.scale_log2e, -row.M, kb, p, sum, pass_turn);
            } else {
              write_penalties(pen, lane, kb.lo, kb.hi);
              softmax_block<false, BIAS>(tm_s, brow, r, pen, a.scale_log2e, -row.M, kb, p, sum, []() {});
            }
            const float ln = row.l + (sum.x + sum.y);
            const bool bad = row.far || !(ln > ROW_SUM_LO && ln < ROW_SUM_HI);
            if (__any_sync(0xffffffffu, bad)) {
              // some row's sum has left the safe range (first block of a row with large logits, only masked keys before this
              // block, or a much larger logit in it): move that row's reference point and redo the block
              if (plain) write_penalties(pen, lane, 0xffffffffu, 0xffffffffu);
              float mx = -INFINITY, alpha = 1.f;
              if (j > 0) wait_o(jt - 1, 34);
#pragma unroll 1
              for (int c = 0; c < 4; ++c) {
                float s[16];
                uint64_t t[8];
                tmem_ld_32x16(tm_s + c * 16, s);
                tmem_ld_wait_for(s);
                logits16<false, BIAS>(t, s, brow, r, c * 16, pen, a.scale_log2e, 0.f);
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                  const float2 f = split2(t[i]);
                  mx = fmaxf(mx, fmaxf(f.x, f.y));
                }
              }
              const float m2 = (row.l > 0.f && !row.far) ? fmaxf(mx, row.M + log2f(row.l)) : mx;
              // a row that leaves the domain of the ordinary path, or that has not re-entered it from above
              const bool out = bad && (!(fabsf(m2) < FAR_LOGIT) || (row.far && row.M > 0.f));
              if (__any_sync(0xffffffffu, out)) {
                row = far_block<BIAS>(row, bad, tm_s, tg + AF_TM_O, j > 0, brow, r, kb, a.n_k - j * AF_BK, a.scale, a.scale_log2e);
                store = false;
              } else {
                if (bad) {
                  if (row.l > 0.f) alpha = ex2f((row.far ? row.M * LOG2E : row.M) - m2);
                  row.M = m2;
                  row.far = 0;
                }
                if (j > 0) {
                  float o[32];                      // D = 16: the upper columns are nobody's
                  tmem_ld_32x32(tg + AF_TM_O, o);
                  tmem_ld_wait_for(o);
#pragma unroll
                  for (int c = 0; c < 32; ++c) o[c] *= alpha;
                  tmem_st_32x32(tg + AF_TM_O, o);
                }
                sum = {0.f, 0.f};
                softmax_block<false, BIAS>(tm_s, brow, r, pen, a.scale_log2e, -row.M, kb, p, sum, []() {});
                row.l = row.l * alpha + (sum.x + sum.y);
              }
            } else {
              row.l = ln;
            }
            if (store) tmem_st_32x32(tm_s, reinterpret_cast<const float*>(p));
          } else {
            // masked keys next to a real one have weight 0; where there has been no other key they all have the same logit
            const bool alone = row.l == 0.f || (row.far && row.M == MASKED_LOGIT);
            if (__any_sync(0xffffffffu, row.far && !alone)) {
              if (j > 0) wait_o(jt - 1, 32);
              row = far_block<BIAS>(row, alone || row.far, tm_s, tg + AF_TM_O, j > 0, brow, r, kb, a.n_k - j * AF_BK, a.scale, a.scale_log2e);
            } else {
              const Keys valid = key_bits(load_keys(nullptr, j * AF_BK, a.n_k, lane));
              if (alone) {
                row.M = MASKED_LOGIT;
                row.far = 1;
                row.l += (float)(__popc(valid.lo) + __popc(valid.hi));
              }
              uint32_t p[32];
#pragma unroll
              for (int i = 0; i < 32; ++i) {
                const uint32_t bits = ((i < 16 ? valid.lo : valid.hi) >> (2 * (i & 15))) & 3u;
                p[i] = alone ? (bits & 1u) * 0x3f80u + (bits >> 1) * 0x3f800000u : 0u;
              }
              tmem_st_32x32(tm_s, reinterpret_cast<const float*>(p));
            }
          }
        }                                           // other warps: nothing of their lanes is ever read
        tmem_st_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(p_full + 8 * (g * 2 + (jt & 1)));        // P is complete, S and the bias have been read
        if (BIAS && ++slot == AF_BSLOTS && !a.bias_resident) {
          slot = 0;
          bpar ^= 1;
        }
        ++jt;
      }
      // ---- the item's output row ----
      if (!mine) continue;
      wait_o(jt - 1, 33);
      float o[32];                                  // D = 16: the upper columns are nobody's
      tmem_ld_32x32(tg + AF_TM_O, o);
      tmem_ld_wait_for(o);
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
  static int sm_count = 0;
  if (!sm_count) {
    int dev = 0;
    cudaGetDevice(&dev);
    if (cudaDeviceGetAttribute(&sm_count, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sm_count <= 0) sm_count = 148;
  }
  // Batch rows per round: three at a time give the most per SM (blocks of 64 keys with one, two, three softmax warps on a scheduler
  // take 1020, 1500, 2000 cycles), but a grid of few rounds is done sooner with less in each.
  long long best = 0;
  for (int c = AF_GROUPS; c > 0; --c) {
    const long long per_tile = (B + c - 1) / c, time = ((long long)H * a.n_qt * per_tile + sm_count - 1) / sm_count * (c + 1);
    if (c == AF_GROUPS || time < best) {
      best = time;
      a.rounds = (int)per_tile;
    }
  }
  a.few = B / a.rounds;
  a.rest = B - a.few * a.rounds;
  // Last query tile with rows for 1 .. 4 warps of a group (n_k 512 with bias, B 3552, H 1: 69, 78, 100, 105 us; n_k 192: 31, 34, 46, 49).
  static const int cost[4] = {10, 12, 15, AF_COST};
  const bool one_each = (long long)H * a.n_qt * a.rounds <= sm_count;
  a.cost_last = one_each ? AF_COST : cost[(n_q - (a.n_qt - 1) * AF_BQ + 31) / 32 - 1];
  const long long work = (long long)H * a.rounds * (AF_COST * (a.n_qt - 1) + a.cost_last);
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
  const long long rounds = (long long)H * a.n_qt * a.rounds;
  const int grid = rounds < sm_count ? (int)rounds : sm_count;
  a.share = work / grid;
  a.extra = (int)(work % grid);
  launch_k(kern, grid, AF_THREADS, AttnInferSmem::TOTAL,
           reinterpret_cast<cudaStream_t>(stream), tq, tk, tv, tb, a);
  return cudaGetLastError() == cudaSuccess ? 0 : -15;
}

}  // extern "C"

// LayerNorm of the rows of an activation and the small GEMMs that follow it, in one kernel:
//
//   chains       out = resid + b2 + f(LN(x) W1^T + b1) W2^T      f = relu (transition) or sigmoid(.) * o (gated attention output)
//   projections  y_s = act(LN(x) W_s^T + b_s) ...                up to three weights that read the same rows (QKV and pair bias;
//                                                                gated operands and output gate of the triangle multiplication)
//
// The modules of the trunk are made of these: a LayerNorm over 64, 128 or 256 channels and one or two products with weights of a
// few hundred kilobytes.  As single kernels each wrote its result to memory and the next one read it back, the hidden
// activation of a transition (four times its input) among them, and on short inputs each was a launch.  Here a tile of 128 rows is
// read once; its normalised form (rounded to bf16, as the LayerNorm kernel stores it) and the hidden activation never leave the SM.
//
// Persistent, one CTA per SM, 448 or 704 threads, tiles of 128 rows:
//   warps 0-3    LayerNorm, a thread per row (channels-first input: per pair of rows and half of the channels), in place in the
//                shared-memory tile that becomes the A operand.  The 128-byte swizzle makes a thread's 16-byte accesses to its own row
//                free of conflicts, so no shuffles are needed
//   then         epilogues, a team of eight warps, two per tensor-memory quadrant with 64 columns each; 64 and 128 channels have two
//                teams: the epilogues are the longest chain there, most of it latency (1600 cycles for 64 columns that are only
//                converted), and two warps per scheduler do not hide it.  Of projections they take the chunks in turn, of chains one
//                has the hidden activation and the other the result.  At 256 channels, whose staging tiles would cost two boxes of the
//                ring, two teams are slower (block of 128 x 203 588 -> 591, of 256 x 384 in chunks 2172 -> 2183)
//   then a warp  TMA: rows of the next tile, weights through a ring of 16 KB boxes (128 rows x 64 columns; out of L2 for all but the
//                first CTA)
//   and one      MMA issue, 128 x 128 x 16
// Weights come in chunks of 128 rows.  Of a chain, chunk h of the hidden activation goes through tensor memory: the epilogue
// reads the accumulator, applies f and writes bf16 pairs over it, and the second product takes them from there as its A operand.
// The products of chunk h + 1 are issued before the second product of chunk h, which hides the epilogue; at 64 and 128 channels, with
// two tiles of rows, so are those of the next tile's first chunk (triangle attention 389 243 -> 240 us, extra-MSA stack 511 -> 498: in the
// gated outputs, which have one chunk a tile, the epilogue had waited for the products of every tile).
//
// What bounds it: the weights, which every tile of 128 rows streams from L2 again (1 MB a tile for the transition of 256 channels, which
// at 32768 rows runs at 0.44 of the tensor cores' rate), the output bytes of the wide projections, and with few tiles the chain of one.
//   Measured (B200, against LayerNorm and GEMM kernels in the same order, us): transition 262144 x 64 89 -> 46, 65536 x 128
//   47 -> 32, 589824 x 128 341 -> 208, 32768 x 256 54 -> 48, 2048 x 256 16 -> 26 (one launch in place of three: host/dispatch.cpp, which chooses,
//   has the line between the two); gated output with the norm (left side without it) 589824 x 128 192 -> 139, 32768 x 256 30 -> 24; QKV 589824 x 128
//   181 -> 130; operands and gate of the triangle multiplication at 1024 residues 539 -> 480, its output 293 -> 177.
//   Two teams instead of one, projections, then chains too: triangle multiplication 1024 1004 -> 932, a block of 128 x 256
//   729 -> 698 -> 694, of 256 x 384 in chunks 2240 -> 2182 -> 2172, the extra-MSA stack of 1024 x 256 531 -> 517 -> 511; a block of 32 x 64
//   as before.
//
// Stands for the nn.LayerNorm / nn.Linear / elementwise chains of the reference (fastfold/model/fastnn/ops.py:85-106, 143-160,
// 275-324, 393-404).
#include "common.cuh"
#include "gemm_api.h"
#include "ln_gemm_api.h"
#include "tmap.h"

namespace ffb {

constexpr int LG_EPI = 8;                 // epilogue warps of a chunk
constexpr int LG_BOX = 16384;             // weight box: 128 rows x 64 columns
constexpr int LG_MAX_N = 1280;            // columns of all weights (biases in shared memory)

struct LgMaps {
  CUtensorMap x, w[3], mul, resid, out[3];
};

struct LgSeg {
  int kind, act, scaled, n;
  bf16* out;
};

struct LgArgs {
  int rows, batch, tiles_m, num_tiles;
  int bpt;                                // batches per tile: 128 / rows where that is 2 or 4, else 1
  const bf16 *gamma, *beta;
  float eps;
  int hidden, has_mul;
  const float* mul_f32;
  int mul_mod;
  const bf16 *b1, *b2;
  int nseg, chunks;                       // projections: segments, chunks of 128 weight rows in all
  LgSeg seg[3];
  const bf16* seg_bias[3];
  const void* rowscale;
  int rs_bf16;
  long long pb_h, pb_i, pb_j;
  int pb_n;
};

// TEAMS: teams of eight epilogue warps.  Two teams make 22 warps, which leaves a thread 80 registers; the epilogues keep 32 columns of
// their row in them then, and some bytes are spilled (gated chain of 64 channels 40, projections of 128 channels 16, projections and relu
// chain of 64 channels 12).  NARROW: projections of 256 channels to few columns, which need two tiles of rows on their way
// more than boxes of weights
template <int C, int MODE, int TEAMS, bool NARROW>
struct LgCfg {
  static constexpr int EPI = LG_EPI * TEAMS, THREADS = (6 + EPI) * 32, TMA = 4 + EPI, MMA = 5 + EPI;       // the last two are warps
  static_assert(C != 256 || TEAMS == 1, "no room for the staging tiles of two teams");
  static constexpr int KB = C / 64;
  static constexpr int A_BYTES = KB * 16384;
  static constexpr int TILES = C == 256 || TEAMS == 2 ? 1 : 2;      // 4 KB staging tiles per epilogue warp (two: channels-first rows)
  static constexpr int NA = C == 256 && !NARROW ? 1 : 2;             // tiles of rows: one less, and the ring holds four boxes more
  static constexpr int RING = NARROW ? 3 : C == 256 ? 7 : 5;
  static constexpr int NB2 = C < 128 ? C : 128;                      // columns of one second product
  static constexpr int NACC = MODE == LN_PROJECT ? 4 : (C == 256 ? 2 : 3);      // 128-column accumulators of the first product
  static constexpr int ACC2 = NACC * 128;                            // tensor-memory column of the second product's accumulator
  static constexpr int A0 = 0, W0 = NA * A_BYTES, STG = W0 + RING * LG_BOX, VEC = STG + EPI * TILES * 4096;
  static constexpr int VEC_FLOATS = 2 * C + LG_MAX_N + 256 + (MODE == LN_PROJECT ? 1280 : 0);     // gamma, beta, biases, channel sums
  static constexpr int BARS = VEC + VEC_FLOATS * 4;
  static constexpr int SMEM = BARS + 512 + 1024;
  static_assert(SMEM <= 232448, "shared memory");
};

__device__ __forceinline__ void lg_unpack(uint4 u, float (&v)[8]) {
  const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    v[2 * i] = __uint_as_float(w[i] << 16);
    v[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
  }
}
__device__ __forceinline__ uint32_t lg_pack2(float a, float b) {
  const bf162 h = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<const uint32_t*>(&h);
}
__device__ __forceinline__ uint4 lg_pack(const float* v) { return make_uint4(lg_pack2(v[0], v[1]), lg_pack2(v[2], v[3]), lg_pack2(v[4], v[5]), lg_pack2(v[6], v[7])); }

__device__ __forceinline__ uint64_t lg_bf2(uint32_t w) { return pair2(__uint_as_float(w << 16), __uint_as_float(w & 0xffff0000u)); }
__device__ __forceinline__ uint32_t lg_pack2v(uint64_t v) {
  const float2 f = split2(v);
  return lg_pack2(f.x, f.y);
}

// One row of a [kb][128 rows][64] swizzled tile, in place.  A warp per scheduler does this, so what counts are its instructions and
// the independent ones among them: two-wide arithmetic in four chains.
// The sums are taken in the order of the LayerNorm kernel (ln_fwd_mr_kernel: eight channels per lane one by one, then lanes half a row
// apart, a quarter apart, ...), so that both give the same bits; the two halves of a pair of floats are the same channel of two pieces of
// eight channels.  Against sums in whatever order suits the registers (us, in a graph with the kernels around them): MSA half of a block of
// 128 x 256 246.9 -> 248.9, pair half 376.2 -> 375.9, extra-MSA core of 1024 x 256 617 -> 619.
template <int C>
__device__ __forceinline__ void lg_norm_row(uint8_t* tile, int row, const float* gamma, const float* beta, float eps) {
  constexpr int KB = C / 64;
  uint8_t* p = tile + row * 128;
  const int x = row & 7;
  auto load = [&](uint4 (&raw)[8], int kb) {
#pragma unroll
    for (int u = 0; u < 8; ++u) raw[u] = *reinterpret_cast<const uint4*>(p + kb * 16384 + ((u ^ x) << 4));
  };
  // the first and the second channel of word w of two pieces
  auto word = [](const uint4& v, int w) { return w == 0 ? v.x : w == 1 ? v.y : w == 2 ? v.z : v.w; };
  auto even = [&](const uint4& a, const uint4& b, int w) { return pair2(__uint_as_float(word(a, w) << 16), __uint_as_float(word(b, w) << 16)); };
  auto odd = [&](const uint4& a, const uint4& b, int w) {
    return pair2(__uint_as_float(word(a, w) & 0xffff0000u), __uint_as_float(word(b, w) & 0xffff0000u));
  };
  if constexpr (KB == 1) {
    // the row stays unpacked in registers: pieces 2 h and 2 h + 1 side by side, gamma and beta too
    uint4 raw[8];
    load(raw, 0);
    uint64_t v[4][8], t[4];
    auto fold = [&]() {
      const float2 f = split2(add2(add2(t[0], t[2]), add2(t[1], t[3])));
      return f.x + f.y;
    };
#pragma unroll
    for (int h = 0; h < 4; ++h) {
      t[h] = pair2(0.f, 0.f);
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        v[h][j] = j & 1 ? odd(raw[2 * h], raw[2 * h + 1], j >> 1) : even(raw[2 * h], raw[2 * h + 1], j >> 1);
        t[h] = add2(t[h], v[h][j]);
      }
    }
    const float mean = fold() * (1.f / C);
    const uint64_t m2 = pair2(-mean, -mean);
#pragma unroll
    for (int h = 0; h < 4; ++h) {
      t[h] = pair2(0.f, 0.f);
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        v[h][j] = add2(v[h][j], m2);
        t[h] = fma2(v[h][j], v[h][j], t[h]);
      }
    }
    const float rstd = rsqrtf(fold() * (1.f / C) + eps);
    const uint64_t r2 = pair2(rstd, rstd);
#pragma unroll
    for (int h = 0; h < 4; ++h) {
      uint32_t lo[4], hi[4];
#pragma unroll
      for (int w = 0; w < 4; ++w) {
        const ulonglong2 g = *reinterpret_cast<const ulonglong2*>(gamma + h * 16 + 4 * w), b = *reinterpret_cast<const ulonglong2*>(beta + h * 16 + 4 * w);
        const float2 e = split2(fma2(mul2(v[h][2 * w], r2), g.x, b.x));
        const float2 o = split2(fma2(mul2(v[h][2 * w + 1], r2), g.y, b.y));
        lo[w] = lg_pack2(e.x, o.x);
        hi[w] = lg_pack2(e.y, o.y);
      }
      *reinterpret_cast<uint4*>(p + (((2 * h) ^ x) << 4)) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
      *reinterpret_cast<uint4*>(p + (((2 * h + 1) ^ x) << 4)) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
    }
  } else {
    // Four chains at a time: a pair of neighbouring pieces (2 i and 2 i + 1) of each of four blocks, or of two blocks and then also the pair
    // half a block on.  Pairs half a block apart are added first
    auto total = [&](auto&& add) {
      uint64_t s[4], half, t;
      auto combine = [&](int n) {
        const uint64_t u = add2(KB == 4 ? add2(s[0], s[2]) : add2(s[0], s[1]), KB == 4 ? add2(s[1], s[3]) : add2(s[2], s[3]));
        if (KB == 4) {
          const uint64_t w = add2(half, u);
          if (n & 1) t = n > 1 ? add2(t, w) : w;
          half = u;
        } else {
          t = n ? add2(t, u) : u;
        }
      };
      half = t = 0;
#pragma unroll 1
      for (int n = 0; n < KB; ++n) {
        uint4 ra[4], rb[4];
        const int i = KB == 4 ? (n >> 1) + 2 * (n & 1) : n;
        const int oa = ((2 * i) ^ x) << 4, ob = oa ^ 16;
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          const int at = KB == 4 ? c * 16384 : (c & 1) * 16384, off = KB == 4 ? 0 : (c >> 1) * 64;       // 64: four pieces on
          ra[c] = *reinterpret_cast<const uint4*>(p + at + (oa ^ off));
          rb[c] = *reinterpret_cast<const uint4*>(p + at + (ob ^ off));
        }
        if (n) combine(n - 1);          // here, with the loads under way, and not at the end of the pass, where it would wait for the sums
#pragma unroll
        for (int c = 0; c < 4; ++c) s[c] = pair2(0.f, 0.f);
#pragma unroll
        for (int w = 0; w < 4; ++w) {
#pragma unroll
          for (int c = 0; c < 4; ++c) s[c] = add(s[c], even(ra[c], rb[c], w));
#pragma unroll
          for (int c = 0; c < 4; ++c) s[c] = add(s[c], odd(ra[c], rb[c], w));
        }
      }
      combine(KB - 1);
      asm volatile("" ::: "memory");
      const float2 f = split2(t);
      return f.x + f.y;
    };
    const float mean = total([](uint64_t s, uint64_t v) { return add2(s, v); }) * (1.f / C);
    const uint64_t m2 = pair2(-mean, -mean);
    const float var = total([&](uint64_t s, uint64_t v) {
      const uint64_t d = add2(v, m2);
      return fma2(d, d, s);
    });
    const float rstd = rsqrtf(var * (1.f / C) + eps);
    const uint64_t r2 = pair2(rstd, rstd);
#pragma unroll 1
    for (int kb = 0; kb < KB; ++kb) {
      uint4 ra[8];
      load(ra, kb);
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        const ulonglong2* g = reinterpret_cast<const ulonglong2*>(gamma + kb * 64 + u * 8);       // the same in every lane
        const ulonglong2* b = reinterpret_cast<const ulonglong2*>(beta + kb * 64 + u * 8);
        const ulonglong2 g0 = g[0], g1 = g[1], b0 = b[0], b1 = b[1];
        uint4 o;
        o.x = lg_pack2v(fma2(mul2(add2(lg_bf2(ra[u].x), m2), r2), g0.x, b0.x));
        o.y = lg_pack2v(fma2(mul2(add2(lg_bf2(ra[u].y), m2), r2), g0.y, b0.y));
        o.z = lg_pack2v(fma2(mul2(add2(lg_bf2(ra[u].z), m2), r2), g1.x, b1.x));
        o.w = lg_pack2v(fma2(mul2(add2(lg_bf2(ra[u].w), m2), r2), g1.y, b1.y));
        *reinterpret_cast<uint4*>(p + kb * 16384 + ((u ^ x) << 4)) = o;
      }
    }
  }
}

// Channels-first tile [kb][2 chunks of 64 rows][64 channels][64 rows], in place: thread t holds rows 2 (t % 64) and the next for
// the 64 channels of block t / 64.  Sums in the order of ln_fwd_transposed128_kernel, so that both give the same bits: four
// channels, four such quads, then the eight groups of 16 channels one by one; the two threads of a pair of rows exchange theirs through
// `part` ([2][5][64] float2: the first four groups added up, the other four each).
__device__ __forceinline__ void lg_norm_columns(uint8_t* tile, int t, float2* part, const float* gamma, const float* beta, float eps) {
  const int pr = t & 63, kb = t >> 6;
  uint8_t* p = tile + kb * 16384 + (pr >> 5) * 8192 + ((pr & 3) << 2);
  const int u = (pr & 31) >> 2;
  auto sweep = [&](auto&& each) {         // 16 channels at a time
#pragma unroll 1
    for (int k0 = 0; k0 < 64; k0 += 16) {
      uint32_t raw[16];
#pragma unroll
      for (int k = 0; k < 16; ++k) raw[k] = *reinterpret_cast<const uint32_t*>(p + (k0 + k) * 128 + ((u ^ (k & 7)) << 4));
      each(k0, raw);
    }
  };
  auto total = [&](float2* at, auto&& quad) {
    uint64_t first = pair2(0.f, 0.f);
    sweep([&](int k0, const uint32_t (&raw)[16]) {
      const uint64_t g = add2(add2(quad(raw), quad(raw + 4)), add2(quad(raw + 8), quad(raw + 12)));
      if (kb == 0) first = add2(first, g);
      else at[(1 + (k0 >> 4)) * 64 + pr] = split2(g);
    });
    if (kb == 0) at[pr] = split2(first);
    asm volatile("bar.sync 2, 128;" ::: "memory");
    float2 sum = at[pr];
#pragma unroll
    for (int i = 1; i < 5; ++i) {
      const float2 g = at[i * 64 + pr];
      sum.x += g.x;
      sum.y += g.y;
    }
    return sum;
  };
  const float2 ms = total(part, [&](const uint32_t* r) { return add2(add2(lg_bf2(r[0]), lg_bf2(r[1])), add2(lg_bf2(r[2]), lg_bf2(r[3]))); });
  const uint64_t m2 = pair2(-ms.x * (1.f / 128), -ms.y * (1.f / 128));
  const float2 qs = total(part + 320, [&](const uint32_t* r) {
    uint64_t q = pair2(0.f, 0.f);
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const uint64_t d = add2(lg_bf2(r[k]), m2);
      q = fma2(d, d, q);
    }
    return q;
  });
  const uint64_t r2 = pair2(rsqrtf(qs.x * (1.f / 128) + eps), rsqrtf(qs.y * (1.f / 128) + eps));
  sweep([&](int k0, const uint32_t (&raw)[16]) {
#pragma unroll
    for (int k = 0; k < 16; k += 4) {
      const float4 g = *reinterpret_cast<const float4*>(gamma + kb * 64 + k0 + k), b = *reinterpret_cast<const float4*>(beta + kb * 64 + k0 + k);
      const float gv[4] = {g.x, g.y, g.z, g.w}, bv[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const uint64_t y = fma2(mul2(add2(lg_bf2(raw[k + i]), m2), r2), pair2(gv[i], gv[i]), pair2(bv[i], bv[i]));
        *reinterpret_cast<uint32_t*>(p + (k0 + k + i) * 128 + ((u ^ ((k + i) & 7)) << 4)) = lg_pack2v(y);
      }
    }
  });
}

// Whether `ok` holds in all four LayerNorm warps.
__device__ __forceinline__ bool lg_norm_warps_agree(bool ok) {
  uint32_t all;
  asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.u32 p, %1, 0;\n\tbarrier.cta.red.and.pred q, 2, 128, p;\n\tselp.u32 %0, 1, 0, q;\n\t}" : "=r"(all) : "r"((uint32_t)ok) : "memory");
  return all != 0;
}

__device__ __forceinline__ void lg_store_tile(const CUtensorMap* map, uint32_t smem, int x, int y, int z) {
  asm volatile("cp.async.bulk.tensor.3d.global.shared::cta.bulk_group [%0, {%2, %3, %4}], [%1];" ::"l"(map), "r"(smem), "r"(x), "r"(y), "r"(z) : "memory");
  asm volatile("cp.async.bulk.commit_group;" ::: "memory");
}

template <int C, int MODE, bool CF, int TEAMS, bool NARROW>
__global__ void __launch_bounds__((6 + LG_EPI * TEAMS) * 32, 1) ln_gemm_kernel(const __grid_constant__ LgMaps maps, const __grid_constant__ LgArgs a) {
  pdl_launch_dependents();
  using Cfg = LgCfg<C, MODE, TEAMS, NARROW>;
  static_assert(TEAMS == (C == 256 || CF ? 1 : 2), "one team at 256 channels and for channels-first rows");
  constexpr int KB = Cfg::KB, RING = Cfg::RING, NACC = Cfg::NACC, NB2 = Cfg::NB2, NA = Cfg::NA;
  // chains run a chunk ahead across tiles where there are two tiles of rows; with one that would wait for rows that wait for this tile
  constexpr bool AHEAD = MODE != LN_PROJECT && NA == 2;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* sm = smem_raw + (base - smem_u32(smem_raw));
  float* gamma = reinterpret_cast<float*>(sm + Cfg::VEC);
  float* beta = gamma + C;
  float* bias1 = beta + C;                  // [LG_MAX_N]
  float* bias2 = bias1 + LG_MAX_N;          // [256]
  float2* part = reinterpret_cast<float2*>(bias2 + 256);
  const uint32_t b0 = base + Cfg::BARS;
  const uint32_t x_full = b0, a_full = b0 + 16, a_empty = b0 + 32, acc_full = b0 + 48, acc_free = b0 + 80, h_full = b0 + 112;
  const uint32_t acc2_full = b0 + 144, acc2_empty = b0 + 152, w_full = b0 + 160, w_empty = b0 + 216, ld_bar = b0 + 272;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(sm + Cfg::BARS + 400);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    for (int i = 0; i < 2; ++i) {
      mbar_init(x_full + 8 * i, 1);
      mbar_init(a_full + 8 * i, 4);
      mbar_init(a_empty + 8 * i, 1);
    }
    for (int i = 0; i < NACC; ++i) {
      mbar_init(acc_full + 8 * i, 1);
      mbar_init(acc_free + 8 * i, MODE == LN_PROJECT ? LG_EPI : 1);
      mbar_init(h_full + 8 * i, LG_EPI);
    }
    mbar_init(acc2_full, 1);
    mbar_init(acc2_empty, LG_EPI);
    for (int i = 0; i < RING; ++i) {
      mbar_init(w_full + 8 * i, 1);
      mbar_init(w_empty + 8 * i, 1);
    }
    for (int i = 0; i < Cfg::EPI; ++i) mbar_init(ld_bar + 8 * i, 1);
    *abort_flag = 0;
    fence_mbar_init();
    prefetch_tmap(&maps.x);
    prefetch_tmap(&maps.w[0]);
  }
  if (warp == 0) {
    __syncwarp();
    tmem_alloc(smem_u32(tmem_slot), 512);
    tmem_relinquish();
  }
  pdl_wait();
  // gamma, beta and all biases as fp32; read back as broadcasts
  for (int i = threadIdx.x; i < C; i += Cfg::THREADS) {
    const int at = C == 64 ? (i & 48) + (i & 7) * 2 + ((i >> 3) & 1) : i;       // for lg_norm_row<64>: the same channel of two pieces side by side
    gamma[at] = __bfloat162float(a.gamma[i]);
    beta[at] = __bfloat162float(a.beta[i]);
  }
  if (MODE != LN_PROJECT) {
    for (int i = threadIdx.x; i < ((a.hidden + 127) & ~127); i += Cfg::THREADS) bias1[i] = (a.b1 && i < a.hidden) ? __bfloat162float(a.b1[i]) : 0.f;
    for (int i = threadIdx.x; i < C; i += Cfg::THREADS) bias2[i] = a.b2 ? __bfloat162float(a.b2[i]) : 0.f;
  } else {
    int off = 0;
    for (int s = 0; s < a.nseg; ++s) {
      const int n = a.seg[s].n, nc = (n + 127) & ~127;
      for (int i = threadIdx.x; i < nc; i += Cfg::THREADS) bias1[off + i] = (a.seg_bias[s] && i < n) ? __bfloat162float(a.seg_bias[s][i]) : 0.f;
      off += nc;
    }
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = __shfl_sync(0xffffffffu, *tmem_slot, 0);
  const int chunks = MODE == LN_PROJECT ? a.chunks : (a.hidden + 127) / 128;

  if (warp < 4) {
    // ---------------- LayerNorm ----------------
    bool ok = true;
    uint32_t t = 0;
#pragma unroll 1
    for (int tile = blockIdx.x; tile < a.num_tiles; tile += gridDim.x, ++t) {
      const uint32_t s = t % NA;
      ok = __all_sync(0xffffffffu, mbar_wait(x_full + 8 * s, (t / NA) & 1));
      // lg_norm_columns has barriers across the four warps: all of them take the tile, or none does and each leaves here
      if (CF) ok = lg_norm_warps_agree(ok);
      if (!ok) break;
      uint8_t* At = sm + Cfg::A0 + s * Cfg::A_BYTES;
      if (CF) lg_norm_columns(At, threadIdx.x, part, gamma, beta, a.eps);
      else lg_norm_row<C>(At, threadIdx.x, gamma, beta, a.eps);
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) mbar_arrive(a_full + 8 * s);
    }
    if (!ok && lane == 0) {
      if (*abort_flag == 0) report(ST_TIMEOUT_TMA, 50);
      *abort_flag = 1;
    }
  } else if (warp == Cfg::TMA) {
    // ---------------- TMA: rows and weights ----------------
    if (lane == 0) {
      bool ok = true;
      uint32_t wi = 0, t = 0;
      auto load_x = [&](int tile, uint32_t n) {
        const uint32_t s = n % NA, dst = base + Cfg::A0 + s * Cfg::A_BYTES, bar = x_full + 8 * s;
        if (!mbar_wait(a_empty + 8 * s, ((n / NA) & 1) ^ 1)) {
          ok = false;
          return;
        }
        const int m0 = (tile % a.tiles_m) * 128, b = tile / a.tiles_m * a.bpt;
        mbar_expect_tx(bar, Cfg::A_BYTES);
#pragma unroll 1
        for (int kb = 0; kb < KB; ++kb) {
          if (CF) {
            tma_load_3d(dst + kb * 16384, &maps.x, bar, m0, kb * 64, b);
            tma_load_3d(dst + kb * 16384 + 8192, &maps.x, bar, m0 + 64, kb * 64, b);
          } else {
            tma_load_3d(dst + kb * 16384, &maps.x, bar, kb * 64, m0, b);
          }
        }
      };
      auto load_w = [&](const CUtensorMap* map, int x, int y, uint32_t bytes) {
        const uint32_t s = wi % RING;
        if (!ok) return;
        ok = mbar_wait(w_empty + 8 * s, ((wi / RING) & 1) ^ 1);
        if (!ok) return;
        mbar_expect_tx(w_full + 8 * s, bytes);
        tma_load_3d(base + Cfg::W0 + s * LG_BOX, map, w_full + 8 * s, x, y, 0);
        ++wi;
      };
      load_x(blockIdx.x, 0);
#pragma unroll 1
      for (int tile = blockIdx.x; tile < a.num_tiles && ok; tile += gridDim.x, ++t) {
        const bool more = tile + gridDim.x < a.num_tiles;       // with one tile of rows its place is free after the last first product
        if (MODE == LN_PROJECT) {
          int seg = 0, row = 0;
#pragma unroll 1
          for (int h = 0; h < chunks && ok; ++h) {
#pragma unroll 1
            for (int kb = 0; kb < KB; ++kb) load_w(&maps.w[seg], kb * 64, row, LG_BOX);
            row += 128;
            if (row >= a.seg[seg].n) {
              ++seg;
              row = 0;
            }
            if (h == (NA == 1 ? chunks - 1 : 0) && more) load_x(tile + gridDim.x, t + 1);
          }
        } else {
          // the boxes in the order in which the issuer takes them
          if (AHEAD && more) load_x(tile + gridDim.x, t + 1);
#pragma unroll 1
          for (int h = AHEAD && t > 0 ? 1 : 0; h <= chunks && ok; ++h) {
#pragma unroll 1
            for (int kb = 0; kb < KB && (h < chunks || (AHEAD && more)); ++kb) load_w(&maps.w[0], kb * 64, h < chunks ? h * 128 : 0, LG_BOX);
            if (h > 0) {
#pragma unroll 1
              for (int kk = 0; kk < 2; ++kk)
#pragma unroll 1
                for (int n = 0; n < C; n += NB2) load_w(&maps.w[1], (h - 1) * 128 + kk * 64, n, NB2 * 128);
            }
            if (!AHEAD && h == chunks && more) load_x(tile + gridDim.x, t + 1);
          }
        }
      }
      if (!ok) {
        if (*abort_flag == 0) report(ST_TIMEOUT_MMA, 51);
        *abort_flag = 1;
      }
    }
    __syncwarp();
  } else if (warp == Cfg::MMA) {
    // ---------------- MMA issue (the whole warp, see umma_bf16_by) ----------------
    constexpr uint32_t idesc1 = make_idesc_bf16(128, 128, CF ? 1 : 0, 0), idesc2 = make_idesc_bf16(128, NB2, 0, 0);
    const uint32_t lead = elect_one();
    // descriptors of the first row tile and ring slot; the address field counts 16 bytes, so slots and steps are additions
    const uint64_t ad0 = CF ? make_smem_desc(base + Cfg::A0, 8192, 1024) : make_smem_desc(base + Cfg::A0, 16, 1024);
    const uint64_t wd0 = make_smem_desc(base + Cfg::W0, 16, 1024);
    bool ok = true;
    uint32_t ws = 0, wphase = 0, t = 0, c1 = 0, c2 = 0;          // ring slot and parity, tiles, chunks of the first and second products so far
    auto await = [&](uint32_t bar, uint32_t parity, int code) {
      if (!ok) return;
      ok = __all_sync(0xffffffffu, mbar_wait(bar, parity));
      if (!ok && lead && *abort_flag == 0) report(code, 52);
    };
    auto box_done = [&]() {
      umma_commit_by(lead, w_empty + 8 * ws);
      if (++ws == RING) {
        ws = 0;
        wphase ^= 1;
      }
    };
    auto first = [&](uint64_t ad) {                    // chunk of the first product
      const uint32_t b = c1 % NACC;
      await(acc_free + 8 * b, ((c1 / NACC) & 1) ^ 1, ST_TIMEOUT_EPI);
#pragma unroll 1
      for (int kb = 0; kb < KB && ok; ++kb) {
        await(w_full + 8 * ws, wphase, ST_TIMEOUT_TMA);
        if (!ok) break;
        tc_fence_after();
        const uint64_t wd = wd0 + ws * (LG_BOX >> 4);
#pragma unroll
        for (int k = 0; k < 4; ++k)
          umma_bf16_by(lead, tmem + b * 128, ad + kb * (16384 >> 4) + k * ((CF ? 2048 : 32) >> 4), wd + k * (32 >> 4), idesc1, (kb > 0 || k > 0) ? 1u : 0u);
        box_done();
      }
      if (ok) umma_commit_by(lead, acc_full + 8 * b);
      ++c1;
    };
    auto second = [&](int h) {                         // chunk of the second product
      const uint32_t b = c2 % NACC;
      await(h_full + 8 * b, (c2 / NACC) & 1, ST_TIMEOUT_EPI);
      if (h == 0) await(acc2_empty, (t & 1) ^ 1, ST_TIMEOUT_EPI);
#pragma unroll 1
      for (int kk = 0; kk < 2; ++kk)
#pragma unroll 1
        for (int n = 0; n < C && ok; n += NB2) {
          await(w_full + 8 * ws, wphase, ST_TIMEOUT_TMA);
          if (!ok) break;
          tc_fence_after();
          const uint64_t wd = wd0 + ws * (LG_BOX >> 4);
#pragma unroll
          for (int k = 0; k < 4; ++k)                  // columns 0-31 and 64-95 of the accumulator hold the two halves
            umma_bf16_ts_by(lead, tmem + Cfg::ACC2 + n, tmem + b * 128 + kk * 64 + k * 8, wd + k * (32 >> 4), idesc2, (h > 0 || kk > 0 || k > 0) ? 1u : 0u);
          box_done();
        }
      if (!ok) return;
      umma_commit_by(lead, acc_free + 8 * b);
      if (h + 1 == chunks) umma_commit_by(lead, acc2_full);
      ++c2;
    };
    if constexpr (AHEAD) {
      // The next chunk's first product goes out before this one's second, which waits for the epilogue between them; the next tile's too
      auto first_of = [&](uint32_t n, int h) {           // chunk h of the n-th tile
        const uint32_t s = n % NA;
        if (h == 0) {
          await(a_full + 8 * s, (n / NA) & 1, ST_TIMEOUT_EPI);
          if (!ok) return;
          tc_fence_after();
        }
        first(ad0 + s * (Cfg::A_BYTES >> 4));
        if (h + 1 == chunks && ok) umma_commit_by(lead, a_empty + 8 * s);        // the last product that reads the rows is in
      };
      first_of(0, 0);
#pragma unroll 1
      for (int tile = blockIdx.x; tile < a.num_tiles && ok; tile += gridDim.x, ++t)
#pragma unroll 1
        for (int h = 0; h < chunks && ok; ++h) {
          if (h + 1 < chunks) first_of(t, h + 1);
          else if (tile + gridDim.x < a.num_tiles) first_of(t + 1, 0);
          if (ok) second(h);
        }
    } else {
#pragma unroll 1
      for (int tile = blockIdx.x; tile < a.num_tiles && ok; tile += gridDim.x, ++t) {
        const uint32_t s = t % NA;
        await(a_full + 8 * s, (t / NA) & 1, ST_TIMEOUT_EPI);
        if (!ok) break;
        tc_fence_after();
#pragma unroll 1
        for (int h = 0; h <= chunks && ok; ++h) {
          if (h < chunks) first(ad0 + s * (Cfg::A_BYTES >> 4));
          if (h + 1 == chunks && ok) umma_commit_by(lead, a_empty + 8 * s);        // the last product that reads the rows is in
          if (MODE != LN_PROJECT && h > 0 && ok) second(h - 1);
        }
      }
    }
    if (!ok && lead) *abort_flag = 1;
    __syncwarp();
  } else {
    // ---------------- epilogues (from warp 4 on) ----------------
    const int quad = warp & 3, half = ((warp - 4) >> 2) & 1, team = (warp - 4) >> 3;
    uint8_t* stg = sm + Cfg::STG + (warp - 4) * (Cfg::TILES * 4096);
    const uint32_t stg_u = smem_u32(stg), my_ld = ld_bar + 8 * (warp - 4);
    const uint32_t lane_base = tmem + ((uint32_t)(quad * 32) << 16);
    uint32_t c1 = 0, t = 0, ld_phase = 0;
    uint32_t ob = 0;                            // projections: byte offset of the staging tile of the next store
    constexpr uint32_t OTHER = Cfg::TILES == 2 ? 4096 : 0;
    bool ok = true;
    auto wait = [&](uint32_t bar, uint32_t parity, int code) -> bool {
      ok = __all_sync(0xffffffffu, mbar_wait(bar, parity));
      if (!ok && lane == 0 && *abort_flag == 0) report(code, 53);
      return ok;
    };
    // 64 columns of this thread's row of an accumulator, bias added
    auto read64 = [&](uint32_t col, const float* bias, float (&v)[64]) {
      tmem_ld_32x32(lane_base + col, v);
      tmem_ld_32x32(lane_base + col + 32, v + 32);
      tmem_ld_wait();
      const float4* bp = reinterpret_cast<const float4*>(bias);
#pragma unroll
      for (int q = 0; q < 16; ++q) {
        const float4 f = bp[q];
        v[4 * q] += f.x;
        v[4 * q + 1] += f.y;
        v[4 * q + 2] += f.z;
        v[4 * q + 3] += f.w;
      }
    };
    auto mul_tile = [&](const uint8_t* buf, float (&v)[64]) {
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        float m[8];
        lg_unpack(*reinterpret_cast<const uint4*>(buf + lane * 128 + ((u ^ (lane & 7)) << 4)), m);
#pragma unroll
        for (int j = 0; j < 8; ++j) v[u * 8 + j] *= m[j];
      }
    };
    // the tile that leaves, with the residual tile in the same place added where there is one
    auto write_tile = [&](uint8_t* buf, float (&v)[64], bool resid) {
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        uint4* at = reinterpret_cast<uint4*>(buf + lane * 128 + ((u ^ (lane & 7)) << 4));
        if (resid) {
          float m[8];
          lg_unpack(*at, m);
#pragma unroll
          for (int j = 0; j < 8; ++j) v[u * 8 + j] += m[j];
        }
        *at = lg_pack(v + u * 8);
      }
      fence_proxy_async_smem();
      __syncwarp();
    };
#pragma unroll 1
    for (int tile = blockIdx.x; tile < a.num_tiles && ok; tile += gridDim.x, ++t) {
      int row0 = (tile % a.tiles_m) * 128 + quad * 32, batch = tile / a.tiles_m;
      if (a.bpt > 1) {
        batch = tile * a.bpt + row0 / a.rows;
        row0 %= a.rows;
      }
      const bool valid = row0 < a.rows && batch < a.batch;
      if constexpr (MODE != LN_PROJECT && TEAMS == 2) {
        // One team for the hidden activation, one for the result: the result of a tile leaves while the next one's hidden activation is
        // made.  32 columns at a time, see LgCfg
        auto read32 = [&](uint32_t col, const float* bias, float (&v)[32]) {
          tmem_ld_32x32(lane_base + col, v);
          const float4* bp = reinterpret_cast<const float4*>(bias);
          tmem_ld_wait();
#pragma unroll
          for (int q = 0; q < 8; ++q) {
            const float4 f = bp[q];
            v[4 * q] += f.x;
            v[4 * q + 1] += f.y;
            v[4 * q + 2] += f.z;
            v[4 * q + 3] += f.w;
          }
        };
        if (team == 0) {
          auto fetch_mul = [&](int h) {
            if (lane == 0) {
              mbar_expect_tx(my_ld, 4096);
              tma_load_3d(stg_u, &maps.mul, my_ld, h * 128 + half * 64, row0, batch);
            }
          };
          if (MODE == LN_GATE_CHAIN && !a.mul_f32) fetch_mul(0);
#pragma unroll 1
          for (int h = 0; h < chunks; ++h, ++c1) {
            const uint32_t b = c1 % NACC;
            if (!wait(acc_full + 8 * b, (c1 / NACC) & 1, ST_TIMEOUT_MMA)) break;
            tc_fence_after();
            if (MODE == LN_GATE_CHAIN && !a.mul_f32) {
              if (!wait(my_ld, ld_phase, ST_TIMEOUT_TMA)) break;
              ld_phase ^= 1;
            }
#pragma unroll 1
            for (int e = 0; e < 2; ++e) {
              float v[32];
              const int col = h * 128 + half * 64 + e * 32;
              read32(b * 128 + half * 64 + e * 32, bias1 + col, v);
              if (MODE == LN_RELU_CHAIN) {
#pragma unroll
                for (int j = 0; j < 32; ++j) v[j] = fmaxf(v[j], 0.f);
              } else {
#pragma unroll
                for (int j = 0; j < 32; ++j) v[j] = sigmoidf_(v[j]);
                if (a.mul_f32) {
                  // one row of 32-bit factors for all rows of a column: a few ten kilobytes that stay in L1
                  const float4* m = reinterpret_cast<const float4*>(a.mul_f32 + ((long long)batch * a.rows + row0 + lane) % a.mul_mod * a.hidden + col);
#pragma unroll
                  for (int q = 0; q < 8; ++q) {
                    const float4 f = col + 4 * q < a.hidden ? m[q] : make_float4(0.f, 0.f, 0.f, 0.f);
                    v[4 * q] *= f.x;
                    v[4 * q + 1] *= f.y;
                    v[4 * q + 2] *= f.z;
                    v[4 * q + 3] *= f.w;
                  }
                } else {
#pragma unroll
                  for (int u = 0; u < 4; ++u) {
                    float m[8];
                    lg_unpack(*reinterpret_cast<const uint4*>(stg + lane * 128 + (((e * 4 + u) ^ (lane & 7)) << 4)), m);
#pragma unroll
                    for (int j = 0; j < 8; ++j) v[u * 8 + j] *= m[j];
                  }
                }
              }
              uint32_t p[16];                                   // bf16 pairs, over columns that have been read
#pragma unroll
              for (int j = 0; j < 16; ++j) p[j] = lg_pack2(v[2 * j], v[2 * j + 1]);
              tmem_st_32x16(lane_base + b * 128 + half * 64 + e * 16, p);
            }
            tmem_st_wait();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(h_full + 8 * b);
            if (MODE == LN_GATE_CHAIN && !a.mul_f32 && h + 1 < chunks) fetch_mul(h + 1);
          }
        } else {
          bool waited = false;
#pragma unroll 1
          for (int c = half; c < C / 64; c += 2) {
            if (lane == 0) {
              asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
              mbar_expect_tx(my_ld, 4096);
              tma_load_3d(stg_u, &maps.resid, my_ld, c * 64, row0, batch);
            }
            __syncwarp();
            if (!waited && !wait(acc2_full, t & 1, ST_TIMEOUT_MMA)) break;
            waited = true;
            tc_fence_after();
            if (!wait(my_ld, ld_phase, ST_TIMEOUT_TMA)) break;
            ld_phase ^= 1;
#pragma unroll 1
            for (int e = 0; e < 2; ++e) {
              float v[32];
              read32(Cfg::ACC2 + c * 64 + e * 32, bias2 + c * 64 + e * 32, v);
#pragma unroll
              for (int u = 0; u < 4; ++u) {
                uint4* at = reinterpret_cast<uint4*>(stg + lane * 128 + (((e * 4 + u) ^ (lane & 7)) << 4));
                float m[8];
                lg_unpack(*at, m);
#pragma unroll
                for (int j = 0; j < 8; ++j) v[u * 8 + j] += m[j];
                *at = lg_pack(v + u * 8);
              }
            }
            fence_proxy_async_smem();
            __syncwarp();
            if (lane == 0 && valid) lg_store_tile(&maps.out[0], stg_u, c * 64, row0, batch);
          }
          if (!ok) break;
          if (!waited && !wait(acc2_full, t & 1, ST_TIMEOUT_MMA)) break;
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(acc2_empty);
        }
      } else if constexpr (MODE != LN_PROJECT) {
        static_assert(Cfg::TILES == 1, "mul tiles, residual and result take turns in one staging tile");
        auto fetch_mul = [&](int h) {
          if (lane == 0) {
            asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
            mbar_expect_tx(my_ld, 4096);
            tma_load_3d(stg_u, &maps.mul, my_ld, h * 128 + half * 64, row0, batch);
          }
        };
        if (MODE == LN_GATE_CHAIN && !a.mul_f32) fetch_mul(0);
#pragma unroll 1
        for (int h = 0; h < chunks; ++h, ++c1) {
          const uint32_t b = c1 % NACC;
          if (!wait(acc_full + 8 * b, (c1 / NACC) & 1, ST_TIMEOUT_MMA)) break;
          tc_fence_after();
          float v[64];
          read64(b * 128 + half * 64, bias1 + h * 128 + half * 64, v);
          if (MODE == LN_RELU_CHAIN) {
#pragma unroll
            for (int j = 0; j < 64; ++j) v[j] = fmaxf(v[j], 0.f);
          } else {
#pragma unroll
            for (int j = 0; j < 64; ++j) v[j] = sigmoidf_(v[j]);
            if (a.mul_f32) {
              // one row of 32-bit factors for all rows of a column: a few ten kilobytes that stay in L1
              const int col = h * 128 + half * 64;
              const float4* m = reinterpret_cast<const float4*>(a.mul_f32 + ((long long)batch * a.rows + row0 + lane) % a.mul_mod * a.hidden + col);
#pragma unroll
              for (int q = 0; q < 16; ++q) {
                const float4 f = col + 4 * q < a.hidden ? m[q] : make_float4(0.f, 0.f, 0.f, 0.f);
                v[4 * q] *= f.x;
                v[4 * q + 1] *= f.y;
                v[4 * q + 2] *= f.z;
                v[4 * q + 3] *= f.w;
              }
            } else {
              if (!wait(my_ld, ld_phase, ST_TIMEOUT_TMA)) break;
              ld_phase ^= 1;
              mul_tile(stg, v);
              __syncwarp();
              if (h + 1 < chunks) fetch_mul(h + 1);
            }
          }
          float p[32];                                          // bf16 pairs
#pragma unroll
          for (int j = 0; j < 32; ++j) p[j] = __uint_as_float(lg_pack2(v[2 * j], v[2 * j + 1]));
          tmem_st_32x32(lane_base + b * 128 + half * 64, p);
          tmem_st_wait();
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(h_full + 8 * b);
        }
        if (!ok) break;
        bool waited = false;
#pragma unroll 1
        for (int c = half; c < C / 64; c += 2) {
          if (lane == 0) {
            asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
            mbar_expect_tx(my_ld, 4096);
            tma_load_3d(stg_u, &maps.resid, my_ld, c * 64, row0, batch);
          }
          __syncwarp();
          if (!waited && !wait(acc2_full, t & 1, ST_TIMEOUT_MMA)) break;
          waited = true;
          tc_fence_after();
          float v[64];
          read64(Cfg::ACC2 + c * 64, bias2 + c * 64, v);
          if (!wait(my_ld, ld_phase, ST_TIMEOUT_TMA)) break;
          ld_phase ^= 1;
          write_tile(stg, v, true);
          if (lane == 0 && valid) lg_store_tile(&maps.out[0], stg_u, c * 64, row0, batch);
        }
        if (!ok) break;
        if (!waited && !wait(acc2_full, t & 1, ST_TIMEOUT_MMA)) break;
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(acc2_empty);
      } else {
        const int row = row0 + lane;
        float rs = 1.f;
        if (a.rowscale && valid && row < a.rows) {
          const long long i = (long long)batch * a.rows + row;
          rs = a.rs_bf16 ? __bfloat162float(reinterpret_cast<const bf16*>(a.rowscale)[i]) : reinterpret_cast<const float*>(a.rowscale)[i];
        }
        int seg = 0, col = 0;                                   // segment and first column of the chunk
#pragma unroll 1
        for (int h = 0; h < chunks; ++h, ++c1) {
          const LgSeg sg = a.seg[seg];
          const int mycol = col + half * 64, b = c1 % NACC;
          auto next = [&]() {
            col += 128;
            if (col >= sg.n) {
              ++seg;
              col = 0;
            }
          };
          if (TEAMS == 2 && (c1 & 1) != team) {                 // the other team's
            next();
            continue;
          }
          const bool work = mycol < sg.n && valid;
          uint8_t* obuf = stg + ob;
          const bool fused = CF && a.has_mul != 0 && seg == 0;  // mul and residual tiles (two staging tiles; first segment)
          // The tiles alternate by the stores that this warp has issued, not by chunks: with all but the newest store done reading,
          // the other tile is free.  Chunks without a store (pair bias, columns or rows past the end) would break the alternation
          if (work && sg.kind != LN_PAIR_BIAS && lane == 0) {
            if (fused || Cfg::TILES == 1) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
            else asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory");
            if (fused) {
              mbar_expect_tx(my_ld, 8192);
              tma_load_3d(stg_u + ob, &maps.resid, my_ld, mycol, row0, batch);
              tma_load_3d(stg_u + (ob ^ OTHER), &maps.mul, my_ld, mycol, row0, batch);
            }
          }
          __syncwarp();
          if (!wait(acc_full + 8 * b, (c1 / NACC) & 1, ST_TIMEOUT_MMA)) break;
          tc_fence_after();
          if (work) {
            if (sg.kind == LN_PAIR_BIAS) {
              float v[32];
              tmem_ld_32x32(lane_base + b * 128 + half * 64, v);
              tmem_ld_wait();
              if (row < a.rows) {
                const long long r = (long long)batch * a.rows + row;
                bf16* dst = sg.out + (r / a.pb_n) * a.pb_i + (r % a.pb_n) * a.pb_j;
#pragma unroll
                for (int j = 0; j < 32; ++j)
                  if (j < sg.n) dst[j * a.pb_h] = __float2bfloat16(v[j]);
              }
            } else if constexpr (TEAMS == 2) {
              // 32 columns at a time, see LgCfg
#pragma unroll 1
              for (int e = 0; e < 2; ++e) {
                float v[32];
                tmem_ld_32x32(lane_base + b * 128 + half * 64 + e * 32, v);
                const float4* bp = reinterpret_cast<const float4*>(bias1 + h * 128 + half * 64 + e * 32);
                tmem_ld_wait();
#pragma unroll
                for (int q = 0; q < 8; ++q) {
                  const float4 f = bp[q];
                  v[4 * q] += f.x;
                  v[4 * q + 1] += f.y;
                  v[4 * q + 2] += f.z;
                  v[4 * q + 3] += f.w;
                }
                if (sg.kind == LN_GLU_T) {
                  bf16* o = reinterpret_cast<bf16*>(obuf) + e * 512 + lane;       // [32 columns][32 rows]
#pragma unroll
                  for (int j = 0; j < 16; ++j) o[j * 32] = __float2bfloat16(v[2 * j] * sigmoidf_(v[2 * j + 1]) * rs);
                } else {
                  if (sg.act == ACT_SIGMOID) {
#pragma unroll
                    for (int j = 0; j < 32; ++j) v[j] = sigmoidf_(v[j]);
                  }
                  if (sg.scaled) {
#pragma unroll
                    for (int j = 0; j < 32; ++j) v[j] *= rs;
                  }
#pragma unroll
                  for (int u = 0; u < 4; ++u) *reinterpret_cast<uint4*>(obuf + lane * 128 + (((e * 4 + u) ^ (lane & 7)) << 4)) = lg_pack(v + u * 8);
                }
              }
              fence_proxy_async_smem();
              __syncwarp();
              if (lane == 0) {
                if (sg.kind == LN_GLU_T) lg_store_tile(&maps.out[seg], stg_u, row0, mycol >> 1, batch);
                else lg_store_tile(&maps.out[seg], stg_u, mycol, row0, batch);
              }
            } else {
              float v[64];
              read64(b * 128 + half * 64, bias1 + h * 128 + half * 64, v);
              if (sg.kind == LN_GLU_T) {
                bf16* o = reinterpret_cast<bf16*>(obuf) + lane;       // [32 columns][32 rows]
#pragma unroll
                for (int j = 0; j < 32; ++j) o[j * 32] = __float2bfloat16(v[2 * j] * sigmoidf_(v[2 * j + 1]) * rs);
                fence_proxy_async_smem();
                __syncwarp();
                if (lane == 0) lg_store_tile(&maps.out[seg], stg_u + ob, row0, mycol >> 1, batch);
                ob ^= OTHER;
              } else {
                if (sg.act == ACT_SIGMOID) {
#pragma unroll
                  for (int j = 0; j < 64; ++j) v[j] = sigmoidf_(v[j]);
                }
                if (sg.scaled) {
#pragma unroll
                  for (int j = 0; j < 64; ++j) v[j] *= rs;
                }
                if (fused) {
                  if (!wait(my_ld, ld_phase, ST_TIMEOUT_TMA)) break;
                  ld_phase ^= 1;
                  mul_tile(stg + (ob ^ OTHER), v);
                }
                write_tile(obuf, v, fused);
                if (lane == 0) lg_store_tile(&maps.out[seg], stg_u + ob, mycol, row0, batch);
                ob ^= OTHER;
              }
            }
          }
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(acc_free + 8 * b);
          next();
        }
      }
    }
    if (lane == 0) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
    if (!ok && lane == 0) *abort_flag = 1;
    __syncwarp();
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 0) {
    tc_fence_after();
    tmem_dealloc(tmem, 512);
  }
}

static int lg_sm_count() {
  static int sm_count = 0;
  if (!sm_count) {
    int dev = 0;
    cudaGetDevice(&dev);
    if (cudaDeviceGetAttribute(&sm_count, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sm_count <= 0) sm_count = 148;
  }
  return sm_count;
}

template <int C, int MODE, bool CF, int TEAMS = 1, bool NARROW = false>
static int lg_launch(const LgMaps& maps, const LgArgs& a, cudaStream_t st) {
  using Cfg = LgCfg<C, MODE, TEAMS, NARROW>;
  auto kern = ln_gemm_kernel<C, MODE, CF, TEAMS, NARROW>;
  static SmemLimit limit;
  if (!limit.raise(kern, Cfg::SMEM)) return -30;
  const int grid = a.num_tiles < lg_sm_count() ? a.num_tiles : lg_sm_count();
  launch_k(kern, grid, Cfg::THREADS, Cfg::SMEM, st, maps, a);
  return cudaGetLastError() == cudaSuccess ? 0 : -31;
}

}  // namespace ffb

using namespace ffb;

extern "C" int ffb_ln_gemm(const LnGemmArgs* p, void* stream) {
  const LnGemmArgs& q = *p;
  if ((q.C != 64 && q.C != 128 && q.C != 256) || q.rows < 1 || q.batch < 1 || (q.channels_first && (q.C != 128 || q.mode != LN_PROJECT))) return -1;
  // short rows of many batches (a slice of columns of the pair or MSA tensor): several batches share a tile
  const int bpt = (!q.channels_first && q.batch > 1 && (q.rows == 32 || q.rows == 64)) ? (int)(128 / q.rows) : 1;
  const long long tiles_m = (q.rows + 127) / 128, tiles = tiles_m * ((q.batch + bpt - 1) / bpt);
  if (tiles > 0x7fffffffLL || q.rows > 0x7fffffffLL || q.batch > 0x7fffffffLL) return -2;
  auto bad = [](const void* ptr, long long rs, long long bs) { return !ptr || (reinterpret_cast<uintptr_t>(ptr) & 15) || (rs % 8) || (bs % 8); };
  if (bad(q.x, q.x_rstride, q.x_bstride)) return -3;
  LgMaps m;
  LgArgs a = {};
  a.rows = (int)q.rows;
  a.batch = (int)q.batch;
  a.tiles_m = (int)tiles_m;
  a.num_tiles = (int)tiles;
  a.bpt = bpt;
  a.gamma = (const bf16*)q.gamma;
  a.beta = (const bf16*)q.beta;
  a.eps = q.eps;
  a.rowscale = q.rowscale;
  a.rs_bf16 = q.rs_bf16;
  a.pb_h = q.pb_h;
  a.pb_i = q.pb_i;
  a.pb_j = q.pb_j;
  a.pb_n = q.pb_n > 0 ? q.pb_n : 1;
  // d0 is the contiguous extent
  auto map = [&](CUtensorMap* t, const void* ptr, long long d0, long long d1, long long d2, long long s1, long long s2, int b0, int b1, int swizzle, int b2 = 1) {
    return encode_tmap3_bf16(t, ptr, d0, d1, d2, s1, s2, b0, b1, swizzle, b2);
  };
  int r = q.channels_first ? map(&m.x, q.x, q.rows, q.C, q.batch, q.x_rstride, q.x_bstride, 64, 64, 128)
                           : map(&m.x, q.x, q.C, q.rows, q.batch, q.x_rstride, q.x_bstride, 64, 128 / bpt, 128, bpt);
  if (r) return 1000 + r;
  m.mul = m.resid = m.out[0] = m.out[1] = m.out[2] = m.w[0] = m.w[1] = m.w[2] = m.x;
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  if (q.mode != LN_PROJECT) {
    const bool f32 = q.mode == LN_GATE_CHAIN && q.mul_f32;
    if (f32 && (q.mul_mod < 1 || (reinterpret_cast<uintptr_t>(q.mul_f32) & 15))) return -4;
    if (q.hidden < 8 || q.hidden % 8 || q.hidden > LG_MAX_N || bad(q.w1, 0, 0) || bad(q.w2, 0, 0) || bad(q.resid, q.r_rstride, q.r_bstride) ||
        bad(q.out, q.o_rstride, q.o_bstride) || (q.mode == LN_GATE_CHAIN && !f32 && bad(q.mul, q.m_rstride, q.m_bstride)))
      return -4;
    a.hidden = q.hidden;
    a.mul_f32 = f32 ? q.mul_f32 : nullptr;
    a.mul_mod = f32 ? q.mul_mod : 1;
    a.b1 = (const bf16*)q.b1;
    a.b2 = (const bf16*)q.b2;
    r = map(&m.w[0], q.w1, q.C, q.hidden, 1, q.C, 0, 64, 128, 128);
    if (!r) r = map(&m.w[1], q.w2, q.hidden, q.C, 1, q.hidden, 0, 64, q.C < 128 ? q.C : 128, 128);
    if (!r) r = map(&m.resid, q.resid, q.C, q.rows, q.batch, q.r_rstride, q.r_bstride, 64, 32, 128);
    if (!r) r = map(&m.out[0], q.out, q.C, q.rows, q.batch, q.o_rstride, q.o_bstride, 64, 32, 128);
    if (!r && q.mode == LN_GATE_CHAIN && !f32) r = map(&m.mul, q.mul, q.hidden, q.rows, q.batch, q.m_rstride, q.m_bstride, 64, 32, 128);
    if (r) return 2000 + r;
    if (q.mode == LN_RELU_CHAIN) {
      if (q.C == 64) return lg_launch<64, LN_RELU_CHAIN, false, 2>(m, a, st);
      if (q.C == 128) return lg_launch<128, LN_RELU_CHAIN, false, 2>(m, a, st);
      return lg_launch<256, LN_RELU_CHAIN, false>(m, a, st);
    }
    if (q.C == 64) return lg_launch<64, LN_GATE_CHAIN, false, 2>(m, a, st);
    if (q.C == 128) return lg_launch<128, LN_GATE_CHAIN, false, 2>(m, a, st);
    return lg_launch<256, LN_GATE_CHAIN, false>(m, a, st);
  }
  if (q.nseg < 1 || q.nseg > 3) return -5;
  a.nseg = q.nseg;
  for (int s = 0; s < q.nseg; ++s) {
    const LnSegment& g = q.seg[s];
    if (g.n < 1 || bad(g.w, 0, 0) || !g.out) return -6;
    if (g.kind != LN_PAIR_BIAS && bad(g.out, g.o_rstride, g.o_bstride)) return -7;
    if ((g.kind == LN_PAIR_BIAS && g.n > 32) || (g.kind == LN_GLU_T && (g.n & 1))) return -8;
    a.seg[s] = {g.kind, g.act, g.scaled, g.n, (bf16*)g.out};
    a.seg_bias[s] = (const bf16*)g.bias;
    a.chunks += (g.n + 127) / 128;
    r = map(&m.w[s], g.w, q.C, g.n, 1, q.C, 0, 64, 128, 128);
    if (!r && g.kind == LN_ROWS) r = map(&m.out[s], g.out, g.n, q.rows, q.batch, g.o_rstride, g.o_bstride, 64, 32, 128);
    if (!r && g.kind == LN_GLU_T) r = map(&m.out[s], g.out, q.rows, g.n / 2, q.batch, g.o_rstride, g.o_bstride, 32, 32, 0);
    if (r) return 3000 + r;
  }
  if (a.chunks * 128 > LG_MAX_N) return -9;
  if (q.mul || q.resid) {
    if (!q.channels_first || bad(q.mul, q.m_rstride, q.m_bstride) || bad(q.resid, q.r_rstride, q.r_bstride) || q.seg[0].kind != LN_ROWS) return -10;
    a.has_mul = 1;
    r = map(&m.mul, q.mul, q.seg[0].n, q.rows, q.batch, q.m_rstride, q.m_bstride, 64, 32, 128);
    if (!r) r = map(&m.resid, q.resid, q.seg[0].n, q.rows, q.batch, q.r_rstride, q.r_bstride, 64, 32, 128);
    if (r) return 4000 + r;
  }
  if (q.channels_first) return lg_launch<128, LN_PROJECT, true>(m, a, st);
  if (q.C == 64) return lg_launch<64, LN_PROJECT, false, 2>(m, a, st);
  if (q.C == 128) return lg_launch<128, LN_PROJECT, false, 2>(m, a, st);
  // Few columns (the masked projections of the outer product mean) of many tiles: the next tile's rows matter more than four boxes of the
  // ring.  Both lines are those of the three workloads that were measured: outer product mean of 512 x 384, ten tiles a CTA, 327 -> 325 us;
  // block of 256 x 384 in chunks, five, 2159 -> 2155; block of 128 x 256, not two, 688 -> 691.  What lies between two and five tiles is not
  // known, nor are other widths; the QKV projection of 768 columns gained too at ten tiles a CTA (138 -> 117 us), in the same layout for
  // every projection of 256 channels, which was not kept.
  bool narrow = a.num_tiles >= 4 * lg_sm_count();
  for (int s = 0; s < q.nseg; ++s) narrow = narrow && q.seg[s].n <= 64;
  return narrow ? lg_launch<256, LN_PROJECT, false, 1, true>(m, a, st) : lg_launch<256, LN_PROJECT, false>(m, a, st);
}

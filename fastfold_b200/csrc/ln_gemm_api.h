// Argument block of the LayerNorm + GEMM kernels (ln_gemm.cu), filled by csrc/host/dispatch.cpp.
#pragma once

enum LnMode { LN_RELU_CHAIN = 0, LN_GATE_CHAIN = 1, LN_PROJECT = 2 };
enum LnOut { LN_ROWS = 0, LN_GLU_T = 1, LN_PAIR_BIAS = 2 };

// One projection of the normalised rows.
struct LnSegment {
  const void* w;            // bf16 [n][C] contiguous
  const void* bias;         // bf16 [n] or null
  int n;                    // weight rows (LN_GLU_T: interleaved value / gate rows, n / 2 outputs)
  int kind;                 // LnOut
  int act;                  // GemmAct (LN_ROWS)
  int scaled;               // multiply by the row factor
  void* out;                // LN_ROWS: [batch][rows][n]; LN_GLU_T: [n / 2][batch][rows]; LN_PAIR_BIAS: see pb_*
  long long o_rstride, o_bstride;   // LN_GLU_T: o_rstride is the distance between channels
};

struct LnGemmArgs {
  const void* x;            // bf16 [batch][rows][C], channels adjacent; channels_first: [C][batch][rows], rows adjacent
  int channels_first;
  int C;                    // 64, 128 or 256 (channels_first: 128)
  long long rows, batch, x_rstride, x_bstride;      // channels_first: x_rstride is the distance between channels
  const void *gamma, *beta; // bf16 [C]
  float eps;
  int mode;                 // LnMode
  // chains: out = resid + b2 + f(LN(x) w1^T + b1) w2^T, f = relu, or sigmoid(.) * mul
  const void *w1, *b1, *w2, *b2;    // [hidden][C], [hidden], [C][hidden], [C]
  int hidden;               // multiple of 8
  const float* mul_f32;     // gated chain: [mul_mod][hidden] in 32 bits instead of mul; row r (batches counted through) takes r % mul_mod
  int mul_mod;
  // mul: [batch][rows][hidden] (chain) or [batch][rows][n] (first segment); resid, out: [batch][rows][C] (chain) or of the first segment.
  // Of projections only those of channels-first rows take mul and resid, and both
  const void* mul;
  long long m_rstride, m_bstride;
  const void* resid;
  long long r_rstride, r_bstride;
  void* out;
  long long o_rstride, o_bstride;
  // projections
  int nseg;
  LnSegment seg[3];
  const void* rowscale;     // [batch * rows], fp32, or bf16 when rs_bf16
  int rs_bf16;
  // LN_PAIR_BIAS: value of row r (all batches counted through) and head h goes to out[h * pb_h + (r / pb_n) * pb_i + (r % pb_n) * pb_j]
  long long pb_h, pb_i, pb_j;
  int pb_n;
};

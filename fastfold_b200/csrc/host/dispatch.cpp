// Host side of the operator calls: argument checks, output allocation and the launch, from tensors to the C entry points
// of libffb200.so, without a trip through Python objects for every pointer, stride and flag.
//
// Why it is native: a block of the trunk is 50 - 100 launches (the training pass of its two halves 290), and with the argument
// block of a launch filled through ctypes each cost the host 20 - 35 us, so that calls of up to 256 residues were bound by the
// host: a block of 32 x 64 took 1.98 ms and takes 0.9 ms (57 launches), 128 x 256 the same, the training pass of the pair half
// at 256 residues 5.3 and 3.5 ms (198 launches).
//
// Nothing is kept between calls.  Work goes to the caller's current stream; tensors are allocated by PyTorch's allocator
// on that stream, exactly as the Python code did.
#include <torch/extension.h>

#include <ATen/cuda/CUDAContext.h>
#include <c10/cuda/CUDAGraphsC10Utils.h>
#include <c10/cuda/CUDAStream.h>

#include "gemm_api.h"
#include "ipa_api.h"
#include "ln_gemm_api.h"

extern "C" {
int ffb_gemm_bf16(const void* A, const void* B, int a_mn, int b_mn, long long lda, long long ldb, long long a_bstride, long long b_bstride,
                  int batch, int bn, GemmArgs* args, void* stream);
int ffb_layernorm_fwd(const void* x, const void* gamma, const void* beta, void* y, float* mean, float* rstd, long long rows, int C, float eps,
                      int dtype, void* stream);
int ffb_layernorm_bwd(const void* dy, const void* x, const void* gamma, const float* mean, const float* rstd, void* dx, float* part, int nblocks,
                      void* dgamma, void* dbeta, long long rows, int C, int dtype, void* stream);
int ffb_layernorm_fwd_transposed(const void* x, const void* gamma, const void* beta, void* y, float* mean, float* rstd, long long rows, int C,
                                 float eps, void* stream);
int ffb_attention_fwd(const void* q, const void* k, const void* v, long long q_bstride, long long q_rstride, long long kv_bstride,
                      long long kv_rstride, const void* bias, const void* mask, long long mask_bstride, void* out, long long out_bstride,
                      long long out_rstride, float* lse2, int B, int H, int n_q, int n_k, int D, float scale, void* stream);
int ffb_attention_infer(const void* q, const void* k, const void* v, long long q_bstride, long long q_rstride, long long kv_bstride,
                        long long kv_rstride, const void* bias, long long bias_rstride, const void* mask, long long mask_bstride, void* out,
                        long long out_bstride, long long out_rstride, int B, int H, int n_q, int n_k, int D, float scale, void* stream);
int ffb_bias_sigmoid_mul_fwd(const void* g, const void* b, const void* o, void* y, long long rows, int C, void* stream);
int ffb_bias_sigmoid_mul_bwd(const void* dy, const void* g, const void* b, const void* o, void* dg, void* dob, long long rows, int C, void* stream);
int ffb_bias_dropout_add_fwd(const void* x, const void* b, const void* m, const void* r, void* y, long long rows, int C, int div, int mod, void* stream);
int ffb_mask_mul(const void* dy, const void* m, void* dx, long long rows, int C, int div, int mod, void* stream);
int ffb_bias_ele_dropout_res_fwd(const void* ab, const void* b, const void* g, const void* m, const void* r, void* y, long long rows, int C, int div,
                                 int mod, void* stream);
int ffb_bias_ele_dropout_res_bwd(const void* dy, const void* ab, const void* b, const void* g, const void* m, void* dab, void* dg, long long rows,
                                 int C, int div, int mod, void* stream);
int ffb_glu_mask_t_fwd(const void* pre, const void* mask, void* out, int C2, long long R, void* stream);
int ffb_glu_mask_t_bwd(const void* dout, const void* pre, const void* mask, void* dpre, int C2, long long R, void* stream);
int ffb_act_bwd(const void* dy, const void* y, void* dx, long long rows, int C, int mode, void* stream);
int ffb_colsum(const void* x, float* out, long long rows, int C, void* stream);
int ffb_ln_gemm(const LnGemmArgs* p, void* stream);
int ffb_mask_norm(const void* mask, float* out, int S, int N, float eps, int is_bf16, void* stream);
int ffb_global_column(const void* x, const void* gamma, const void* beta, float eps, const void* wq, const void* kv, const void* mask, float* out,
                      long long S, long long N, float scaling, void* stream);
int ffb_ipa_prep(const void* q, const void* kv, const void* q_pts, const void* kv_pts, const float* rot, int is_quat, const float* trans, float* oq,
                 float* ok, float* ov, float* oq_pts, float* ok_pts, float* ov_pts, int N, int H, int C, int Pq, int Pv, void* stream);
int ffb_ipa_fwd_mixed(const float* q, const float* k, const float* v, const float* q_pts, const float* k_pts, const float* v_pts, const void* z,
                      const void* wb, const void* bb, const void* gamma, const void* mask, int bf, float* o, float* o_pt, float* o_pair, int N, int H,
                      int C, int Pq, int Pv, int CZ, int row0, int rows, float w_c, float w_b, float inf, void* stream);
int ffb_ipa_cat(const float* o, const float* o_pt, const float* o_pair, const float* rot, int is_quat, const float* trans, void* out, int N, int H,
                int C, int Pv, int CZ, float eps, void* stream);
}

namespace {

using at::Tensor;
using OptTensor = std::optional<Tensor>;

long long g_launches = 0;        // guarded by the interpreter lock: every entry below holds it

void* stream() { return c10::cuda::getCurrentCUDAStream().stream(); }
void* ptr(const Tensor& t) { return t.data_ptr(); }
void* ptr(const OptTensor& t) { return t ? t->data_ptr() : nullptr; }

// The checks that the Python wrappers made with ``assert`` raise the same exception type here.
void expect(bool ok, const char* what) {
  if (!ok) {
    PyErr_SetString(PyExc_AssertionError, what);
    throw pybind11::error_already_set();
  }
}

void check(int rc, const char* what) {
  ++g_launches;
  TORCH_CHECK(rc == 0, "fastfold_b200 kernel launch failed: ", what, " returned ", rc);
}

Tensor f32(at::IntArrayRef shape, const Tensor& like) { return at::empty(shape, like.options().dtype(at::kFloat)); }

// See ``gemm`` in ops/gemm.py for the meaning of the arguments.
Tensor gemm(Tensor a, Tensor b, bool a_mn, bool b_mn, double alpha, OptTensor bias, int act, bool glu, OptTensor rowscale, OptTensor mul,
            OptTensor dmask, int64_t dm_div, int64_t dm_mod, OptTensor resid, bool trans_out, OptTensor out, bool out_f32, int64_t splits,
            bool accumulate, int64_t bn, std::optional<std::vector<int64_t>> block_out) {
  expect(a.scalar_type() == at::kBFloat16 && b.scalar_type() == at::kBFloat16, "tcgen05 GEMM takes bf16 operands");
  if (a.stride(-1) != 1) a = a.contiguous();
  if (b.stride(-1) != 1) b = b.contiguous();
  const bool a3 = a.dim() == 3, b3 = b.dim() == 3, batched = a3 || b3;
  expect((a3 || a.dim() == 2) && (b3 || b.dim() == 2), "operands are matrices or batches of matrices");
  int64_t batch = 1;
  if (a3) batch = a.size(0);
  if (b3) batch = std::max(batch, b.size(0));
  const int64_t K = a_mn ? a.size(-2) : a.size(-1), M = a_mn ? a.size(-1) : a.size(-2);
  const int64_t Kb = b_mn ? b.size(-2) : b.size(-1), N = b_mn ? b.size(-1) : b.size(-2);
  expect(K == Kb, "contraction extents differ");
  const int64_t n_out = glu ? N / 2 : N;
  GemmArgs g = {};
  Tensor result;
  std::vector<int64_t> oshape;
  if (batched) oshape.push_back(batch);
  oshape.push_back(trans_out ? n_out : M);
  oshape.push_back(trans_out ? M : n_out);
  if (block_out) {
    const auto& q = *block_out;      // [shape ..., mdiv, sr2, sr1, sc1]
    const size_t n = q.size() - 4;
    expect(!out && M % 32 == 0 && n_out % 32 == 0 && q[n] > 0 && (M / 32) % q[n] == 0 && !out_f32, "block-permuted output");
    result = at::empty(at::IntArrayRef(q.data(), n), a.options());
    expect(result.numel() == M * n_out, "block-permuted output");
    g.cq = 1;
    g.cq_mdiv = (int)q[n];
    g.cq_sr2 = q[n + 1];
    g.cq_sr1 = q[n + 2];
    g.cq_sc1 = q[n + 3];
    g.ldc = 8;
    g.out_mode = OUT_BF16;
  } else {
    if (out) {
      result = *out;
      expect(result.sizes() == at::IntArrayRef(oshape), "out has another shape than the result");
      expect(result.stride(-1) == 1, "out rows must be contiguous");
    } else {
      result = out_f32 ? f32(oshape, a) : at::empty(oshape, a.options());
    }
    if (result.scalar_type() == at::kBFloat16) {
      expect(!accumulate, "accumulation needs an fp32 output");
      g.out_mode = OUT_BF16;
    } else {
      expect(result.scalar_type() == at::kFloat, "output type");
      g.out_mode = accumulate ? OUT_F32_ATOMIC : OUT_F32;
    }
    g.ldc = result.stride(-2);
    g.c_bstride = batched ? result.stride(0) : 0;
  }
  g.M = (int)M;
  g.N = (int)N;
  g.K = (int)K;
  g.splits = accumulate ? (int)splits : 1;
  g.trans_out = trans_out;
  g.act = act;
  g.glu = glu;
  g.alpha = (float)alpha;
  g.C = ptr(result);
  g.dm_div = g.dm_mod = 1;
  if (bias) {
    bias = bias->to(at::kBFloat16).contiguous();
    expect(bias->numel() == N, "bias length");
    g.bias = ptr(bias);
  }
  if (rowscale) {
    // bf16 masks are read as they are, which saves the conversion's launch; not so in the gated projection of the triangle
    // multiplication: with them the whole operator took 1250 us at 1024 residues, with the converted mask 1215 us (why is not
    // known, and only that size was measured)
    g.rs_bf16 = rowscale->scalar_type() == at::kBFloat16 && !glu;
    rowscale = (g.rs_bf16 ? *rowscale : rowscale->to(at::kFloat)).contiguous();
    g.rowscale = ptr(rowscale);
    g.rs_bstride = (batched && rowscale->dim() == 2) ? M : 0;
    expect(rowscale->numel() >= (g.rs_bstride ? batch : 1) * M, "fewer row factors than rows");
    expect(rowscale->device() == a.device(), "row factors on another device");
  }
  if (mul) {
    expect(mul->scalar_type() == at::kBFloat16 && mul->stride(-1) == 1, "mul operand");
    g.mul = ptr(mul);
    g.ldmul = mul->stride(-2);
    g.mul_bstride = (batched && mul->dim() == 3) ? mul->stride(0) : 0;
  }
  if (dmask) {
    expect(dmask->scalar_type() == at::kBFloat16 && dmask->stride(-1) == 1 && dmask->size(-1) == n_out, "dropout mask");
    g.dmask = ptr(dmask);
    g.lddm = dmask->dim() >= 2 ? dmask->stride(-2) : 0;
    g.dm_div = (int)dm_div;
    g.dm_mod = (int)dm_mod;
  }
  if (resid) {
    expect(resid->scalar_type() == at::kBFloat16 && resid->stride(-1) == 1, "residual");
    g.resid = ptr(resid);
    g.ldres = resid->stride(-2);
    g.res_bstride = (batched && resid->dim() == 3) ? resid->stride(0) : 0;
  }
  const int rc = ffb_gemm_bf16(ptr(a), ptr(b), a_mn, b_mn, a.stride(-2), b.stride(-2), a3 ? a.stride(0) : 0, b3 ? b.stride(0) : 0, (int)batch,
                               (int)bn, &g, stream());
  ++g_launches;
  TORCH_CHECK(rc == 0, "fastfold_b200 kernel launch failed: ffb_gemm_bf16(M=", M, ",N=", N, ",K=", K, ",batch=", batch, ") returned ", rc);
  return result;
}

// Gradients of y = x W^T + b on [rows, c]: each None unless asked for.  The weight gradient is a split-K product into fp32
// that is then rounded, the bias gradient column sums in fp32.
std::tuple<OptTensor, OptTensor, OptTensor> linear_bwd(const Tensor& dy, const Tensor& x, const Tensor& w, bool need_x, bool need_w, bool need_b,
                                                       int64_t splits) {
  OptTensor dx, dw, db;
  const OptTensor none;
  if (need_x) dx = gemm(dy, w, false, true, 1.0, none, ACT_NONE, false, none, none, none, 1, 1, none, false, none, false, 1, false, 0, std::nullopt);
  if (need_w) {
    const Tensor acc = at::zeros({dy.size(1), x.size(1)}, dy.options().dtype(at::kFloat));
    gemm(dy, x, true, true, 1.0, none, ACT_NONE, false, none, none, none, 1, 1, none, false, acc, false, splits, true, 0, std::nullopt);
    dw = acc.to(w.scalar_type());
  }
  if (need_b) {
    const Tensor acc = at::zeros({dy.size(1)}, dy.options().dtype(at::kFloat));
    check(ffb_colsum(ptr(dy), static_cast<float*>(ptr(acc)), dy.size(0), (int)dy.size(1), stream()), "colsum");
    db = acc.to(w.scalar_type());
  }
  return {dx, dw, db};
}

// An extent that lengths are divided by; integers do not raise by themselves here.
int64_t divisor(int64_t extent) {
  expect(extent > 0, "empty last dimension");
  return extent;
}

int dtype_code(const Tensor& t) {
  return t.scalar_type() == at::kFloat ? 0 : (t.scalar_type() == at::kHalf ? 1 : 2);
}

// y, and mean / rstd when `stats`
std::tuple<Tensor, OptTensor, OptTensor> layer_norm_fwd(const Tensor& x, const Tensor& weight, const Tensor& bias, double eps, bool stats) {
  const Tensor w = weight.contiguous(), b = bias.contiguous();
  const int64_t C = divisor(x.size(-1)), rows = x.numel() / C;
  Tensor y = at::empty_like(x);
  OptTensor mean, rstd;
  if (stats) {
    mean = f32({rows}, x);
    rstd = f32({rows}, x);
  }
  check(ffb_layernorm_fwd(ptr(x), ptr(w), ptr(b), ptr(y), static_cast<float*>(ptr(mean)), static_cast<float*>(ptr(rstd)), rows, (int)C, (float)eps,
                          dtype_code(x), stream()),
        "layernorm_fwd");
  return {y, mean, rstd};
}

std::tuple<Tensor, Tensor, Tensor> layer_norm_bwd(const Tensor& dy, const Tensor& x, const Tensor& w, const Tensor& mean, const Tensor& rstd,
                                                  int64_t nblocks) {
  const int64_t C = divisor(x.size(-1)), rows = x.numel() / C;
  Tensor dx = at::empty_like(x), dg = at::empty_like(w), db = at::empty_like(w), part = f32({nblocks * 2 * C}, x);
  check(ffb_layernorm_bwd(ptr(dy), ptr(x), ptr(w), static_cast<const float*>(ptr(mean)), static_cast<const float*>(ptr(rstd)), ptr(dx),
                          static_cast<float*>(ptr(part)), (int)nblocks, ptr(dg), ptr(db), rows, (int)C, dtype_code(x), stream()),
        "layernorm_bwd");
  return {dx, dg, db};
}

std::tuple<Tensor, OptTensor, OptTensor> layer_norm_transposed_fwd(const Tensor& x_cm, const Tensor& weight, const Tensor& bias, double eps,
                                                                   bool stats) {
  const Tensor w = weight.contiguous(), b = bias.contiguous();
  const int64_t C = x_cm.size(0), rows = x_cm.size(1);
  Tensor y = at::empty({rows, C}, x_cm.options());
  OptTensor mean, rstd;
  if (stats) {
    mean = f32({rows}, x_cm);
    rstd = f32({rows}, x_cm);
  }
  check(ffb_layernorm_fwd_transposed(ptr(x_cm), ptr(w), ptr(b), ptr(y), static_cast<float*>(ptr(mean)), static_cast<float*>(ptr(rstd)), rows, (int)C,
                                     (float)eps, stream()),
        "layernorm_fwd_transposed");
  return {y, mean, rstd};
}

// qkv [1, B, n, 3, H, d] (transposed: [1, n, B, 3, H, d]); bias [H, n, n] at row pitch `pitch`; mask [B, n] bf16
std::tuple<Tensor, OptTensor> attention_packed_fwd(const Tensor& qkv, const OptTensor& mask, const OptTensor& bias, int64_t pitch, double scale,
                                                   bool want_lse, bool transposed) {
  const int64_t B = qkv.size(transposed ? 2 : 1), n = qkv.size(transposed ? 1 : 2), H = qkv.size(4), d = qkv.size(5), HD = H * d;
  expect(!mask || mask->device() == qkv.device(), "mask on another device");
  Tensor out = transposed ? at::empty({1, n, B, HD}, qkv.options()) : at::empty({1, B, n, HD}, qkv.options());
  OptTensor lse;
  if (want_lse) lse = f32({B, H, n}, qkv);
  const int64_t bs = transposed ? 3 * HD : n * 3 * HD, rs = transposed ? B * 3 * HD : 3 * HD;
  char* base = static_cast<char*>(ptr(qkv));
  const int64_t obs = transposed ? HD : n * HD, ors = transposed ? B * HD : HD;
  if (want_lse)           // a pass with gradients: contiguous bias rows
    check(ffb_attention_fwd(base, base + 2 * HD, base + 4 * HD, bs, rs, bs, rs, ptr(bias), ptr(mask), n, ptr(out), obs, ors,
                            static_cast<float*>(ptr(lse)), (int)B, (int)H, (int)n, (int)n, (int)d, (float)scale, stream()),
          "ffb_attention_fwd packed");
  else
    check(ffb_attention_infer(base, base + 2 * HD, base + 4 * HD, bs, rs, bs, rs, ptr(bias), pitch, ptr(mask), n, ptr(out), obs, ors, (int)B, (int)H,
                              (int)n, (int)n, (int)d, (float)scale, stream()),
          "ffb_attention_infer packed");
  return {out, lse};
}

int64_t rows_of(const Tensor& x) { return x.numel() / divisor(x.size(-1)); }

// The elementwise kernels move 16 bytes per thread and operand and do not look at the pointers: a view that starts off a
// 16-byte boundary is copied.
void dense16(Tensor& t) {
  t = t.contiguous();
  if (reinterpret_cast<uintptr_t>(t.data_ptr()) & 15) t = t.clone();
}
void dense16(OptTensor& t) {
  if (t) dense16(*t);
}
template <class... T>
void dense16(T&... ts) {
  (dense16(ts), ...);
}

Tensor bias_sigmoid_mul_fwd(Tensor g, Tensor b, Tensor o) {
  dense16(g, b, o);
  Tensor y = at::empty_like(g);
  check(ffb_bias_sigmoid_mul_fwd(ptr(g), ptr(b), ptr(o), ptr(y), rows_of(g), (int)g.size(-1), stream()), "bias_sigmoid_mul_fwd");
  return y;
}

std::tuple<Tensor, Tensor> bias_sigmoid_mul_bwd(Tensor dy, Tensor g, Tensor b, Tensor o) {
  dense16(dy, g, b, o);
  Tensor dg = at::empty_like(g), dob = at::empty_like(o);
  check(ffb_bias_sigmoid_mul_bwd(ptr(dy), ptr(g), ptr(b), ptr(o), ptr(dg), ptr(dob), rows_of(g), (int)g.size(-1), stream()), "bias_sigmoid_mul_bwd");
  return {dg, dob};
}

Tensor bias_dropout_add_fwd(Tensor x, OptTensor b, OptTensor m, Tensor r, int64_t div, int64_t mod) {
  dense16(x, b, m, r);
  Tensor y = at::empty_like(x);
  check(ffb_bias_dropout_add_fwd(ptr(x), ptr(b), ptr(m), ptr(r), ptr(y), rows_of(x), (int)x.size(-1), (int)div, (int)mod, stream()),
        "bias_dropout_add_fwd");
  return y;
}

Tensor mask_mul(Tensor dy, Tensor m, int64_t div, int64_t mod) {
  dense16(dy, m);
  Tensor dx = at::empty_like(dy);
  check(ffb_mask_mul(ptr(dy), ptr(m), ptr(dx), rows_of(dy), (int)dy.size(-1), (int)div, (int)mod, stream()), "mask_mul");
  return dx;
}

Tensor bias_ele_dropout_res_fwd(Tensor ab, Tensor b, Tensor g, OptTensor m, Tensor r, int64_t div, int64_t mod) {
  dense16(ab, b, g, m, r);
  Tensor y = at::empty_like(ab);
  check(ffb_bias_ele_dropout_res_fwd(ptr(ab), ptr(b), ptr(g), ptr(m), ptr(r), ptr(y), rows_of(ab), (int)ab.size(-1), (int)div, (int)mod, stream()),
        "bias_ele_dropout_res_fwd");
  return y;
}

std::tuple<Tensor, Tensor> bias_ele_dropout_res_bwd(Tensor dy, Tensor ab, Tensor b, Tensor g, OptTensor m,
                                                    int64_t div, int64_t mod) {
  dense16(dy, ab, b, g, m);
  Tensor dab = at::empty_like(ab), dg = at::empty_like(g);
  check(ffb_bias_ele_dropout_res_bwd(ptr(dy), ptr(ab), ptr(b), ptr(g), ptr(m), ptr(dab), ptr(dg), rows_of(ab), (int)ab.size(-1), (int)div, (int)mod,
                                     stream()),
        "bias_ele_dropout_res_bwd");
  return {dab, dg};
}

Tensor glu_mask_t_fwd(Tensor pre, Tensor mask) {
  dense16(pre, mask);
  const int64_t C2 = pre.size(0) / 2, R = pre.size(1);
  Tensor out = at::empty({C2, R}, pre.options());
  check(ffb_glu_mask_t_fwd(ptr(pre), ptr(mask), ptr(out), (int)C2, R, stream()), "glu_mask_t_fwd");
  return out;
}

Tensor glu_mask_t_bwd(Tensor dout, Tensor pre, Tensor mask) {
  dense16(dout, pre, mask);
  Tensor dpre = at::empty_like(pre);
  check(ffb_glu_mask_t_bwd(ptr(dout), ptr(pre), ptr(mask), ptr(dpre), (int)(pre.size(0) / 2), pre.size(1), stream()), "glu_mask_t_bwd");
  return dpre;
}

Tensor act_bwd(Tensor dy, Tensor y, int mode) {
  dense16(dy, y);
  Tensor dx = at::empty_like(dy);
  check(ffb_act_bwd(ptr(dy), ptr(y), ptr(dx), rows_of(dy), (int)dy.size(-1), mode, stream()), "act_bwd");
  return dx;
}

Tensor colsum(const Tensor& x, OptTensor out) {
  if (!out) out = at::zeros({x.size(1)}, x.options().dtype(at::kFloat));
  check(ffb_colsum(ptr(x), static_cast<float*>(ptr(*out)), x.size(0), (int)x.size(1), stream()), "colsum");
  return *out;
}

// ---- LayerNorm + GEMM kernels (ln_gemm.cu) ----
// Rows [.., C] as [batch][rows][C]; weights, norm parameters and biases contiguous bf16 (the callers in ops/ln_gemm.py see to it).
struct Rows {
  int64_t batch, rows, rstride, bstride;
};
Rows rows3(const Tensor& t) {
  expect(t.scalar_type() == at::kBFloat16 && t.stride(-1) == 1 && (t.dim() == 2 || t.dim() == 3), "rows of adjacent bf16 channels");
  if (t.dim() == 2) return {1, t.size(0), t.stride(0), 0};
  return {t.size(0), t.size(1), t.stride(1), t.size(0) > 1 ? t.stride(0) : 0};
}
LnGemmArgs ln_args(const Tensor& x, const Tensor& gamma, const Tensor& beta, double eps, int mode) {
  LnGemmArgs g = {};
  const Rows r = rows3(x);
  g.x = ptr(x);
  g.C = (int)x.size(-1);
  g.rows = r.rows;
  g.batch = r.batch;
  g.x_rstride = r.rstride;
  g.x_bstride = r.bstride;
  expect(gamma.numel() == g.C && beta.numel() == g.C, "norm parameters");
  g.gamma = ptr(gamma);
  g.beta = ptr(beta);
  g.eps = (float)eps;
  g.mode = mode;
  return g;
}
void ln_run(const LnGemmArgs& g, const char* what) {
  if (g.rows * g.batch == 0) return;
  check(ffb_ln_gemm(&g, stream()), what);
}
void same_rows(const Rows& a, const LnGemmArgs& g) { expect(a.batch == g.batch && a.rows == g.rows, "operands with other rows than the input"); }
void same_shape(const Tensor& t, const LnGemmArgs& g, int64_t n) {
  same_rows(rows3(t), g);
  expect(t.size(-1) == n, "operands with other columns than the result");
}

// resid + b2 + f(LN(x) w1^T + b1) w2^T; f = relu, or sigmoid(.) * mul (fp32 `mul`: one row of factors for every mul.size(0)-th row)
Tensor ln_chain(const Tensor& x, const Tensor& gamma, const Tensor& beta, double eps, const Tensor& w1, const OptTensor& b1, const Tensor& w2,
                const OptTensor& b2, const OptTensor& mul, const Tensor& resid, OptTensor out) {
  LnGemmArgs g = ln_args(x, gamma, beta, eps, mul ? LN_GATE_CHAIN : LN_RELU_CHAIN);
  g.hidden = (int)w1.size(0);
  expect(w1.size(1) == g.C && w2.size(0) == g.C && w2.size(1) == g.hidden && (!b1 || b1->numel() == g.hidden) && (!b2 || b2->numel() == g.C), "weights");
  g.w1 = ptr(w1);
  g.b1 = ptr(b1);
  g.w2 = ptr(w2);
  g.b2 = ptr(b2);
  if (mul && mul->scalar_type() == at::kFloat) {
    expect(mul->dim() == 2 && mul->is_contiguous() && mul->size(1) == g.hidden && mul->size(0) > 0, "gated operand");
    g.mul_f32 = static_cast<const float*>(ptr(mul));
    g.mul_mod = (int)mul->size(0);
  } else if (mul) {
    const Rows r = rows3(*mul);
    same_shape(*mul, g, g.hidden);
    g.mul = ptr(mul);
    g.m_rstride = r.rstride;
    g.m_bstride = r.bstride;
  }
  const Rows r = rows3(resid);
  same_shape(resid, g, g.C);
  g.resid = ptr(resid);
  g.r_rstride = r.rstride;
  g.r_bstride = r.bstride;
  Tensor y = out ? *out : at::empty(resid.sizes(), resid.options());
  const Rows o = rows3(y);
  same_shape(y, g, g.C);
  g.out = ptr(y);
  g.o_rstride = o.rstride;
  g.o_bstride = o.bstride;
  ln_run(g, "ln_chain");
  return y;
}

LnSegment ln_rows(const LnGemmArgs& g, const Tensor& w, const OptTensor& bias, int act, bool scaled, const Tensor& out) {
  const Rows o = rows3(out);
  expect(w.size(1) == g.C && (!bias || bias->numel() == w.size(0)), "weights");
  same_shape(out, g, w.size(0));
  LnSegment s = {};
  s.w = ptr(w);
  s.bias = ptr(bias);
  s.n = (int)w.size(0);
  s.kind = LN_ROWS;
  s.act = act;
  s.scaled = scaled;
  s.out = ptr(out);
  s.o_rstride = o.rstride;
  s.o_bstride = o.bstride;
  return s;
}
Tensor like_rows(const Tensor& x, int64_t n) {
  auto shape = x.sizes().vec();
  shape.back() = n;
  return at::empty(shape, x.options());
}

// LN(x) w^T of rows [.., C], and / or the pair bias LN(x) wb^T of a pair tensor's rows (i j): bias [H, q, k] with q = i and k = j,
// or q = j and k = i (`transposed`), into `bias`, whose last two axes may have any pitch
OptTensor ln_qkv(const Tensor& x, const Tensor& gamma, const Tensor& beta, double eps, const OptTensor& w, const OptTensor& wb, const OptTensor& bias,
                 bool transposed) {
  LnGemmArgs g = ln_args(x, gamma, beta, eps, LN_PROJECT);
  OptTensor y;
  if (w) {
    y = like_rows(x, w->size(0));
    g.seg[g.nseg++] = ln_rows(g, *w, std::nullopt, ACT_NONE, false, *y);
  }
  if (wb) {
    expect(bias && bias->dim() == 3 && wb->size(1) == g.C, "pair bias");
    const int64_t ni = bias->size(transposed ? 2 : 1), nj = bias->size(transposed ? 1 : 2);
    expect(bias->scalar_type() == at::kBFloat16 && bias->size(0) == wb->size(0) && ni * nj == g.rows * g.batch, "pair bias");
    LnSegment& s = g.seg[g.nseg++];
    s.w = ptr(wb);
    s.n = (int)wb->size(0);
    s.kind = LN_PAIR_BIAS;
    s.out = ptr(bias);
    g.pb_n = (int)nj;
    g.pb_h = bias->stride(0);
    g.pb_i = bias->stride(transposed ? 2 : 1);
    g.pb_j = bias->stride(transposed ? 1 : 2);
  }
  ln_run(g, "ln_qkv");
  return y;
}

// Value vectors [N, 64] (fp32) of the global column attention over x [S, N, 64] with keys and values kv [S * N, 16]
Tensor global_column(const Tensor& x, const Tensor& gamma, const Tensor& beta, double eps, const Tensor& wq, const Tensor& kv, Tensor mask, double scaling) {
  const int64_t S = x.size(0), N = x.size(1);
  mask = mask.to(at::kBFloat16).contiguous();
  expect(x.dim() == 3 && x.is_contiguous() && x.size(2) == 64 && gamma.numel() == 64 && beta.numel() == 64 && wq.is_contiguous() && wq.size(0) == 64 &&
             wq.size(1) == 64 && kv.is_contiguous() && kv.numel() == S * N * 16 && mask.numel() == S * N,
         "global column attention");
  const Tensor out = f32({N, 64}, x);
  if (x.numel() == 0) return out;
  check(ffb_global_column(ptr(x), ptr(gamma), ptr(beta), (float)eps, ptr(wq), ptr(kv), ptr(mask), static_cast<float*>(ptr(out)), S, N, (float)scaling,
                          stream()),
        "global_column");
  return out;
}

void ln_scale(LnGemmArgs& g, Tensor& scale) {
  g.rs_bf16 = scale.scalar_type() == at::kBFloat16;
  scale = (g.rs_bf16 ? scale : scale.to(at::kFloat)).contiguous();
  expect(scale.numel() >= g.rows * g.batch, "fewer row factors than rows");
  g.rowscale = ptr(scale);
}

// Operands of the triangle multiplication: the gated projections, channels first, into lr [2c, batch, rows] (any pitch), times one
// factor per row; returns the output gate sigmoid(LN(x) wg^T + bg)
Tensor ln_tri_in(const Tensor& x, const Tensor& gamma, const Tensor& beta, double eps, const Tensor& w, const Tensor& b, const Tensor& wg,
                 const Tensor& bg, Tensor scale, const Tensor& lr) {
  LnGemmArgs g = ln_args(x, gamma, beta, eps, LN_PROJECT);
  ln_scale(g, scale);
  expect(lr.dim() == 3 && lr.scalar_type() == at::kBFloat16 && lr.size(0) * 2 == w.size(0) && lr.size(1) == g.batch && lr.size(2) == g.rows &&
             lr.stride(2) == 1 && w.size(1) == g.C && b.numel() == w.size(0),
         "gated operands");
  LnSegment& s = g.seg[0];
  s.w = ptr(w);
  s.bias = ptr(b);
  s.n = (int)w.size(0);
  s.kind = LN_GLU_T;
  s.scaled = 1;
  s.out = ptr(lr);
  s.o_rstride = lr.stride(0);
  s.o_bstride = g.batch > 1 ? lr.stride(1) : 0;
  const Tensor y = like_rows(x, wg.size(0));
  g.seg[1] = ln_rows(g, wg, bg, ACT_SIGMOID, false, y);
  g.nseg = 2;
  ln_run(g, "ln_tri_in");
  return y;
}

// Output of the triangle multiplication: resid + mul * (LN(p) w^T + b) of a channels-first p [c, batch, rows] (any pitch)
Tensor ln_tri_out(const Tensor& p, const Tensor& gamma, const Tensor& beta, double eps, const Tensor& w, const Tensor& b, const Tensor& mul,
                  const Tensor& resid, OptTensor out) {
  LnGemmArgs g = {};
  expect(p.scalar_type() == at::kBFloat16 && p.dim() == 3 && p.stride(2) == 1, "channels-first operand");
  g.x = ptr(p);
  g.channels_first = 1;
  g.C = (int)p.size(0);
  g.batch = p.size(1);
  g.rows = p.size(2);
  g.x_rstride = p.stride(0);
  g.x_bstride = g.batch > 1 ? p.stride(1) : 0;
  expect(gamma.numel() == g.C && beta.numel() == g.C, "norm parameters");
  g.gamma = ptr(gamma);
  g.beta = ptr(beta);
  g.eps = (float)eps;
  g.mode = LN_PROJECT;
  const Rows m = rows3(mul), r = rows3(resid);
  same_shape(mul, g, w.size(0));
  same_shape(resid, g, w.size(0));
  g.mul = ptr(mul);
  g.m_rstride = m.rstride;
  g.m_bstride = m.bstride;
  g.resid = ptr(resid);
  g.r_rstride = r.rstride;
  g.r_bstride = r.bstride;
  Tensor y = out ? *out : at::empty(resid.sizes(), resid.options());
  g.seg[0] = ln_rows(g, w, b, ACT_NONE, false, y);
  g.nseg = 1;
  ln_run(g, "ln_tri_out");
  return y;
}

// (LN(x) wa^T + ba) * scale and (LN(x) wb^T + bb) * scale
std::tuple<Tensor, Tensor> ln_pair(const Tensor& x, const Tensor& gamma, const Tensor& beta, double eps, const Tensor& wa, const OptTensor& ba,
                                   const Tensor& wb, const OptTensor& bb, Tensor scale) {
  LnGemmArgs g = ln_args(x, gamma, beta, eps, LN_PROJECT);
  ln_scale(g, scale);
  const Tensor ya = like_rows(x, wa.size(0)), yb = like_rows(x, wb.size(0));
  g.seg[0] = ln_rows(g, wa, ba, ACT_NONE, true, ya);
  g.seg[1] = ln_rows(g, wb, bb, ACT_NONE, true, yb);
  g.nseg = 2;
  ln_run(g, "ln_pair");
  return {ya, yb};
}

// ---- whole modules without gradients, from their input to their result ----
// A module is two to four launches, and checks, views and calls made one by one from Python took three times as long as the
// launches: a block of 32 x 64 was 830 us of host time for 265 us of kernels.  Each returns None where the kernels do not cover the
// call; the caller then composes the module from its parts.
bool plain(const Tensor& t) {
  return t.is_cuda() && t.scalar_type() == at::kBFloat16 && t.is_contiguous() && (reinterpret_cast<uintptr_t>(t.data_ptr()) & 15) == 0;
}
bool plain(const OptTensor& t) { return !t || plain(*t); }
template <class... T>
bool all_plain(const T&... ts) {
  return (plain(ts) && ...);
}
bool rows_of_channels(const Tensor& x) {
  const int64_t C = x.dim() > 0 ? x.size(-1) : 0;
  return x.is_cuda() && x.scalar_type() == at::kBFloat16 && (C == 64 || C == 128 || C == 256) && x.numel() > 0;
}
bool matrix(const Tensor& w, int64_t rows, int64_t cols) { return w.dim() == 2 && w.size(0) == rows && w.size(1) == cols; }
bool vector(const OptTensor& b, int64_t n) { return !b || b->numel() == n; }
constexpr int64_t LN_MAX_COLUMNS = 1280;      // weight rows of one call of the LayerNorm + GEMM kernels

// x as the kernels address it: contiguous rows on a 16-byte boundary
Tensor dense_rows(Tensor x) {
  dense16(x);
  return x;
}

// `inplace`: the caller's tensor receives the result, also where the kernels worked on a dense copy of it
Tensor settle(const Tensor& x0, const Tensor& out, bool inplace) {
  if (!inplace || out.data_ptr() == x0.data_ptr()) return out;
  x0.copy_(out);
  return x0;
}

// mul * act(x w^T + b) + resid
Tensor linear(const Tensor& x, const Tensor& w, const OptTensor& b, int act, const OptTensor& mul, const OptTensor& resid, const OptTensor& out) {
  const OptTensor none;
  return gemm(x, w, false, false, 1.0, b, act, false, none, mul, none, 1, 1, resid, false, out, false, 1, false, 0, std::nullopt);
}

// Few rows of 256 channels under stream capture.  A tile of 128 rows walks all weights on one SM, 25 us for a transition whether there are
// 64 rows or 16384, where LayerNorm and two GEMMs, whose tiles spread over the SMs, take less.  In a graph (B200, us, one kernel / separate
// ones): transition 64 rows 24 / 13, 2048 25 / 15, 4096 25 / 16, 8192 26 / 21, 12288 26 / 28, 16384 26 / 30; column attention 32 x 64 37 / 28,
// 128 x 64 40 / 35, 128 x 96 45 / 45, 128 x 128 48 / 51; row attention 32 x 64 47 / 35, 128 x 64 54 / 45, 128 x 96 60 / 57, 128 x 128 60 / 63;
// the MSA half of a block of 32 x 64 110 / 77.  So up to a tile for every second SM.  Calls that are not captured are bound by the host there and
// keep the fewer launches: a block of 32 x 64 356 / 388, 128 x 64 358 / 394, 64 x 100 359 / 394.  With 64 and 128 channels the one kernel is
// the faster one at every length.  Both give the same bits.
bool few_rows_captured(int64_t C, int64_t rows) {
  return C == 256 && (rows + 127) / 128 * 2 <= at::cuda::getCurrentDeviceProperties()->multiProcessorCount &&
         c10::cuda::currentStreamCaptureStatusMayInitCtx() != c10::cuda::CaptureStatus::None;
}

OptTensor transition_module(const Tensor& x0, const Tensor& gamma, const Tensor& beta, double eps, const Tensor& w1, const OptTensor& b1, const Tensor& w2,
                            const OptTensor& b2, bool inplace) {
  if (!rows_of_channels(x0) || !all_plain(gamma, beta, w1, b1, w2, b2)) return std::nullopt;
  const int64_t C = x0.size(-1), hidden = w1.size(0);
  if (hidden % 128 || hidden > LN_MAX_COLUMNS || !matrix(w1, hidden, C) || !matrix(w2, C, hidden) || !vector(b1, hidden) || !vector(b2, C) ||
      gamma.numel() != C || beta.numel() != C)
    return std::nullopt;
  const Tensor x = dense_rows(x0), x2 = x.view({-1, C});
  const OptTensor dst = inplace ? OptTensor(x2) : std::nullopt;
  if (few_rows_captured(C, x2.size(0))) {
    const Tensor h = linear(std::get<0>(layer_norm_fwd(x2, gamma, beta, eps, false)), w1, b1, ACT_RELU, std::nullopt, std::nullopt, std::nullopt);
    return settle(x0, linear(h, w2, b2, ACT_NONE, std::nullopt, x2, dst).view(x.sizes()), inplace);
  }
  return settle(x0, ln_chain(x2, gamma, beta, eps, w1, b1, w2, b2, std::nullopt, x2, dst).view(x.sizes()), inplace);
}

// A pair bias [H, n, n] with rows at an 8-element pitch
Tensor pitched(int64_t H, int64_t n, const Tensor& like) { return at::empty({H, n, (n + 7) / 8 * 8}, like.options()).narrow(2, 0, n); }

// x [1, A, B, C] plus the gated attention over norm(x) along its second axis (first with `transposed`), `chunk` rows (columns) at a
// time where that is > 0.  Pair bias: none, or pair_w applied to norm(x), or to norm_z(z) where z is given.
OptTensor attention_module(const Tensor& x0, const Tensor& gamma, const Tensor& beta, double eps, const Tensor& wq, const Tensor& wg, const Tensor& bg,
                           const Tensor& wo, const OptTensor& bo, const OptTensor& mask, const OptTensor& pair_w, const OptTensor& z0,
                           const OptTensor& z_gamma, const OptTensor& z_beta, double z_eps, int64_t H, int64_t D, double scale, bool transposed,
                           int64_t chunk, bool inplace) {
  if (!rows_of_channels(x0) || x0.dim() != 4 || x0.size(0) != 1 || !all_plain(gamma, beta, wq, wg, bg, wo, bo, pair_w, z_gamma, z_beta)) return std::nullopt;
  const int64_t A = x0.size(1), B = x0.size(2), C = x0.size(3), HD = H * D;
  const int64_t n = transposed ? A : B, rows = transposed ? B : A;
  if ((D != 16 && D != 32) || HD % 128 || 3 * HD + 128 > LN_MAX_COLUMNS || !matrix(wq, 3 * HD, C) || !matrix(wg, HD, C) || bg.numel() != HD || !matrix(wo, C, HD) ||
      !vector(bo, C) || gamma.numel() != C || beta.numel() != C)
    return std::nullopt;
  if (mask && (mask->numel() != rows * n || mask->device() != x0.device())) return std::nullopt;
  if (pair_w) {
    const Tensor& src = z0 ? *z0 : x0;
    if (H > 32 || !rows_of_channels(src) || src.dim() != 4 || src.size(0) != 1 || src.size(1) != n || src.size(2) != n || !matrix(*pair_w, H, src.size(3)))
      return std::nullopt;
    if (z0 && (!z_gamma || !z_beta || z_gamma->numel() != src.size(3) || z_beta->numel() != src.size(3))) return std::nullopt;
  }
  const Tensor x = dense_rows(x0), x3 = x.view({A, B, C}), x2 = x.view({-1, C});
  const Tensor out = inplace ? x3 : at::empty_like(x3);
  OptTensor m2, bias;
  if (mask) m2 = mask->reshape({rows, n}).to(at::kBFloat16).contiguous();
  const bool whole = chunk <= 0 || chunk >= rows;
  OptTensor own_w;                                    // pair weight that rides along with QKV
  if (pair_w) {
    bias = pitched(H, n, x);
    if (z0) ln_qkv(dense_rows(*z0).view({n * n, -1}), *z_gamma, *z_beta, z_eps, std::nullopt, pair_w, bias, false);
    else if (whole) own_w = pair_w;
    else ln_qkv(x2, gamma, beta, eps, std::nullopt, pair_w, bias, transposed);
  }
  const int64_t pitch = bias ? bias->stride(1) : n;
  OptTensor norm;                                     // of the whole input, where its projections are kernels of their own
  if (few_rows_captured(C, n * (whole ? rows : std::min(chunk, rows)))) {
    norm = std::get<0>(layer_norm_fwd(x2, gamma, beta, eps, false)).view(x3.sizes());
    if (own_w) ln_qkv(x2, gamma, beta, eps, std::nullopt, own_w, bias, transposed);
  }
  for (int64_t at = 0; at < rows; at += whole ? rows : chunk) {
    const int64_t len = whole ? rows : std::min(chunk, rows - at);
    // rows are contiguous: one matrix; columns are not: a batch of them, one per position along the attention
    auto cut = [&](const Tensor& t) {
      if (whole) return t.view({-1, t.size(2)});
      const Tensor slice = t.narrow(transposed ? 1 : 0, at, len);
      return transposed ? slice : slice.view({-1, t.size(2)});
    };
    const Tensor part = cut(x3), dst = cut(out);
    const Tensor qkv = norm ? linear(cut(*norm), wq, std::nullopt, ACT_NONE, std::nullopt, std::nullopt, std::nullopt)
                            : *ln_qkv(part, gamma, beta, eps, wq, own_w, own_w ? bias : OptTensor(), transposed);
    const OptTensor m = m2 ? OptTensor(whole ? *m2 : m2->narrow(0, at, len)) : std::nullopt;
    const Tensor o4 = std::get<0>(attention_packed_fwd(transposed ? qkv.view({1, n, len, 3, H, D}) : qkv.view({1, len, n, 3, H, D}), m, bias, pitch, scale,
                                                       false, transposed));
    const Tensor o = part.dim() == 3 ? o4.view({part.size(0), part.size(1), HD}) : o4.view({-1, HD});
    if (norm) linear(linear(cut(*norm), wg, bg, ACT_SIGMOID, o, std::nullopt, std::nullopt), wo, bo, ACT_NONE, std::nullopt, part, dst);
    else ln_chain(part, gamma, beta, eps, wg, bg, wo, bo, o, part, dst);
  }
  return settle(x0, out.unsqueeze(0), inplace);
}

// Triangle multiplication of a square pair tensor [1, n, n, 128].  w / b: projection and gate weights interleaved by rows.  Extents
// that are no multiple of 8 make the first axis the batch, so that the channels-first tensors get rows at an 8-element pitch (TMA
// wants 16-byte strides); the padding is neither written nor read.
OptTensor triangle_module(const Tensor& z0, const Tensor& g1, const Tensor& b1, double eps1, const Tensor& w, const Tensor& b, const Tensor& wg, const Tensor& bg,
                          const Tensor& g2, const Tensor& b2, double eps2, const Tensor& wo, const Tensor& bo, const Tensor& mask, bool outgoing, bool inplace) {
  if (!rows_of_channels(z0) || z0.dim() != 4 || z0.size(0) != 1 || z0.size(1) != z0.size(2) || z0.size(3) != 128 || mask.device() != z0.device() ||
      !all_plain(g1, b1, w, b, wg, bg, g2, b2, wo, bo))
    return std::nullopt;
  constexpr int64_t c = 128;
  const int64_t n = z0.size(1), pitch = (n + 7) / 8 * 8;
  if (!matrix(w, 4 * c, c) || b.numel() != 4 * c || !matrix(wg, c, c) || bg.numel() != c || !matrix(wo, c, c) || bo.numel() != c || g1.numel() != c ||
      b1.numel() != c || g2.numel() != c || b2.numel() != c)
    return std::nullopt;
  const Tensor z = dense_rows(z0), scale = mask.numel() == n * n ? mask.reshape({-1}) : mask.expand({1, n, n}).reshape({-1});
  const Tensor lr = at::empty({2 * c, n, pitch}, z.options()), p = at::empty({c, n, pitch}, z.options());
  const bool flat = pitch == n;
  const Tensor z3 = flat ? z.view({1, n * n, c}) : z.view({n, n, c});
  auto cut = [&](const Tensor& t) { return flat ? t.view({t.size(0), 1, n * n}) : t.narrow(2, 0, n); };
  const Tensor gate = ln_tri_in(z3, g1, b1, eps1, w, b, wg, bg, scale, cut(lr));
  const Tensor lr_n = lr.narrow(2, 0, n), p_n = p.narrow(2, 0, n);
  const OptTensor none;
  gemm(lr_n.narrow(0, 0, c), lr_n.narrow(0, c, c), !outgoing, !outgoing, 1.0, none, ACT_NONE, false, none, none, none, 1, 1, none, false, p_n, false, 1,
       false, 0, std::nullopt);
  return settle(z0, ln_tri_out(cut(p), g2, b2, eps2, wo, bo, gate, z3, inplace ? OptTensor(z3) : std::nullopt).view(z.sizes()), inplace);
}

// Global column attention of the extra-MSA stack over x [1, S, N, 64], 8 heads of 8 channels
OptTensor global_column_module(const Tensor& x0, const Tensor& gamma, const Tensor& beta, double eps, const Tensor& wq, const Tensor& wkv, const Tensor& wg,
                               const Tensor& bg, const Tensor& wo, const OptTensor& bo, const Tensor& mask, double scale, bool inplace) {
  if (!rows_of_channels(x0) || x0.dim() != 4 || x0.size(0) != 1 || x0.size(3) != 64 || !all_plain(gamma, beta, wq, wkv, wg, bg, wo, bo)) return std::nullopt;
  if (!matrix(wq, 64, 64) || !matrix(wkv, 16, 64) || !matrix(wg, 64, 64) || bg.numel() != 64 || !matrix(wo, 64, 64) || !vector(bo, 64) || gamma.numel() != 64 ||
      beta.numel() != 64 || mask.numel() != x0.size(1) * x0.size(2) || mask.device() != x0.device())
    return std::nullopt;
  const Tensor x = dense_rows(x0), x2 = x.view({-1, 64});
  const Tensor kv = *ln_qkv(x2, gamma, beta, eps, wkv, std::nullopt, std::nullopt, false);
  const Tensor o = global_column(x.view({x.size(1), x.size(2), 64}), gamma, beta, eps, wq, kv, mask, scale);
  return settle(x0, ln_chain(x2, gamma, beta, eps, wg, bg, wo, bo, o, x2, inplace ? OptTensor(x2) : std::nullopt).view(x.sizes()), inplace);
}

// Masked projections of the outer product mean
std::optional<std::tuple<Tensor, Tensor>> masked_pair(const Tensor& x0, const Tensor& gamma, const Tensor& beta, double eps, const Tensor& wa,
                                                      const OptTensor& ba, const Tensor& wb, const OptTensor& bb, const Tensor& mask) {
  if (!rows_of_channels(x0) || !all_plain(gamma, beta, wa, ba, wb, bb) || mask.device() != x0.device()) return std::nullopt;
  const int64_t C = x0.size(-1);
  if (!matrix(wa, wa.size(0), C) || !matrix(wb, wb.size(0), C) || !vector(ba, wa.size(0)) || !vector(bb, wb.size(0)) || wa.size(0) % 8 || wb.size(0) % 8 ||
      wa.size(0) + wb.size(0) + 256 > LN_MAX_COLUMNS || gamma.numel() != C || beta.numel() != C)
    return std::nullopt;
  const Tensor x = dense_rows(x0);
  auto shape = x.sizes().vec();
  shape.back() = 1;
  const Tensor factors = mask.numel() == x.numel() / C ? mask.reshape({-1}) : mask.expand(shape).reshape({-1});
  auto [a, b] = ln_pair(x.view({-1, C}), gamma, beta, eps, wa, ba, wb, bb, factors);
  shape.back() = wa.size(0);
  const Tensor a4 = a.view(shape);
  shape.back() = wb.size(0);
  return std::make_tuple(a4, b.view(shape));
}

// 1 / (mask^T mask + eps) of a mask [1, S, N], as [1, N, N, 1] in fp32; None for other shapes and types
OptTensor mask_norm(const Tensor& mask, double eps) {
  const bool half = mask.scalar_type() == at::kBFloat16;
  if (!mask.is_cuda() || (!half && mask.scalar_type() != at::kFloat) || mask.dim() != 3 || mask.size(0) != 1 || mask.numel() == 0) return std::nullopt;
  const Tensor m = mask.contiguous();
  const int64_t S = m.size(1), N = m.size(2);
  const Tensor out = f32({1, N, N, 1}, m);
  check(ffb_mask_norm(ptr(m), static_cast<float*>(ptr(out)), (int)S, (int)N, (float)eps, half, stream()), "mask_norm");
  return out;
}

// Invariant point attention between its input projections [N, .] and its output projection, in three kernels; rot: [N, 3, 3] matrices or
// [N, 4] quaternions, trans [N, 3], both fp32.  Parameters and mask in bf16 or fp32 as they come: as four conversions, with the 13 tensors of
// the three calls allocated and passed one by one, the layer's host side took 220 us at 512 residues, the kernels 215.
Tensor ipa_layer(const Tensor& q, const Tensor& kv, const Tensor& q_pts, const Tensor& kv_pts, const Tensor& rot, bool is_quat, const Tensor& trans,
                 const Tensor& z, const Tensor& wb, const Tensor& bb, const Tensor& gamma, const Tensor& mask, double w_c, double w_b, double inf,
                 double eps) {
  constexpr int H = 12, C = 16, PQ = 4, PV = 8, CZ = 128;
  const int64_t N = z.dim() == 3 ? z.size(0) : -1;
  expect(N >= 0 && z.size(1) == N && z.size(2) == CZ && z.scalar_type() == at::kBFloat16 && z.is_contiguous(), "invariant point attention: dense bf16 pair tensor");
  // the kernels index these by N alone
  for (auto [t, width] : {std::pair(&q, H * C), std::pair(&kv, 2 * H * C), std::pair(&q_pts, 3 * H * PQ), std::pair(&kv_pts, 3 * H * (PQ + PV))})
    expect(t->device() == z.device() && t->scalar_type() == at::kBFloat16 && t->is_contiguous() && t->numel() == N * width,
           "invariant point attention: dense bf16 projections with a row for each of the pair tensor's, on its device");
  int bf = 0;
  auto operand = [&](const Tensor& t, int64_t numel, int bit) {
    expect(t.device() == z.device() && t.numel() == numel, "invariant point attention: parameters and mask on the device of the pair tensor");
    if (t.scalar_type() == at::kBFloat16) {
      bf |= bit;
      return t.contiguous();
    }
    return t.to(at::kFloat).contiguous();
  };
  const Tensor w = operand(wb, H * CZ, IPA_BF16_WB), b = operand(bb, H, IPA_BF16_BB), g = operand(gamma, H, IPA_BF16_GAMMA),
               m = operand(mask, N, IPA_BF16_MASK);
  expect(rot.numel() == N * (is_quat ? 4 : 9) && trans.numel() == 3 * N && rot.scalar_type() == at::kFloat && trans.scalar_type() == at::kFloat &&
             rot.device() == z.device() && trans.device() == z.device() && rot.is_contiguous() && trans.is_contiguous(),
         "invariant point attention: frames");
  expect(z.is_cuda(), "invariant point attention: operands on a CUDA device");
  // one workspace: queries, keys, values, their points, and the core's outputs (extents are multiples of 16 bytes a residue)
  const Tensor work = f32({N * H * (3 * C + 3 * (2 * PQ + PV) + C + 3 * PV + CZ)}, z);
  float* at = static_cast<float*>(ptr(work));
  auto take = [&](int per_head) {
    float* p = at;
    at += N * H * per_head;
    return p;
  };
  float *qf = take(C), *kf = take(C), *vf = take(C), *qp = take(3 * PQ), *kp = take(3 * PQ), *vp = take(3 * PV), *o = take(C), *o_pt = take(3 * PV),
        *o_pair = take(CZ);
  const float *r = static_cast<const float*>(ptr(rot)), *t = static_cast<const float*>(ptr(trans));
  check(ffb_ipa_prep(ptr(q), ptr(kv), ptr(q_pts), ptr(kv_pts), r, is_quat, t, qf, kf, vf, qp, kp, vp, (int)N, H, C, PQ, PV, stream()), "ipa_prep");
  check(ffb_ipa_fwd_mixed(qf, kf, vf, qp, kp, vp, ptr(z), ptr(w), ptr(b), ptr(g), ptr(m), bf, o, o_pt, o_pair, (int)N, H, C, PQ, PV, CZ, 0, (int)N,
                          (float)w_c, (float)w_b, (float)inf, stream()),
        "ipa_fwd");
  const Tensor out = at::empty({N, H * (C + 4 * PV + CZ)}, z.options());
  check(ffb_ipa_cat(o, o_pt, o_pair, r, is_quat, t, ptr(out), (int)N, H, C, PV, CZ, (float)eps, stream()), "ipa_cat");
  return out;
}

}  // namespace

PYBIND11_MODULE(_ffb_dispatch, m) {
  m.def("gemm", &gemm);
  m.def("linear_bwd", &linear_bwd);
  m.def("layer_norm_fwd", &layer_norm_fwd);
  m.def("layer_norm_bwd", &layer_norm_bwd);
  m.def("layer_norm_transposed_fwd", &layer_norm_transposed_fwd);
  m.def("attention_packed_fwd", &attention_packed_fwd);
  m.def("bias_sigmoid_mul_fwd", &bias_sigmoid_mul_fwd);
  m.def("bias_sigmoid_mul_bwd", &bias_sigmoid_mul_bwd);
  m.def("bias_dropout_add_fwd", &bias_dropout_add_fwd);
  m.def("mask_mul", &mask_mul);
  m.def("bias_ele_dropout_res_fwd", &bias_ele_dropout_res_fwd);
  m.def("bias_ele_dropout_res_bwd", &bias_ele_dropout_res_bwd);
  m.def("glu_mask_t_fwd", &glu_mask_t_fwd);
  m.def("glu_mask_t_bwd", &glu_mask_t_bwd);
  m.def("act_bwd", &act_bwd);
  m.def("colsum", &colsum);
  m.def("ln_chain", &ln_chain);
  m.def("ln_qkv", &ln_qkv);
  m.def("ln_tri_in", &ln_tri_in);
  m.def("ln_pair", &ln_pair);
  m.def("transition_module", &transition_module);
  m.def("attention_module", &attention_module);
  m.def("triangle_module", &triangle_module);
  m.def("global_column_module", &global_column_module);
  m.def("masked_pair", &masked_pair);
  m.def("mask_norm", &mask_norm);
  m.def("ipa_layer", &ipa_layer);
  m.def("launches", []() { return g_launches; });
}

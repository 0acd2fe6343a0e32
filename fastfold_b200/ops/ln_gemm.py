"""LayerNorm and the GEMMs that read its rows, in one kernel each (csrc/ln_gemm.cu), without gradients.

The callers (``models/fastnn``) ask ``ready`` first and otherwise compose LayerNorm and GEMM; the two agree up to
the rounding of the LayerNorm's sums.
"""
import torch
from torch.autograd import forward_ad
from torch.nn.modules import module as _nn_module

from . import _lib

CHANNELS = (64, 128, 256)
MAX_COLUMNS = 1280          # weight rows of one call (their biases are kept in shared memory)


def hooked(mod):
    return bool(mod._forward_hooks or mod._forward_pre_hooks)


def ready(x, norm, modules=(), tensors=()):
    """True when the kernels may stand for ``norm(x)`` and what follows: bf16 activations in GPU memory, contiguous bf16
    parameters, no gradients or forward-mode level, and no hook on a module that would be passed by."""
    if torch.is_grad_enabled() or not (x.is_cuda and x.dtype == torch.bfloat16 and x.shape[-1] in CHANNELS and x.numel() > 0):
        return False
    if forward_ad._current_level >= 0 or _nn_module._global_forward_hooks or _nn_module._global_forward_pre_hooks:
        return False
    if hooked(norm) or any(hooked(m) for m in modules):
        return False
    return all(t is None or (t.dtype == torch.bfloat16 and t.is_contiguous() and t.data_ptr() % 16 == 0 and t.is_cuda)
               for t in (norm.weight, norm.bias, *tensors))


def dense(x):
    """``x`` as the kernels address it: contiguous rows on a 16-byte boundary (a copy of anything else)."""
    x = x.contiguous()
    return x.clone() if x.data_ptr() % 16 else x


def chain(x, norm, w1, b1, w2, b2, resid, mul=None, out=None):
    """``resid + b2 + f(LN(x) w1^T + b1) w2^T`` with ``f`` = relu, or sigmoid times ``mul`` (one row of it per row of ``x``; in fp32,
    ``[n, hidden]``, row ``r`` of ``x`` takes row ``r % n``)."""
    return _lib.native().ln_chain(x, norm.weight, norm.bias, norm.eps, w1, b1, w2, b2, mul, resid, out)


def qkv(x, norm, w=None, pair_w=None, pair_out=None, transposed=False):
    """``LN(x) w^T`` (None without ``w``); with ``pair_w [H, C]`` also the pair bias ``pair_out[h, q, k] = LN(x)[q, k] . pair_w[h]``
    (``LN(x)[k, q]`` with ``transposed``) of rows ``(i j)``."""
    return _lib.native().ln_qkv(x, norm.weight, norm.bias, norm.eps, w, pair_w, pair_out, transposed)


def tri_in(x, norm, w, b, wg, bg, scale, lr):
    """Gated, channels-first operands of the triangle multiplication into ``lr``; returns its output gate."""
    return _lib.native().ln_tri_in(x, norm.weight, norm.bias, norm.eps, w, b, wg, bg, scale, lr)


def tri_out(p, norm, w, b, mul, resid, out=None):
    """``resid + mul * (LN(p) w^T + b)`` of a channels-first ``p [c, batch, rows]``."""
    return _lib.native().ln_tri_out(p, norm.weight, norm.bias, norm.eps, w, b, mul, resid, out)


def pair(x, norm, wa, ba, wb, bb, scale):
    """``(LN(x) wa^T + ba) * scale`` and the same with ``wb``, ``bb``; one factor per row."""
    return _lib.native().ln_pair(x, norm.weight, norm.bias, norm.eps, wa, ba, wb, bb, scale)


def global_column(x, norm, wq, kv, mask, scaling):
    """Value vectors ``[N, 64]`` (fp32) of the global column attention over ``x [S, N, 64]``: one mean query per column and head."""
    return _lib.native().global_column(x, norm.weight, norm.bias, norm.eps, wq, kv, mask, scaling)

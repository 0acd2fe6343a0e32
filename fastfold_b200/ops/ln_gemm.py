"""LayerNorm and the GEMMs that read its rows, in one kernel each (csrc/ln_gemm.cu), without gradients.

``models/fastnn`` calls whole modules through the native functions below, which return None for tensors that the
kernels do not cover, and otherwise composes LayerNorm and GEMM; both give the same bits.  (The global column attention does not: its
mean query, which the composition rounds to bf16 three times, stays in 32 bits.)
"""
import torch
from torch.autograd import forward_ad
from torch.nn.modules import module as _nn_module

from . import _lib
from .layer_norm import LayerNorm

_known = {LayerNorm}


def stands_for(cls):
    """Class decorator: ``ready`` takes modules of exactly this class for what their parameters say."""
    _known.add(cls)
    return cls


def ready(*modules):
    """True when the kernels may stand for calls of ``modules``: no gradients or forward-mode level, and each of the modules that
    would be passed by is one of this package's own, unchanged - no subclass, parametrisation, replaced ``forward`` or hook.
    Whether the kernels cover the tensors is checked by the native functions, which return None where not."""
    if torch.is_grad_enabled() or forward_ad._current_level >= 0 or _nn_module._global_forward_hooks or _nn_module._global_forward_pre_hooks:
        return False
    for m in modules:
        if type(m) not in _known or m._forward_hooks or m._forward_pre_hooks or "forward" in m.__dict__:
            return False
    return True


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


def pair(x, norm, wa, ba, wb, bb, scale):
    """``(LN(x) wa^T + ba) * scale`` and the same with ``wb``, ``bb``; one factor per row."""
    return _lib.native().ln_pair(x, norm.weight, norm.bias, norm.eps, wa, ba, wb, bb, scale)


def transition(x, norm, l1, l2, inplace):
    return _lib.native().transition_module(x, norm.weight, norm.bias, norm.eps, l1.weight, l1.bias, l2.weight, l2.bias, inplace)


def attention(x, norm, wq, wg, bg, wo, bo, mask, H, D, scaling, transposed=False, chunk=None, inplace=False, pair_w=None, z=None, norm_z=None):
    """``x [1, A, B, C]`` plus the gated attention over ``norm(x)``: one kernel from the rows to QKV (and the pair bias
    ``pair_w . norm(x)``), the attention, and one kernel from the rows and its output to the result.  With ``z`` the pair bias is
    ``pair_w . norm_z(z)``."""
    zg, zb, ze = (None, None, 0.0) if z is None else (norm_z.weight, norm_z.bias, norm_z.eps)
    return _lib.native().attention_module(x, norm.weight, norm.bias, norm.eps, wq, wg, bg, wo, bo, mask, pair_w, z, zg, zb, ze, H, D, scaling, transposed,
                                          chunk or 0, inplace)


def triangle(z, norm1, w, b, gate, norm2, wo, bo, mask, outgoing, inplace):
    """Triangle multiplication in three kernels: the norm with the gated operands (channels first) and the output gate, the
    contraction, and the norm over its channels with the output projection, gate and residual."""
    return _lib.native().triangle_module(z, norm1.weight, norm1.bias, norm1.eps, w, b, gate.weight, gate.bias, norm2.weight, norm2.bias, norm2.eps, wo, bo,
                                         mask, outgoing, inplace)


def global_column_attention(x, norm, ga, mask, inplace):
    return _lib.native().global_column_module(x, norm.weight, norm.bias, norm.eps, ga.to_q.weight, ga.to_kv.weight, ga.gating_linear.weight, ga.gating_bias,
                                              ga.o_linear.weight, ga.o_linear.bias, mask, ga.scaling, inplace)


def masked_pair(x, norm, la, lb, mask):
    """``la(norm(x)) * mask`` and ``lb(norm(x)) * mask`` with one mask value per row, or None."""
    return _lib.native().masked_pair(x, norm.weight, norm.bias, norm.eps, la.weight, la.bias, lb.weight, lb.bias, mask)


def mask_norm(mask, eps):
    """``1 / (mask^T mask + eps)`` of ``mask [1, S, N]`` as ``[1, N, N, 1]`` in fp32, or None."""
    return _lib.native().mask_norm(mask, eps)

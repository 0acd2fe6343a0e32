"""Argument checks of the extension module: they come before any launch, so they need no GPU."""
import os

import pytest
import torch

from fastfold_b200 import _build
from fastfold_b200.ops import _lib

pytestmark = pytest.mark.skipif(not os.path.exists(_build.dispatch_path()), reason="extension module not built")


def _gemm(a, b, rowscale):
    return _lib.native().gemm(a, b, False, False, 1.0, None, 0, False, rowscale, None, None, 1, 1, None, False, None, False, 1, False, 0, None)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("batch,shape", [(0, (127,)), (0, (1, 16)), (3, (127,)), (3, (3, 127)), (3, (2, 128)), (3, (1, 128))])
def test_gemm_refuses_fewer_row_factors_than_rows(batch, shape, dtype):
    """The kernel reads one factor per row through a bare pointer."""
    a = torch.zeros(*([batch] if batch else []), 128, 64, dtype=torch.bfloat16)
    with pytest.raises(AssertionError, match="fewer row factors than rows"):
        _gemm(a, torch.zeros(64, 64, dtype=torch.bfloat16), torch.ones(shape, dtype=dtype))


def test_factors_and_masks_on_another_device_raise():
    """Their pointers would be read by a kernel of the other operands' device."""
    x = torch.zeros(128, 64, dtype=torch.bfloat16)
    with pytest.raises(AssertionError, match="another device"):
        _gemm(x, x[:64], torch.ones(128, device="meta"))
    qkv = torch.zeros(1, 4, 8, 3, 2, 16, dtype=torch.bfloat16)
    with pytest.raises(AssertionError, match="another device"):
        _lib.native().attention_packed_fwd(qkv, torch.ones(4, 8, dtype=torch.bfloat16, device="meta"), None, 8, 0.25, False, False)


def test_empty_extents_raise():
    """Integer division by an extent of 0 ends the process in native code; it raised in Python."""
    n, w = _lib.native(), torch.ones(0, dtype=torch.bfloat16)
    x = torch.empty(3, 0, dtype=torch.bfloat16)
    calls = [lambda: n.layer_norm_fwd(x, w, w, 1e-5, False), lambda: n.layer_norm_bwd(x, x, w, w.float(), w.float(), 1),
             lambda: n.bias_sigmoid_mul_fwd(x, w, x), lambda: n.bias_dropout_add_fwd(x, None, None, x, 1, 1), lambda: n.act_bwd(x, x, 1),
             lambda: n.gemm(torch.empty(32, 64).bfloat16(), torch.empty(32, 64).bfloat16(), False, False, 1.0, None, 0, False, None, None, None,
                            1, 1, None, False, None, False, 1, False, 0, [32, 32, 0, 1024, 1024, 1024])]
    for call in calls:
        with pytest.raises((AssertionError, RuntimeError)):        # RuntimeError: the stream, asked for first, needs a GPU
            call()


def _ipa_operands(N=6):
    b = lambda *s: torch.zeros(*s, dtype=torch.bfloat16)
    return {"q": b(N, 192), "kv": b(N, 384), "q_pts": b(N, 144), "kv_pts": b(N, 432), "rot": torch.zeros(N, 4), "is_quat": True, "trans": torch.zeros(N, 3),
            "z": b(N, N, 128), "wb": b(12, 128), "bb": b(12), "gamma": b(12), "mask": b(N)}


@pytest.mark.parametrize("name", ["q", "kv", "q_pts", "kv_pts", "z"])
@pytest.mark.parametrize("change", [lambda t: t[:-1], lambda t: t.float(), lambda t: t.transpose(0, 1), lambda t: t[..., :-1].contiguous(), lambda t: t.to("meta")],
                         ids=["rows", "type", "order", "columns", "device"])
def test_ipa_layer_refuses_operands_that_its_kernels_would_misread(name, change):
    """The kernels take the projections and the pair tensor as dense bf16 rows of fixed widths, as many as the pair tensor has."""
    args = _ipa_operands()
    args[name] = change(args[name])
    with pytest.raises(AssertionError, match="invariant point attention"):
        _lib.native().ipa_layer(*args.values(), 0.1, 0.5, 1e5, 1e-8)


def test_ipa_layer_refuses_host_memory():
    with pytest.raises(AssertionError, match="CUDA device"):
        _lib.native().ipa_layer(*_ipa_operands().values(), 0.1, 0.5, 1e5, 1e-8)

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

"""Lengths that are no multiple of 8: the fused no-grad path of every trunk module against the module in fp32 on the CPU."""
import copy

import pytest
import torch

from fastfold_b200.models.fastnn import ops as fops
from fastfold_b200.models.fastnn.msa import ExtraMSACore, MSAColumnAttention, MSARowAttentionWithPairBias
from fastfold_b200.models.fastnn.triangle import (TriangleAttentionEndingNode, TriangleAttentionStartingNode, TriangleMultiplicationIncoming,
                                                  TriangleMultiplicationOutgoing)
from fastfold_b200.ops import flash

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _random_parameters(mod):
    with torch.no_grad():
        for name, p in mod.named_parameters():
            p.normal_(std=p.shape[-1] ** -0.5 if p.dim() >= 2 else 0.1)
            if "norm" in name and name.endswith("weight"):
                p.add_(1.0)
    return mod.to(torch.bfloat16).float()        # weights that bf16 holds exactly


def _check(mod, inputs, call, tol=2e-2):
    """Relative 2-norm error of the module's update; bf16 roundings of a handful of chained tensors, 2^-9 each."""
    gpu = copy.deepcopy(mod).to(DEV, torch.bfloat16)
    with torch.no_grad():
        ref = call(mod, [t.float() for t in inputs])
        got = call(gpu, [t.to(DEV, torch.bfloat16) for t in inputs]).float().cpu()
    assert got.shape == ref.shape
    err = ((got - ref).norm() / ref.norm()).item()
    assert err < tol, err


def _masks(n, s=0):
    pm = torch.ones(1, n, n)
    pm[:, :, n - 3:] = 0
    pm[:, 1] = 0                                 # a row without any key: uniform weights over the true length
    if not s:
        return pm
    mm = torch.ones(1, s, n)
    mm[:, :, n - 2:] = 0
    mm[:, s // 2] = 0
    return pm, mm


@pytest.mark.parametrize("n", [33, 61, 68, 129, 203, 261])
@pytest.mark.parametrize("cls", [TriangleAttentionStartingNode, TriangleAttentionEndingNode, TriangleMultiplicationOutgoing, TriangleMultiplicationIncoming])
def test_pair_modules(cls, n, device_status):
    torch.manual_seed(n)
    att = cls in (TriangleAttentionStartingNode, TriangleAttentionEndingNode)
    mod = _random_parameters(cls(128, p_drop=0.25, c=32 if att else 128, **({"n_head": 4} if att else {}))).eval()
    _check(mod, [torch.randn(1, n, n, 128).bfloat16(), _masks(n)], lambda m, x: m(*x))
    fops.set_chunk_size(16)
    try:
        _check(mod, [torch.randn(1, n, n, 128).bfloat16(), _masks(n)], lambda m, x: m(*x))
    finally:
        fops.set_chunk_size(None)


@pytest.mark.parametrize("n", [16, 45, 64, 200, 320])
@pytest.mark.parametrize("cls", [TriangleAttentionStartingNode, TriangleAttentionEndingNode])
def test_sixteen_channel_heads(cls, n, device_status):
    """Heads of 16 channels (template pair stack) have their own instance of the forward attention kernel."""
    torch.manual_seed(n)
    mod = _random_parameters(cls(64, p_drop=0.25, c=16, n_head=4)).eval()
    _check(mod, [torch.randn(1, n, n, 64).bfloat16(), _masks(n)], lambda m, x: m(*x))


@pytest.mark.parametrize("n", [61, 130])
def test_triangle_multiplication_with_dropout_mask(n, device_status):
    """The first pass of activation checkpointing: no gradients, training mode, a mask shared along the first axis."""
    torch.manual_seed(n)
    mod = _random_parameters(TriangleMultiplicationOutgoing(128, p_drop=0.25, c=128)).train()
    drop = ((torch.rand(1, 1, n, 128) > 0.25).float() / 0.75).bfloat16()
    _check(mod, [torch.randn(1, n, n, 128).bfloat16(), _masks(n), drop], lambda m, x: m(*x))


@pytest.mark.parametrize("s,n", [(5, 33), (29, 61), (130, 71)])
def test_msa_modules(s, n, device_status):
    torch.manual_seed(s + n)
    pm, mm = _masks(n, s)
    m, z = torch.randn(1, s, n, 256).bfloat16(), torch.randn(1, n, n, 128).bfloat16()
    _check(_random_parameters(MSARowAttentionWithPairBias(256, 128)).eval(), [m, z, mm], lambda f, x: f(*x))
    _check(_random_parameters(MSAColumnAttention(256)).eval(), [m, mm], lambda f, x: f(*x))
    _check(_random_parameters(ExtraMSACore(64, 128)).eval(), [m[..., :64], z, mm], lambda f, x: f(*x))


@pytest.mark.parametrize("s,n", [(7, 2), (16, 3), (24, 33), (40, 77), (128, 100)])
def test_outer_product_mean(s, n, device_status):
    torch.manual_seed(s + n)
    mod = _random_parameters(fops.OutProductMean(256, 128, 32)).eval()
    _check(mod, [torch.randn(1, s, n, 256).bfloat16(), torch.ones(1, s, n), torch.randn(1, n, n, 128).bfloat16()], lambda m, x: m(*x))


@pytest.mark.parametrize("S,n", [(5, 16), (83, 24), (131, 40), (517, 8)])
def test_column_attention_gradients_for_any_number_of_sequences(S, n, device_status):
    torch.manual_seed(S)
    mod = _random_parameters(MSAColumnAttention(256)).eval()
    x, up = torch.randn(1, S, n, 256).bfloat16(), torch.randn(1, S, n, 256).bfloat16()
    mask = torch.ones(1, S, n)
    mask[:, S - S // 8:] = 0
    grads = []
    for dev, dt in (("cpu", torch.float32), (DEV, torch.bfloat16)):
        m = copy.deepcopy(mod).to(dev, dt)
        xi = x.to(dev, dt).requires_grad_(True)
        out = m(xi, mask.to(dev, dt))
        grads.append([out.float().cpu()] + [g.float().cpu() for g in torch.autograd.grad(out, [xi] + list(m.parameters()), up.to(dev, dt))])
    for a, b in zip(*grads):
        assert ((a - b).norm() / a.norm()).item() < 3e-2


def test_bias_pitch(device_status):
    """Every layout of the pair bias that the forward kernel takes gives the result of the contiguous one."""
    torch.manual_seed(0)
    H, n = 4, 75
    qkv = torch.randn(1, 6, n, 3, H, 32, device=DEV).bfloat16()
    bias = torch.randn(1, 1, H, n, n, device=DEV).bfloat16()
    with torch.no_grad():
        want = flash.flash_attention_packed(qkv, None, bias, 32 ** -0.5)
        for pitch in (80, 88, 200):
            wide = torch.full((1, 1, H, n, pitch), float("nan"), device=DEV, dtype=torch.bfloat16)
            wide[..., :n] = bias
            assert torch.equal(flash.flash_attention_packed(qkv, None, wide[..., :n], 32 ** -0.5), want)
        odd = torch.full((1, 1, H, n, 81), float("nan"), device=DEV, dtype=torch.bfloat16)
        odd[..., :n] = bias
        assert torch.equal(flash.flash_attention_packed(qkv, None, odd[..., :n], 32 ** -0.5), want)


@pytest.mark.parametrize("rows", [8, 56, 64, 72, 4096, 203 * 208])
@pytest.mark.parametrize("offset", [0.0, 30.0])
def test_channel_major_layer_norm_of_128_channels(rows, offset, device_status):
    """Tile edges, remainders and rows whose mean is large against their spread; bf16 output: 2^-8 of its range."""
    from fastfold_b200 import ops as K
    torch.manual_seed(rows)
    x = (torch.randn(128, rows, device=DEV) + offset).bfloat16()
    w, b = (1 + 0.1 * torch.randn(128, device=DEV)).bfloat16(), (0.1 * torch.randn(128, device=DEV)).bfloat16()
    ref = torch.nn.functional.layer_norm(x.double().t(), (128,), w.double(), b.double(), 1e-5)
    with torch.no_grad():
        out = K.layer_norm_transposed(x, w, b, 1e-5)
    assert (out.double() - ref).abs().max().item() <= 2.0 ** -8 * ref.abs().max().item()


@pytest.mark.parametrize("chunk", [1, 5, 16, 64])
@pytest.mark.parametrize("n", [24, 61])
def test_chunked_attention_is_the_unchunked_one(n, chunk, device_status):
    """Chunks that divide the rows or do not, in place and not, for every attention module (the block in-place mode writes
    each slice over its residual)."""
    torch.manual_seed(n)
    s = 37
    pm, mm = _masks(n, s)
    z, m = torch.randn(1, n, n, 128).bfloat16().to(DEV), torch.randn(1, s, n, 256).bfloat16().to(DEV)
    pm, mm = pm.bfloat16().to(DEV), mm.bfloat16().to(DEV)
    mods = [(TriangleAttentionStartingNode(128, p_drop=0.25, c=32, n_head=4), (z, pm)), (TriangleAttentionEndingNode(128, p_drop=0.25, c=32, n_head=4), (z, pm)),
            (MSARowAttentionWithPairBias(256, 128), (m, z, mm)), (MSAColumnAttention(256), (m, mm)),
            (TriangleAttentionEndingNode(128, p_drop=0.25, c=16, n_head=8), (z, pm))]
    for mod, args in mods:
        mod = _random_parameters(mod).eval().to(DEV, torch.bfloat16)
        with torch.no_grad():
            want = mod(*args).float()
            fops.set_chunk_size(chunk)
            try:
                got = mod(*args).float()
                with fops.inplace_scope():
                    first = args[0].clone()
                    over = mod(first, *args[1:])
            finally:
                fops.set_chunk_size(None)
        assert ((got - want).norm() / want.norm()).item() < 4e-3
        assert torch.equal(over.float(), got)


@pytest.mark.parametrize("chunk", [None, 16])
def test_inputs_stored_channel_first(chunk, device_status):
    """Residual inputs whose channels are not adjacent, at lengths that are no multiple of 8: the bits of dense ones."""
    torch.manual_seed(0)
    s, n = 29, 61
    pm, mm = (t.bfloat16().to(DEV) for t in _masks(n, s))
    z, m = torch.randn(1, n, n, 128, device=DEV).bfloat16(), torch.randn(1, s, n, 256, device=DEV).bfloat16()
    zt, mt = (t.movedim(-1, 1).contiguous().movedim(1, -1) for t in (z, m))
    mods = [(TriangleMultiplicationOutgoing(128, p_drop=0.25, c=128), (z, pm), (zt, pm)),
            (TriangleAttentionEndingNode(128, p_drop=0.25, c=32, n_head=4), (z, pm), (zt, pm)),
            (MSAColumnAttention(256), (m, mm), (mt, mm)), (fops.OutProductMean(256, 128, 32), (m, mm, z), (mt, mm, zt))]
    for mod, dense, strided in mods:
        mod = _random_parameters(mod).eval().to(DEV, torch.bfloat16)
        with torch.no_grad():
            fops.set_chunk_size(chunk)
            try:
                want, got = mod(*dense), mod(*strided)
            finally:
                fops.set_chunk_size(None)
        assert torch.equal(got, want), type(mod).__name__


@pytest.mark.parametrize("n", [33, 61])
def test_masks_that_broadcast(n, device_status):
    """Masks with an extent of 1 give the bits of the masks that they stand for."""
    torch.manual_seed(n)
    s = 29
    z, m = torch.randn(1, n, n, 128, device=DEV).bfloat16(), torch.randn(1, s, n, 256, device=DEV).bfloat16()
    tri = _random_parameters(TriangleMultiplicationIncoming(128, p_drop=0.25, c=128)).eval().to(DEV, torch.bfloat16)
    opm = _random_parameters(fops.OutProductMean(256, 128, 32)).eval().to(DEV, torch.bfloat16)
    with torch.no_grad():
        for shape in ((1, 1, n), (1, n, 1), (1, 1, 1)):
            mask = (torch.rand(shape, device=DEV) > 0.2).bfloat16()
            assert torch.equal(tri(z, mask), tri(z, mask.expand(1, n, n).contiguous()))
        mask = (torch.rand(1, s, 1, device=DEV) > 0.2).bfloat16()
        mask[:, 0] = 1
        assert torch.equal(opm(m, mask, z), opm(m, mask.expand(1, s, n).contiguous(), z))


@pytest.mark.parametrize("n", [61, 64])
def test_biases_of_another_type_or_extent(n, device_status):
    """A pair bias in fp32, and one that all heads share, next to the bf16 ``[1, H, n, n]`` that the kernel reads.  bf16 roundings
    of the logits (2^-9 of up to 8) and of the output."""
    torch.manual_seed(n)
    att = _random_parameters(fops.SelfAttention(qkv_dim=128, c=32, n_head=4, out_dim=128)).eval().to(DEV, torch.bfloat16)
    x, mask = torch.randn(1, 9, n, 128, device=DEV).bfloat16(), torch.ones(1, 9, n, device=DEV).bfloat16()
    shared = torch.randn(1, 1, n, n, device=DEV).bfloat16()
    bias = shared.expand(1, 4, n, n).contiguous()
    with torch.no_grad():
        want = att(x, mask, (bias, -1))[0].float()
        for b in (bias.float(), shared):
            got = att(x, mask, (b, -1))[0].float()
            assert ((got - want).norm() / want.norm()).item() < 2e-2


@pytest.mark.parametrize("n", [24, 32])
def test_outer_product_mean_with_only_its_bias_trainable(n, device_status):
    torch.manual_seed(n)
    mod = _random_parameters(fops.OutProductMean(256, 128, 32)).to(DEV, torch.bfloat16).requires_grad_(False)
    mod.o_linear.bias.requires_grad_(True)
    m, z, mask = torch.randn(1, 8, n, 256, device=DEV).bfloat16(), torch.randn(1, n, n, 128, device=DEV).bfloat16(), torch.ones(1, 8, n, device=DEV)
    up = torch.randn(1, n, n, 128, device=DEV).bfloat16()
    (grad,) = torch.autograd.grad(mod(m, mask.bfloat16(), z), [mod.o_linear.bias], up)
    want = up.float().sum((0, 1, 2)) / (8 + 1e-3)                  # 1 / (sequences + 1e-3) for every pair
    assert ((grad.float() - want).norm() / want.norm()).item() < 2e-2


@pytest.mark.parametrize("s,n", [(7, 33), (40, 77), (64, 64), (128, 100)])
def test_outer_product_mean_with_masks(s, n, device_status):
    """Whole sequences, whole residues and single positions masked: every row of both projections has its own mask value.
    Pairs without a common sequence are divided by 1e-3, so their update is that of the bias."""
    torch.manual_seed(s * n)
    mod = _random_parameters(fops.OutProductMean(256, 128, 32)).eval()
    mask = (torch.rand(1, s, n) > 0.3).float()
    mask[:, s // 2] = 0
    mask[:, :, n // 3] = 0
    m, z = torch.randn(1, s, n, 256).bfloat16(), torch.randn(1, n, n, 128).bfloat16()
    _check(mod, [m, mask, z], lambda f, x: f(*x))
    both = mask[0].t() @ mask[0] > 0                              # and the pairs that have one, where the operands matter
    _check(mod, [m, mask, z], lambda f, x: (f(*x) - x[2])[0][both.to(x[0].device)])


@pytest.mark.parametrize("n", [1, 2, 5, 9, 17])
def test_a_few_residues(n, device_status):
    """The smallest lengths of every pair and MSA module: extents below a tile, a vector and a warp."""
    torch.manual_seed(n)
    pm, mm = torch.ones(1, n, n), torch.ones(1, 3, n)
    z, m = torch.randn(1, n, n, 128).bfloat16(), torch.randn(1, 3, n, 256).bfloat16()
    for cls in (TriangleAttentionStartingNode, TriangleAttentionEndingNode, TriangleMultiplicationOutgoing, TriangleMultiplicationIncoming):
        att = cls in (TriangleAttentionStartingNode, TriangleAttentionEndingNode)
        mod = _random_parameters(cls(128, p_drop=0.25, c=32 if att else 128, **({"n_head": 4} if att else {}))).eval()
        _check(mod, [z, pm], lambda f, x: f(*x))
    _check(_random_parameters(MSARowAttentionWithPairBias(256, 128)).eval(), [m, z, mm], lambda f, x: f(*x))
    _check(_random_parameters(MSAColumnAttention(256)).eval(), [m, mm], lambda f, x: f(*x))
    _check(_random_parameters(ExtraMSACore(64, 128)).eval(), [m[..., :64], z, mm], lambda f, x: f(*x))
    _check(_random_parameters(fops.OutProductMean(256, 128, 32)).eval(), [m, mm, z], lambda f, x: f(*x))


def test_widths_that_are_no_multiple_of_8(device_status):
    """The GEMM reads rows at a pitch of 16 bytes; layers of other widths are the library's."""
    torch.manual_seed(0)
    s, n = 9, 61
    m, z, mask = torch.randn(1, s, n, 20).bfloat16(), torch.randn(1, n, n, 128).bfloat16(), torch.ones(1, s, n)
    _check(_random_parameters(fops.OutProductMean(20, 128, 32)).eval(), [m, mask, z], lambda f, x: f(*x))
    _check(_random_parameters(fops.SelfAttention(qkv_dim=20, c=8, n_head=4, out_dim=64, gating=False)).eval(), [m, mask], lambda f, x: f(*x)[0])


@pytest.mark.parametrize("n", [61, 64])
def test_triangle_multiplication_with_fp32_norms(n, device_status):
    """Norm parameters kept in fp32 next to bf16 activations: the kernels take one type only, other parameters are converted."""
    torch.manual_seed(n)
    mod = _random_parameters(TriangleMultiplicationOutgoing(128, p_drop=0.25, c=128)).eval().to(DEV, torch.bfloat16)
    z, mask = torch.randn(1, n, n, 128, device=DEV).bfloat16(), torch.ones(1, n, n, device=DEV).bfloat16()
    with torch.no_grad():
        want = mod(z, mask).float()
        mod.layernorm1.float()
        mod.layernorm2.float()
        got = mod(z, mask).float()
    assert ((got - want).norm() / want.norm()).item() < 1e-2


@pytest.mark.parametrize("n", [61, 64])
def test_dropout_masks_in_fp32(n, device_status):
    """The first pass of activation checkpointing with a mask of another type than the activations."""
    torch.manual_seed(n)
    z, mask = torch.randn(1, n, n, 128, device=DEV).bfloat16(), torch.ones(1, n, n, device=DEV).bfloat16()
    for mod, shape in ((TriangleMultiplicationOutgoing(128, p_drop=0.25, c=128), (1, 1, n, 128)),
                       (TriangleAttentionEndingNode(128, p_drop=0.25, c=32, n_head=4), (1, n, 1, 128))):
        mod = _random_parameters(mod).train().to(DEV, torch.bfloat16)
        drop = (torch.rand(shape, device=DEV) > 0.25).float() * 1.25             # 1.25 is a bf16 value
        with torch.no_grad():
            assert torch.equal(mod(z, mask, drop), mod(z, mask, drop.bfloat16()))


@pytest.mark.parametrize("n", [40, 64])
def test_outer_product_mean_of_an_fp32_msa(n, device_status):
    """An fp32 module and MSA next to a bf16 pair tensor."""
    torch.manual_seed(n)
    mod = _random_parameters(fops.OutProductMean(256, 128, 32)).eval().to(DEV)
    m, z, mask = torch.randn(1, 9, n, 256, device=DEV), torch.randn(1, n, n, 128, device=DEV).bfloat16(), torch.ones(1, 9, n, device=DEV)
    with torch.no_grad():
        want = mod(m, mask, z.float())
        got = mod(m, mask, z).float()
    assert ((got - want).norm() / want.norm()).item() < 1e-2

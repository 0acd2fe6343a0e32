"""Fast (DAP-aware) modules against the OpenFold-layout modules they replace, one module per test, with and without
chunking - the module list of the reference's tests/test_fastnn/ (test_msa_att_row, test_msa_att_col,
test_msa_global_att_col, test_out_product_mean, test_evoformer_stack, test_extramsa_stack), on the CPU in fp32.
The fast modules return the residual stream (input + update); the OpenFold-layout modules return the update."""
import pytest
import torch

from fastfold_b200.models import fastnn
from fastfold_b200.models import nn as ref
from fastfold_b200.models.fastnn import ops as fops
from fastfold_b200.models.nn.evoformer import EvoformerStack as RefEvoformerStack, ExtraMSAStack as RefExtraMSAStack
from fastfold_b200.models.nn.msa import MSAColumnAttention, MSAColumnGlobalAttention, MSARowAttentionWithPairBias
from fastfold_b200.models.nn.pair import OuterProductMean
import importlib

inj = importlib.import_module("fastfold_b200.utils.inject_fastnn")          # ``fastfold_b200.utils.inject_fastnn`` is also a function

S, N, C_M, C_Z = 6, 10, 32, 16


@pytest.fixture(autouse=True)
def _reset_chunk():
    yield
    fops.set_chunk_size(None)


def _randomize(module, seed):
    g = torch.Generator().manual_seed(seed)
    with torch.no_grad():
        for p in module.parameters():
            p.copy_(torch.randn(p.shape, generator=g) * 0.2)
    return module.eval()


def _inputs(seed=0):
    g = torch.Generator().manual_seed(seed)
    m = torch.randn(S, N, C_M, generator=g)
    z = torch.randn(N, N, C_Z, generator=g)
    msa_mask = (torch.rand(S, N, generator=g) > 0.15).float()
    msa_mask[0] = 1
    pair_mask = (torch.rand(N, N, generator=g) > 0.1).float()
    return m, z, msa_mask, pair_mask


@pytest.mark.parametrize("chunk", [None, 4])
def test_msa_att_row(chunk):
    m, z, msa_mask, _ = _inputs()
    ori = _randomize(MSARowAttentionWithPairBias(C_M, C_Z, 8, 4), 1)
    fast = fastnn.msa.MSARowAttentionWithPairBias(d_node=C_M, d_pair=C_Z, c=8, n_head=4).eval()
    inj._copy_row_attention(fast, ori)
    fops.set_chunk_size(chunk)
    with torch.no_grad():
        want = m + ori(m, z=z, mask=msa_mask, chunk_size=chunk)
        got = fast(m[None], z[None], msa_mask[None])[0]
    assert (got - want).abs().max() < 2e-5


@pytest.mark.parametrize("chunk", [None, 4])
def test_msa_att_col(chunk):
    m, _, msa_mask, _ = _inputs(1)
    ori = _randomize(MSAColumnAttention(C_M, 8, 4), 2)
    fast = fastnn.msa.MSAColumnAttention(d_node=C_M, c=8, n_head=4).eval()
    inj._copy_layernorm(fast.layernormM, ori._msa_att.layer_norm_m)
    inj._copy_attention(fast.attention, ori._msa_att.mha)
    fops.set_chunk_size(chunk)
    with torch.no_grad():
        want = m + ori(m, mask=msa_mask, chunk_size=chunk)
        got = fast(m[None], msa_mask[None])[0]
    assert (got - want).abs().max() < 2e-5


@pytest.mark.parametrize("chunk", [None, 4])
def test_msa_global_att_col(chunk):
    m, _, msa_mask, _ = _inputs(2)
    ori = _randomize(MSAColumnGlobalAttention(C_M, 8, 4), 3)
    fast = fastnn.msa.MSAColumnGlobalAttention(d_node=C_M, c=8, n_head=4).eval()
    inj._copy_layernorm(fast.layernormM, ori.layer_norm_m)
    inj._copy_global_attention(fast.global_attention, ori.global_attention)
    fops.set_chunk_size(chunk)
    with torch.no_grad():
        want = m + ori(m, mask=msa_mask, chunk_size=chunk)
        got = fast(m[None], msa_mask[None])[0]
    assert (got - want).abs().max() < 2e-5


@pytest.mark.parametrize("chunk", [None, 4])
def test_out_product_mean(chunk):
    m, z, msa_mask, _ = _inputs(3)
    ori = _randomize(OuterProductMean(C_M, C_Z, 8), 4)
    fast = fastnn.ops.OutProductMean(n_feat=C_M, n_feat_out=C_Z, n_feat_proj=8).eval()
    inj._copy_layernorm(fast.layernormM, ori.layer_norm)
    inj._copy_linear(fast.linear_a, ori.linear_1)
    inj._copy_linear(fast.linear_b, ori.linear_2)
    inj._copy_linear(fast.o_linear, ori.linear_out)
    fops.set_chunk_size(chunk)
    with torch.no_grad():
        want = z + ori(m, mask=msa_mask, chunk_size=chunk)
        got = fast(m[None], msa_mask[None], z[None])[0]
    assert (got - want).abs().max() < 2e-5


def _stack_cfg(c_hidden_msa_att):
    # hidden sizes of the published model (the fast modules are built for them); small c_m / c_z keep the test quick
    return dict(c_m=C_M, c_z=C_Z, c_hidden_msa_att=c_hidden_msa_att, c_hidden_opm=32, c_hidden_mul=C_Z, c_hidden_pair_att=C_Z // 4, no_heads_msa=8,
                no_heads_pair=4, transition_n=4, msa_dropout=0.15, pair_dropout=0.25, inf=1e9, eps=1e-8)


@pytest.mark.parametrize("chunk", [None, 4])
def test_evoformer_stack(chunk):
    m, z, msa_mask, pair_mask = _inputs(4)
    ori = _randomize(RefEvoformerStack(c_s=24, no_blocks=3, blocks_per_ckpt=None, clear_cache_between_blocks=False, **_stack_cfg(32)), 5)
    fast = fastnn.EvoformerStack(c_m=C_M, c_z=C_Z, c_s=24, no_blocks=3, blocks_per_ckpt=None).eval()
    for fb, ob in zip(fast.blocks, ori.blocks):
        inj.copy_evoformer_block(fb, ob)
    inj._copy_linear(fast.linear, ori.linear)
    fops.set_chunk_size(chunk)
    with torch.no_grad():
        m1, z1, s1 = ori(m, z, msa_mask=msa_mask, pair_mask=pair_mask, chunk_size=chunk, _mask_trans=False)   # as the model config sets it
        m2, z2, s2 = fast(m, z, msa_mask=msa_mask, pair_mask=pair_mask, chunk_size=chunk, _mask_trans=False)
    for a, b in ((m1, m2), (z1, z2), (s1, s2)):          # the reference's gate: mean absolute difference below 2e-3
        assert torch.isfinite(b).all() and (a - b).abs().mean() < 2e-3 * max(1.0, float(a.abs().mean()))


@pytest.mark.parametrize("chunk", [None, 4])
def test_extramsa_stack(chunk):
    m, z, msa_mask, pair_mask = _inputs(5)
    ori = _randomize(RefExtraMSAStack(no_blocks=2, ckpt=False, clear_cache_between_blocks=False, **_stack_cfg(8)), 6)
    fast = fastnn.ExtraMSAStack(c_m=C_M, c_z=C_Z, no_blocks=2).eval()
    for fb, ob in zip(fast.blocks, ori.blocks):
        inj.copy_extra_msa_block(fb, ob)
    fops.set_chunk_size(chunk)
    with torch.no_grad():
        z1 = ori(m, z, chunk_size=chunk, msa_mask=msa_mask, pair_mask=pair_mask, _mask_trans=False)
        z2 = fast(m, z, chunk_size=chunk, msa_mask=msa_mask, pair_mask=pair_mask, _mask_trans=False)
    assert torch.isfinite(z2).all() and (z1 - z2).abs().mean() < 2e-3 * max(1.0, float(z1.abs().mean()))


@pytest.mark.parametrize("c", [8, 16, 24, 32, 40, 64])
def test_chunked_attention_takes_any_head_width(c, monkeypatch):
    """Chunked rows without gradients where the fused path may be tried: head widths that its kernels do not have - wider ones
    among them - give what the plain evaluation gives."""
    monkeypatch.setattr(fops, "_fusable", lambda x: not torch.is_grad_enabled())
    torch.manual_seed(c)
    att = fops.SelfAttention(qkv_dim=64, c=c, n_head=2, out_dim=64).eval()
    with torch.no_grad():
        for p in att.parameters():
            p.normal_(std=0.1)
        x, mask = torch.randn(1, 7, 12, 64), torch.ones(1, 7, 12)
        mask[..., 9:] = 0
        want = att(x, mask)[0]
        fops.set_chunk_size(3)
        try:
            got = att(x, mask)[0]
        finally:
            fops.set_chunk_size(None)
    torch.testing.assert_close(got, want, rtol=1e-4, atol=1e-5)


def test_stack_entry_passes_on_only_what_needs_no_copy():
    """Evoformer and extra-MSA stacks hand their input on without a copy only where it is dense, 16-byte aligned, not needed
    by a backward pass and not written over."""
    from fastfold_b200.models.fastnn.triangle import pad_or_pass
    flat = torch.randn(8 * 16 * 32 + 8).bfloat16()
    start = (-flat.data_ptr() // 2) % 8                       # first 16-byte boundary
    dense = flat[start:start + 4096].view(1, 8, 16, 32)
    views = {"off the boundary": flat[start + 1:start + 4097].view(1, 8, 16, 32), "every other channel": dense[..., ::2],
             "expanded channel": dense[..., :1].expand(1, 8, 16, 8), "channels first": dense.permute(0, 1, 3, 2)}
    with torch.no_grad():
        assert pad_or_pass(dense, (0, 0, 0, 0)).data_ptr() == dense.data_ptr()
        for name, v in views.items():
            out = pad_or_pass(v, (0, 0, 0, 0))
            assert torch.equal(out, v) and out.data_ptr() != v.data_ptr() and out.data_ptr() % 16 == 0, name
        assert pad_or_pass(dense, (0, 0, 0, 2)).shape == (1, 8, 18, 32)
        with fops.inplace_scope():
            assert pad_or_pass(dense, (0, 0, 0, 0)).data_ptr() != dense.data_ptr()
    kept = dense.detach().requires_grad_(True)
    assert pad_or_pass(kept, (0, 0, 0, 0)).data_ptr() != dense.data_ptr()


class _Forwarding(torch.nn.Module):
    """A module around another that only passes the call on."""

    def __init__(self, inner):
        super().__init__()
        self.inner = inner

    def forward(self, *args, **kw):
        return self.inner(*args, **kw)


@pytest.mark.parametrize("grad", [False, True])
@pytest.mark.parametrize("which", ["row", "column", "start", "end"])
def test_wrapped_attention(which, grad):
    """The attention of a module may be any module: nothing but the call is asked of it."""
    m, z, msa_mask, pair_mask = _inputs(3)
    if which == "row":
        net = _randomize(fastnn.msa.MSARowAttentionWithPairBias(d_node=C_M, d_pair=C_Z, c=8, n_head=4), 1)
        args = (m[None], z[None], msa_mask[None])
    elif which == "column":
        net, args = _randomize(fastnn.msa.MSAColumnAttention(d_node=C_M, c=8, n_head=4), 1), (m[None], msa_mask[None])
    else:
        cls = fops.ChunkTriangleAttentionStartingNode if which == "start" else fops.ChunkTriangleAttentionEndingNode
        net, args = _randomize(cls(C_Z, p_drop=0.0, c=8, n_head=2), 1), (z[None], pair_mask[None])
    with torch.set_grad_enabled(grad):
        want = net(*args)
        net.attention = _Forwarding(net.attention)
        assert torch.equal(net(*args), want)


def _change(module, name, how):
    """Other values in one parameter of a module in evaluation."""
    with torch.no_grad():
        old = getattr(module, name)
        if how == "in place":
            old.add_(1.0)
        elif how == "data":
            old.data = old.data + 1.0
        else:                                    # another tensor with the same version count
            setattr(module, name, torch.nn.Parameter(old + 1.0))


@pytest.mark.parametrize("how", ["in place", "data", "replaced"])
@pytest.mark.parametrize("which", ["to_qkv.weight", "gating_linear.weight", "gating_bias", "o_linear.weight"])
def test_widened_heads_follow_their_parameters(which, how):
    """The widened weights of narrow heads, kept in evaluation, are built again when any of the parameters changes."""
    torch.manual_seed(0)
    net = fops.SelfAttention(qkv_dim=64, c=8, n_head=4, out_dim=64).eval()
    first = net._padded_heads(16)
    assert all(a is b for a, b in zip(net._padded_heads(16), first))
    owner = net if "." not in which else getattr(net, which.split(".")[0])
    _change(owner, which.split(".")[-1], how)
    got = net._padded_heads(16)
    net._pad_cache = None
    for a, b in zip(got, net._padded_heads(16)):
        assert torch.equal(a, b)


@pytest.mark.parametrize("how", ["in place", "data", "replaced"])
@pytest.mark.parametrize("name", ["weight", "bias"])
@pytest.mark.parametrize("which", ["left_right_projection", "left_right_gate"])
def test_gated_weights_follow_their_parameters(which, name, how):
    torch.manual_seed(0)
    net = fops.AsyncChunkTriangleMultiplicationOutgoing(16, p_drop=0.0, c=16).eval()
    first = net._glu_weights()
    assert all(a is b for a, b in zip(net._glu_weights(), first))
    _change(getattr(net, which), name, how)
    got = net._glu_weights()
    net._glu_cache = None
    for a, b in zip(got, net._glu_weights()):
        assert torch.equal(a, b)

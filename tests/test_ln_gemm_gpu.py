"""LayerNorm + GEMM kernels (csrc/ln_gemm.cu) and the column kernel of global_attention.cu against the separate kernels, whose bits the
former give, and against the same mathematics in 64 bits with the roundings to bf16 that the kernels make (normalised rows, hidden
activation) made there too.  Bound: what is left are the fp32 sums and the rounding of the result, 2^-9 of each value at most, so 2^-9 in
the 2-norm; a normalised or hidden value that rounds the other way adds less than that again."""
import pytest
import torch

from fastfold_b200.models.fastnn import ops as fops
from fastfold_b200.models.fastnn.msa import MSAColumnAttention
from fastfold_b200.ops import LayerNorm, ln_gemm

pytestmark = pytest.mark.gpu
DEV = "cuda"
TOL = 2.0 ** -8


def _randn(*shape, scale=1.0):
    return (torch.randn(*shape, device=DEV) * scale).to(torch.bfloat16)


def _norm(C):
    norm = LayerNorm(C).to(DEV, torch.bfloat16).requires_grad_(False)
    norm.weight.copy_(1 + 0.1 * torch.randn(C, device=DEV))
    norm.bias.copy_(0.1 * torch.randn(C, device=DEV))
    return norm


def _ln(x, norm):
    y = torch.nn.functional.layer_norm(x.double(), (x.shape[-1],), norm.weight.double(), norm.bias.double(), norm.eps)
    return y.bfloat16().double()


def _close(a, ref):
    assert a.shape == ref.shape
    assert torch.isfinite(a.float()).all()
    assert (a.double() - ref).norm() <= TOL * ref.norm()


def _lin(x, w, b=None):
    y = x @ w.double().t()
    return y if b is None else y + b.double()


@pytest.mark.parametrize("C", [64, 128, 256])
@pytest.mark.parametrize("M", [1, 31, 128, 129, 19000, 60007])
def test_chains(C, M, device_status):
    """Transition and gated output: less than a tile, a whole one, a remainder of one row, more tiles than CTAs, several per CTA; one and
    two chunks of gated columns; the result over the residual."""
    torch.manual_seed(C + M)
    with torch.no_grad():
        x, norm, H = _randn(M, C), _norm(C), 4 * C
        w1, b1, w2, b2 = _randn(H, C, scale=C ** -0.5), _randn(H, scale=0.1), _randn(C, H, scale=H ** -0.5), _randn(C, scale=0.1)
        X = _ln(x, norm)
        _close(ln_gemm.chain(x, norm, w1, b1, w2, b2, x), x.double() + _lin(torch.relu(_lin(X, w1, b1)).bfloat16().double(), w2, b2))
        for G in (128, 256):
            o, wg, bg, wo = _randn(M, G), _randn(G, C, scale=C ** -0.5), _randn(G, scale=0.1), _randn(C, G, scale=G ** -0.5)
            ref = x.double() + _lin((torch.sigmoid(_lin(X, wg, bg)) * o.double()).bfloat16().double(), wo)
            _close(ln_gemm.chain(x, norm, wg, bg, wo, None, x, mul=o), ref)
        y = x.clone()
        assert ln_gemm.chain(y, norm, wg, bg, wo, None, y, mul=o, out=y).data_ptr() == y.data_ptr()
        _close(y, ref)


@pytest.mark.parametrize("batch,rows", [(5, 64), (7, 32), (3, 16), (6, 96), (4, 200), (2, 1)])
def test_rows_in_batches(batch, rows, device_status):
    """Slices of columns: two or four batches share a tile (64 and 32 rows), one otherwise; nothing outside the slice is written."""
    torch.manual_seed(batch * rows)
    with torch.no_grad():
        whole, norm = _randn(batch, rows + 24, 128), _norm(128)
        x = whole[:, 8:8 + rows]
        w, b, wo, o = _randn(128, 128, scale=0.09), _randn(128, scale=0.1), _randn(128, 128, scale=0.09), _randn(batch, rows, 128)
        out = torch.zeros_like(whole)
        X = _ln(x, norm)
        ln_gemm.chain(x, norm, w, b, wo, b, x, mul=o, out=out[:, 8:8 + rows])
        _close(out[:, 8:8 + rows], x.double() + _lin((torch.sigmoid(_lin(X, w, b)) * o.double()).bfloat16().double(), wo, b))
        assert not out[:, :8].any() and not out[:, 8 + rows:].any()
        _close(ln_gemm.qkv(x, norm, w), _lin(X, w))


@pytest.mark.parametrize("C,n", [(128, 5), (128, 16), (128, 77), (128, 130), (64, 33), (256, 40)])
@pytest.mark.parametrize("transposed", [False, True])
def test_qkv_and_pair_bias(C, n, transposed, device_status):
    torch.manual_seed(n)
    with torch.no_grad():
        z, norm, w, wb = _randn(n, n, C), _norm(C), _randn(384, C, scale=C ** -0.5), _randn(8, C, scale=C ** -0.5)
        buf = torch.full((8, n, (n + 7) // 8 * 8), 7.0, device=DEV, dtype=torch.bfloat16)
        y = ln_gemm.qkv(z.view(-1, C), norm, w, wb, buf[:, :, :n], transposed)
        X = _ln(z, norm)
        _close(y.view(n, n, -1), _lin(X, w))
        _close(buf[:, :, :n], _lin(X, wb).permute(2, 1, 0) if transposed else _lin(X, wb).permute(2, 0, 1))
        assert (buf[:, :, n:] == 7.0).all()


def _close_blocks(a, ref, rows=32, cols=64):
    """The bound in the 2-norm, for every tile that an epilogue warp stores: one that holds values of another stays far below it in the whole."""
    pad = (0, -a.shape[1] % cols, 0, -a.shape[0] % rows)
    cut = lambda t: torch.nn.functional.pad(t.double(), pad).unfold(0, rows, rows).unfold(1, cols, cols)  # noqa: E731
    assert ((cut(a) - cut(ref)).norm(dim=(2, 3)) <= TOL * cut(ref).norm(dim=(2, 3))).all()


@pytest.mark.parametrize("C,n", [(64, 203), (128, 203), (128, 256), (128, 389)])
@pytest.mark.parametrize("transposed", [False, True])
def test_tiles_without_a_store(C, n, transposed, device_status):
    """Two to eight tiles per CTA, one chunk of four without a store (the pair bias) and a last tile that ends between two warps: the
    staging tiles are filled again in another order than one by one.  The same bits every time."""
    torch.manual_seed(n)
    with torch.no_grad():
        z, norm, w, wb = _randn(n * n, C), _norm(C), _randn(384, C, scale=C ** -0.5), _randn(4, C, scale=C ** -0.5)
        X = _ln(z, norm)
        ref, ref_b = _lin(X, w), _lin(X, wb).view(n, n, 4)
        first = None
        for _ in range(6):
            bias = torch.empty(4, n, (n + 7) // 8 * 8, device=DEV, dtype=torch.bfloat16)[:, :, :n]
            y = ln_gemm.qkv(z, norm, w, wb, bias, transposed)
            if first is None:
                first = (y, bias)
                _close_blocks(y, ref)
                _close(bias, ref_b.permute(2, 1, 0) if transposed else ref_b.permute(2, 0, 1))
            assert torch.equal(y, first[0]) and torch.equal(bias, first[1])


@pytest.mark.parametrize("n", [131, 203, 301])
def test_partial_tiles_in_batches(n, device_status):
    """Odd lengths of the triangle multiplication: five chunks a tile, a partial tile in every row of the pair tensor whose last warps
    store nothing, several tiles per CTA.  The gated operands against 64 bits, block by block; the same bits every time."""
    torch.manual_seed(n)
    with torch.no_grad():
        z, norm, w, b = _randn(n, n, 128), _norm(128), _randn(512, 128, scale=0.09), _randn(512, scale=0.1)
        wg, bg, mask = _randn(128, 128, scale=0.09), _randn(128, scale=0.1), (torch.rand(n * n, device=DEV) > 0.2).to(torch.bfloat16)
        X = _ln(z, norm)
        pre = _lin(X, w, b)
        lr_ref = (pre[..., 0::2] * torch.sigmoid(pre[..., 1::2]) * mask.double().view(n, n, 1)).permute(2, 0, 1)
        first = None
        for _ in range(6):
            lr = torch.zeros(256, n, (n + 7) // 8 * 8, device=DEV, dtype=torch.bfloat16)[:, :, :n]
            gate = ln_gemm.tri_in(z, norm, w, b, wg, bg, mask, lr)
            if first is None:
                first = (lr, gate)
                for i in range(n):
                    _close_blocks(lr[:, i], lr_ref[:, i], 32, 32)
                _close_blocks(gate.view(n * n, 128), torch.sigmoid(_lin(X, wg, bg)).view(n * n, 128))
            assert torch.equal(lr, first[0]) and torch.equal(gate, first[1])


@pytest.mark.parametrize("M,dtype", [(3, torch.bfloat16), (300, torch.float32), (5000, torch.bfloat16), (60007, torch.float32)])
@pytest.mark.parametrize("C", [64, 256])
def test_pair_of_projections(C, M, dtype, device_status):
    torch.manual_seed(M)
    with torch.no_grad():
        x, norm, s = _randn(M, C), _norm(C), torch.rand(M, device=DEV).to(dtype)
        ws = [_randn(32, C, scale=C ** -0.5) for _ in range(2)]
        bs = [_randn(32, scale=0.1) for _ in range(2)]
        for y, w, b in zip(ln_gemm.pair(x, norm, ws[0], bs[0], ws[1], bs[1], s), ws, bs):
            _close(y, _lin(_ln(x, norm), w, b) * s.double()[:, None])


@pytest.mark.parametrize("S,N", [(1, 1), (7, 64), (32, 65), (33, 130), (100, 200)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_mask_normaliser(S, N, dtype, device_status):
    """fp32 sums of at most 100 products of values in [0, 1], one reciprocal: 100 x 2^-24 relative, and 2 ulp."""
    torch.manual_seed(N)
    mask = torch.rand(1, S, N, device=DEV).to(dtype)
    ref = 1.0 / (mask[0].double().t() @ mask[0].double() + 1e-3)
    out = ln_gemm.mask_norm(mask, 1e-3)
    assert out.shape == (1, N, N, 1)
    assert ((out[0, :, :, 0].double() - ref).abs() <= 1e-5 * ref).all()
    assert ln_gemm.mask_norm(mask[0], 1e-3) is None and ln_gemm.mask_norm(mask.double(), 1e-3) is None


def _randomise(net):
    for p in net.parameters():
        p.copy_(torch.randn_like(p) * (p.shape[-1] ** -0.5 if p.dim() == 2 else 0.1) + (1.0 if p.dim() == 1 and p.float().mean() > 0.5 else 0.0))


@pytest.mark.parametrize("n", [1, 8, 27, 64, 131, 200])
@pytest.mark.parametrize("cls", [fops.AsyncChunkTriangleMultiplicationOutgoing, fops.AsyncChunkTriangleMultiplicationIncoming])
def test_triangle_multiplication(cls, n, device_status):
    """The three-kernel path against the layer in 64 bits (its roundings are not restated here: operands, their product, its norm and
    the gate are rounded to bf16, 2^-9 each, and the update is added to a residual of about its size)."""
    torch.manual_seed(n)
    net = cls(128, p_drop=0.25).to(DEV, torch.bfloat16).eval().requires_grad_(False)
    with torch.no_grad():
        _randomise(net)
        z, mask = _randn(1, n, n, 128), (torch.rand(1, n, n, device=DEV) > 0.2).to(torch.bfloat16)
        assert net._from_raw(z, mask) is not None
        P = {k: v.double() for k, v in net.named_parameters()}
        lin = lambda x, name: torch.nn.functional.linear(x, P[name + ".weight"], P.get(name + ".bias"))  # noqa: E731
        ln = lambda x, name: torch.nn.functional.layer_norm(x, (128,), P[name + ".weight"], P[name + ".bias"], 1e-5)  # noqa: E731
        x = ln(z[0].double(), "layernorm1")
        a, b = (lin(x, "left_right_projection") * torch.sigmoid(lin(x, "left_right_gate")) * mask[0].double()[..., None]).chunk(2, -1)
        p = torch.einsum("ikc,jkc->ijc", a, b) if net.outgoing else torch.einsum("kic,kjc->ijc", a, b)
        ref = z.double() + torch.sigmoid(lin(x, "output_gate")) * (lin(ln(p, "layernorm2"), "output_projection") + P["output_bias"])
        out = net(z, mask)
        assert (out.double() - ref).norm() <= 4 * TOL * ref.norm()


@pytest.mark.parametrize("n", [16, 27])
def test_masks_of_other_shapes(n, device_status):
    """A mask with an axis more, and one that broadcasts, give what the mask of the pair tensor's shape gives."""
    torch.manual_seed(n)
    net = fops.AsyncChunkTriangleMultiplicationOutgoing(128, p_drop=0.25).to(DEV, torch.bfloat16).eval().requires_grad_(False)
    with torch.no_grad():
        _randomise(net)
        z, row = _randn(1, n, n, 128), (torch.rand(1, 1, n, device=DEV) > 0.2).to(torch.bfloat16)
        whole = row.expand(1, n, n).contiguous()
        ref = net._from_raw(z, whole)
        assert torch.equal(net._from_raw(z, whole[None]), ref) and torch.equal(net._from_raw(z, row), ref)


@pytest.mark.parametrize("S,N", [(1, 3), (5, 40), (31, 8), (130, 33), (700, 17), (512, 3), (2049, 37), (5120, 5), (1030, 148), (600, 149)])
def test_global_column_attention(S, N, device_status):
    """The layer against the same in 64 bits, with masked sequences and a wholly masked column.  Bound as above, once for the gated
    product that is rounded before the output projection."""
    torch.manual_seed(S)
    net = fops.ChunkMSAColumnGlobalAttention(64, c=8, n_head=8).to(DEV, torch.bfloat16).eval().requires_grad_(False)
    with torch.no_grad():
        _randomise(net)
        m, mask = _randn(1, S, N, 64), (torch.rand(1, S, N, device=DEV) > 0.2).to(torch.bfloat16)
        mask[0, :, 1] = 0
        assert net._from_raw(m, mask) is not None
        ga = net.global_attention
        x, mk = _ln(m[0], net.layernormM).transpose(0, 1), mask[0].double().t()                       # [N, S, c]
        q = (x * mk[..., None]).sum(1) / (mk.sum(-1, keepdim=True) + 1e-10)
        q = (_lin(q, ga.to_q.weight) * ga.scaling).view(N, 8, 8)
        k, v = _lin(x, ga.to_kv.weight).bfloat16().double().chunk(2, -1)
        a = (q @ k.transpose(1, 2)).masked_fill(mk[:, None] == 0, -1e9).softmax(-1)
        o = (a @ v).reshape(N, 1, 64) * torch.sigmoid(_lin(x, ga.gating_linear.weight, ga.gating_bias))
        ref = m[0].double() + _lin(o, ga.o_linear.weight, ga.o_linear.bias).transpose(0, 1)
        _close(net(m, mask)[0], ref)


def test_calls_that_stay_with_the_composition():
    """What the kernels do not cover goes the way of the separate kernels: None from the native functions, or `ready` says no."""
    with torch.no_grad():
        net = fops.Transition(128).to(DEV, torch.bfloat16)
        x = _randn(1, 6, 7, 128)
        assert net._one_kernel(x) is not None
        assert net._one_kernel(x.float()) is None
        assert net._one_kernel(x[:0]) is None
        assert net._one_kernel(x[..., :96]) is None
        assert ln_gemm.transition(x, LayerNorm(128).to(DEV), net.linear1, net.linear2, False) is None            # fp32 norm
        for odd in (x.transpose(1, 3).contiguous().transpose(1, 3), _randn(6 * 7 * 128 + 4)[4:].view(1, 6, 7, 128)):
            assert torch.equal(net(odd), net(odd.clone(memory_format=torch.contiguous_format)))
        handle = net.linear1.register_forward_hook(lambda *a: None)
        assert net._one_kernel(x) is None
        handle.remove()
        assert net._one_kernel(x) is not None
        with torch.autograd.forward_ad.dual_level():
            assert net._one_kernel(x) is None

        class Doubled(fops.Linear):
            def forward(self, x, act=None):
                return 2 * super().forward(x, act)

        plain, net.linear1 = net.linear1, Doubled(128, 512).to(DEV, torch.bfloat16)                              # a module of another class
        assert net._one_kernel(x) is None
        net.linear1 = plain
        net.norm.forward = lambda x: x                                               # a replaced forward
        assert net._one_kernel(x) is None
        del net.norm.forward
        assert net._one_kernel(x) is not None
    assert net._one_kernel(x) is None                                                # gradients


@pytest.mark.parametrize("n", [24, 100])
@pytest.mark.parametrize("chunk", [None, 16, 64])
@pytest.mark.parametrize("cls", [fops.ChunkTriangleAttentionStartingNode, fops.ChunkTriangleAttentionEndingNode])
def test_triangle_attention(cls, chunk, n, device_status):
    """Whole and in chunks of rows / columns, in place and not, against the composition from separate kernels."""
    torch.manual_seed(n)
    net = cls(128, p_drop=0.25, c=32, n_head=4).to(DEV, torch.bfloat16).eval().requires_grad_(False)
    z, mask = _randn(1, n, n, 128), (torch.rand(1, n, n, device=DEV) > 0.2).to(torch.bfloat16)
    with torch.no_grad():
        _randomise(net)
        handle = net.linear_b.register_forward_hook(lambda *a: None)
        ref = net(z, mask)
        handle.remove()
        fops.set_chunk_size(chunk)
        try:
            _close(net(z, mask), ref.double())
            held = z.clone()
            out = net.inplace([held], mask)[0]
            assert out.data_ptr() == held.data_ptr()
            _close(out, ref.double())
        finally:
            fops.set_chunk_size(None)


class _composed:
    """Inside, the module runs as separate kernels: one of the modules that would be passed by has a hook."""

    def __init__(self, mod):
        self.mod = mod

    def __enter__(self):
        self.handle = self.mod.register_forward_hook(lambda *a: None)

    def __exit__(self, *exc):
        self.handle.remove()


def _net(cls, *args, **kw):
    net = cls(*args, **kw).to(DEV, torch.bfloat16).eval().requires_grad_(False)
    _randomise(net)
    return net


@pytest.mark.parametrize("C", [64, 128, 256])
@pytest.mark.parametrize("shape", [(1, 1), (1, 31), (3, 43), (74, 128), (1, 9473), (100, 203)])
def test_transition_same_bits(C, shape, device_status):
    """The sums of the LayerNorm and the roundings are those of the separate kernels, so nothing may differ."""
    torch.manual_seed(C)
    with torch.no_grad():
        net, x = _net(fops.Transition, C), _randn(1, *shape, C) * 3 + 0.5
        fused = net(x)
        with _composed(net.linear1):
            assert torch.equal(net(x), fused)


@pytest.mark.parametrize("n", [8, 27, 64, 203])
@pytest.mark.parametrize("chunk", [None, 16, 64])
def test_pair_modules_same_bits(chunk, n, device_status):
    torch.manual_seed(n)
    with torch.no_grad():
        z, mask = _randn(1, n, n, 128) * 2 + 0.25, (torch.rand(1, n, n, device=DEV) > 0.2).to(torch.bfloat16)
        fops.set_chunk_size(chunk)
        try:
            for cls in (fops.AsyncChunkTriangleMultiplicationOutgoing, fops.AsyncChunkTriangleMultiplicationIncoming):
                net = _net(cls, 128, p_drop=0.25)
                fused = net(z, mask)
                with _composed(net.output_projection):
                    assert torch.equal(net(z, mask), fused), cls
            for cls in (fops.ChunkTriangleAttentionStartingNode, fops.ChunkTriangleAttentionEndingNode):
                net = _net(cls, 128, p_drop=0.25, c=32, n_head=4)
                fused = net(z, mask)
                with _composed(net.attention.o_linear):
                    assert torch.equal(net(z, mask), fused), cls
        finally:
            fops.set_chunk_size(None)


@pytest.mark.parametrize("S,n", [(5, 8), (33, 27), (64, 64), (40, 203), (74, 128), (130, 150)])
@pytest.mark.parametrize("chunk", [None, 16])
def test_msa_modules_same_bits(chunk, S, n, device_status):
    torch.manual_seed(n)
    with torch.no_grad():
        m, e, z = _randn(1, S, n, 256) * 2 + 0.25, _randn(1, S, n, 64), _randn(1, n, n, 128)
        mask = (torch.rand(1, S, n, device=DEV) > 0.2).to(torch.bfloat16)
        row, extra = _net(fops.ChunkMSARowAttentionWithPairBias, 256, 128), _net(fops.ChunkMSARowAttentionWithPairBias, 64, 128, c=8)
        col, opm = _net(MSAColumnAttention, 256), _net(fops.OutProductMean, 256, 128, 32)
        fops.set_chunk_size(chunk)
        try:
            for call, inner in ((lambda: row(m, z, mask), row.attention.o_linear), (lambda: extra(e, z, mask), extra.attention.o_linear),
                                (lambda: col(m, mask), col.attention.o_linear), (lambda: opm(m, mask, z), opm.linear_a)):
                fused = call()
                with _composed(inner):
                    assert torch.equal(call(), fused)
        finally:
            fops.set_chunk_size(None)


class _DoubledNorm(LayerNorm):
    def forward(self, x):
        return 2 * super().forward(x)


@pytest.mark.parametrize("how", ["subclass", "forward", "identity", "hook"])
def test_replaced_pair_norm(how, device_status):
    """The norm of the pair tensor in the row attention is evaluated from its parameters only where it is the package's own, unchanged."""
    torch.manual_seed(5)
    with torch.no_grad():
        net = _net(fops.ChunkMSARowAttentionWithPairBias, 256, 128)
        m, z, mask = _randn(1, 9, 24, 256), _randn(1, 24, 24, 128), torch.ones(1, 9, 24, device=DEV, dtype=torch.bfloat16)
        plain = net(m, z, mask)
        if how == "subclass":
            net.layernormZ = _DoubledNorm(128).to(DEV, torch.bfloat16)
        elif how == "forward":
            net.layernormZ.forward = lambda x: 2 * x
        elif how == "identity":
            net.layernormZ = torch.nn.Identity()
        else:
            net.layernormZ.register_forward_hook(lambda mod, args, out: 2 * out)
        out = net(m, z, mask)
        assert not torch.equal(out, plain)
        with _composed(net.attention.o_linear):
            assert torch.equal(net(m, z, mask), out)


class _Forwarding(torch.nn.Module):
    def __init__(self, inner):
        super().__init__()
        self.inner = inner

    def forward(self, *args, **kw):
        return self.inner(*args, **kw)


def test_wrapped_attention(device_status):
    """An attention inside a module that only passes the call on gives what the attention itself gives (the global one from separate
    kernels, whose mean query is rounded to bf16)."""
    torch.manual_seed(6)
    with torch.no_grad():
        m, z = _randn(1, 9, 24, 256), _randn(1, 24, 24, 128)
        mask, zmask = torch.ones(1, 9, 24, device=DEV, dtype=torch.bfloat16), torch.ones(1, 24, 24, device=DEV, dtype=torch.bfloat16)
        row, col = _net(fops.ChunkMSARowAttentionWithPairBias, 256, 128), _net(MSAColumnAttention, 256)
        start, end = _net(fops.ChunkTriangleAttentionStartingNode, 128, p_drop=0.0), _net(fops.ChunkTriangleAttentionEndingNode, 128, p_drop=0.0)
        for net, args in ((row, (m, z, mask)), (col, (m, mask)), (start, (z, zmask)), (end, (z, zmask))):
            want = net(*args)
            net.attention = _Forwarding(net.attention)
            assert torch.equal(net(*args), want), type(net)
        e, net = _randn(1, 40, 24, 64), _net(fops.ChunkMSAColumnGlobalAttention, 64)
        emask = torch.ones(1, 40, 24, device=DEV, dtype=torch.bfloat16)
        assert net._from_raw(e, emask) is not None
        with _composed(net.layernormM):
            want = net(e, emask)
        net.global_attention = _Forwarding(net.global_attention)
        assert torch.equal(net(e, emask), want)


@pytest.mark.parametrize("layout", ["dense", "off the boundary", "channels apart"])
@pytest.mark.parametrize("chunk", [None, 16])
def test_in_place_calls_write_into_the_tensor_itself(chunk, layout, device_status):
    """`inplace` leaves its result in the caller's tensor, not only in the list: dense tensors on any address, and those of another
    layout where the separate kernels did (global column attention; transitions in chunks)."""
    torch.manual_seed(7)

    def held(*shape):
        if layout == "dense":
            return _randn(*shape)
        if layout == "off the boundary":
            n = 4 + torch.Size(shape).numel()
            return _randn(n)[4:].view(shape)
        return _randn(shape[0], shape[3], shape[2], shape[1]).transpose(1, 3)

    with torch.no_grad():
        mask, zmask = torch.ones(1, 40, 24, device=DEV, dtype=torch.bfloat16), torch.ones(1, 24, 24, device=DEV, dtype=torch.bfloat16)
        cases = [(_net(fops.ChunkMSAColumnGlobalAttention, 64), held(1, 40, 24, 64), (mask,))]
        if layout != "channels apart" or chunk:
            cases.append((_net(fops.Transition, 128), held(1, 40, 24, 128), ()))
        if layout != "channels apart":
            cases += [(_net(fops.AsyncChunkTriangleMultiplicationOutgoing, 128, p_drop=0.0), held(1, 24, 24, 128), (zmask,)),
                      (_net(fops.ChunkTriangleAttentionStartingNode, 128, p_drop=0.0), held(1, 24, 24, 128), (zmask,)),
                      (_net(fops.ChunkTriangleAttentionEndingNode, 128, p_drop=0.0), held(1, 24, 24, 128), (zmask,))]
        fops.set_chunk_size(chunk)
        try:
            for net, x, args in cases:
                want = net(x.clone(), *args)
                out = net.inplace([x], *args)[0]
                assert out.data_ptr() == x.data_ptr() and torch.equal(out, want) and torch.equal(x, want), type(net)
        finally:
            fops.set_chunk_size(None)


@pytest.mark.parametrize("S,n", [(3, 40), (74, 128), (75, 128)])
@pytest.mark.parametrize("chunk", [None, 16])
def test_captured_calls_same_bits(chunk, S, n, device_status):
    """Few rows of 256 channels run as separate kernels under stream capture, up to 9472 rows on 148 SMs."""
    torch.manual_seed(S)
    with torch.no_grad():
        m, z, mask = _randn(1, S, n, 256), _randn(1, n, n, 128), (torch.rand(1, S, n, device=DEV) > 0.2).to(torch.bfloat16)
        row, col, tr = _net(fops.ChunkMSARowAttentionWithPairBias, 256, 128), _net(MSAColumnAttention, 256), _net(fops.Transition, 256)
        fops.set_chunk_size(chunk)
        try:
            for call in (lambda x: row(x, z, mask), lambda x: col(x, mask), tr, lambda x: tr.inplace([x.clone()])[0]):
                want = call(m)
                graph = torch.cuda.CUDAGraph()
                with torch.cuda.graph(graph):
                    got = call(m)
                graph.replay()
                assert torch.equal(got, want)
        finally:
            fops.set_chunk_size(None)


def test_masks_in_host_memory_raise(device_status):
    """No kernel is launched with them: the native calls leave them to the composition, which refuses them."""
    with torch.no_grad():
        m, e, z = _randn(1, 9, 24, 256), _randn(1, 9, 24, 64), _randn(1, 24, 24, 128)
        mask, zmask = torch.ones(1, 9, 24, dtype=torch.bfloat16), torch.ones(1, 24, 24, dtype=torch.bfloat16)
        row, col, opm = _net(fops.ChunkMSARowAttentionWithPairBias, 256, 128), _net(MSAColumnAttention, 256), _net(fops.OutProductMean, 256, 128, 32)
        glob, start = _net(fops.ChunkMSAColumnGlobalAttention, 64), _net(fops.ChunkTriangleAttentionStartingNode, 128, p_drop=0.0)
        mul = _net(fops.AsyncChunkTriangleMultiplicationOutgoing, 128, p_drop=0.0)
        for call in (lambda: row(m, z, mask), lambda: col(m, mask), lambda: opm(m, mask, z), lambda: glob(e, mask), lambda: start(z, zmask),
                     lambda: mul(z, zmask)):
            with pytest.raises((AssertionError, RuntimeError)):
                call()


@pytest.mark.parametrize("S,N", [(64, 40), (65, 40), (128, 33), (129, 64), (515, 70)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_mask_normaliser_of_many_sequences(S, N, dtype, device_status):
    """One pass of 64 sequences in one group, and one, two and five passes of 128 in four: fp32 sums of at most 515 products of
    values in [0, 1], one reciprocal: 515 x 2^-24 relative, and 2 ulp.  Of masks of zeros and ones the sums are exact."""
    torch.manual_seed(N)
    for mask in (torch.rand(1, S, N, device=DEV).to(dtype), (torch.rand(1, S, N, device=DEV) > 0.3).to(dtype)):
        ref = 1.0 / (mask[0].double().t() @ mask[0].double() + 1e-3)
        out = ln_gemm.mask_norm(mask, 1e-3)
        assert ((out[0, :, :, 0].double() - ref).abs() <= 3.2e-5 * ref).all()


@pytest.mark.parametrize("M", [4 * 148 * 128 - 128, 4 * 148 * 128 - 127, 90001])
def test_pair_of_projections_of_many_rows(M, device_status):
    """256 channels, on both sides of four tiles of 128 rows per SM: every element, the same bits as in two halves."""
    torch.manual_seed(M)
    with torch.no_grad():
        x, norm, s = _randn(M, 256), _norm(256), torch.rand(M, device=DEV).to(torch.bfloat16)
        ws, bs = [_randn(32, 256, scale=1 / 16) for _ in range(2)], [_randn(32, scale=0.1) for _ in range(2)]
        ys = ln_gemm.pair(x, norm, ws[0], bs[0], ws[1], bs[1], s)
        h = M // 256 * 128
        halves = [ln_gemm.pair(x[i:j].contiguous(), norm, ws[0], bs[0], ws[1], bs[1], s[i:j].contiguous()) for i, j in ((0, h), (h, M))]
        for y, a, b, w, c in zip(ys, *halves, ws, bs):
            assert torch.equal(y, torch.cat([a, b]))
            _close(y, _lin(_ln(x, norm), w, c) * s.double()[:, None])

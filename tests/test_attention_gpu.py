"""Fused tcgen05 attention against an fp32 PyTorch reference of the same op."""
import pytest
import torch

from fastfold_b200.ops.attention import attention_core, attention_core_ref
from fastfold_b200.ops import flash

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _qkv(B, n, H, d=32):
    qkv = torch.randn(1, B, n, 3, H, d, device=DEV).to(torch.bfloat16)
    return tuple(qkv[:, :, :, i].permute(0, 1, 3, 2, 4) for i in range(3))


@pytest.mark.parametrize("B,n,H,use_bias,use_mask", [
    (4, 128, 8, True, True), (128, 256, 8, True, True), (37, 256, 4, True, False), (256, 128, 8, False, True),
    (3, 384, 4, True, True), (2, 200, 4, True, True), (5, 1024, 4, True, True), (9, 72, 8, False, False),
    (3, 40, 4, True, True), (300, 256, 4, True, False),
])
def test_forward(B, n, H, use_bias, use_mask, device_status):
    torch.manual_seed(B * 1000 + n)
    q, k, v = _qkv(B, n, H)
    bias = torch.randn(1, 1, H, n, n, device=DEV).to(torch.bfloat16) if use_bias else None
    mask = None
    if use_mask:
        mask = (torch.rand(1, B, n, device=DEV) > 0.2).to(torch.bfloat16)
        mask[..., 0] = 1
        if B > 1:
            mask[0, 1] = 0            # one fully masked row: uniform weights, as in the reference kernels
    assert flash.supported(q, k, v, mask, bias)
    with torch.no_grad():
        out = attention_core(q, k, v, mask, bias)
    ref = attention_core_ref(q.float(), k.float(), v.float(), None if mask is None else mask.float(), None if bias is None else bias.float())
    err = (out.float() - ref).abs().max().item()
    assert err < 2e-2, "max abs err %g" % err


@pytest.mark.parametrize("B,n,H,use_bias", [(1, 64, 4, True), (5, 72, 4, True), (6, 256, 8, True), (7, 320, 4, False), (9, 640, 4, True)])
def test_forward_rows_that_leave_the_exponent_range(B, n, H, use_bias, device_status):
    """Rows whose reference point has to move: logits of several hundred, a much larger (smaller) level from some key on,
    leading blocks that are masked as a whole, a fully masked row.  Bound: |v| < 5.5; the
    output is rounded to bf16 (half a step of 2^-5 at 4 .. 8), and P is (2^-9 relative, so up to 2 x 2^-9 x 5.5 between a
    row's keys): 1.6e-2 + 2.2e-2; the logits agree to fp32."""
    torch.manual_seed(n + B)
    q, k, v = _qkv(B, n, H)
    q = q * 8.0
    bias = None
    if use_bias:
        bias = torch.randn(1, 1, H, n, n, device=DEV)
        bias[..., : n // 3, n // 2:] += 300.0
        bias[..., n // 3: 2 * (n // 3), n // 2:] -= 300.0
        bias[:, :, 0] -= 500.0
        bias = bias.to(torch.bfloat16)
    mask = torch.ones(1, B, n, device=DEV, dtype=torch.bfloat16)
    mask[0, 0, : (n * 3) // 4] = 0
    if B > 1:
        mask[0, 1] = 0
    with torch.no_grad():
        out = attention_core(q, k, v, mask, bias)
    ref = attention_core_ref(q.float(), k.float(), v.float(), mask.float(), None if bias is None else bias.float())
    assert (out.float() - ref).abs().max().item() < 3.8e-2


def _infer(xq, xkv, bias, mask, n_k):
    """The kernel without gradients: queries from ``xq [B, n_q, 3, H, d]``, the first ``n_k`` rows of ``xkv [B, .., 3, H, d]`` as
    keys and values, ``bias [H, n_q, n_k]`` in rows at a pitch of 8, ``mask [B, n_k]``."""
    from fastfold_b200.ops import _lib
    B, n_q, _, H, d = xq.shape
    pitch = (n_k + 7) // 8 * 8
    b = None if bias is None else torch.nn.functional.pad(bias, (0, pitch - n_k)).contiguous()
    out = torch.full((B, n_q, H * d), float("nan"), device=DEV, dtype=torch.bfloat16)
    kv, rs = xkv.data_ptr(), 3 * H * d
    rc = _lib.get().ffb_attention_infer(xq.data_ptr(), kv + 2 * H * d, kv + 4 * H * d, n_q * rs, rs, xkv.shape[1] * rs, rs, _lib.ptr(b), pitch,
                                        _lib.ptr(mask), n_k, out.data_ptr(), n_q * H * d, H * d, B, H, n_q, n_k, d, d ** -0.5, _lib.stream_ptr())
    assert rc == 0
    return out.view(B, n_q, H, d).transpose(1, 2)


@pytest.mark.parametrize("B,H,n_q,n_k,d", [
    (1, 1, 1, 1, 32), (3, 2, 33, 17, 32), (7, 4, 97, 64, 16), (5, 2, 64, 127, 32),      # one round per CTA, one to four warps with rows
    (445, 1, 129, 65, 32), (446, 1, 161, 129, 16), (447, 2, 225, 256, 32),  # several rounds per CTA, resident bias, last query tile in part
    (100, 8, 257, 257, 32), (64, 4, 390, 390, 16), (67, 4, 520, 389, 32),   # streamed bias, rounds with fewer than three rows, key tails
    (1000, 4, 64, 321, 32),
])
@pytest.mark.parametrize("use_bias", [True, False])
@pytest.mark.parametrize("use_mask", [True, False])
def test_forward_rounds_and_tails(B, H, n_q, n_k, d, use_bias, use_mask, device_status):
    """Query tiles and key blocks that are filled in part, more queries than keys and fewer, batch rows in rounds of one to three,
    several rounds per CTA: every element, twice the same bits.  What lies behind the last key is NaN.  Bound: P and the output are rounded to
    bf16 and |v| < 5.5, as above, with logits of order 1."""
    g = torch.Generator(device=DEV).manual_seed(B + n_k)
    xq = torch.randn(B, n_q, 3, H, d, device=DEV, generator=g).to(torch.bfloat16)
    xkv = torch.randn(B, n_k + 3, 3, H, d, device=DEV, generator=g).to(torch.bfloat16)
    xkv[:, n_k:] = float("nan")
    bias = torch.randn(H, n_q, n_k, device=DEV, generator=g).to(torch.bfloat16) if use_bias else None
    mask = None
    if use_mask:
        mask = (torch.rand(B, n_k, device=DEV, generator=g) > 0.3).to(torch.bfloat16)
        mask[:, 0] = 1
        mask[B // 2:] = 1
    out = _infer(xq, xkv, bias, mask, n_k)
    assert torch.equal(out, _infer(xq, xkv, bias, mask, n_k))
    for i in range(0, B, 64):
        q = xq[i:i + 64, :, 0].float().transpose(1, 2)
        k, v = (xkv[i:i + 64, :n_k, j].float().transpose(1, 2) for j in (1, 2))
        ref = attention_core_ref(q, k, v, None if mask is None else mask[i:i + 64].float(), None if bias is None else bias.float())
        assert (out[i:i + 64].float() - ref).abs().max().item() < 2.2e-2


@pytest.mark.parametrize("n", [128, 200, 640])
@pytest.mark.parametrize("level", [-8e8, -1e9])
def test_forward_masked_block_before_keys_of_a_low_bias(level, n, device_status):
    """A wholly masked block of 64 keys, then keys that the pair bias pushes to the level that masks are written with: still
    above the logit of a masked key (-2^30), so all weight is theirs.  Values of 1 there and -1 on masked keys: exactly 1."""
    torch.manual_seed(n)
    q, k, _ = _qkv(3, n, 4)
    v = torch.ones_like(q)
    v[..., :64, :] = -1
    mask = torch.ones(1, 3, n, device=DEV, dtype=torch.bfloat16)
    mask[..., :64] = 0
    bias = torch.full((1, 1, 4, n, n), level, device=DEV, dtype=torch.bfloat16)
    with torch.no_grad():
        assert torch.equal(attention_core(q, k, v, mask, bias), torch.ones_like(v))


@pytest.mark.parametrize("B,n,H,d", [(1, 64, 4, 32), (5, 75, 4, 32), (6, 256, 8, 32), (9, 320, 4, 32), (9, 640, 4, 32), (6, 128, 4, 16), (7, 333, 4, 16)])
def test_forward_biases_that_are_masks(B, n, H, d, device_status):
    """Pair biases of -1e9, the lowest and the largest bf16 value, -inf and ordinary ones in blocks of keys, next to blocks that
    are masked wholly, in part or not at all.  Rows without a single finite logit are NaN in both.  Bound as above: |v| < 5.5,
    output and P rounded to bf16."""
    g = torch.Generator().manual_seed(n + B + d)
    qkv = torch.randn(1, B, n, 3, H, d, generator=g).to(DEV, torch.bfloat16)
    low = torch.finfo(torch.bfloat16).min
    levels = torch.tensor([0.0, -600.0, 600.0, -2e6, 2e6, -1e9, 1e9, low, -low, float("-inf")])
    blocks = (n + 63) // 64
    pick = torch.randint(0, len(levels), (1, 1, H, n, blocks), generator=g)
    pick[..., : n // 2, :] = pick[..., : n // 2, :1]                # half of the rows at one level,
    pick[..., : n // 4, :] = 5 + 2 * (pick[..., : n // 4, :] % 3)   # some of them at one that is a mask
    bias = (levels[pick].repeat_interleave(64, -1)[..., :n] + torch.randn(1, 1, H, n, n, generator=g)).to(DEV, torch.bfloat16)
    share = torch.tensor([0.0, 0.1, 0.5, 1.0])[torch.randint(0, 4, (1, B, blocks), generator=g)].repeat_interleave(64, -1)[..., :n]
    mask = (torch.rand(1, B, n, generator=g) >= share).to(DEV, torch.bfloat16)
    mask[0, 0] = 1
    mask[0, -1, :64] = 0
    with torch.no_grad():
        out = flash.flash_attention_packed(qkv, mask, bias, d ** -0.5).float()
    q, k, v = qkv.float().permute(3, 0, 1, 4, 2, 5)
    ref = attention_core_ref(q, k, v, mask.float(), bias.float()).transpose(2, 3).flatten(3)
    assert torch.equal(out.isnan(), ref.isnan())
    assert (out - ref).nan_to_num().abs().max().item() < 3.8e-2


@pytest.mark.parametrize("B,n,H,use_bias,use_mask", [
    (4, 128, 8, True, True), (16, 256, 8, True, True), (7, 256, 4, False, True), (5, 384, 4, True, False), (3, 200, 4, True, True),
    (6, 512, 4, True, True),
])
def test_backward(B, n, H, use_bias, use_mask, device_status):
    torch.manual_seed(B * 77 + n)
    qkv = (torch.randn(1, B, n, 3, H, 32, device=DEV) * 0.7).to(torch.bfloat16).requires_grad_(True)
    bias = torch.randn(1, 1, H, n, n, device=DEV).to(torch.bfloat16).requires_grad_(True) if use_bias else None
    mask = None
    if use_mask:
        mask = (torch.rand(1, B, n, device=DEV) > 0.2).to(torch.bfloat16)
        mask[..., 0] = 1
    q, k, v = (qkv[:, :, :, i].permute(0, 1, 3, 2, 4) for i in range(3))
    assert flash.supported(q, k, v, mask, bias)
    out = attention_core(q, k, v, mask, bias)
    g = torch.randn_like(out)
    out.backward(g)
    qkv_r = qkv.detach().float().requires_grad_(True)
    bias_r = bias.detach().float().requires_grad_(True) if use_bias else None
    qr, kr, vr = (qkv_r[:, :, :, i].permute(0, 1, 3, 2, 4) for i in range(3))
    ref = attention_core_ref(qr, kr, vr, None if mask is None else mask.float(), bias_r)
    ref.backward(g.float())
    assert (out.float() - ref).abs().max() < 2e-2
    gerr = (qkv.grad.float() - qkv_r.grad).abs().max().item()
    gmax = qkv_r.grad.abs().max().item()
    assert gerr < 3e-2 * max(1.0, gmax), "dqkv err %g (max %g)" % (gerr, gmax)
    if use_bias:
        berr = (bias.grad.float() - bias_r.grad).abs().max().item()
        bmax = bias_r.grad.abs().max().item()
        assert berr < 3e-2 * max(1.0, bmax), "dbias err %g (max %g)" % (berr, bmax)


@pytest.mark.parametrize("n", [256, 200])
def test_backward_fully_masked_row_is_exact(n, device_status):
    """A batch row whose keys are all masked (a padded MSA row) has uniform attention weights; its gradients must be
    those of the uniform softmax (a backward pass that is off by a constant factor there grows exponentially through a
    deep stack), and the other rows must be unaffected."""
    torch.manual_seed(5)
    B, H = 6, 4
    qkv = (torch.randn(1, B, n, 3, H, 32, device=DEV) * 0.7).to(torch.bfloat16).requires_grad_(True)
    bias = torch.randn(1, 1, H, n, n, device=DEV).to(torch.bfloat16).requires_grad_(True)
    mask = torch.ones(1, B, n, device=DEV, dtype=torch.bfloat16)
    mask[0, 2] = 0
    mask[0, 4] = 0
    q, k, v = (qkv[:, :, :, i].permute(0, 1, 3, 2, 4) for i in range(3))
    out = attention_core(q, k, v, mask, bias)
    g = torch.randn_like(out)
    out.backward(g)
    assert torch.isfinite(out.float()).all()
    assert torch.isfinite(qkv.grad.float()).all() and torch.isfinite(bias.grad.float()).all()
    qkv_r = qkv.detach().float().requires_grad_(True)
    bias_r = bias.detach().float().requires_grad_(True)
    qr, kr, vr = (qkv_r[:, :, :, i].permute(0, 1, 3, 2, 4) for i in range(3))
    ref = attention_core_ref(qr, kr, vr, mask.float(), bias_r)
    ref.backward(g.float())
    assert (out.float() - ref).abs().max().item() < 2e-2
    gerr = (qkv.grad.float() - qkv_r.grad).abs().max().item()
    assert gerr < 3e-2 * max(1.0, qkv_r.grad.abs().max().item()), gerr
    # the masked rows on their own: dV there is mean(dO) / 1, small numbers that a factor-n error would swamp
    merr = (qkv.grad.float()[:, [2, 4]] - qkv_r.grad[:, [2, 4]]).abs().max().item()
    assert merr < 3e-2 * max(0.05, qkv_r.grad[:, [2, 4]].abs().max().item()), merr
    berr = (bias.grad.float() - bias_r.grad).abs().max().item()
    assert berr < 3e-2 * max(1.0, bias_r.grad.abs().max().item())


@pytest.mark.parametrize("B,n,H,use_bias", [(6, 256, 4, True), (5, 128, 8, False), (3, 200, 4, True)])
def test_packed_qkv_path(B, n, H, use_bias, device_status):
    """The packed entry (one QKV tensor in, one gradient tensor out) against the fp32 reference."""
    torch.manual_seed(B + n)
    qkv = (torch.randn(1, B, n, 3, H, 32, device=DEV) * 0.7).to(torch.bfloat16).requires_grad_(True)
    bias = torch.randn(1, 1, H, n, n, device=DEV).to(torch.bfloat16).requires_grad_(True) if use_bias else None
    mask = (torch.rand(1, B, n, device=DEV) > 0.2).to(torch.bfloat16)
    mask[..., 0] = 1
    assert flash.packed_supported(qkv, mask, bias)
    out = flash.flash_attention_packed(qkv, mask, bias, 32 ** -0.5)
    g = torch.randn_like(out)
    out.backward(g)
    qkv_r = qkv.detach().float().requires_grad_(True)
    bias_r = bias.detach().float().requires_grad_(True) if use_bias else None
    qr, kr, vr = (qkv_r[:, :, :, i].permute(0, 1, 3, 2, 4) for i in range(3))
    ref = attention_core_ref(qr, kr, vr, mask.float(), bias_r).permute(0, 1, 3, 2, 4).reshape(out.shape)
    ref.backward(g.float())
    assert (out.float() - ref).abs().max() < 2e-2
    gerr = (qkv.grad.float() - qkv_r.grad).abs().max().item()
    assert gerr < 3e-2 * max(1.0, qkv_r.grad.abs().max().item())
    if use_bias:
        berr = (bias.grad.float() - bias_r.grad).abs().max().item()
        assert berr < 3e-2 * max(1.0, bias_r.grad.abs().max().item())


def test_ending_node_strided_matches_transposed_reference(device_status):
    """Triangle attention around the ending node: GPU path (row / batch strides, no transposes; fused tail under
    no_grad, autograd under grad) against the same module in fp32 on the CPU (explicit transposes)."""
    from fastfold_b200.models.fastnn.ops import ChunkTriangleAttentionEndingNode
    torch.manual_seed(11)
    N, c = 64, 128
    ref = ChunkTriangleAttentionEndingNode(c, p_drop=0.25, c=32, n_head=4)
    with torch.no_grad():
        for p in ref.parameters():
            p.copy_(torch.randn_like(p) * 0.1)
    gpu = ChunkTriangleAttentionEndingNode(c, p_drop=0.25, c=32, n_head=4)
    gpu.load_state_dict(ref.state_dict())
    gpu = gpu.to(DEV, torch.bfloat16)
    ref.eval(); gpu.eval()
    z = torch.randn(1, N, N, c)
    mask = (torch.rand(1, N, N) > 0.1).float()
    mask[:, 0, :] = 1
    zg = z.to(DEV, torch.bfloat16)
    zr = zg.float().cpu().requires_grad_(True)
    with torch.no_grad():
        for p, q in zip(ref.parameters(), gpu.parameters()):
            p.copy_(q.float().cpu())
    out_ref = ref(zr, mask)
    assert gpu.strided(zg)
    with torch.no_grad():
        out_nograd = gpu(zg, mask.to(DEV, torch.bfloat16))
    assert (out_nograd.float().cpu() - out_ref.detach()).abs().max() < 0.06
    zg2 = zg.clone().requires_grad_(True)
    out_grad = gpu(zg2, mask.to(DEV, torch.bfloat16))
    assert (out_grad.float().cpu() - out_ref.detach()).abs().max() < 0.06
    g = torch.randn_like(out_ref)
    out_ref.backward(g)
    out_grad.backward(g.to(DEV, torch.bfloat16))
    err = (zg2.grad.float().cpu() - zr.grad).abs().max().item()
    assert err < 0.05 * max(1.0, zr.grad.abs().max().item()), err
    for (n_, p), q in zip(ref.named_parameters(), gpu.parameters()):
        e = (q.grad.float().cpu() - p.grad).abs().max().item()
        assert e < 0.06 * max(1.0, p.grad.abs().max().item()), (n_, e)


@pytest.mark.parametrize("B,n,H,use_bias,transposed", [(3, 640, 4, True, False), (2, 1024, 4, True, False), (2, 1024, 8, False, True),
                                                        (1, 2048, 4, True, False)])
def test_packed_backward_long_rows(B, n, H, use_bias, transposed, device_status):
    """Rows longer than the 512 queries whose gradient fits tensor memory: backward runs in blocks of 512 queries and sums
    the key / value gradients across the blocks; forward and all gradients against the fp32 reference."""
    torch.manual_seed(B * 31 + n)
    shape = (1, n, B, 3, H, 32) if transposed else (1, B, n, 3, H, 32)
    qkv = (torch.randn(*shape, device=DEV) * 0.7).to(torch.bfloat16).requires_grad_(True)
    bias = (torch.randn(1, 1, H, n, n, device=DEV)).to(torch.bfloat16).requires_grad_(True) if use_bias else None
    mask = (torch.rand(1, B, n, device=DEV) > 0.2).to(torch.bfloat16)
    mask[..., 0] = 1
    assert flash.packed_supported(qkv, mask, bias, transposed=transposed)
    out = flash.flash_attention_packed(qkv, mask, bias, 32 ** -0.5, transposed=transposed)
    g = torch.randn_like(out)
    out.backward(g)
    qkv_r = qkv.detach().float().requires_grad_(True)
    bias_r = bias.detach().float().requires_grad_(True) if use_bias else None
    src = qkv_r.transpose(1, 2) if transposed else qkv_r
    qr, kr, vr = (src[:, :, :, i].permute(0, 1, 3, 2, 4) for i in range(3))
    ref = attention_core_ref(qr, kr, vr, mask.float(), bias_r).permute(0, 1, 3, 2, 4).reshape(1, B, n, H * 32)
    if transposed:
        ref = ref.transpose(1, 2)
    ref.backward(g.float())
    assert (out.float() - ref).abs().max() < 2e-2
    gerr = (qkv.grad.float() - qkv_r.grad).abs().max().item()
    assert gerr < 3e-2 * max(1.0, qkv_r.grad.abs().max().item()), gerr
    if use_bias:
        berr = (bias.grad.float() - bias_r.grad).abs().max().item()
        assert berr < 3e-2 * max(1.0, bias_r.grad.abs().max().item()), berr


@pytest.mark.parametrize("c,heads", [(8, 8), (16, 4)])
def test_narrow_heads_train_on_the_fused_kernels(c, heads, device_status):
    """Gated self attention with 8- / 16-channel heads (extra-MSA rows, template triangles) under autograd: the module runs
    the fused kernels through differentiably zero-padded weights; outputs and every gradient against fp32 on the CPU."""
    from fastfold_b200.models.fastnn.ops import SelfAttention
    from fastfold_b200.ops import _lib
    torch.manual_seed(c)
    att = SelfAttention(64, c, heads, 64, gating=True)
    with torch.no_grad():
        for p in att.parameters():
            p.copy_(torch.randn_like(p) * 0.2)
    gpu = SelfAttention(64, c, heads, 64, gating=True)
    gpu.load_state_dict(att.state_dict())
    gpu = gpu.to(DEV, torch.bfloat16)
    with torch.no_grad():
        for p, q in zip(att.parameters(), gpu.parameters()):
            p.copy_(q.float().cpu())
    x = torch.randn(1, 6, 72, 64)
    xg = x.to(DEV, torch.bfloat16).requires_grad_(True)
    xr = xg.detach().float().cpu().requires_grad_(True)
    mask = (torch.rand(1, 6, 72) > 0.2).float()
    mask[..., 0] = 1
    bias = torch.randn(1, heads, 72, 72)
    n0 = _lib.LAUNCHES[0]
    out, _ = gpu(xg, mask.to(DEV, torch.bfloat16), (bias.to(DEV, torch.bfloat16), -1))
    assert _lib.LAUNCHES[0] - n0 >= 3
    ref, _ = att(xr, mask, (bias, -1))
    assert (out.float().cpu() - ref.detach()).abs().max() < 6e-2 * max(1.0, ref.abs().max().item())
    g = torch.randn_like(ref)
    ref.backward(g)
    out.backward(g.to(DEV, torch.bfloat16))
    assert (xg.grad.float().cpu() - xr.grad).abs().max() < 6e-2 * max(1.0, xr.grad.abs().max().item())
    for (name, p), q in zip(att.named_parameters(), gpu.parameters()):
        e = (q.grad.float().cpu() - p.grad).abs().max().item()
        assert e < 8e-2 * max(1.0, p.grad.abs().max().item()), (name, e)

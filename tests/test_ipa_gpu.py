"""Invariant point attention kernel (csrc/ipa.cu) against its fp32 PyTorch statement, and the module that calls it."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _inputs(N, seed=0, masked=True):
    g = torch.Generator().manual_seed(seed)
    H, C, PQ, PV, CZ = 12, 16, 4, 8, 128
    r = lambda *s: torch.randn(*s, generator=g)
    q, k, v = r(N, H, C), r(N, H, C), r(N, H, C)
    q_pts, k_pts, v_pts = r(N, H, PQ, 3) * 8, r(N, H, PQ, 3) * 8, r(N, H, PV, 3) * 8
    z = r(N, N, CZ).to(torch.bfloat16)
    wb, bb = r(H, CZ) * 0.1, r(H) * 0.1
    gamma = torch.nn.functional.softplus(r(H)) * math.sqrt(1.0 / (3 * (PQ * 9.0 / 2)))
    mask = (torch.rand(N, generator=g) > 0.15).float() if masked else torch.ones(N)
    return [t.to(DEV) for t in (q, k, v, q_pts, k_pts, v_pts, z, wb, bb, gamma, mask)]


@pytest.mark.parametrize("N", [64, 200, 333])
def test_ipa_core_matches_reference(N, device_status):
    from fastfold_b200.ops.ipa import ipa_core, ipa_core_ref
    args = _inputs(N)
    w_c, w_b, inf = math.sqrt(1.0 / 48), math.sqrt(1.0 / 3), 1e5
    with torch.no_grad():
        o, o_pt, o_pair = ipa_core(*args, w_c, w_b, inf)
        ro, ro_pt, ro_pair = ipa_core_ref(*args, w_c, w_b, inf)
    for a, b, tol in ((o, ro, 2e-3), (o_pt, ro_pt, 2e-2), (o_pair, ro_pair, 2e-3)):
        assert a.shape == b.shape
        assert (a - b).abs().max().item() <= tol * max(1.0, b.abs().max().item())


def test_ipa_core_row_block(device_status):
    """A rank that holds rows [64, 128) of the pair tensor computes exactly those query rows."""
    from fastfold_b200.ops.ipa import ipa_core
    args = _inputs(192, seed=3)
    w_c, w_b, inf = math.sqrt(1.0 / 48), math.sqrt(1.0 / 3), 1e5
    with torch.no_grad():
        full = ipa_core(*args, w_c, w_b, inf)
        shard = list(args)
        shard[6] = args[6][64:128].contiguous()
        part = ipa_core(*shard, w_c, w_b, inf, row0=64)
    for a, b in zip(part, full):
        assert torch.equal(a, b[64:128])


@pytest.mark.parametrize("N", [1, 15, 16, 17, 70, 127, 130])
def test_ipa_core_infinite_values_of_the_last_key(N, device_status):
    """A sum that holds an infinite value is infinite, whatever the length: keys past the end must not take part.  The other
    channels as in ``test_ipa_core_matches_reference``."""
    from fastfold_b200.ops.ipa import ipa_core, ipa_core_ref
    args = _inputs(N, seed=N, masked=False)
    args[0], args[3], args[4] = args[0] * 0.1, args[3] * 0.05, args[4] * 0.05        # every probability well above 0
    args[2][-1, 3, 5], args[2][-1, 7, 0] = math.inf, -math.inf
    args[5][-1, 2, 6, 1], args[5][-1, 11, 7, 2] = -math.inf, math.inf
    w = (math.sqrt(1.0 / 48), math.sqrt(1.0 / 3), 1e5)
    with torch.no_grad():
        out, ref = ipa_core(*args, *w), ipa_core_ref(*args, *w)
    for i, (a, b) in enumerate(zip(out, ref)):
        far = b.isinf()
        assert not b.isnan().any() and far.sum().item() == (0 if i == 2 else 2 * N)
        assert torch.equal(a[far], b[far]) and torch.isfinite(a[~far]).all()
        assert (a[~far] - b[~far]).abs().max().item() <= (2e-2 if i == 1 else 2e-3) * max(1.0, b[~far].abs().max().item())


def test_ipa_module_uses_kernel_and_matches_cpu(device_status):
    from fastfold_b200.models.nn.structure_module import InvariantPointAttention
    from fastfold_b200.ops import _lib
    from fastfold_b200.utils.rigid_utils import Rigid, Rotation
    torch.manual_seed(0)
    N = 96
    ipa = InvariantPointAttention(384, 128, 16, 12, 4, 8).eval()
    with torch.no_grad():
        for p in ipa.parameters():
            if float(p.abs().sum()) == 0.0:
                p.normal_(0, 0.05)
    s, z = torch.randn(N, 384), torch.randn(N, N, 128)
    quats, trans = torch.randn(N, 4), torch.randn(N, 3) * 5
    mask = torch.ones(N)
    with torch.no_grad():
        ref = ipa(s, z, Rigid(Rotation(quats=quats, normalize_quats=True), trans), mask)
        ipa_g = ipa.to(DEV, torch.bfloat16)
        n0 = _lib.LAUNCHES[0]
        got = ipa_g(s.to(DEV, torch.bfloat16), z.to(DEV, torch.bfloat16), Rigid(Rotation(quats=quats.to(DEV), normalize_quats=True), trans.to(DEV)),
                    mask.to(DEV, torch.bfloat16))
        assert _lib.LAUNCHES[0] > n0            # the native kernel ran
    err = (got.float().cpu() - ref).abs().mean().item()
    assert err <= 5e-2 * max(1.0, ref.abs().mean().item()), err


@pytest.mark.parametrize("N,fmt", [(1, "quat"), (33, "quat"), (96, "rot_mat"), (130, "quat")])
def test_ipa_layer_in_three_kernels(N, fmt, device_status):
    """Points, core and concatenated features against the operations they stand for, from the same bf16 projections.  The
    features are rounded to bf16 (2^-9 relative); coordinates of up to ~50 cancel against translations in fp32."""
    from fastfold_b200.ops import ipa as ipa_op
    from fastfold_b200.utils.rigid_utils import Rigid, Rotation
    g = torch.Generator().manual_seed(N)
    H, C, PQ, PV, CZ = 12, 16, 4, 8, 128
    r = lambda *s: torch.randn(*s, generator=g).to(DEV)
    b = lambda *s: r(*s).to(torch.bfloat16)
    q, kv, qp, kvp, z = b(N, 192), b(N, 384), b(N, 144), b(N, 432), b(N, N, CZ)
    rots = Rotation(quats=r(N, 4), normalize_quats=True)
    if fmt == "rot_mat":
        rots = Rotation(rot_mats=rots.get_rot_mats())
    frames = Rigid(rots, r(N, 3) * 8)
    wb, bb, gamma, mask = r(H, CZ) * 0.1, r(H) * 0.1, torch.rand(H, generator=g).to(DEV) * 0.1, (torch.rand(N, generator=g) > 0.2).float().to(DEV)
    w = (math.sqrt(1.0 / 48), math.sqrt(1.0 / 3), 1e5)
    with torch.no_grad():
        assert ipa_op.layer_supported(torch.empty(N, 384, device=DEV), z, q, kv, qp, kvp, frames)
        out = ipa_op.ipa_layer(q, kv, qp, kvp, frames, z, wb, bb, gamma, mask, *w, 1e-8)
        k, v = kv.view(N, H, 2 * C).split(C, dim=-1)
        pts = [frames[..., None].apply(torch.stack(p.split(p.shape[-1] // 3, dim=-1), dim=-1)).view(N, H, -1, 3) for p in (qp, kvp)]
        o, o_pt, o_pair = ipa_op.ipa_core_ref(q.view(N, H, C), k, v, pts[0], pts[1][:, :, :PQ], pts[1][:, :, PQ:], z, wb, bb, gamma, mask, *w)
        o_pt = frames[..., None, None].invert_apply(o_pt).reshape(N, -1, 3)
        ref = torch.cat([o.flatten(1), *o_pt.unbind(-1), torch.sqrt((o_pt ** 2).sum(-1) + 1e-8), o_pair.flatten(1)], dim=-1)
    assert out.shape == ref.shape and out.dtype == torch.bfloat16
    assert ((out.float() - ref).norm() / ref.norm()).item() < 4e-3
    assert (out.float() - ref).abs().max().item() < 2.0 ** -8 * ref.abs().max().item() + 1e-3


@pytest.mark.parametrize("half", [(0,), (1,), (2,), (3,), (0, 1, 2, 3)])
def test_ipa_layer_takes_parameters_and_mask_as_they_come(half, device_status):
    """Pair-bias weight and bias, point weights and mask in bf16 give the bits of the same values in fp32."""
    from fastfold_b200.ops import ipa as ipa_op
    from fastfold_b200.utils.rigid_utils import Rigid, Rotation
    g = torch.Generator().manual_seed(3)
    b = lambda *s: torch.randn(*s, generator=g).to(DEV, torch.bfloat16)
    N = 70
    frames = Rigid(Rotation(quats=torch.randn(N, 4, generator=g).to(DEV), normalize_quats=True), torch.randn(N, 3, generator=g).to(DEV))
    params = [b(12, 128), b(12), b(12).abs(), (b(N) > -1).to(torch.bfloat16)]
    args = (b(N, 192), b(N, 384), b(N, 144), b(N, 432), frames, b(N, N, 128))
    with torch.no_grad():
        want = ipa_op.ipa_layer(*args, *(p.float() for p in params), 0.1, 0.5, 1e5, 1e-8)
        got = ipa_op.ipa_layer(*args, *(p if i in half else p.float() for i, p in enumerate(params)), 0.1, 0.5, 1e5, 1e-8)
    assert torch.equal(got, want)


@pytest.mark.parametrize("case", ["layer", "fp32", "batched"])
def test_ipa_module_projects_once(case, device_status):
    """Each input projection is evaluated once, whichever path the rest of the layer takes."""
    from fastfold_b200.models.nn.structure_module import InvariantPointAttention
    from fastfold_b200.utils.rigid_utils import Rigid, Rotation
    torch.manual_seed(0)
    dt = torch.float32 if case == "fp32" else torch.bfloat16
    lead = (1,) if case == "batched" else ()
    mod = InvariantPointAttention(384, 128, 16, 12, 4, 8).to(DEV, dt)
    calls = []
    for name in ("linear_q", "linear_kv", "linear_q_points", "linear_kv_points"):
        getattr(mod, name).register_forward_hook(lambda m, x, y, name=name: calls.append(name))
    N = 24
    frames = Rigid(Rotation(quats=torch.randn(*lead, N, 4, device=DEV), normalize_quats=True), torch.randn(*lead, N, 3, device=DEV))
    with torch.no_grad():
        mod(torch.randn(*lead, N, 384, device=DEV, dtype=dt), torch.randn(*lead, N, N, 128, device=DEV, dtype=dt), frames,
            torch.ones(*lead, N, device=DEV, dtype=dt))
    assert sorted(calls) == ["linear_kv", "linear_kv_points", "linear_q", "linear_q_points"]


def test_ipa_core_takes_key_points_off_a_16_byte_boundary(device_status):
    from fastfold_b200.ops.ipa import ipa_core
    args = _inputs(70, seed=5)
    w = (math.sqrt(1.0 / 48), math.sqrt(1.0 / 3), 1e5)
    with torch.no_grad():
        want = ipa_core(*args, *w)
        flat = torch.empty(args[4].numel() + 1, device=DEV)
        args[4] = flat[1:].view(args[4].shape).copy_(args[4])
        got = ipa_core(*args, *w)
    assert all(torch.equal(a, b) for a, b in zip(got, want))


@pytest.mark.parametrize("N,row0,rows", [(1024, 0, 1024), (1027, 0, 1027), (1101, 50, 1026)])
def test_ipa_core_from_1024_rows_on(N, row0, rows, device_status):
    """The instance with four query rows per CTA: whole and partial last groups, and a block of rows.  Bounds as above."""
    from fastfold_b200.ops.ipa import ipa_core, ipa_core_ref
    args = _inputs(N, seed=N)
    args[6] = args[6][row0:row0 + rows].contiguous()
    w = (math.sqrt(1.0 / 48), math.sqrt(1.0 / 3), 1e5)
    with torch.no_grad():
        got, want = ipa_core(*args, *w, row0=row0), ipa_core_ref(*args, *w, row0=row0)
    for a, b, tol in zip(got, want, (2e-3, 2e-2, 2e-3)):
        assert a.shape == b.shape
        assert (a - b).abs().max().item() <= tol * max(1.0, b.abs().max().item())

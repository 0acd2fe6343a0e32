"""Performance cases: the layers and blocks of the trunk and of the structure module, as programs call them.

Every case goes through public module entry points in bfloat16 with bfloat16 weights.  ``exact`` restates the same mathematics in
plain PyTorch in 64 bits.
"""
import math

import torch

from fastfold_b200.models.fastnn import ops as fast_ops
from fastfold_b200.models.fastnn.evoformer import Evoformer
from fastfold_b200.models.fastnn.msa import ExtraMSACore, MSACore
from fastfold_b200.models.fastnn.ops import OutProductMean
from fastfold_b200.models.fastnn.triangle import (PairCore, TriangleAttentionEndingNode, TriangleAttentionStartingNode,
                                                  TriangleMultiplicationIncoming, TriangleMultiplicationOutgoing)
from fastfold_b200.models.nn.structure_module import InvariantPointAttention
from fastfold_b200.utils.rigid_utils import Rigid, Rotation

C_M, C_Z, C_E, C_S = 256, 128, 64, 384        # MSA, pair, extra-MSA and single channels of every preset
IPA_HEADS, IPA_C, IPA_QP, IPA_VP = 12, 16, 4, 8


def listed():
    return [
        # a peptide: one block of the trunk where launches and latency are all there is
        {"name": "block s32 n64", "kind": "block", "s": 32, "n": 64, "chunk": 0},
        # prediction of an ordinary domain: 128 clustered sequences, 256 residues (also the headline configuration)
        {"name": "block s128 n256", "kind": "block", "s": 128, "n": 256, "chunk": 0},
        # prediction of a protein of whatever length it happens to have
        {"name": "block s128 n203", "kind": "block", "s": 128, "n": 203, "chunk": 0},
        # the same with the memory-bounding option that long predictions are run with
        {"name": "block s256 n384 chunked", "kind": "block", "s": 256, "n": 384, "chunk": 64},
        # long predictions: triangle attention is most of their time
        {"name": "tri_att_start n1536", "kind": "tri_att_start", "n": 1536},
        # ending node at a length that is no multiple of anything
        {"name": "tri_att_end n389", "kind": "tri_att_end", "n": 389},
        # long predictions: the cubic contraction of the pair representation
        {"name": "tri_mul_out n1024", "kind": "tri_mul_out", "n": 1024},
        # extra-MSA stack: many sequences, narrow channels, 8-channel heads, global column attention
        {"name": "extra_msa s1024 n256", "kind": "extra_msa", "s": 1024, "n": 256},
        # outer product mean with the full cluster count
        {"name": "opm s512 n384", "kind": "opm", "s": 512, "n": 384},
        # structure module: eight calls of this per pass through the model
        {"name": "ipa n512", "kind": "ipa", "n": 512},
        # training at the crop size of the training preset, padded crops among them, with dropout masks: pair half and MSA half
        {"name": "pair_train n256", "kind": "pair_train", "n": 256},
        {"name": "msa_train s128 n256", "kind": "msa_train", "s": 128, "n": 256},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["block", "block", "block", "tri_att_start", "tri_att_end", "tri_mul_out", "tri_mul_in", "extra_msa", "opm", "ipa",
                       "pair_train", "msa_train"])
    if kind == "block":
        n, chunk = _log(rng, 32, 384), rng.choice([0, 0, 64])
        # the slab-wise triangle multiplication of chunked runs takes multiples of 8
        return {"kind": kind, "s": _log(rng, 16, 256), "n": n // 8 * 8 if chunk else n, "chunk": chunk}
    if kind in ("tri_att_start", "tri_att_end"):
        n = _log(rng, 64, 768)
        return {"kind": kind, "n": n}
    if kind in ("tri_mul_out", "tri_mul_in"):
        return {"kind": kind, "n": _log(rng, 64, 1024)}
    if kind == "extra_msa":
        return {"kind": kind, "s": _log(rng, 64, 1536), "n": _log(rng, 64, 320)}
    if kind == "opm":
        return {"kind": kind, "s": _log(rng, 16, 512), "n": _log(rng, 32, 448)}
    if kind == "ipa":
        return {"kind": kind, "n": _log(rng, 32, 768)}
    # training crops and their cluster counts are padded to configured sizes
    n = 8 * rng.randint(8, 40)
    return {"kind": kind, "n": n} if kind == "pair_train" else {"kind": kind, "s": 8 * rng.randint(4, 20), "n": n}


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _module(case):
    kind = case["kind"]
    if kind == "block":
        return Evoformer(C_M, C_Z, first_block=True, last_block=True)
    if kind == "tri_att_start":
        return TriangleAttentionStartingNode(C_Z, p_drop=0.25, c=32, n_head=4)
    if kind == "tri_att_end":
        return TriangleAttentionEndingNode(C_Z, p_drop=0.25, c=32, n_head=4)
    if kind == "tri_mul_out":
        return TriangleMultiplicationOutgoing(C_Z, p_drop=0.25, c=C_Z)
    if kind == "tri_mul_in":
        return TriangleMultiplicationIncoming(C_Z, p_drop=0.25, c=C_Z)
    if kind == "extra_msa":
        return ExtraMSACore(C_E, C_Z)
    if kind == "opm":
        return OutProductMean(n_feat=C_M, n_feat_out=C_Z, n_feat_proj=32)
    if kind == "ipa":
        return InvariantPointAttention(C_S, C_Z, IPA_C, IPA_HEADS, IPA_QP, IPA_VP)
    return PairCore(d_pair=C_Z) if kind == "pair_train" else MSACore(C_M, C_Z)


def prepare(case, seed):
    kind, n, s = case["kind"], case["n"], case.get("s", 0)
    g = torch.Generator(device="cuda").manual_seed(seed)

    def randn(*shape, scale=1.0):
        return (torch.randn(*shape, device="cuda", generator=g) * scale).to(torch.bfloat16)

    net = _module(case).to("cuda", torch.bfloat16)
    with torch.no_grad():
        for name, p in net.named_parameters():
            if p.dim() == 2:
                p.copy_(randn(*p.shape, scale=1.0 / math.sqrt(p.shape[1])))
            elif name.endswith(("gating_bias", "gate.bias")) or ("norm" in name and name.endswith("weight")):
                p.copy_(1.0 + randn(*p.shape, scale=0.1))
            else:
                p.copy_(randn(*p.shape, scale=0.1))
    train = kind.endswith("_train")
    net.train(train)
    net.requires_grad_(train)
    st = {"kind": kind, "net": net, "chunk": case.get("chunk", 0)}
    # predictions have whole masks; training crops end in padding
    res = torch.ones(n, device="cuda")
    seq = torch.ones(max(s, 1), device="cuda")
    if train:
        res[n - n // 10:] = 0.0
        seq[max(s, 1) - s // 10:] = 0.0
    st["msa_mask"] = (seq[:, None] * res[None, :]).to(torch.bfloat16)
    st["pair_mask"] = (res[:, None] * res[None, :]).to(torch.bfloat16)
    st["z"] = randn(n, n, C_Z)
    if s:
        st["m"] = randn(s, n, C_E if kind == "extra_msa" else C_M)
    if kind == "ipa":
        st["s"] = randn(n, C_S)
        quats = torch.randn(n, 4, device="cuda", generator=g)
        st["trans"] = torch.randn(n, 3, device="cuda", generator=g) * 5.0
        st["frames"] = Rigid(Rotation(quats=quats, normalize_quats=True), st["trans"])
        st["quats"] = quats
        st["mask"] = torch.ones(n, device="cuda", dtype=torch.bfloat16)
    if train:
        keep = lambda p, c, *shape: ((torch.rand(n, c, device="cuda", generator=g) >= p).to(torch.bfloat16) / (1.0 - p)).reshape(*shape, c)  # noqa: E731
        st["drop"] = {"tri_mul_out": keep(0.25, C_Z, 1, 1, n), "tri_mul_in": keep(0.25, C_Z, 1, 1, n),
                      "tri_att_start": keep(0.25, C_Z, 1, 1, n), "tri_att_end": keep(0.25, C_Z, 1, n, 1)}
        st["drop_msa"] = keep(0.15, C_M, 1, 1, n)
        st["up"] = randn(1, n, n, C_Z) if kind == "pair_train" else randn(1, s, n, C_M)
        st["z"].requires_grad_(True)
        if s:
            st["m"].requires_grad_(True)
    return st


def _rounding_only(name):
    """The one gradient that is zero in exact arithmetic: this bias shifts all logits of a row alike."""
    return name == "MSARowAttentionWithPairBias.layernormZ.bias"


def run(st):
    kind, net = st["kind"], st["net"]
    if kind == "pair_train":
        out = net(st["z"].unsqueeze(0), st["pair_mask"].unsqueeze(0), st["drop"])
        return [out] + list(torch.autograd.grad(out, [st["z"]] + list(net.parameters()), st["up"]))
    if kind == "msa_train":
        out = net(st["m"].unsqueeze(0), st["z"].unsqueeze(0), st["msa_mask"].unsqueeze(0), st["drop_msa"])
        grads = torch.autograd.grad(out, [st["m"], st["z"]] + list(net.parameters()), st["up"])
        return [out] + [g for g, name in zip(grads, ["m", "z"] + [k for k, _ in net.named_parameters()]) if not _rounding_only(name)]
    with torch.no_grad():
        if kind == "block":
            fast_ops.set_chunk_size(st["chunk"] or None)
            try:
                return net(st["m"], st["z"], st["msa_mask"], st["pair_mask"])
            finally:
                fast_ops.set_chunk_size(None)
        if kind == "extra_msa":
            return net(st["m"].unsqueeze(0), st["z"].unsqueeze(0), st["msa_mask"].unsqueeze(0))
        if kind == "opm":
            return net(st["m"].unsqueeze(0), st["msa_mask"].unsqueeze(0), st["z"].unsqueeze(0))
        if kind == "ipa":
            return net(st["s"], st["z"], st["frames"], st["mask"])
        return net(st["z"].unsqueeze(0), st["pair_mask"].unsqueeze(0))


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
def _attention_flops(rows, n, c, heads_c, extra=0):
    """Projections (qkv, gate, output) and the two products of ``rows`` attentions of length ``n``."""
    return 2.0 * rows * n * c * 5 * heads_c + 4.0 * rows * n * n * heads_c + 2.0 * extra


def _flops(case):
    kind, n, s = case["kind"], case["n"], case.get("s", 0)
    tri_att = _attention_flops(n, n, C_Z, 128, n * n * C_Z * 4)
    tri_mul = 2.0 * n * n * C_Z * C_Z * 6 + 2.0 * n ** 3 * C_Z
    opm = 2.0 * s * n * C_M * 64 + 2.0 * s * n * n * 1024 + 2.0 * n * n * 1024 * C_Z
    pair = 2 * tri_att + 2 * tri_mul + 2.0 * n * n * C_Z * 8 * C_Z
    msa = _attention_flops(s, n, C_M, 256, n * n * C_Z * 8) + _attention_flops(n, s, C_M, 256) + 2.0 * s * n * C_M * 8 * C_M
    if kind == "block":
        return msa + opm + pair
    if kind.startswith("tri_att"):
        return tri_att
    if kind.startswith("tri_mul"):
        return tri_mul
    if kind == "opm":
        return opm
    if kind == "extra_msa":
        return _attention_flops(s, n, C_E, 64, n * n * C_Z * 8) + 2.0 * s * n * C_E * (16 + 64 + 64) + 4.0 * s * n * 64 + 2.0 * s * n * C_E * 8 * C_E
    if kind == "ipa":
        per_pair = IPA_HEADS * (IPA_C + 3 * IPA_QP + C_Z + IPA_C + 3 * IPA_VP + C_Z)
        return 2.0 * n * n * per_pair + 2.0 * n * C_S * (3 * 192 + 144 + 432) + 2.0 * n * 2112 * C_S
    return 3.0 * (pair if kind == "pair_train" else msa)        # forward, and two products for each in backward


def work(case):
    kind, n, s = case["kind"], case["n"], case.get("s", 0)
    z, m = 2.0 * n * n * C_Z, 2.0 * s * n * (C_E if kind == "extra_msa" else C_M)
    weights = 2.0 * sum(p.numel() for p in _module(case).parameters())
    if kind == "block":
        moved = 2 * (z + m)
    elif kind == "extra_msa":
        moved = z + 2 * m
    elif kind == "opm":
        moved = 2 * z + m
    elif kind == "ipa":
        moved = z + 4.0 * n * C_S
    elif kind == "pair_train":
        moved = 4 * z + weights         # input, upstream gradient, output, gradient; a gradient for each weight
    elif kind == "msa_train":
        moved = 2 * z + 4 * m + weights
    else:
        moved = 2 * z
    return {"bytes": moved + weights, "flops": _flops(case)}


def tolerance(case):
    # about four times what the path shows against 64 bits, measured over the ranges of ``draw``
    kind = case["kind"]
    if kind == "block":
        return {"rel": 2.4e-2}
    if kind in ("pair_train", "msa_train"):
        return {"rel": 1.5e-1}
    return {"rel": 1.4e-2}


# ---------------------------------------------------------------------------
# the same in 64 bits
# ---------------------------------------------------------------------------
def _norm(x, P, name):
    return torch.nn.functional.layer_norm(x, (x.shape[-1],), P[name + ".weight"], P[name + ".bias"], 1e-5)


def _lin(x, P, name):
    y = x @ P[name + ".weight"].t()
    return y + P[name + ".bias"] if name + ".bias" in P else y


def _sdpa(q, k, v, mask, bias):
    """q, k, v [b, h, n, d], mask [b, n], bias [h, n, n]; a slab of b at a time unless gradients are wanted."""
    def part(q, k, v, mask):
        a = (q * q.shape[-1] ** -0.5) @ k.transpose(-1, -2)
        if bias is not None:
            a = a + bias
        a = torch.where(mask[:, None, None, :] == 0, torch.full_like(a, -1e9), a)
        return torch.softmax(a, -1) @ v
    step = q.shape[0] if torch.is_grad_enabled() else max(1, int(2 ** 28 / (q.shape[1] * q.shape[2] ** 2)))
    return torch.cat([part(q[i:i + step], k[i:i + step], v[i:i + step], mask[i:i + step]) for i in range(0, q.shape[0], step)])


def _gated(x, mask, bias, P, name, heads):
    b, n, _ = x.shape
    q, k, v = (t.transpose(1, 2) for t in _lin(x, P, name + ".to_qkv").view(b, n, 3, heads, -1).unbind(2))
    o = _sdpa(q, k, v, mask, bias).transpose(1, 2).reshape(b, n, -1)
    o = o * torch.sigmoid(_lin(x, P, name + ".gating_linear") + P[name + ".gating_bias"])
    return _lin(o, P, name + ".o_linear")


def _tri_att(z, mask, P, name, end, drop=None):
    x = _norm(z, P, name + "layernorm1")
    if end:
        x, mask = x.transpose(0, 1), mask.t()
    o = _gated(x, mask, _lin(x, P, name + "linear_b").permute(2, 0, 1), P, name + "attention", 4) + P[name + "out_bias"]
    o = o.transpose(0, 1) if end else o
    return z + (o if drop is None else o * drop)


def _tri_mul(z, mask, P, name, outgoing, drop=None):
    x = _norm(z, P, name + "layernorm1")
    ab = _lin(x, P, name + "left_right_projection") * torch.sigmoid(_lin(x, P, name + "left_right_gate")) * mask.unsqueeze(-1)
    a, b = (t.permute(2, 0, 1) for t in ab.chunk(2, -1))
    p = a @ b.transpose(1, 2) if outgoing else a.transpose(1, 2) @ b
    p = _norm(p.permute(1, 2, 0), P, name + "layernorm2")
    o = torch.sigmoid(_lin(x, P, name + "output_gate")) * (_lin(p, P, name + "output_projection") + P[name + "output_bias"])
    return z + (o if drop is None else o * drop)


def _transition(x, P, name):
    return x + _lin(torch.relu(_lin(_norm(x, P, name + "norm"), P, name + "linear1")), P, name + "linear2")


def _row_att(m, z, mask, P, name, drop=None):
    bias = (_norm(z, P, name + "layernormZ") @ P[name + "linear_b_weights"].t()).permute(2, 0, 1)
    o = _gated(_norm(m, P, name + "layernormM"), mask, bias, P, name + "attention", 8) + P[name + "out_bias"]
    return m + (o if drop is None else o * drop)


def _msa(m, z, mask, P, name, drop=None):
    m = _row_att(m, z, mask, P, name + "MSARowAttentionWithPairBias.", drop)
    col = name + "MSAColumnAttention."
    x = _norm(m, P, col + "layernormM").transpose(0, 1)
    m = m + _gated(x, mask.t(), None, P, col + "attention", 8).transpose(0, 1)
    return _transition(m, P, name + "MSATransition.")


def _pair(z, mask, P, name, drop=None):
    d = drop or {}
    z = _tri_mul(z, mask, P, name + "TriangleMultiplicationOutgoing.", True, d.get("tri_mul_out"))
    z = _tri_mul(z, mask, P, name + "TriangleMultiplicationIncoming.", False, d.get("tri_mul_in"))
    z = _tri_att(z, mask, P, name + "TriangleAttentionStartingNode.", False, d.get("tri_att_start"))
    z = _tri_att(z, mask, P, name + "TriangleAttentionEndingNode.", True, d.get("tri_att_end"))
    return _transition(z, P, name + "PairTransition.")


def _opm(m, mask, z, P, name):
    x = _norm(m, P, name + "layernormM")
    a, b = (_lin(x, P, name + t) * mask.unsqueeze(-1) for t in ("linear_a", "linear_b"))
    count = mask.t() @ mask + 1e-3
    w = P[name + "o_linear.weight"].view(-1, 32, 32)
    s, n = mask.shape
    out = torch.empty_like(z)
    for i in range(0, n, 16):
        o = (a[:, i:i + 16].reshape(s, -1).t() @ b.reshape(s, -1)).view(-1, 32, n, 32).permute(0, 2, 1, 3).reshape(-1, 1024)
        o = (o @ w.reshape(-1, 1024).t()).view(-1, n, z.shape[-1])
        out[i:i + 16] = z[i:i + 16] + (o + P[name + "o_linear.bias"]) / count[i:i + 16].unsqueeze(-1)
    return out


def _extra(m, z, mask, P):
    m = _row_att(m, z, mask, P, "MSARowAttentionWithPairBias.")
    col = "MSAColumnAttention."
    x, mk = _norm(m, P, col + "layernormM").transpose(0, 1), mask.t()
    g = col + "global_attention."
    q = (x * mk.unsqueeze(-1)).sum(1) / (mk.sum(-1, keepdim=True) + 1e-10)
    q = (_lin(q, P, g + "to_q") * 8 ** -0.5).view(-1, 8, 8)
    k, v = _lin(x, P, g + "to_kv").chunk(2, -1)
    a = q @ k.transpose(1, 2)
    a = torch.softmax(torch.where(mk[:, None, :] == 0, torch.full_like(a, -1e9), a), -1)
    o = (a @ v).reshape(a.shape[0], 1, -1) * torch.sigmoid(_lin(x, P, g + "gating_linear") + P[g + "gating_bias"])
    m = m + _lin(o, P, g + "o_linear").transpose(0, 1)
    return _transition(m, P, "MSATransition.")


def _ipa(st, P):
    n, h = st["s"].shape[0], IPA_HEADS
    s, z = st["s"].double(), st["z"].double()
    w, x, y, u = (st["quats"].double() / st["quats"].double().norm(dim=-1, keepdim=True)).unbind(-1)
    rot = torch.stack([1 - 2 * (y * y + u * u), 2 * (x * y - w * u), 2 * (x * u + w * y), 2 * (x * y + w * u), 1 - 2 * (x * x + u * u),
                       2 * (y * u - w * x), 2 * (x * u - w * y), 2 * (y * u + w * x), 1 - 2 * (x * x + y * y)], -1).view(n, 3, 3)
    trans = st["trans"].double()

    def points(name):                       # components lie apart: [x of all points | y | z]
        p = _lin(s, P, name).view(n, 3, -1).transpose(1, 2)
        return (p @ rot.transpose(1, 2) + trans[:, None]).view(n, h, -1, 3)
    q = _lin(s, P, "linear_q").view(n, h, -1)
    k, v = _lin(s, P, "linear_kv").view(n, h, -1).chunk(2, -1)
    qp, kvp = points("linear_q_points"), points("linear_kv_points")
    kp, vp = kvp[:, :, :IPA_QP], kvp[:, :, IPA_QP:]
    a = math.sqrt(1 / (3 * IPA_C)) * torch.einsum("ihc,jhc->hij", q, k) + math.sqrt(1 / 3) * _lin(z, P, "linear_b").permute(2, 0, 1)
    gamma = torch.nn.functional.softplus(P["head_weights"]) * math.sqrt(1.0 / (3 * (IPA_QP * 9.0 / 2)))
    a = a - 0.5 * gamma[:, None, None] * torch.cdist(qp.transpose(0, 1).flatten(2), kp.transpose(0, 1).flatten(2), compute_mode="donot_use_mm_for_euclid_dist") ** 2
    a = torch.softmax(a, -1)
    o = torch.einsum("hij,jhc->ihc", a, v).flatten(1)
    o_pt = (torch.einsum("hij,jhpx->ihpx", a, vp).flatten(1, 2) - trans[:, None]) @ rot
    o_pair = torch.einsum("hij,ijc->ihc", a, z).flatten(1)
    length = torch.sqrt((o_pt ** 2).sum(-1) + 1e-8)
    return _lin(torch.cat([o, *o_pt.unbind(-1), length, o_pair], -1), P, "linear_out")


def exact(case, seed):
    st = prepare(case, seed)
    kind = st["kind"]
    train = kind.endswith("_train")
    P = {k: p.detach().double().requires_grad_(train) for k, p in st["net"].named_parameters()}
    z = st["z"].detach().double().requires_grad_(train)
    m = st["m"].detach().double().requires_grad_(train) if "m" in st else None
    mm, pm = st["msa_mask"].double(), st["pair_mask"].double()
    if kind == "pair_train":
        drop = {"tri_mul_out": st["drop"]["tri_mul_out"].double()[0], "tri_mul_in": st["drop"]["tri_mul_in"].double()[0],
                "tri_att_start": st["drop"]["tri_att_start"].double()[0], "tri_att_end": st["drop"]["tri_att_end"].double()[0]}
        out = _pair(z, pm, P, "", drop)
        return [out[None]] + list(torch.autograd.grad(out, [z] + list(P.values()), st["up"].double()[0]))
    if kind == "msa_train":
        out = _msa(m, z, mm, P, "", st["drop_msa"].double()[0])
        grads = torch.autograd.grad(out, [m, z] + list(P.values()), st["up"].double()[0])
        return [out[None]] + [g for g, name in zip(grads, ["m", "z"] + list(P)) if not _rounding_only(name)]
    with torch.no_grad():
        if kind == "block":
            m = _msa(m, z, mm, P, "msa.")
            return m, _pair(_opm(m, mm, z, P, "communication."), pm, P, "pair.")
        if kind == "extra_msa":
            return _extra(m, z, mm, P)[None]
        if kind == "opm":
            return _opm(m, mm, z, P, "")[None]
        if kind == "ipa":
            return _ipa(st, P)
        if kind.startswith("tri_att"):
            return _tri_att(z, pm, P, "", kind == "tri_att_end")[None]
        return _tri_mul(z, pm, P, "", kind == "tri_mul_out")[None]

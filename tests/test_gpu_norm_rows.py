"""Rows of the joined norms and of the normed rotation at the sizes where their wide forms begin, end and wrap."""
from __future__ import annotations

import pytest
import torch

DEV = "cuda:0"
pytestmark = pytest.mark.gpu


def _norm(x, center, eps):
    x = x - x.mean(-1, keepdim=True) if center else x
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)


@pytest.mark.parametrize("H", [4, 508, 2048, 2052, 4096, 4100])       # a lone group; a group a thread to its end; two; the other form
@pytest.mark.parametrize("parts", [0, 2, 17])                          # a tensor; slabs in one round of loads; in two
@pytest.mark.parametrize("center", [False, True])
def test_joined_norms_of_every_row_size(H, parts, center):
    from wllm_b200.kernels import ops
    g = torch.Generator().manual_seed(H + parts)
    n, eps = 5, 1e-5
    x, bias = torch.randn(n, H, generator=g) * 2, torch.randn(H, generator=g)
    a = torch.randn(*([parts] if parts else []), n, H, generator=g)
    a = a if parts else a.bfloat16()
    wp, w = (torch.randn(H, generator=g).bfloat16() for _ in range(2))
    u = (a.double().sum(0) if parts else a.double()) + bias.double()
    r = x.double() + _norm(u, center, eps) * (1 + wp.double())
    want = _norm(r, center, eps) * (0.5 + w.double())
    resid, out = x.to(DEV), torch.empty(n, H, device=DEV)
    ops.sandwich_norm(resid, (a.to(DEV), parts), out, wp.to(DEV), center, eps, w.to(DEV), 0.5, center, eps, post_offset=1.0, bias=bias.to(DEV))
    # 32-bit sums of some twenty parts and of a row's squares: a few 2^-24 of values up to ten
    assert (resid.cpu().double() - r).abs().max() < 2e-5 and (out.cpu().double() - want).abs().max() < 2e-5
    rows = torch.tensor([3, 0], dtype=torch.int32, device=DEV)
    before, some = resid.clone(), torch.empty(2, H, device=DEV, dtype=torch.bfloat16)
    ops.sandwich_norm(resid, (a.to(DEV), parts), some, wp.to(DEV), center, eps, None, 0.0, False, 0.0, rows=rows, post_offset=1.0, bias=bias.to(DEV))
    r2 = (before.cpu().double() + _norm(u, center, eps) * (1 + wp.double()))[[3, 0]]
    assert torch.equal(before, resid) and (some.cpu().double() - r2).abs().max() <= 2.0 ** -8 * r2.abs().max() + 2e-5


@pytest.mark.parametrize("heads", [(1, 1, 8, 8, 8), (16, 4, 128, 128, 64), (16, 4, 128, 256, 128), (2, 1, 64, 64, 24)])    # one group a part; all threads once; a second round; partners that are no whole groups
@pytest.mark.parametrize("parts", [0, 1, 8, 9])                       # a bfloat16 tensor; slabs in one round of loads, in two
@pytest.mark.parametrize("biased", [False, True])
def test_turned_rows_from_tensors_and_slabs(heads, parts, biased):
    from wllm_b200.kernels import ops
    nq, nkv, hd, vd, rot = heads
    g = torch.Generator().manual_seed(hd + parts)
    n, ps, eps, qw, kw = 5, 16, 1e-5, nq * hd, nkv * hd
    x = torch.randn(*([parts] if parts else []), n, qw + kw + nkv * vd, generator=g)
    x = x if parts else x.bfloat16()
    bias = torch.randn(qw + kw + nkv * vd, generator=g) if biased else None
    q_gain, k_gain = (torch.randn(m, generator=g).bfloat16() for m in (qw, kw))
    freq = torch.tensor([100.0 ** (-2.0 * i / rot) for i in range(rot // 2)])
    positions, slots = torch.arange(40, 40 + n, dtype=torch.int32), torch.randperm(3 * ps, generator=g)[:n].to(torch.int32)
    slots[2] = -1                                                     # a row whose key and value go nowhere
    kp, vp = torch.zeros(3, nkv, ps, hd, dtype=torch.bfloat16, device=DEV), torch.zeros(3, nkv, ps, vd, dtype=torch.bfloat16, device=DEV)
    q_out = torch.empty(n, qw, dtype=torch.bfloat16, device=DEV)
    ops.rope_row_norm_kv_write(x.to(DEV), q_out, positions.to(DEV), slots.to(DEV), freq.to(DEV), kp, vp, nq, nkv, hd, rot, ps, q_gain.to(DEV),
                               k_gain.to(DEV), eps, qw, kw, in_splits=parts, vd=vd, bias=bias.to(DEV) if biased else None)
    W = x.double().sum(0) if parts else x.double()
    W = W + bias.double() if biased else W

    def turned(y, gain, m):
        y = (_norm(y, False, eps) * gain.double()).view(n, m, hd)
        a = positions.double()[:, None] * freq.double()
        c, s, lo, hi = a.cos()[:, None], a.sin()[:, None], y[..., :rot // 2], y[..., rot // 2:rot]
        return torch.cat([lo * c - hi * s, hi * c + lo * s, y[..., rot:]], -1)
    want_q, want_k, want_v = turned(W[:, :qw], q_gain, nq), turned(W[:, qw:qw + kw], k_gain, nkv), W[:, qw + kw:].view(n, nkv, vd)
    keep = slots >= 0
    sl = slots[keep].long()
    got_k, got_v = kp.cpu()[sl // ps, :, sl % ps].double(), vp.cpu()[sl // ps, :, sl % ps].double()
    for got, want in ((q_out.cpu().double().view(n, nq, hd), want_q), (got_k, want_k[keep]), (got_v, want_v[keep])):
        assert ((got - want).abs() <= 2.0 ** -8 * want.abs() + 2e-5 * want.abs().max()).all()       # one rounding to bfloat16, 32-bit before
    assert int((kp.float().abs().sum(-1) > 0).sum()) == int(keep.sum()) * nkv


@pytest.mark.parametrize("H", [4, 508, 2048, 2052, 4096, 4100])       # as above
@pytest.mark.parametrize("parts", [(0, 0), (2, 0), (17, 9)])           # of the two branches
@pytest.mark.parametrize("center", [False, True])
def test_joined_norms_of_two_branches(H, parts, center):
    from wllm_b200.kernels import ops
    g = torch.Generator().manual_seed(H + sum(parts))
    n, eps, factor = 5, 1e-5, 0.7
    x = torch.randn(n, H, generator=g) * 2
    a, b = (torch.randn(*([p] if p else []), n, H, generator=g) for p in parts)
    a, b = a if parts[0] else a.bfloat16(), b if parts[1] else b.bfloat16()
    wp, w, ga, gb = (torch.randn(H, generator=g).bfloat16() for _ in range(4))
    whole = lambda t, p: t.double().sum(0) if p else t.double()
    u = factor * (_norm(whole(a, parts[0]), False, eps) * ga.double() + _norm(whole(b, parts[1]), False, eps) * gb.double())
    r = x.double() + _norm(u, center, eps) * wp.double()
    want = _norm(r, center, eps) * (1 + w.double())
    resid, out = x.to(DEV), torch.empty(n, H, device=DEV)
    ops.sandwich_norm(resid, (a.to(DEV), parts[0]), out, wp.to(DEV), center, eps, w.to(DEV), 1.0, center, eps, gain_a=ga.to(DEV), b=(b.to(DEV), parts[1]),
                      gain_b=gb.to(DEV), inner_eps=eps, factor=factor)
    # 32-bit sums of some twenty parts and of a row's squares: a few 2^-24 of values up to ten.  (H = 4 with the mean off: u may nearly cancel, and its norm
    # divides by what is left, so the bound grows by the ratio.)
    c = u - u.mean(-1, keepdim=True) if center else u
    grown = max(1.0, float((u.abs().amax(-1) / c.pow(2).mean(-1).sqrt()).max()))
    assert (resid.cpu().double() - r).abs().max() < 2e-5 * grown and (out.cpu().double() - want).abs().max() < 2e-5 * grown * max(1.0, float(want.abs().max()))

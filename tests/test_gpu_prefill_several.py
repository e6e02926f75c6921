"""Prefill attention beside decoding requests: a launch that counts the requests of several tokens alone writes what one over all requests writes."""
from __future__ import annotations

import math

import pytest
import torch

DEV = "cuda:0"
pytestmark = pytest.mark.gpu


# several among more than a warp's lanes; at its ends and borders; all of them
@pytest.mark.parametrize("several", [{5: 70}, {0: 33, 31: 300, 32: 2, 63: 129}, {40: 17, 69: 40}, "all"])
@pytest.mark.parametrize("hd", [128, 256])
def test_requests_of_several_tokens_are_found(several, hd):
    from wllm_b200.kernels import ops
    R, nq, nkv, ps = 70, 8, 1, 64
    several = {r: 20 + r % 3 for r in range(R)} if several == "all" else several
    g = torch.Generator().manual_seed(len(several) + hd)
    q_lens = [several.get(r, 1) for r in range(R)]
    ctx = [n + (37 * r) % 150 for r, n in enumerate(q_lens)]
    starts = [sum(q_lens[:r]) for r in range(R)]
    width = -(-max(ctx) // ps)
    pages = torch.randperm(R * width, generator=g).view(R, width).to(torch.int32).to(DEV)
    q = torch.randn(sum(q_lens), nq * hd, generator=g).bfloat16().to(DEV)
    k, v = (torch.randn(R * width, nkv, ps, hd, generator=g).bfloat16().to(DEV) for _ in range(2))
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)
    outs = []
    for multi in (0, len(several)):
        out = torch.full_like(q, 7.0)
        ops.attention_mma_prefill(q, out, k, v, i32(starts), i32(q_lens), i32(ctx), pages, max(q_lens), nq, nkv, hd, ps, 0, 1 / math.sqrt(hd),
                                  skip_single=True, multi=multi)
        outs.append(out)
    assert torch.equal(*outs)
    rows = torch.zeros(q.shape[0], dtype=torch.bool)
    for r in several:
        rows[starts[r]:starts[r] + q_lens[r]] = True
    assert bool((outs[0][~rows.to(DEV)] == 7).all()) and bool((outs[0][rows.to(DEV)] != 7).any(dim=1).all())
    r = max(several)                                        # the last one against the formula
    keys, vals = (t[pages[r].long()].permute(1, 0, 2, 3).reshape(width * ps, hd)[:ctx[r]].double() for t in (k, v))
    x = q[starts[r]:starts[r] + q_lens[r]].double().view(q_lens[r], nq, hd) @ keys.t() / math.sqrt(hd)
    pos = torch.arange(ctx[r] - q_lens[r], ctx[r], device=DEV)
    x = x.masked_fill(torch.arange(ctx[r], device=DEV)[None, None] > pos[:, None, None], -math.inf)
    want = torch.softmax(x, -1) @ vals
    got = outs[1][starts[r]:starts[r] + q_lens[r]].double().view_as(want)
    assert float((got - want).norm() / want.norm()) < 6e-3          # weights and results rounded to bfloat16

"""32-bit attention of portions of prompts, dealt out by chunks of keys, beside the tiled kernel: the same bits."""
from __future__ import annotations

import pytest
import torch

DEV = "cuda:0"
pytestmark = pytest.mark.gpu


# portions that end in a tile of rows, of keys, of a chunk, one past and one short of them; on cached keys; single tokens beside them
@pytest.mark.parametrize("lens,before", [([64], [0]), ([1, 33, 65], [0, 5, 63]), ([31, 1, 127, 128], [200, 300, 1, 0]), ([190], [131])])
@pytest.mark.parametrize("nq,nkv,hd,vd,ps", [(8, 1, 256, 256, 64), (4, 4, 16, 16, 16), (6, 2, 72, 40, 16), (4, 2, 128, 256, 32)])
@pytest.mark.parametrize("extra", ["plain", "all"])
def test_chunks_give_the_tiled_kernels_bits(lens, before, nq, nkv, hd, vd, ps, extra):
    from wllm_b200.kernels import ops
    g = torch.Generator().manual_seed(sum(lens) + hd)
    R, n, ctx = len(lens), sum(lens), [m + b for m, b in zip(lens, before)]
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)
    pages = [-(-c // ps) for c in ctx]
    table, at = torch.zeros(R, max(pages) + 1, dtype=torch.int32), 1
    order = torch.randperm(sum(pages), generator=g) + 1
    for r, p in enumerate(pages):
        table[r, :p] = order[at - 1:at - 1 + p]
        at += p
    # what lies behind a request's last key in its page is no number
    k, v = (torch.full((sum(pages) + 1, nkv, ps, d), float("nan")) for d in (hd, vd))
    for r, c in enumerate(ctx):
        for key in range(c):
            page = int(table[r, key // ps])
            k[page, :, key % ps], v[page, :, key % ps] = torch.randn(nkv, hd, generator=g), torch.randn(nkv, vd, generator=g)
    q = torch.randn(n, nq * hd + 8, generator=g).to(DEV)[:, :nq * hd]
    meta = (i32([sum(lens[:r]) for r in range(R)]), i32(lens), i32(ctx), table.to(DEV))
    positions = i32([b + j for m, b in zip(lens, before) for j in range(m)])
    more = dict(sinks=torch.randn(nq, generator=g).to(DEV), cap=3.0, slopes=torch.rand(nq, generator=g).to(DEV)) if extra == "all" else {}
    want, got = (torch.full((n, nq * vd), float("nan"), device=DEV) for _ in range(2))
    ops.paged_attention_simt_tiled(q, want, k.to(DEV), v.to(DEV), *meta, max(lens), nq, nkv, hd, ps, 0, hd ** -0.5, vd=vd, **more)
    chunks = -(-max(ctx) // 64)
    scratch = torch.full((n * nq * chunks * (vd + 2),), float("nan"), device=DEV)
    ops.paged_attention_simt_chunks(q, got, k.to(DEV), v.to(DEV), positions, *meta, max(lens), nq, nkv, hd, ps, hd ** -0.5, scratch, chunks, vd=vd, **more)
    assert bool(want.isfinite().all()) and torch.equal(want, got)


def test_pools_and_tables_that_do_not_fit_are_refused():
    """What the kernel indexes by: rows of hd and vd elements, a table of two axes, chunks that hold the longest context."""
    from wllm_b200.kernels import ops
    n, nq, nkv, hd, vd, ps, ctx = 4, 2, 1, 32, 16, 16, 70
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)
    z = lambda *shape: torch.zeros(shape, device=DEV)
    args = dict(q=z(n, nq * hd), out=z(n, nq * vd), k_pages=z(6, nkv, ps, hd), v_pages=z(6, nkv, ps, vd), positions=i32([66, 67, 68, 69]), req_q_start=i32([0]),
                req_q_len=i32([n]), req_ctx_len=i32([ctx]), block_table=i32([[1, 2, 3, 4, 5]]), max_q_len=n, nq=nq, nkv=nkv, hd=hd, page_size=ps, scale=0.2,
                scratch=z(n * nq * 2 * (vd + 2)), max_chunks=2, vd=vd, max_ctx=ctx)
    ops.paged_attention_simt_chunks(**args)
    for wrong in (dict(k_pages=z(6, nkv, ps, 16)), dict(v_pages=z(6, nkv, ps, 8)), dict(k_pages=args["v_pages"], v_pages=args["k_pages"]),
                  dict(block_table=i32([1, 2, 3, 4, 5])), dict(max_chunks=1), dict(scratch=args["scratch"][:-1])):
        with pytest.raises(AssertionError):
            ops.paged_attention_simt_chunks(**{**args, **wrong})


# requests of more than a warp's lanes, some that bring nothing, long contexts behind few rows and the other way round
@pytest.mark.parametrize("lens,before", [([70, 0, 1, 33], [10, 40, 300, 63]), ([1, 0, 3] * 15 + [150] + [1] * 30, [5 + 29 * i for i in range(76)]), ([17], [1000])])
@pytest.mark.parametrize("nq,nkv,hd", [(8, 1, 64), (6, 2, 32)])
def test_every_request_has_ctas_of_its_own_rows_and_keys(lens, before, nq, nkv, hd):
    import numpy as np

    from wllm_b200.kernels import ops
    ps, R, n, ctx = 16, len(lens), sum(lens), [m + b for m, b in zip(lens, before)]
    g = torch.Generator().manual_seed(n)
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)
    width = -(-max(ctx) // ps)
    table = torch.arange(R * width, dtype=torch.int32, device=DEV).view(R, width)
    k, v = (torch.randn(R * width, nkv, ps, hd, generator=g).to(DEV) for _ in range(2))
    q = torch.randn(n, nq * hd, generator=g).to(DEV)
    meta = (i32([sum(lens[:r]) for r in range(R)]), i32(lens), i32(ctx), table)
    positions = i32([b + j for m, b in zip(lens, before) for j in range(m)])
    want, got = (torch.full((n, nq * hd), float("nan"), device=DEV) for _ in range(2))
    ops.paged_attention_simt_tiled(q, want, k, v, *meta, max(lens), nq, nkv, hd, ps, 0, 0.1)
    chunks, rep = -(-max(ctx) // 64), nq // nkv
    pairs = ops.simt_chunk_pairs(np.array(lens, dtype=np.int32), np.array(ctx, dtype=np.int32), rep)
    assert pairs == sum(-(-m * rep // 32) * -(-c // 64) for m, c in zip(lens, ctx))
    scratch = torch.full((n * nq * chunks * (hd + 2),), float("nan"), device=DEV)
    ops.paged_attention_simt_chunks(q, got, k, v, positions, *meta, max(lens), nq, nkv, hd, ps, 0.1, scratch, chunks, max_ctx=max(ctx), pairs=pairs)
    assert bool(want.isfinite().all()) and torch.equal(want, got)

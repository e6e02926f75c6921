"""32-bit products of more than 32 rows: tile edges, segments' ends, tiles of 64 and 128 rows whose CTAs walk their segments or that are cut by them, beside the same
rows in smaller products."""
from __future__ import annotations

import math

import pytest
import torch

DEV = "cuda:0"
pytestmark = pytest.mark.gpu


# rows and columns one past, at and one short of a tile; K within a stage, of one segment, one group past it, of several, its last one short;
# (M, N) of few tiles, whose segments have CTAs of their own (tiles of 64 rows; the sixth and eighth of 128), and of more, of 128 rows, whose CTAs walk them
@pytest.mark.parametrize("M,N,K", [(65, 1, 4), (127, 129, 1024), (128, 128, 1028), (129, 255, 2048), (300, 130, 5000), (1100, 8501, 1060), (1030, 8320, 3076),
                                   (1030, 5300, 2052), (2100, 15801, 1060)])
def test_every_row_has_the_bits_of_a_smaller_product(M, N, K):
    from wllm_b200.kernels import ops
    g = torch.Generator().manual_seed(M + N + K)
    a, w = torch.randn(M, K + 4, generator=g).to(DEV)[:, :K], torch.randn(N, K, generator=g).to(DEV)
    out = torch.full((M, N + 3), float("nan"), device=DEV)
    ops.gemm_f32(a, w, out[:, :N])
    # 32-bit accumulation error grows with sqrt(K)
    assert float((out[:, :N].double() - a.double() @ w.double().t()).abs().max()) < 2e-5 * math.sqrt(K)
    assert bool(out[:, N:].isnan().all())
    for rows in (slice(0, 32), slice(M - 40, M), slice(M // 2, M // 2 + 1)):        # the few-rows kernels and the 64-row tile
        assert torch.equal(ops.gemm_f32(a[rows], w), out[rows, :N])


# K of 3 to 5 segments; the last one short; two and more turns, the last of one segment; tiles of 64 rows, and of 128 (the last)
@pytest.mark.parametrize("M,N,K", [(65, 130, 2060), (300, 129, 5120), (130, 256, 4100), (1400, 2050, 4100)])
def test_less_scratch_gives_the_same_bits(M, N, K, monkeypatch):
    """Room for every slab, for four, three and two, for one and for none; memory that runs out on the way; operands that lie across 16 bytes ask for none."""
    import ctypes

    from wllm_b200.kernels import ops
    from wllm_b200.kernels.build import load_family
    g = torch.Generator().manual_seed(M + K)
    a, w = torch.randn(M, K + 4, generator=g).to(DEV), torch.randn(N, K, generator=g).to(DEV)
    want = ops.gemm_f32(a[:, :K], w)
    lib = load_family("gemm_f32")
    query = lambda x: lib.wllm_gemm_f32_scratch_floats(ops._ptr(x), x.stride(0), ops._ptr(w), K, M, N, K)
    assert query(a[:, :K]) == -(-K // 1024) * M * N and query(a[:, 1:K + 1]) == 0
    for slabs in (4, 3, 2, 1, 0):
        out, scratch = torch.full((M, N + 3), float("nan"), device=DEV), torch.full((max(slabs, 1) * M * N,), float("nan"), device=DEV)
        status = lib.wllm_gemm_f32(ops._ptr(a), K + 4, ops._ptr(w), K, ops._ptr(out), N + 3, M, N, K, ops._ptr(scratch if slabs else None),
                                   ctypes.c_longlong(slabs * M * N), ops._stream())
        assert status == 0 and torch.equal(out[:, :N], want) and bool(out[:, N:].isnan().all()), slabs
    out, empty = torch.empty(M, N, device=DEV), torch.empty

    def no_room(*args, **kw):
        raise torch.OutOfMemoryError("none left")
    monkeypatch.setattr(torch, "empty", no_room)
    ops.gemm_f32(a[:, :K], w, out)
    monkeypatch.setattr(torch, "empty", empty)
    assert torch.equal(out, want)


def test_scratch_of_a_large_product_is_bounded():
    import ctypes

    from wllm_b200.kernels.build import load_family
    lib = load_family("gemm_f32")
    lib.wllm_gemm_f32_scratch_floats.restype = ctypes.c_longlong
    query = lambda M, N, K: lib.wllm_gemm_f32_scratch_floats(ctypes.c_void_p(4096), K, ctypes.c_void_p(4096), K, M, N, K)       # (pointers are looked at, not read)
    assert query(509, 2048, 16384) == 16 * 509 * 2048
    assert 0 < query(2400, 2048, 16384) <= 64 << 20 and 0 < query(2048, 2048, 1 << 20) <= 64 << 20 and 0 < query(4096, 2048, 16384) <= 64 << 20

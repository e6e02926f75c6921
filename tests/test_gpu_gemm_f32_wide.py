"""32-bit products of more than 64 rows: tile edges, segments' ends, both ways of adding the segments, beside the same rows in smaller products."""
from __future__ import annotations

import math

import pytest
import torch

DEV = "cuda:0"
pytestmark = pytest.mark.gpu


# rows and columns one past, at and one short of a tile; K within a stage, of one segment, one group past it, of several, its last one short;
# (M, N) of many tiles, whose segments one CTA walks, and of few, whose segments have CTAs of their own
@pytest.mark.parametrize("M,N,K", [(65, 1, 4), (127, 129, 1024), (128, 128, 1028), (129, 255, 2048), (300, 130, 5000), (1100, 8501, 1060), (1030, 8320, 3076)])
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

"""Latent attention over whole prompts with every head's own keys and values: how they are laid out, and steps beside the same steps over the latent rows and beside a
64-bit statement."""
from __future__ import annotations

import pytest
import torch

DEV = "cuda:0"
pytestmark = pytest.mark.gpu


# pages that end with a prompt, one past and one short of it; prompts shorter than a page, that begin anywhere in the step
@pytest.mark.parametrize("lens", [[64], [1, 65, 63], [130, 3, 64, 127, 200]])
@pytest.mark.parametrize("heads,dim", [(3, 64), (2, 128)])
def test_pages_hold_every_token_once(lens, heads, dim):
    from wllm_b200.kernels import ops
    n, R = sum(lens), len(lens)
    starts = [sum(lens[:r]) for r in range(R)]
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)
    kv = torch.randn(n, 2 * heads * dim, generator=torch.Generator().manual_seed(n)).bfloat16().to(DEV)
    keys, values = (torch.full((n // 64 + R, heads, 64, dim), float("nan"), dtype=torch.bfloat16, device=DEV) for _ in range(2))
    table = torch.full((R, -(-max(lens) // 64)), -9, dtype=torch.int32, device=DEV)
    req = i32([r for r, m in enumerate(lens) for _ in range(m)])
    ops.latent_expand(kv, req, i32(starts), i32(lens), keys, values, table, heads, dim)
    used = set()
    for r, m in enumerate(lens):
        pages, k = table[r].tolist(), -(-m // 64)
        assert all(p == 0 for p in pages[k:]) and not used & set(pages[:k])
        used |= set(pages[:k])
        for part, src in ((keys, kv[:, :heads * dim]), (values, kv[:, heads * dim:])):
            got = part[pages[:k]].transpose(1, 2).reshape(-1, heads * dim)
            assert torch.equal(got[:m], src[starts[r]:starts[r] + m]) and bool(got[m:].isnan().all())


@pytest.mark.parametrize("dim,q_rank", [(64, 40), (128, 48)])
def test_whole_prompts_are_no_further_from_64_bits_than_over_latent_rows(dim, q_rank, monkeypatch):
    import plain_gudarax as plain

    from wllm_b200.config import EngineConfig, resolve_architecture
    from wllm_b200.engine import ComposedModel, StepEntry, build_runner
    from wllm_b200.kernels import ops
    from wllm_b200.parts.latent_attention import LatentAttention
    layer = {"type": "latent_attention", "mlp": {"kind": "dense", "ff": 96},
             "mixer": {"heads": 4, "dim": dim, "vdim": dim, "kv_rank": 96, "q_rank": q_rank, "scale": dim ** -0.5}}
    raw = {"architecture": "Gudarax", "vocab": 211, "width": 64, "max_positions": 4096, "norm": {"eps": 1e-6}, "embedding": {"scale": 1.0},
           "token_side": {"dim": 16}, "layers": [layer] * 2}
    arch = resolve_architecture("Gudarax")
    cfg = arch.config_class.from_dict(raw, where="test")
    ran, far = [], {1: 0.0, 1 << 30: 0.0}
    expand = ops.latent_expand

    def spy(*args):
        ran.append(1)
        expand(*args)
    monkeypatch.setattr(ops, "latent_expand", spy)
    for seed in range(4):
        gen = torch.Generator().manual_seed(dim + seed)
        weights = {}
        for ps in ComposedModel(arch.make_plan(cfg), torch.bfloat16).param_specs():
            shape = tuple(ps.shape)
            t = torch.randn(shape, generator=gen) * (1.0 if ps.name.endswith("embed") else 0.3 if len(shape) > 1 else 0.1)
            weights[ps.name] = (t + (1.0 if len(shape) == 1 else 0.0)).bfloat16()
        draw = lambda n: torch.randint(0, 211, (n,), generator=gen).tolist()
        prompts, tails = [draw(n) for n in (300, 129, 64, 2)], [draw(n) for n in (1, 70, 1, 1)]
        wide = {k: v.double() for k, v in weights.items()}
        want = [plain.forward(raw, wide, p + t) for p, t in zip(prompts, tails)]
        for least in far:
            monkeypatch.setattr(LatentAttention, "EXPAND_FROM", least)
            model = ComposedModel(arch.make_plan(cfg), torch.bfloat16)
            model.load(lambda name: weights[name].to(DEV))
            model.config = cfg
            runner = build_runner(model, EngineConfig(dtype="bfloat16", block_size=16, max_num_seqs=4, device=DEV), num_pages=80)
            rcs = [runner.cache.open(i) for i in range(4)]
            ran.clear()
            got = runner.step([StepEntry(rc, p, range(len(p))) for rc, p in zip(rcs, prompts)])
            ref = torch.cat([w[:len(p)] for w, p in zip(want, prompts)])
            far[least] += float((got.cpu().double() - ref).norm() / ref.norm()) ** 2
            assert len(ran) == (2 if least == 1 else 0)
            # portions and single tokens on the cached rows
            got = runner.step([StepEntry(rc, t, [len(t) - 1]) for rc, t in zip(rcs, tails)]).cpu().double()
            ref = torch.stack([w[-1] for w in want])
            assert len(ran) == (2 if least == 1 else 0) and float((got - ref).norm() / ref.norm()) < 0.1
    # roundings to bfloat16 that fall on keys and values in place of mapped queries and mixed rows: as many, and over 2,000 rows of two layers as far
    assert far[1] <= 1.1 * far[1 << 30], far

"""The mixers that go in chunks of 64 tokens, at sizes that reach them: steps of bfloat16 models beside the 64-bit statement and beside the same steps walked token by
token; the decay's low-rank map on the tensor cores."""
from __future__ import annotations

import pytest
import torch

DEV = "cuda:0"
pytestmark = pytest.mark.gpu


def _weights(specs, gen) -> dict:
    """Matrices that keep the heads' numbers near one; gains around one; decays from about a token's memory to a thousand's."""
    out = {}
    for ps in specs:
        name, shape = ps.name, tuple(ps.shape)
        if name.endswith(".a2.b"):
            t = torch.rand(shape, generator=gen) * 8.0 - 3.0
        elif name.endswith((".A_log", ".dt_bias")):
            t = torch.rand(shape, generator=gen) * 4.0 - 3.0
        elif len(shape) == 1:
            t = 1.0 + 0.3 * torch.randn(shape, generator=gen)
        else:
            t = torch.randn(shape, generator=gen) * (1.0 if name.endswith("embed") else 0.1)
        out[name] = t.bfloat16()
    return out


def _pesanex(*layers):
    return {"architecture": "Pesanex", "vocab": 97, "width": 128, "norm": {"eps": 1e-6}, "layers": list(layers)}


def _gla(heads, dim, vdim, tau, rank):
    return {"heads": heads, "dim": dim, "vdim": vdim, "tau": tau, "rank": rank}


def _delta(kind, heads, kv_heads):
    more = {"decay_rank": 24, "gate_rank": 16} if kind == "channel_delta" else {}
    return {"type": kind, "mlp": {"kind": "dense", "ff": 64}, "mixer": {"heads": heads, "kv_heads": kv_heads, "dim": 128, "vdim": 128, "conv": 4, **more}}


MODELS = {
    "gla 64": _pesanex({"type": "gla", "mlp": None, "mixer": _gla(2, 64, 64, 4.0, 24)}),
    "gla 128": _pesanex({"type": "gla", "mlp": None, "mixer": _gla(2, 128, 128, 16.0, 40)}),
    "retention 64, turned": _pesanex({"type": "retention", "mlp": None, "mixer": {"heads": 3, "dim": 64, "vdim": 128, "decay": [0.9, 0.99, 1.0], "rot": {"dims": 32, "base": 500.0}}}),
    "retention 128, turned": _pesanex({"type": "retention", "mlp": None, "mixer": {"heads": 2, "dim": 128, "vdim": 64, "decay": [0.97, 0.999], "rot": {"dims": 128, "base": 1e4}}}),
    "parallel": _pesanex({"type": "parallel", "mlp": None, "mixer": {"left": {"heads": 2, "kv_heads": 1, "dim": 64, "vdim": 64, "scale": 0.2, "rot": {"dims": 32, "base": 1e4}},
                                                                     "right": _gla(2, 64, 128, 8.0, 16)}}),
    "delta": {"architecture": "Gudarax", "vocab": 97, "width": 128, "max_positions": 4096, "embedding": {"scale": 1.0}, "norm": {"eps": 1e-6}, "token_side": {"dim": 16},
              "layers": [_delta("delta", 4, 2)]},
    "channel_delta": {"architecture": "Vifirax", "vocab": 97, "width": 128, "norm": {"eps": 1e-6}, "logit_scale": 0.5, "layers": [_delta("channel_delta", 3, 3)]},
}


def _plain(name, cfg, w, tokens):
    import plain_gudarax
    import plain_pesanex
    import plain_vifirax
    if cfg["architecture"] == "Pesanex":
        return plain_pesanex.forward(tokens, w, cfg)
    return (plain_gudarax if cfg["architecture"] == "Gudarax" else plain_vifirax).forward(cfg, w, tokens)


@pytest.mark.parametrize("name", list(MODELS))
def test_steps_in_chunks_are_no_further_from_64_bits_than_walked_ones(name, monkeypatch):
    from wllm_b200.config import EngineConfig, resolve_architecture
    from wllm_b200.engine import ComposedModel, StepEntry, build_runner
    from wllm_b200.kernels import ops
    from wllm_b200.parts.linear_attention import DeltaRule, LinearAttention
    raw = MODELS[name]
    arch = resolve_architecture(raw["architecture"])
    cfg = arch.config_class.from_dict(raw, where="test")
    mixer, which = (DeltaRule, "delta_chunks") if "delta" in name else (LinearAttention, "linattn_chunks")
    ran, fn = [], getattr(ops, which)

    def spy(*args, **kw):
        ran.append(1)
        return fn(*args, **kw)
    monkeypatch.setattr(ops, which, spy)
    far = {True: 0.0, False: 0.0}
    for seed in range(2):
        gen = torch.Generator().manual_seed(40 + seed)
        weights = _weights(ComposedModel(arch.make_plan(cfg), torch.bfloat16).param_specs(), gen)
        draw = lambda n: torch.randint(0, 97, (n,), generator=gen).tolist()
        # a prompt beside ones of a chunk and a bit, short and single ones; then a portion from the states that these left, beside single tokens
        prompts, tails = [draw(n) for n in (620, 70, 20, 9, 1)], [draw(n) for n in (1, 640, 1, 3, 40)]
        wide = {k: v.double() for k, v in weights.items()}
        want = [_plain(name, raw, wide, p + t) for p, t in zip(prompts, tails)]
        ref = torch.cat([w[:len(p)] for w, p in zip(want, prompts)] + [w[len(p):] for w, p in zip(want, prompts)])
        rows = {}
        for chunks in (True, False):
            with monkeypatch.context() as m:
                if not chunks:
                    m.setattr(mixer, "_chunk_room", lambda self, ctx: 0)
                    if mixer is DeltaRule:
                        m.setattr(mixer, "REQUEST_FROM", 1 << 30)          # not in blocks either
                model = ComposedModel(arch.make_plan(cfg), torch.bfloat16)
                model.load(lambda key: weights[key].to(DEV))
                model.config = cfg
                runner = build_runner(model, EngineConfig(dtype="bfloat16", block_size=16, max_num_seqs=6, device=DEV), num_pages=200)
                caches = [runner.cache.open(i) for i in range(6)]
                runner.cache.close(caches.pop(0))                         # (slots and places in the step differ)
                ran.clear()
                got = [runner.step([StepEntry(rc, t, range(len(t))) for rc, t in zip(caches, part)]).cpu().double() for part in (prompts, tails)]
                assert len(ran) == (2 if chunks else 0)
                rows[chunks] = torch.cat(got)
                far[chunks] += float((rows[chunks] - ref).norm() / ref.norm()) ** 2
        assert bool(rows[True].isfinite().all())
    # the same products in bfloat16 around a recurrence whose 32-bit sums run in another order
    assert far[True] <= 1.1 * far[False] and far[False] < 2 * 0.1 ** 2, far


# tokens at the edges of the 64 that a CTA takes; ranks that are no steps of 16, channels that are no steps of 128; too few tokens for the tensor cores
@pytest.mark.parametrize("n", [63, 64, 65, 200])
@pytest.mark.parametrize("heads,dim,rank,tau", [(2, 64, 8, 4.0), (3, 40, 24, 1.0), (5, 64, 72, 16.0), (8, 128, 64, 16.0), (8, 128, 256, 16.0)])
def test_the_decay_of_linear_attention_alone(n, heads, dim, rank, tau):
    from wllm_b200.kernels import ops
    gen = torch.Generator().manual_seed(n + rank)
    HD, off = heads * dim, 16
    low = torch.randn(n, off + rank + 8, generator=gen).bfloat16().to(DEV)
    w2, b2 = (torch.randn(HD, rank, generator=gen) * 0.4).bfloat16().to(DEV), (torch.rand(HD, generator=gen) * 8 - 3).bfloat16().to(DEV)
    want = torch.nn.functional.logsigmoid(low[:, off:off + rank].double() @ w2.double().t() + b2.double()) / tau
    alone, beside = (torch.full((n, HD), float("nan"), device=DEV) for _ in range(2))
    ops.linattn_decay(low, 0, off, w2, b2, heads, dim, alone, tau=tau)
    # what the walk's preparation makes of the same columns, on the FMA pipes
    wide = torch.cat([torch.zeros(n, 3 * HD, device=DEV).bfloat16(), low], 1)
    q, k, v = (torch.empty(n, HD, device=DEV) for _ in range(3))
    ops.linattn_prepare(wide, 0, 0, HD, 2 * HD, heads, dim, dim, torch.arange(n, dtype=torch.int32, device=DEV), q, k, v, low_off=3 * HD + off, w2=w2, b2=b2, tau=tau,
                        decay=beside)
    far = lambda a: float((a.double() - want.exp()).norm() / want.exp().norm())
    # a decay of 32 bits is within some roundings of 2^-24; the map's sum of `rank` products, in either order, is no further off
    assert far(alone) <= 1.03 * far(beside), (far(alone), far(beside))
    forgets = want < -0.01                       # where the logarithm tells more than the rounding of the decay itself
    logs = lambda a: float(((a.double().log() - want)[forgets] / want[forgets]).abs().max())
    assert logs(alone) <= max(1.5 * logs(beside), 2e-5), (logs(alone), logs(beside))

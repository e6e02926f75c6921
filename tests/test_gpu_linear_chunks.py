"""The decayed-state recurrence in chunks on the tensor cores: ends of chunks and of blocks, several requests, turns, fast and slow decays, against 64 bits and beside
the token by token walk."""
from __future__ import annotations

import numpy as np
import pytest
import torch

DEV = "cuda:0"
pytestmark = pytest.mark.gpu


def _case(lens, H, D, V, rot, per_channel, seed, speed="mixed"):
    g = torch.Generator().manual_seed(seed)
    n, W = sum(lens), 2 * H * D + H * V + 40
    c = dict(lens=lens, H=H, D=D, V=V, rot=rot, off=(8, 8 + H * D, 16 + 2 * H * D), q_scale=0.37, k_scale=1.9)
    c["fused"] = torch.randn(n, W, generator=g).bfloat16()
    # channels that forget within a token, within some, hardly, never and at once
    low, high = {"mixed": (-30.0, 12.0), "slow": (4.0, 9.0)}[speed]
    a = torch.sigmoid(torch.rand(n, H * D, generator=g) * (high - low) + low)
    if speed == "mixed":
        a[torch.rand(n, H * D, generator=g) < 0.02] = 0.0
        a[torch.rand(n, H * D, generator=g) < 0.02] = 1.0
    c["decay"] = a if per_channel else None
    c["head_decay"] = None if per_channel else torch.tensor([0.5, 1.0, 0.999, 0.97][:H])
    c["inv_freq"] = torch.tensor([1e4 ** (-2.0 * i / max(rot, 1)) for i in range(rot // 2)])
    c["positions"] = torch.cat([torch.arange(7 * i, 7 * i + m) for i, m in enumerate(lens)]).int()
    c["slots"] = [2, 0, 3, 1, 5, 6][:len(lens)]
    c["state"] = torch.randn(7, H, D, V, generator=g)
    return c


def _meta(c):
    lens = c["lens"]
    starts = [sum(lens[:i]) for i in range(len(lens))]
    return [torch.tensor(x, dtype=torch.int32, device=DEV) for x in (starts, lens, c["slots"])]


def _run(c, scratch_bytes=None):
    from wllm_b200.kernels import ops
    H, D, V, lens = c["H"], c["D"], c["V"], np.array(c["lens"], dtype=np.int32)
    n = int(lens.sum())
    dev = lambda t: None if t is None else t.to(DEV)
    state, out = dev(c["state"]).clone(), torch.full((n, H * V), float("nan"), device=DEV)
    need = ops.linattn_chunks_bytes(lens, H, D, V)
    scratch = torch.full((need if scratch_bytes is None else scratch_bytes,), 0xff, dtype=torch.uint8, device=DEV)      # (NaN in every type)
    ops.linattn_chunks(dev(c["fused"]), *c["off"], H, D, V, dev(c["positions"]), dev(c["decay"]), dev(c["head_decay"]), state, out, *_meta(c), lens, scratch,
                       q_scale=c["q_scale"], k_scale=c["k_scale"], inv_freq=dev(c["inv_freq"]) if c["rot"] else None, rot_dim=c["rot"])
    return out, state


def _walk(c):
    from wllm_b200.kernels import ops
    H, D, V, n = c["H"], c["D"], c["V"], sum(c["lens"])
    dev = lambda t: None if t is None else t.to(DEV)
    q, k, v = (torch.empty(n, H * x, device=DEV) for x in (D, D, V))
    state, out = dev(c["state"]).clone(), torch.empty(n, H * V, device=DEV)
    ops.linattn_prepare(dev(c["fused"]), 0, *c["off"], H, D, V, dev(c["positions"]), q, k, v, q_scale=c["q_scale"], k_scale=c["k_scale"],
                        inv_freq=dev(c["inv_freq"]) if c["rot"] else None, rot_dim=c["rot"])
    ops.linattn_scan(q, k, v, dev(c["decay"]), dev(c["head_decay"]), state, out, *_meta(c), H, D, V)
    return out, state


def _exact(c):
    H, D, V, lens = c["H"], c["D"], c["V"], c["lens"]
    f, rot = c["fused"].double().to(DEV), c["rot"]
    angle = c["positions"].float()[:, None].to(DEV) * c["inv_freq"][None].to(DEV)          # (the turn's angle is a 32-bit product in both)
    sn, cs = torch.sin(angle.double())[:, None], torch.cos(angle.double())[:, None]

    def turned(x):
        u, w = x[..., :rot // 2], x[..., rot // 2:rot]
        return torch.cat([u * cs - w * sn, w * cs + u * sn, x[..., rot:]], -1)
    n = sum(lens)
    q = turned(f[:, c["off"][0]:][:, :H * D].reshape(n, H, D)) * c["q_scale"]
    k = turned(f[:, c["off"][1]:][:, :H * D].reshape(n, H, D)) * c["k_scale"]
    v = f[:, c["off"][2]:][:, :H * V].reshape(n, H, V)
    a = c["decay"].double().to(DEV).view(n, H, D) if c["decay"] is not None else c["head_decay"].double().to(DEV)[None, :, None].expand(n, H, D)
    state, out, t = c["state"].double().to(DEV).clone(), torch.empty(n, H, V, dtype=torch.float64, device=DEV), 0
    for length, slot in zip(lens, c["slots"]):
        S = state[slot]
        for _ in range(length):
            S = S * a[t][:, :, None] + k[t][:, :, None] * v[t][:, None, :]
            out[t] = (q[t][:, None, :] @ S)[:, 0]
            t += 1
        state[slot] = S
    return out.view(n, H * V), state


def _off(x, want):
    return float((x.double() - want).norm() / want.norm())


# ends of a block, a chunk and a tile of the chunk's rows, one past and one short of them; requests too short for chunks
@pytest.mark.parametrize("per_channel,speed", [(True, "mixed"), (True, "slow"), (False, "mixed")])
@pytest.mark.parametrize("lens,H,D,V,rot", [([64], 1, 64, 64, 0), ([1, 16, 8, 9, 15, 17], 2, 64, 64, 16), ([65, 127, 128, 129, 63], 3, 128, 64, 128), ([300, 1, 40], 4, 128, 192, 64),
                                            ([1000], 2, 128, 256, 128)])
def test_chunks_are_no_further_from_64_bits_than_the_walk(lens, H, D, V, rot, per_channel, speed):
    c = _case(lens, H, D, V, rot, per_channel, seed=sum(lens) + D, speed=speed)
    want, want_state = _exact(c)
    (o, s), (wo, ws) = _run(c), _walk(c)
    # a rounding at 2^-24 for every of some hundred additions, at random; the walk's own distance where that is larger
    assert _off(o, want) <= max(1.05 * _off(wo, want), 4e-7), (_off(o, want), _off(wo, want))
    assert _off(s, want_state) <= max(1.05 * _off(ws, want_state), 2e-7), (_off(s, want_state), _off(ws, want_state))
    assert torch.equal(s[4], c["state"][4].to(DEV))        # nobody's slot


def test_less_scratch_takes_more_turns_and_gives_the_same_bits():
    from wllm_b200.kernels import ops
    c = _case([500, 64, 130, 1], 2, 128, 64, 0, True, 5)
    o, s = _run(c)
    one = ops.linattn_chunks_bytes(np.array([64], dtype=np.int32), 2, 128, 64)
    for chunks in (3, 5, 7, 11):
        o2, s2 = _run(c, scratch_bytes=chunks * one)
        assert torch.equal(o, o2) and torch.equal(s, s2), chunks
    with pytest.raises(ops.KernelError):
        _run(c, scratch_bytes=2 * one)                     # not a chunk of every request that goes in chunks


def test_many_requests_and_empty_ones():
    lens = [3 if i % 5 else 0 for i in range(70)] + [150]
    c = _case(lens, 1, 64, 64, 0, False, 9)
    c["slots"], c["state"] = list(range(len(lens))), torch.randn(len(lens), 1, 64, 64)
    want, want_state = _exact(c)
    o, s = _run(c)
    assert _off(o, want) < 4e-7 and _off(s, want_state) < 4e-7


@pytest.mark.parametrize("value", [float("nan"), float("inf"), 3e38])
@pytest.mark.parametrize("column", ["q", "k", "v"])
def test_a_token_that_is_no_number_reaches_none_in_front_of_it(column, value):
    c = _case([100, 90], 2, 128, 64, 0, True, 3, speed="slow")
    clean, _ = _run(c)
    at = 100 + 41                                          # inside the second request's first chunk
    c["fused"][at, c["off"]["qkv".index(column)] + 5] = value
    o, s = _run(c)
    same = torch.ones(190, dtype=torch.bool)
    same[at:] = False
    assert torch.equal(o[same], clean[same]) if column != "v" else torch.allclose(o[same], clean[same], rtol=1e-4, atol=1e-4)
    assert torch.equal(o[:100], clean[:100]) and bool(o[:at].isfinite().all())
    if value != value:
        assert bool(o[at].isnan().any()) and bool(s[0].isnan().any()) == (column != "q")

"""The delta rule in chunks of 64 tokens on the tensor cores, beside the walk token by token, the walk in blocks and the recurrence in 64 bits."""
from __future__ import annotations

import numpy as np
import pytest
import torch
from test_gpu_delta_blocks import _plain

DEV = "cuda:0"
pytestmark = pytest.mark.gpu
D = 128


def _case(lens, H, G, memory, channel, seed):
    gen = torch.Generator().manual_seed(seed)
    n, R = sum(lens), len(lens)
    unit = lambda x: x / x.norm(dim=-1, keepdim=True)
    q, k = unit(torch.randn(n, G, D, generator=gen)) * D ** -0.5, unit(torch.randn(n, G, D, generator=gen) + 0.3)
    v, beta = torch.randn(n, H, D, generator=gen), torch.rand(n, H, generator=gen)
    lo, hi = {"short": (0.5, 40.0), "long": (1e-4, 1e-2), "mixed": (1e-4, 40.0)}[memory]
    rate = lo * (hi / lo) ** torch.rand(n, H, D if channel else 1, generator=gen).double()
    decay = (torch.expm1(-rate) if channel else torch.exp(-rate)[..., 0]).float()
    state = torch.randn(2 * R, H, D, D, generator=gen)
    return q, k, v, beta, decay, state, [(2 * i + 1) % (2 * R) for i in range(R)]


def _run(way, lens, H, G, channel, q, k, v, beta, decay, state, slots, share=1.0):
    from wllm_b200.kernels import ops
    n, R = sum(lens), len(lens)
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)
    d = lambda x: x.reshape(x.shape[0], -1).contiguous().to(DEV)
    starts, host = [sum(lens[:i]) for i in range(R)], np.array(lens, dtype=np.int32)
    S, o = state.clone().to(DEV), torch.full((n, H * D), float("nan"), device=DEV)
    if way == "chunks":
        scratch = torch.full((int(ops.delta_chunks_bytes(host, H) * share),), 255, dtype=torch.uint8, device=DEV)
        ops.delta_chunks(d(q), d(k), d(v), d(beta), d(decay), S, o, i32(starts), i32(lens), i32(slots), host, H, G, channel, scratch)
    else:
        scratch = torch.full((ops.delta_block_floats(n, R, H, D),), float("nan"), device=DEV) if way == "blocks" else None
        ops.delta_scan(d(q), d(k), d(v), d(beta), d(decay), S, o, i32(starts), i32(lens), i32(slots), H, G, D, D, channel, scratch, max(lens))
    return o.view(n, H, D).cpu(), S.cpu()


# around a chunk and the first length that goes in one, beside requests that do not; several chunks
@pytest.mark.parametrize("lens", [[64], [16, 1, 65, 15, 63], [0, 200, 24], [333, 2]])
@pytest.mark.parametrize("heads", [(2, 1), (3, 3)])
@pytest.mark.parametrize("memory", ["short", "long", "mixed"])                   # decays near 0, near 1, both
@pytest.mark.parametrize("channel", [False, True])
def test_chunks_give_the_recurrence(lens, heads, memory, channel):
    H, G = heads
    case = _case(lens, H, G, memory, channel, sum(lens) * 7 + H + channel)
    q, k, v, beta, decay, state, slots = case
    g = (1 + decay.double()) if channel else decay.double()[..., None]
    want, want_o, s0 = state.double().clone(), torch.zeros(sum(lens), H, D, dtype=torch.float64), 0
    for m, slot in zip(lens, slots):
        part, rep = slice(s0, s0 + m), H // G
        s0 += m
        if m:
            want_o[part], want[slot] = _plain(q[part].double().repeat_interleave(rep, 1), k[part].double().repeat_interleave(rep, 1), v[part].double(),
                                              beta[part].double(), g[part], state[slot].double())
    errors = {}
    for way in ("walk", "blocks", "chunks"):
        o, S = _run(way, lens, H, G, channel, *case)
        errors[way] = float((o.double() - want_o).norm() / want_o.norm()), float((S.double() - want).norm() / want.norm())
    # 32-bit sums of 128 channels and up to 64 tokens in another order, on numbers of 24 bits: of the size of the two walks' own roundings
    for i in range(2):
        assert errors["chunks"][i] <= 1.5 * max(errors["walk"][i], errors["blocks"][i]) + 2e-7, errors


def test_turns_give_the_same_bits():
    lens = [300, 1, 130]
    case = _case(lens, 2, 1, "long", True, 3)
    want = _run("chunks", lens, 2, 1, True, *case)
    for share in (0.5, 0.26):          # of eight chunks four and two: the fewest, one of each request
        got = _run("chunks", lens, 2, 1, True, *case, share=share)
        assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])


@pytest.mark.parametrize("channel", [False, True])
def test_a_value_that_is_no_number_stays_with_its_column_and_later_tokens(channel):
    lens = [150]
    q, k, v, beta, decay, state, slots = _case(lens, 2, 2, "long", channel, 5)
    want = _run("chunks", lens, 2, 2, channel, q, k, v, beta, decay, state, slots)
    for bad in (float("inf"), float("nan")):
        v2 = v.clone()
        v2[70, 1, 17] = bad
        o, _ = _run("chunks", lens, 2, 2, channel, q, k, v2, beta, decay, state, slots)
        other = torch.ones(D, dtype=torch.bool)
        other[17] = False
        assert not bool(o[70:, 1, 17].isfinite().any())
        assert torch.equal(o[:, 0], want[0][:, 0]) and torch.equal(o[:64, 1], want[0][:64, 1])
        # (the chunk's rows are added up token by token then)
        assert bool(o[64:70, 1].isfinite().all()) and float((o[64:, 1][:, other] - want[0][64:, 1][:, other]).abs().max()) < 1e-5


# a block's first token, inside a tile of sixteen, a chunk's first, the last of a partly filled chunk
@pytest.mark.parametrize("at", [72, 85, 64, 149])
@pytest.mark.parametrize("bad", ["v", "k", "q", "beta", "decay"])
@pytest.mark.parametrize("what", [float("inf"), float("nan")])
@pytest.mark.parametrize("channel", [False, True])
def test_what_is_no_number_reaches_no_earlier_token(at, bad, what, channel):
    lens, H = [150], 2
    case = dict(zip(("q", "k", "v", "beta", "decay", "state", "slots"), _case(lens, H, 2, "long", channel, 7)))
    run = lambda way: _run(way, lens, H, 2, channel, *case.values())
    clean_o, clean_S = run("chunks")
    case[bad] = case[bad].clone()
    case[bad][(at, 0, 9) if case[bad].dim() == 3 else (at, 0)] = what
    (o, S), (walk_o, walk_S) = run("chunks"), run("walk")
    slot, chunk = case["slots"][0], at - at % 64
    assert torch.equal(o[:chunk], clean_o[:chunk]) and torch.equal(o[:, 1], clean_o[:, 1]) and torch.equal(S[slot, 1], clean_S[slot, 1])
    # (the chunk's earlier tokens are added up one by one then: up to 64 sums of numbers of the outputs' size, each rounded at 2^-24)
    assert float((o[chunk:at] - clean_o[chunk:at]).abs().max() if at > chunk else 0.0) < 1e-5
    assert bool(o.isfinite()[walk_o.isfinite()].all()) and bool(S.isfinite()[walk_S.isfinite()].all())
    assert not bool(o[at, 0].isfinite().all())


# (lens, whether the chunks pay): full chunks, mostly empty ones, a portion beside single tokens, too short
@pytest.mark.parametrize("lens,chunks", [([2048], True), ([704, 20], True), ([512] + [20] * 30, False), ([1531] + [1] * 24, True), ([127], False), ([130], False)])
def test_which_steps_go_in_chunks(lens, chunks):
    from types import SimpleNamespace

    from wllm_b200.kernels import ops
    from wllm_b200.parts.linear_attention import DeltaRule
    host = np.array(lens, dtype=np.int32)
    rule = DeltaRule.__new__(DeltaRule)
    rule.heads, rule.dim, rule.vdim, rule.model_dtype = 16, 128, 128, torch.bfloat16
    ctx = lambda: SimpleNamespace(host={"req_q_len": host}, memo={}, max_q_len=max(lens))
    assert rule._chunk_room(ctx()) == (ops.delta_chunks_bytes(host, 16) if chunks else 0)
    rule.model_dtype = torch.float32              # (the same bits under every cut)
    assert rule._chunk_room(ctx()) == 0
    rule.model_dtype, rule.vdim = torch.bfloat16, 64
    assert rule._chunk_room(ctx()) == 0


@pytest.mark.parametrize("channel", [False, True])
def test_chunks_are_no_further_from_64_bits_than_the_walks(channel):
    """Decays as such models are initialised and stay: rates A softplus(a + bias), A of 1 to 16, steps of 1e-3 to 1e-1."""
    lens, H, far = [700, 130], 3, {}
    for seed in range(3):
        gen = torch.Generator().manual_seed(seed)
        q, k, v, beta, _, state, slots = _case(lens, H, H, "long", channel, 20 + seed)
        width = D if channel else 1
        A, step = 1 + 15 * torch.rand(H, 1, generator=gen), 1e-3 * 100.0 ** torch.rand(H, width, generator=gen)
        rate = (A * torch.nn.functional.softplus(0.9 * torch.randn(sum(lens), H, width, generator=gen) + step + torch.log(-torch.expm1(-step)))).double()
        decay = (torch.expm1(-rate) if channel else torch.exp(-rate)[..., 0]).float()
        g = (1 + decay.double()) if channel else decay.double()[..., None]
        want, want_o = state.double().clone(), torch.zeros(sum(lens), H, D, dtype=torch.float64)
        for m, slot, s0 in zip(lens, slots, (0, lens[0])):
            part = slice(s0, s0 + m)
            want_o[part], want[slot] = _plain(q[part].double(), k[part].double(), v[part].double(), beta[part].double(), g[part], state[slot].double())
        for way in ("walk", "blocks", "chunks"):
            o, S = _run(way, lens, H, H, channel, q, k, v, beta, decay, state, slots)
            a, b = far.get(way, (0.0, 0.0))
            far[way] = a + float((o.double() - want_o).norm() / want_o.norm()) / 3, b + float((S.double() - want)[slots].norm() / want[slots].norm()) / 3
    # (three drawings; a hundredth or two between them)
    for i in range(2):
        assert far["chunks"][i] <= 1.02 * max(far["walk"][i], far["blocks"][i]), far

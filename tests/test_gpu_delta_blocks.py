"""The delta rule in blocks of tokens, beside the walk token by token and the recurrence in 64 bits."""
from __future__ import annotations

import pytest
import torch

DEV = "cuda:0"
pytestmark = pytest.mark.gpu


def _plain(q, k, v, beta, g, S):
    """q, k [n, H, D], v [n, H, V], beta [n, H], g [n, H, D or 1], S [H, D, V]; 64 bits."""
    out = []
    for t in range(q.shape[0]):
        S = S * g[t][:, :, None]
        u = beta[t][:, None] * (v[t] - torch.einsum("hdv,hd->hv", S, k[t]))
        S = S + k[t][:, :, None] * u[:, None, :]
        out.append(torch.einsum("hdv,hd->hv", S, q[t]))
    return torch.stack(out), S


# lengths around a block and the first length that is walked in blocks, beside requests that are not; a long one
@pytest.mark.parametrize("lens", [[16], [1, 23, 15, 17, 1], [24, 0, 200]])
@pytest.mark.parametrize("sizes", [(2, 1, 8, 5), (3, 3, 72, 16), (4, 2, 128, 128), (1, 1, 256, 33)])      # channels a thread; ragged columns
@pytest.mark.parametrize("memory", ["short", "long", "mixed"])                                           # decays near 0, near 1, both
@pytest.mark.parametrize("channel", [False, True])
def test_blocks_of_tokens_give_the_recurrence(lens, sizes, memory, channel):
    from wllm_b200.kernels import ops
    H, G, D, V = sizes
    gen = torch.Generator().manual_seed(sum(lens) * 7 + D + channel)
    n, R = sum(lens), len(lens)
    unit = lambda x: x / x.norm(dim=-1, keepdim=True)
    q, k = unit(torch.randn(n, G, D, generator=gen)) * D ** -0.5, unit(torch.randn(n, G, D, generator=gen) + 0.3)
    v, beta = torch.randn(n, H, V, generator=gen), torch.rand(n, H, generator=gen)
    lo, hi = {"short": (0.5, 40.0), "long": (1e-4, 1e-2), "mixed": (1e-4, 40.0)}[memory]
    x = torch.rand(n, H, D if channel else 1, generator=gen)
    rate = lo * (hi / lo) ** x.double()
    decay = (torch.expm1(-rate) if channel else torch.exp(-rate)[..., 0]).float()
    g = (1 + decay.double()) if channel else decay.double()[..., None]
    starts = [sum(lens[:i]) for i in range(R)]
    slots = [(2 * i + 1) % (2 * R) for i in range(R)]
    state = torch.randn(2 * R, H, D, V, generator=gen)
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)
    rep = H // G
    want = state.double().clone()
    want_o = torch.zeros(n, H, V, dtype=torch.float64)
    for s0, m, slot in zip(starts, lens, slots):
        if m:
            part = slice(s0, s0 + m)
            want_o[part], want[slot] = _plain(q[part].double().repeat_interleave(rep, 1), k[part].double().repeat_interleave(rep, 1), v[part].double(),
                                              beta[part].double(), g[part], state[slot].double())
    d = lambda x: x.reshape(x.shape[0], -1).contiguous().to(DEV)
    errors = {}
    for way in ("walk", "blocks"):
        S, o = state.clone().to(DEV), torch.full((n, H * V), float("nan"), device=DEV)
        scratch = torch.full((ops.delta_block_floats(n, R, H, D),), float("nan"), device=DEV) if way == "blocks" else None
        ops.delta_scan(d(q), d(k), d(v), d(beta), d(decay), S, o, i32(starts), i32(lens), i32(slots), H, G, D, V, channel, scratch, max(lens))
        err_o = (o.cpu().double().view(n, H, V) - want_o).norm() / want_o.norm()
        err_s = (S.cpu().double() - want).norm() / want.norm()
        errors[way] = float(err_o), float(err_s)
    # 32-bit sums over D channels and eight tokens: some 2^-24 sqrt(D) of the result, and no further off than token by token by more
    # than the scatter of such sums
    for a, b in zip(errors["walk"], errors["blocks"]):
        assert b < 2e-6 and b < 1.5 * a + 1e-7, errors


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("sizes", [(2, 1, 8, 5), (4, 2, 128, 128), (1, 1, 200, 256)])       # a part of a warp's lanes; all of them; two rounds
@pytest.mark.parametrize("lens", [[2800], [3, 2797, 1], [1030, 7, 1766]])                  # runs that end in the middle and hold several requests
def test_runs_of_tokens_are_prepared_as_one_by_one(lens, sizes, dtype):
    """A step of so many tokens takes the kernel that walks runs; the same requests in portions of at most 31 tokens do not: the same bits."""
    from wllm_b200.kernels import ops
    H, G, D, V = sizes
    gen = torch.Generator().manual_seed(sum(lens) + D)
    n, R, C, T = sum(lens), len(lens), 2 * G * D + H * V, 4
    off = {"q": 0, "k": G * D, "v": 2 * G * D, "b": C, "a": C + H}
    fused = torch.randn(n, C + 2 * H + 3, generator=gen).to(dtype).to(DEV)
    taps = [torch.randn(c, T, generator=gen).to(dtype).to(DEV) for c in (G * D, G * D, H * V)]
    a_log, dt_bias = (torch.randn(H, generator=gen).to(dtype).to(DEV) for _ in range(2))
    starts = [sum(lens[:i]) for i in range(R)]
    conv0 = torch.randn(R, T - 1, C, generator=gen)
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)

    def run(pieces):
        """pieces: [(request, from, to)] lists, one a step; the outputs of all tokens."""
        conv, res = conv0.clone().to(DEV), [torch.empty(n, w, device=DEV) for w in (G * D, G * D, H * V, H, H)]
        for step in pieces:
            rows = torch.cat([torch.arange(starts[r] + a, starts[r] + b) for r, a, b in step]).to(DEV)
            x, m = fused[rows].contiguous(), [b - a for _, a, b in step]
            at = [sum(m[:i]) for i in range(len(m))]
            req = torch.cat([torch.full((c,), i, dtype=torch.int32) for i, c in enumerate(m)]).to(DEV)
            part = [torch.empty(sum(m), t.shape[1], device=DEV) for t in res]
            slots = i32([r for r, _, _ in step])
            ops.delta_prepare(x, 0, off, H, G, D, V, T, *taps, a_log, dt_bias, req, i32(at), slots, conv, 1e-6, D ** -0.5, *part)
            ops.delta_conv_update(x, 0, off, H, G, D, V, T, i32(at), i32(m), slots, conv)
            for t, p in zip(res, part):
                t[rows] = p
        return res + [conv]
    whole = run([[(r, 0, m) for r, m in enumerate(lens)]])
    cut = run([[(r, a, min(a + 31, m))] for r, m in enumerate(lens) for a in range(0, m, 31)])
    assert all(torch.equal(a, b) for a, b in zip(whole, cut))


@pytest.mark.parametrize("sizes", [(2, 1, 33, 5), (3, 3, 64, 64), (4, 2, 128, 128), (2, 2, 100, 65), (1, 1, 256, 200)])     # channels a thread; ragged columns
@pytest.mark.parametrize("channel", [False, True])
def test_single_tokens_have_the_walks_bits(sizes, channel):
    from wllm_b200.kernels import ops
    H, G, D, V = sizes
    R = 5
    gen = torch.Generator().manual_seed(D + V + channel)
    rand = lambda *shape: torch.randn(*shape, generator=gen).to(DEV)
    q, k, v, beta = rand(R, G * D), rand(R, G * D), rand(R, H * V), torch.sigmoid(rand(R, H))
    rate = torch.exp(3 * rand(R, H * D if channel else H) - 3)
    decay = torch.expm1(-rate) if channel else torch.exp(-rate)
    state = rand(2 * R, H, D, V)
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)
    index = i32([0, 1, 2, 3, 4]), i32([1, 1, 0, 1, 1]), i32([3, 0, 5, -1, 9])          # one brings no token, one has no slot
    res = []
    for single in (False, True):
        S, o = state.clone(), torch.full((R, H * V), float("nan"), device=DEV)
        ops.delta_scan(q, k, v, beta, decay, S, o, *index, H, G, D, V, channel, single=single)
        res.append((S, torch.nan_to_num(o, nan=-1.0)))
    assert torch.equal(res[0][0], res[1][0]) and torch.equal(res[0][1], res[1][1])
    assert not torch.equal(res[1][0], state)


@pytest.mark.parametrize("parts", [0, 1, 17])                         # a tensor; a slab; more than are asked for at once
@pytest.mark.parametrize("sizes", [(2, 1, 8, 5), (4, 2, 128, 128), (1, 1, 200, 256)])
def test_single_tokens_are_prepared_as_portions_of_one(parts, sizes):
    """With the slots' inputs brought up to date in the same kernel, beside the two kernels of steps with portions: the same bits."""
    from wllm_b200.kernels import ops
    H, G, D, V = sizes
    gen = torch.Generator().manual_seed(parts + D)
    R, C, T = 5, 2 * G * D + H * V, 4
    off = {"q": 0, "k": G * D, "v": 2 * G * D, "b": C, "a": C + H}
    fused = torch.randn(*([parts] if parts else []), R, C + 2 * H, generator=gen).to(DEV)
    taps = [torch.randn(c, T, generator=gen).to(DEV) for c in (G * D, G * D, H * V)]
    a_log, dt_bias = (torch.randn(H, generator=gen).to(DEV) for _ in range(2))
    conv0 = torch.randn(2 * R, T - 1, C, generator=gen).to(DEV)
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)
    starts, lens, slots = i32([0, 1, 2, 3, 4]), i32([1, 1, 0, 1, 1]), i32([3, 0, 5, -1, 9])      # one brings no token, one has no slot
    res = []
    for shift in (None, lens):
        conv, out = conv0.clone(), [torch.empty(R, w, device=DEV) for w in (G * D, G * D, H * V, H, H)]
        ops.delta_prepare(fused, parts, off, H, G, D, V, T, *taps, a_log, dt_bias, starts, starts, slots, conv, 1e-6, D ** -0.5, *out, shift=shift)
        if shift is None:
            ops.delta_conv_update(fused, parts, off, H, G, D, V, T, starts, lens, slots, conv)
        res.append(out + [conv])
    assert all(torch.equal(a, b) for a, b in zip(*res))


@pytest.mark.parametrize("bad", ["v", "k", "q", "beta", "decay"])
@pytest.mark.parametrize("what", [float("inf"), float("nan")])
@pytest.mark.parametrize("n,at", [(24, 13), (24, 8), (17, 16)])                # inside a block; its first token; a portion's last, beside places past its end
@pytest.mark.parametrize("channel", [False, True])
def test_what_is_no_number_reaches_no_earlier_token(n, at, what, bad, channel):
    """One input that overflowed: the tokens in front of it, the other head and (for a value) the other columns keep their bits, and what the walk
    token by token leaves finite is finite."""
    from wllm_b200.kernels import ops
    H, D, V = 2, 72, 20
    gen = torch.Generator().manual_seed(n + at)
    rand = lambda *shape: torch.randn(*shape, generator=gen).to(DEV)
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)
    unit = lambda x: (x / x.norm(dim=-1, keepdim=True)).reshape(n, -1).contiguous()
    arg = {"q": unit(rand(n, H, D)), "k": unit(rand(n, H, D)), "v": rand(n, H * V), "beta": torch.sigmoid(rand(n, H))}
    rate = torch.exp(rand(n, H * D if channel else H) - 3)
    arg["decay"], state = torch.expm1(-rate) if channel else torch.exp(-rate), rand(1, H, D, V)
    place = {"v": 5, "k": 7, "q": 7, "beta": 0, "decay": 7 if channel else 0}[bad]         # head 0

    def run(arg, blocks):
        S, o = state.clone(), torch.empty(n, H * V, device=DEV)
        scratch = torch.full((ops.delta_block_floats(n, 1, H, D),), float("nan"), device=DEV) if blocks else None
        ops.delta_scan(*arg.values(), S, o, i32([0]), i32([n]), i32([0]), H, H, D, V, channel, scratch, n)
        return o.view(n, H, V), S[0]
    clean_o, clean_S = run(arg, True)
    arg[bad] = arg[bad].clone()
    arg[bad][at, place] = what
    (o, S), (walk_o, walk_S) = run(arg, True), run(arg, False)
    assert torch.equal(o[:at], clean_o[:at]) and torch.equal(o[:, 1], clean_o[:, 1]) and torch.equal(S[1], clean_S[1])
    if bad == "v":
        others = [c for c in range(V) if c != 5]
        assert torch.equal(o[:, 0, others], clean_o[:, 0, others]) and torch.equal(S[0][:, others], clean_S[0][:, others])
    assert bool(o.isfinite()[walk_o.isfinite()].all()) and bool(S.isfinite()[walk_S.isfinite()].all())
    assert not bool(o[at, 0].isfinite().all())


@pytest.mark.parametrize("several", [{40: 50, 71: 16, 72: 200}, {0: 31, 31: 17, 32: 24, 63: 90}, {69: 70}])      # among more than a warp's lanes; at its borders
@pytest.mark.parametrize("order", ["ascending", "descending"])                                                       # of the requests' tokens in the step
@pytest.mark.parametrize("channel", [False, True])
def test_requests_in_blocks_are_found_beside_single_tokens(several, order, channel):
    """A launch that counts the requests in blocks alone, one over all requests, and the walk token by token, beside 70 requests of one token."""
    from wllm_b200.kernels import ops
    H, G, D, V = 2, 1, 40, 20
    R = max(70, max(several) + 1)
    lens = [several.get(r, 1) for r in range(R)]
    n, gen = sum(lens), torch.Generator().manual_seed(len(several))
    by_place = range(R) if order == "ascending" else range(R - 1, -1, -1)
    starts, at = [0] * R, 0
    for r in by_place:
        starts[r], at = at, at + lens[r]
    rand = lambda *shape: torch.randn(*shape, generator=gen).to(DEV)
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)
    unit = lambda x: (x / x.norm(dim=-1, keepdim=True)).reshape(n, -1).contiguous()
    rate = torch.exp(rand(n, H * D if channel else H) - 3)
    args = unit(rand(n, G, D)), unit(rand(n, G, D)), rand(n, H * V), torch.sigmoid(rand(n, H)), torch.expm1(-rate) if channel else torch.exp(-rate)
    state, res = rand(R, H, D, V), []
    for walked in (len(several), 0, None):
        S, o = state.clone(), torch.full((n, H * V), float("nan"), device=DEV)
        scratch = None if walked is None else torch.full((ops.delta_block_floats(n, R, H, D),), float("nan"), device=DEV)
        ops.delta_scan(*args, S, o, i32(starts), i32(lens), i32(range(R)), H, G, D, V, channel, scratch, max(lens), walked=walked or 0)
        res.append((o, S))
    (o, S), (all_o, all_S), (walk_o, walk_S) = res
    assert torch.equal(o, all_o) and torch.equal(S, all_S)
    # two orders of 32-bit sums over 40 channels and 200 tokens
    assert float((o - walk_o).norm() / walk_o.norm()) < 2e-6 and float((S - walk_S).norm() / walk_S.norm()) < 2e-6
    ones = [starts[r] for r in range(R) if lens[r] == 1]
    assert torch.equal(o[ones], walk_o[ones])


@pytest.mark.parametrize("channel", [False, True])
def test_portions_in_turns_have_the_bits_of_one(channel):
    """Scratch for every block, for some blocks of each request down to one, and for less."""
    from wllm_b200.kernels import ops
    H, G, D, V, lens = 2, 1, 72, 20, [24, 1, 0, 203, 16, 9]
    R, n, gen = len(lens), sum(lens), torch.Generator().manual_seed(3)
    rand = lambda *shape: torch.randn(*shape, generator=gen).to(DEV)
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)
    unit = lambda x: (x / x.norm(dim=-1, keepdim=True)).reshape(n, -1).contiguous()
    rate = torch.exp(rand(n, H * D if channel else H) - 3)
    args = unit(rand(n, G, D)), unit(rand(n, G, D)), rand(n, H * V), torch.sigmoid(rand(n, H)), torch.expm1(-rate) if channel else torch.exp(-rate)
    state, res = rand(R, H, D, V), []
    floats = ops.delta_block_floats(8, 0, H, D)                       # of a block
    starts = [sum(lens[:r]) for r in range(R)]
    for blocks, walked in ((n // 8 + R, 3), (15, 3), (3 * 13, 3), (6, 3), (3, 3), (6, 0)):
        S, o = state.clone(), torch.full((n, H * V), float("nan"), device=DEV)
        scratch = torch.full((blocks * floats,), float("nan"), device=DEV)
        ops.delta_scan(*args, S, o, i32(starts), i32(lens), i32(range(R)), H, G, D, V, channel, scratch, max(lens), walked=walked)
        res.append((o, S))
    assert all(torch.equal(o, res[0][0]) and torch.equal(S, res[0][1]) for o, S in res) and bool(res[0][0].isfinite().all())
    with pytest.raises(ops.KernelError):
        ops.delta_scan(*args, state.clone(), o, i32(starts), i32(lens), i32(range(R)), H, G, D, V, channel, scratch[:2 * floats], max(lens), walked=3)


def test_scratch_of_long_portions_is_bounded():
    from wllm_b200.kernels import ops
    assert ops.delta_block_floats(2048, 1, 16, 128) == 257 * 16 * (25 * 128 + 64)
    assert ops.delta_block_floats(16384, 1, 64, 128) <= 32 << 20 and ops.delta_block_floats(1 << 20, 4, 32, 256) <= 32 << 20


@pytest.mark.parametrize("design", ["Vifirax", "Gudarax"])                  # a decay per key channel, per head
def test_a_long_portion_beside_many_single_tokens(design, monkeypatch):
    """A whole bfloat16 step: a prompt that is walked in blocks, a short one and forty decoded tokens that are not; then a step of single tokens from the
    states it left.  Beside the same steps by the walk alone."""
    from wllm_b200.config import EngineConfig, resolve_architecture
    from wllm_b200.engine import ComposedModel, StepEntry, build_runner
    from wllm_b200.kernels import ops
    from wllm_b200.parts.linear_attention import DeltaRule
    dense, mixer = {"kind": "dense", "ff": 96}, {"heads": 4, "kv_heads": 2, "dim": 40, "vdim": 24, "conv": 4}
    raw = {"architecture": design, "vocab": 211, "width": 64, "norm": {"eps": 1e-6}, "layers": [
        {"type": "delta", "mlp": dense, "mixer": mixer} if design == "Gudarax" else
        {"type": "channel_delta", "mlp": dense, "mixer": {**mixer, "kv_heads": 4, "decay_rank": 8, "gate_rank": 8}}] * 2}
    if design == "Gudarax":
        raw.update(max_positions=4096, embedding={"scale": 1.0}, token_side={"dim": 16})
    arch = resolve_architecture(design)
    cfg = arch.config_class.from_dict(raw, where=design)
    gen = torch.Generator().manual_seed(5)
    weights = {}
    model = ComposedModel(arch.make_plan(cfg), torch.bfloat16)
    for ps in model.param_specs():
        shape = tuple(ps.shape)
        t = torch.randn(shape, generator=gen) * (1.0 if ps.name.endswith("embed") else 0.3 if len(shape) > 1 else 0.1)
        weights[ps.name] = (t + (1.0 if len(shape) == 1 and design == "Gudarax" else 0.0)).bfloat16().to(DEV)
    draw = lambda n: torch.randint(0, 211, (n,), generator=gen).tolist()
    prompt, short, firsts, seconds, thirds = draw(620), draw(30), [draw(3) for _ in range(40)], draw(40), draw(42)
    asked = []
    plain_scan = ops.delta_scan

    def spy(*args, **kw):
        asked.append((args[15] is not None, args[18]))
        return plain_scan(*args, **kw)
    monkeypatch.setattr(ops, "delta_scan", spy)

    def steps(blocks):
        if not blocks:
            monkeypatch.setattr(DeltaRule, "BLOCKS_FROM", 1 << 30)
            monkeypatch.setattr(DeltaRule, "CHANNEL_BLOCKS_FROM", 1 << 30)
        model = ComposedModel(arch.make_plan(cfg), torch.bfloat16)
        model.load(weights.__getitem__)
        model.config = cfg
        runner = build_runner(model, EngineConfig(dtype="bfloat16", block_size=64, max_num_seqs=42, device=DEV), num_pages=64)
        rcs = [runner.cache.open(i) for i in range(42)]
        runner.step([StepEntry(rc, t, []) for rc, t in zip(rcs, firsts)])
        asked.clear()
        out = [runner.step([StepEntry(rc, [t], [0]) for rc, t in zip(rcs[:20], seconds)] + [StepEntry(rcs[40], prompt, [0, 299, 619])] +
                           [StepEntry(rc, [t], [0]) for rc, t in zip(rcs[20:40], seconds[20:])] + [StepEntry(rcs[41], short, [29])])]
        assert asked == [(blocks, 1 if blocks else 0)] * 2, asked
        return out + [runner.step([StepEntry(rc, [t], [0]) for rc, t in zip(rcs, thirds)])]
    for got, want in zip(steps(True), steps(False)):
        # two programs whose 32-bit sums fall differently, rounded to bfloat16 in two layers
        assert bool(got.isfinite().all()) and float((got - want).norm() / want.norm()) < 2.5e-2


@pytest.mark.parametrize("parts", [0, 1, 2, 9, 17])                    # a tensor; a slab; fewer than are asked for at once; more
@pytest.mark.parametrize("lens", [[5, 1, 9], [120, 1, 40], [3] * 40])    # CTAs that lie on the device at once; more of them; more requests
def test_inputs_in_slabs_are_their_sums(parts, lens):
    """The convolutions' inputs and kept inputs from slabs, however many loads are in flight, beside the same from their sum, added up in order."""
    from wllm_b200.kernels import ops
    H, G, D, V, T = 32, 16, 40, 24, 4
    gen = torch.Generator().manual_seed(parts + len(lens))
    n, R, C = sum(lens), len(lens), 2 * G * D + H * V
    off = {"q": 0, "k": G * D, "v": 2 * G * D, "b": C, "a": C + H}
    fused = torch.randn(*([parts] if parts else []), n, C + 2 * H, generator=gen).to(DEV)
    whole = fused if not parts else fused[0].clone()
    for part in fused[1:] if parts else ():
        whole += part
    taps = [torch.randn(c, T, generator=gen).to(DEV) for c in (G * D, G * D, H * V)]
    a_log, dt_bias = (torch.randn(H, generator=gen).to(DEV) for _ in range(2))
    conv0 = torch.randn(R, T - 1, C, generator=gen).to(DEV)
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)
    starts, slots = i32([sum(lens[:r]) for r in range(R)]), i32(range(R))
    req = torch.cat([torch.full((m,), r, dtype=torch.int32) for r, m in enumerate(lens)]).to(DEV)
    res = []
    for x, p in ((fused, parts), (whole, 0)):
        conv, out = conv0.clone(), [torch.empty(n, w, device=DEV) for w in (G * D, G * D, H * V, H, H)]
        ops.delta_prepare(x, p, off, H, G, D, V, T, *taps, a_log, dt_bias, req, starts, slots, conv, 1e-6, D ** -0.5, *out)
        ops.delta_conv_update(x, p, off, H, G, D, V, T, starts, i32(lens), slots, conv)
        res.append(out + [conv])
    assert all(torch.equal(a, b) for a, b in zip(*res))

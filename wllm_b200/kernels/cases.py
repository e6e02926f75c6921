"""Single-kernel cases: run one kernel of the engine on synthetic operands, time it with CUDA events and
print what it achieved against the roofline.  The same command under `ncu` gives the profiles in profiles/.

    python -m wllm_b200.kernels.cases gemm --m 2048 --n 32768 --k 2048 --epilogue gelu_tanh
    python -m wllm_b200.kernels.cases gemm --m 8 --n 2048 --k 16384 --split
    python -m wllm_b200.kernels.cases attention-decode --requests 16 --context 8192
    python -m wllm_b200.kernels.cases attention-prefill --requests 1 --tokens 2048 --context 2048
    python -m wllm_b200.kernels.cases sampling --rows 8 --vocab 256000 --top-k 50 --top-p 0.9
    python -m wllm_b200.kernels.cases gemm-f32 --m 16 --n 49152 --k 3072
    python -m wllm_b200.kernels.cases attention-f32 --requests 16 --context 6000 --tokens 1 --heads 16 --kv-heads 16
    python -m wllm_b200.kernels.cases recurrence --requests 1 --tokens 2048 --heads 8 --dim 128 --vdim 256
    python -m wllm_b200.kernels.cases recurrence --chunks --requests 1 --tokens 2048 --heads 8 --dim 128 --vdim 256
    python -m wllm_b200.kernels.cases recurrence --delta --requests 1 --tokens 2048 --heads 16 --dim 128 --vdim 128
    python -m wllm_b200.kernels.cases experts --tokens 2048 --experts 32 --top 4 --width 2048 --ff 1024

Operands are larger than L2 where the case is bound by memory (several weight copies are cycled), so the
figures are DRAM figures.  Peaks: MEASURED_PEAKS.json at the repository root when present, else the fallback
6.65 TB/s and 1.59 PFLOP/s.
"""
from __future__ import annotations

import argparse
import json
import math
import os
import sys

import numpy as np
import torch

from . import ops

DEV = "cuda:0"


def peaks():
    path = os.path.join(os.path.dirname(os.path.dirname(os.path.dirname(os.path.abspath(__file__)))), "MEASURED_PEAKS.json")
    try:
        with open(path) as f:
            raw = json.load(f)
        return float(raw["hbm_gbs"]), float(raw["bf16_tflops"]), "measured"
    except (OSError, ValueError, KeyError):
        return 6650.0, 1590.0, "fallback"


def timed(fn, iters: int, warmup: int = 3) -> float:
    """Milliseconds per call, CUDA events around `iters` calls after `warmup`."""
    for _ in range(warmup):
        fn()
    torch.cuda.synchronize()
    start, end = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    start.record()
    for _ in range(iters):
        fn()
    end.record()
    torch.cuda.synchronize()
    return start.elapsed_time(end) / iters


def gemm(args) -> None:
    M, N, K = args.m, args.n, args.k
    a = (torch.randn(M, K, device=DEV) * 0.1).to(torch.bfloat16)
    copies = max(1, min(8, int(300e6 // (N * K * 2)) + 1))       # cycle weights so that they come from DRAM
    ws = [(torch.randn(N, K, device=DEV) * 0.1).to(torch.bfloat16) for _ in range(copies)]
    parts = ops.split_plan(M, N, K) if args.split else 1
    code = args.epilogue
    if parts > 1:
        out = torch.empty((parts, M, N), dtype=torch.float32, device=DEV)
    else:
        cols = N // 2 if code in ("gelu_tanh", "silu") else N
        out = torch.empty((M, cols), dtype=torch.float32 if code == "f32" or args.split else torch.bfloat16, device=DEV)
    i = [0]

    def run():
        i[0] += 1
        w = ws[i[0] % copies]
        if parts > 1:
            ops.gemm_bf16_tc(a, w, out, "f32", k_splits=parts)
        else:
            ops.gemm_bf16_tc(a, w, out, "f32" if args.split else code, half_rows=args.half_rows or None)
    ms = timed(run, args.iters)
    hbm, tf, src = peaks()
    flops, byts = 2.0 * M * N * K, (N * K + M * K) * 2.0 + out.numel() * out.element_size()
    print(f"gemm_bf16_tc M={M} N={N} K={K} epilogue={code} parts={parts}: {ms * 1e3:.1f} us, "
          f"{flops / ms / 1e9:.1f} TFLOP/s ({flops / ms / 1e9 / tf:.3f} of {src} {tf:.0f}), "
          f"{byts / ms / 1e6:.0f} GB/s ({byts / ms / 1e6 / hbm:.3f} of {src} {hbm:.0f}), status {ops.tc_gemm_status(DEV)}")


def gemm_f32(args) -> None:
    """The 32-bit FMA product against a measured loop of fused multiply-adds (no tensor cores)."""
    M, N, K = args.m, args.n, args.k
    a = torch.randn(M, K, device=DEV) * 0.1
    copies = max(1, min(8, int(300e6 // (N * K * 4)) + 1))
    ws = [torch.randn(N, K, device=DEV) * 0.1 for _ in range(copies)]
    out = torch.empty((M, N), device=DEV)
    i = [0]

    def run():
        i[0] += 1
        ops.gemm_f32(a, ws[i[0] % copies], out)
    ms = timed(run, args.iters)
    hbm, _, src = peaks()
    fma_peak = ops.fma_peak_tflops(DEV)
    flops, byts = 2.0 * M * N * K, (N * K + M * K + M * N) * 4.0
    print(f"gemm_f32 M={M} N={N} K={K}: {ms * 1e3:.1f} us, {flops / ms / 1e9:.2f} TFLOP/s "
          f"({flops / ms / 1e9 / fma_peak:.3f} of a measured FMA loop's {fma_peak:.1f}), "
          f"{byts / ms / 1e6:.0f} GB/s ({byts / ms / 1e6 / hbm:.3f} of {src} {hbm:.0f})")


def attention_f32(args) -> None:
    """The 32-bit attention (one warp per row, or per row and chunk of 64 keys) as a step context would call it."""
    nq, nkv, hd, ps = args.heads, args.kv_heads, args.head_dim, args.page_size
    R, ctx, q_len = args.requests, args.context, args.tokens
    pages_each = -(-ctx // ps)
    num_pages = R * pages_each + 1
    k = torch.randn(num_pages, nkv, ps, hd, device=DEV) * 0.5
    v = torch.randn(num_pages, nkv, ps, hd, device=DEV) * 0.5
    table = torch.randperm(num_pages - 1, device=DEV).to(torch.int32).view(R, pages_each).contiguous()
    n = R * q_len
    q = torch.randn(n, nq * hd, device=DEV) * 0.5
    out = torch.empty_like(q)
    treq = torch.arange(R, dtype=torch.int32, device=DEV).repeat_interleave(q_len)
    pos = (torch.arange(ctx - q_len, ctx, dtype=torch.int32, device=DEV)).repeat(R)
    rows, chunks = n * nq, ops.simt_chunks(ctx, 0)
    scratch = None
    if not args.walk and chunks > 1 and rows <= 4096 and rows * chunks <= 65536:
        scratch = torch.empty(rows * chunks * (hd + 2), device=DEV)
    if q_len > 1 and not args.walk:          # portions of prompts: the tiled kernel, as the attention part chooses
        starts = torch.arange(0, n, q_len, dtype=torch.int32, device=DEV)
        qlens = torch.full((R,), q_len, dtype=torch.int32, device=DEV)
        ctxs = torch.full((R,), ctx, dtype=torch.int32, device=DEV)
        ms = timed(lambda: ops.paged_attention_simt_tiled(q, out, k, v, starts, qlens, ctxs, table, q_len, nq, nkv, hd, ps, 0,
                                                          1.0 / math.sqrt(hd)), args.iters)
        how = "tiled"
    else:
        ms = timed(lambda: ops.paged_attention_simt(q, out, k, v, treq, pos, table, nq, nkv, hd, ps, 0, 1.0 / math.sqrt(hd),
                                                    scratch, chunks), args.iters)
        how = "split by chunks" if scratch is not None else "walk"
    hbm, _, src = peaks()
    kv_bytes = 2.0 * R * ctx * nkv * hd * 4
    keys_seen = R * sum(ctx - q_len + i + 1 for i in range(q_len))
    print(f"attention f32 requests={R} context={ctx} tokens={q_len} heads={nq}/{nkv} head_dim={hd} "
          f"{how}: {ms * 1e3:.1f} us, {kv_bytes / ms / 1e6:.0f} GB/s of keys "
          f"and values ({kv_bytes / ms / 1e6 / hbm:.3f} of {src} {hbm:.0f}), {4.0 * nq * hd * keys_seen / ms / 1e9:.2f} TFLOP/s")


def attention(args, decode: bool) -> None:
    nq, nkv, hd, ps = args.heads, args.kv_heads, args.head_dim, args.page_size
    R, ctx = args.requests, args.context
    q_len = 1 if decode else args.tokens
    pages_each = -(-ctx // ps)
    num_pages = R * pages_each + 1
    k = (torch.randn(num_pages, nkv, ps, hd, device=DEV) * 0.5).to(torch.bfloat16)
    v = (torch.randn(num_pages, nkv, ps, hd, device=DEV) * 0.5).to(torch.bfloat16)
    table = torch.randperm(num_pages - 1, device=DEV).to(torch.int32).view(R, pages_each).contiguous()
    n = R * q_len
    q = (torch.randn(n, nq * hd, device=DEV) * 0.5).to(torch.bfloat16)
    out = torch.empty_like(q)
    starts = torch.arange(0, n, q_len, dtype=torch.int32, device=DEV)
    qlens = torch.full((R,), q_len, dtype=torch.int32, device=DEV)
    ctxs = torch.full((R,), ctx, dtype=torch.int32, device=DEV)
    scale = 1.0 / math.sqrt(hd)
    if decode:
        split_keys, max_splits = ops.decode_split_plan(R * nkv, ctx, 32 if hd % 64 == 0 else 64)
        scratch = torch.empty(ops.attention_mma_scratch_floats(R, nq, hd, max_splits), device=DEV)

        def run():
            ops.attention_mma_decode(q, out, k, v, starts, qlens, ctxs, table, nq, nkv, hd, ps, 0, scale, split_keys,
                                     max_splits, scratch)
    else:
        split_above = 0 if args.no_share else ops.prefill_share_plan([q_len] * R, [ctx] * R, nq, nkv, hd, False)
        halves = torch.empty(ops.attention_prefill_halves_floats(R, q_len, nq, nkv, hd), device=DEV) if split_above else None

        def run():
            ops.attention_mma_prefill(q, out, k, v, starts, qlens, ctxs, table, q_len, nq, nkv, hd, ps, 0, scale, False,
                                      split_above=split_above, halves=halves)
    ms = timed(run, args.iters)
    hbm, tf, src = peaks()
    kv_bytes = 2.0 * R * ctx * nkv * hd * 2
    first = ctx - q_len
    keys_seen = R * sum(first + i + 1 for i in range(q_len)) if q_len < 4096 else R * q_len * (first + q_len / 2)
    flops = 4.0 * nq * hd * keys_seen
    what = "attention decode" if decode else "attention prefill"
    print(f"{what} requests={R} context={ctx} tokens={q_len} heads={nq}/{nkv} head_dim={hd} page={ps}: {ms * 1e3:.1f} us, "
          f"{kv_bytes / ms / 1e6:.0f} GB/s of keys and values ({kv_bytes / ms / 1e6 / hbm:.3f} of {src} {hbm:.0f}), "
          f"{flops / ms / 1e9:.1f} TFLOP/s ({flops / ms / 1e9 / tf:.3f} of {src} {tf:.0f}), status {ops.tc_gemm_status(DEV)}")


def sampling(args) -> None:
    """The sampling passes on rows of logits that lie in L2 (as the head's product leaves them), options on the device."""
    from ..sampling import SamplingParams
    from ..sampling.sampler import Sampler
    rows, V = args.rows, args.vocab
    sp = SamplingParams(temperature=args.temperature, top_k=args.top_k, top_p=args.top_p, min_p=args.min_p, seed=1)
    sampler = Sampler(DEV)
    logits = torch.randn(rows, V, device=DEV) * 3.0
    logits[:, 77] += 8.0                                        # a peaked row, as a model's is
    lists = ([sp] * rows, [3] * rows, [7] * rows, [set()] * rows)
    sampler.launch(logits, *lists)                              # sends the options once
    greedy = args.temperature == 0.0
    if greedy:
        ms = timed(lambda: sampler.launch(logits, *lists), args.iters)
    else:
        from ..sampling.sampler import pack_options
        filters = pack_options(*lists)[1]
        ms = timed(lambda: sampler.launch_packed(logits, filters), args.iters)
    passes = 1 if greedy else 2 + (1 if filters & 1 else 0) + (2 if filters & 2 else 0)
    print(f"sampling rows={rows} vocab={V} temperature={args.temperature} top_k={args.top_k} top_p={args.top_p} "
          f"min_p={args.min_p}: {ms * 1e3:.1f} us, {passes} passes over {rows * V * 4 / 1e6:.1f} MB of logits "
          f"({passes * rows * V * 4 / ms / 1e6:.0f} GB/s out of L2)")


def recurrence(args) -> None:
    """The decayed-state recurrence of linear attention (csrc/linear_attention.cu) over `requests` portions of `tokens`
    tokens each (1: a decode step), decay per key channel or per head."""
    if args.chunks or args.delta:
        return recurrence_chunks(args)
    R, T, H, D, V = args.requests, args.tokens, args.heads, args.dim, args.vdim
    n = R * T
    g = torch.Generator(device=DEV).manual_seed(1)
    q, k = (torch.randn(n, H * D, device=DEV, generator=g) for _ in range(2))
    v = torch.randn(n, H * V, device=DEV, generator=g)
    decay = None if args.per_head else torch.rand(n, H * D, device=DEV, generator=g) * 0.1 + 0.9
    head_decay = torch.full((H,), 0.97, device=DEV) if args.per_head else None
    state = torch.zeros(R, H, D, V, device=DEV)
    out = torch.empty(n, H * V, device=DEV)
    starts = torch.arange(R, dtype=torch.int32, device=DEV) * T
    lens = torch.full((R,), T, dtype=torch.int32, device=DEV)
    slots = torch.arange(R, dtype=torch.int32, device=DEV)
    seg_len, max_seg = (0, 1) if args.no_segments else ops.linattn_segment_plan(T, R if T > 1 else 0, H, V)
    seg_state = torch.empty(R * max_seg * H * D * V, device=DEV)
    seg_decay = torch.empty(R * max_seg * H * D, device=DEV)
    ms = timed(lambda: ops.linattn_scan(q, k, v, decay, head_decay, state, out, starts, lens, slots, H, D, V, seg_len, max_seg,
                                        seg_state, seg_decay), args.iters)
    hbm, _, src = peaks()
    moved = n * ((3 if decay is not None else 2) * H * D + 2 * H * V) * 4 + 2 * R * H * D * V * 4
    fma = 3.0 * n * H * D * V * (2 if max_seg > 1 else 1)
    print(f"recurrence requests={R} tokens={T} heads={H} dim={D} vdim={V} segments={max_seg}x{seg_len}: {ms * 1e3:.1f} us, "
          f"{moved / 1e6:.1f} MB that must move ({moved / ms / 1e6:.0f} GB/s, {moved / ms / 1e6 / hbm:.3f} of {src} copy bandwidth), "
          f"{fma / ms / 1e9:.2f} T 32-bit multiply-adds and multiplies a second")


def recurrence_chunks(args) -> None:
    """The same recurrence, or the gated delta rule (`--delta`), in chunks of 64 tokens on the tensor cores (csrc/linear_attention_chunks.cu,
    csrc/delta_rule_chunks.cu)."""
    R, T, H, D, V = args.requests, args.tokens, args.heads, args.dim, args.vdim
    n, g = R * T, torch.Generator(device=DEV).manual_seed(1)
    rand = lambda *shape: torch.randn(*shape, device=DEV, generator=g)
    host = np.full(R, T, dtype=np.int32)
    starts, lens, slots = torch.arange(R, dtype=torch.int32, device=DEV) * T, torch.full((R,), T, dtype=torch.int32, device=DEV), torch.arange(R, dtype=torch.int32, device=DEV)
    decay = torch.rand(n, H * D, device=DEV, generator=g) * 0.1 + 0.9
    state, out = torch.zeros(R, H, D, V, device=DEV), torch.empty(n, H * V, device=DEV)
    if args.delta:
        unit = lambda x: (x / x.norm(dim=-1, keepdim=True)).view(n, H * D).contiguous()
        q, k, v, beta = unit(rand(n, H, D)), unit(rand(n, H, D)), rand(n, H * V), torch.rand(n, H, device=DEV, generator=g)
        per = decay[:, ::D].contiguous() if args.per_head else decay - 1.0
        room, turns = ops.delta_chunks_plan(host, H)
        scratch = torch.empty(room, dtype=torch.uint8, device=DEV)
        ms = timed(lambda: ops.delta_chunks(q, k, v, beta, per, state, out, starts, lens, slots, host, H, H, not args.per_head, scratch), args.iters)
    else:
        fused, positions = rand(n, 2 * H * D + H * V).bfloat16(), torch.arange(n, dtype=torch.int32, device=DEV) % T
        head_decay = torch.full((H,), 0.97, device=DEV)
        room, turns = ops.linattn_chunks_plan(host, H, D, V)
        scratch = torch.empty(room, dtype=torch.uint8, device=DEV)
        ms = timed(lambda: ops.linattn_chunks(fused, 0, H * D, 2 * H * D, H, D, V, positions, None if args.per_head else decay, head_decay, state, out, starts, lens,
                                              slots, host, scratch, q_scale=D ** -0.5), args.iters)
    print(f"{'delta rule' if args.delta else 'recurrence'} in chunks requests={R} tokens={T} heads={H} dim={D} vdim={V}: {ms * 1e3:.1f} us, {room / 1e6:.0f} MB of scratch, "
          f"{turns} turns")


def experts(args) -> None:
    """Routed experts at a layer's shape: router, the pairs sorted by expert, the two grouped products, the weighted sum."""
    n, E, top, W, I = args.tokens, args.experts, args.top, args.width, args.ff
    bf, f32, i32 = torch.bfloat16, torch.float32, torch.int32
    x = (torch.randn(n, W, device=DEV)).to(bf)
    wr, wg = torch.randn(E, W, device=DEV) * 0.05, torch.randn(W, device=DEV) * 0.05
    copies = max(1, min(4, int(300e6 // (E * 3 * I * W * 2)) + 1))       # cycle the experts' weights so that they come from DRAM
    w_gu = [(torch.randn(E, 2 * I, W, device=DEV) * 0.02).to(bf) for _ in range(copies)]
    w_d = [(torch.randn(E, W, I, device=DEV) * 0.02).to(bf) for _ in range(copies)]
    pairs = n * top
    chosen, weights, gate = torch.empty(n, top, dtype=i32, device=DEV), torch.empty(n, top, device=DEV), torch.empty(n, device=DEV)
    count, offset = torch.empty(E, dtype=i32, device=DEV), torch.empty(E + 1, dtype=i32, device=DEV)
    order, place = torch.empty(pairs, dtype=i32, device=DEV), torch.empty(pairs, dtype=i32, device=DEV)
    act, y, out = torch.empty(pairs, I, dtype=bf, device=DEV), torch.empty(pairs, W, device=DEV), torch.empty(n, W, device=DEV)
    groups = args.groups
    ops.moe_route(x, wr, wg, chosen, weights, gate, groups, max(1, groups // 2))
    ops.moe_plan(chosen, count, offset, order, place)
    used = int((count > 0).sum())
    state = {"i": 0}

    def nxt():
        state["i"] = (state["i"] + 1) % copies
        return state["i"]
    hbm, tflops, src = peaks()
    rows = [("router", lambda: ops.moe_route(x, wr, wg, chosen, weights, gate, groups, max(1, groups // 2)), n * W * 2 + (E + 1) * W * 4, 2.0 * n * (E + 1) * W),
            ("pairs sorted by expert", lambda: ops.moe_plan(chosen, count, offset, order, place), pairs * 12, 0.0),
            ("gate|up with the clamped unit", lambda: ops.moe_grouped(x, w_gu[nxt()], act, offset, order, top, True, 7.0, 1.702),
             used * 2 * I * W * 2 + pairs * (W + I) * 2, 4.0 * pairs * I * W),
            ("down", lambda: ops.moe_grouped(act, w_d[nxt()], y, offset, order, top, False), used * I * W * 2 + pairs * (I * 2 + W * 4), 2.0 * pairs * I * W),
            ("weighted sum", lambda: ops.moe_combine(y, place, weights, None, None, out), pairs * W * 4 + n * W * 4, 0.0)]
    if ops.tc_grouped_ok(x, w_gu[0]) and I % 8 == 0:
        tiles = torch.empty(1 + 3 * ops.moe_row_tiles(pairs, E), dtype=i32, device=DEV)
        ops.moe_plan(chosen, count, offset, order, place, tiles)
        xs = torch.empty(pairs, W, dtype=bf, device=DEV)
        rows += [("rows into sorted order", lambda: ops.moe_gather(x, order, top, xs), pairs * W * 4, 0.0),
                 ("gate|up, clamped unit (tcgen05)", lambda: ops.gemm_bf16_tc_grouped(xs, w_gu[nxt()], act, tiles, True, 7.0, 1.702),
                  used * 2 * I * W * 2 + pairs * (W + I) * 2, 4.0 * pairs * I * W),
                 ("down (tcgen05)", lambda: ops.gemm_bf16_tc_grouped(act, w_d[nxt()], y, tiles, False),
                  used * I * W * 2 + pairs * (I * 2 + W * 4), 2.0 * pairs * I * W)]
    print(f"experts: {n} tokens, {E} experts ({used} used), top {top}, width {W}, ff {I}; peaks {src}: {hbm:.0f} GB/s, {tflops:.0f} TFLOP/s")
    for name, fn, moved, flops in rows:
        ms = timed(fn, args.iters)
        floor = max(moved / (hbm * 1e6), flops / (tflops * 1e9))
        print(f"  {name:32s} {ms * 1e3:9.1f} us   {moved / ms / 1e6:8.0f} GB/s   {flops / ms / 1e9:8.1f} TFLOP/s   {ms / max(floor, 1e-9):6.1f} x its floor")


def main(argv=None) -> int:
    ap = argparse.ArgumentParser(prog="python -m wllm_b200.kernels.cases", description=__doc__.split("\n\n")[0])
    sub = ap.add_subparsers(dest="case", required=True)
    g = sub.add_parser("gemm")
    g.add_argument("--m", type=int, default=2048)
    g.add_argument("--n", type=int, default=32768)
    g.add_argument("--k", type=int, default=2048)
    g.add_argument("--epilogue", default="bf16", choices=["bf16", "f32", "gelu_tanh", "silu"])
    g.add_argument("--split", action="store_true", help="cut K into parts as a step of few rows does (float32 slabs)")
    g.add_argument("--half-rows", type=int, default=0, help="half the W tile's rows (0: the plan's choice)")
    g32 = sub.add_parser("gemm-f32")
    g32.add_argument("--m", type=int, default=16)
    g32.add_argument("--n", type=int, default=49152)
    g32.add_argument("--k", type=int, default=3072)
    for name in ("attention-decode", "attention-prefill", "attention-f32"):
        a = sub.add_parser(name)
        a.add_argument("--requests", type=int, default=16)
        a.add_argument("--context", type=int, default=8192)
        a.add_argument("--tokens", type=int, default=2048, help="new tokens per request (prefill)")
        a.add_argument("--heads", type=int, default=8)
        a.add_argument("--kv-heads", type=int, default=1)
        a.add_argument("--head-dim", type=int, default=256)
        a.add_argument("--page-size", type=int, default=64)
        a.add_argument("--no-share", action="store_true", help="prefill: never share a heavy tile between two CTAs")
        a.add_argument("--walk", action="store_true", help="attention-f32: one warp per row even where chunks would be split or rows tiled")
    rc = sub.add_parser("recurrence")
    rc.add_argument("--requests", type=int, default=1)
    rc.add_argument("--tokens", type=int, default=2048)
    rc.add_argument("--heads", type=int, default=8)
    rc.add_argument("--dim", type=int, default=128)
    rc.add_argument("--vdim", type=int, default=256)
    rc.add_argument("--per-head", action="store_true", help="one decay per head (retention) instead of one per key channel")
    rc.add_argument("--chunks", action="store_true", help="in chunks of 64 tokens on the tensor cores, as bfloat16 models' long portions go")
    rc.add_argument("--delta", action="store_true", help="the gated delta rule in such chunks (heads of 128 by 128)")
    rc.add_argument("--no-segments", action="store_true", help="walk every portion in one go")
    ex = sub.add_parser("experts")
    ex.add_argument("--tokens", type=int, default=2048)
    ex.add_argument("--experts", type=int, default=32)
    ex.add_argument("--top", type=int, default=4)
    ex.add_argument("--groups", type=int, default=4)
    ex.add_argument("--width", type=int, default=2048)
    ex.add_argument("--ff", type=int, default=1024)
    sm = sub.add_parser("sampling")
    sm.add_argument("--rows", type=int, default=8)
    sm.add_argument("--vocab", type=int, default=256000)
    sm.add_argument("--temperature", type=float, default=0.8)
    sm.add_argument("--top-k", type=int, default=0)
    sm.add_argument("--top-p", type=float, default=1.0)
    sm.add_argument("--min-p", type=float, default=0.0)
    for p in sub.choices.values():
        p.add_argument("--iters", type=int, default=10)
    args = ap.parse_args(argv)
    if not torch.cuda.is_available():
        print("a CUDA device is needed", file=sys.stderr)
        return 1
    if args.case == "gemm":
        gemm(args)
    elif args.case == "gemm-f32":
        gemm_f32(args)
    elif args.case == "attention-f32":
        attention_f32(args)
    elif args.case == "sampling":
        sampling(args)
    elif args.case == "recurrence":
        recurrence(args)
    elif args.case == "experts":
        experts(args)
    else:
        attention(args, decode=args.case == "attention-decode")
    return 0


if __name__ == "__main__":
    sys.exit(main())

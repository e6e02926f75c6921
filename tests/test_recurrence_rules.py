"""Which steps the recurrences take in chunks of 64 tokens: mostly full ones, no portion beside many short requests, none whose scratch goes in many turns."""
from __future__ import annotations

from types import SimpleNamespace

import numpy as np
import pytest
import torch


def _ctx(lens):
    return SimpleNamespace(host={"req_q_len": np.array(lens, dtype=np.int32)}, memo={}, max_q_len=max(lens))


def _linear(heads, dim, vdim, rank):
    from wllm_b200.parts.linear_attention import LinearAttention
    mixer = LinearAttention.__new__(LinearAttention)
    mixer.heads, mixer.dim, mixer.vdim, mixer.rank, mixer.decay_kind = heads, dim, vdim, rank, "low_rank" if rank else "per_head"
    return mixer


# (sizes, lens, whether chunks were the faster way on the device, by more than a tenth)
@pytest.mark.parametrize("sizes,lens,chunks", [
    ((8, 128, 256, 64), [130], True), ((8, 128, 256, 64), [2048], True), ((8, 128, 256, 64), [130] * 16, True), ((8, 128, 256, 64), [512] * 16, True),
    ((8, 128, 256, 64), [1531] + [1] * 24, True), ((8, 128, 256, 64), [512] + [20] * 20, True), ((8, 128, 256, 64), [2048] + [20] * 40, True),
    ((8, 128, 256, 64), [130] + [20] * 20, False), ((8, 128, 256, 64), [130] + [20] * 40, False), ((8, 128, 256, 64), [130] + [20] * 90, False),
    ((8, 128, 256, 64), [512] + [20] * 90, False), ((8, 128, 256, 64), [2048] + [20] * 90, False), ((8, 128, 256, 64), [2048] + [20] * 200, False),
    ((8, 128, 256, 0), [2048], True), ((8, 128, 256, 0), [130] + [40] * 16, False), ((8, 128, 256, 0), [512] + [20] * 90, False),
    ((4, 64, 64, 64), [130] + [20] * 90, True), ((4, 64, 64, 64), [2048] + [20] * 200, True),
    ((16, 64, 128, 64), [130] + [20] * 90, False), ((16, 64, 128, 64), [2048] + [20] * 90, True), ((16, 64, 128, 64), [2048] + [20] * 200, False),
    ((32, 128, 128, 64), [2048], True), ((32, 128, 128, 64), [130] * 16, False), ((32, 128, 128, 64), [512] * 4, True), ((32, 128, 128, 64), [130] + [20] * 20, False), ((32, 128, 128, 64), [512] + [20] * 40, False)])
def test_linear_attention_goes_in_chunks_where_they_are_faster(sizes, lens, chunks):
    from wllm_b200.kernels import ops
    mixer, ctx = _linear(*sizes), _ctx(lens)
    assert mixer._chunk_room(ctx) == (ops.linattn_chunks_bytes(ctx.host["req_q_len"], *sizes[:3]) if chunks else 0)
    assert mixer._chunk_room(ctx) == mixer._chunk_room(_ctx(lens))


def test_steps_without_lengths_on_the_host_are_walked():
    assert _linear(8, 128, 256, 64)._chunk_room(SimpleNamespace(host=None, memo={}, max_q_len=2048)) == 0


def test_turns_are_those_that_the_scratch_leaves():
    from wllm_b200.kernels import ops
    plan = lambda lens: ops.linattn_chunks_plan(np.array(lens, dtype=np.int32), 8, 128, 256)
    assert plan([2048]) == (32 * 2560000, 1) and plan([1, 15]) == (0, 0)
    room, turns = plan([64 * 200])              # 512 MB at once
    assert turns == 4 and room == 50 * 2560000
    assert plan([2048] + [20] * 90) == (91 * 2560000, 32)


# (heads, lens, whether chunks were the faster way on the device)
@pytest.mark.parametrize("heads,lens,chunks", [
    (16, [2048], True), (16, [512], True), (16, [1021, 680, 340], True), (16, [1531] + [1] * 24, True), (16, [256], False), (16, [130] * 16, False),
    (16, [512] + [20] * 100, False), (16, [256] + [1] * 47, False), (2, [384], True), (2, [130] * 16, False), (4, [300] * 4, False), (4, [512] * 16, True),
    (8, [384], True), (8, [256], False), (8, [512] + [20] * 100, False), (32, [2048], True), (32, [512], True), (32, [1021, 680, 340], False),
    (32, [300] * 4, False), (32, [512] * 16, False), (64, [2048], True), (64, [1021, 680, 340], False), (64, [300] * 4, False)])
def test_the_delta_rule_goes_in_chunks_where_they_are_faster(heads, lens, chunks):
    from wllm_b200.kernels import ops
    from wllm_b200.parts.linear_attention import DeltaRule
    mixer, ctx = DeltaRule.__new__(DeltaRule), _ctx(lens)
    mixer.heads, mixer.dim, mixer.vdim, mixer.model_dtype = heads, 128, 128, torch.bfloat16
    assert mixer._chunk_room(ctx) == (ops.delta_chunks_bytes(ctx.host["req_q_len"], heads) if chunks else 0)

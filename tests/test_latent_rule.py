"""Which steps latent attention runs over keys and values of every head's own: where they are the faster way."""
from __future__ import annotations

from types import SimpleNamespace

import numpy as np
import pytest


def _mixer(heads, dim, rank, window=None):
    from wllm_b200.parts.latent_attention import LatentAttention
    mixer = LatentAttention.__new__(LatentAttention)
    mixer.heads, mixer.dim, mixer.rank, mixer.window, mixer.w_ukv = heads, dim, rank, window, object()
    return mixer


def _ctx(lens, cached=0):
    lens = np.array(lens, dtype=np.int32)
    return SimpleNamespace(host={"req_q_len": lens, "req_ctx_len": lens + np.int32(cached)}, memo={}, num_single=int((lens == 1).sum()), n_tokens=int(lens.sum()))


# (heads, dim, rank), lens, whether that was the faster way on the device
@pytest.mark.parametrize("sizes,lens,expands", [
    ((16, 128, 512), [64], True), ((16, 128, 512), [2048], True), ((16, 128, 512), [340, 680, 1021], True), ((16, 128, 512), [64] * 16, True),
    ((16, 128, 512), [130] * 8, True), ((16, 128, 512), [2048] + [20] * 16, True), ((16, 128, 512), [20] * 16, False), ((64, 128, 512), [33] * 8, False),
    ((64, 128, 512), [200] * 16, True), ((16, 128, 256), [1021], True), ((16, 128, 256), [130] * 8, False), ((16, 128, 256), [20] * 16, False),
    ((16, 128, 128), [1021], True), ((16, 128, 128), [130] * 8, False), ((16, 128, 96), [130] * 8, False), ((16, 128, 64), [128], False), ((16, 128, 64), [512], False),
    ((16, 128, 64), [130] * 8, False), ((16, 64, 512), [130] * 8, True), ((16, 256, 64), [256], False), ((16, 256, 64), [340, 680, 1021], False),
    ((16, 256, 64), [130] * 8, False), ((16, 256, 512), [2048], True), ((16, 256, 512), [130] * 16, False), ((4, 128, 96), [256], False), ((4, 128, 96), [2048], True)])
def test_prompts_make_keys_and_values_where_that_is_faster(sizes, lens, expands):
    mixer, ctx = _mixer(*sizes), _ctx(lens)
    assert mixer._expands(ctx) is expands and mixer._expands(ctx) is expands


def test_only_whole_prompts_do():
    mixer = _mixer(16, 128, 512)
    assert mixer._expands(_ctx([500])) and not mixer._expands(_ctx([500], cached=1)) and not mixer._expands(_ctx([500, 1])) and not mixer._expands(_ctx([63]))
    assert not mixer._expands(SimpleNamespace(host=None, memo={}, num_single=0, n_tokens=500))
    mixer.w_ukv = None
    assert not mixer._expands(_ctx([500]))


def test_keys_behind_a_window_are_no_gain():
    from wllm_b200.kernels import ops
    lens = np.array([4096], dtype=np.int32)
    worth = lambda window: ops.latent_expand_worth(lens, lens, 16, 128, 512, window)
    assert worth(64) < worth(0) / 4 and worth(4096) == worth(0) and ops.latent_expand_worth(lens, lens + np.int32(1), 16, 128, 512, 0) == 0


@pytest.mark.parametrize("rot", [0, 16])
def test_the_values_maps_are_held_once(rot):
    """Where every head's keys and values are made by one matrix, the maps of the values alone are its second half."""
    import torch

    from wllm_b200.config import resolve_architecture
    from wllm_b200.engine import ComposedModel
    layer = {"type": "latent_attention", "mlp": {"kind": "dense", "ff": 32}, "mixer": {"heads": 2, "dim": 64, "vdim": 64, "kv_rank": 24, "q_rank": 16, "scale": 0.1}}
    raw = {"architecture": "Gudarax", "vocab": 31, "width": 32, "max_positions": 64, "norm": {"eps": 1e-6}, "embedding": {"scale": 1.0}, "token_side": {"dim": 8},
           "layers": [layer]}
    arch = resolve_architecture("Gudarax")
    model = ComposedModel(arch.make_plan(arch.config_class.from_dict(raw, where="test")), torch.bfloat16)
    weights = {p.name: torch.randn(tuple(p.shape)).bfloat16() for p in model.param_specs()}
    mixer = model.blocks[0].mixer
    mixer.rot = rot                       # (with a turned part nothing is expanded)
    mixer.load(weights.__getitem__)
    up_k, up_v = weights[mixer.names["up_k"]], weights[mixer.names["up_v"]]
    assert torch.equal(mixer.w_uv.flatten(0, 1), up_v) and torch.equal(mixer.w_uk_t, up_k.view(2, 64, 24).transpose(1, 2))
    assert (mixer.w_ukv is None) == (rot > 0)
    if rot == 0:
        assert torch.equal(mixer.w_ukv, torch.cat([up_k, up_v])) and mixer.w_uv.untyped_storage().data_ptr() == mixer.w_ukv.untyped_storage().data_ptr()

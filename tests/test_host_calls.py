"""The native checks and launches (csrc/host_calls.cpp): what they refuse, with which errors, and that they refuse before anything is compiled or loaded."""
from __future__ import annotations

import pytest
import torch

BF, F32, I32 = torch.bfloat16, torch.float32, torch.int32


def _calls(dev: str) -> dict:
    """Calls that fit, small ones: name -> (function, arguments by name)."""
    from wllm_b200.kernels import ops
    z = lambda *shape, dtype=BF: torch.zeros(shape, dtype=dtype, device=dev)
    ints = lambda *x: torch.tensor(x, dtype=I32, device=dev)
    pages = dict(k_pages=z(2, 1, 64, 64), v_pages=z(2, 1, 64, 64))
    rows = dict(positions=ints(0, 1), slots=ints(0, 1), inv_freq=z(16, dtype=F32), **pages, nq=2, nkv=1, hd=64, rot_dim=32, page_size=64)
    batch = dict(q=z(2, 128), out=z(2, 128), **pages, req_q_start=ints(0), req_q_len=ints(2), req_ctx_len=ints(2), block_table=ints(0, 1).view(1, 2))
    return {
        "rmsnorm": (ops.rmsnorm, dict(resid=z(2, 64, dtype=F32), delta=z(2, 64), weight=z(64), eps=1e-6, offset=0.0, out=z(2, 64))),
        "sandwich_norm": (ops.sandwich_norm, dict(resid=z(2, 64, dtype=F32), a=(z(2, 64), 0), out=z(2, 64), post_weight=z(64), post_center=False, post_eps=1e-6,
                                                  weight=z(64), offset=0.0, center=False, eps=1e-6)),
        "rope_kv_write": (ops.rope_kv_write, dict(qkv=z(2, 256), q_out=z(2, 128), **rows)),
        "rope_row_norm_kv_write": (ops.rope_row_norm_kv_write, dict(qkv=z(2, 256), q_out=z(2, 128), **rows, q_gain=z(128), k_gain=z(64), eps=1e-6, q_count=128,
                                                                    k_count=64)),
        "attention_mma_decode": (ops.attention_mma_decode, dict(batch, req_q_len=ints(1), nq=2, nkv=1, hd=64, page_size=64, window=0, scale=0.1, split_keys=128, max_splits=1,
                                                                scratch=z(1 * 2 * 1 * 66, dtype=F32))),
        "attention_mma_prefill": (ops.attention_mma_prefill, dict(batch, max_q_len=2, nq=2, nkv=1, hd=64, page_size=64, window=0, scale=0.1, skip_single=False)),
        "gemm_bf16_tc": (ops.gemm_bf16_tc, dict(a=z(2, 64), w=z(64, 64), out=z(2, 64, dtype=F32), epilogue="f32", half_rows=ops.tile_plan(2, 64, 64)[0])),
    }


NAMES = ["rmsnorm", "sandwich_norm", "rope_kv_write", "rope_row_norm_kv_write", "attention_mma_decode", "attention_mma_prefill", "gemm_bf16_tc"]


@pytest.mark.parametrize("name", NAMES)
def test_tensors_on_the_host_are_refused_before_anything_is_compiled(name, monkeypatch):
    from wllm_b200.kernels import ops

    def compiles(*args):
        raise AssertionError(f"compiled or loaded {args}")
    monkeypatch.setattr(ops, "load_family", compiles)
    status = dict(ops._tc_status)
    fn, args = _calls("cpu")[name]
    with pytest.raises(ops.KernelError, match="CUDA device only; got a tensor on cpu"):
        fn(**args)
    assert ops._tc_status == status


def test_products_that_the_kernel_takes_are_told_without_it(monkeypatch):
    from wllm_b200.kernels import ops

    def compiles(*args):
        raise AssertionError(f"compiled or loaded {args}")
    monkeypatch.setattr(ops, "load_family", compiles)
    a, w = torch.zeros(4, 64, dtype=BF), torch.zeros(8, 64, dtype=BF)
    assert ops.tc_gemm_ok(a, w) and not ops.tc_gemm_ok(a.float(), w) and not ops.tc_gemm_ok(a[:, :60], w[:, :60]) and not ops.tc_gemm_ok(a[0], w)
    assert not ops.tc_gemm_ok(torch.zeros(4, 70, dtype=BF)[:, :64], w) and not ops.tc_gemm_ok(torch.zeros(4 * 64 + 8, dtype=BF)[1:257].view(4, 64), w)


def _strided(t):
    """The same tensor with a gap behind every element of its last axis."""
    return torch.zeros(*t.shape[:-1], 2 * t.shape[-1], dtype=t.dtype, device=t.device)[..., ::2]


# name: {argument: (what takes its place, error)}; the kernels' own refusals (sizes that none of them is built for) are not among them
WRONG = {
    "rmsnorm": {"resid": (lambda t: t.to(BF), AssertionError), "delta": (lambda t: t[:1], AssertionError), "weight": (lambda t: t[:32], AssertionError),
                "out": (lambda t: t[:, :32], AssertionError), "rows": (lambda _: torch.zeros(2, dtype=torch.int64, device="cuda"), "KernelError")},
    "sandwich_norm": {"resid": (_strided, AssertionError), "a": (lambda a: (a[0][:1], 0), AssertionError), "out": (lambda t: t[:1], AssertionError),
                      "post_weight": (lambda t: t.float(), AssertionError), "weight": (lambda t: t[:32], AssertionError),
                      "bias": (lambda _: torch.zeros(64, dtype=BF, device="cuda"), AssertionError), "b": (lambda _: (torch.zeros(3, 2, 64, device="cuda"), 2), AssertionError)},
    "rope_kv_write": {"qkv": (lambda t: t[:, :248], AssertionError), "q_out": (lambda t: t[:1], AssertionError), "inv_freq": (lambda t: t.to(BF), AssertionError),
                      "k_pages": (lambda t: t.float(), AssertionError), "v_pages": (_strided, AssertionError), "positions": (lambda t: t.long(), "KernelError"),
                      "slots": (lambda t: t.long(), "KernelError"), "in_splits": (lambda _: 2, AssertionError), "pairing": (lambda _: "odd", "KernelError")},
    "rope_row_norm_kv_write": {"qkv": (lambda t: t[:, :248], AssertionError), "q_gain": (lambda t: t[:64], AssertionError), "k_gain": (lambda t: None, AssertionError),
                               "bias": (lambda _: torch.zeros(8, device="cuda"), AssertionError), "mix": (lambda _: "first", AssertionError)},
    "attention_mma_decode": {"q": (_strided, AssertionError), "out": (lambda t: t.float(), AssertionError), "k_pages": (_strided, AssertionError),
                             "scratch": (lambda t: t[:131], AssertionError), "req_q_len": (lambda t: t.long(), "KernelError"),
                             "sinks": (lambda _: torch.zeros(3, device="cuda"), AssertionError), "slopes": (lambda _: torch.zeros(2, dtype=BF, device="cuda"), AssertionError)},
    "attention_mma_prefill": {"q": (lambda t: t.float(), AssertionError), "v_pages": (_strided, AssertionError), "block_table": (lambda t: t.long(), "KernelError"),
                              "split_above": (lambda _: 1, AssertionError), "sinks": (lambda _: torch.zeros(2, dtype=BF, device="cuda"), AssertionError)},
    "gemm_bf16_tc": {"a": (lambda t: t.float(), "KernelError"), "w": (lambda t: t[:, :56], AssertionError), "out": (lambda t: t.to(BF), AssertionError),
                     "k_splits": (lambda _: 2, AssertionError)},
}


@pytest.mark.gpu
@pytest.mark.parametrize("name", NAMES)
def test_operands_that_do_not_fit_are_refused(name):
    from wllm_b200.kernels import ops
    fn, args = _calls("cuda")[name]
    before = ops.launches
    fn(**args)
    fits = ops.launches
    assert fits == before + 1
    for which, (change, error) in WRONG[name].items():
        with pytest.raises(ops.KernelError if error == "KernelError" else error):
            fn(**{**args, which: change(args.get(which))})
    assert ops.launches == fits
    torch.cuda.synchronize()


@pytest.mark.gpu
def test_a_refused_product_names_its_operands():
    from wllm_b200.kernels import ops
    fn, args = _calls("cuda")["gemm_bf16_tc"]
    with pytest.raises(ops.KernelError, match=r"a\[2, 60\] stride \[64, 1\] w\[64, 60\] stride \[64, 1\]"):
        fn(**{**args, "a": args["a"][:, :60], "w": args["w"][:, :60]})

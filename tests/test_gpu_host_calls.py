"""The operators' native call path (csrc/host_calls.cpp) against the checks and ctypes calls behind it."""
import ctypes
import importlib

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda:0")
K, H, E, T = 1024, 512, 8, 3


def calls(rt, qz):
    """name -> (C entry, call(**kw)) of every operator on that path, with well-formed arguments."""
    g = torch.Generator(device=DEV).manual_seed(1)

    def act(*shape):
        return torch.randn(*shape, generator=g, device=DEV).to(torch.bfloat16)

    p4, p8 = qz.quantize_mxfp4((torch.randn(640, K, generator=g, device=DEV) * 0.02).to(torch.bfloat16)), {}
    for kind in ("e8m0", "f32"):
        p8[kind] = qz.quantize_fp8_block128(torch.randn(640, K, generator=g, device=DEV) * 0.02, kind)
    shared = {}
    for name, n, k in (("w1", H, K), ("w3", H, K), ("w2", K, H)):
        shared[name], shared[name + "s"] = qz.quantize_fp8_block128(torch.randn(n, k, generator=g, device=DEV) * 0.02)
    bank = qz.make_expert_bank(E, K, H, DEV, seed=2)
    six = [{"packed": bank[n + "p"][:6], "scale": bank[n + "s"][:6]} for n in ("w1", "w3", "w2")]
    x, xs, logits, r = act(K), act(T, K), torch.randn(T, E, generator=g, device=DEV), torch.rand(6, generator=g, device=DEV)
    ids = torch.arange(2, 8, dtype=torch.int32, device=DEV)
    picks, w = torch.arange(2 * T, dtype=torch.int32, device=DEV).view(T, 2), torch.rand(T, 2, generator=g, device=DEV)
    return {
        "mxfp4_gemv": ("mxfp4_gemv_m1", lambda **kw: rt.mxfp4_gemv(*p4, x, **kw)),
        "fp8_gemv": ("fp8_e4m3_gemv_m1", lambda **kw: rt.fp8_e4m3_gemv(*p8["e8m0"], x, **kw)),
        "fp8_gemv_f32scale": ("fp8_e4m3_gemv_m1_f32scale", lambda **kw: rt.fp8_e4m3_gemv_f32scale(*p8["f32"], x, **kw)),
        "fp8_gemv_batched": ("fp8_e4m3_gemv_batched", lambda **kw: rt.fp8_e4m3_gemv_batched(*p8["e8m0"], xs, **kw)),
        "fp8_shared_swiglu": ("fp8_e4m3_shared_swiglu_m1", lambda **kw: rt.fp8_shared_swiglu(shared, x, **kw)),
        "grouped_gemv": ("mxfp4_grouped_gemv_topk", lambda **kw: rt.mxfp4_grouped_gemv(*six, None, x, r, **kw)),
        "grouped_gemv_ids": ("mxfp4_grouped_gemv_topk_ids_stages", lambda **kw: rt.mxfp4_grouped_gemv_ids(bank, ids, x, r, **kw)),
        "route_topk": ("mxfp4_moe_route_topk", lambda **kw: rt.moe_route_topk(logits, k=2, **kw)),
        "decode_layer": ("mxfp4_moe_decode_layer", lambda **kw: rt.moe_decode_layer(bank, logits[0], x, k=2, **kw)),
        "moe_forward": ("mxfp4_moe_forward", lambda **kw: rt.moe_forward(bank, xs, picks, w, **kw)),
        "moe_forward_path": ("mxfp4_moe_forward_path", lambda **kw: rt.moe_forward(bank, xs, picks, w, path="fp16", **kw)),
    }


@pytest.fixture(scope="module")
def capi(rt):
    return importlib.import_module("dsv4_b200.runtime._capi")


@pytest.fixture(scope="module")
def ops(rt, qz, capi):
    for key in capi.SIGNATURES:
        capi.load(key)
    capi.host()
    return calls(rt, qz)


OPS = ["mxfp4_gemv", "fp8_gemv", "fp8_gemv_f32scale", "fp8_gemv_batched", "fp8_shared_swiglu", "grouped_gemv", "grouped_gemv_ids",
       "route_topk", "decode_layer", "moe_forward", "moe_forward_path"]


@pytest.mark.parametrize("name", OPS)
def test_interpreter_lock_is_released_around_the_call(ops, capi, name):
    """The C entry replaced by one that answers 1 while its thread holds the lock: a return code the operator raises for."""
    entry, call = ops[name]
    try:
        capi.host().bind(entry, ctypes.cast(ctypes.pythonapi.PyGILState_Check, ctypes.c_void_p).value)
        call()
    finally:
        for lib in capi._loaded.values():
            capi._bind(lib)


def test_failed_allocation_raises_what_torch_raises(rt, ops):
    logits = torch.zeros(1, 8, device=DEV)
    with pytest.raises(torch.OutOfMemoryError):
        rt.moe_route_topk(logits, k=1 << 42)        # 16 TB of ids
    ids, _ = rt.moe_route_topk(logits, k=2)
    assert ids.tolist() == [[0, 1]]


@pytest.mark.parametrize("name", OPS)
def test_same_bits_through_ctypes(ops, capi, monkeypatch, name):
    def tensors(result):
        return list(result) if isinstance(result, tuple) else [result]

    native = tensors(ops[name][1]())
    with monkeypatch.context() as m:
        m.setattr(capi, "_host", capi._Declines())
        through_ctypes = tensors(ops[name][1]())
    assert [(t.dtype, t.shape, t.device) for t in native] == [(t.dtype, t.shape, t.device) for t in through_ctypes]
    assert all(torch.equal(a.view(torch.uint8), b.view(torch.uint8)) for a, b in zip(native, through_ctypes))

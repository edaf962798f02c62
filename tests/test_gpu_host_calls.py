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


@pytest.mark.parametrize("kind", ["mxfp4", "fp8", "fp8_batched"])
def test_calls_out_of_the_ordinary(rt, qz, capi, kind):
    """Strides, an explicit stream and given outputs give the ordinary call's bits, whichever way they take; what does not fit
    raises."""
    g = torch.Generator(device=DEV).manual_seed(9)
    w = torch.randn(256, K, generator=g, device=DEV) * 0.02
    p, s = qz.quantize_mxfp4(w.to(torch.bfloat16)) if kind == "mxfp4" else qz.quantize_fp8_block128(w)
    op = {"mxfp4": rt.mxfp4_gemv, "fp8": rt.fp8_e4m3_gemv, "fp8_batched": rt.fp8_e4m3_gemv_batched}[kind]
    x = torch.randn(K, generator=g, device=DEV).to(torch.bfloat16)
    want = op(p, s, x).view(torch.int16)
    apart = torch.zeros(256, p.shape[1] + 48, dtype=p.dtype, device=DEV)[:, : p.shape[1]].copy_(p)      # rows with gaps
    column = torch.zeros(K, 2, dtype=x.dtype, device=DEV)[:, 0].copy_(x)                                # every second element
    turned = torch.zeros(p.shape[1], 256, dtype=p.dtype, device=DEV).t().copy_(p)                       # rows not dense
    odd = torch.zeros(K + 1, dtype=x.dtype, device=DEV)[1:].copy_(x)                                    # not 16-byte aligned
    side = torch.cuda.Stream(device=DEV)
    side.wait_stream(torch.cuda.current_stream(DEV))
    out = torch.empty(256, dtype=torch.bfloat16, device=DEV)
    results = [op(apart, s, x), op(p, s, column), op(turned, s, x), op(p, s, x, stream=side), op(p, s, x, out=out)]
    torch.cuda.synchronize()
    assert results[-1].data_ptr() == out.data_ptr()
    assert all(torch.equal(r.view(torch.int16), want) for r in results)
    if kind == "fp8_batched":
        with pytest.raises(RuntimeError):
            op(p, s, odd)
    else:
        err = (op(p, s, odd).float() - want.view(torch.bfloat16).float()).abs().max()      # the byte-wise kernel: FP32 sums, where the other's are fp16 inside a block; bf16 rounding of both is 2^-8
        assert err <= 2 ** -7 * want.view(torch.bfloat16).float().abs().max()
    for bad in (dict(out=out.float()), dict(out=out[:128]), dict(out=out.cpu())):
        with pytest.raises(RuntimeError):
            op(p, s, x, **bad)
    for args in ((p, s[:1], x), (p, s, x[:-128]), (p.int(), s, x), (p, s, x.float()), (p.cpu(), s, x)):
        with pytest.raises(RuntimeError):
            op(*args)


def test_workspace_that_is_too_small_is_refused(rt, qz, ops):
    call = ops["fp8_shared_swiglu"][1]
    good = call(workspace=torch.empty(2 * H, dtype=torch.uint8, device=DEV))
    assert torch.equal(good.view(torch.int16), call().view(torch.int16))
    for ws in (torch.empty(2 * H - 1, dtype=torch.uint8, device=DEV), torch.empty(2 * H, dtype=torch.uint8)):
        with pytest.raises(RuntimeError):
            call(workspace=ws)

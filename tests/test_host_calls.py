"""Tensors of several GPUs: the native call path hands them to the checks in Python, and those refuse them (fake tensors: no GPU
needed, nothing is launched)."""
import importlib

import pytest
import torch
from torch._subclasses.fake_tensor import FakeTensorMode

K, H, E, T = 256, 256, 8, 3


def cases(rt):
    """name -> (native arguments in order, index of the argument or of (argument, key) to move, operator call)."""
    def u8(*shape):
        return lambda dev: torch.empty(*shape, dtype=torch.uint8, device=dev)

    def of(dtype, *shape):
        return lambda dev: torch.empty(*shape, dtype=dtype, device=dev)

    bf, f32, i32 = torch.bfloat16, torch.float32, torch.int32
    bank = {"w1p": u8(E, H, K // 2), "w3p": u8(E, H, K // 2), "w2p": u8(E, K, H // 2), "w1s": u8(E, H, K // 32), "w3s": u8(E, H, K // 32),
            "w2s": u8(E, K, H // 32)}
    shared = {"w1": u8(H, K), "w3": u8(H, K), "w2": u8(K, H), "w1s": u8(2, 2), "w3s": u8(2, 2), "w2s": u8(2, 2)}
    stack = [{"packed": bank[n + "p"], "scale": bank[n + "s"]} for n in ("w1", "w3", "w2")]
    x, out = of(bf, K), of(bf, K)
    return {
        "mxfp4_gemv": ([u8(64, K // 2), u8(64, K // 32), x, of(bf, 64), None], lambda a: rt.mxfp4_gemv(*a)),
        "fp8_gemv": ([u8(128, K), u8(1, 2), x, of(bf, 128), None], lambda a: rt.fp8_e4m3_gemv(*a)),
        "fp8_gemv_f32scale": ([u8(128, K), of(f32, 1, 2), x, of(bf, 128), None], lambda a: rt.fp8_e4m3_gemv_f32scale(*a)),
        "fp8_gemv_batched": ([u8(128, K), u8(1, 2), of(bf, T, K), 1, None, None], lambda a: rt.fp8_e4m3_gemv_batched(*a)),
        "fp8_shared_swiglu": ([shared, x, 10.0, 0.0, out, u8(2 * H), None], lambda a: rt.fp8_shared_swiglu(*a)),
        "grouped_gemv": ([*stack, x, of(f32, E), out, u8(1 << 16)], lambda a: rt.mxfp4_grouped_gemv(*a[:3], None, *a[3:])),
        "grouped_gemv_ids": ([bank, of(i32, 6), x, of(f32, 6), out, u8(1 << 16), 3], lambda a: rt.mxfp4_grouped_gemv_ids(*a)),
        "route_topk": ([of(f32, T, E), 2, "softmax", 1e-20, 1.0, of(i32, T, 2), of(f32, T, 2)], lambda a: rt.moe_route_topk(*a)),
        "decode_layer": ([bank, of(f32, E), x, 2, "softmax", 1e-20, 1.0, out, u8(1 << 16)], lambda a: rt.moe_decode_layer(*a)),
        "moe_forward": ([bank, of(bf, T, K), of(i32, T, 2), of(f32, T, 2), of(bf, T, K), u8(1 << 20), -1],
                        lambda a: rt.moe_forward(*a[:6])),
    }


NAMES = ["mxfp4_gemv", "fp8_gemv", "fp8_gemv_f32scale", "fp8_gemv_batched", "fp8_shared_swiglu", "grouped_gemv", "grouped_gemv_ids",
         "route_topk", "decode_layer", "moe_forward"]


@pytest.mark.parametrize("name", NAMES)
def test_tensors_of_two_devices(rt, name):
    capi = importlib.import_module("dsv4_b200.runtime._capi")
    for key in capi.SIGNATURES:
        capi.load(key)
    native = getattr(capi.host(), name)
    makers, operator = cases(rt)[name]
    places = []
    for i, m in enumerate(makers):
        places += [(i, k) for k in m] if isinstance(m, dict) else [(i, None)] if callable(m) else []
    for moved in places:
        def build(i, m):
            if isinstance(m, dict):
                return {k: v("cuda:1" if (i, k) == moved else "cuda:0") for k, v in m.items()}
            return m("cuda:1" if (i, None) == moved else "cuda:0") if callable(m) else m

        with FakeTensorMode():
            args = [build(i, m) for i, m in enumerate(makers)]
        assert native(*args) is None, moved
        with pytest.raises((RuntimeError, ValueError), match="CUDA device"):
            operator(args)


def test_integers_beyond_64_bits_are_declined(rt):
    capi = importlib.import_module("dsv4_b200.runtime._capi")
    for key in capi.SIGNATURES:
        capi.load(key)
    makers, _ = cases(rt)["fp8_gemv_batched"]
    with FakeTensorMode():
        args = [m("cuda:0") if callable(m) else m for m in makers]
    args[3] = 1 << 70
    assert capi.host().fp8_gemv_batched(*args) is None
    makers, _ = cases(rt)["route_topk"]
    with FakeTensorMode():
        args = [m("cuda:0") if callable(m) else m for m in makers]
    args[1] = 1 << 70
    assert capi.host().route_topk(*args) is None


@pytest.mark.parametrize("content", [None, b"not a library"])
def test_operators_do_without_the_module(rt, pkg, monkeypatch, tmp_path, content):
    """A lib/ without the module, or with one that does not load: one warning, then the checks in Python and ctypes."""
    capi = importlib.import_module("dsv4_b200.runtime._capi")
    if content is not None:
        (tmp_path / pkg.host_file()).write_bytes(content)
    monkeypatch.setattr(capi, "LIB_DIR", str(tmp_path))
    monkeypatch.setattr(capi, "_host", None)
    with pytest.warns(RuntimeWarning, match="ctypes"):
        with pytest.raises(RuntimeError, match="CUDA device"):
            rt.mxfp4_gemv(torch.zeros(8, 32, dtype=torch.uint8), torch.zeros(8, 2, dtype=torch.uint8), torch.zeros(64, dtype=torch.bfloat16))
    assert capi.host().moe_forward(None) is None
    capi.load("mxfp4")


def test_module_is_named_for_its_torch(pkg):
    assert torch.__version__ in pkg.host_file()


def test_device_that_is_not_current_is_made_so(rt, monkeypatch):
    """The call then goes through Python, which enters the tensors' device; on the current one it enters nothing."""
    capi = importlib.import_module("dsv4_b200.runtime._capi")
    entered = []
    monkeypatch.setattr(torch.cuda, "current_device", lambda: 0)
    monkeypatch.setattr(torch.cuda, "device", lambda d: entered.append(d))
    with FakeTensorMode():
        here, other = torch.empty(1, device="cuda:0"), torch.empty(1, device="cuda:1")
    with capi.on_device(here):
        assert not entered
    capi.on_device(other)
    assert entered == [torch.device("cuda:1")]
    assert capi.elsewhere(here, a=None, b=here, c=torch.zeros(1), d=other) == "d"

"""Calls from two threads whose shapes need different, and ever larger, amounts of shared memory: what a kernel may use is an
attribute of the kernel on its device, so setting it for one call must not leave the other, or a later one, with too little.
The library is loaded from fresh copies, each with its own record of what has been set."""
import ctypes
import importlib
import shutil
import threading

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda:0")


def race(pkg, tmp_path, key, copies, pairs):
    """pairs: (call, call), a call being (lib, stream) -> return code; both of a pair are made at the same time."""
    capi = importlib.import_module("dsv4_b200.runtime._capi")
    streams = [torch.cuda.Stream(device=DEV) for _ in range(2)]
    handles = [ctypes.c_void_p(s.cuda_stream) for s in streams]
    for i in range(copies):
        path = tmp_path / f"{key}_{i}.so"
        shutil.copy(pkg.lib_path(key), path)
        lib = ctypes.CDLL(str(path))
        for name, (restype, argtypes) in capi.SIGNATURES[key].items():
            if hasattr(lib, name):
                getattr(lib, name).restype, getattr(lib, name).argtypes = restype, argtypes
        codes = [[None] * len(pairs) for _ in range(2)]
        gate = threading.Barrier(2)

        def run(side):
            torch.cuda.set_device(DEV)
            for n, pair in enumerate(pairs):
                gate.wait()
                codes[side][n] = pair[side](lib, handles[side])
                if n % 16 == 15:
                    streams[side].synchronize()

        threads = [threading.Thread(target=run, args=(side,)) for side in range(2)]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
        again = [call(lib, handles[side]) for pair in pairs[-2:] for side, call in enumerate(pair)]
        torch.cuda.synchronize()
        assert not any(codes[0]) and not any(codes[1]) and not any(again), (i, codes, again)


def byte_bank(E, K, H, O):
    shapes = {"w1p": (E, H, K // 2), "w3p": (E, H, K // 2), "w2p": (E, O, H // 2), "w1s": (E, H, K // 32), "w3s": (E, H, K // 32),
              "w2s": (E, O, H // 32)}
    return [torch.full(shapes[n], 0x21 if n.endswith("p") else 118, dtype=torch.uint8, device=DEV)
            for n in ("w1p", "w3p", "w2p", "w1s", "w3s", "w2s")]


def test_grouped_experts(pkg, tmp_path):
    def call(K, E=2, H=64, O=64):
        t = [torch.ones(K, dtype=torch.bfloat16, device=DEV), *byte_bank(E, K, H, O),
             torch.arange(E, dtype=torch.int32, device=DEV), torch.ones(E, device=DEV)]
        out = torch.empty(O, dtype=torch.bfloat16, device=DEV)
        ws = torch.empty(E * H * 8 + 64, dtype=torch.uint8, device=DEV)
        return lambda lib, stream: lib.mxfp4_grouped_gemv_topk_ids(*(v.data_ptr() for v in t), K, H, O, E, out.data_ptr(), ws.data_ptr(), stream)

    race(pkg, tmp_path, "grouped", 8, [(call(K), call(K + 32)) for K in range(32, 384, 64)])


def test_batched_layer(pkg, rt, tmp_path):
    T, K, H, O, E_most = 4, 256, 256, 128, 1024
    bank = byte_bank(E_most, K, H, O)
    x, w = torch.ones(T, K, dtype=torch.bfloat16, device=DEV), torch.ones(T, 1, device=DEV)
    ids = torch.arange(T, dtype=torch.int32, device=DEV).view(T, 1)

    def call(E, side):
        out, ws = outs[side]
        return lambda lib, stream: lib.mxfp4_moe_forward_path(1, *(v.data_ptr() for v in (x, *bank, ids, w)), T, E, K, H, O, 1,
                                                              out.data_ptr(), ws.data_ptr(), stream)

    outs = [(torch.empty(T, O, dtype=torch.bfloat16, device=DEV),
             torch.empty(rt.forward_workspace_bytes(T, 1, K, H, O, E_most), dtype=torch.uint8, device=DEV)) for _ in range(2)]
    race(pkg, tmp_path, "moe", 2, [(call(E, 0), call(E + 4, 1)) for E in range(4, E_most, 8)])

import os
import sys

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
if ROOT not in sys.path:
    sys.path.insert(0, ROOT)

import __graft_entry__ as entry  # noqa: E402


def pytest_configure(config):
    config.addinivalue_line("markers", "gpu: needs a CUDA device (run on the B200 box)")


@pytest.fixture(scope="session")
def pkg():
    """The package, with its libraries built (nvcc cross-compiles without a GPU)."""
    p = entry.load_package()
    if not all(os.path.exists(f) for f in [*(p.lib_path(k) for k in p.LIB_FILES), os.path.join(p.LIB_DIR, p.host_file())]):
        p.build()
    return p


@pytest.fixture(scope="session")
def rt(pkg):
    import importlib
    return importlib.import_module(entry.PKG_ALIAS + ".runtime")


@pytest.fixture(scope="session")
def qz(pkg):
    import importlib
    return importlib.import_module(entry.PKG_ALIAS + ".runtime.quantize")


@pytest.fixture(scope="session")
def golden():
    return np.load(os.path.join(ROOT, "tests", "golden", "reference_vectors.npz"))


@pytest.fixture(scope="session")
def odd_bank():
    """A bank's tensors at addresses that are 16 modulo 32: the TMA cannot lay such weights down padded, so the batched layer's path "fp16"
    dequantises them."""
    import torch

    def at_odd_16_bytes(t):
        buf = torch.empty(t.numel() + 48, dtype=t.dtype, device=t.device)
        shift = (16 - buf.data_ptr() % 32) % 32
        view = buf[shift:shift + t.numel()].view(t.shape)
        assert view.data_ptr() % 32 == 16
        return view.copy_(t)
    return lambda bank: {n: at_odd_16_bytes(t) for n, t in bank.items()}

import ctypes
import os
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PKG = os.path.join(ROOT, "kernel-independent-fast-multipole-method_b200")
for p in (PKG, os.path.join(ROOT, "oracle")):
    if p not in sys.path:
        sys.path.insert(0, p)


def pytest_configure(config):
    config.addinivalue_line("markers", "gpu: needs a CUDA device (B200); run with -m gpu")


def has_gpu() -> bool:
    try:
        import torch
        return torch.cuda.is_available()
    except Exception:
        return False


@pytest.fixture(scope="session")
def gpu():
    if not has_gpu():
        pytest.skip("no CUDA device")
    return True


@pytest.fixture(scope="session")
def harness(tmp_path_factory):
    """tests/device_harness.cu, compiled beside the built library."""
    out = str(tmp_path_factory.mktemp("harness") / "libharness.so")
    lib = os.path.join(PKG, "lib")
    nvcc = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")
    subprocess.run([nvcc, "-std=c++17", "-O2", "-gencode", "arch=compute_100a,code=sm_100a", "-shared", "-Xcompiler",
                    "-fPIC", "-cudart", "shared", "-I", os.path.join(PKG, "csrc"), "-o", out,
                    os.path.join(ROOT, "tests", "device_harness.cu"), "-L", lib, "-lkifmm_b200", "-Xlinker",
                    "-rpath," + lib], check=True)
    return ctypes.CDLL(out)

import os
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
if ROOT not in sys.path:
    sys.path.insert(0, ROOT)


def pytest_configure(config):
    config.addinivalue_line("markers", "gpu: needs a CUDA GPU (GB300, sm_103a)")
    config.addinivalue_line("markers", "slow: long-running CPU test")


@pytest.fixture(scope="session")
def orc():
    from oracle import oracle as o
    o.lib()
    return o


@pytest.fixture(scope="session")
def kernels(tmp_path_factory):
    """Kernels of the library that no entry point runs alone
    (native/kernels_harness.cu), built against it."""
    import ctypes
    import subprocess

    from bem_gmsh_gb300 import _build
    so = str(tmp_path_factory.mktemp("kernels") / "kernels_harness.so")
    subprocess.check_call([_build._nvcc(), *_build.ARCH, "-O2", "-std=c++17", "-shared", "-Xcompiler", "-fPIC",
                           "-cudart", "static", os.path.join(ROOT, "tests", "native", "kernels_harness.cu"), "-o", so,
                           _build.LIB, "-Xlinker", "-rpath=" + _build.BUILD])
    return ctypes.CDLL(so)

import os
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
for p in (os.path.join(ROOT, "cp-paw_b200"), os.path.join(ROOT, "oracle"), ROOT):
    if p not in sys.path:
        sys.path.insert(0, p)


def pytest_configure(config):
    config.addinivalue_line("markers", "gpu: needs a CUDA device (B200)")


@pytest.fixture(scope="session")
def oracle():
    import binding

    binding.build()
    return binding


@pytest.fixture(scope="session")
def engine_lib():
    import build as b

    b.build()
    import cuwaves

    return cuwaves


class FakeEngine:
    """The engine's host side on the device-less runtime of fake_cuda.cpp."""

    def __init__(self, path):
        import ctypes

        from cuwaves import capi

        self.lib = ctypes.CDLL(path, mode=ctypes.RTLD_LOCAL)
        for n in ("fake_in_use", "fake_peak", "fake_mallocs", "fake_waits"):
            getattr(self.lib, n).restype = ctypes.c_longlong
        self.lib.fake_fail_malloc.argtypes = [ctypes.c_longlong]
        self.lib.fake_fail_malloc.restype = None
        self.lib.fake_launches.argtypes = [ctypes.c_char_p, ctypes.c_int]
        self.fns = capi.bind(self.lib, "cuwaves_")

    def open(self, inp, precision=0):
        from cuwaves import capi

        return capi.Waves(self.fns, inp, precision)

    def launches(self):
        """Names of the kernels launched since the last call."""
        import ctypes

        buf = ctypes.create_string_buffer(1 << 20)
        self.lib.fake_launches(buf, len(buf))
        return buf.value.decode().split()


@pytest.fixture(scope="session")
def fake_engine(engine_lib, tmp_path_factory):
    import glob
    import shutil
    import subprocess

    import build as b

    out = str(tmp_path_factory.mktemp("fake") / "libfake.so")
    nvcc = shutil.which(b.nvcc()) or b.nvcc()
    cuda = os.path.join(os.path.dirname(os.path.dirname(nvcc)), "include")
    subprocess.run(["g++", "-O1", "-std=c++17", "-fPIC", "-shared", "-Wl,--no-undefined,-Bsymbolic", f"-I{cuda}", "-o", out,
                    os.path.join(ROOT, "tests", "fake_cuda.cpp"), *sorted(glob.glob(os.path.join(b.OBJ, "*.o"))),
                    "-lpthread"], check=True)
    return FakeEngine(out)

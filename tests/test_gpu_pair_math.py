"""The packed pair arithmetic of the forward passes (physica_b200/csrc/pbf_math.cuh) against the IEEE
square root and division, bit for bit."""
import ctypes
import pathlib
import subprocess

import pytest

ROOT = pathlib.Path(__file__).resolve().parent.parent

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def check(tmp_path_factory):
    from physica_b200 import build
    out = tmp_path_factory.mktemp("pair_math") / "libpair_math.so"
    subprocess.run([build.nvcc(), *build.ARCH, *build.FLAGS, "-w", "-shared", "-cudart=static", "-Xcompiler",
                    "-fvisibility=default", "-o", str(out), str(ROOT / "tests" / "cpp" / "pair_math_check.cu")], check=True)
    lib = ctypes.CDLL(str(out))
    for name in ("check_roots", "check_root_quotients", "check_constant_quotients", "check_kernels", "check_cubic"):
        getattr(lib, name).restype = ctypes.c_longlong
    lib.check_roots.argtypes = [ctypes.c_uint32, ctypes.c_uint32]
    for name in ("check_kernels", "check_cubic"):
        getattr(lib, name).argtypes = [ctypes.c_float, ctypes.c_uint32, ctypes.POINTER(ctypes.c_longlong)]
    return lib


def test_every_root_of_the_range(check):
    """r2 from 2^-80 (h = 2^-10, r = 2^-30 h) to 2^20 (h = 2^10): every float."""
    first, last = (127 - 80) << 23, (127 + 20) << 23
    step = 1 << 28
    for at in range(first, last, step):
        assert check.check_roots(at, min(step, last - at)) == 0


def test_quotients_nearest_a_rounding_boundary(check):
    """Every divisor with the numerators that bring a / b within 12 units of a rounding boundary (the
    correction's error is below 4 units), and pseudo-random ones."""
    assert check.check_root_quotients(12) == 0
    assert check.check_constant_quotients(12) == 0


@pytest.mark.parametrize("h", [2.0 ** -10, 0.00123, 0.0125, 0.025, 0.05, 0.1, 1.0 / 3.0, 1.0, 7.7, 333.0, 1024.0])
def test_kernel_values(check, h):
    tested = ctypes.c_longlong()
    for entry in (check.check_kernels, check.check_cubic):
        assert entry(h, 1 << 22, ctypes.byref(tested)) == 0
        assert tested.value > 1 << 21


@pytest.mark.parametrize("h", [2.0 ** -11, 2048.0])
def test_radii_outside_the_range_take_the_scalar_path(check, h):
    tested = ctypes.c_longlong()
    assert check.check_kernels(h, 1 << 16, ctypes.byref(tested)) == 0
    assert tested.value == 0

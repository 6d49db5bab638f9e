"""Host checks of spnet's float-float expressions (voltage step, weight
derivative), of products with short decimals and of voltage steps near rest against
their double evaluation, bit for bit where the rounding test accepts."""
import ctypes
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("spnetff") / "libspnetff.so")
    subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-fopenmp", "-shared", "-fPIC", "-I",
                    os.path.join(ROOT, "synaptogenesis_gb300", "csrc"),
                    os.path.join(ROOT, "tests", "cpu_checks", "spnet_ff_check.cpp"), "-o", out],
                   check=True)
    lib = ctypes.CDLL(out)
    for f in (lib.check_spnet, lib.check_near, lib.check_decimal, lib.check_single):
        f.restype = ctypes.c_ulonglong
    return lib


# exponents: operands alike, as in a running network, far apart, near the
# smallest results the test takes, and beyond them
@pytest.mark.parametrize("lo,hi", [(-2, 2), (-20, 8), (-60, 60), (-104, -96), (-126, -90)])
@pytest.mark.parametrize("which", [0, 1])
def test_spnet_expressions(lib, which, lo, hi):
    accepted = ctypes.c_ulonglong()
    n = 3_000_000
    bad = lib.check_spnet(which, lo, hi, ctypes.c_ulonglong(97 * which + hi), ctypes.c_ulonglong(n),
                          ctypes.byref(accepted))
    assert bad == 0
    assert accepted.value > (0.9 * n if lo > -90 else 0)


@pytest.mark.parametrize("spread", [2, 12, 20, 26, 40])
@pytest.mark.parametrize("izhikevich", [0, 1])
def test_voltage_steps_near_rest(lib, izhikevich, spread):
    accepted = ctypes.c_ulonglong()
    n = 2_000_000
    assert lib.check_near(izhikevich, spread, ctypes.c_ulonglong(5 + spread), ctypes.c_ulonglong(n),
                          ctypes.byref(accepted)) == 0
    if spread >= 12 and not izhikevich:
        assert accepted.value > 0.999 * n


# every pattern of one binade of mantissas (ties fall on one in 10, 20 or 1000) at
# exponents of running traces, the smallest and largest taken, and the subnormals
@pytest.mark.parametrize("c", [0.9, 0.95, 0.933])
@pytest.mark.parametrize("begin,end,step", [
    (0, 0x01800000, 1), (0x0D000000, 0x0D000000 + (1 << 24), 1), (0x3B000000, 0x3B000000 + (1 << 24), 1),
    (0x7E000000, 0x7E800000, 7), (0x01800000, 0x7F800000, 1001)])
def test_products_with_short_decimals(lib, c, begin, end, step):
    accepted = ctypes.c_ulonglong()
    assert lib.check_decimal(ctypes.c_double(c), begin, end, step, ctypes.byref(accepted)) == 0
    assert accepted.value > (0.99 if begin < 0x7E000000 else 0.4) * 2 * ((end - begin) // step)


@pytest.mark.parametrize("c,units", [(0.95, 10), (0.933, 7), (0.9, 4)])
def test_fixed_points_of_decays(c, units):
    """Where a trace or derivative that only decays ends, in units of 2^-149."""
    import numpy as np
    p = np.uint32(1 << 20).view(np.float32)
    for _ in range(1000):
        p = np.float32(np.float64(p) * c)
    assert p.view(np.uint32) == units and np.float32(np.float64(p) * c) == p


def test_derivative_of_subnormal_size_is_gone_in_the_sum():
    import numpy as np
    for dw in (2.0**-60, -2.0**-60, 2.0**-149):
        assert np.float32(np.float64(np.float32(dw)) + 0.01) == np.float32(0.01)


# every 61st float here (a minute and more on a few cores for every one, which is
# what the expressions rest on: SG_EVERY_FLOAT=1)
@pytest.mark.parametrize("which", range(8))
def test_single_argument_expressions(lib, which):
    step = 1 if os.environ.get("SG_EVERY_FLOAT") else 61
    accepted = ctypes.c_ulonglong()
    assert lib.check_single(which, ctypes.c_ulonglong(which if step > 1 else 0),
                            ctypes.c_ulonglong(step), ctypes.byref(accepted)) == 0
    # what is rejected: non-finite and huge operands
    assert accepted.value > 0.7 * (1 << 32) / step

"""Host checks of what the kernels decide without a rounding test on the result at hand:
decays over every mantissa, and substep voltages of both neuron models from the function
that the kernels call."""
import ctypes
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("decided") / "libdecided.so")
    subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-shared", "-fPIC", "-I",
                    os.path.join(ROOT, "synaptogenesis_gb300", "csrc"),
                    os.path.join(ROOT, "tests", "cpu_checks", "decided_check.cpp"), "-o", out],
                   check=True)
    lib = ctypes.CDLL(out)
    lib.check_decay.restype = lib.check_substep.restype = ctypes.c_ulonglong
    return lib


# every mantissa, both signs, at the ends of the range taken without any test (2^-100 to
# 2^100: the operations do not depend on the exponent in between) and beyond it
@pytest.mark.parametrize("exponent", [-126, -101, -100, -8, 99, 100, 126])
@pytest.mark.parametrize("c", [0.9, 0.95, 0.933])
def test_decay_of_every_mantissa(lib, c, exponent):
    taken = ctypes.c_ulonglong()
    assert lib.check_decay(ctypes.c_double(c), exponent, ctypes.byref(taken)) == 0
    if -100 <= exponent < 100:
        assert taken.value == 1 << 24


# within the derivative's own bound nearly all voltages are decided, most of them without
# it; with conductances the drive's float roundings are larger and some are left
@pytest.mark.parametrize("spread", [0, 12, 20, 26, 40])
@pytest.mark.parametrize("izhikevich", [0, 1])
@pytest.mark.parametrize("quiet", [0, 1])
def test_substep_voltages(lib, quiet, izhikevich, spread):
    taken, near = ctypes.c_ulonglong(), ctypes.c_ulonglong()
    n = 2_000_000
    assert lib.check_substep(izhikevich, quiet, spread, ctypes.c_ulonglong(31 + spread), ctypes.c_ulonglong(n),
                             ctypes.byref(taken), ctypes.byref(near)) == 0
    if quiet or not izhikevich:
        assert taken.value > 0.99 * n
    if spread >= 26 and (quiet or not izhikevich):
        assert near.value > 0.5 * n

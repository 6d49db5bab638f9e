"""What the step kernels take without a run-time rounding test, over every float (about a
second an expression): decays, midpoints and subnormal products, sums and derivatives of
one operand, bit for bit the double expressions on the FP64 pipe.  And whole neuron
updates of both models against their expressions written in double, on random neurons
near rest and anywhere else."""
import ctypes
import os
import subprocess

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("decided") / "libdecided.so")
    nvcc = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "bin", "nvcc")
    subprocess.run([nvcc, "-std=c++17", "-O3", "--fmad=false", "-shared", "-Xcompiler", "-fPIC",
                    "-gencode", "arch=compute_103a,code=sm_103a",
                    "-I", os.path.join(ROOT, "synaptogenesis_gb300", "csrc"),
                    os.path.join(ROOT, "tests", "gpu_checks", "decided_check.cu"), "-o", out],
                   check=True)
    return ctypes.CDLL(out)


# non-finite and huge operands are left to the double expression: at most a quarter
@pytest.mark.parametrize("which", range(11))
def test_every_float(lib, which):
    out = (ctypes.c_ulonglong * 4)()
    assert lib.check_every_float(which, out) == 0
    assert out[1] == 1 << 32
    assert out[0] == 0, "mismatch at %#x" % out[3]
    assert out[2] > 0.7 * out[1]


@pytest.mark.parametrize("spnet", [0, 1])
def test_neuron_updates(lib, spnet):
    out = (ctypes.c_ulonglong * 4)()
    n = 1 << 28
    assert lib.check_neurons(spnet, ctypes.c_ulonglong(n), ctypes.c_ulonglong(11 + spnet), out) == 0
    assert out[1] == n
    assert out[0] == 0, "mismatch at neuron %d" % out[3]

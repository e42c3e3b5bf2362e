"""The fixed-point FFTs of the FP64 path (csrc/fx.cuh, fx_fft.cuh) compiled for the host: lines that one element
dominates, against NumPy.

A single element gives outputs of its own magnitude at every index: the largest values that the scale (the sum of the
magnitudes of all real and imaginary parts below 2^61) lets a butterfly meet.  Tolerance: input, twiddles and output are
rounded below 2 eps of the line's sum of magnitudes, the reference below eps log2(L) of it.
"""

import ctypes as C
import os
import shutil
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
EPS = np.finfo(float).eps
# every radix first and behind others; radix 8 behind the first stage: 64, 256, 320, 384, 448, 512
LENGTHS = [2, 4, 6, 8, 10, 14, 16, 22, 26, 30, 32, 34, 36, 48, 50, 64, 72, 84, 90, 96, 128, 144, 160, 192, 210, 224, 254,
           256, 270, 320, 384, 448, 512]


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    gxx = shutil.which("g++") or shutil.which("c++")
    if gxx is None:
        pytest.skip("no C++ compiler")
    so = str(tmp_path_factory.mktemp("fx") / "fx_host.so")
    r = subprocess.run([gxx, "-std=c++17", "-O2", "-fwrapv", "-w", "-shared", "-fPIC", "-I",
                        os.path.join(ROOT, "channelflow_gb300", "csrc"), "-I", "/usr/local/cuda/include",
                        os.path.join(ROOT, "tests", "cpp", "fx_host.cpp"), "-o", so], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
    return C.CDLL(so)


def _fft(lib, x, inverse):
    out = np.empty_like(x)
    lib.fx_line(len(x), int(inverse), x.ctypes.data_as(C.c_void_p), out.ctypes.data_as(C.c_void_p))
    return out


def _numpy(x, inverse):
    return np.fft.ifft(x) * len(x) if inverse else np.fft.fft(x)


@pytest.mark.parametrize("L", LENGTHS)
def test_one_element_dominates(lib, L):
    """Real, imaginary and any phase, leading factors from 1 to 2, every index; alone and with 10% of the sum elsewhere."""
    rng = np.random.default_rng(L)
    tol = (4 + np.log2(L)) * EPS
    for inverse in (False, True):
        for k in range(L):
            for phase in (1, -1, 1j, -1j, np.exp(2j * np.pi * rng.random())):
                x = np.zeros(L, complex)
                if k % 3 == 2:
                    x = (rng.standard_normal(L) + 1j * rng.standard_normal(L)) * (0.07 / L)
                x[k] = phase * rng.choice([rng.uniform(1, 2), 1.4375, 1.5, 1.99])
                s = np.abs(x.view(float)).sum()
                assert np.abs(_fft(lib, x, inverse) - _numpy(x, inverse)).max() <= tol * s

"""The single-precision face velocities of Mom2Face against 64 bits, on the CPU: the device's function compiled for the
host. The yardstick is the sum it stands for, volume * velocity formed in double and rounded once, then summed in single
precision: the error may nowhere be larger."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
W = np.array([-3, 29, -139, 533, 533, -139, 29, -3]) / 840.0
SRC = """
#include "gam_mom2face.cuh"
extern "C" void faces(const float* vol, const float* vel, float* out, long long n) {
    for (long long f = 0; f < n; ++f) {
        float a, b;
        gam::mom2face_sum<float>(vol + f, vel + f, vel + f, vel + f, out[f], a, b);
    }
}
"""


@pytest.fixture(scope="module")
def faces(tmp_path_factory):
    from kaiju_b200 import build as kb
    d = tmp_path_factory.mktemp("m2f")
    (d / "m2f.cu").write_text(SRC)
    subprocess.run([kb.NVCC, *kb.ARCH, "-O2", "-std=c++17", "-shared", "-Xcompiler", "-fPIC,-ffp-contract=off", "-I",
                    kb.CSRC, str(d / "m2f.cu"), "-o", str(d / "m2f.so")], check=True)
    lib = C.CDLL(str(d / "m2f.so"))

    def run(vol, vel):
        n = len(vol) - 7
        v, u, out = vol.astype(np.float32), vel.astype(np.float32), np.empty(n, np.float32)
        p = lambda a: a.ctypes.data_as(C.c_void_p)  # noqa: E731
        lib.faces(p(v), p(u), p(out), C.c_longlong(n))
        return out
    return run


def _exact(vol, vel):
    n = len(vol) - 7
    return sum(W[m] * (vol * vel)[m:m + n] for m in range(8)) / sum(W[m] * vol[m:m + n] for m in range(8))


def _summands_in_double(vol, vel):
    f, n = np.float32, len(vol) - 7
    fma = lambda a, b, c: f(np.float64(a) * b.astype(np.float64) + c)  # noqa: E731  (the product is exact)
    v, u, w = vol.astype(f), (vol * vel).astype(f), W.astype(f)
    sV, s = np.zeros(n, f), np.zeros(n, f)
    for m in range(8):
        sV, s = fma(w[m], v[m:m + n], sV), fma(w[m], u[m:m + n], s)
    return s * (f(1) / sV)


def _cases():
    r, x = np.random.default_rng(0), np.arange(200007.0)
    for per in (12, 32, 256):
        ph = 2 * np.pi * x / per
        vel = np.sin(ph) * (1 + 0.2 * np.cos(0.37 * ph))
        yield f"smooth{per}", np.full(len(x), 1.0 / per ** 3), vel
        yield f"warped{per}", (1 + 0.3 * np.sin(0.71 * ph)) / per ** 3, vel
    yield "random", np.exp(0.1 * r.normal(size=len(x))), r.normal(size=len(x))
    yield "stream", np.exp(0.1 * r.normal(size=len(x))), 3.0 + 0.01 * r.normal(size=len(x))
    yield "jumps", np.full(len(x), 96.0 ** -3), np.where((x // 20) % 2, 1.0, -1.0) * (1 + 0.01 * r.normal(size=len(x)))


@pytest.mark.parametrize("name,vol,vel", list(_cases()), ids=lambda q: q if isinstance(q, str) else "")
def test_no_larger_error_than_summands_in_double(faces, name, vol, vel):
    ex = _exact(vol, vel)
    err = [np.sqrt(np.mean((np.float64(q) - ex) ** 2)) for q in (faces(vol, vel), _summands_in_double(vol, vel))]
    assert err[0] <= err[1], err


def test_volumes_below_the_floor(faces):
    """Volume sums below TINY divide by TINY, as max(sum, TINY) does."""
    vol, vel = np.full(40, 1.0e-13), np.linspace(1.0, 2.0, 40)
    want = _exact(vol, vel) * 0.1
    assert np.abs(faces(vol, vel) - want).max() <= 4 * 2.0 ** -24 * np.abs(want).max()

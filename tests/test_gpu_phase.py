"""The quadrature kernels' own phase factors and reciprocal square roots
(csrc/phase.cuh) against extended precision and against CUDA's functions.

Phase factors, absolute error: the table entries are sincospi's (2 ulp of a value
below 1: 2.2e-16), the last two fused multiply-adds round at half an ulp each
(1.1e-16), the polynomials, their rounding and the remainder's stay below
5e-17: 3.8e-16 in all, 4e-16 is used whatever the phase is. CUDA's sincos adds its own 2 ulp.

Reciprocal square root, relative error: half an ulp of the last step, at most 2^-53,
and half the rounding of x y, 2^-54: 1.67e-16; the truncated series adds 5/16
e^3 < 2^-57 for estimates good to 2^-20. CUDA's rsqrt is good to 1 ulp, so the two
differ by 2 ulp at most."""

import ctypes
import shutil
import subprocess
from pathlib import Path

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
ROOT = Path(__file__).resolve().parents[1]
PHASE_MAX = 1e7  # kPhaseMax
LD = np.longdouble


@pytest.fixture(scope="module")
def probe(tmp_path_factory):
    so = tmp_path_factory.mktemp("phase") / "libphase_probe.so"
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    subprocess.run([nvcc, "-std=c++17", "-O3", "-gencode", "arch=compute_100a,code=sm_100a", "-shared", "-Xcompiler",
                    "-fPIC", "-I", str(ROOT / "sie-gstc-2026_b200" / "csrc"), "-I", str(ROOT / "include"), "-o", str(so),
                    str(ROOT / "tests" / "phase_probe.cu")], check=True)
    return ctypes.CDLL(str(so))


def _run(fn, x, rows, *args):
    import torch
    n = x.size
    dx = torch.from_numpy(x).cuda()
    out = torch.zeros((rows, n), dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    ptr = ctypes.c_void_p
    assert fn(n, *args, ptr(dx.data_ptr()), ptr(out.data_ptr())) == 0
    return out.cpu().numpy()


def _product(k, x):
    """k x = hi + lo exactly (Dekker's product)."""
    def halves(a):
        c = 134217729.0 * a
        h = c - (c - a)
        return h, a - h
    hi = k * x
    (kh, kl), (xh, xl) = halves(k), halves(x)
    return hi, ((kh * xh - hi) + kh * xl + kl * xh) + kl * xl


@pytest.mark.parametrize("k", [1.0, 2 * np.pi, 0.37, 209.58, 4.0e5])
def test_phase_factors(k, probe):
    rng = np.random.default_rng(int(k * 100))
    steps = np.arange(-300, 300) * (np.pi / 128 / k)  # the middle and the ends of the table's steps
    ends = np.array([0.0, 1e-300, -1e-300, 1e-12, PHASE_MAX / k, -PHASE_MAX / k])
    x = np.concatenate([ends, steps, np.nextafter(steps, 1.0), np.nextafter(steps, -1.0),
                        rng.uniform(-10, 10, 20000) / k, rng.uniform(-PHASE_MAX, PHASE_MAX, 40000) / k])
    x = x[np.abs(k * x) <= PHASE_MAX]
    c, s, cc, cs = _run(probe.probe_phase, x, 4, ctypes.c_double(k))
    hi, lo = _product(k, x)
    ch, sh = np.cos(LD(hi)), np.sin(LD(hi))
    assert np.abs(LD(c) - (ch - lo * sh)).max() <= 4e-16
    assert np.abs(LD(s) - (sh + lo * ch)).max() <= 4e-16
    if k == 1.0:  # sincos gets the exact product
        assert np.abs(c - cc).max() <= 4e-16 + 2.2e-16
        assert np.abs(s - cs).max() <= 4e-16 + 2.2e-16


def test_reciprocal_square_root(probe):
    rng = np.random.default_rng(1)
    e = 2.0 ** np.arange(-80, 81)  # squared distances from 1e-24 on: R below 1e-12 is left out
    x = np.concatenate([e, np.nextafter(e, 0.0), np.nextafter(e, 1e300), 3.0 * e, 10.0 ** rng.uniform(-24, 24, 100000),
                        rng.uniform(1.0, 4.0, 100000)])
    got, cuda = _run(probe.probe_rsqrt, x, 2)
    want = 1 / np.sqrt(LD(x))
    assert np.abs((LD(got) - want) / want).max() <= 1.67e-16 + 2.0 ** -57
    assert np.abs(got.view(np.int64) - cuda.view(np.int64)).max() <= 2

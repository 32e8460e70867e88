"""The library's own reciprocal and reciprocal square root (csrc/common.cuh)
against extended precision, over random mantissas and the whole range of
exponents that their callers accept, its ends, and arguments close to 1.

Bounds, in ulp of the result.  With E the largest residual |1 - d r| or
|1 - a r^2| of the hardware's approximation r (which has at most 21 significant
bits, so that r^2 is exact), the step leaves out E^3 or 5/16 E^3 of the value
and rounds once: at most 1/2 + 2^53 E^3 (times 5/16); the rounding of the
correction itself is 2^53 2^-53 E, below 2^-15.  The rounding errors of N values
with random last bits average to 0 within 6 / sqrt(12 N).
"""
import os
import subprocess

import numpy as np
import pytest

from conftest import PKG, ROOT

pytestmark = pytest.mark.gpu

N = 1 << 20


@pytest.fixture(scope="module")
def driver(tmp_path_factory):
    out = tmp_path_factory.mktemp("approx") / "approx_gpu_driver"
    nvcc = "/usr/local/cuda/bin/nvcc"
    subprocess.check_call([nvcc if os.path.exists(nvcc) else "nvcc", "-std=c++20", "-O3", "--fmad=false",
                           "-gencode", "arch=compute_100a,code=sm_100a", "-I", os.path.join(PKG, "csrc"),
                           "-I", os.path.join(ROOT, "include"),
                           os.path.join(ROOT, "tests", "cpp", "approx_gpu_driver.cu"), "-o", str(out)])
    return str(out)


def inputs(which, kind, rng):
    mant = 1.0 + rng.random(N)
    if kind == "range":  # the ends of the range among them
        lo, hi = (-1000, 1000) if which == 0 else (-996, 997)
        x = np.ldexp(mant, rng.integers(lo, hi, N))
        x[:4] = [np.ldexp(1.0, lo), np.nextafter(np.ldexp(1.0, lo), 1), np.nextafter(np.ldexp(1.0, hi), 0),
                 np.ldexp(1.0, hi - 1)]
        return x
    if kind == "half_to_one":  # the squared cosines of the rotation
        return 0.5 * mant
    return 1.0 - np.ldexp(rng.integers(1, 1 << 40, N).astype(np.float64), -53)  # "below_one"


@pytest.mark.parametrize("kind", ["range", "half_to_one", "below_one"])
@pytest.mark.parametrize("which", [0, 1])
def test_error_in_ulp(cuda_device, driver, tmp_path, which, kind):
    assert np.finfo(np.longdouble).nmant >= 63
    x = inputs(which, kind, np.random.default_rng(17 + which))
    fin, fout = tmp_path / "x.bin", tmp_path / "y.bin"
    x.tofile(fin)
    subprocess.run([driver, str(which), str(fin), str(fout)], check=True)
    raw, got = np.fromfile(fout).reshape(2, N)
    assert not np.any(raw.view(np.uint64) & np.uint64(0xFFFFFFFF))
    xl, rl = x.astype(np.longdouble), raw.astype(np.longdouble)
    big_e = float(np.max(np.abs(1 - (xl * rl if which == 0 else (xl * rl) * rl))))
    assert big_e <= 2.0 ** -18
    exact = 1 / xl if which == 0 else 1 / np.sqrt(xl)
    err = ((got - exact) / np.spacing(got).astype(np.longdouble)).astype(np.float64)
    left_out = 2.0 ** 53 * big_e ** 3 * (1.0 if which == 0 else 5.0 / 16.0)
    assert np.abs(err).max() <= 0.5 + left_out + 2.0 ** -9
    assert abs(err.mean()) <= left_out + 6.0 / np.sqrt(12.0 * N) + 2.0 ** -9

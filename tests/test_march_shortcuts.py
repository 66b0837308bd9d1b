"""The raycast march's shortcuts (csrc/tsdf.cu) against the expressions they
stand for: the division by a hoisted reciprocal equals IEEE division for
every significand, and the voxel and cell indices taken from the rounded
product p * (1 / vs) equal the reference's (tsdf.cu:189-193 of the reference)
wherever the march's margin lets it take them."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
f = np.float32


@pytest.fixture(scope="module")
def host(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("march") / "march.so")
    subprocess.run(["g++", "-O2", "-march=native", "-ffp-contract=off", "-shared", "-fPIC",
                    os.path.join(HERE, "cpp", "march_host.cpp"), "-o", so], check=True)
    lib = C.CDLL(so)
    lib.march_div_mismatches.restype = C.c_int64
    lib.march_div_mismatches.argtypes = [C.c_float, C.c_float]
    return lib


@pytest.mark.parametrize("b", [525.0, 262.5, 131.25, 910.0, 519.257812, 0.005, 0.0079, 1.0,
                               1.99999988, 1.00000012, 1048576.0, 9.53674316e-07])
def test_division_by_a_hoisted_reciprocal_is_exact(host, b):
    for lo in (2.0 ** -40, 1.0, 2.0 ** 38):
        assert host.march_div_mismatches(b, lo) == 0


def ref_index(p, vs):
    s = ((p / vs).astype(f) + np.sign(p).astype(f) * f(0.5)).astype(f)
    return np.trunc(s).astype(np.int64)


@pytest.mark.parametrize("vs", [0.004, 0.005, 0.0079, 0.01, 0.0123])
def test_indices_from_the_rounded_product(vs):
    vs = f(vs)
    inv = (f(1.0) / vs).astype(f)
    rng = np.random.default_rng(7)
    k = rng.integers(-3000, 3000, 1_000_000)
    near = ((k * 0.5) * float(vs) + rng.normal(0, 2e-6, k.size)).astype(f)  # rounding boundaries
    wide = rng.uniform(-1200, 1200, 200_000).astype(f)
    used = 0
    for p in (rng.uniform(-8, 8, 1_000_000).astype(f), near, wide,
              np.array([0.0, -0.0, 1e-9, -1e-9], f)):
        vp = (p * inv).astype(f)
        n = ((vp + f(12582912.0)).astype(f) - f(12582912.0)).astype(f)
        assert np.array_equal(n, np.rint(vp))
        d = (vp - n).astype(f)
        low = n.astype(np.int64) + np.where(d < 0, -1, 0)
        assert np.array_equal(low, np.floor(vp).astype(np.int64))
        thr = (np.abs(vp).astype(np.float64) * -4.76837158203125e-7
               + (0.25 - 9.5367431640625e-7)).astype(f)
        sure = np.abs((np.abs(d) - f(0.25)).astype(f)) < thr
        pd = (p - vs / f(2.0)).astype(f)
        g, g0 = ref_index(p, vs), ref_index(pd, vs)
        g1 = ref_index((pd + vs).astype(f), vs)
        assert np.array_equal(n.astype(np.int64)[sure], g[sure])
        assert np.array_equal(low[sure], g0[sure])
        assert np.array_equal(low[sure] + 1, g1[sure])
        used += int(sure.sum())
    assert used > 1_000_000


def test_division_by_merge_weights_is_exact(host):
    """The merge's quotient by weight + 1 through its tabulated reciprocal."""
    for d in list(range(1, 67)) + [100, 127, 128, 129, 200, 251, 255, 256]:
        assert host.march_div_mismatches(float(d), 2.0 ** -60) == 0
        assert host.march_div_mismatches(float(d), 0.0078125) == 0


def test_colour_quotient_by_multiplication_is_exact():
    """(old * w + obs) / (w + 1) as the high part of a product, every weight
    and numerator."""
    for d in range(1, 257):
        n = np.arange(0, 255 * (d - 1) + 256, dtype=np.uint64)
        m = np.uint64((0x1000000 + d - 1) // d)
        assert np.array_equal((n * m) >> np.uint64(24), n // np.uint64(d)), d


@pytest.mark.parametrize("cols,cx,fx", [(160, 79.5, 131.25), (640, 319.5, 525.0), (1280, 639.5, 910.0),
                                        (8192, 4000.0, 5000.0), (633, 316.0, 519.25)])
def test_pixels_from_the_approximate_quotient(cols, cx, fx):
    """The voxel's pixel from (fx x) * rcp(z) + cx equals round(fx x / z + cx)
    outside the margin, for reciprocals an ulp either way."""
    rng = np.random.default_rng(11)
    n = 500_000
    z = rng.uniform(0.1, 8.0, n).astype(f)
    u = np.concatenate([rng.uniform(-2, cols + 2, n // 2),
                        rng.integers(-1, cols + 1, n // 2) + 0.5 + rng.normal(0, 1e-4, n // 2)])
    x = ((u - cx) * z / fx).astype(f)
    ax = (f(fx) * x).astype(f)
    ref = ((ax / z).astype(f) + f(cx)).astype(f)
    want = np.trunc(ref.astype(np.float64) + np.copysign(0.5, ref)).astype(np.int64)
    margin = 0.5 - 6e-7 * (cols + abs(cx) + 1.0)
    for k in (-1, 0, 1):
        rz = ((f(1.0) / z).astype(np.float64) * (1 + k * 2.0 ** -23)).astype(f)
        a = (ax.astype(np.float64) * rz.astype(np.float64) + cx).astype(f)  # one rounding
        t = np.rint(a)
        sure = np.abs(a - t) < margin
        inside = (want >= 0) & (want < cols)
        assert np.array_equal(t[sure & inside].astype(np.int64), want[sure & inside])
        out = sure & ~inside
        assert not ((t[out] >= 0) & (t[out] < cols)).any()
        assert sure.mean() > 0.45

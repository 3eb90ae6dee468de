"""Device unit tests of the arithmetic of the kernels by lines (marked gpu),
against long-double evaluations.  Bounds in units of eps = 2^-53, counted from the
operations: sqrt_pos ends in one fused step from a value within an ulp (1 ulp);
log_ratio and atanh(f)/f form f from a difference, a sum, a reciprocal (1 ulp) and
a product and take a series or the logarithm of a rounded quotient, whose error
the logarithm divides by |ln| >= 0.4 (12 eps as for the logarithmic mean in
test_gpu_device_math, 3/|ln| more on the logarithm's branch); a component of the
two-point flux is a sum of at most four products of such values (40 eps of the
sum of their magnitudes)."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
EPS = 2.0 ** -53
LD = np.longdouble


@pytest.fixture(scope="module")
def lm(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("lm") / "libline_math.so")
    subprocess.run(["nvcc", "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17", "--expt-relaxed-constexpr",
                    "-Xcompiler", "-fPIC", "-shared", os.path.join(ROOT, "tests", "cpp", "line_math.cu"), "-o", out],
                   check=True)
    L = C.CDLL(out)
    p = C.POINTER(C.c_double)
    L.lm_scalar.argtypes = [C.c_int, p, p, p, C.c_int]
    L.lm_flux.argtypes = [C.c_int, p, p, p, C.c_double, p, C.c_int]
    return L


def _p(a):
    assert a.dtype == np.float64 and a.flags.c_contiguous
    return a.ctypes.data_as(C.POINTER(C.c_double))


def scalar(lm, which, x, y=None):
    x = np.ascontiguousarray(x, dtype=np.float64)
    y = x if y is None else np.ascontiguousarray(y, dtype=np.float64)
    out = np.empty_like(x)
    assert lm.lm_scalar(which, _p(x), _p(y), _p(out), len(x)) == 0
    return out


def pairs():
    """x, y with ratios from 1 to 1e6 on both sides of the branch points (u = 1e-4, 1e-3, 0.04)."""
    rng = np.random.default_rng(3)
    f = np.concatenate([np.logspace(-12, np.log10(0.999998), 60001), *(np.sqrt(u) * (1 + np.linspace(-2e-3, 2e-3, 2001))
                                                                       for u in (1e-4, 1e-3, 0.04))])
    x = 10 ** rng.uniform(-3, 3, len(f))
    y = x * (1 + f) / (1 - f)
    swap = rng.uniform(size=len(f)) < 0.5
    return np.where(swap, y, x), np.where(swap, x, y)


def ln(x, y):
    """ln(y / x) without cancellation: log1p of a positive number."""
    x, y = x.astype(LD), y.astype(LD)
    r = np.log1p(np.abs(y - x) / np.minimum(x, y))
    return np.where(y < x, -r, r)


def test_square_root(lm):
    rng = np.random.default_rng(5)
    x = np.concatenate([10 ** rng.uniform(-300, 300, 200000), 10 ** rng.uniform(-3, 3, 200000), [1.0, 2.0, 4.0, 1.4],
                        [np.finfo(float).tiny, np.finfo(float).max]])
    got, ref = scalar(lm, 0, x), np.sqrt(x)
    assert np.abs(got.view(np.int64) - ref.view(np.int64)).max() <= 1
    assert np.isnan(scalar(lm, 0, [-1.0, -1e-310, -1e300, -np.inf, np.nan])).all()
    np.testing.assert_array_equal(scalar(lm, 0, [0.0, -0.0, np.inf]), [0.0, 0.0, np.inf])
    small = np.array([5e-324, 1e-310, 2e-308])
    assert np.abs(scalar(lm, 0, small) - np.sqrt(small)).max() <= 2e-154


def test_logarithm_of_a_ratio(lm):
    x, x0 = pairs()
    got, ref = scalar(lm, 1, x, x0), ln(x0, x)
    bound = 12 * EPS * np.abs(ref) + 3 * EPS
    near = ref ** 2 < 0.15   # u < 0.04: series, relative to the value itself
    assert (np.abs(got - ref)[near] <= 12 * EPS * np.abs(ref)[near]).all()
    assert (np.abs(got - ref) <= bound).all()
    assert np.isnan(scalar(lm, 1, [-1.0, -0.5, -2.0, np.nan], [1.0, 1.0, 1.0, 1.0])).all()


def test_series_of_the_logarithmic_mean(lm):
    x, y = pairs()
    f = (y.astype(LD) - x) / (y.astype(LD) + x)
    L = ln(x, y)
    ref = L / (2 * f)
    got = scalar(lm, 2, x, y)
    assert (np.abs(got - ref) / ref <= 12 * EPS + np.where(f ** 2 >= 0.0399, 3 * EPS / np.abs(L), 0)).all()


@pytest.mark.parametrize("near", [True, False])
def test_two_point_flux(lm, near):
    """The rearranged flux against the textbook form, on the branch every pair of a line shares."""
    rng = np.random.default_rng(7)
    n, g = 40000, 1.4
    amp = 0.009 if near else 0.6   # near: |f| < 0.01
    a = np.empty((n, 5))
    a[:, 0], a[:, 4] = 10 ** rng.uniform(-2, 2, n), 10 ** rng.uniform(-2, 2, n)
    a[:, 1:4] = rng.uniform(-2, 2, (n, 3))
    b = a.copy()
    b[:, [0, 4]] *= 1 + amp * rng.uniform(-1, 1, (n, 2))
    b[:, 1:4] += rng.uniform(-0.5, 0.5, (n, 3))
    m = rng.uniform(-1, 1, (n, 3))
    F = np.empty((n, 5))
    assert lm.lm_flux(int(near), _p(a), _p(b), _p(m), 1 / (g - 1), _p(F), n) == 0
    A, B, M = a.astype(LD), b.astype(LD), m.astype(LD)
    rho_ln, beta_ln = [(B[:, k] - A[:, k]) / ln(a[:, k], b[:, k]) for k in (0, 4)]
    vm, v2 = (A[:, 1:4] + B[:, 1:4]) / 2, ((A[:, 1:4] ** 2).sum(1) + (B[:, 1:4] ** 2).sum(1)) / 2
    p_hat = (A[:, 0] + B[:, 0]) / (2 * (A[:, 4] + B[:, 4]))
    vn = (vm * M).sum(1)
    terms = np.stack([1 / (2 * LD(1 / (g - 1)) ** -1 * beta_ln), p_hat / rho_ln, (vm ** 2).sum(1), -v2 / 2])
    ref = np.concatenate([(rho_ln * vn)[:, None], (rho_ln * vn)[:, None] * vm + p_hat[:, None] * M,
                          (rho_ln * vn * terms.sum(0))[:, None]], axis=1)
    mass = rho_ln * (np.abs(A[:, 1:4] * M).sum(1) + np.abs(B[:, 1:4] * M).sum(1)) / 2
    v_abs = (np.abs(A[:, 1:4]) + np.abs(B[:, 1:4])) / 2
    scale = np.concatenate([mass[:, None], mass[:, None] * v_abs + (p_hat[:, None] * np.abs(M)),
                            (mass * np.abs(terms).sum(0))[:, None]], axis=1)
    assert (np.abs(F - ref) <= 40 * EPS * scale).all(), float((np.abs(F - ref) / scale).max() / EPS)

"""The element pass's arithmetic in pairs of FP32 numbers (csrc/dnl_ff.cuh), compiled for the host
and compared with extended precision: conversions, ln U and R - I of the polar decomposition with the
reference's rotations and stopping test, the binomial series of the hardening law.

Bounds: a pair holds 2^-48 of its value and every operation adds at most 2^-46; the polar
decomposition's dropped off-diagonal terms go through single precision, 2^-22 of 1e-9 each, three
of them: 8e-16 absolute at most."""

import ctypes as C
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
WRAP = r"""
#define __host__
#define __device__
#define __forceinline__ inline
#include "dnl_ff.cuh"
using namespace dnl;
extern "C" {
void of_f64(int n, const double *x, int k, double *back) {
  for (int i = 0; i < n; i++) back[i] = f64_of(ff_of(x[i], k * (1 << 20)), -k * (1 << 20));
}
void polar(int n, const double *g, double *L, double *Q) {
  const ff tol = ff_host(1e-9);
  for (int i = 0; i < n; i++) {
    ff G[3][3], E[6], l[6], q[3][3];
    for (int k = 0; k < 9; k++) G[k / 3][k % 3] = ff_of(g[9 * i + k]);
    const float mg = green_ff<false>(G, E);
    strain_ff<false, false>(G, E, mg, tol, 29, -1, l, q);
    for (int k = 0; k < 9; k++) {
      L[9 * i + k] = f64_of(l[sym_of(k / 3, k % 3)]);
      Q[9 * i + k] = f64_of(q[k / 3][k % 3]);
    }
  }
}
void pow1p(int n, const double *q, double e, double *out) {
  const MatFF m = make_mat_ff(2., 3., 2., 1., 1., e, 1., 1.);
  for (int i = 0; i < n; i++) out[i] = f64_of(pow1p_ff(m, ff_host(q[i])));
}
void slope(int n, const double *a, const double *b, double *out) {
  for (int i = 0; i < n; i++) out[i] = f64_of(half_log_slope_ff(ff_host(a[i]), ff_host(b[i])));
}
void powq(int n, const double *q, double e, double *out) {
  const MatFF m = make_mat_ff(2., 3., 2., 1., 1., e, 1., 1.);
  for (int i = 0; i < n; i++) out[i] = f64_of(powq_ff(m.n, m.n3, ff_host(q[i])));
}
}
"""


@pytest.fixture(scope="module")
def pairs(tmp_path_factory):
    d = tmp_path_factory.mktemp("pairs")
    (d / "w.cc").write_text(WRAP)
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-fPIC", "-shared", "-w",
                    "-I" + os.path.join(ROOT, "redynela_gb300", "csrc"), "-o", str(d / "w.so"), str(d / "w.cc")], check=True)
    return C.CDLL(str(d / "w.so"))


def _p(a):
    return a.ctypes.data_as(C.POINTER(C.c_double))


def test_conversions(pairs):
    rng = np.random.default_rng(0)
    x = rng.normal(size=4000) * 2.0 ** rng.integers(-60, 60, size=4000)
    x[:3] = 0.0, -0.0, 1.0
    for k in (0, -36, 7):
        back = np.empty_like(x)
        pairs.of_f64(len(x), _p(x), k, _p(back))
        small = np.abs(x) * 2.0 ** k < 2.0 ** -70  # by definition 0
        assert np.all(back[small] == 0.0)
        assert np.all(np.abs(back - x)[~small] <= 2.0 ** -48 * np.abs(x[~small]))


def _reference_polar(G):
    """ln U and R - I in extended precision: the reference's pivots, rotations and stop at 1e-9."""
    LD = np.longdouble
    F = G.astype(LD) + np.eye(3, dtype=LD)
    A, V = F.T @ F, np.eye(3, dtype=LD)
    for _ in range(29):
        q = 1 if abs(A[0, 1]) > abs(A[0, 2]) else 2
        p, q = (0, q) if abs(A[0, q]) > abs(A[1, 2]) else (1, 2)
        if abs(A[p, q]) < LD("1e-9"):
            break
        al = (A[q, q] - A[p, p]) / (2 * A[p, q])
        t = 1 / (abs(al) + np.sqrt(al * al + 1)) * (-1 if al < 0 else 1)
        R = np.eye(3, dtype=LD)
        R[p, p] = R[q, q] = 1 / np.sqrt(1 + t * t)
        R[p, q], R[q, p] = t * R[p, p], -t * R[p, p]
        A, V = R.T @ A @ R, V @ R
    lam = np.diag(A)
    return (V * (np.log1p(lam - 1) / 2)) @ V.T, F @ ((V / np.sqrt(lam)) @ V.T) - np.eye(3, dtype=LD)


@pytest.mark.parametrize("exponent", [-40, -30, -20, -14, -11, -10, -9, -8, -7])
def test_polar_decomposition(pairs, exponent):
    rng = np.random.default_rng(exponent + 100)
    n = 300
    G = rng.normal(size=(n, 3, 3))
    G[::3] *= np.where(np.eye(3) > 0, 1.0, 1e-3)  # nearly diagonal
    G[1::7, 0, 1] = G[1::7, 1, 0] = 0.0
    G *= 2.0 ** exponent / np.abs(G).max(axis=(1, 2))[:, None, None]
    G[0] = 0.0
    G = G.astype(np.float32).astype(np.float64)  # exact as pairs
    L, Q = np.empty_like(G), np.empty_like(G)
    pairs.polar(n, _p(np.ascontiguousarray(G)), _p(L), _p(Q))
    bound = 8e-16 + 2.0 ** -44 * 2.0 ** exponent
    for i in range(n):
        l, q = _reference_polar(G[i])
        assert np.abs(L[i] - l).max() <= bound and np.abs(Q[i] - q).max() <= bound, i


@pytest.mark.parametrize("n", [0.05, 0.31, 0.5, 1.0, 1.7, 2.0])
def test_power_series(pairs, n):
    q = np.concatenate([[0.0], np.geomspace(1e-12, 2.0 ** -6, 400)])
    out = np.empty_like(q)
    pairs.pow1p(len(q), _p(q), C.c_double(n), _p(out))
    want = np.expm1(np.longdouble(n) * np.log1p(q.astype(np.longdouble)))
    # relative to (1 + q)^n: the omitted q^9 term (below 2^-54) and 2^-46 of the sum
    assert np.abs(out - want).max() <= 2.0 ** -46 * 2.0 ** -6 * 2 + 2.0 ** -52


@pytest.mark.parametrize("n", [0.05, 0.31, 1.0, 2.0, 5.0])
def test_power_at_large_ratios(pairs, n):
    """(1 + q)^n - 1 beyond the series' range: q from 1e-3 to 1e9 (a point's first plastic steps)."""
    q = np.geomspace(1e-3, min(1e9, 2.0 ** (50 / n)), 3000)
    out = np.empty_like(q)
    pairs.powq(len(q), _p(q), C.c_double(n), _p(out))
    want = np.expm1(np.longdouble(n) * np.log1p(q.astype(np.longdouble)))
    # the exponent's fraction, below 1, and its logarithm n log2 z / ln 2 carry 2^-46 each
    assert np.abs((out - want) / (1 + want)).max() <= (2 + n) * 2.0 ** -46


def test_power_at_random_exponents(pairs):
    rng = np.random.default_rng(4)
    for n in rng.uniform(0.05, 2.0, 200):
        q = 10.0 ** rng.uniform(-2, 8, 500)
        out = np.empty_like(q)
        pairs.powq(len(q), _p(q), C.c_double(n), _p(out))
        want = np.expm1(np.longdouble(n) * np.log1p(q.astype(np.longdouble)))
        assert np.abs((out - want) / (1 + want)).max() <= (2 + n) * 2.0 ** -46


@pytest.mark.parametrize("apart", [0.0, 1e-12, 1e-6, 1e-3, 0.33, 0.36, 0.6])
def test_slope_of_the_logarithm(pairs, apart):
    """(ln(1 + a) - ln(1 + b)) / (2 (a - b)), equal arguments, near ones and both sides of the series' end."""
    rng = np.random.default_rng(8)
    a = rng.uniform(-0.4, 0.4 - apart, 2000)
    b = a + apart
    out = np.empty_like(a)
    pairs.slope(len(a), _p(a), _p(b), _p(out))
    la, lb = (x.astype(np.longdouble) for x in (a, b))
    d = la - lb
    u = d / (2 + la + lb)
    # atanh(u) / u: its series for small u, where the quotient of differences would cancel
    ratio = np.where(np.abs(u) > 0.01, np.arctanh(u) / np.where(u == 0, 1, u), sum(u ** (2 * k) / (2 * k + 1) for k in range(8)))
    want = ratio / (2 + la + lb)
    # a dozen pair operations of 2^-46 each; logarithms subtracted: below 0.52 and at least 0.17 apart
    assert np.abs((out - want) / want).max() <= 12 * 2.0 ** -46

"""The pair arithmetic of csrc/dnl_ff.cuh at the ends of the ranges that it is used in, compiled for the
host and compared with extended precision: nearly rank-one displacement gradients, whose eigenvalues are
three times their entries, at the lines between the lengths of the series; the eigenvalues' functions.

Bounds: those of the pair itself, 2^-44 of the increment for a few dozen operations, and three times
2^-22 of the stop's 1e-9 (terms that the reference drops go through single precision)."""

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
template <bool TWO_D, bool KEEP> void polar_t(int n, const double *g, double *L, double *Q, double *H, double *rest) {
  const ff tol = ff_host(1e-9);
  for (int i = 0; i < n; i++) {
    ff G[3][3], E[6], E0[6], l[6], q[3][3], V[3][3], lam[3], h[6];
    for (int k = 0; k < 9; k++) G[k / 3][k % 3] = ff_of(g[9 * i + k]);
    const float mg = green_ff<TWO_D>(G, E);
    for (int k = 0; k < 6; k++) E0[k] = E[k];
    strain_ff<TWO_D, KEEP>(G, E, mg, tol, 29, -1, l, q, V, lam, h);
    for (int k = 0; k < 9; k++) {
      L[9 * i + k] = f64_of(l[sym_of(k / 3, k % 3)]);
      Q[9 * i + k] = f64_of(q[k / 3][k % 3]);
      H[9 * i + k] = KEEP ? f64_of(h[sym_of(k / 3, k % 3)]) : 0.;
    }
    // E V = V lambda but for what the stop leaves off the diagonal
    double r = 0.;
    if (KEEP)
      for (int a = 0; a < 3; a++)
        for (int c = 0; c < 3; c++) {
          double s = -f64_of(V[a][c]) * f64_of(lam[c]);
          for (int b = 0; b < 3; b++) s += f64_of(E0[sym_of(a, b)]) * f64_of(V[b][c]);
          if (fabs(s) > r) r = fabs(s);
        }
    rest[i] = r;
  }
}
extern "C" {
void functions(int n, const double *x, double *half_log, double *rsqrt) {
  for (int i = 0; i < n; i++) {
    half_log[i] = f64_of(half_log1p_ff(ff_host(x[i])));
    rsqrt[i] = f64_of(rsqrt1p_ff(ff_host(x[i])));
  }
}
void polar(int two, int keep, int n, const double *g, double *L, double *Q, double *H, double *rest) {
  if (two)
    keep ? polar_t<true, true>(n, g, L, Q, H, rest) : polar_t<true, false>(n, g, L, Q, H, rest);
  else
    keep ? polar_t<false, true>(n, g, L, Q, H, rest) : polar_t<false, false>(n, g, L, Q, H, rest);
}
}
"""


@pytest.fixture(scope="module")
def pairs(tmp_path_factory):
    d = tmp_path_factory.mktemp("pairs_range")
    (d / "w.cc").write_text(WRAP)
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-fPIC", "-shared", "-w",
                    "-I" + os.path.join(ROOT, "redynela_gb300", "csrc"), "-o", str(d / "w.so"), str(d / "w.cc")], check=True)
    return C.CDLL(str(d / "w.so"))


def _p(a):
    return a.ctypes.data_as(C.POINTER(C.c_double))


def _reference_polar(G):
    """ln U, R - I and U^-1 - I in extended precision: the reference's pivots, rotations and stop at 1e-9."""
    LD = np.longdouble
    one = np.eye(3, dtype=LD)
    F = G.astype(LD) + one
    E, V = F.T @ F - one, one.copy()
    for _ in range(29):
        q = 1 if abs(E[0, 1]) > abs(E[0, 2]) else 2
        p, q = (0, q) if abs(E[0, q]) > abs(E[1, 2]) else (1, 2)
        if abs(E[p, q]) < LD("1e-9"):
            break
        al = (E[q, q] - E[p, p]) / (2 * E[p, q])
        t = 1 / (abs(al) + np.sqrt(al * al + 1)) * (-1 if al < 0 else 1)
        R = one.copy()
        R[p, p] = R[q, q] = 1 / np.sqrt(1 + t * t)
        R[p, q], R[q, p] = t * R[p, p], -t * R[p, p]
        E, V = R.T @ E @ R, V @ R
    lam = np.diag(E)
    Ui = (V / np.sqrt(1 + lam)) @ V.T
    return (V * (np.log1p(lam) / 2)) @ V.T, F @ Ui - one, Ui - one


def rank_one(rng, n, size, two):
    """Nearly a a^T with a = (+-1, +-1, +-1), either sign: eigenvalues of 3 (plane: 2) times the entries."""
    a = rng.choice([-1.0, 1.0], size=(n, 3))
    G = a[:, :, None] * a[:, None, :] * rng.choice([-1.0, 1.0], size=(n, 1, 1)) * (1 + 0.02 * rng.uniform(-1, 1, (n, 3, 3)))
    if two:
        G[:, :2, 2] = G[:, 2, :2] = 0.0
    G *= size / np.abs(G).max(axis=(1, 2))[:, None, None]
    return np.ascontiguousarray(G.astype(np.float32).astype(np.float64))  # exact as pairs


def check_polar(pairs, G, two, size):
    n = len(G)
    for keep in (0, 1):
        L, Q, H, rest = np.empty_like(G), np.empty_like(G), np.empty_like(G), np.empty(n)
        pairs.polar(int(two), keep, n, _p(G), _p(L), _p(Q), _p(H), _p(rest))
        bound = 8e-16 + 2.0 ** -44 * size
        for i in range(n):
            l, q, h = _reference_polar(G[i])
            assert np.abs(L[i] - l).max() <= bound and np.abs(Q[i] - q).max() <= bound, i
            if keep:
                assert np.abs(H[i] - h).max() <= bound, i
        if keep:  # two dropped entries of 1e-9 a column, E and V as pairs
            assert rest.max() <= 1.5e-9


@pytest.mark.parametrize("two", [False, True])
@pytest.mark.parametrize("exponent", [-20, -12.6, -12.5, -11.6, -11.05, -11, -9, -8.6, -8.5, -8, -7.05])
def test_rank_one_increments(pairs, exponent, two):
    size = 2.0 ** exponent
    check_polar(pairs, rank_one(np.random.default_rng(30), 200, size, two), two, size)


def test_functions_of_an_eigenvalue(pairs):
    """ln(1 + x)/2 and (1 + x)^(-1/2) - 1 over their whole range, -1/2 to 1.  Bound: relative, 2^-45 as they
    state (half a dozen pair operations of 2^-47 and the series' 2^-47)."""
    x = np.concatenate([np.linspace(-0.5, 1.0, 3001), np.geomspace(1e-12, 0.5, 200), -np.geomspace(1e-12, 0.5, 200)])
    x = x[x != 0]
    hl, rs = np.empty_like(x), np.empty_like(x)
    pairs.functions(len(x), _p(x), _p(hl), _p(rs))
    # the pair of x holds 2^-48 of it
    hi = x.astype(np.float32).astype(np.float64)
    e = hi.astype(np.longdouble) + (x - hi).astype(np.float32)
    want = np.log1p(e) / 2
    assert np.abs((hl - want) / want).max() <= 2.0 ** -45
    y = 1 + e
    want = -e / (y + np.sqrt(y))
    assert np.abs((rs - want) / want).max() <= 2.0 ** -45

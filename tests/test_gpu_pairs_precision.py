"""How precise the element pass's kinematics and polar decomposition are: ln U and R of single elements
against extended precision, for increments on both sides of every line between the pairs' forms and the FP64
form.

Bounds (root mean square over points and components): rounding F = I + G to FP64 costs its diagonal up to
2^-53, and ln U as much; R = F U^-1 is a sum of products of rounded factors near 1, four times that."""

import os
import re

import numpy as np
import pytest

from redynela_gb300 import meshes

pytestmark = pytest.mark.gpu
LD = np.longdouble
ETYPES = {"axi": meshes.ELQUA4NAX, "plane": meshes.ELQUA4N2D, "hex": meshes.ELHEX8N3D, "tet4": meshes.ELTET4N3D,
          "hex1pt": meshes.ELHEX8N3D_1PT}
CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "redynela_gb300", "csrc")
with open(os.path.join(CSRC, "dnl_ff.cuh")) as src:
    LIMIT = float.fromhex(re.search(r"kFastMax = (\S+)f;", src.read()).group(1))  # |F - I| of the pairs' form
QUAD = np.array([[0, 0], [1, 0], [1, 1], [0, 1]], float)
HEX = np.array([[*xy, z] for z in (0, 1) for xy in QUAD], float)
TET = np.array([[0, 0, 0], [1, 0, 0], [0, 1, 0], [0, 0, 1]], float)


def _nodes(et):
    return QUAD if et in (meshes.ELQUA4NAX, meshes.ELQUA4N2D) else TET if et == meshes.ELTET4N3D else HEX


def _tables(et):
    """Shape values (q, k) and derivatives (q, k, c) at the integration points, extended precision."""
    if et == meshes.ELTET4N3D:
        return np.full((1, 4), LD(1) / 4), np.array([[[-1, -1, -1], [1, 0, 0], [0, 1, 0], [0, 0, 1]]], LD)
    sign = 2 * _nodes(et).astype(LD) - 1
    pts = np.zeros((1, 3), LD) if et == meshes.ELHEX8N3D_1PT else sign / np.sqrt(LD(3))
    f = 1 + pts[:, None, :] * sign[None]
    d = sign.shape[1]
    D = np.stack([sign[None, :, c] * np.prod(np.delete(f, c, axis=2), axis=2) for c in range(d)], axis=2) / LD(2) ** d
    return np.prod(f, axis=2) / LD(2) ** d, D


def _inverse(J):
    d = J.shape[-1]
    A = np.empty_like(J)
    if d == 2:
        A[..., 0, 0], A[..., 0, 1], A[..., 1, 0], A[..., 1, 1] = J[..., 1, 1], -J[..., 0, 1], -J[..., 1, 0], J[..., 0, 0]
    else:
        for r in range(3):
            for c in range(3):
                u, v, p, q = (c + 1) % 3, (c + 2) % 3, (r + 1) % 3, (r + 2) % 3
                A[..., r, c] = J[..., u, p] * J[..., v, q] - J[..., v, p] * J[..., u, q]
    return A / sum(J[..., 0, c] * A[..., c, 0] for c in range(d))[..., None, None]


def _polar(G, tol):
    """ln U and R from G = F - I: the reference's pivots, rotations and stop at tol, on C - I."""
    n, I = len(G), np.arange(len(G))
    one = np.eye(3, dtype=LD)
    E, V = G + G.transpose(0, 2, 1) + np.einsum("nki,nkj->nij", G, G), np.tile(one, (n, 1, 1))
    for _ in range(29):
        q1 = np.abs(E[:, 0, 1]) > np.abs(E[:, 0, 2])
        p0 = np.where(q1, np.abs(E[:, 0, 1]), np.abs(E[:, 0, 2])) > np.abs(E[:, 1, 2])
        p, q = np.where(p0, 0, 1), np.where(p0 & q1, 1, 2)
        x = E[I, p, q]
        go = np.abs(x) >= LD(tol)
        al = (E[I, q, q] - E[I, p, p]) / (2 * np.where(go, x, 1))
        t = np.where(go, 1 / (np.abs(al) + np.sqrt(al * al + 1)) * np.where(al < 0, -1, 1), 0)
        R = np.tile(one, (n, 1, 1))
        R[I, p, p] = R[I, q, q] = 1 / np.sqrt(1 + t * t)
        R[I, p, q], R[I, q, p] = t * R[I, p, p], -t * R[I, p, p]
        E, V = np.einsum("nji,njk,nkl->nil", R, E, R), np.einsum("nij,njk->nik", V, R)
    lam = np.einsum("nii->ni", E)
    F = G + one
    return np.einsum("nik,nk,njk->nij", V, np.log1p(lam) / 2, V), F @ np.einsum("nik,nk,njk->nij", V, 1 / np.sqrt(1 + lam), V)


def _elements(et, size, seed, shear=0.0):
    """Separate distorted elements at some distance from the origin, displaced by gradients whose largest
    entry is `size` (of each element, or of all; a third each random, nearly rank one, simple shear), with
    a little noise."""
    rng = np.random.default_rng(seed)
    ref = _nodes(et)
    dim, E, h = ref.shape[1], 48, 1e-3
    X = ref[None] * h + rng.uniform(-0.1, 0.1, (E,) + ref.shape) * h
    X = X @ (np.eye(dim) + shear * np.triu(np.ones((dim, dim)), 1)).T
    off = rng.uniform(5.0, 60.0, (E, 1, dim)) * h
    G = rng.normal(size=(E, dim, dim))
    a = rng.choice([-1.0, 1.0], size=(E, dim))
    G[::3] = (a[:, :, None] * a[:, None, :] * (1 + 0.02 * rng.uniform(-1, 1, G.shape)))[::3]
    G[1::3] = 0.02 * G[1::3]
    G[1::3, 0, dim - 1] = 1.0
    size = np.broadcast_to(size, E)[:, None, None]
    G *= size / np.abs(G).max(axis=(1, 2), keepdims=True)
    u = np.einsum("eij,ekj->eki", G, X - X.mean(axis=1, keepdims=True)) + 1e-3 * size * h * rng.normal(size=X.shape)
    X = X + off
    N = E * len(ref)
    x3, u3 = np.zeros((N, 3)), np.zeros((N, 3))
    x3[:, :dim], u3[:, :dim] = X.reshape(N, dim), u.reshape(N, dim)
    m = meshes.Model(et, x3, np.arange(N).reshape(E, -1), tend=1.0,
                     method=meshes.PULSE if et == meshes.ELHEX8N3D else meshes.COURANT)
    return m, x3, u3


def _reference(et, x3, u3, tol="1e-9"):
    k = len(_nodes(et))
    dim = _nodes(et).shape[1]
    N, D = _tables(et)
    x, u = (a.reshape(-1, k, 3)[..., :dim].astype(LD) for a in (x3, u3))
    Ji = _inverse(np.einsum("ekr,qkc->eqrc", x, D))
    G = np.zeros(Ji.shape[:2] + (3, 3), LD)
    G[..., :dim, :dim] = np.einsum("ekr,qkl,eqlc->eqrc", u, D, Ji)
    if et == meshes.ELQUA4NAX:
        G[..., 2, 2] = np.einsum("qk,ek->eq", N, u[..., 0]) / np.einsum("qk,ek->eq", N, x[..., 0])
    return _polar(G.reshape(-1, 3, 3), tol)


def _rms(a):
    return float(np.sqrt(np.mean(np.square(a.astype(LD)))))


def check(gpu_lib, name, size, seed, shear=0.0, tol="1e-9"):
    et = ETYPES[name]
    m, x3, u3 = _elements(et, size, seed, shear)
    d = gpu_lib.GpuDomain(m, gpu_lib.FLAG_STEP_TENSORS)
    d.internal_forces(x3, u3)
    lnU, R = (a.reshape(-1, 3, 3) for a in d.step_tensors())
    want = _reference(et, x3, u3, tol)
    assert _rms(lnU - want[0]) <= 2.0 ** -53
    assert _rms(R - want[1]) <= 2.0 ** -51


# (the FP64 form of the one-point hexahedron sums absolute coordinates: 2^-53 up to 2^-5)
@pytest.mark.parametrize("name,exponent", [(n, e) for n in sorted(ETYPES) for e in (-3, -4, -5, -6, -6.5, -7, -8, -9, -10, -11.1, -12.6, -16, -30)
                                           if n != "hex1pt" or e <= -5])
def test_increments(gpu_lib, name, exponent):
    check(gpu_lib, name, 2.0 ** exponent, 40)


@pytest.mark.parametrize("shear", [1.0, 2.0])
@pytest.mark.parametrize("exponent", [-6, -7.5, -8.1, -9, -12])
@pytest.mark.parametrize("name", sorted(ETYPES))
def test_increments_of_sheared_elements(gpu_lib, name, exponent, shear):
    check(gpu_lib, name, 2.0 ** exponent, 42, shear)


@pytest.mark.parametrize("near", [0.97, 1.03, "both"])
@pytest.mark.parametrize("name", sorted(ETYPES))
def test_increments_at_the_limit(gpu_lib, name, near):
    """Below, above, and both in every warp."""
    f = np.where(np.arange(48) % 3 == 1, 0.97, 1.03) if near == "both" else near
    check(gpu_lib, name, LIMIT * f, 43)


@pytest.mark.parametrize("tol", ["1e-5", "1e-7", "1.5e-9", "1e-12"])
@pytest.mark.parametrize("name", ["axi", "hex"])
def test_other_stopping_tolerances(gpu_lib, name, tol):
    """A looser stop leaves larger terms off the diagonal, which the result drops as the reference does."""
    gpu_lib.set_stop_tolerances(float(tol), 1e-8)
    try:
        check(gpu_lib, name, 2.0 ** -9, 44, tol=tol)
    finally:
        gpu_lib.set_stop_tolerances()


def test_hourglass_forces(gpu_lib):
    """Hourglass forces alone, no stress and no increment.  Bound: the coefficient's and the projected
    velocities' chains of some twenty pair operations of 2^-47, root mean square."""
    et = meshes.ELHEX8N3D_1PT
    m, x3, u3 = _elements(et, 2.0 ** -10, 41)
    v = np.random.default_rng(41).normal(scale=50.0, size=x3.shape)
    d = gpu_lib.GpuDomain(m)
    d.set_state(v=v)
    got = d.internal_forces(x3, 0.0 * u3).reshape(-1, 8, 3)
    x, v = (a.reshape(-1, 8, 3).astype(LD) for a in (x3, v))
    sign = 2 * HEX.astype(LD) - 1
    D = _tables(et)[1][0]
    J = np.einsum("ekr,kc->erc", x, D)
    b = np.einsum("kl,elc->ekc", D, _inverse(J))
    V = 8 * np.einsum("ei,ei->e", np.cross(J[:, :, 0], J[:, :, 1]), J[:, :, 2])
    h = np.stack([sign[:, 0] * sign[:, 1], sign[:, 1] * sign[:, 2], sign[:, 2] * sign[:, 0], sign.prod(axis=1)])
    g = h - np.einsum("qk,ekr,ejr->eqj", h, x, b)
    young, nu, rho = LD(m.young), LD(m.poisson), LD(m.density)
    c = np.sqrt(young * (1 - nu) / (rho * (1 + nu) * (1 - 2 * nu)))
    ah = LD(m.hourglass) * rho * c * np.cbrt(V) ** 2 / 4
    want = -ah[:, None, None] * np.einsum("eqk,eqr->ekr", g, np.einsum("eqk,ekr->eqr", g, v))
    assert _rms(got - want) <= np.sqrt(20.0) * 2.0 ** -47 * _rms(want)


def test_radial_return_stops_where_fp64_does(gpu_lib):
    """Trial stresses whose Newton residual, 0 or 1 iterations in, is within 1.5e-7 to 1e-6 of the stopping
    tolerance of 1e-8: FP64 (2^-53 of the trial stress, 3e-8 of the tolerance) can tell on which side, and one
    iteration more or less moves evp by up to 1e-11.  No increments: the trial stress is the given one."""
    rng = np.random.default_rng(45)
    m, x3, u3 = _elements(meshes.ELTET4N3D, 0.0, 45)
    n = 960
    x3, m.coords, m.conn = np.tile(x3, (20, 1)), np.tile(m.coords, (20, 1)), np.arange(4 * n).reshape(n, 4)
    two = LD(2)
    G2 = LD(m.young) / (1 + LD(m.poisson))
    A, B, e = LD(m.A), LD(m.B), LD(m.n)
    r23, r32 = np.sqrt(two / 3), np.sqrt(LD(3) / 2)

    def newton(norm, evp, updates, stop=None):
        """|f / sigma_y| and gamma after that many updates (with stop: until it is met)."""
        h = e * B * evp ** (e - 1)
        gamma = (norm - r23 * (A + B * evp ** e)) / (G2 * (1 + 2 * h / (3 * G2)))
        for k in range(updates + 1):
            x = evp + r23 * gamma
            sigma, h = A + B * x ** e, e * B * x ** (e - 1)
            slope = r32 * G2 + r23 * h
            f = slope * gamma - (r32 * norm - sigma + h * r23 * gamma)
            go = k < updates if stop is None else np.abs(f / sigma) > stop
            gamma = np.where(go, gamma - f / slope, gamma)
        return np.abs(f / sigma), gamma

    evp = rng.uniform(1e-3, 0.3, n)
    at = np.arange(n) % 2
    goal = LD("1e-8") * (1 + rng.choice([-1, 1], n) * rng.uniform(1.5e-7, 1e-6, n).astype(LD))
    lo, hi = np.full(n, LD("1e-9")), np.full(n, LD(3))
    yield0 = (A + B * evp.astype(LD) ** e) / r32
    for _ in range(90):
        mid = np.sqrt(lo * hi)
        r = np.where(at == 0, newton(yield0 * (1 + mid), evp.astype(LD), 0)[0], newton(yield0 * (1 + mid), evp.astype(LD), 1)[0])
        lo, hi = np.where(r < goal, mid, lo), np.where(r < goal, hi, mid)
    S = rng.normal(size=(n, 3, 3))
    S += S.transpose(0, 2, 1)
    S -= np.trace(S, axis1=1, axis2=2)[:, None, None] / 3 * np.eye(3)
    S *= ((yield0 * (1 + lo)).astype(float) / np.sqrt((S * S).sum(axis=(1, 2))))[:, None, None]
    norm = np.sqrt((S.astype(LD) ** 2).sum(axis=(1, 2)))
    want = evp + r23 * newton(norm, evp.astype(LD), 6, LD("1e-8"))[1]
    d = gpu_lib.GpuDomain(m)
    d.set_state(S=S, evp=evp)
    d.internal_forces(x3, 0.0 * x3)
    assert np.abs(d.get_state("evp")["evp"].ravel() - want).max() <= 1e-14

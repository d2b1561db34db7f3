"""The element pass in FP32 pairs (increments |F - I| <= 2^-7) and its fall-back to FP64 (larger
increments, badly shaped elements, state outside the pairs' range) against the oracle, one force
pass from the same state: element counts with a partly filled last warp, increments on both sides of
the limit and within one warp, thin and sheared elements, a first yield.

Tolerance: 1e-12 relative, the parity bound of a single pass; on elements of aspect ratio a the
displacement gradient of either side carries the shortest edge's rounding, a times as much."""

import dataclasses

import numpy as np
import pytest

from oracle import states
from oracle.oracle import Oracle
from redynela_gb300 import meshes

pytestmark = pytest.mark.gpu
TOL = 1e-12


def rel(a, b):
    a, b = np.asarray(a).ravel(), np.asarray(b).ravel()
    return np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-300)


MODELS = {"axi": lambda: meshes.taylor_axi(5, 7), "plane": lambda: meshes.taylor_plane(3, 9),
          "hex": lambda: meshes.taylor_hex(5, 3), "tet4": lambda: meshes.taylor_tet(3, 3),
          "hex1pt": lambda: meshes.taylor_hex_1pt(5, 3)}


def compare(gpu_lib, m, st, tol):
    o = Oracle(m)
    o.inject(**st)
    o.internal_matrices()
    want = o.internal_forces()
    d = gpu_lib.GpuDomain(m)
    d.set_state(**{k: v for k, v in st.items() if k != "dt"})
    assert rel(d.internal_forces(), want) <= tol
    out = d.get_state("S", "Eps", "EpsPlas", "p", "evp")
    for k in out:
        assert rel(out[k], o.array(k)) <= tol, k


@pytest.mark.parametrize("scale", [0.0, 1e-7, 1e-4, 1.5e-3, 4e-3, 2e-2])
@pytest.mark.parametrize("name", sorted(MODELS))
def test_increments_around_the_limit(gpu_lib, name, scale):
    m = MODELS[name]()
    compare(gpu_lib, m, states.random_state(m, seed=11, du_scale=scale), TOL)


@pytest.mark.parametrize("name,aspect,shear", [("axi", 8.0, 0.0), ("plane", 8.0, 0.0), ("hex", 8.0, 0.0), ("tet4", 4.0, 0.0),
                                               ("hex1pt", 8.0, 0.0), ("plane", 1.0, 4.0), ("hex", 1.0, 4.0)])
def test_thin_and_sheared_elements(gpu_lib, name, aspect, shear):
    m = MODELS[name]()
    st = states.random_state(m, seed=12, du_scale=1e-4)
    up = m.dim - 1
    for x in (st["coords"],):
        x[:, up] /= aspect
        x[:, 0] += shear * x[:, up]
    st["du"][:, up] /= aspect
    compare(gpu_lib, m, st, TOL * max(aspect, 1.0 + shear * shear))


@pytest.mark.parametrize("name", sorted(MODELS))
def test_first_yield_and_other_exponents(gpu_lib, name):
    for n in (0.05, 1.0, 2.5):
        m = dataclasses.replace(MODELS[name](), n=n)
        st = states.random_state(m, seed=13, du_scale=5e-4)
        st["evp"][...] = 1e-10
        st["evp"].ravel()[::3] = 1e-4
        compare(gpu_lib, m, st, TOL)


def test_pressure_outside_the_pairs_range(gpu_lib):
    m = MODELS["hex"]()
    st = states.random_state(m, seed=14, du_scale=1e-4)
    st["p"].ravel()[5] = 1e40
    compare(gpu_lib, m, st, TOL)

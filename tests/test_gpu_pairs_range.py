"""The ends of the pair arithmetic's range: elements, states and units whose values the FP32 pairs cannot
carry, or not as precisely as FP64, against the oracle, one force pass from the same state.

Tolerance: 1e-12 relative, the parity bound of a single pass."""

import numpy as np
import pytest

from oracle import states
from oracle.oracle import Oracle
from redynela_gb300 import meshes

pytestmark = pytest.mark.gpu
TOL = 1e-12


def rel(a, b):
    a, b = np.asarray(a).ravel(), np.asarray(b).ravel()
    top = max(np.abs(b).max(initial=0.0), 1e-300)  # squares of large values overflow
    a, b = a / top, b / top
    return np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-300)


def both(gpu_lib, m, st):
    """Forces of the oracle and of the library, the library's handle and the oracle's."""
    o = Oracle(m)
    o.inject(**st)
    o.internal_matrices()
    want = o.internal_forces().copy()
    d = gpu_lib.GpuDomain(m)
    d.set_state(**{k: v for k, v in st.items() if k != "dt"})
    return want, d.internal_forces(), o, d


@pytest.mark.parametrize("hourglass", [0.0, 0.05])
def test_inverted_one_point_hexahedra(gpu_lib, hourglass):
    """Every other element numbered the other way round: a negative volume, no error in 3D."""
    m = meshes.taylor_hex_1pt(5, 3)
    m.hourglass = hourglass
    m.conn = m.conn.copy()
    m.conn[::2] = m.conn[::2][:, [4, 5, 6, 7, 0, 1, 2, 3]]
    want, got, _, _ = both(gpu_lib, m, states.random_state(m, seed=21, du_scale=1e-4))
    assert rel(got, want) <= TOL


@pytest.mark.parametrize("speed", [float("nan"), float("inf"), -1e300, 1e40, 1e-30])
def test_hourglass_velocities_of_any_size(gpu_lib, speed):
    """One node's speed out of the pairs' range, or all tiny: the other nodes' forces are not touched, and
    infinities and NaN come out where the oracle has them."""
    m = meshes.taylor_hex_1pt(5, 3)
    st = states.random_state(m, seed=22, du_scale=1e-4)
    if abs(speed) < 1.0:
        st["v"] *= speed
        st["S"][...] = st["p"][...] = st["du"][...] = 0.0  # hourglass forces alone
    else:
        st["v"][7, 1] = speed
    want, got, _, _ = both(gpu_lib, m, st)
    want, got = want.reshape(m.N, 3), got.reshape(m.N, 3)
    near = np.zeros(m.N, dtype=bool)
    near[np.unique(m.conn[(m.conn == 7).any(axis=1)])] = True
    assert np.array_equal(np.isfinite(want), np.isfinite(got))
    assert rel(got[~near], want[~near]) <= TOL
    for c in range(3):
        ok = np.isfinite(want[near, c])
        assert rel(got[near, c][ok], want[near, c][ok]) <= TOL


@pytest.mark.parametrize("coefficient,density", [(1e-9, 8930.0), (1.0, 8930.0), (0.05, 1e-24), (0.05, 1e30)])
def test_hourglass_factors_of_any_size(gpu_lib, coefficient, density):
    m = meshes.taylor_hex_1pt(5, 3)
    m.hourglass, m.density = coefficient, density
    st = states.random_state(m, seed=23, du_scale=1e-4)
    st["S"][...] = st["p"][...] = st["du"][...] = 0.0
    want, got, _, _ = both(gpu_lib, m, st)
    assert rel(got, want) <= TOL


MODELS = {"axi": lambda: meshes.taylor_axi(5, 7), "plane": lambda: meshes.taylor_plane(3, 9),
          "hex": lambda: meshes.taylor_hex(5, 3), "tet4": lambda: meshes.taylor_tet(3, 3),
          "hex1pt": lambda: meshes.taylor_hex_1pt(5, 3)}


@pytest.mark.parametrize("unit", [1e-40, 1e-16, 1e-12, 1e-9, 1e9, 1e40])
@pytest.mark.parametrize("name", sorted(MODELS))
def test_any_unit_of_length(gpu_lib, name, unit):
    """Increments of 1e-6 of an edge (stresses of 1e5 beside 1e8) in small and large units of length."""
    m = MODELS[name]()
    st = states.random_state(m, seed=24, du_scale=1e-6)
    st["v"][...] = 0.0
    m.coords = m.coords * unit
    st["coords"], st["du"] = st["coords"] * unit, st["du"] * unit
    want, got, o, d = both(gpu_lib, m, st)
    assert rel(got / unit, want / unit) <= TOL
    for k, v in d.get_state("S", "Eps", "EpsPlas", "p", "evp").items():
        assert rel(v, o.array(k)) <= TOL, k
    # the increment itself, not only the state that it is added to
    dS = (d.get_state("p")["p"].ravel() - st["p"].ravel())
    assert rel(dS, o.array("p").ravel() - st["p"].ravel()) <= 1e-9


# (a finite stress of that size has no return mapping: an error status)
@pytest.mark.parametrize("field,value", [(f, v) for f in ("S", "Eps", "EpsPlas", "p") for v in (float("nan"), float("inf"), 1e35, -1e200)
                                         if f != "S" or not np.isfinite(v)])
@pytest.mark.parametrize("name", sorted(MODELS))
def test_state_out_of_range(gpu_lib, name, field, value):
    """One point's component out of the pairs' range: infinities and NaN stay that, numbers are the
    oracle's, and no other element is touched.  (Which other components an infinity reaches depends on
    the zeros that a form leaves out and on its yield test, so they are not compared.)"""
    m = MODELS[name]()
    st = states.random_state(m, seed=25, du_scale=1e-4)
    st["v"][...] = 0.0
    st[field].reshape(m.E * m.nip, -1)[5, 0] = value
    want, got, o, d = both(gpu_lib, m, st)
    own = np.arange(m.E) == 5 // m.nip
    for k, v in d.get_state("S", "Eps", "EpsPlas", "p", "evp").items():
        g, w = v.reshape(m.E, m.nip, -1), o.array(k).reshape(m.E, m.nip, -1)
        rest = np.full(m.E, True) if np.isfinite(value) and k != field else ~own
        assert rel(g[rest], w[rest]) <= TOL, k
        if k == field:
            if np.isfinite(w[own]).all():
                assert rel(g[own], w[own]) <= TOL, k
            assert np.isfinite(g[own][0, 5 % m.nip, 0]) == np.isfinite(w[own][0, 5 % m.nip, 0])
    nodes = np.ones(m.N, dtype=bool)
    nodes[m.conn[own]] = False
    g, w = got.reshape(m.N, m.dim), want.reshape(m.N, m.dim)
    assert rel(g[nodes], w[nodes]) <= TOL
    if field in ("S", "p"):
        assert np.array_equal(np.isfinite(g[~nodes]).all(axis=1), np.isfinite(w[~nodes]).all(axis=1))


@pytest.mark.parametrize("unit", [1e-60, 1e-20, 1e20, 1e60])
@pytest.mark.parametrize("name", sorted(MODELS))
def test_any_unit_of_stress(gpu_lib, name, unit):
    m = MODELS[name]()
    st = states.random_state(m, seed=26, du_scale=1e-4)
    for k in ("young", "A", "B"):
        setattr(m, k, getattr(m, k) * unit)
    m.density *= unit  # the hourglass viscosity with it
    st["S"], st["p"] = st["S"] * unit, st["p"] * unit
    want, got, o, d = both(gpu_lib, m, st)
    assert rel(got / unit, want / unit) <= TOL
    for k, v in d.get_state("S", "Eps", "EpsPlas", "p", "evp").items():
        u = unit if k in ("S", "p") else 1.0
        assert rel(v / u, o.array(k) / u) <= TOL, k


def test_nearly_vertical_segment_of_a_table(gpu_lib):
    """evp = 1e-10 on a segment of the hardening table 1e-22 wide: the points yield there."""
    m = meshes.taylor_hex(5, 3)
    x = np.array([0.0, 1e-10 - 5e-23, 1e-10 + 5e-23, 0.1, 1.0, 10.0])
    assert np.all(np.diff(x) > 0)
    y = np.array([90e6, 90e6, 90e6 + 1e3, 150e6, 250e6, 400e6])
    m.materials = [meshes.MaterialLaw(m.young, m.poisson, m.density, meshes.HARD_TABULAR, (), x, y)]
    m.elem_material = np.zeros(m.E, dtype=np.int64)
    st = states.random_state(m, seed=27, du_scale=1e-3)
    st["evp"][...] = 1e-10
    want, got, o, d = both(gpu_lib, m, st)
    assert (o.array("evp") > 1e-9).sum() > 100  # yielded
    assert rel(got, want) <= TOL
    for k, v in d.get_state("S", "EpsPlas", "p", "evp").items():
        assert rel(v, o.array(k)) <= TOL, k

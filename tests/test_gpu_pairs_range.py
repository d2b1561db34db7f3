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

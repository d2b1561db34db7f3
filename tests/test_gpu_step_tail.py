"""The time logic in the last block of a step's last kernel: after an error that some blocks of the Courant
kernel see and others do not, and in scheduled steps of a run that is over."""

import dataclasses

import numpy as np
import pytest

from redynela_gb300 import meshes

pytestmark = pytest.mark.gpu


def test_time_step_after_a_courant_error(gpu_lib):
    """One element turns over while the nodes move, so that an early block of the Courant kernel records the
    error and later ones meet it.  The error cleared (dnl_internal_forces) and the bar at rest with its last
    row of elements squeezed, the next time step is that row's: the time logic waits for the last blocks."""
    nr, nz = 1500, 1500  # several waves of blocks, more than the caches hold
    m = meshes.taylor_axi(nr, nz, speed=0.0, tend=1.0)
    squeezed = m.coords.copy()
    squeezed[-(nr + 1):, 1] -= 0.95 * (squeezed[-1, 1] - squeezed[-1 - (nr + 1), 1])
    other = gpu_lib.GpuDomain(dataclasses.replace(m, coords=squeezed))
    other.prologue()
    want = other.time_step()
    other.close()
    d = gpu_lib.GpuDomain(m)
    d.prologue()
    d.step(9)
    rest = d.get_state("coords", "du", "v", "a", "disp")
    v = rest["v"].copy()
    v[2 * (nr + 1) + 3, 1] = 1e9
    d.set_state(v=v)
    with pytest.raises(gpu_lib.DnlError):
        d.step(1)  # the tenth: the critical time step is due
    d.internal_forces(rest["coords"], rest["du"])
    d.set_state(**dict(rest, coords=squeezed))
    d.step(10)
    assert abs(d.time_step() / want - 1.0) <= 1e-12
    assert np.array_equal(d.get_state("coords")["coords"], squeezed)


def test_scheduled_steps_of_a_finished_run(gpu_lib, tmp_path):
    """A restart at the end time: its steps do nothing, and a schedule counts its steps all the same."""
    m = meshes.taylor_axi(4, 12, tend=2e-7)
    d = gpu_lib.GpuDomain(m, gpu_lib.FLAG_STEP_TENSORS)
    d.run()
    path = str(tmp_path / "end.res")
    d.write_results(path)
    end = d.get_state("coords")["coords"]
    r = gpu_lib.GpuDomain(m, gpu_lib.FLAG_STEP_TENSORS)
    r.read_results(path)
    assert r.step(1) == 0
    x = r.run_schedule(np.full(7, 1e-9))
    assert np.array_equal(x, end)
    assert r.time_info()["increment"] == 7

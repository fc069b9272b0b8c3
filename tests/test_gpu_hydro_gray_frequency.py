"""A frequency that a gray problem's segments carry along through moving material:
a scatter leaves it with the Doppler factor of the transform back to the lab
frame alone (lorentzTransformToLab, radiation/RadiationIMC.hpp:286-310), since a
gray scatter draws no comoving frequency."""
import numpy as np
import pytest

from conftest import golden
from test_gpu_hydro import _engine_at, _problems

pytestmark = pytest.mark.gpu


def test_gray_scatter_shifts_the_frequency_once(oracle_lib):
    p = _problems()[0]["replay_hydro.npz"]
    g = golden("replay_hydro.npz")
    e = _engine_at(p, g)
    f = 2.0
    b = oracle_lib.ReplayBatch(g["before"], g["cell"], g["tape_offset"], g["tape_length"], g["tape"],
                               frequency=np.full(len(g["cell"]), f), momentum=True)
    e.replay(b)
    moved = np.abs(np.stack([b["phys_v" + a] - g["before"][:, 3 + k] for k, a in enumerate("xyz")])).max(0) > 0
    scatter = (b["phys_status"] == 0) & (b["used_random_walk"] == 0) & moved
    assert scatter.sum() >= 20
    # that factor, gamma (1 + v.u' / c^2) with the comoving direction u', is the reciprocal of
    # the lab-to-comoving one at the lab direction that the scatter left
    c = 2.99792458e10
    v = g["vel_start"][g["cell"]]
    u = np.stack([b["phys_vx"], b["phys_vy"], b["phys_vz"]], 1)
    gamma = 1.0 / np.sqrt(1.0 - (v * v).sum(1) / c ** 2)
    dop = gamma * (1.0 - (v * u).sum(1) / c ** 2)
    assert np.abs(dop[scatter] - 1.0).max() > 1e-3
    np.testing.assert_allclose(b["phys_frequency"][scatter], f / dop[scatter], rtol=1e-9)
    np.testing.assert_array_equal(b["phys_frequency"][(b["phys_status"] == 1)], f)   # a crossing does not
    e.close()

"""Which cell an emitted packet comes from: a warp makes a range of packets and
walks on from the cell of its last pass.  Exactly the allocation's counts, cell
by cell, where ranges take several passes, cells hold few or many packets, and
long runs of cells hold none."""
import numpy as np
import pytest

from storm_b200 import _abi as A
from storm_b200 import problems
from storm_b200.engine import Engine

pytestmark = pytest.mark.gpu


def _check(p):
    e = Engine(p)
    n0 = e.census_count()
    for ph in ("begin", "prestep", "emit"):
        e.phase(ph, p.dt)
    counts, _ = e.emission()
    b = e.bank()
    n = int(counts.sum())
    assert n > 0
    np.testing.assert_array_equal(b.cell[n0:n0 + n], np.repeat(np.arange(p.ncells), counts.astype(np.int64)))
    np.testing.assert_array_equal(b.id[n0:n0 + n], n0 + np.arange(n))
    e.close()


@pytest.mark.parametrize("precision", [A.PRECISION_FP64, A.PRECISION_FP32_TRACK])
@pytest.mark.parametrize("n,per_cell,hot", [
    (1, 31, 1.0), (1, 33, 1.0),              # one cell, a pass and its remainder
    (2, 200001, 1.0), (9, 1201, 0.5),        # more packets than lanes: several passes a warp
    (40, 3, 0.004), (24, 90, 0.02),          # long runs of empty cells, crossed within and between passes
])
def test_packets_lie_in_the_cells_that_emit_them(n, per_cell, hot, precision):
    p = problems.step_cube(n=n, new_photons_per_cell=per_cell, face_packets=3, comb_nmin=4, precision=precision)
    rng = np.random.default_rng(n)
    p.temperature = np.where(rng.random(p.ncells) < hot, p.temperature.max(), 1e-6 * p.temperature.max())
    p.temperature[-1] = p.temperature.max()
    _check(p)


@pytest.mark.parametrize("precision", [A.PRECISION_FP64, A.PRECISION_FP32_TRACK])
@pytest.mark.parametrize("groups", [2, 5, 64, 67])
def test_multigroup_packets(groups, precision):
    _check(problems.mg_cube(n=6, groups=groups, new_photons_per_cell=41, precision=precision))

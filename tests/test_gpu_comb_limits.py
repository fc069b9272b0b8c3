"""The comb at the ends of what it accepts: census weights down to the smallest
doubles."""
import numpy as np
import pytest

from storm_b200 import problems
from storm_b200.engine import Engine

pytestmark = pytest.mark.gpu


def census(p, cell, weight, seed=0):
    """Particles at the centres of `cell`, flying anywhere, of `weight`."""
    from oracle import ref
    n = len(cell)
    q = ref.Particles(n)
    q.cell[:] = cell
    q.id[:] = np.arange(n)
    xc, yc, zc = p.cell_centers()
    q.x, q.y, q.z = xc[cell].copy(), yc[cell].copy(), zc[cell].copy()
    u = np.random.default_rng(seed).standard_normal((3, n))
    q.vx, q.vy, q.vz = (u / np.linalg.norm(u, axis=0) * 2.99792458e10).copy()
    q.weight = np.array(weight, float)
    q.initial_weight = q.weight.copy()
    return q


def same_as_oracle(oracle_lib, p, e, pre):
    post = e.population_control(pre)
    o = oracle_lib.Oracle(p)
    o.set_census(pre)
    o.phase("comb")
    oc = o.census()
    assert post.n == oc.n > 0
    np.testing.assert_array_equal(post.cell, oc.cell)
    for f in ("x", "vx", "weight", "initial_weight"):
        np.testing.assert_array_equal(getattr(post, f), getattr(oc, f), err_msg=f)
    energy = np.zeros(p.ncells)   # the cells' census energy: the copies' weights in output order
    np.add.at(energy, post.cell, post.weight)
    np.testing.assert_array_equal(e.cells()["erad_census"], energy)


@pytest.mark.parametrize("nx", [40, 100003])   # by warps, and a thread per cell
@pytest.mark.parametrize("unit", [1e-290, 6e-309, 1e-309, 1e-318, 4.94065645841246544e-324])
def test_smallest_weights(oracle_lib, unit, nx):
    """Cells of more particles than they keep: their teeth are apart by less than
    the smallest number whose reciprocal is finite."""
    p = problems.gray_slab(nx=nx, new_photons_per_cell=1, face_packets=10, comb_nmin=8, comb_factor=1.5)
    rng = np.random.default_rng(5)
    lengths = (9, 31, 33, 64, 200, 257)
    cell = np.repeat(rng.permutation(nx)[:4 * len(lengths)], np.tile(lengths, 4))
    weight = np.ceil(1000.0 * rng.random(len(cell))) * unit
    same_as_oracle(oracle_lib, p, Engine(p), census(p, cell, weight))

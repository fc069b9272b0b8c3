"""The comb's walks along the cells' runs, by a warp per batch of runs and by a
thread per run, against the oracle: the same particles, copies and weights, bit
for bit.  Run lengths at the edges of a warp, a tile and the sort's classes;
weights spread over decades, so that particles are kept, split into few and into
many copies, and combed."""
import numpy as np
import pytest

from storm_b200 import problems
from storm_b200.engine import Engine

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,lengths,nmin,spread", [
    (40, (1, 2, 7, 8, 9, 31, 32, 33, 63, 64, 65), 8, 1.0),            # combed and split cells, tile remainders
    (40, (127, 128, 129, 255, 256, 257, 511, 512, 513), 300, 2.0),     # kept and split, across tiles
    (12, (1, 3, 40, 2000), 5000, 3.0),                                 # far more copies than particles
    (30000, (1, 2, 5, 9), 6, 2.0),                                     # several runs to a warp
    (100003, (1, 2, 4), 6, 2.0),                                       # a thread per run
])
def test_comb_walks_match_oracle(oracle_lib, nx, lengths, nmin, spread):
    from oracle import ref
    p = problems.gray_slab(nx=nx, new_photons_per_cell=1, face_packets=10, comb_nmin=nmin, comb_factor=1.5)
    rng = np.random.default_rng(nx)
    cells = rng.permutation(nx)[: min(nx - 1, 3 * len(lengths) if nx < 1000 else nx // 2)]
    cell = np.concatenate([np.full(lengths[k % len(lengths)], c) for k, c in enumerate(cells)])
    n = len(cell)
    pre = ref.Particles(n)
    pre.cell[:] = cell
    pre.id[:] = np.arange(n)
    xc, yc, zc = p.cell_centers()
    pre.x, pre.y, pre.z = xc[cell].copy(), yc[cell].copy(), zc[cell].copy()
    u = rng.standard_normal((3, n))
    pre.vx, pre.vy, pre.vz = (u / np.linalg.norm(u, axis=0) * 2.99792458e10).copy()
    pre.weight = np.exp(spread * rng.standard_normal(n))
    pre.weight[rng.random(n) < 0.2] = 1.0    # equal weights among them
    pre.initial_weight = pre.weight.copy()
    e = Engine(p)
    post = e.population_control(pre)
    o = oracle_lib.Oracle(p)
    o.set_census(pre)
    o.phase("comb")
    oc = o.census()
    assert post.n == oc.n
    np.testing.assert_array_equal(post.cell, oc.cell)
    for f in ("x", "vx", "weight", "initial_weight"):
        np.testing.assert_array_equal(getattr(post, f), getattr(oc, f), err_msg=f)
    energy = np.zeros(nx)   # the cells' census energy: the copies' weights in output order
    np.add.at(energy, post.cell, post.weight)
    np.testing.assert_array_equal(e.cells()["erad_census"], energy)

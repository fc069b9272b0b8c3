"""The comb at the ends of what it accepts: census weights down to the smallest
doubles, and cells of more particles than a block sorts."""
import numpy as np
import pytest

from storm_b200 import _abi as A
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


@pytest.mark.parametrize("longest", [8192, 8193, 20000])
@pytest.mark.parametrize("kind", ["plain", "stratified"])
def test_long_runs_on_a_used_block(oracle_lib, kind, longest):
    """A cell whose run is sorted by radix after the first plan has been launched: that
    plan must not touch the weights the first sort left unwritten, here those of
    another handle's last comb on the same memory."""
    def problem():
        p = problems.gray_slab(nx=6, new_photons_per_cell=1, face_packets=10, comb_nmin=2000, comb_factor=1.5)
        if kind == "stratified":
            p.comb_kind = A.COMB_STRATIFIED
        return p
    p = problem()
    n = 6 * 7000
    first = Engine(p)   # tiny weights in every slot of the buffers
    first.population_control(census(p, np.repeat(np.arange(6), 7000), np.full(n, 1e-309)))
    first.close()
    e = Engine(problem())
    cell = np.concatenate([np.full(longest, 2), np.array([0, 1, 3, 4, 5])[np.arange(n - longest) % 5]]).astype(np.uint32)
    weight = np.exp(np.random.default_rng(longest).standard_normal(n))
    pre = census(p, cell, weight)
    if kind == "plain":
        same_as_oracle(oracle_lib, problem(), e, pre)
        return
    a = e.population_control(pre)
    energy = e.cells()["erad_census"]
    b = e.population_control(pre)
    assert a.n == b.n > 0
    np.testing.assert_array_equal(a.cell, b.cell)
    np.testing.assert_array_equal(a.weight, b.weight)
    np.testing.assert_array_equal(energy, e.cells()["erad_census"])
    np.testing.assert_allclose(a.weight.sum(), weight.sum(), rtol=1e-9)


@pytest.mark.parametrize("nx", [20, 100003])   # by warps, and a thread per cell
@pytest.mark.parametrize("kind", ["plain", "stratified"])
def test_weights_too_small_to_split_are_kept(kind, nx):
    """A cell's share of the smallest double is zero: its particles stay as they are,
    beside a cell of ordinary ones that are split."""
    p = problems.gray_slab(nx=nx, new_photons_per_cell=1, face_packets=10, comb_nmin=50, comb_factor=1.5)
    if kind == "stratified":
        p.comb_kind = A.COMB_STRATIFIED
    tiny = 4.94065645841246544e-324
    pre = census(p, np.array([3, 7, 7, 11, 11, 11]), [tiny, tiny, 2 * tiny, 1.0, 0.5, 0.25])
    e = Engine(p)
    for _ in range(2):   # the second time the banks hold the split particles
        post = e.population_control(pre)
        np.testing.assert_array_equal(post.weight[post.cell == 3], [tiny])
        np.testing.assert_array_equal(np.sort(post.weight[post.cell == 7]), [tiny, 2 * tiny])
        hot = post.weight[post.cell == 11]
        assert len(hot) >= 50 and abs(hot.sum() - 1.75) < 1e-12 and (hot > 0).all()
        assert post.n == 3 + len(hot)


@pytest.mark.parametrize("copies", [31, 32, 33, 255, 256, 257, 5000])
@pytest.mark.parametrize("n", [1, 12, 300, 2500])
def test_many_copies(oracle_lib, n, copies):
    """Particles alone in their cells, and some beside others, split into few and many
    copies; the second comb writes into banks that the first one has grown."""
    if n * copies > 2_000_000:
        copies //= 10
    p = problems.gray_slab(nx=n, new_photons_per_cell=1, face_packets=10, comb_nmin=copies, comb_factor=0.5)
    cell = np.concatenate([np.arange(n), np.repeat(np.arange(0, n, 3), 5)]).astype(np.uint32)
    weight = np.concatenate([np.ones(n), 0.01 * np.ones(len(cell) - n)])
    e = Engine(p)
    pre = census(p, cell, weight)
    e.population_control(pre)
    same_as_oracle(oracle_lib, p, e, pre)


@pytest.mark.parametrize("nx", [148, 592, 593, 2000])
def test_run_lengths_either_side_of_the_block_sort(oracle_lib, nx):
    """Runs of 129 to 512 keys: by blocks where there are few runs, else by warps."""
    p = problems.gray_slab(nx=nx, new_photons_per_cell=1, face_packets=10, comb_nmin=100, comb_factor=1.5)
    rng = np.random.default_rng(nx)
    cell = np.repeat(rng.permutation(nx)[:140], np.tile((1, 127, 128, 129, 255, 256, 257, 400, 511, 512, 513, 600, 64, 33), 10))
    same_as_oracle(oracle_lib, p, Engine(p), census(p, cell, np.exp(rng.standard_normal(len(cell)))))

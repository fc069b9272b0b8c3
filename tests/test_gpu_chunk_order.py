"""The order of the transport's chunks and the comb's wide sum against the oracle.
A bank of one to eight waves of lanes is taken longest histories first; which
lanes a history meets, and when, is nothing that its result depends on."""
import numpy as np
import pytest

from storm_b200 import _abi as A
from storm_b200 import problems
from storm_b200.engine import Engine

from test_gpu_comb_limits import census, same_as_oracle

pytestmark = pytest.mark.gpu

LANES = 148 * 4 * 256   # a wave: four blocks of 256 a multiprocessor


def _problem(bank, precision):
    """A slab whose cells differ by decades in opacity, so that chunks differ in level,
    with `bank` packets from its face and its cells together."""
    p = problems.gray_slab(nx=50, new_photons_per_cell=10, face_packets=1000, comb_nmin=2000, comb_factor=1.0,
                           precision=precision)
    p.opacity_kind = A.OPACITY_CELL_TABLE
    p.sigma_a = 10.0 ** (np.arange(50) % 5 - 2.0)
    p.sigma_s = 10.0 ** (np.arange(50) % 3 - 1.0)
    p.dt = 1e-12
    e = Engine(p)   # the cells' own number of packets
    for ph in ("begin", "prestep", "emit"):
        e.phase(ph, p.dt)
    st = e.stats()
    e.close()
    p.faces[0].packets_per_face = bank - st["emitted_cells"]
    return p


@pytest.mark.parametrize("precision", [A.PRECISION_FP64, A.PRECISION_FP32_TRACK])
@pytest.mark.parametrize("bank,ordered", [(LANES, False), (LANES + 1, True), (2 * LANES + 37, True),
                                          (8 * LANES - 31, True), (8 * LANES + 1, False)])
def test_histories_do_not_depend_on_the_chunks_order(oracle_lib, bank, ordered, precision):
    p = _problem(bank, precision)
    e = Engine(p)
    for ph in ("begin", "prestep", "emit"):
        e.phase(ph, p.dt)
    b = e.bank()
    assert b.n == bank
    before = e.launches()
    e.phase("transport")
    # the transport, the fold, the counters' histogram, and the two of the order
    assert e.launches() - before == (5 if ordered else 3)
    e.phase("comb")
    st = e.stats()
    counts = ("segments", "escaped", "cutoff", "rw_steps", "census_out_pre_comb", "census_out")
    if precision == A.PRECISION_FP64:
        o = oracle_lib.Oracle(p)
        for ph in ("begin", "prestep", "emit", "transport", "comb"):
            o.phase(ph, p.dt)
        so, want = o.stats(), o.census()
    else:   # the same step by the other way through the bank
        f = Engine(p)
        f.set_transport_mode(False, 4)
        for ph in ("begin", "prestep", "emit", "transport", "comb"):
            f.phase(ph, p.dt)
        so, want = f.stats(), f.census()
    got = e.census()
    for k in counts:
        assert st[k] == so[k], k
    assert st["segments"] > bank
    np.testing.assert_array_equal(got.cell, want.cell)
    # a few roundings of the box (1 cm), the speed of light and the weight per segment
    for k, atol in (("x", 1e-12), ("vx", 1e-12 * 3e10), ("weight", 0.0)):
        if precision == A.PRECISION_FP64:
            np.testing.assert_allclose(getattr(got, k), getattr(want, k), rtol=1e-11, atol=atol, err_msg=k)
        else:
            np.testing.assert_array_equal(getattr(got, k), getattr(want, k), err_msg=k)


@pytest.mark.parametrize("nx", [1023, 16385, 131072, 131073, 132095, 163841])
def test_total_weight(oracle_lib, nx):
    """The total that every cell's share is taken of: by one block up to 131072 cells, by
    several above, the same partial sums; the first and the last cells weigh most."""
    p = problems.gray_slab(nx=nx, new_photons_per_cell=1, face_packets=10, comb_nmin=2, comb_factor=3.0)
    rng = np.random.default_rng(nx)
    cell = np.sort(np.concatenate([rng.integers(0, nx, 3 * nx), np.arange(nx - 5, nx), np.arange(5)]))
    weight = np.exp(rng.standard_normal(len(cell)))
    weight[cell >= nx - 5] *= nx
    weight[cell < 5] *= nx
    e = Engine(p)
    pre = census(p, cell, weight)
    for _ in range(2):   # the sum's counter is as it was
        same_as_oracle(oracle_lib, p, e, pre)

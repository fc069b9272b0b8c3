"""The gray transports' tallies: one sum per stay in a cell that serves both the
material and the radiation tally.  Against the oracle on identical streams where
the deposits do not follow from the absorption rate alone: cells without
absorption, cells too thin for an attenuation, pure scatterers, cut-off weights,
reflecting walls, Random Walk, no feedback."""
import numpy as np
import pytest

from storm_b200 import _abi as A
from storm_b200 import problems
from storm_b200.engine import Engine

pytestmark = pytest.mark.gpu


def _problem(n, precision, feedback=True):
    p = problems.step_cube(n=n, new_photons_per_cell=6, face_packets=60, comb_nmin=10, precision=precision)
    k = np.arange(p.ncells) % 6
    p.sigma_a = np.choose(k, [0.0, 1e-13, 1e-6, 1.0, 40.0, 2000.0])
    p.sigma_s = np.choose(k[::-1], [0.0, 5.0, 0.0, 300.0, 0.0, 1.0])
    p.faces[2] = problems.BoxFace(A.FACE_REFLECT)
    p.faces[5] = problems.BoxFace(A.FACE_REFLECT)
    p.no_hydro_feedback = not feedback
    return p


@pytest.mark.parametrize("n,feedback", [(1, True), (5, True), (7, False), (12, True)])
def test_fp64_tallies_match_oracle(oracle_lib, n, feedback):
    p = _problem(n, A.PRECISION_FP64, feedback)
    e, o = Engine(p), oracle_lib.Oracle(p)
    se, so = e.step(), o.step()
    for k in ("segments", "escaped", "cutoff", "rw_steps", "census_out_pre_comb"):
        assert se[k] == so[k], k
    assert abs(se["energy_deposited"] - so["energy_deposited"]) <= 1e-9 * max(abs(so["energy_deposited"]), 1e-300)
    ce, co = e.cells(), o.cells()
    np.testing.assert_array_equal(ce["segments"], co["segments"])
    assert ce["segments"].sum() == se["segments"]
    for k in ("internal_energy", "erad_time_avg"):
        np.testing.assert_allclose(ce[k], co[k], rtol=1e-9, atol=1e-9 * np.abs(co[k]).max(), err_msg=k)


@pytest.mark.parametrize("n", [5, 12])
def test_fp32_conserves_energy_and_counts(n):
    p = _problem(n, A.PRECISION_FP32_TRACK)
    e = Engine(p)
    before = p.internal_energy.sum()
    for _ in range(2):
        st = e.step()
        sink = st["energy_deposited"] + st["energy_escaped"] + st["energy_census_pre_comb"]
        source = st["energy_census_in"] + st["energy_emitted"]
        assert abs(sink - source) <= 1e-10 * source
        c = e.cells()
        after = c["internal_energy"].sum()
        assert abs(after - before - st["energy_deposited"] + st["energy_emission_debit"]) <= 1e-10 * (abs(before) + source)
        before = after
        assert c["segments"].sum() == st["segments"]
        assert np.isfinite(c["erad_time_avg"]).all() and (c["erad_time_avg"] >= 0).all()


def _forms():
    for prec in (A.PRECISION_FP32_TRACK, A.PRECISION_FP64):
        yield "gray", prec, lambda prec=prec: _problem(9, prec)
        yield "mg", prec, lambda prec=prec: problems.mg_cube(n=9, groups=30, kappa0=1.0, new_photons_per_cell=4, precision=prec)
        yield "mg_const", prec, lambda prec=prec: problems.mg_cube(n=9, groups=64, new_photons_per_cell=4, precision=prec)
        yield "ddmc", prec, lambda prec=prec: problems.ddmc_cube(n=8, with_random_walk=True, precision=prec)
        yield "voronoi", prec, lambda prec=prec: problems.voronoi_cube(ncells=200, packets_per_step=8000, precision=prec)
        yield "voronoi_ddmc", prec, lambda prec=prec: problems.voronoi_ddmc(ncells=200, packets_per_step=8000, precision=prec,
                                                                           with_random_walk=True)


@pytest.mark.parametrize("name,precision,make", [pytest.param(*f, id=f"{f[0]}-{f[1]}") for f in _forms()])
def test_histories_do_not_depend_on_their_lane(name, precision, make):
    """A history draws from its own stream wherever it runs: with other bursts the
    particles meet other lanes, and other histories' words lie in the rings
    before theirs.  One step from an empty census is the same to the last bit in
    its counts and its census."""
    ref = None
    for burst in (1, 3, 8):
        e = Engine(make())
        e.set_transport_mode(True, burst)
        st = e.step()
        p = e.census()
        got = [st[k] for k in ("segments", "rw_steps", "escaped", "cutoff", "census_out_pre_comb", "census_out")], p
        if ref is None:
            ref = got
            assert st["segments"] > 1000
            continue
        assert got[0] == ref[0], (name, burst)
        for f in ("x", "y", "z", "vx", "vy", "vz", "weight", "cell", "frequency"):
            np.testing.assert_array_equal(getattr(p, f), getattr(ref[1], f), err_msg=f"{name} burst {burst} {f}")

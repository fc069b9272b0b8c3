"""Which transports are followed by the fold of the attenuation sums."""
import pytest

from storm_b200 import _abi as A
from storm_b200.engine import Engine

from test_gpu_run_tally import _forms, _problem

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name,precision,folds", [
    ("gray", A.PRECISION_FP64, 1), ("gray", A.PRECISION_FP32_TRACK, 1), ("ddmc", A.PRECISION_FP32_TRACK, 1),
    ("ddmc", A.PRECISION_FP64, 0), ("voronoi_ddmc", A.PRECISION_FP64, 1), ("mg", A.PRECISION_FP64, 0),
    ("reproducible", A.PRECISION_FP64, 0), ("reproducible", A.PRECISION_FP32_TRACK, 0),
])
def test_fold_runs_only_where_a_transport_adds_to_it(name, precision, folds):
    if name == "reproducible":
        p = _problem(5, precision)
        p.reproducible_tallies = True
    else:
        p = {(f[0], f[1]): f[2] for f in _forms()}[name, precision]()
    p.per_cell_segment_counters = False   # they take a launch of their own
    e = Engine(p)
    for ph in ("begin", "prestep", "emit"):
        e.phase(ph, p.dt)
    before = e.launches()
    e.phase("transport")
    assert e.launches() - before == 1 + folds
    e.close()

"""The LRF accumulation beside the row build and behind it (the batch's rows of
all windows decide): one window, the last batch beside and the first behind
hold the same records and rows, and evaluate to the same bits."""
import numpy as np
import pytest

from q6_gb300.qnb import PREC_MIXED, NonbondedEngine
from q6_gb300.system import make_system

pytestmark = pytest.mark.gpu
CUT = dict(Rcq=99.0, RcLRF=99.0, Rcpp=6.0, Rcpw=5.0, Rcww=5.5)
LINE = 32768   # rows


def test_order_of_the_list_build():
    s = make_system(R=15.0, n_solute=20, nq=3, nstates=2, seed=18)
    first = -(-LINE // (s.ncgp_solute + s.nwat))
    out = []
    for w in (1, first - 1, first):
        with NonbondedEngine(s, precision=PREC_MIXED, windows=w) as e:
            e.set_lambda([0.5, 0.5])
            e.set_coordinates_dev(np.stack([s.x] * w))
            e.make_pair_lists_dev(**CUT)
            E, EQ, _ = e.compute_dev()
            d = e.gradient_dev()
            assert np.array_equal(d, np.stack([d[0]] * w)) and all(v == E[0] for v in E)
            out.append((e.lrf(), d[0], E[0], EQ[0], *e.export_rows(2)))
    for o in out[1:]:
        assert o[2] == out[0][2]
        for k in (0, 1, 3, 4, 5):
            assert np.array_equal(o[k], out[0][k]), k

"""The mixed form's LRF accumulation at the edges of its layout -- target
blocks of 64, source tiles of 16 groups, one to four blocks per cluster, large
groups in the tiles -- against the FP64 form's records, sphere and box: within
2e-5 of each coefficient order's scale (the mixed records' bar); and the order
of the list build (beside the rows for few rows, behind them for many) leaves
a window's records bit-equal."""
import numpy as np
import pytest

from q6_gb300.qnb import PREC_FP64, PREC_MIXED, NonbondedEngine
from q6_gb300.system import make_system

pytestmark = pytest.mark.gpu
CUT = dict(Rcq=9.0, RcLRF=9.5, Rcpp=6.0, Rcpw=5.0, Rcww=5.5)


def records(s, prec, box, cut):
    with NonbondedEngine(s, precision=prec) as e:
        if box:
            e.set_box([box] * 3)
        e.make_pair_lists(s.x, **cut)
        return e.lrf()


@pytest.mark.parametrize("R,n_solute,sizes", [(4.0, 5, (1, 2)), (6.5, 12, (3, 5)), (8.0, 120, (12, 15)),
                                              (9.0, 30, (3, 5)), (12.0, 60, (3, 6)), (16.0, 200, (3, 6))])
@pytest.mark.parametrize("box", [False, True])
def test_lrf_records_against_fp64(R, n_solute, sizes, box):
    s = make_system(R=R, n_solute=n_solute, group_sizes=sizes, nq=3, nstates=2, seed=17)
    L = max(2.0 * R + 8.0, 20.0)   # cut-offs within half the box
    cut = dict(CUT) if box else dict(CUT, RcLRF=99.0, Rcq=99.0)
    a, b = records(s, PREC_FP64, L if box else None, cut), records(s, PREC_MIXED, L if box else None, cut)
    assert a[:, 3].any()
    for k in (slice(0, 3), slice(3, 4), slice(4, 7), slice(7, 16), slice(16, 43)):
        assert np.abs(b[:, k] - a[:, k]).max() <= 2e-5 * np.abs(a[:, k]).max(), k


def test_lrf_beside_and_behind_the_rows_are_bit_equal():
    s = make_system(R=13.0, n_solute=20, nq=3, nstates=2, seed=18)
    W = 16384 // (s.ncgp_solute + s.nwat) + 1
    out = []
    for w in (1, W):
        with NonbondedEngine(s, precision=PREC_MIXED, windows=w) as e:
            e.set_coordinates_dev(np.stack([s.x] * w))
            e.make_pair_lists_dev(**dict(CUT, RcLRF=99.0, Rcq=99.0))
            out.append(e.lrf())
    assert np.array_equal(out[0], out[1])

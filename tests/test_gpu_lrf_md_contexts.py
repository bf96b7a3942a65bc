"""LRF records of the mixed form before and after qnb_md_init, whose contexts
keep another summation: against the FP64 form in the sphere and in a box, from
one source range to all eight, within 6e-6 of each coefficient order's scale
(per term about 4e-7 of rounding, and terms that cancel to about a tenth of
their sum); the two within twice that of each other at the same coordinates;
and the FP64 form's records unchanged by qnb_md_init."""
import numpy as np
import pytest

from q6_gb300.qnb import PREC_FP64, PREC_MIXED, NonbondedEngine
from q6_gb300.system import make_system

pytestmark = pytest.mark.gpu
BAR = 6e-6


def records(s, prec, box, cut):
    """Of lists built before qnb_md_init, and of the same lists built again after it."""
    with NonbondedEngine(s, precision=prec) as e:
        if box:
            e.set_box([box] * 3)
        e.make_pair_lists(s.x, **cut)
        a = e.lrf()
        e.md_init()
        e.make_pair_lists(s.x, **cut)
        return a, e.lrf()


@pytest.mark.parametrize("R,n_solute,sizes", [(6.5, 12, (3, 5)), (9.0, 60, (9, 15)), (12.0, 60, (3, 6)), (18.0, 60, (3, 6))])
@pytest.mark.parametrize("box", [False, True])
def test_records_before_and_after_md_init(R, n_solute, sizes, box):
    s = make_system(R=R, n_solute=n_solute, group_sizes=sizes, nq=3, nstates=2, seed=17)
    L = max(2.0 * R + 8.0, 20.0) if box else None
    far = 9.5 if box else 99.0
    cut = dict(Rcq=far, RcLRF=far, Rcpp=6.0, Rcpw=5.0, Rcww=5.5)
    a, a_md = records(s, PREC_FP64, L, cut)
    b, b_md = records(s, PREC_MIXED, L, cut)
    assert np.array_equal(a, a_md) and a[:, 3].any()
    for k in (slice(0, 3), slice(3, 4), slice(4, 7), slice(7, 16), slice(16, 43)):
        scale = np.abs(a[:, k]).max()
        assert np.abs(b[:, k] - a[:, k]).max() <= BAR * scale, k
        assert np.abs(b_md[:, k] - a[:, k]).max() <= BAR * scale, k
        assert np.abs(b_md[:, k] - b[:, k]).max() <= 2 * BAR * scale, k

"""FP32 rounding of the mixed form's LRF sums: both summations -- that of
contexts with an integrator and that of all others -- fold their FP32 sums
every eight source groups, so their distances from the FP64 form's records
(root mean square over a coefficient order) are the same up to the scatter of
two such samples.  All charges are positive, which makes the sums' own rounding
the largest part of it (a run twice as long would be off by about half as much
again); bar 1.15, the scatter of some 500 targets' records being about 5 %."""
import dataclasses

import numpy as np
import pytest

from q6_gb300.qnb import PREC_FP64, PREC_MIXED, NonbondedEngine
from q6_gb300.system import make_system

pytestmark = pytest.mark.gpu
CUT = dict(Rcq=99.0, RcLRF=99.0, Rcpp=4.0, Rcpw=4.0, Rcww=4.0)


def records(s, prec, md):
    with NonbondedEngine(s, precision=prec) as e:
        if md:
            e.md_init()
        e.make_pair_lists(s.x, **CUT)
        return e.lrf()


@pytest.mark.parametrize("R,n_solute,sizes", [(15.0, 60, (3, 5)), (15.0, 400, (4, 8))])
def test_rounding_of_both_summations(R, n_solute, sizes):
    s = make_system(R=R, n_solute=n_solute, group_sizes=sizes, nq=3, nstates=2, seed=19)
    s = dataclasses.replace(s, crg=np.abs(s.crg))
    a = records(s, PREC_FP64, False)
    b, c = records(s, PREC_MIXED, False), records(s, PREC_MIXED, True)
    for k in (slice(3, 4), slice(4, 7), slice(7, 16), slice(16, 43)):
        eb, ec = (np.sqrt(((v[:, k] - a[:, k]) ** 2).mean()) for v in (b, c))
        assert eb <= 1.15 * ec, (k, eb, ec)

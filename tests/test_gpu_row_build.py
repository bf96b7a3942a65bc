"""Solute rows at the edges of the 32 selected groups that are written together
-- one group, 31 to 33, 63 to 65, Q atoms inside groups, groups of Q atoms
only -- for the cell stencil, the periodic one and every-group candidates:
the pair counts equal the FP64 form's (another kernel), energies within 1e-3
relative, gradient within 2e-3 of max(|F|, median |F|) (the mixed form's
bars)."""
import numpy as np
import pytest

from q6_gb300.qnb import PREC_FP64, PREC_MIXED, NonbondedEngine
from q6_gb300.system import make_system

pytestmark = pytest.mark.gpu


def evaluate(s, prec, box, rc):
    cut = dict(Rcq=9.0, RcLRF=9.0, Rcpp=rc, Rcpw=rc, Rcww=rc)
    with NonbondedEngine(s, precision=prec, use_lrf=False) as e:
        if box:
            e.set_box([box] * 3)
        e.set_lambda(np.full(s.nstates, 1.0 / s.nstates))
        e.make_pair_lists(s.x, **cut)
        n = [e.list_size(k) for k in range(3)]
        d, E, EQ = e.pot_energy_nonbonds(s.x)
        return n, d, np.array(list(E.values())), EQ


@pytest.mark.parametrize("n_solute,sizes,nq,rc", [(3, (1, 1), 2, 9.0), (33, (1, 1), 1, 30.0), (34, (1, 1), 2, 30.0),
                                                  (36, (1, 1), 3, 30.0), (65, (1, 1), 1, 30.0), (67, (1, 1), 2, 30.0),
                                                  (150, (2, 4), 7, 6.0), (200, (9, 15), 5, 9.0)])
@pytest.mark.parametrize("box", [None, 28.0, 44.0])   # 28 with the long cut-offs: fewer than five cells, every group is a candidate
def test_row_build_against_fp64(n_solute, sizes, nq, rc, box):
    s = make_system(R=12.0, n_solute=n_solute, group_sizes=sizes, ntypes=5, nq=nq, nstates=2, seed=37,
                    type2_pairs=((0, 1),))
    if box:
        rc = min(rc, 13.0)
    (n0, d0, E0, EQ0), (n, d, E, EQ) = evaluate(s, PREC_FP64, box, rc), evaluate(s, PREC_MIXED, box, rc)
    assert n == n0
    assert np.all(np.abs(E - E0) <= 1e-3 * np.maximum(1.0, np.abs(E0)))
    assert np.all(np.abs(EQ - EQ0) <= 1e-3 * np.maximum(1.0, np.abs(EQ0)))
    assert np.all(np.abs(d - d0) <= 2e-3 * np.maximum(np.abs(d0), np.median(np.abs(d0))) + 1e-9)

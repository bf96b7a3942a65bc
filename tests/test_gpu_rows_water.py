"""Water rows of the mixed form at their edges -- no solute, no partners, one
partner more or less than a warp or than a prefetched chunk of 128, Q-only
groups, sphere and box, 3- and 4-site solvents -- against the FP64 form:
energies within 1e-3 relative, gradient within 2e-3 of max(|F|, median |F|)
(the mixed form's bars)."""
import dataclasses

import numpy as np
import pytest

from q6_gb300.qnb import PREC_FP64, PREC_MIXED, NonbondedEngine
from q6_gb300.system import make_system
from tests.test_gpu_fp64_pairs import four_site

pytestmark = pytest.mark.gpu


def evaluate(s, prec, box, rc):
    cut = dict(Rcq=9.0, RcLRF=9.0, Rcpp=rc, Rcpw=rc, Rcww=rc)
    with NonbondedEngine(s, precision=prec, use_lrf=False) as e:
        if box:
            e.set_box([box] * 3)
        e.set_lambda(np.full(max(1, s.nstates), 1.0 / max(1, s.nstates)))
        e.make_pair_lists(s.x, **cut)
        d, E, EQ = e.pot_energy_nonbonds(s.x)
        return d, np.array(list(E.values())), EQ


@pytest.mark.parametrize("R,n_solute,nq,rc", [(3.0, 0, 0, 9.0), (6.0, 7, 7, 2.0), (6.0, 12, 3, 5.0), (7.0, 60, 3, 6.5),
                                              (9.0, 200, 4, 9.0), (11.0, 12, 3, 9.9)])
@pytest.mark.parametrize("sites,box", [(3, False), (3, True), (4, False), (4, True)])
def test_water_rows_against_fp64(R, n_solute, nq, rc, sites, box):
    s = make_system(R=R, n_solute=n_solute, group_sizes=(3, 6), nq=nq, nstates=2, seed=23)
    if sites == 4:
        s = four_site(s)
    L = 2.0 * R + 14.0 if box else None
    (d0, E0, EQ0), (d, E, EQ) = evaluate(s, PREC_FP64, L, rc), evaluate(s, PREC_MIXED, L, rc)
    assert np.all(np.abs(E - E0) <= 1e-3 * np.maximum(1.0, np.abs(E0)))
    assert np.all(np.abs(EQ - EQ0) <= 1e-3 * np.maximum(1.0, np.abs(EQ0)))
    assert np.all(np.abs(d - d0) <= 2e-3 * np.maximum(np.abs(d0), np.median(np.abs(d0))) + 1e-9)

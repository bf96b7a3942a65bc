"""Mixed Q-environment kernels at their edges -- one atom or water to just past
a block of 64, Q atoms around the blocks of five whose gradients are summed
together, one to eight states, the largest water-parameter table (4-site
water, 40 Q atoms, 8 states), sphere and box -- against the FP64 form:
energies within 1e-3 relative, gradient within 2e-3 of max(|F|, median |F|)
(the mixed form's bars)."""
import numpy as np
import pytest

from q6_gb300.qnb import PREC_FP64, PREC_MIXED
from q6_gb300.system import make_system
from tests.test_gpu_fp64_pairs import four_site
from tests.test_gpu_rows_water import evaluate

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("R,n_solute,nq,nstates", [(4.0, 2, 1, 1), (7.0, 32, 5, 2), (9.0, 64, 6, 4), (9.0, 65, 4, 5),
                                                   (11.0, 129, 11, 8), (12.0, 80, 40, 8)])
@pytest.mark.parametrize("sites,box", [(3, False), (3, True), (4, False), (4, True)])
def test_q_lanes_against_fp64(R, n_solute, nq, nstates, sites, box):
    s = make_system(R=R, n_solute=n_solute, nq=nq, nstates=nstates, seed=31)
    if sites == 4:
        s = four_site(s)
    L = 2.0 * R + 14.0 if box else None
    (d0, E0, EQ0), (d, E, EQ) = evaluate(s, PREC_FP64, L, 6.0), evaluate(s, PREC_MIXED, L, 6.0)
    assert np.all(np.abs(EQ - EQ0) <= 1e-3 * np.maximum(1.0, np.abs(EQ0)))
    assert np.all(np.abs(d - d0) <= 2e-3 * np.maximum(np.abs(d0), np.median(np.abs(d0))) + 1e-9)

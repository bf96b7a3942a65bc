"""Solute rows of the mixed form at their edges -- group sizes from one atom to
the largest of each compiled size (odd ones included), Q atoms inside groups,
rows around a prefetched chunk of 128 plain and special entries, type-2 LJ
pairs, the arithmetic rule, sphere and box -- against the FP64 form: energies
within 1e-3 relative, gradient within 2e-3 of max(|F|, median |F|) (the mixed
form's bars)."""
import copy

import numpy as np
import pytest

from q6_gb300.system import make_system
from tests.test_gpu_rows_water import evaluate
from q6_gb300.qnb import PREC_FP64, PREC_MIXED

pytestmark = pytest.mark.gpu


def arithmetic(s):
    """The same system under the arithmetic rule, with LJ factors of its kind (sigma / 2, sqrt epsilon)."""
    s = copy.deepcopy(s)
    rng = np.random.default_rng(3)
    s.ivdw_rule = 2
    for a, b in ((s.avdw, s.bvdw), (s.qavdw, s.qbvdw)):
        a[:] = rng.uniform(0.6, 1.4, a.shape[0])[:, None]
        b[:] = rng.uniform(0.1, 0.4, b.shape[0])[:, None]
    return s


@pytest.mark.parametrize("sizes,n_solute,rc", [((1, 1), 40, 6.0), ((2, 3), 90, 7.0), ((4, 4), 300, 9.0), ((5, 6), 330, 9.0),
                                               ((7, 8), 200, 8.0), ((9, 15), 260, 9.0)])
@pytest.mark.parametrize("rule,box", [(1, False), (1, True), (2, False), (2, True)])
def test_solute_rows_against_fp64(sizes, n_solute, rc, rule, box):
    s = make_system(R=12.0, n_solute=n_solute, group_sizes=sizes, ntypes=5, nq=3, nstates=2, seed=29,
                    type2_pairs=((0, 1), (2, 2)))
    if rule == 2:
        s = arithmetic(s)
    L = 38.0 if box else None
    (d0, E0, EQ0), (d, E, EQ) = evaluate(s, PREC_FP64, L, rc), evaluate(s, PREC_MIXED, L, rc)
    assert np.all(np.abs(E - E0) <= 1e-3 * np.maximum(1.0, np.abs(E0)))
    assert np.all(np.abs(EQ - EQ0) <= 1e-3 * np.maximum(1.0, np.abs(EQ0)))
    assert np.all(np.abs(d - d0) <= 2e-3 * np.maximum(np.abs(d0), np.median(np.abs(d0))) + 1e-9)

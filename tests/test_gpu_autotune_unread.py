"""The autotuner leaves the values that no kernel reads (the Q chunk, the LRF
accumulation) as the caller set them."""
import pytest

from q6_gb300.qnb import PREC_MIXED, TUNE_NAMES, NonbondedEngine
from q6_gb300.system import default_solvent_params, make_system

pytestmark = pytest.mark.gpu


def test_unread_values_are_kept():
    s = make_system(R=8.0, n_solute=20, nq=3, nstates=2, seed=6)
    with NonbondedEngine(s, precision=PREC_MIXED) as e:
        e.set_solvent_params(default_solvent_params(s))
        e.set_lambda([0.5, 0.5])
        e.make_pair_lists(s.x, Rcpp=6.0, Rcpw=6.0, Rcww=6.0)
        t = e.tuning()
        t.update({TUNE_NAMES[4]: 13, TUNE_NAMES[6]: 7})   # no candidate of any search
        e.set_tuning(t)
        out = e.autotune(reps=1)
        assert out[TUNE_NAMES[4]] == 13 and out[TUNE_NAMES[6]] == 7
        assert e.tuning() == out

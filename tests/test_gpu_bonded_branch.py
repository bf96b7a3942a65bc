"""The bonded terms' branch (none without bonded terms; behind the kernel that
puts the excluded atoms back under excluded_freeze): with the branches on and
off, replayed and kernel by kernel, the mixed form's energies and gradients
are the same bits, and the FP64 form's agree to the rounding of their atomic
sums: at most 1e5 terms whose magnitudes sum to at most 100 times the largest
result, 1e5 * 100 * 1.1e-16 = 1e-9 of it."""
import numpy as np
import pytest

from q6_gb300.bonded import synthetic_bonded
from q6_gb300.md import make_shell
from q6_gb300.qnb import PREC_FP64, PREC_MIXED, NonbondedEngine
from q6_gb300.system import config_small, default_solvent_params

pytestmark = pytest.mark.gpu
CUT = dict(Rcq=99.0, RcLRF=99.0, Rcpp=10.0, Rcpw=10.0, Rcww=10.0)


def run(s, prec, bonded, freeze, branches, graphs):
    out = []
    with NonbondedEngine(s, precision=prec, windows=2) as e:
        e.set_solvent_params(default_solvent_params(s, itdis=2.0))
        e.set_concurrency(branches)
        e.set_graphs(graphs)
        for w in range(2):
            e.set_lambda([0.3 + 0.4 * w, 0.7 - 0.4 * w], window=w)
        if bonded:
            e.set_bonded(synthetic_bonded(s, seed=5))
        if freeze:
            e.set_shell_restraint(s.x, make_shell(s, 0.85))
            e.set_freeze(True)
        e.set_coordinates_dev(np.stack([s.x, s.x + 0.01]))
        e.make_pair_lists_dev(**CUT)
        for k in range(3):
            E, EQ, R = e.compute_dev(Tfree=300.0, istep=k, sync=True)
            out += [np.array([list(v.values()) for v in E]), EQ.copy(), R.copy(), e.gradient_dev()]
        if bonded:
            out += [np.array(v) for v in e.bonded_energies()]
    return out


@pytest.mark.parametrize("prec", [PREC_MIXED, PREC_FP64])
@pytest.mark.parametrize("bonded,freeze", [(True, False), (True, True), (False, False)])
def test_bonded_branch(prec, bonded, freeze):
    s = config_small()
    ref = run(s, prec, bonded, freeze, False, False)
    for graphs in (True, False):
        for a, b in zip(ref, run(s, prec, bonded, freeze, True, graphs)):
            if prec == PREC_MIXED:
                assert np.array_equal(a, b)
            else:
                assert np.all(np.abs(a - b) <= 1e-9 * max(1.0, np.abs(a).max()))

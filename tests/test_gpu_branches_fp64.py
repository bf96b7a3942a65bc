"""The FP64 form's evaluation branches (qnb_set_concurrency): its sums are FP64
atomics, so a run with the branches on agrees with the single-stream run to
rounding.  With 10^5 terms per sum, each within 2^-53 of its operands, the two
orders differ by at most 1e5 * 2^-53 = 1.1e-11 of the sum of magnitudes; the
bars use the largest energy term and gradient component for that scale."""
import numpy as np
import pytest

from q6_gb300.qnb import PREC_FP64, NonbondedEngine
from q6_gb300.system import config_small, default_solvent_params, lambdas_for_window

pytestmark = pytest.mark.gpu
CUT = dict(Rcq=99.0, RcLRF=99.0, Rcpp=10.0, Rcpw=10.0, Rcww=10.0)


@pytest.mark.parametrize("graphs", [True, False])
def test_fp64_branches_agree_with_single_stream(graphs):
    s, W, out = config_small(), 2, []
    xs = np.stack([s.x + np.random.default_rng(8 + w).normal(0.0, 0.02, s.x.shape) for w in range(W)])
    for branches in (True, False):
        with NonbondedEngine(s, precision=PREC_FP64, windows=W) as e:
            e.set_solvent_params(default_solvent_params(s))
            e.set_concurrency(branches)
            e.set_graphs(graphs)
            for w in range(W):
                e.set_lambda(lambdas_for_window(0.3 + 0.4 * w, s.nstates), window=w)
            e.set_coordinates_dev(xs)
            e.make_pair_lists_dev(**CUT)
            E, EQ, R = e.compute_dev(Tfree=300.0, istep=1, sync=True)
            out.append((np.array([list(v.values()) for v in E]), EQ, R, e.gradient_dev()))
    for a, b in zip(*out):
        assert np.abs(a - b).max() <= 1.1e-11 * np.abs(b).max()

"""Adjoint kernels at the edges of their lane layout (Q atoms around the powers
of two up to 32 and in two rounds of 32) and with soft-core alphas that some
states share and others do not, against the FP64 reference gradient within
1e-9 of it (the bar of the config-4 test: sums of 10^4 terms in another
order)."""
import numpy as np
import pytest

from oracle.adjoint import QEnergyReference
from q6_gb300.qnb import PREC_MIXED, NonbondedEngine
from q6_gb300.system import make_system

pytestmark = pytest.mark.gpu
CUT = dict(Rcq=99.0, RcLRF=99.0, Rcpp=10.0, Rcpw=10.0, Rcww=10.0)


@pytest.mark.parametrize("nq,nstates", [(1, 1), (2, 5), (3, 2), (8, 4), (9, 2), (17, 3), (32, 2), (33, 2), (64, 4)])
def test_adjoint_lane_edges(nq, nstates):
    s = make_system(R=12.0, n_solute=max(nq + 12, 20), nq=nq, nstates=nstates, seed=70 + nq)
    rng = np.random.default_rng(nq)
    s.sc_lookup[:, : s.natyps, :] = rng.choice([0.0, 0.4, 0.7], size=(nq, 1, nstates))
    with NonbondedEngine(s, precision=PREC_MIXED) as e:
        e.set_coordinates_dev(s.x[None])
        e.make_pair_lists_dev(**CUT)
        got = e.q_adjoint_dev()
    for g, r in zip(got, QEnergyReference(s).evaluate(s.x)[1:]):
        assert np.all(np.abs(g[0] - r) <= 1e-9 * np.maximum(np.abs(r), 1e-3 * np.abs(r).max()))

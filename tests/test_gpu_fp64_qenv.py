"""FP64 Q-environment kernels at the edges of their blocks of five Q atoms, up
to five states, soft-core alphas that some states share and others do not,
against the oracle (sphere) and the numpy restatement (box): the FP64 form's
bars, 1e-6 kcal/mol per energy and 1e-6 relative per gradient component."""
import numpy as np
import pytest

from oracle.oracle import Oracle
from q6_gb300.qnb import PREC_FP64, NonbondedEngine
from q6_gb300.system import make_system

pytestmark = pytest.mark.gpu
CUT = dict(Rcq=99.0, RcLRF=99.0, Rcpp=8.0, Rcpw=8.0, Rcww=8.0)


def system(nq, nstates):
    s = make_system(R=9.0, n_solute=24, nq=nq, nstates=nstates, seed=40 + nq)
    s.sc_lookup[:, : s.natyps, :] = np.random.default_rng(nq).choice([0.0, 0.5, 0.5], size=(nq, 1, nstates))
    return s


def ok(d, d0):
    return np.all(np.abs(d - d0) <= 1e-6 * np.maximum(np.abs(d0), np.median(np.abs(d0))) + 1e-9)


@pytest.mark.parametrize("nq,nstates", [(1, 1), (4, 2), (5, 3), (6, 4), (11, 5)])
def test_fp64_q_environment(nq, nstates):
    s, lam = system(nq, nstates), np.full(nstates, 1.0 / nstates)
    o = Oracle(s)
    o.set_lambda(lam)
    o.make_pair_lists(s.x, **CUT)
    d0, _, EQ0 = o.pot_energy_nonbonds(s.x)
    with NonbondedEngine(s, precision=PREC_FP64) as e:
        e.set_lambda(lam)
        e.make_pair_lists(s.x, **CUT)
        d, _, EQ = e.pot_energy_nonbonds(s.x)
    assert np.all(np.abs(EQ - EQ0) <= 1e-6) and ok(d, d0)


@pytest.mark.parametrize("nq,nstates", [(4, 1), (6, 5)])
def test_fp64_q_environment_box(nq, nstates):
    from oracle.box import box_energies, box_lists
    s, lam, L = system(nq, nstates), np.full(nstates, 1.0 / nstates), np.full(3, 21.0)
    cut = dict(CUT, RcLRF=8.0, Rcq=9.0)
    qs = int(s.iqseq[0])
    lists = box_lists(s, s.x, L, qs, cut)
    d0, _, EQ0 = box_energies(s, s.x, lam, L, qs, cut, lists)
    with NonbondedEngine(s, precision=PREC_FP64, use_lrf=False) as e:
        e.set_box(L, qs)
        e.set_lambda(lam)
        e.make_pair_lists(s.x, **cut)
        d, _, EQ = e.pot_energy_nonbonds(s.x)
    assert np.all(np.abs(EQ[:, 2:] - EQ0[:, 2:]) <= 1e-6) and ok(d, d0)

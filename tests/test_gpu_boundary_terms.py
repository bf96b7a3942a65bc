"""The step's boundary terms (radial restraint with watpol's angles, then rank,
force and averages in one kernel) against the oracle over several steps and an
update: shells from a few waters to more than one block's rounds, both forms;
then watpol without md on the last call's order.  FP64 form: 1e-6 kcal/mol and
1e-6 relative per gradient component; mixed form: 1e-3 and 2e-3 (the forms'
bars); running averages within 1e-9 and 1e-5."""
import numpy as np
import pytest

from oracle.oracle import Oracle
from q6_gb300.qnb import PREC_FP64, PREC_MIXED, NonbondedEngine
from q6_gb300.system import default_solvent_params, make_system

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec,bar,gbar,abar", [(PREC_FP64, 1e-6, 1e-6, 1e-9), (PREC_MIXED, 1e-3, 2e-3, 1e-5)])
@pytest.mark.parametrize("R,nlayer", [(4.0, 0.5), (9.0, 3.0001), (18.0, 6.0)])
def test_boundary_terms(prec, bar, gbar, abar, R, nlayer):
    s = make_system(R=R, n_solute=6, nq=2, nstates=1, seed=33)
    sp = default_solvent_params(s, itdis=3.0, wpolr_layer=nlayer)
    cut = dict(Rcq=99.0, RcLRF=99.0, Rcpp=3.0, Rcpw=3.0, Rcww=3.0)
    rng = np.random.default_rng(4)
    o = Oracle(s, use_lrf=False)
    o.set_solvent_params(sp)
    o.set_lambda([1.0])
    with NonbondedEngine(s, precision=prec, use_lrf=False) as e:
        e.set_solvent_params(sp)
        e.set_lambda([1.0])
        o.make_pair_lists(s.x, **cut)
        e.make_pair_lists(s.x, **cut)
        for k in range(1, 6):
            x = s.x + rng.normal(0.0, 0.05, s.x.shape)
            d0, _, EQ = o.pot_energy_nonbonds(x)
            d0, _ = o.nonbond_qq(x, d0, EQ)
            r0 = [o.restrain_solvent(x, d0, 300.0), o.watpol(x, d0, k, True)]
            d, _, _, r = e.pot_energy_step(x, Tfree=300.0, istep=k)
            assert np.all(np.abs(r - r0) <= bar * np.maximum(1.0, np.abs(r0))), k
            assert np.all(np.abs(d - d0) <= gbar * np.maximum(np.abs(d0), np.median(np.abs(d0))) + 1e-9), k
            for a, b in zip(e.watpol_state(), o.watpol_state()):
                assert np.allclose(a, b, rtol=abar, atol=abar), k
        d0, d = np.zeros_like(x), np.zeros_like(x)
        x = x + rng.normal(0.0, 0.001, x.shape)
        assert abs(e.watpol(x, d, 7, md=False) - o.watpol(x, d0, 7, False)) <= max(bar, 0.05)

"""Water polarisation restraint in shells of more waters than the ranking
kernel stages at a time (1,024) and than its blocks have threads (2,048),
against the oracle over several steps and an update; then watpol without md,
energy and gradient, on the last call's order.

FP64 form: 1e-6 kcal/mol relative per energy and 1e-6 per gradient component.
Mixed form: 1e-3 and 2e-3; two waters whose angles agree to FP32 rounding may
take each other's rank, which moves their target angles by about 4/n (n
waters) and their forces by fkwpol 4/n (2/|dipole| + 1/r) <= 20 * 4/n * 1.9,
allowed on top.  Running averages within 1e-9 and 1e-5."""
import numpy as np
import pytest

from oracle.oracle import Oracle
from q6_gb300.qnb import PREC_FP64, PREC_MIXED, NonbondedEngine
from q6_gb300.system import default_solvent_params, make_system

pytestmark = pytest.mark.gpu
CUT = dict(Rcq=99.0, RcLRF=99.0, Rcpp=3.0, Rcpw=3.0, Rcww=3.0)


def close(a, b, bar, extra=0.0):
    return np.all(np.abs(a - b) <= bar * np.maximum(np.abs(b), np.median(np.abs(b))) + 1e-9 + extra)


@pytest.mark.parametrize("prec,bar,gbar,abar", [(PREC_FP64, 1e-6, 1e-6, 1e-9), (PREC_MIXED, 1e-3, 2e-3, 1e-5)])
@pytest.mark.parametrize("R,drout,least", [(9.0, 0.5, 0), (22.0, 9.0, 1025), (27.0, 14.0, 2049)])
def test_large_shells(prec, bar, gbar, abar, R, drout, least):
    s = make_system(R=R, n_solute=6, nq=2, nstates=1, seed=33)
    sp = default_solvent_params(s, itdis=2.0, drout=drout, wpolr_layer=drout + 0.5 if least else 3.0001)
    r = np.linalg.norm(s.x[s.nat_solute::3] - s.xwcent, axis=1)
    n = max(int(((r <= sp.shell_rout[k]) & (r > sp.shell_rout[k] - sp.shell_dr[k])).sum()) for k in range(sp.nwpolr_shell))
    assert n >= least
    swap = 0.0 if prec == PREC_FP64 else 20.0 * 4.0 / n * 1.9
    rng = np.random.default_rng(4)
    o = Oracle(s, use_lrf=False)
    o.set_solvent_params(sp)
    with NonbondedEngine(s, precision=prec, use_lrf=False) as e:
        e.set_solvent_params(sp)
        for k in range(1, 4):
            x = s.x + rng.normal(0.0, 0.02, s.x.shape)
            d, d0 = np.zeros_like(x), np.zeros_like(x)
            E, E0 = e.watpol(x, d, k, md=True), o.watpol(x, d0, k, True)
            assert abs(E - E0) <= bar * max(1.0, abs(E0)), (k, E, E0)
            assert close(d, d0, gbar, swap), k
            for a, b in zip(e.watpol_state(), o.watpol_state()):
                assert np.allclose(a, b, rtol=abar, atol=abar), k
        x = x + rng.normal(0.0, 0.001, x.shape)
        d, d0 = np.zeros_like(x), np.zeros_like(x)
        E, E0 = e.watpol(x, d, 7, md=False), o.watpol(x, d0, 7, False)
        assert d.any()
        assert abs(E - E0) <= bar * max(1.0, abs(E0)), (E, E0)
        assert close(d, d0, gbar, swap)
        for a, b in zip(e.watpol_state(), o.watpol_state()):
            assert np.allclose(a, b, rtol=abar, atol=abar)

"""MD step of systems whose constrained molecules are all rigid 3-site waters
(SHAKE in registers, fused with newvel and the velocity update) against the
oracle's strict-IEEE step, FP64 form: sizes around the kernels' blocks of 32
molecules and 128 atoms, with and without free solute atoms.  Bars as for the
general molecules: given the same gradient the integrator is bit-equal, and
the gradients differ by the order of their sums (1e-9 relative); the SHAKE
sweeps are equal as counts."""
import dataclasses

import numpy as np
import pytest

from oracle.oracle import Oracle, OracleMD
from q6_gb300.md import MdSetup, build_constraints, maxwell_velocities, md_params
from q6_gb300.qnb import PREC_FP64, NonbondedEngine
from q6_gb300.system import default_solvent_params, make_system

pytestmark = pytest.mark.gpu
CUT = dict(Rcq=99.0, RcLRF=99.0, Rcpp=10.0, Rcpw=10.0, Rcww=10.0)


@pytest.mark.parametrize("R,n_solute,sep", [(5.0, 6, True), (9.0, 12, False), (11.0, 33, True)])
def test_triangle_step_matches_oracle(R, n_solute, sep):
    s = make_system(R=R, n_solute=n_solute, nq=4, nstates=2, seed=61)
    setup = MdSetup(stepsize=1.0, temp0=300.0, tau_t=50.0, nbcycle=4, separate_scaling=sep, cut=CUT)
    sp, lam, n = default_solvent_params(s, itdis=4.0), [0.6, 0.4], 6
    v0 = maxwell_velocities(s, 300.0, 11)
    with NonbondedEngine(s, precision=PREC_FP64) as e:
        e.set_solvent_params(sp)
        e.set_lambda(lam)
        e.set_coordinates_dev(s.x[None])
        e.md_init(setup)
        e.md_set_velocities(v0)
        e.md_prepare(stop_cm=True)
        rec, EQ, _ = e.md_run(n)
        xd, vd = e.md_state(0)
    o = Oracle(s)
    o.set_solvent_params(sp)
    cons = build_constraints(s, setup)
    md = OracleMD(o, md_params(s, setup, cons), cons, sp=sp, lam=lam)
    x, v = md.prepare(s.x, v0)
    for k in range(n):
        r = md.step(x, v, k, CUT)
        for key in ("ekin", "temp", "tfree"):
            assert abs(rec[k, 0][key] - r[key]) <= 1e-9 * abs(r[key]), (k, key)
        assert rec[k, 0]["shake_iterations"] == r["shake_iterations"], k
        assert np.allclose(EQ[k, 0], r["EQ"], rtol=1e-9, atol=1e-9), k
    assert np.allclose(xd, x, rtol=0, atol=1e-9)
    assert np.allclose(vd, v, rtol=1e-8, atol=1e-10)


def test_an_impossible_triangle_fails():
    s = make_system(R=8.0, n_solute=6, nq=4, nstates=2, seed=61)
    from q6_gb300 import md as qmd
    setup = MdSetup(stepsize=1.0, cut=CUT)
    cons = qmd.build_constraints(s, setup)
    cons = dataclasses.replace(cons, dist=np.where(np.arange(len(cons.dist)) == 5, 3.0, cons.dist))
    import ctypes
    from q6_gb300.qnb import _p
    with NonbondedEngine(s, precision=PREC_FP64) as e:
        e.set_solvent_params(default_solvent_params(s))
        e.set_coordinates_dev(s.x[None])
        p = md_params(s, setup, cons)
        mass = np.ascontiguousarray(s.mass[s.iac], dtype=np.float64)
        ij = np.ascontiguousarray(cons.ij, dtype=np.int32)
        d = np.ascontiguousarray(cons.dist)
        assert e.lib.qnb_md_init(e.h, ctypes.byref(p), _p(mass), len(cons.mol_first) - 1, _p(cons.mol_first), _p(ij),
                                 _p(d)) == 0
        assert e.lib.qnb_md_prepare(e.h, 1) == 7   # QNB_ERR_CONSTRAINT
        assert b"molecule 1" in e.lib.qnb_last_error()

"""qnb_pot_energy_step with its host transfers in the step's graph: bit-equal
(mixed form) to the kernel-by-kernel run and to a batched context's
evaluation, over steps with other coordinates, other Tfree, rebuilt lists and
watpol's update step; the gradient is added to the caller's and cleared
between steps."""
import numpy as np
import pytest

from q6_gb300.qnb import PREC_MIXED, NonbondedEngine
from q6_gb300.system import default_solvent_params, make_system

pytestmark = pytest.mark.gpu
CUT = dict(Rcq=99.0, RcLRF=99.0, Rcpp=8.0, Rcpw=8.0, Rcww=8.0)


@pytest.mark.parametrize("R,n_solute", [(5.0, 6), (10.0, 41)])
def test_host_step_graph(R, n_solute):
    s = make_system(R=R, n_solute=n_solute, nq=3, nstates=2, seed=12)
    sp = default_solvent_params(s, itdis=3.0)
    rng = np.random.default_rng(1)
    xs = [s.x + rng.normal(0.0, 0.02, s.x.shape) for _ in range(7)]
    out = []
    for mode in ("graph", "direct", "device"):
        res = []
        with NonbondedEngine(s, precision=PREC_MIXED) as e:
            e.set_graphs(mode != "direct")
            e.set_solvent_params(sp)
            e.set_lambda([0.3, 0.7])
            e.make_pair_lists(xs[0], **CUT)
            for k, x in enumerate(xs):
                if k == 4:
                    e.make_pair_lists(x, **CUT)
                T = 300.0 if k < 5 else 310.0
                if mode == "device":
                    e.set_coordinates_dev(x[None])
                    E, EQ, R2 = e.compute_dev(Tfree=T, istep=k)
                    res.append((e.gradient_dev()[0], list(E[0].values()), EQ[0], R2[0]))
                else:
                    d0 = np.full(s.x.shape, 0.5)
                    d, E, EQ, R2 = e.pot_energy_step(x, d0, Tfree=T, istep=k)
                    res.append((d - 0.5, list(E.values()), EQ, R2))
        out.append(res)
    for a, b, c in zip(*out):
        for u, v, w in zip(a, b, c):
            assert np.array_equal(u, v)
            assert np.allclose(u, w, rtol=0, atol=2e-13 * max(1.0, np.abs(w).max()))   # (the 0.5 added and taken off)

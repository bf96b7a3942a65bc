"""FP64 Q-environment kernels with one to five Q atoms per warp (the number of
windows decides: all windows' warps are kept to eight per SM) against the
oracle, sphere, and against the numpy restatement, box: every window has
coordinates of its own and is compared; 1e-6 kcal/mol per energy and 1e-6
relative per gradient component, the FP64 form's bars."""
import numpy as np
import pytest

from oracle.box import box_energies, box_lists
from oracle.oracle import Oracle
from q6_gb300.qnb import PREC_FP64, NonbondedEngine
from q6_gb300.system import make_system

pytestmark = pytest.mark.gpu
CUT = dict(Rcq=99.0, RcLRF=99.0, Rcpp=8.0, Rcpw=8.0, Rcww=8.0)


def ok(d, d0):
    return np.all(np.abs(d - d0) <= 1e-6 * np.maximum(np.abs(d0), np.median(np.abs(d0))) + 1e-9)


def run(s, xs, lam, windows, box, cut):
    """The evaluation of `windows` windows that hold the coordinates xs in turn."""
    with NonbondedEngine(s, precision=PREC_FP64, windows=windows, use_lrf=box is None) as e:
        if box is not None:
            e.set_box(box, int(s.iqseq[0]))
        e.set_lambda(lam)
        e.set_coordinates_dev(np.stack([xs[w % len(xs)] for w in range(windows)]))
        e.make_pair_lists_dev(**cut)
        _, EQ, _ = e.compute_dev()
        return EQ, e.gradient_dev()


@pytest.mark.parametrize("box", [False, True])
@pytest.mark.parametrize("nq,nstates,windows", [(11, 2, w) for w in (1, 37, 50, 90, 130, 200)] + [(5, 5, 1), (5, 5, 300)])
def test_q_blocks(nq, nstates, windows, box):
    s, lam = make_system(R=9.0, n_solute=24, nq=nq, nstates=nstates, seed=51), np.full(nstates, 1.0 / nstates)
    rng = np.random.default_rng(2)
    xs = [s.x + rng.normal(0.0, 0.02, s.x.shape) for _ in range(3)]
    L, qs = np.full(3, 21.0), int(s.iqseq[0])
    cut = dict(CUT, RcLRF=8.0, Rcq=9.0) if box else CUT
    want = []
    for x in xs:
        if box:
            d0, _, EQ0 = box_energies(s, x, lam, L, qs, cut, box_lists(s, x, L, qs, cut))
        else:
            o = Oracle(s)
            o.set_lambda(lam)
            o.make_pair_lists(x, **cut)
            d0, _, EQ0 = o.pot_energy_nonbonds(x)
        o = Oracle(s, use_lrf=False)
        o.set_lambda(lam)
        EQ0 = np.array(EQ0)
        EQ0[:, :2] = 0.0
        d0, EQ0 = o.nonbond_qq(x, d0, EQ0)
        want.append((EQ0, d0))
    EQ, d = run(s, xs, lam, windows, L if box else None, cut)
    for w in range(windows):
        EQ0, d0 = want[w % 3]
        assert np.all(np.abs(EQ[w] - EQ0) <= 1e-6) and ok(d[w], d0), w

"""Rounding of the FP64 form's pair terms: 1/r and 1/r^2 as good as a correctly
rounded division and square root give them.  One pair per window at random
distances; every energy, gradient component and LRF coefficient against
quad- or 80-bit arithmetic on the same squared distance and parameters, as a
root mean square relative error, which may be at most 1.15 times that of the
same terms taken in FP64 from 1/r^2 by division and 1/r by its square root
(1,024 pairs: the ratio of two such estimates scatters by about 4 %)."""
import dataclasses

import numpy as np
import pytest

from q6_gb300.qnb import PREC_FP64, NonbondedEngine
from q6_gb300.system import make_system

pytestmark = pytest.mark.gpu
L = np.longdouble
BAR = 1.15


def pair(q_atom):
    """Two atoms in groups of their own; the first a Q atom or not.  Repulsive LJ term only."""
    s = make_system(R=4.0, n_solute=2, group_sizes=(1, 1), nq=1, nstates=1, seed=3)
    none = np.zeros((0, 2), np.int32)
    s = dataclasses.replace(s, natom=2, nwat=0, x=s.x[:2], crg=np.array([7.31, -5.17]), iac=s.iac[:2], excl=s.excl[:2] * 0,
                            heavy=s.heavy[:2], cgp_first=s.cgp_first[:2], cgp_last=s.cgp_last[:2],
                            cgp_iswitch=s.cgp_iswitch[:2], cgpatom=s.cgpatom[:2], excl_pairs=none, rexcl_o=1.0e3,
                            qcrg=np.array([[6.83]]), sc_lookup=s.sc_lookup * 0.0, qconn=np.full_like(s.qconn, 9),
                            ljcod=np.ones_like(s.ljcod))
    s.qconn[:, 0] = 1   # the Q atom itself
    s.bvdw[:] = 0.0
    s.qbvdw[:] = 0.0
    if not q_atom:
        s = dataclasses.replace(s, nqat=0, iqseq=s.iqseq[:0], qcrg=s.qcrg[:0], qiac=s.qiac[:0], sc_lookup=s.sc_lookup[:0, : s.natyps],
                                qconn=s.qconn[:, :, :0])
    return s


def positions(s, n, seed):
    rng = np.random.default_rng(seed)
    u = rng.normal(size=(n, 3))
    d = np.exp(rng.uniform(np.log(1.0), np.log(30.0), (n, 1))) * u / np.linalg.norm(u, axis=1, keepdims=True)
    a = rng.normal(0.0, 3.0, (n, 3))
    return np.stack([a, a + d], 1)


def inverses(t, exact):
    """1/r and 1/r^2 of the squared length the kernels form (one rounding per term)."""
    f = lambda a, c: (L(a) * a + c).astype(np.float64)
    d2 = f(t[:, 2], f(t[:, 0], t[:, 1] * t[:, 1]))
    if exact:
        r2 = 1 / L(d2)
    else:
        r2 = 1.0 / d2
    return np.sqrt(r2), r2


def rms(a, b, scale):
    return float(np.sqrt((((a - b) / scale).astype(np.float64) ** 2).mean()))


@pytest.mark.parametrize("q_atom", [False, True])
def test_pair_terms(q_atom):
    s = pair(q_atom)
    W, rounds = 256, 4
    x = positions(s, W * rounds, 5)
    got = []
    with NonbondedEngine(s, precision=PREC_FP64, use_lrf=False, windows=W) as e:
        e.set_lambda([1.0])
        for k in range(rounds):
            e.set_coordinates_dev(x[k * W:(k + 1) * W])
            e.make_pair_lists_dev(Rcpp=99.0)
            E, EQ, _ = e.compute_dev()
            g = e.gradient_dev()
            v = EQ[:, 0, 2:4] if q_atom else np.array([[w["pp_el"], w["pp_vdw"]] for w in E])
            got.append(np.concatenate([v, g[:, 1]], 1))
    got = np.concatenate(got)
    j = x[:, 1] - x[:, 0]
    ti, tj = s.iac
    A = (s.qavdw[0, 0] if q_atom else s.avdw[ti, 0]) * s.avdw[tj, 0]
    el = (6.83 if q_atom else 7.31) * -5.17

    def terms(exact):
        r, r2 = inverses(j, exact)
        r6 = r2 * r2 * r2
        vel, va = el * r, A * (r6 * r6)
        dv = r2 * (-vel - 12 * va)
        return np.stack([vel, va, *(j[:, c] * dv for c in range(3))], 1)
    ex, plain = terms(True), terms(False)
    for c in (slice(0, 1), slice(1, 2), slice(2, 5)):
        a, b = (rms(v[:, c], ex[:, c], ex[:, c]) for v in (got, plain))
        assert a <= BAR * b, (c, a, b)


def test_lrf_records():
    s = pair(False)
    n = 1024
    x = positions(s, n, 6)
    got = np.zeros((n, 2, 40))
    with NonbondedEngine(s, precision=PREC_FP64) as e:
        for k in range(n):
            e.make_pair_lists(x[k], Rcpp=0.1)
            got[k] = e.lrf()[:, 3:]
    delta = np.eye(3)
    errs = {"got": [], "plain": []}
    for g in range(2):
        t, q = x[:, 1 - g] - x[:, g], s.crg[1 - g]

        def record(exact):
            _, r2 = inverses(t, exact)
            d2 = 1 / r2 if exact else inverses(t, True)[1] ** -1
            d2 = d2 if exact else d2.astype(np.float64)
            f0 = q / (d2 * np.sqrt(d2))
            d = t.astype(f0.dtype)
            f1 = 3 * f0 * r2
            S2 = f1[:, None, None] * d[:, :, None] * d[:, None, :] - f0[:, None, None] * delta
            h = 5 * f1 * r2
            U = f1[:, None] * d
            S3 = -h[:, None, None, None] * d[:, :, None, None] * d[:, None, :, None] * d[:, None, None, :]
            S3 = S3 + U[:, None, None, :] * delta[:, :, None] + U[:, None, :, None] * delta[:, None, :] \
                + U[:, :, None, None] * delta[None, :, :]
            return np.concatenate([(f0 * d2)[:, None], -f0[:, None] * d, S2.reshape(n, 9), S3.reshape(n, 27)], 1)
        ex, plain = record(True), record(False)
        r = np.sqrt((t * t).sum(1))[:, None]
        scale = np.abs(q) * np.concatenate([r ** -1, np.repeat(r ** -2, 3, 1), np.repeat(r ** -3, 9, 1), np.repeat(r ** -4, 27, 1)], 1)
        for name, v in (("got", got[:, g]), ("plain", plain)):
            errs[name].append(((v - ex) / scale).astype(np.float64))
    for c in (slice(0, 1), slice(1, 4), slice(4, 13), slice(13, 40)):
        a, b = (float(np.sqrt((np.concatenate(errs[k])[:, c] ** 2).mean())) for k in ("got", "plain"))
        assert a <= BAR * b, (c, a, b)

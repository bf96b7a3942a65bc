"""The mixed form's rows and Q-environment terms against the FP64 form at bars
near their rounding.  The coordinates are multiples of 2^-18 A and the boxes
whole numbers, so that they and their differences are exact in FP32 and what
remains is the arithmetic: per pair term about 3e-7 (the powers of a reciprocal
square root of 2^-22.9 at most, a dozen roundings), random in sign.

Gradient: root mean square within 1e-5 of the gradients' own (forces that
cancel to a fifth, with a factor of six in hand), each component within 2e-4 of
max(|F|, median |F|) (the pairs' magnitudes sum to at most 150 times that, at
1.2e-6 each if all signs agreed).  Energies: errors of random sign add up to
3e-7 of the root of the sum of the terms' squares; six times that, and the
fixed-point quantum of the rows.  An error of 1e-4 in every term fails on the
gradient, and on the energies that do not cancel."""
import dataclasses

import numpy as np
import pytest

from q6_gb300.qnb import (LIST_PP, LIST_PP14, LIST_PW, LIST_QP, LIST_QW, LIST_WW, PREC_FP64, PREC_MIXED,
                          NonbondedEngine)
from q6_gb300.system import make_system
from tests.test_gpu_fp64_pairs import four_site
from tests.test_gpu_rows_solute import arithmetic
from tests.test_gpu_rows_water import evaluate

pytestmark = pytest.mark.gpu


def distance2(s, i, j, L):
    t = s.x[j] - s.x[i]
    if L:
        t -= L * np.round(t / L)
    return (t * t).sum(1)


def term_squares(s, L, rc):
    """Roots of the sums of squares of the pair terms: pp, pw, ww (el, vdw) and per state qp, qw (el, vdw)."""
    with NonbondedEngine(s, precision=PREC_FP64, use_lrf=False) as e:
        if L:
            e.set_box([L] * 3)
        e.make_pair_lists(s.x, Rcq=9.0, RcLRF=9.0, Rcpp=rc, Rcpw=rc, Rcww=rc)
        pairs = {k: e.export_pairs(k) for k in (LIST_PP, LIST_PW, LIST_WW, LIST_QP, LIST_QW, LIST_PP14)}
    geo = s.ivdw_rule == 1
    combine = lambda a, b, c, d: (a * b, c * d) if geo else ((a + b) ** 12 * c * d, 2.0 * (a + b) ** 6 * c * d)
    root = lambda *v: [float(np.sqrt((u * u).sum())) for u in v]
    E, EQ = [], np.zeros((s.nstates, 4))
    for kind in (LIST_PP, LIST_PW, LIST_WW):
        i, j = pairs[kind]
        code = s.ljcod[s.iac[i], s.iac[j]].astype(int) - 1
        A, B = combine(s.avdw[s.iac[i], code], s.avdw[s.iac[j], code], s.bvdw[s.iac[i], code], s.bvdw[s.iac[j], code])
        r2 = distance2(s, i, j, L)
        E += root(s.crg[i] * s.crg[j] / np.sqrt(r2), np.hypot(A / r2 ** 6, B / r2 ** 3))
    for c, kind in ((0, LIST_QP), (2, LIST_QW)):
        iq, j = pairs[kind]
        r2 = distance2(s, s.iqseq[iq], j, L)
        for st in range(s.nstates):
            q = s.qiac[iq, st]
            A, B = combine(s.qavdw[q, 0], s.avdw[s.iac[j], 0], s.qbvdw[q, 0], s.bvdw[s.iac[j], 0])
            u = 1.0 / (r2 ** 3 + s.sc_lookup[iq, s.iac[j], st])
            EQ[st, c:c + 2] = root(s.qcrg[iq, st] * s.crg[j] / np.sqrt(r2), np.hypot(A * u * u, B * u))
    return np.array(E), EQ


def check(s, L, rc):
    s = dataclasses.replace(s, x=np.round(s.x * 2.0 ** 18) / 2.0 ** 18)
    sE, sEQ = term_squares(s, L, rc)
    (d0, E0, EQ0), (d, E, EQ) = evaluate(s, PREC_FP64, L, rc), evaluate(s, PREC_MIXED, L, rc)
    assert np.sqrt(((d - d0) ** 2).mean()) <= 1e-5 * np.sqrt((d0 ** 2).mean())
    assert np.all(np.abs(d - d0) <= 2e-4 * np.maximum(np.abs(d0), np.median(np.abs(d0))))
    quantum = s.natom * 2.0 ** -32
    assert np.all(np.abs(E - E0)[:6] <= 1.8e-6 * sE + quantum), (E - E0, sE)
    assert np.all(np.abs(EQ - EQ0)[:, 2:] <= 1.8e-6 * sEQ + quantum), (EQ - EQ0, sEQ)


@pytest.mark.parametrize("sizes,n_solute,rc", [((1, 1), 40, 6.0), ((2, 3), 90, 7.0), ((4, 4), 300, 9.0), ((5, 6), 330, 9.0),
                                               ((7, 8), 200, 8.0), ((9, 15), 260, 9.0)])
@pytest.mark.parametrize("rule", [1, 2])
@pytest.mark.parametrize("box", [None, 38.0])
def test_solute_rows(sizes, n_solute, rc, rule, box):
    s = make_system(R=12.0, n_solute=n_solute, group_sizes=sizes, ntypes=5, nq=3, nstates=2, seed=29,
                    type2_pairs=((0, 1), (2, 2)))
    check(arithmetic(s) if rule == 2 else s, box, rc)


@pytest.mark.parametrize("R,n_solute,nq,rc", [(6.0, 12, 3, 5.0), (7.0, 60, 3, 6.5), (9.0, 200, 4, 9.0), (11.0, 12, 3, 9.9)])
@pytest.mark.parametrize("sites", [3, 4])
@pytest.mark.parametrize("box", [False, True])
def test_water_rows(R, n_solute, nq, rc, sites, box):
    s = make_system(R=R, n_solute=n_solute, group_sizes=(3, 6), nq=nq, nstates=2, seed=23)
    check(four_site(s) if sites == 4 else s, 2.0 * R + 14.0 if box else None, rc)


@pytest.mark.parametrize("R,n_solute,nq,nstates", [(7.0, 32, 5, 2), (9.0, 65, 4, 5), (11.0, 129, 11, 8), (12.0, 80, 40, 8)])
@pytest.mark.parametrize("box", [False, True])
def test_q_environment(R, n_solute, nq, nstates, box):
    s = make_system(R=R, n_solute=n_solute, nq=nq, nstates=nstates, seed=31)
    check(s, 2.0 * R + 14.0 if box else None, 6.0)


@pytest.mark.parametrize("n_solute,sizes,nq,rc", [(33, (1, 1), 1, 30.0), (67, (1, 1), 2, 30.0), (150, (2, 4), 7, 6.0),
                                                  (200, (9, 15), 5, 9.0)])
@pytest.mark.parametrize("box", [None, 28.0, 44.0])
def test_row_build(n_solute, sizes, nq, rc, box):
    s = make_system(R=12.0, n_solute=n_solute, group_sizes=sizes, ntypes=5, nq=nq, nstates=2, seed=37)
    check(s, box, min(rc, 13.0) if box else rc)

"""FP32 rounding of the solute rows' energies over long rows.  One atom's charge
is ten million times the others', so in every row one lane meets a term of
which the others are less than half a unit in the last place: they are lost if
they are added to it one after the other, and kept if every prefetched chunk of
128 partners has a sum of its own.  Against the FP64 form: within 2e-7 of the
energy, the reciprocal square root's largest error (2^-22.9) and the rounding
of short runs (4e-8); lost terms make 6e-7 of it."""
import numpy as np
import pytest

from q6_gb300.qnb import PREC_FP64, PREC_MIXED, NonbondedEngine
from q6_gb300.system import make_system

pytestmark = pytest.mark.gpu


def test_energy_of_long_rows():
    s = make_system(R=25.0, n_solute=2955, group_sizes=(3, 6), nq=3, nstates=2, seed=7)
    s.crg[: s.nat_solute] = 0.1
    s.crg[s.nat_solute // 2] = 1.0e6
    E = []
    for prec in (PREC_FP64, PREC_MIXED):
        with NonbondedEngine(s, precision=prec, use_lrf=False) as e:
            e.set_lambda([0.5, 0.5])
            e.make_pair_lists(s.x, Rcpp=99.0, Rcpw=3.0, Rcww=3.0)
            E.append(e.pot_energy_nonbonds(s.x)[1]["pp_el"])
    assert abs(E[1] - E[0]) <= 2e-7 * abs(E[0]), (E[1] - E[0]) / E[0]

"""qnb_pot_energy_step with profiling on: every class is counted once per step
whether or not the caller collects between the steps, the results are those of
the unprofiled step, bit for bit, and a long run whose times nobody collects
does not pile up events (about 26 a step, some 100 bytes each of host memory:
the 3,000 steps measured here would add 8 MB or more; 2 MB are allowed)."""
import os

import numpy as np
import pytest

from q6_gb300.qnb import PREC_MIXED, NonbondedEngine
from q6_gb300.system import default_solvent_params, make_system

pytestmark = pytest.mark.gpu
CUT = dict(Rcq=99.0, RcLRF=99.0, Rcpp=8.0, Rcpw=8.0, Rcww=8.0)


def rss():
    with open("/proc/self/statm") as f:
        return int(f.read().split()[1]) * os.sysconf("SC_PAGE_SIZE")


def test_profiled_host_steps():
    s = make_system(R=5.0, n_solute=6, nq=3, nstates=2, seed=12)
    with NonbondedEngine(s, precision=PREC_MIXED) as e:
        e.set_solvent_params(default_solvent_params(s, itdis=1.0e6))
        e.set_lambda([0.3, 0.7])
        e.make_pair_lists(s.x, **CUT)
        want = e.pot_energy_step(s.x)
        e.profile(True)
        e.kernel_times()
        for k in range(5):
            d, E, EQ, _ = e.pot_energy_step(s.x)
            assert np.array_equal(d, want[0]) and E == want[1] and np.array_equal(EQ, want[2])
        t = e.kernel_times()
        for name in ("ww", "pp", "qw", "qp", "qq", "lrf_taylor", "restrain", "watpol"):
            assert t[name][1] == 5 and t[name][0] > 0.0, (name, t[name])
        for k in range(500):
            e.pot_energy_step(s.x)
        m0 = rss()
        for k in range(3000):
            e.pot_energy_step(s.x)
        grown = rss() - m0
    assert grown <= 2 << 20, grown

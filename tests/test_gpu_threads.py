"""Eight host threads with a context each, of topologies whose LRF accumulation
asks for different amounts of shared memory: every list build succeeds, and
each context then holds the records that it gave by itself, bit for bit."""
import threading

import numpy as np
import pytest

from q6_gb300.qnb import PREC_MIXED, NonbondedEngine
from q6_gb300.system import make_system

pytestmark = pytest.mark.gpu
CUT = dict(Rcq=99.0, RcLRF=99.0, Rcpp=6.0, Rcpw=5.0, Rcww=5.5)


def test_list_builds_of_several_threads():
    systems = [make_system(R=8.0, n_solute=n, group_sizes=sizes, nq=3, nstates=2, seed=17)
               for n, sizes in ((120, (12, 15)), (6, (3, 5)))] * 4
    engines = [NonbondedEngine(s, precision=PREC_MIXED) for s in systems]
    alone = []
    for e, s in zip(engines, systems):
        e.make_pair_lists(s.x, **CUT)
        alone.append(e.lrf())
    start, errors = threading.Barrier(len(engines)), []

    def work(e, s, want):
        start.wait()
        try:
            for _ in range(3000):
                e.make_pair_lists(s.x, **CUT)
            assert np.array_equal(e.lrf(), want)
        except Exception as err:
            errors.append(err)

    threads = [threading.Thread(target=work, args=a) for a in zip(engines, systems, alone)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for e in engines:
        e.close()
    assert not errors, errors

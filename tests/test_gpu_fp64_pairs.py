"""FP64 form of the water-water and solute-water pairs for solvents of 3 and 4
atoms, with and without the SPC fast path (the kernels' compile-time molecule
sizes and the Coulomb-only atoms), against the oracle: 1e-6 kcal/mol per term
and 1e-6 relative per gradient component, the FP64 form's bars."""
import dataclasses

import numpy as np
import pytest

from oracle.oracle import Oracle
from q6_gb300.qnb import PREC_FP64, NonbondedEngine
from q6_gb300.system import make_system

pytestmark = pytest.mark.gpu
CUT = dict(Rcq=99.0, RcLRF=99.0, Rcpp=8.0, Rcpw=8.0, Rcww=8.0)


def four_site(s):
    """The same droplet with a fourth solvent atom (copy of the last type) 0.3 A off the first."""
    w = s.x[s.nat_solute:].reshape(s.nwat, 3, 3)
    m = w[:, :1] + np.array([0.0, 0.0, 0.3])
    x = np.concatenate([s.x[: s.nat_solute], np.concatenate([w, m], 1).reshape(-1, 3)])
    per = lambda a: np.concatenate([a[: s.nat_solute], np.repeat(a[s.nat_solute:].reshape(s.nwat, 3), [1, 1, 2], 1).ravel()])
    nat = s.nat_solute + 4 * s.nwat
    ns, W = s.ncgp_solute, np.arange(s.nwat)
    first = np.concatenate([s.cgp_first[:ns], s.nat_solute + 4 * W]).astype(np.int32)
    last = np.concatenate([s.cgp_last[:ns], s.nat_solute + 4 * W + 3]).astype(np.int32)
    sw = np.concatenate([s.cgp_iswitch[:ns], s.nat_solute + 4 * W]).astype(np.int32)
    return dataclasses.replace(s, x=x, natom=nat, solv_atom=4, crg=per(s.crg), iac=per(s.iac), excl=per(s.excl),
                               heavy=per(s.heavy), cgp_first=first, cgp_last=last, cgp_iswitch=sw,
                               cgpatom=np.arange(nat, dtype=np.int32))


@pytest.mark.parametrize("sites,solvent_type", [(3, 0), (3, 2), (4, 0), (4, 2)])
def test_fp64_water_pairs(sites, solvent_type):
    s = make_system(R=9.0, n_solute=15, nq=4, nstates=2, seed=91)
    s = dataclasses.replace(s if sites == 3 else four_site(s), solvent_type=solvent_type)
    o = Oracle(s)
    o.set_lambda([0.4, 0.6])
    o.make_pair_lists(s.x, **CUT)
    d0, E0, EQ0 = o.pot_energy_nonbonds(s.x)
    with NonbondedEngine(s, precision=PREC_FP64) as e:
        e.set_lambda([0.4, 0.6])
        e.make_pair_lists(s.x, **CUT)
        d, E, EQ = e.pot_energy_nonbonds(s.x)
    assert all(abs(E[k] - E0[k]) <= 1e-6 for k in E0)
    assert np.all(np.abs(EQ - EQ0) <= 1e-6)
    assert np.all(np.abs(d - d0) <= 1e-6 * np.maximum(np.abs(d0), np.median(np.abs(d0))))

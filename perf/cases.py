"""Performance cases of the nonbonded engine: what its users have it do.

A case is one call sequence of the public entry points (q6_gb300.qnb, the
Python mirror of the C ABI) on a generated system:

  host      qnb_pot_energy_step: a qdyn process's pot_energy call, one window,
            host buffers in and out
  batch     qnb_compute_dev: one step of all lambda windows of a perturbation
            on device-resident coordinates, energies read back (EVB/FEP
            sampling reads them), gradient left in HBM
  md        qnb_md_run: the device-resident MD step, one list-update cycle
  adjoint   qnb_q_adjoint_dev: parameter gradients of the Q-atom energies

With ``lists`` the pair lists (and the LRF moments) are rebuilt in the pass,
as qdyn does every NBcycle steps; without it the pass runs on lists built a
few steps earlier, from slightly different coordinates.

The mixed form computes its pairs in FP32, so its outputs are handed on as
float32; the FP64 form's as float64.
"""
import ctypes
import functools
import math

import numpy as np
import torch

from q6_gb300.bonded import remove_shaken, synthetic_bonded
from q6_gb300.md import MdSetup, maxwell_velocities
from q6_gb300.qnb import PREC_FP64, PREC_MIXED, NonbondedEngine
from q6_gb300.system import default_solvent_params, make_system

TFREE = 300.0
ISTEP = 7          # a step that does not update watpol's theta_corr
MD_STEPS = 25      # one NBcycle of qdyn's default input
MAX_ATOMS = 51 * 6060   # window-atoms of the largest batches


def _case(kind, prec, R, n_solute, nq, nstates, windows, lists, box=False, rc=10.0, name=None):
    c = dict(kind=kind, prec=prec, R=float(R), n_solute=int(n_solute), nq=int(nq), nstates=int(nstates),
             windows=int(windows), lists=bool(lists), box=bool(box), rc=float(rc))
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # one qdyn process, the small droplet of the regression-test size: the smallest call
        _case("host", "mixed", 15, 20, 6, 2, 1, False, name="host_r15"),
        # the same in the all-FP64 form
        _case("host", "fp64", 15, 20, 6, 2, 1, False, name="host_r15_fp64"),
        # one qdyn process on the 25 A sphere with a protein-sized solute
        _case("host", "mixed", 25, 3000, 20, 2, 1, False, name="host_r25"),
        # ... and its list-update step
        _case("host", "mixed", 25, 3000, 20, 2, 1, True, name="host_r25_lists"),
        # 51 lambda windows of the droplet: many small windows
        _case("batch", "mixed", 15, 20, 6, 2, 51, False, name="w51_r15"),
        # 51 lambda windows of the 25 A sphere: the benchmark's plain step
        _case("batch", "mixed", 25, 3000, 20, 2, 51, False, name="w51_r25"),
        # ... and its list-update step
        _case("batch", "mixed", 25, 3000, 20, 2, 51, True, name="w51_r25_lists"),
        # windows in the all-FP64 form (reference trajectories for dG checks)
        _case("batch", "fp64", 25, 3000, 20, 2, 16, False, name="w16_r25_fp64"),
        # periodic box with LRF, the solute of the 25 A sphere
        _case("batch", "mixed", 25, 3000, 20, 2, 51, False, box=True, name="w51_box"),
        # a large sphere, 40 Q atoms in 4 states, 12 A cut-offs, lists rebuilt
        _case("batch", "mixed", 34, 1500, 40, 4, 8, True, rc=12.0, name="w8_r34_lists"),
        # a replica's device-resident MD over one list-update cycle
        _case("md", "mixed", 20, 40, 10, 2, 16, True, name="md_r20"),
        # parameter gradients of 4-state EVB over 200 snapshots
        _case("adjoint", "mixed", 15, 40, 30, 4, 200, True, name="adjoint_r15"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["host", "host", "batch", "batch", "batch", "batch", "batch", "md", "adjoint"])
    prec = "fp64" if kind in ("host", "batch") and rng.random() < 0.2 else "mixed"
    R = round(rng.uniform(13.0, 27.0), 2)
    n_solute = _log_int(rng, 12, 1200)
    if kind in ("md", "adjoint"):
        R, n_solute = round(rng.uniform(13.0, 21.0), 2), _log_int(rng, 12, 60)
    n_solute = min(n_solute, int(0.06 * (R - 2.0) ** 3 * 2.0))
    nq = rng.randint(2, min(40, n_solute))
    nstates = rng.choice([1, 2, 2, 2, 3, 4])
    atoms = n_solute + 0.1 * 4.19 * R ** 3
    most = MAX_ATOMS * (0.15 if kind == "md" else 0.25 if prec == "fp64" else 0.8)
    W = 1 if kind == "host" else _log_int(rng, 1, max(1, min(200 if kind == "adjoint" else 64, int(most / atoms))))
    lists = kind in ("md", "adjoint") or rng.random() < 0.4
    box = kind == "batch" and rng.random() < 0.3
    rc = rng.choice([10.0, 10.0, 9.0, 12.0])
    return _case(kind, prec, R, n_solute, nq, nstates, W, lists, box, rc)


# ---- the systems ------------------------------------------------------------
@functools.lru_cache(maxsize=4)
def _system(R, n_solute, nq, nstates):
    """A topology (a user's program has one for all its frames and windows)."""
    return make_system(R=R, n_solute=n_solute, group_sizes=(3, 6) if n_solute > 60 else (3, 5),
                       ntypes=12 if n_solute > 60 else 6, nq=nq, nstates=nstates, q_sigma=0.4,
                       lognormal_q=nstates > 2, seed=2000)


def _topology(case):
    return _system(case["R"], case["n_solute"], case["nq"], case["nstates"])


def _box_edge(s):
    return 2.0 * round(float(np.sqrt((s.x ** 2).sum(1)).max())) + 3.0


def _cuts(case, s):
    rc = case["rc"]
    if case["box"]:
        half = 0.499 * _box_edge(s)
        return dict(Rcq=min(12.0, half), RcLRF=20.0, Rcpp=min(rc, half), Rcpw=min(rc, half), Rcww=min(rc, half))
    return dict(Rcq=99.0, RcLRF=99.0, Rcpp=rc, Rcpw=rc, Rcww=rc)


def _inputs(case, seed):
    """Coordinates of every window when its lists are built and when it is
    evaluated, and its lambdas."""
    s = _topology(case)
    rng = np.random.default_rng(seed)
    W = case["windows"]
    x0 = s.x + rng.normal(0.0, 0.002 if case["kind"] == "md" else 0.02, (W,) + s.x.shape)
    x = x0 if case["lists"] else x0 + rng.normal(0.0, 0.03, x0.shape)
    lam = np.zeros((W, s.nstates))
    l0 = (np.arange(W) + rng.uniform(0.0, 1.0)) / W
    if s.nstates == 1:
        lam[:, 0] = 1.0
    else:
        lam[:, 0], lam[:, 1] = l0, 1.0 - l0
    return s, x0, x, lam


class _DeviceArray:
    """The engine's gradient accumulators as a CUDA array."""

    def __init__(self, ptr, shape):
        self.__cuda_array_interface__ = dict(shape=shape, typestr="<f8", data=(ptr, False), version=2)


class _State:
    pass


def prepare(case, seed):
    s, x0, x, lam = _inputs(case, seed)
    st = _State()
    st.case, st.cut, st.W, st.s = case, _cuts(case, s), case["windows"], s
    st.out = torch.float32 if case["prec"] == "mixed" else torch.float64
    st.np_out = np.float32 if case["prec"] == "mixed" else np.float64
    st.eng = e = NonbondedEngine(s, precision=PREC_MIXED if case["prec"] == "mixed" else PREC_FP64, windows=st.W)
    if case["box"]:
        e.set_box([_box_edge(s)] * 3)
    else:
        e.set_solvent_params(default_solvent_params(s))
    for w in range(st.W):
        e.set_lambda(lam[w], window=w)
    if case["kind"] == "host":
        e.make_pair_lists(x0[0], **st.cut)
        st.x = np.ascontiguousarray(x[0])
        return st
    e.set_coordinates_dev(x0)
    if case["kind"] == "md":
        heavy = np.asarray(s.heavy).astype(bool)
        e.set_bonded(remove_shaken(synthetic_bonded(s, seed=21), heavy, s.nat_solute))
        e.md_init(MdSetup(stepsize=0.5, temp0=300.0, tau_t=100.0, nbcycle=MD_STEPS, cut=st.cut))
        st.x = x0
        st.v = np.stack([maxwell_velocities(s, 300.0, seed + w) for w in range(st.W)])
        return st
    e.make_pair_lists_dev(**st.cut)
    e.set_coordinates_dev(x)
    _, d = e.device_buffers()
    st.d = torch.as_tensor(_DeviceArray(d, (st.W, s.natom, 3)), device="cuda")
    st.stream = torch.cuda.ExternalStream(e.stream())
    return st


def run(st):
    e, case, W, S = st.eng, st.case, st.W, st.s.nstates
    if case["kind"] == "host":
        if case["lists"]:
            e.make_pair_lists(st.x, **st.cut)
        d, E, EQ, R = e.pot_energy_step(st.x, Tfree=TFREE, istep=ISTEP)
        t = st.np_out
        return {"gradient": d.astype(t, copy=False), "E": np.array(list(E.values()), t)[None],
                "EQ": EQ.astype(t)[None], "restraints": R.astype(t)[None]}
    if case["kind"] == "md":
        e.set_coordinates_dev(st.x)
        e.md_set_velocities(st.v)
        e.md_prepare(stop_cm=False)
        rec, EQ, _ = e.md_run(MD_STEPS, 0)
        xv = [e.md_state(w) for w in range(W)]
        t = st.np_out
        return {"x": np.stack([a for a, _ in xv]).astype(t), "v": np.stack([b for _, b in xv]).astype(t),
                "temp": rec["temp"].astype(t), "EQ": EQ.astype(t)}
    if case["lists"]:
        e.make_pair_lists_dev(**st.cut)
    if case["kind"] == "adjoint":
        dq, dA, dB = e.q_adjoint_dev()
        return {"dq": dq, "dA": dA, "dB": dB}
    with torch.cuda.stream(st.stream):
        st.d.zero_()
    E, EQ, R = np.zeros((W, 7)), np.zeros((W, S, 6)), np.zeros((W, 2))
    p = [a.ctypes.data_as(ctypes.c_void_p) for a in (E, EQ, R)]
    e._check(e.lib.qnb_compute_dev(e.h, TFREE, ISTEP, 1, *p))
    with torch.cuda.stream(st.stream):
        g = st.d.to(st.out, copy=True)
    t = st.np_out
    return {"gradient": g, "E": E.astype(t), "EQ": EQ.astype(t), "restraints": R.astype(t)}


# ---- the work a pass cannot do without ------------------------------------------
def _sizes(s):
    n = np.asarray(s.cgp_last) - np.asarray(s.cgp_first) + 1
    isq = np.zeros(s.natom, bool)
    isq[np.asarray(s.iqseq, np.int64)] = True
    unit = np.repeat(np.arange(s.ncgp), n)
    return n, isq, unit


@functools.lru_cache(maxsize=32)
def _pair_counts(R, n_solute, nq, nstates, box, rc, rlrf):
    """Atom pairs within the cut-offs (pp, pw, ww) and (unit, source atom)
    pairs of the LRF moments at the topology's coordinates."""
    s = _system(R, n_solute, nq, nstates)
    _, isq, unit = _sizes(s)
    free = torch.from_numpy(np.bincount(unit[~isq], minlength=s.ncgp).astype(np.float64))
    xs = torch.from_numpy(s.x[np.asarray(s.cgp_iswitch, np.int64)])
    G = s.ncgp_solute
    pp = pw = ww = far = 0.0
    for a in range(0, s.ncgp, 1024):
        d = xs[a:a + 1024, None, :] - xs[None, :, :]
        if box:
            L = _box_edge(s)
            d = d - L * torch.round(d / L)
        d = (d * d).sum(-1)
        near = (d <= rc * rc).double()
        m = near * free[a:a + 1024, None] * free[None, :]
        k = max(0, min(G - a, 1024))
        pp += float(m[:k, :G].sum())
        pw += float(m[:k, G:].sum())
        ww += float(m[k:, G:].sum())
        far += float((((d > rc * rc) & (d <= rlrf * rlrf)).double() @ free).sum())
    return 0.5 * pp, pw, 0.5 * (ww - 9.0 * s.nwat), far


def work(case):
    s = _topology(case)
    W, S, nq, N = case["windows"], case["nstates"], s.nqat, s.natom
    cut = _cuts(case, s)
    pp, pw, ww, far = _pair_counts(case["R"], case["n_solute"], case["nq"], S, case["box"], case["rc"], cut["RcLRF"])
    share = min(1.0, 4.19 * cut["Rcq"] ** 3 / _box_edge(s) ** 3) if case["box"] else 1.0
    q = share * nq * ((22 + 17 * S) * (s.nat_solute - nq + s.nwat) + 2 * (19 + 5 * S) * s.nwat)
    step = 33 * pp + 26 * pw + 23 * ww + q + 75 * N
    build = 46 * far + 8 * (pp + pw + ww) / 9
    word = 8 if case["prec"] == "fp64" else 4
    if case["kind"] == "md":
        return {"bytes": W * N * 24 * 4, "flops": W * (MD_STEPS * (step + 60 * N) + build)}
    if case["kind"] == "adjoint":
        return {"bytes": W * (N * 24 + 3 * nq * S * 8), "flops": W * (q + build)}
    return {"bytes": W * N * (24 + 3 * word), "flops": W * (step + (build if case["lists"] else 0.0))}


# ---- the same in plain torch, 64 bits ---------------------------------------------
class _Model:
    """The topology's arrays in torch, for the evaluation below."""

    def __init__(self, s, dev):
        def t(a, dt=torch.float64):
            return torch.as_tensor(np.ascontiguousarray(a)).to(dev, dt)

        self.s, self.dev = s, dev
        n, isq, unit = _sizes(s)
        self.unit, self.isq = t(unit, torch.int64), t(isq, torch.bool)
        self.ref = t(s.cgp_iswitch, torch.int64)
        self.size = t(n)
        self.solute_u = torch.arange(s.ncgp, device=dev) < s.ncgp_solute
        self.crg, self.iac = t(s.crg), t(s.iac, torch.int64)
        self.avdw, self.bvdw = t(s.avdw), t(s.bvdw)
        self.code = t(s.ljcod, torch.int64)
        self.excl_pairs, self.pairs14 = t(s.excl_pairs, torch.int64), t(s.pairs14, torch.int64)
        self.iq = t(s.iqseq, torch.int64)
        self.qcrg, self.qt = t(s.qcrg), t(s.qiac, torch.int64)
        self.qa, self.qb = t(s.qavdw), t(s.qbvdw)
        self.sc, self.qconn = t(s.sc_lookup), t(s.qconn, torch.int64)


def _lrf_gradient(M, x0, x, cut, box, grad, chunk):
    """LRF moments from x0, their Taylor terms at x: adds the gradient,
    returns the energy (lrf_update and lrf_taylor of the reference)."""
    s = M.s
    U = s.ncgp
    cent = torch.zeros(U, 3, dtype=x.dtype, device=x.device).index_add_(0, M.unit, x0) / M.size[:, None]
    src = torch.nonzero(~M.isq)[:, 0]
    xs, q, us = x0[src], M.crg[src], M.unit[src]
    xr = x0[M.ref]
    eye = torch.eye(3, dtype=x.dtype, device=x.device)
    p0 = torch.zeros(U, dtype=x.dtype, device=x.device)
    p1, p2 = p0.new_zeros(U, 3), p0.new_zeros(U, 3, 3)
    p3 = p0.new_zeros(U, 3, 3, 3)
    for a in range(0, U, chunk):
        sl = slice(a, min(a + chunk, U))
        du = xr[sl, None, :] - xr[None, :, :]
        if box:
            du = du - box * torch.round(du / box)
        du = (du * du).sum(-1)
        both, one = M.solute_u[sl, None] & M.solute_u[None, :], M.solute_u[sl, None] ^ M.solute_u[None, :]
        rc = torch.where(both, cut["Rcpp"], torch.where(one, cut["Rcpw"], cut["Rcww"]))
        far = (du > rc * rc) & (du <= cut["RcLRF"] ** 2)
        far &= torch.arange(U, device=x.device)[sl, None] != torch.arange(U, device=x.device)[None, :]
        d = xs[None, :, :] - cent[sl, None, :]
        if box:
            d = d - box * torch.round((xr[None, us, :] - cent[sl, None, :]) / box)
        m = far[:, us]
        r2 = torch.where(m, (d * d).sum(-1), 1.0)
        qm = torch.where(m, q[None, :], 0.0)
        f0 = qm / (r2 * torch.sqrt(r2))
        f1 = 3.0 * f0 / r2
        f2 = -f1 / r2
        p0[sl] = (f0 * r2).sum(1)
        p1[sl] = -torch.einsum("tn,tna->ta", f0, d)
        p2[sl] = torch.einsum("tn,tna,tnb->tab", f1, d, d) - f0.sum(1)[:, None, None] * eye
        u = torch.einsum("tn,tna->ta", f2 * r2, d)
        t3 = 5.0 * torch.einsum("tna,tnb,tnc->tabc", f2[..., None] * d, d, d)
        p3[sl] = t3 - (torch.einsum("ab,tc->tabc", eye, u) + torch.einsum("ac,tb->tabc", eye, u)
                       + torch.einsum("bc,ta->tabc", eye, u))
    dr = (cent[M.unit] - x)[src]
    p0, p1, p2, p3 = p0[us], p1[us], p2[us], p3[us]
    v = p0 + (dr * p1).sum(1) + 0.5 * torch.einsum("na,nab,nb->n", dr, p2, dr)
    df = p1 + torch.einsum("nab,nb->na", p2, dr) + 0.5 * torch.einsum("nabc,nb,nc->na", p3, dr, dr)
    grad[src] -= df * q[:, None]
    return 0.5 * (q * v).sum()


def _pairs(M, x0, x, cut, box, grad, chunk):
    """The classical pairs: adds the gradient, returns (pp, pw, ww) x (el, vdw)."""
    s = M.s
    N, ns = s.natom, s.nat_solute
    E = torch.zeros(3, 2, dtype=x.dtype, device=x.device)
    xr0, xr = x0[M.ref], x[M.ref]
    kind = torch.zeros(ns, ns, dtype=torch.int8, device=x.device)
    for p, k in ((M.excl_pairs, 1), (M.pairs14, 3)):
        kind[p[:, 0], p[:, 1]] = k
        kind[p[:, 1], p[:, 0]] = k
    a1, b1 = M.avdw[M.iac], M.bvdw[M.iac]
    for a in range(0, N, chunk):
        sl = slice(a, min(a + chunk, N))
        ui = M.unit[sl]
        du = xr0[ui][:, None, :] - xr0[None, :, :]
        if box:
            du = du - box * torch.round(du / box)
        du = (du * du).sum(-1)
        both, one = M.solute_u[ui][:, None] & M.solute_u[None, :], M.solute_u[ui][:, None] ^ M.solute_u[None, :]
        rc = torch.where(both, cut["Rcpp"], torch.where(one, cut["Rcpw"], cut["Rcww"]))
        inside = (du <= rc * rc)
        inside &= M.solute_u[None, :] | (ui[:, None] != torch.arange(s.ncgp, device=x.device)[None, :])
        m = inside[:, M.unit]
        m &= ~(M.isq[sl, None] | M.isq[None, :])
        m &= torch.arange(N, device=x.device)[sl, None] != torch.arange(N, device=x.device)[None, :]
        k = M.code[M.iac[sl]][:, M.iac]
        el = M.crg[sl, None] * M.crg[None, :]
        if a < ns:
            kk = kind[a:min(a + chunk, ns)]
            r = kk.shape[0]
            m[:r, :ns] &= kk != 1
            k[:r, :ns] = torch.where(kk == 3, 3, k[:r, :ns])
            el[:r, :ns] *= torch.where(kk == 3, s.el14_scale, 1.0)
        A = torch.zeros_like(el)
        B = torch.zeros_like(el)
        for c in (1, 2, 3):
            A = torch.where(k == c, a1[sl, c - 1][:, None] * a1[None, :, c - 1], A)
            B = torch.where(k == c, b1[sl, c - 1][:, None] * b1[None, :, c - 1], B)
        t = x[None, :, :] - x[sl, None, :]
        if box:
            t = t + box * torch.round((xr[ui][:, None, :] - xr[M.unit][None, :, :]) / box)
        r2 = torch.where(m, 1.0 / torch.where(m, (t * t).sum(-1), 1.0), 0.0)
        r6 = r2 ** 3
        vel, va, vb = el * torch.sqrt(r2), A * r6 * r6, B * r6
        dv = r2 * (-vel - 12.0 * va + 6.0 * vb)
        grad[sl] -= torch.einsum("ij,ija->ia", dv, t)
        n = max(0, min(ns - a, sl.stop - a))
        for row, v in ((0, vel), (1, va - vb)):
            E[0, row] += 0.5 * v[:n, :ns].sum()
            E[1, row] += v[:n, ns:].sum()
            E[2, row] += 0.5 * v[n:, ns:].sum()
    return E


def _q_pairs(M, x0, x, cut, box, qcrg, qa, qb):
    """Every pair of a Q atom with the solute, the water or another Q atom:
    (Q atom, partner, vector, A, B, el, alpha, LJ?, kind) in blocks."""
    s = M.s
    S, nq, ns, nw = s.nstates, s.nqat, s.nat_solute, s.nwat
    centre = x0[M.iq[0]] if box else torch.as_tensor(s.xpcent).to(x)
    t = [M.qt[:, st] for st in range(S)]
    # solute partners
    j = torch.nonzero(~M.isq[:ns])[:, 0]
    out = []
    if len(j):
        conn = M.qconn[0][j].T                                     # [nq, nj]
        near = (M.qconn[:, j, :] <= 3).any(0).any(1)              # Q-bonded partners: static list
        if box:
            rel = x0[:ns] - centre
            inside = ((rel - box * torch.round(rel / box)) ** 2).sum(-1) <= cut["Rcq"] ** 2
            listed = torch.zeros(s.ncgp, dtype=torch.bool, device=x.device)
            listed[M.unit[:ns][inside]] = True
            rel = x[:ns] - x[M.iq[0]]
            inside = ((rel - box * torch.round(rel / box)) ** 2).sum(-1) <= cut["Rcq"] ** 2
            first = torch.arange(ns, device=x.device) + torch.where(inside, 0, ns)
            ref = torch.full((s.ncgp,), 4 * ns, dtype=torch.int64, device=x.device)
            ref = ref.scatter_reduce(0, M.unit[:ns], first, "amin") % ns
            sh = box * torch.round((x[M.iq[0]] - x[ref[M.unit[j]]]) / box)
            sh = torch.where(near[:, None], 0.0, sh)
        else:
            listed = ((x0[M.ref] - centre) ** 2).sum(-1) <= cut["Rcq"] ** 2
            sh = torch.zeros(len(j), 3, dtype=x.dtype, device=x.device)
        use = torch.where(near[None, :], conn >= 4, listed[M.unit[j]][None, :])
        code = torch.where(near[None, :], 1, M.code[M.iac[j]][:, M.iac[M.iq]].T)
        code = torch.where(conn == 4, 3, code)
        vec = x[j][None, :, :] + sh[None, :, :] - x[M.iq][:, None, :]
        aj, bj = M.avdw[M.iac[j]], M.bvdw[M.iac[j]]
        A, B, el, sc = [], [], [], []
        for st in range(S):
            Aq = torch.where(code == 3, qa[t[st], 2][:, None], qa[t[st], 0][:, None])
            Bq = torch.where(code == 3, qb[t[st], 2][:, None], qb[t[st], 0][:, None])
            A.append(Aq * torch.gather(aj.T, 0, code - 1))
            B.append(Bq * torch.gather(bj.T, 0, code - 1))
            el.append(qcrg[:, st][:, None] * M.crg[j][None, :] * torch.where(code == 3, s.el14_scale, 1.0))
            sc.append(M.sc[:, :, st][:, M.iac[j]])
        out.append((M.iq, j, vec, use, torch.stack(A), torch.stack(B), torch.stack(el), torch.stack(sc), 1))
    # water partners: LJ for the first atom, Coulomb for the others
    o = ns + 3 * torch.arange(nw, device=x.device)
    if nw:
        if box:
            rel = x0[o] - centre
            listed = ((rel - box * torch.round(rel / box)) ** 2).sum(-1) <= cut["Rcq"] ** 2
            sh = box * torch.round((x[M.iq[0]] - x[o]) / box)
        else:
            listed = ((x0[o] - centre) ** 2).sum(-1) <= cut["Rcq"] ** 2
            sh = torch.zeros(nw, 3, dtype=x.dtype, device=x.device)
        for k in range(3):
            j = o + k
            vec = x[j][None, :, :] + sh[None, :, :] - x[M.iq][:, None, :]
            tw = M.iac[ns + k]
            lj = 1.0 if k == 0 else 0.0
            A = torch.stack([lj * (qa[t[st], 0] * M.avdw[tw, 0])[:, None].expand(nq, nw) for st in range(S)])
            B = torch.stack([lj * (qb[t[st], 0] * M.bvdw[tw, 0])[:, None].expand(nq, nw) for st in range(S)])
            el = torch.stack([qcrg[:, st][:, None] * M.crg[j][None, :] for st in range(S)])
            sc = torch.stack([M.sc[:, tw, st][:, None].expand(nq, nw) for st in range(S)])
            out.append((M.iq, j, vec, listed[None, :].expand(nq, nw), A, B, el, sc, 2))
    # Q-Q pairs
    conn = M.qconn[0][M.iq].T
    upper = torch.ones(nq, nq, dtype=torch.bool, device=x.device).triu(1)
    c3 = conn == 4
    vec = x[M.iq][None, :, :] - x[M.iq][:, None, :]
    A, B, el, sc = [], [], [], []
    for st in range(S):
        a, b = qa[t[st]], qb[t[st]]
        A.append(torch.where(c3, a[:, None, 2] * a[None, :, 2], a[:, None, 0] * a[None, :, 0]))
        B.append(torch.where(c3, b[:, None, 2] * b[None, :, 2], b[:, None, 0] * b[None, :, 0]))
        el.append(qcrg[:, None, st] * qcrg[None, :, st] * torch.where(c3, s.el14_scale, 1.0))
        sc.append(M.sc[:, s.natyps:, st])
    out.append((M.iq, M.iq, vec, upper & (conn >= 4), torch.stack(A), torch.stack(B), torch.stack(el),
                torch.stack(sc), 0))
    return out


def _q_terms(M, x0, x, cut, box, lam, grad, qcrg=None, qa=None, qb=None):
    """Per-state Q energies [S, 6] = (qq, qp, qw) x (el, vdw); adds the
    lambda-weighted gradient when given."""
    s = M.s
    S = s.nstates
    E = [[0.0] * 6 for _ in range(S)]
    for i, j, vec, use, A, B, el, sc, kind in _q_pairs(M, x0, x, cut, box, M.qcrg if qcrg is None else qcrg,
                                                       M.qa if qa is None else qa, M.qb if qb is None else qb):
        d2 = torch.where(use, (vec * vec).sum(-1), 1.0)
        r2, w = 1.0 / d2, use.to(d2.dtype)
        d6 = d2 ** 3
        dvs = 0.0
        for st in range(S):
            r6 = 1.0 / (d6 + sc[st])
            vel, va, vb = el[st] * torch.sqrt(r2) * w, A[st] * r6 * r6 * w, B[st] * r6 * w
            E[st][2 * kind] = E[st][2 * kind] + vel.sum()
            E[st][2 * kind + 1] = E[st][2 * kind + 1] + (va - vb).sum()
            if grad is not None:
                dvs = dvs + r2 * (-vel - (12.0 * va - 6.0 * vb) * r6 * d6) * lam[st]
        if grad is not None:
            grad.index_add_(0, i, -torch.einsum("ij,ija->ia", dvs, vec))
            grad.index_add_(0, j, torch.einsum("ij,ija->ja", dvs, vec))
    return E


def _restraints(M, x, p, grad):
    """restrain_solvent and watpol (theta_corr 0)."""
    s = M.s
    ns, nw = s.nat_solute, s.nwat
    if nw == 0:
        return 0.0, 0.0
    o = ns + 3 * torch.arange(nw, device=x.device)
    wc = torch.as_tensor(s.xwcent).to(x)
    u = x[o] - wc
    b = u.norm(dim=1)
    db = b - (p.rwat - math.sqrt(p.boltz * TFREE / p.fk_wsphere))
    ex = torch.exp(p.awmz * torch.clamp(db, max=0.0))
    erad = torch.where(db > 0, 0.5 * p.fk_wsphere * db * db - p.Dwmz, p.Dwmz * (ex * ex - 2.0 * ex)).sum()
    dv = torch.where(db > 0, p.fk_wsphere * db / b, -2.0 * p.Dwmz * p.awmz * (ex - ex * ex) / b)
    grad[o] += u * dv[:, None]
    mu = x[o + 1] + x[o + 2] - 2.0 * x[o]
    rm = mu.norm(dim=1, keepdim=True)
    mu, rc, r = mu / rm, u / b[:, None], b[:, None]
    cos = torch.clamp((mu * rc).sum(1, keepdim=True), -1.0, 1.0)
    theta = torch.acos(cos[:, 0])
    n = p.nwpolr_shell
    shell = torch.full((nw,), -1, dtype=torch.int64, device=x.device)
    for k in range(n):   # the innermost shell whose outer radius holds the water, else the outermost
        shell = torch.where((b <= p.shell_rout[k]) | (k == 0), k, shell)
    shell = torch.where(b > p.shell_rout[n - 1] - p.shell_dr[n - 1], shell, -1)
    epol = 0.0
    for k in range(n):
        w = torch.nonzero(shell == k)[:, 0]
        if not len(w):
            continue
        w = w[torch.argsort(theta[w], stable=True)]
        il = torch.arange(1, len(w) + 1, device=x.device, dtype=x.dtype)
        t0 = torch.acos(1.0 + (1.0 - 2.0 * il) / len(w))
        t0 = torch.clamp(t0 - 1.5 * torch.sin(t0) * p.shell_cstb[k], 0.0, math.pi)
        dth = theta[w] - t0
        epol = epol + 0.5 * p.fkwpol * (dth * dth).sum()
        f0 = (-p.fkwpol * dth / torch.clamp(torch.sin(theta[w]), min=1e-10))[:, None]
        f3 = (rc[w] - mu[w] * cos[w]) / rm[w]
        f2 = (mu[w] - rc[w] * cos[w]) / r[w]
        grad[o[w]] += (f2 - 2.0 * f3) * f0
        grad[o[w] + 1] += f3 * f0
        grad[o[w] + 2] += f3 * f0
    return erad, epol


def exact(case, seed):
    if case["kind"] == "md":
        return None   # the trajectory of a whole MD cycle
    s, x0, x, lam = _inputs(case, seed)
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    M = _Model(s, dev)
    cut, box = _cuts(case, s), _box_edge(s) if case["box"] else 0.0
    W, S = case["windows"], s.nstates
    a0, a = torch.from_numpy(x0).to(dev), torch.from_numpy(x).to(dev)
    if case["kind"] == "adjoint":
        out = {k: np.zeros((W, s.nqat, S)) for k in ("dq", "dA", "dB")}
        for w in range(W):
            par = [v.clone().requires_grad_(True) for v in (M.qcrg, M.qa, M.qb)]
            E = _q_terms(M, a0[w], a[w], cut, box, lam[w], None, *par)
            for st in range(S):
                g = torch.autograd.grad(sum(E[st]), par, retain_graph=st + 1 < S)
                out["dq"][w, :, st] = g[0][:, st].cpu().numpy()
                out["dA"][w, :, st] = g[1][M.qt[:, st], 0].cpu().numpy()
                out["dB"][w, :, st] = g[2][M.qt[:, st], 0].cpu().numpy()
        return out
    p = default_solvent_params(s)
    chunk = max(32, int(4e7 / s.natom))
    grad = torch.zeros_like(a)
    E, EQ, R = np.zeros((W, 7)), np.zeros((W, S, 6)), np.zeros((W, 2))
    for w in range(W):
        E[w, :6] = _pairs(M, a0[w], a[w], cut, box, grad[w], chunk).cpu().numpy().ravel()
        E[w, 6] = float(_lrf_gradient(M, a0[w], a[w], cut, box, grad[w], max(16, chunk // 4)))
        EQ[w] = np.array([[float(v) for v in e] for e in _q_terms(M, a0[w], a[w], cut, box, lam[w], grad[w])])
        if not case["box"]:
            R[w] = [float(v) for v in _restraints(M, a[w], p, grad[w])]
    return {"gradient": grad[0] if case["kind"] == "host" else grad, "E": E, "EQ": EQ, "restraints": R}

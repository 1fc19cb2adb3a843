"""Timed workloads of the impurity solver, called as a user's program calls them.

A case is a dict of plain values; its "op" is one of

  product   H*v on one sector: the procedure-pointer contract on host vectors
            (dtype "c128"), or device vectors (dtype "f64" / "f32")
  solve     one impurity solve read back (G, Sigma, observables); nup < 0 scans
            every sector, nstates > 1 is finite temperature, loop adds the
            local Green's function and the Weiss field of a Bethe iteration
  chi2      chi^2 of the bath fit and its gradient for a batch of parameter sets
  fit       ed_chi2_fitgf: the conjugate-gradient bath fit of every orbital

The sizes are those of the repository's own configurations (single-orbital
Nbath = 7, 11, 13; two orbitals with four or five levels each; beta = 50 and
100; 4096 Matsubara points) and the doped, odd-sized and large sectors that a
DMFT run meets around them.  Baths are seeded: e_k ~ U[-1, 1] (U[-1.5, 1.5]
for two orbitals), V_k = 0.5 (0.4) + U[-0.1, 0.1].
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "dmft-ed_b200"))

import dmfted  # noqa: E402
from dmfted import bethe  # noqa: E402

LE = 500  # points of the semicircular density of states


def listed():
    return [
        # the plug-in product of a host program that owns its vectors (a
        # Fortran driver's ARPACK), smallest configuration: all latency
        dict(name="product_host_ns8", op="product", norb=1, nbath=7, nup=4, ndw=4, dtype="c128",
             u=2.0, jhflag=False),
        # device vectors, the doped sector of a mid-size bath: the rows of the
        # vector matrix are odd in number (1287 x 1716)
        dict(name="product_odd_ns13", op="product", norb=1, nbath=12, nup=5, ndw=6, dtype="f64",
             u=3.0, jhflag=False),
        # two orbitals: more hops per word than a single-orbital bath has
        dict(name="product_2orb_ns12", op="product", norb=2, nbath=5, nup=6, ndw=6, dtype="f64",
             u=3.0, jhflag=False),
        # the headline sector in the mixed form's vector precision
        dict(name="product_f32_ns14", op="product", norb=1, nbath=13, nup=7, ndw=7, dtype="f32",
             u=3.0, jhflag=False),
        # the largest sector one GPU serves in earnest: 12870 x 12870, 1.3 GB a vector
        dict(name="product_f64_ns16", op="product", norb=1, nbath=15, nup=8, ndw=8, dtype="f64",
             u=3.0, jhflag=False),
        # one iteration of the Bethe driver at the small configuration: every
        # sector at T=0, then Sigma, G_loc and the Weiss field
        dict(name="iteration_scan_ns8", op="solve", norb=1, nbath=7, nspin=1, nup=-1, ndw=-1,
             u=2.0, beta=100.0, precision="f64", nstates=1, lmats=4096, loop=True),
        # the middle configuration, one sector, mixed precision
        dict(name="solve_mixed_ns12", op="solve", norb=1, nbath=11, nspin=1, nup=6, ndw=6,
             u=3.0, beta=100.0, precision="mixed", nstates=1, lmats=4096, loop=False),
        # the FP64 drop-in between the two large configurations, away from half filling
        dict(name="solve_f64_ns13", op="solve", norb=1, nbath=12, nspin=1, nup=6, ndw=7,
             u=3.0, beta=100.0, precision="f64", nstates=1, lmats=4096, loop=False),
        # the headline configuration
        dict(name="solve_mixed_ns14", op="solve", norb=1, nbath=13, nspin=1, nup=7, ndw=7,
             u=3.0, beta=100.0, precision="mixed", nstates=1, lmats=4096, loop=False),
        # finite temperature, two orbitals, two spins: every sector, all chains
        dict(name="solve_thermal_ns10", op="solve", norb=2, nbath=4, nspin=2, nup=-1, ndw=-1,
             u=3.0, beta=50.0, precision="f64", nstates=16, lmats=4096, loop=False),
        # a multi-start bath fit's function and gradient
        dict(name="chi2_batch_4096", op="chi2", nbatch=4096, nbath=9, lfit=1000, beta=100.0),
        # the fit that closes each DMFT iteration
        dict(name="fit_ns8", op="fit", norb=1, nbath=7, beta=100.0, lfit=1000),
    ]


def _around(rng, ns):
    """Particle numbers of a sector at or near half filling."""
    return [min(ns - 1, max(1, ns // 2 + rng.choice((-2, -1, 0, 0, 1)))) for _ in range(2)]


def draw(rng):
    op = rng.choice(("product", "product", "solve", "solve", "chi2"))
    if op == "product":
        norb = rng.choice((1, 1, 2))
        nbath = rng.randint(6, 13) if norb == 1 else rng.randint(2, 5)
        nup, ndw = _around(rng, (nbath + 1) * norb)
        dtype = rng.choice(("f64", "f32", "c128")) if norb * (nbath + 1) < 13 else \
            rng.choice(("f64", "f32"))
        return dict(op=op, norb=norb, nbath=nbath, nup=nup, ndw=ndw, dtype=dtype,
                    u=round(rng.uniform(1.0, 4.0), 2), jhflag=norb == 2 and rng.random() < 0.5)
    if op == "solve":
        kind = rng.choice(("scan", "sector", "sector", "thermal"))
        case = dict(op=op, norb=1, nspin=1, u=round(rng.uniform(1.0, 4.0), 2), nstates=1,
                    beta=round(rng.uniform(40.0, 120.0), 1), loop=False,
                    lmats=rng.choice((512, 1000, 2048, 4096)))
        if kind == "scan":
            return dict(case, nbath=rng.randint(3, 7), nup=-1, ndw=-1, precision="f64", loop=True)
        if kind == "sector":
            nbath = rng.randint(6, 13)
            nup = ndw = (nbath + 1) // 2
            return dict(case, nbath=nbath, nup=nup, ndw=min(nbath, ndw + rng.randint(0, 1)),
                        precision=rng.choice(("f64", "mixed")))
        norb = rng.choice((1, 2))
        return dict(case, norb=norb, nbath=rng.randint(4, 7) if norb == 1 else rng.randint(2, 3),
                    nspin=rng.choice((1, 2)), nup=-1, ndw=-1, precision="f64", nstates=16,
                    beta=round(rng.uniform(20.0, 60.0), 1))
    return dict(op=op, nbatch=int(round(math.exp(rng.uniform(math.log(16), math.log(4096))))),
                nbath=rng.randint(3, 13), lfit=rng.randint(200, 1500), beta=100.0)


# ---------------------------------------------------------------- inputs ---
def _bath(case, seed):
    """(e[norb, nbath], V[norb, nbath]) of the case's bath."""
    rng = np.random.default_rng(seed)
    no, nb = case["norb"], case["nbath"]
    e = rng.uniform(-1.0, 1.0, (no, nb)) * (1.0 if no == 1 else 1.5)
    v = (0.5 if no == 1 else 0.4) + rng.uniform(-0.1, 0.1, (no, nb))
    return e, v


def _interaction(case):
    no, u = case["norb"], case["u"]
    kw = dict(uloc=[u] * no)
    if no > 1:
        kw.update(ust=u - 1.0, jh=0.5)
        if case.get("jhflag"):
            kw.update(jhflag=1, jx=0.5, jp=0.5)
    return kw


def _dim(case):
    ns = case["norb"] * (case["nbath"] + 1)
    return math.comb(ns, case["nup"]) * math.comb(ns, case["ndw"])


def _vector(case, seed):
    """The case's vector: CUDA for device types, a complex host array for "c128"."""
    n = _dim(case)
    if case["dtype"] == "c128":
        rng = np.random.default_rng(seed + 1)
        return rng.standard_normal(n) + 1j * rng.standard_normal(n)
    g = torch.Generator(device="cuda").manual_seed(seed + 1)
    dt = torch.float64 if case["dtype"] == "f64" else torch.float32
    return torch.randn(n, generator=g, device="cuda", dtype=dt)


def _chi2_inputs(case, seed):
    rng = np.random.default_rng(seed)
    nbath, L = case["nbath"], case["lfit"]
    wm = np.pi / case["beta"] * (2.0 * np.arange(1, L + 1) - 1.0)
    e = rng.uniform(-1.0, 1.0, nbath)
    v = 0.5 + rng.uniform(-0.1, 0.1, nbath)
    delta = (v ** 2 / (1j * wm[:, None] - e)).sum(axis=1)
    delta = delta + 1e-4 * (rng.normal(size=L) + 1j * rng.normal(size=L))
    a = np.concatenate([e, v]) + 0.05 * rng.normal(size=(case["nbatch"], 2 * nbath))
    return a, wm, delta, 1.0 / wm


def prepare(case, seed):
    op = case["op"]
    if op == "product":
        e, v = _bath(case, seed)
        s = dmfted.EDSolver(dmfted.default_params(
            norb=case["norb"], nbath=case["nbath"], beta=100.0, lmats=16, lreal=0,
            **_interaction(case)))
        s.set_bath(np.concatenate([e.reshape(-1), v.reshape(-1)]))
        s.setup_hv_sector(s.sector_index(case["nup"], case["ndw"]))
        x = _vector(case, seed)
        y = torch.empty_like(x) if case["dtype"] != "c128" else None
        return dict(case=case, solver=s, x=x, y=y)
    if op == "solve":
        e, v = _bath(case, seed)
        ns = case["nspin"]
        s = dmfted.EDSolver(dmfted.default_params(
            norb=case["norb"], nbath=case["nbath"], nspin=ns, beta=case["beta"],
            lmats=case["lmats"], lreal=0, lanc_nstates_total=case["nstates"],
            lanc_nstates_sector=1 if case["nup"] >= 0 else 6,
            precision=dmfted.MIXED if case["precision"] == "mixed" else dmfted.FP64,
            **_interaction(case)))
        bath = np.concatenate([e.reshape(-1)] * ns + [v.reshape(-1)] * ns)
        sectors = None if case["nup"] < 0 else [s.sector_index(case["nup"], case["ndw"])]
        return dict(case=case, solver=s, bath=bath, sectors=sectors, dos=bethe.bethe_dos(LE, 1.0))
    if op == "chi2":
        a, wm, delta, w = _chi2_inputs(case, seed)
        s = dmfted.EDSolver(dmfted.default_params(nbath=case["nbath"], lmats=16, lreal=0))
        dev = [torch.from_numpy(np.ascontiguousarray(t)).cuda()
               for t in (a, wm, delta.view(np.float64), w)]
        out = [torch.empty(a.shape[0], dtype=torch.float64, device="cuda"),
               torch.empty(a.shape, dtype=torch.float64, device="cuda")]
        return dict(case=case, solver=s, inputs=dev, out=out)
    # fit: the Weiss field of a bath twice as fine as the one fitted
    rng = np.random.default_rng(seed)
    no, nb, L = case["norb"], case["nbath"], case["lfit"]
    s = dmfted.EDSolver(dmfted.default_params(
        norb=no, nbath=nb, beta=case["beta"], lmats=L, lfit=L, lreal=0))
    z = 1j * np.pi / case["beta"] * (2.0 * np.arange(1, L + 1) - 1.0)
    fg = np.zeros((1, 1, no, no, L), np.complex128)
    for o in range(no):
        e = rng.uniform(-1.0, 1.0, 2 * nb)
        v = 0.35 + rng.uniform(-0.07, 0.07, 2 * nb)
        fg[0, 0, o, o] = 1.0 / (z - (v ** 2 / (z[:, None] - e)).sum(axis=1))
    start = np.concatenate([np.tile(np.linspace(-1.0, 1.0, nb), no), np.full(no * nb, 0.5)])
    return dict(case=case, solver=s, fg=fg, bath=start)


def run(state):
    case, s = state["case"], state["solver"]
    op = case["op"]
    if op == "product":
        if case["dtype"] == "c128":
            return s.hxv(state["x"])
        lib = dmfted.lib()
        f = lib.dmfted_hxv_device_f64 if case["dtype"] == "f64" else lib.dmfted_hxv_device_f32
        rc = f(s.ctx, state["x"].data_ptr(), state["y"].data_ptr(), 1)
        if rc != dmfted.OK:
            raise RuntimeError(lib.dmfted_last_error().decode())
        return state["y"]
    if op == "solve":
        s.ed_solve(state["bath"], sectors=state["sectors"])
        out = dict(egs=s.egs(), sigma=s.ed_get_sigma_matsubara(), **s.observables())
        if case["loop"]:
            out["gloc"] = s.gloc_matsubara_diag(*state["dos"], out["sigma"])
            out["weiss"] = s.get_weiss(out["gloc"], out["sigma"])
        else:
            out["gimp"] = s.ed_get_gimp_matsubara()
        if case["nstates"] > 1:
            energies, _, zeta = s.eigenspace()
            out.update(energies=energies, zeta=zeta)
        return out
    if op == "chi2":
        a, wm, delta, w = state["inputs"]
        chi2, grad = state["out"]
        lib = dmfted.lib()
        rc = lib.dmfted_chi2_delta_batch_device(
            s.ctx, case["nbatch"], case["nbath"], case["lfit"], a.data_ptr(), wm.data_ptr(),
            delta.data_ptr(), w.data_ptr(), chi2.data_ptr(), grad.data_ptr())
        if rc != dmfted.OK:
            raise RuntimeError(lib.dmfted_last_error().decode())
        return chi2, grad
    bath, steps, chi2 = s.ed_chi2_fitgf(state["fg"], state["bath"])
    return bath, steps, chi2


# ------------------------------------------------------------------ work ---
def _hops(case):
    """Hops per word and spin, about: each bath level differs from its
    impurity level in half of the words."""
    return case["norb"] * (case["nbath"] + 1) / 2.0


def work(case):
    op = case["op"]
    if op == "product":
        size = {"c128": 16, "f64": 8, "f32": 4}[case["dtype"]]
        n = _dim(case)
        return dict(bytes=2.0 * n * size,
                    flops=n * (4.0 * _hops(case) + 2.0) * (2 if case["dtype"] == "c128" else 1))
    if op == "solve":
        # a Lanczos step reads two vectors and writes one.  One sector: about
        # 100 ground-state steps and 2 x 200 chain steps; a scan: about 50
        # steps in each sector and the chains of the kept states
        ns = case["norb"] * (case["nbath"] + 1)
        size = 4 if case["precision"] == "mixed" else 8
        dims = [math.comb(ns, i) * math.comb(ns, j) for i in range(ns + 1) for j in range(ns + 1)]
        if case["nup"] >= 0:
            elements = _dim(case) * 500.0
        else:
            chains = 2 * case["norb"] * case["nspin"] * case["nstates"]
            elements = sum(dims) * 50.0 + max(dims) * 200.0 * chains
        return dict(bytes=3.0 * size * elements, flops=elements * (4.0 * _hops(case) + 8.0))
    if op == "chi2":
        n = case["nbatch"] * case["nbath"]
        return dict(bytes=8.0 * (4 * n + case["nbatch"] + 4 * case["lfit"]),
                    flops=25.0 * n * case["lfit"])
    # fit: tens of conjugate-gradient steps of some ten evaluations each
    n = case["norb"] * case["nbath"]
    return dict(bytes=8.0 * (4 * n + 4 * case["lfit"]), flops=400 * 15.0 * n * case["lfit"])


# ----------------------------------------------------------------- exact ---
def _words(ns, n):
    w = np.arange(1 << ns)
    bits = ((w[:, None] >> np.arange(ns)) & 1).sum(axis=1)
    return w[bits == n]


def _spin_operator(case, words, e, v):
    """(bath energy per word, [(rows, partner rows, amplitude)]) of one spin."""
    no, nb = case["norb"], case["nbath"]
    rank = {int(w): i for i, w in enumerate(words)}
    diag = np.zeros(words.size)
    hops = []
    for o in range(no):
        for k in range(nb):
            site = no + o * nb + k
            diag += e[o, k] * ((words >> site) & 1)
            rows = np.nonzero(((words >> o) ^ (words >> site)) & 1)[0]
            w = words[rows]
            partner = np.array([rank[int(t)] for t in w ^ (1 << o) ^ (1 << site)], np.int64)
            between = (w >> (o + 1)) & ((1 << (site - o - 1)) - 1)
            parity = np.array([bin(int(b)).count("1") & 1 for b in between])
            hops.append((rows, partner, v[o, k] * (1.0 - 2.0 * parity)))
    return diag, hops


def _sign(word, src, dst):
    """Sign of c^+_dst c_src on a word with src occupied and dst empty."""
    lo, hi = min(src, dst), max(src, dst)
    return 1.0 - 2.0 * (bin((int(word) >> (lo + 1)) & ((1 << (hi - lo - 1)) - 1)).count("1") & 1)


def _exact_product(case, seed):
    e, v = _bath(case, seed)
    no, ns = case["norb"], case["norb"] * (case["nbath"] + 1)
    wu, wd = _words(ns, case["nup"]), _words(ns, case["ndw"])
    du, hu = _spin_operator(case, wu, e, v)
    dd, hd = _spin_operator(case, wd, e, v)
    u = case["u"]
    ust, jh = (u - 1.0, 0.5) if no > 1 else (0.0, 0.0)
    nu = np.array([(wu >> a) & 1 for a in range(no)], float)
    nd = np.array([(wd >> a) & 1 for a in range(no)], float)
    x = _vector(case, seed)
    host = isinstance(x, np.ndarray)
    x = (torch.from_numpy(x).cuda() if host else x.double()).reshape(wd.size, wu.size)
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
    d = t(dd)[:, None] + t(du)[None, :]
    for a in range(no):
        d += u * t(nd[a] - 0.5)[:, None] * t(nu[a] - 0.5)[None, :]
        for b in range(a + 1, no):
            d += ust * (t(nd[b] - 0.5)[:, None] * t(nu[a] - 0.5)[None, :]
                        + t(nd[a] - 0.5)[:, None] * t(nu[b] - 0.5)[None, :])
            d += (ust - jh) * (t((nu[a] - 0.5) * (nu[b] - 0.5))[None, :]
                               + t((nd[a] - 0.5) * (nd[b] - 0.5))[:, None])
            # the constant of the repository's shift counts each pair once
            d -= 0.25 * ust + 0.25 * (ust - jh)
    y = d * x
    del d
    for rows, partner, amp in hu:
        y[:, t(rows)] += t(amp)[None, :] * x[:, t(partner)]
    for rows, partner, amp in hd:
        y[t(rows)] += t(amp)[:, None] * x[t(partner)]
    if case["jhflag"]:
        # spin exchange and pair hopping: one two-spin move per orbital pair
        ru = {int(w): i for i, w in enumerate(wu)}
        rd = {int(w): i for i, w in enumerate(wd)}

        def moves(words, rank, src, dst):
            at = [i for i, w in enumerate(words) if (w >> src) & 1 and not (w >> dst) & 1]
            to = [rank[int(words[i]) ^ (1 << src) ^ (1 << dst)] for i in at]
            return t(np.array(at, np.int64)), t(np.array(to, np.int64)), \
                t(np.array([_sign(words[i], src, dst) for i in at]))

        for a in range(no):
            for b in range(no):
                if a == b:
                    continue
                up, up_to, up_sign = moves(wu, ru, b, a)
                for src, dst, j in ((a, b, 0.5), (b, a, 0.5)):
                    dn, dn_to, dn_sign = moves(wd, rd, src, dst)
                    if len(up) and len(dn):
                        y[dn_to[:, None], up_to[None, :]] += (
                            j * dn_sign[:, None] * up_sign[None, :] * x[dn[:, None], up[None, :]])
    y = y.reshape(-1)
    return y.cpu().numpy() if host else y


def _exact_chi2(case, seed):
    a, wm, delta, w = (torch.from_numpy(np.ascontiguousarray(t)).cuda()
                       for t in _chi2_inputs(case, seed))
    nb = case["nbath"]
    chi2, grad = [], []
    for part in a.split(256):
        e, v = part[:, :nb, None], part[:, nb:, None]
        r = 1.0 / (1j * wm - e)
        res = delta - (v ** 2 * r).sum(dim=1)
        chi2.append((res.abs() ** 2 / w).sum(dim=1))
        conj = res.conj()[:, None, :] / w
        grad.append(torch.cat([-2.0 * (conj * v ** 2 * r * r).real.sum(dim=2),
                               -2.0 * (conj * 2.0 * v * r).real.sum(dim=2)], dim=1))
    return torch.cat(chi2), torch.cat(grad)


def exact(case, seed):
    if case["op"] == "product":
        return _exact_product(case, seed)
    if case["op"] == "chi2":
        return _exact_chi2(case, seed)
    return None

"""The work a user of this package has it do, as cases that can be timed.

A program that uses the package initialises one solver, keeps H_k in hand and
calls `solve` for one variational point after another; some programs pass a
batch of points, some apply the sector Hamiltonian to vectors of their own,
and most read Green's functions and self-energies after a solve.  The cases
are those calls at the sizes of this repository's configurations, tests and
benchmark.  The variational parameters, vectors and frequencies come from the
seed; the solver is initialised once per configuration and kept, as such a
program keeps it.
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch

from vca_gb300 import clusters
from vca_gb300.config import ARITH_AUTO, ARITH_FP64
from vca_gb300.solver import VcaSolver


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------
def _solve(model, nx, ny, nspin, nk, steps, nodes, lmats, **kw):
    """nx, ny: cluster sites per direction (a chain has ny = 1); nk: k-points
    per direction; nb: bath levels; symmetric: two-channel off-diagonal
    Green's functions; fp64: FP64 Lanczos vectors where fixed point would
    apply; nstates > 1: finite temperature with that list size."""
    c = {"kind": "solve", "model": model, "nx": nx, "ny": ny, "nspin": nspin, "nb": 0, "nk": nk, "steps": steps,
         "nodes": nodes, "lmats": lmats, "symmetric": 0, "fp64": 0, "nstates": 1, "points": 1}
    c.update(kw)
    return c


def _hxv(model, nx, ny, nspin, nup, ndw, cols, **kw):
    c = {"kind": "hxv", "model": model, "nx": nx, "ny": ny, "nspin": nspin, "nb": 0, "nup": nup, "ndw": ndw,
         "cols": cols, "permuted": 0, "fp64": 0}
    c.update(kw)
    return c


def _functions(nx, ny, nspin, nk, steps, lmats, nz, nw):
    return {"kind": "functions", "model": "square", "nx": nx, "ny": ny, "nspin": nspin, "nb": 0, "nk": nk,
            "steps": steps, "nodes": 512, "lmats": lmats, "symmetric": 0, "fp64": 0, "nstates": 1, "points": 1,
            "nz": nz, "nw": nw}


def listed():
    return [
        # a t' sweep of the 4-site chain: the smallest solve, all launches and latency
        dict(_solve("chain", 4, 1, 1, 64, 100, 4096, 512), name="solve_chain4"),
        # one call of a stationary-point search on the 2x2 plaquette (t', M, charge field)
        dict(_solve("square", 2, 2, 2, 8, 100, 512, 512), name="solve_square2x2"),
        # a Weiss-field sweep on a mid-size cluster (sectors up to 15,876 states)
        dict(_solve("square", 3, 3, 2, 16, 200, 4096, 512), name="solve_square3x3"),
        # the same cluster at finite temperature (Matsubara sum and contour)
        dict(_solve("square", 3, 3, 2, 8, 100, 256, 256, nstates=2), name="solve_square3x3_thermal"),
        # the two-orbital BHZ cluster: complex Hamiltonian, 48x48 k-points
        dict(_solve("bhz", 2, 2, 2, 48, 200, 4096, 256), name="solve_bhz"),
        # 2x2 cluster with 8 bath levels: FP64 vectors, dense one-body part, Delta(z)
        dict(_solve("bath", 2, 2, 1, 24, 200, 4096, 256, nb=8), name="solve_bath8"),
        # the 4x3 cluster, sectors up to 853,776 states, both spins alike, 100-step
        # chains: the large solve (the benchmark's point has four times its chain steps)
        dict(_solve("square", 4, 3, 1, 32, 100, 8192, 256), name="solve_square4x3"),
        # four BHZ points in one call: the batched form
        dict(_solve("bhz", 2, 2, 2, 48, 200, 4096, 256, points=4), name="batch_bhz"),
        # H x v with its Rayleigh numerators on the 408 particle-chain columns of the
        # 4x3 cluster, in the chains' layout
        dict(_hxv("square", 4, 3, 2, 7, 6, 408, permuted=1), name="hxv_columns_4x3"),
        # H x v on one vector of the half-filled 4x4 cluster (165,636,900 states)
        dict(_hxv("square", 4, 4, 1, 8, 8, 1), name="hxv_vector_4x4"),
        # H x v on 16 columns of a 4x4 chain sector (147,232,800 states each)
        dict(_hxv("square", 4, 4, 2, 9, 8, 16), name="hxv_columns_4x4"),
        # what a program reads after a solve: G' at its own points, the Omega
        # integrand, the self-energy grid and the observables
        dict(_functions(3, 2, 2, 16, 200, 2000, 5000, 1024), name="functions_3x2"),
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    largest = max(_cost(c) for c in listed())
    while True:
        c = _draw(rng)
        if _cost(c) <= 0.6 * largest and _fits(c):
            return c


def _draw(rng):
    what = rng.choices(["solve", "thermal", "bhz", "bath", "batch", "hxv", "functions"], [4, 1, 1, 1, 1, 3, 1])[0]
    steps, nodes = _log_int(rng, 30, 200), _log_int(rng, 512, 8192)
    if what == "solve":
        sym, fp64 = int(rng.random() < 0.25), int(rng.random() < 0.15)
        if rng.random() < 0.3:
            return _solve("chain", rng.randint(2, 6), 1, 1, _log_int(rng, 16, 128), steps, nodes,
                          _log_int(rng, 64, 1024), symmetric=sym, fp64=fp64)
        nx, ny = rng.choice([(2, 2), (3, 2), (4, 2), (3, 3), (5, 2), (4, 3)])
        if (nx, ny) == (4, 3):
            steps, fp64 = _log_int(rng, 20, 60), 0
        return _solve("square", nx, ny, rng.choice([1, 2]) if (nx, ny) != (4, 3) else 1, _log_int(rng, 4, 32),
                      steps, nodes, _log_int(rng, 64, 512), symmetric=sym, fp64=fp64)
    if what == "thermal":
        nx, ny = rng.choice([(2, 2), (3, 2), (4, 2), (3, 3)])
        return _solve("square", nx, ny, 2, _log_int(rng, 4, 16), _log_int(rng, 30, 100), 256, _log_int(rng, 64, 256),
                      nstates=2)
    if what == "bhz":
        return _solve("bhz", 2, 2, 2, _log_int(rng, 8, 48), steps, _log_int(rng, 512, 4096), _log_int(rng, 64, 256))
    if what == "bath":
        return _solve("bath", 2, 2, 1, _log_int(rng, 8, 24), steps, _log_int(rng, 512, 4096),
                      _log_int(rng, 64, 256), nb=rng.randint(2, 8))
    if what == "batch":
        if rng.random() < 0.5:
            return _solve("bhz", 2, 2, 2, _log_int(rng, 8, 24), steps, _log_int(rng, 512, 2048), 128,
                          points=rng.randint(2, 5))
        return _solve("bath", 2, 2, 1, _log_int(rng, 8, 16), steps, _log_int(rng, 512, 2048), 128,
                      nb=rng.randint(3, 6), points=rng.randint(2, 6))
    if what == "functions":
        nx, ny = rng.choice([(2, 2), (3, 2)])
        return _functions(nx, ny, rng.choice([1, 2]), _log_int(rng, 8, 32), steps, _log_int(rng, 200, 4000),
                          _log_int(rng, 100, 5000), _log_int(rng, 64, 2048))
    form = rng.choice(["columns", "few", "fp64", "bhz", "bath", "large"])
    if form == "large":
        return _hxv("square", 4, 4, 1, rng.choice([5, 6, 7, 8]), rng.choice([6, 7, 8]), 1)
    if form == "bhz":
        return _hxv("bhz", 2, 2, 2, rng.randint(2, 6), rng.randint(2, 6), 1)
    if form == "bath":
        nb = rng.randint(4, 8)
        return _hxv("bath", 2, 2, 1, (4 + nb) // 2, (4 + nb) // 2 + rng.choice([-1, 0, 1]), _log_int(rng, 1, 48),
                    nb=nb)
    nx, ny = rng.choice([(3, 3), (5, 2), (4, 3)])
    n = nx * ny
    up, dw = n // 2 + rng.choice([0, 1]), n // 2 - rng.choice([0, 1])
    if form == "fp64":
        return _hxv("square", nx, ny, 2, up, dw, _log_int(rng, 1, 48), fp64=1)
    if form == "few":
        return _hxv("square", nx, ny, 2, up, dw, rng.choice([1, 2, 3, 5, 7, 8]))
    return _hxv("square", nx, ny, 2, up, dw, 8 * _log_int(rng, 2, 51), permuted=rng.choice([0, 1]))


# ---------------------------------------------------------------------------
# sizes
# ---------------------------------------------------------------------------
def _orbitals(c):
    """Orbitals of one spin: of the cluster alone, and with the bath."""
    n = c["nx"] * c["ny"] * (2 if c["model"] == "bhz" else 1)
    return n, n + c["nb"]


def _pairs(c):
    """Directed one-body hops of one spin."""
    if c["model"] == "chain":
        return 2 * (c["nx"] - 1)
    nx, ny = c["nx"], c["ny"]
    bonds = (nx - 1) * ny + nx * (ny - 1)
    if c["model"] == "bhz":
        return 2 * bonds * 4 + nx * ny * 2
    return 2 * bonds + c["nb"] * (c["nb"] - 1) + 2 * c["nb"] * nx * ny


def _hops(c, n):
    """Mean hops of one configuration with n particles of one spin."""
    ns = _orbitals(c)[1]
    return _pairs(c) * n * (ns - n) / (ns * (ns - 1)) if ns > 1 else 0.0


def _columns(c):
    """Real (or complex) chain columns of one spin and one of particle | hole."""
    n = _orbitals(c)[0]
    off = n * (n - 1)
    if c["symmetric"]:
        return n + off
    return n + 2 * off if c["model"] == "bhz" else n + off + 2 * off


def _cost(c):
    w = work(c)
    return max(w["bytes"] / 1e12, w["flops"] / 0.5e12)


def _fits(c):
    # the batch's exact partial sums have to fit the product's static scratch, and
    # the chains' layout needs the up block in shared memory
    if c["kind"] != "hxv":
        return True
    ns = _orbitals(c)[1]
    return c["cols"] * math.comb(ns, c["ndw"]) * 16 <= 8 << 20 or ns > 12


def work(case):
    c = case
    norb, ns = _orbitals(c)
    cplx = c["model"] == "bhz"
    mac = 8 if cplx else 2  # operations of one multiply-add
    size = 16 if cplx else 8
    if c["kind"] == "hxv":
        d = math.comb(ns, c["nup"]) * math.comb(ns, c["ndw"])
        return {"bytes": 2.0 * size * d * c["cols"],
                "flops": mac * d * c["cols"] * (_hops(c, c["nup"]) + _hops(c, c["ndw"]) + 1.0)}
    n = norb * c["nspin"]  # matrix size of G', per frequency
    nk = c["nk"] if c["model"] == "chain" else c["nk"] ** 2
    blocks, nb = c["nspin"], norb
    lu = blocks * (8.0 / 3.0) * nb ** 3  # one complex determinant per k and frequency
    hk = 16.0 * n * n * nk
    # Green's function chains: their steps on the two target sectors next to the
    # half-filled one, which stream a vector in and out where it is larger than
    # an SM's shared memory
    half = ns // 2
    d = math.comb(ns, half) * math.comb(ns, min(ns, half + 1))
    steps = min(d, c["steps"])
    cols = 2 * c["nspin"] * _columns(c)
    hops = _hops(c, half) + _hops(c, min(ns, half + 1))
    chain_flops = cols * steps * mac * d * (hops + 5.0)
    chain_bytes = cols * steps * 2.0 * size * d if d * size > 227 * 1024 else 0.0
    if c["kind"] == "functions":
        # chain fractions per point and element, the integrand, one inversion per grid point
        per_z = cols * steps * 10.0
        return {"bytes": hk + 16.0 * n * n * (c["nz"] + c["lmats"]),
                "flops": (c["nz"] + c["nw"] + c["lmats"]) * per_z + c["nw"] * nk * lu + 16.0 * c["lmats"] * n ** 3}
    # ground-state search: every sector, about 40 steps each
    search = sum(min(40, math.comb(ns, u) * math.comb(ns, w)) * math.comb(ns, u) * math.comb(ns, w) *
                 (_hops(c, u) + _hops(c, w) + 5.0) for u in range(ns + 1) for w in range(ns + 1)) * mac
    omega = c["nodes"] * (nk * lu + cols * steps * 10.0)
    if c["nstates"] > 1:
        omega *= 2.0
    p = c["points"]
    return {"bytes": hk + p * chain_bytes + 16.0 * n * n * c["lmats"],
            "flops": p * (search + c["nstates"] * chain_flops + omega)}


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _point(c, rng):
    """One variational point of a case's model: a solve's arguments."""
    kw = dict(lanc_nstates_total=c.get("nstates", 1), vca_gf_symmetric=c.get("symmetric", 0),
              Lmats=c.get("lmats", 64), arith=ARITH_FP64 if c["fp64"] else ARITH_AUTO,
              ngfiter=c.get("steps", 100), omega_nodes=c.get("nodes", 512))
    if c.get("nstates", 1) > 1:
        kw.update(beta=20.0, bandwidth=8.0)
    if c["kind"] == "hxv":
        kw.update(hxv_variant=2 if c["permuted"] else 0)
    if c["model"] == "chain":
        return clusters.chain1d(tprime=rng.uniform(0.8, 1.2), nlat=c["nx"], nk=1, **kw)
    if c["model"] == "bath":
        return clusters.square_bath(s_h=rng.uniform(0.5, 1.5), s_v=rng.uniform(0.5, 1.5),
                                    mu_prime=rng.uniform(1.5, 2.5), nk1=1, nb=c["nb"], **kw)
    if c["model"] == "bhz":
        return clusters.bhz(mass=rng.uniform(1.5, 2.5), delta=rng.uniform(-0.2, 0.2), nk1=1, **kw)
    return clusters.square(nx=c["nx"], ny=c["ny"], nspin=c["nspin"], tprime=rng.uniform(0.9, 1.2),
                           maf=rng.uniform(0.05, 0.3), cdw=rng.uniform(0.02, 0.1), nkx=1, nky=1, **kw)


@functools.lru_cache(maxsize=4)
def _hk(model, nx, ny, nspin, nk):
    """H_k of the lattice, the same for every variational point."""
    if model == "chain":
        return clusters.chain1d(nlat=nx, nk=nk).Hk
    if model == "bhz":
        return clusters.bhz(nk1=nk).Hk
    return clusters.square(nx=nx, ny=ny, nspin=nspin, nkx=nk, nky=nk).Hk


class _Kept:
    """The one solver of the program: initialised when the configuration
    changes, with the fixed Hamiltonian of the cases that have one."""

    def __init__(self):
        self.key, self.solver = None, None

    def get(self, c):
        key = tuple(sorted((k, v) for k, v in c.items() if k not in ("name", "points", "nz", "nw", "cols")))
        if key != self.key:
            self.key = None
            pt = _point(c, np.random.default_rng(11))
            self.solver = VcaSolver(pt.cfg, pt.bath_h, pt.bath_v)
            if c["kind"] == "hxv":
                self.solver.set_hamiltonian(pt.Hloc, pt.bath_h, pt.bath_v)
            elif c["kind"] == "functions":
                self.solver.solve(pt.Hloc, _hk(c["model"], c["nx"], c["ny"], c["nspin"], c["nk"]))
            self.key = key
        return self.solver


_kept = _Kept()


def _vectors(c, d, seed):
    """Unit-norm random columns [d][cols] in FP64 (complex: [d][2])."""
    gen = torch.Generator(device="cuda").manual_seed(seed)
    w = 2 if c["model"] == "bhz" else c["cols"]
    x = torch.randn(d, w, dtype=torch.float64, device="cuda", generator=gen)
    return x.div_(torch.linalg.vector_norm(x) if w == 2 and c["cols"] == 1 else torch.linalg.vector_norm(x, dim=0))


def _slabs(x):
    """[d][m] -> slabs of 8 adjacent columns, the library's layout for 8 or more."""
    d, m = x.shape
    return x.reshape(d, m // 8, 8).permute(1, 0, 2).contiguous() if m >= 8 else x.contiguous()


def prepare(case, seed):
    c = case
    rng = np.random.default_rng(seed)
    s = _kept.get(c)
    if c["kind"] == "hxv":
        ns = _orbitals(c)[1]
        isector = 1 + c["ndw"] + c["nup"] * (ns + 1)
        d = math.comb(ns, c["nup"]) * math.comb(ns, c["ndw"])
        x = _vectors(c, d, seed)
        fx, scale, _ = s.arith_info()
        if fx:
            x = _slabs(x.mul_(2.0 ** scale).round_().to(torch.int64))
        alpha = torch.zeros(c["cols"], dtype=torch.float64, device="cuda")
        return {"case": c, "solver": s, "sector": isector, "x": x, "y": torch.zeros_like(x), "alpha": alpha}
    if c["kind"] == "functions":
        lo, hi = s.cfg.wini, s.cfg.wfin
        half = c["nz"] // 2
        z = np.concatenate([1j * np.exp(rng.uniform(np.log(0.01), np.log(100.0), half)),
                            np.sort(rng.uniform(lo, hi, c["nz"] - half)) + 0.1j])
        w = np.sort(np.exp(rng.uniform(np.log(1e-3), np.log(1e3), c["nw"])))
        return {"case": c, "solver": s, "z": z, "w": w}
    pts = [_point(c, rng) for _ in range(c["points"])]
    hk = _hk(c["model"], c["nx"], c["ny"], c["nspin"], c["nk"])
    st = {"case": c, "solver": s, "Hk": hk}
    if c["points"] == 1:
        st.update(Hloc=pts[0].Hloc, bath_h=pts[0].bath_h, bath_v=pts[0].bath_v)
    else:
        def cat(xs):
            return None if xs[0] is None else np.asfortranarray(np.stack(xs, axis=-1))
        st.update(Hloc=cat([p.Hloc for p in pts]), bath_h=cat([p.bath_h for p in pts]),
                  bath_v=cat([p.bath_v for p in pts]))
    return st


def run(state):
    c, s = state["case"], state["solver"]
    if c["kind"] == "hxv":
        x, y = state["x"], state["y"]
        if c["model"] == "bhz" or c["cols"] == 1:
            rc = s.L.vca_gpu_hxv_device(state["sector"], x.data_ptr(), y.data_ptr(), int(c["model"] == "bhz"))
            if rc:
                raise RuntimeError(f"vca_gpu_hxv_device: {rc}")
            return y
        s.hxv_alpha_noalloc(state["sector"], x.data_ptr(), y.data_ptr(), c["cols"], state["alpha"].data_ptr())
        return {"y": y, "alpha": state["alpha"]}
    if c["kind"] == "functions":
        return {"g": s.gf_cluster(state["z"]), "f": s.sum_kmesh(state["w"]), "sigma": s.sigma_matsubara(),
                **s.observables()}
    if c["points"] == 1:
        omega = s.solve(state["Hloc"], state["Hk"], state["bath_h"], state["bath_v"])
    else:
        omega = s.solve_batch(state["Hloc"], state["Hk"], state["bath_h"], state["bath_v"])
    egs, integral = s.energies()
    return {"omega": np.asarray(omega), "egs": np.asarray(egs), "integral": np.asarray(integral),
            "sectors": s.sector_energies(),
            "g": s.gimp_matsubara()}


# ---------------------------------------------------------------------------
# the same in 64 bits, by plain numpy and torch
# ---------------------------------------------------------------------------
def _words(ns, n):
    return np.array([w for w in range(1 << ns) if bin(w).count("1") == n], dtype=np.int64)


def _moves(words, a, b):
    """c+_a c_b on every word it does not annihilate: (to row, from row, sign)."""
    src = np.nonzero(((words >> b) & 1 == 1) & ((words >> a) & 1 == 0))[0]
    w = words[src]
    lo, hi = min(a, b), max(a, b)
    between = (w >> (lo + 1)) & ((1 << (hi - lo - 1)) - 1)
    sign = np.ones(len(w))
    for k in range(hi - lo - 1):
        sign *= 1.0 - 2.0 * ((between >> k) & 1)
    return np.searchsorted(words, w ^ (1 << a) ^ (1 << b)), src, sign


def _one_body(pt, spin):
    """The one-body matrix of one spin: cluster, bath and hybridisation, -xmu."""
    h = pt.Hloc[:, :, spin, spin]
    nl, norb = h.shape[0], h.shape[2]
    m = np.transpose(h, (0, 2, 1, 3)).reshape(nl * norb, nl * norb)
    if pt.bath_h is not None:
        bh, bv = pt.bath_h[:, :, spin, spin, 0, 0], pt.bath_v[:, :, spin, spin, 0, 0]
        m = np.block([[m, bv], [bv.conj().T, bh]])
    return m - pt.cfg.xmu * np.eye(len(m))


def _hop_list(words, m):
    """[(to, from, amplitude)] of the off-diagonal one-body part, and its diagonal."""
    hops = []
    for a in range(len(m)):
        for b in range(len(m)):
            if a != b and m[a, b] != 0.0:
                to, src, sign = _moves(words, a, b)
                if len(to):
                    hops.append((to, src, m[a, b] * sign))
    occ = (words[:, None] >> np.arange(len(m))) & 1
    return hops, occ @ np.diagonal(m).real


def _exact_hxv(c, seed):
    ns = _orbitals(c)[1]
    if c["model"] == "bhz" or (c["cols"] == 1 and not c["fp64"] and c["model"] != "bath"):
        return None  # (the two-orbital interaction; whole numbers)
    pt = _point(c, np.random.default_rng(11))
    up, dw = _words(ns, c["nup"]), _words(ns, c["ndw"])
    hu, eu = _hop_list(up, _one_body(pt, 0))
    hd, ed = _hop_list(dw, _one_body(pt, c["nspin"] - 1))
    x = _vectors(c, len(up) * len(dw), seed).reshape(len(dw), len(up), c["cols"])
    fixed = not c["fp64"] and c["model"] != "bath"
    if c["permuted"]:  # rows of the up role by decreasing hop count
        count = np.zeros(len(up), dtype=np.int64)
        for to, _, _ in hu:
            np.add.at(count, to, 1)
        perm = np.argsort(-count, kind="stable")
        back = np.empty_like(perm)
        back[perm] = np.arange(len(perm))
        hu = [(back[to], back[src], amp) for to, src, amp in hu]
        up, eu = up[perm], eu[perm]
    nl = c["nx"] * c["ny"]
    docc = np.zeros((len(dw), len(up)))
    for i in range(nl):
        docc += np.outer((dw >> i) & 1, (up >> i) & 1)

    def dev(v, kind=torch.float64):
        return torch.as_tensor(np.ascontiguousarray(v), dtype=kind, device="cuda")

    y = x * dev(ed[:, None] + eu[None, :] + pt.cfg.Uloc[0] * docc)[:, :, None]
    for to, src, amp in hd:
        y[dev(to, torch.int64)] += x[dev(src, torch.int64)] * dev(amp.real)[:, None, None]
    for to, src, amp in hu:
        y[:, dev(to, torch.int64)] += x[:, dev(src, torch.int64)] * dev(amp.real)[None, :, None]
    y = y.reshape(-1, c["cols"])
    if c["cols"] == 1:
        return y
    alpha = torch.einsum("dc,dc->c", x.reshape(-1, c["cols"]), y)
    return {"y": None if fixed else y, "alpha": alpha}


def _small_solve(c, pt):
    """Every sector of a small real cluster in dense form: energies, the
    ground states, and G'(z) per spin as a function."""
    ns = _orbitals(c)[1]
    m = [_one_body(pt, 0).real, _one_body(pt, c["nspin"] - 1).real]
    words = [_words(ns, n) for n in range(ns + 1)]
    one = []
    for spin in range(2):
        hs = []
        for n in range(ns + 1):
            hops, diag = _hop_list(words[n], m[spin])
            h = np.diag(diag)
            for to, src, amp in hops:
                np.add.at(h, (to, src), amp.real)
            hs.append(h)
        one.append(hs)

    @functools.lru_cache(maxsize=None)
    def sector(nu, nd):
        u, w = words[nu], words[nd]
        docc = np.zeros((len(u), len(w)))
        for i in range(c["nx"] * c["ny"]):
            docc += np.outer((u >> i) & 1, (w >> i) & 1)
        h = np.kron(one[0][nu], np.eye(len(w))) + np.kron(np.eye(len(u)), one[1][nd])
        return np.linalg.eigh(h + np.diag(pt.cfg.Uloc[0] * docc.reshape(-1)))

    energies = np.array([sector(nu, nd)[0][0] for nu in range(ns + 1) for nd in range(ns + 1)])
    e0 = energies.min()
    ground = [(k // (ns + 1), k % (ns + 1)) for k in range(len(energies)) if energies[k] < e0 + 1e-9]

    def ladder(n, dag):
        """c+_j (or c_j) between the words of n and n +- 1 particles of one spin."""
        out = []
        to = words[n + 1] if dag else words[n - 1]
        for j in range(_orbitals(c)[0]):
            a = np.zeros((len(to), len(words[n])))
            src = np.nonzero(((words[n] >> j) & 1) == (0 if dag else 1))[0]
            sign = np.ones(len(src))
            for k in range(j):
                sign *= 1.0 - 2.0 * ((words[n][src] >> k) & 1)
            a[np.searchsorted(to, words[n][src] ^ (1 << j)), src] = sign
            out.append(a)
        return out

    terms = {0: [], 1: []}  # per spin: (pole, residue vector)
    for nu, nd in ground:
        psi = sector(nu, nd)[1][:, 0].reshape(len(words[nu]), len(words[nd]))
        for spin in range(c["nspin"]):
            for dag in (True, False):
                n = (nu if spin == 0 else nd) + (1 if dag else -1)
                if n < 0 or n > ns:
                    continue
                tn = (n, nd) if spin == 0 else (nu, n)
                e, v = sector(*tn)
                phi = [(a @ psi if spin == 0 else psi @ a.T).reshape(-1) for a in ladder(nu if spin == 0 else nd, dag)]
                terms[spin].append(((e - e0) if dag else (e0 - e), v.T @ np.array(phi).T))

    def green(z, spin):
        g = 0.0
        for pole, q in terms[spin]:
            f = 1.0 / (np.asarray(z)[:, None] - pole[None, :])
            g = g + np.einsum("zn,na,nb->zab", f, q, q, optimize=True)
        return g / len(ground)

    docc_of = [(np.abs(sector(nu, nd)[1][:, 0].reshape(len(words[nu]), len(words[nd]))) ** 2, words[nu], words[nd])
               for nu, nd in ground]
    return energies, e0, green, docc_of


def _grid(c, z, green):
    """(Nlat,Nlat,Nspin,Nspin,1,1,nz) of a function of (z, spin)."""
    nl = _orbitals(c)[0]
    out = np.zeros((nl, nl, c["nspin"], c["nspin"], 1, 1, len(z)), dtype=np.complex128)
    for s in range(c["nspin"]):
        out[:, :, s, s, 0, 0, :] = np.moveaxis(green(z, s), 0, -1)
    return out


def _integrand(c, pt, hk, green, w):
    f = np.zeros(len(w))
    for s in range(c["nspin"]):
        mk = np.moveaxis(pt.Hloc[:, :, s, s, 0, 0, None] - hk[:, :, s, s, 0, 0, :], -1, 0)
        g = green(1j * w, s)
        eye = np.eye(g.shape[1])
        for i in range(0, len(w), 64):
            f[i:i + 64] += np.linalg.slogdet(eye + mk[None] @ g[i:i + 64, None])[1].mean(axis=1)
    return f


def exact(case, seed):
    c = case
    if c["kind"] == "hxv":
        return _exact_hxv(c, seed)
    if c["model"] not in ("chain", "square") or c["nx"] * c["ny"] > 6 or c["nstates"] > 1 or c["points"] > 1:
        return None  # many-second dense problems, the thermal list and the two-orbital interaction
    hk = _hk(c["model"], c["nx"], c["ny"], c["nspin"], c["nk"])
    if c["kind"] == "functions":
        state = prepare(c, seed)
        pt = _point(c, np.random.default_rng(11))
        _, _, green, rho = _small_solve(c, pt)
        wm = np.pi / pt.cfg.beta * (2 * np.arange(c["lmats"]) + 1)
        nl = _orbitals(c)[0]

        def sigma(z, s):
            h = _one_body(pt, s)  # holds -xmu
            return z[:, None, None] * np.eye(nl) - h - np.linalg.inv(green(z, s))

        up = sum(np.einsum("uw,ui->i", p, (u[:, None] >> np.arange(nl)) & 1) for p, u, _ in rho) / len(rho)
        dw = sum(np.einsum("uw,wi->i", p, (w[:, None] >> np.arange(nl)) & 1) for p, _, w in rho) / len(rho)
        dd = sum(np.einsum("uw,ui,wi->i", p, (u[:, None] >> np.arange(nl)) & 1, (w[:, None] >> np.arange(nl)) & 1)
                 for p, u, w in rho) / len(rho)
        obs = {"dens": up + dw, "dens_up": up, "dens_dw": dw, "docc": dd, "mag": up - dw}
        return {"g": _grid(c, state["z"], green), "f": _integrand(c, pt, hk, green, state["w"]),
                "sigma": _grid(c, 1j * wm, sigma), **{k: v.reshape(nl, 1) for k, v in obs.items()}}
    pt = _point(c, np.random.default_rng(seed))
    energies, e0, green, _ = _small_solve(c, pt)
    # composite Gauss-Legendre on w = s/(1-s), 48 panels of 16 nodes graded to s = 0
    x, wt = np.polynomial.legendre.leggauss(16)
    edge = np.linspace(0.0, 1.0, 49) ** 2
    half, mid = 0.5 * np.diff(edge), 0.5 * (edge[1:] + edge[:-1])
    s = (mid[:, None] + half[:, None] * x[None, :]).reshape(-1)
    wts = (half[:, None] * wt[None, :]).reshape(-1) / (1.0 - s) ** 2
    integral = (3.0 - c["nspin"]) / np.pi * float(wts @ _integrand(c, pt, hk, green, s / (1.0 - s)))
    wm = np.pi / pt.cfg.beta * (2 * np.arange(c["lmats"]) + 1)
    return {"omega": np.asarray(e0 - integral), "egs": np.asarray(e0), "integral": np.asarray(integral),
            "sectors": energies,
            "g": _grid(c, 1j * wm, green)}

"""Timed cases of the engine: the calls a user's program makes, over the sizes it makes them at.

A case is one call path (its "kind") on one Hamiltonian (its "model" and sizes):

  krylov   T_steps(H/a)|v>: the Chebyshev recurrence t_{k+1} = 2 (H/a) t_k - t_{k-1} on device
           vectors, as kernel-polynomial, filtering and time-propagation programs write it over
           to_native / mltply_device_async / from_native; returns the vector and <t_k|H|t_k>
  device   one v0 = H v1 on device vectors in HPhi's own order (mltply_device), the drop-in call
  lanczos  a fixed number of Lanczos steps (lanczos_steps), the ground-state driver's loop
  tpq      microcanonical TPQ of several samples (calc_by_tpq) with HPhi's output files
  tem      real-time evolution under a time-dependent Peierls phase (calc_by_tem)
  green    one- and two-body Green's functions of a device vector (expec_green_device)
  batch    Lanczos steps of many chains in one batch (Batch.lanczos)

Vectors are FP64 (real or complex); the batch also has its FP32 storage option.
"""
from __future__ import annotations

import math
import os
import tempfile

import numpy as np
import torch

import hphi_b200
from hphi_b200 import expert

DEV = "cuda" if torch.cuda.is_available() else "cpu"
F64, C128, I64 = torch.float64, torch.complex128, torch.int64
CHUNK = 1 << 25
U_HUBBARD, J_KONDO, TWIST = 8.0, 1.5, 0.3


def listed():
    return [
        # the smallest sector a user runs (tutorials, scans over many couplings): launches count
        dict(name="lanczos_chain16", kind="lanczos", model="chain", L=16, j2=0.0, steps=40),
        # an ordinary spin-chain sector whose vectors stay in L2
        dict(name="krylov_j1j2_24", kind="krylov", model="chain", L=24, j2=0.35, vec="real", steps=16),
        # the largest sector of this repository's benchmark: 601 M rows, 4.8 GB per vector
        dict(name="krylov_heisenberg4x8", kind="krylov", model="square", W=4, L=8, vec="real", steps=3),
        # the headline sector, half-filled 4x4 Hubbard, real vectors
        dict(name="krylov_hubbard4x4", kind="krylov", model="hubbard", W=4, L=4, nup=8, ndown=8, twist=0, vec="real",
             steps=6),
        # complex hoppings (twisted boundary / flux), complex vectors
        dict(name="krylov_hubbard14_twist", kind="krylov", model="hubbard", W=14, L=1, nup=7, ndown=7, twist=1,
             vec="complex", steps=8),
        # no conserved Sz: Kitaev-Heisenberg honeycomb, complex vectors as HPhi's default start gives them
        dict(name="krylov_kitaev24", kind="krylov", model="kitaev", W=4, L=3, vec="complex", steps=8),
        # Kondo lattice: the general row kernel with crossing terms
        dict(name="krylov_kondo8", kind="krylov", model="kondo", L=8, vec="real", steps=12),
        # HPhi's row order in and out, doped Hubbard
        dict(name="device_hubbard4x4_6e", kind="device", model="hubbard", W=4, L=4, nup=6, ndown=6, twist=0,
             vec="real"),
        # finite temperature: 5 samples, HPhi's default NumAve
        dict(name="tpq_j1j2_22", kind="tpq", model="chain", L=22, j2=0.35, steps=30, samples=5),
        # pulse on a Hubbard cluster, Taylor order 10 as standard mode writes it
        dict(name="tem_hubbard3x4", kind="tem", model="hubbard", W=3, L=4, nup=6, ndown=6, twist=0, steps=8),
        # all one-body and density / spin-flip two-body functions of a ground-state sized vector
        dict(name="green_hubbard14", kind="green", model="hubbard", W=14, L=1, nup=7, ndown=7, twist=0, vec="real"),
        # coupling scan: many short chains at once
        dict(name="batch_j1j2_32", kind="batch", lo=14, hi=20, members=32, steps=48, fp32=0),
    ]


def draw(rng):
    def between(a, b):  # whole numbers spread over their logarithm
        return int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))

    kind = rng.choice(["krylov"] * 5 + ["device", "lanczos", "tpq", "tem", "green", "batch"])
    if kind == "lanczos":
        return dict(kind=kind, model="chain", L=rng.randint(13, 24), j2=rng.choice([0.0, 0.35, 0.6]), steps=between(24, 44))
    if kind == "tpq":
        return dict(kind=kind, model="chain", L=rng.randint(16, 23), j2=rng.choice([0.0, 0.35]), steps=between(10, 40),
                    samples=rng.randint(1, 8))
    if kind == "batch":
        lo = rng.randint(12, 17)
        return dict(kind=kind, lo=lo, hi=lo + rng.randint(1, 5), members=between(4, 48), steps=between(96, 128),
                    fp32=rng.randint(0, 1))
    if kind in ("tem", "green"):
        n = rng.randint(9, 12) if kind == "tem" else rng.randint(10, 14)
        c = dict(kind=kind, model="hubbard", W=n, L=1, nup=rng.randint(n // 3, n // 2), ndown=rng.randint(n // 3, n // 2),
                 twist=0)
        return dict(c, steps=rng.randint(3, 10)) if kind == "tem" else dict(c, vec=rng.choice(["real", "complex"]))
    steps = dict(steps=rng.randint(2, 12)) if kind == "krylov" else {}
    what = "hubbard" if kind == "device" else rng.choice(["chain", "square", "hubbard", "hubbard", "kitaev", "kondo", "spin1"])
    vec = rng.choice(["real", "complex"])
    if what == "chain":
        return dict(kind=kind, model=what, L=rng.randint(17, 28), j2=rng.choice([0.0, 0.35]), vec=vec, **steps)
    if what == "square":
        W, L = rng.choice([(3, 7), (5, 5), (4, 6), (3, 9), (4, 7), (3, 10)])
        return dict(kind=kind, model=what, W=W, L=L, vec=vec, **steps)
    if what == "hubbard":
        W, L = rng.choice([(11, 1), (13, 1), (14, 1), (15, 1), (3, 4), (3, 5), (4, 4)])
        n = W * L
        twist = rng.randint(0, 1) if n < 15 else 0
        return dict(kind=kind, model=what, W=W, L=L, nup=rng.randint(n // 4, n // 2), ndown=rng.randint(n // 4, n // 2),
                    twist=twist, vec="complex" if twist else vec, **steps)
    if what == "kitaev":
        W, L = rng.choice([(3, 3), (3, 4), (4, 3), (5, 2)])
        return dict(kind=kind, model=what, W=W, L=L, vec=vec, **steps)
    return dict(kind=kind, model=what, L=rng.randint(5, 8) if what == "kondo" else rng.randint(9, 14), vec=vec, **steps)


# ------------------------------------------------------------------ Hamiltonians
def _bonds(case):
    """(i, j, J) of a spin lattice, or (i, j, phase winds) of a Hubbard one; site = x + W*y."""
    m = case["model"]
    if m in ("chain", "spin1"):
        L = case["L"]
        out = [(i, (i + 1) % L, 1.0) for i in range(L)]
        if case.get("j2"):
            out += [(i, (i + 2) % L, case["j2"]) for i in range(L)]
        return out
    W, L = case["W"], case["L"]
    out = []
    for y in range(L):
        for x in range(W):
            out.append((x + W * y, (x + 1) % W + W * y, 1.0 if m == "square" else float(x + 1 == W)))
            if L > 1:
                out.append((x + W * y, x + W * ((y + 1) % L), 1.0 if m == "square" else 0.0))
    return out


def _hops(case):
    """(i, j, t) of a Hubbard lattice: H += -t c+_i c_j, both directions listed."""
    out = []
    for i, j, wind in _bonds(case):
        t = complex(math.cos(TWIST), math.sin(TWIST)) if (case["twist"] and wind) else complex(1.0, 0.0)
        out += [(i, j, t), (j, i, t.conjugate())]
    return out


def _sites(case):
    m = case["model"]
    if m in ("chain", "spin1"):
        return case["L"]
    if m == "kondo":
        return 2 * case["L"]
    return case["W"] * case["L"] * (2 if m == "kitaev" else 1)


def _kitaev_bonds(case):
    W, L = case["W"], case["L"]
    out = []
    for y in range(L):
        for x in range(W):
            a = 2 * (x + W * y)
            out += [(a, a + 1, 0), (a + 1, 2 * ((x + 1) % W + W * y), 1), (a + 1, 2 * (x + W * ((y + 1) % L)), 2)]
    return out


def _model(case, **kw):
    m, n = case["model"], _sites(case)
    kw.setdefault("initial_vec_type", 0 if case.get("vec") == "complex" else 1)
    if m in ("chain", "square"):
        b = _bonds(case)
        return expert.heisenberg(n, [(i, j) for i, j, _ in b], [J for _, _, J in b], two_sz=n % 2, **kw)
    if m == "hubbard":
        h = expert.hubbard(n, [], 1.0, U_HUBBARD, case["nup"], case["ndown"], **kw)
        h.trans = [(i, s, j, s, t.real, t.imag) for i, j, t in _hops(case) for s in (0, 1)]
        return h
    if m == "kitaev":
        return expert.kitaev_heisenberg(case["W"], case["L"], -1.0, 0.3, **kw)
    if m == "kondo":
        return expert.kondo_chain(case["L"], 1.0, J_KONDO, ncond=case["L"], two_sz=0, **kw)
    return expert.general_heisenberg([2] * n, [(i, j) for i, j, _ in _bonds(case)], 1.0, two_sz=0, **kw)


def _dim(case):
    m, n = case["model"], _sites(case)
    if m in ("chain", "square"):
        return math.comb(n, n // 2)
    if m == "hubbard":
        return math.comb(n, case["nup"]) * math.comb(n, case["ndown"])
    if m == "kitaev":
        return 1 << n
    if m == "kondo":  # L conduction electrons and L local spins, total Sz 0
        L = case["L"]
        return sum(math.comb(L, u) * math.comb(L, L - u) * math.comb(L, L - u) for u in range(L + 1))
    return sum(math.comb(n, u) * math.comb(n - u, u) for u in range(n // 2 + 1))


def _elements(case):
    """Off-diagonal matrix elements of H per row, on average."""
    m, n = case["model"], _sites(case)
    if m in ("chain", "square"):
        return len(_bonds(case)) * 0.5 * n / (n - 1)
    if m == "hubbard":
        return sum(2 * len(_bonds(case)) * k * (n - k) / (n * (n - 1)) for k in (case["nup"], case["ndown"]))
    if m == "kitaev":
        return 1.0 * len(_kitaev_bonds(case))
    return 2.0 * case["L"] if m == "kondo" else 1.3 * n


def _norm_bound(case):
    """A bound on |H| (the sum over the terms), the scale of the Chebyshev recurrence."""
    m, n = case["model"], _sites(case)
    if m in ("chain", "square"):
        return sum(0.75 * J for _, _, J in _bonds(case))
    if m == "hubbard":
        return 2.0 * len(_bonds(case)) + 0.5 * U_HUBBARD * n
    if m == "kitaev":
        return 0.75 * len(_kitaev_bonds(case))
    return 4.0 * case["L"] if m == "kondo" else 2.0 * n


# ------------------------------------------------------------------ the calls
def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed))


def _start(case, seed, dim):
    dt = C128 if case.get("vec") == "complex" else F64
    v = torch.randn(dim, dtype=dt, device=DEV, generator=_gen(seed))
    return v / torch.linalg.vector_norm(v)


def _host_starts(case, seed, dim, count):
    """Normal start vectors in HPhi's host layout (element 0 unused)."""
    v = np.zeros((count, dim + 1), dtype=np.complex128)
    v[:, 1:] = torch.randn(count, dim, dtype=F64, device=DEV, generator=_gen(seed)).cpu().numpy()
    return v / np.linalg.norm(v, axis=1, keepdims=True)


def _tem_rows(case):
    """TEOneBody rows per time index: every hop t -> t e^{+-iA}, A = 0.5 sin 4t, dt = 0.01."""
    out = []
    for k in range(case["steps"]):
        a = 0.5 * math.sin(4.0 * 0.01 * k)
        rows = []
        for i, j, t in _hops(case):
            p = t * complex(math.cos(a), math.sin(a) if i < j else -math.sin(a))
            rows += [(i, s, j, s, p.real, p.imag) for s in (0, 1)]
        out.append((0.01 * k, rows))
    return out


def _green_rows(case):
    n = _sites(case)
    one = [(i, s, j, s) for i in range(n) for j in range(n) for s in (0, 1)]
    two = [(i, s, i, s, j, t, j, t) for i in range(n) for j in range(n) for s in (0, 1) for t in (0, 1)]
    two += [(i, 0, i, 1, j, 1, j, 0) for i in range(n) for j in range(n) if i != j]
    return one, two


def _members(case):
    n = case["members"]
    return [dict(model="chain", L=case["lo"] + i % (case["hi"] - case["lo"] + 1), j2=0.05 + 0.5 * i / n)
            for i in range(n)]


def _open(model, keep):
    d = tempfile.TemporaryDirectory()
    keep.append(d)
    return hphi_b200.Hamiltonian(model.write(d.name)), d.name


def prepare(case, seed):
    kind, keep = case["kind"], []
    st = dict(case=case, keep=keep, seed=int(seed) % (1 << 31))
    if kind == "batch":
        st["H"] = [_open(_model(m), keep)[0] for m in _members(case)]
        st["batch"] = hphi_b200.Batch(st["H"], hphi_b200.FP32 if case["fp32"] else hphi_b200.FP64)
        return st
    kw = {}
    if kind == "tpq":
        kw = dict(calc_type="TPQ", lanczos_max=case["steps"], num_ave=case["samples"], large_value=2.0)
    elif kind == "tem":
        kw = dict(calc_type="TimeEvolution", lanczos_max=case["steps"], input_eigenvec=1, expand_coef=10,
                  spectrum_vec="zvo_eigenvec_0")
    model = _model(case, **kw)
    if kind == "tem":
        model.trans, model.te_onebody = [], _tem_rows(case)
    H, folder = _open(model, keep)
    st["H"], st["out"] = H, os.path.join(folder, "output")
    st["vt"] = hphi_b200.COMPLEX128 if case.get("vec") == "complex" else hphi_b200.REAL64
    if kind == "krylov":
        a = _norm_bound(case)
        st["v"] = _start(case, seed, H.dim)
        st["buf"] = [torch.empty_like(st["v"]) for _ in range(3)]
        st["coef"] = torch.tensor([[0.0, 1.0 / a], [-1.0, 2.0 / a]], dtype=F64, device=DEV)
        st["mu"] = torch.zeros(case["steps"], 2, dtype=F64, device=DEV)
    elif kind == "device":
        st["v"] = _start(case, seed, H.dim)
        st["buf"] = torch.empty_like(st["v"])
    elif kind == "green":
        st["v"] = _start(case, seed, H.dim)
        st["rows"] = [np.array(r, dtype=np.int32) for r in _green_rows(case)]
    elif kind in ("tpq", "tem"):
        st["starts"] = list(_host_starts(case, seed, H.dim, case.get("samples", 1)))
    return st


def run(state):
    case, H = state["case"], state["H"]
    kind = case["kind"]
    if kind == "krylov":
        vt, (a, b, out), coef, mu = state["vt"], state["buf"], state["coef"], state["mu"]
        H.to_native(state["v"].data_ptr(), a.data_ptr(), vt)
        for k in range(case["steps"]):
            H.mltply_device_async(b.data_ptr(), a.data_ptr(), vt, coef[min(k, 1)].data_ptr(), mu[k].data_ptr())
            a, b = b, a
        H.from_native(a.data_ptr(), out.data_ptr(), vt)
        return {"t": out, "mu": mu}
    if kind == "device":
        p = H.mltply_device(state["buf"].data_ptr(), state["v"].data_ptr(), state["vt"], acc=0.0, scale=1.0)
        return {"v0": state["buf"], "prdct": [p.real, p.imag]}
    if kind == "lanczos":
        return H.lanczos_steps(case["steps"], seed=state["seed"], nev=4)
    if kind == "tpq":
        return H.calc_by_tpq(v_init=state["starts"], output_dir=state["out"])
    if kind == "tem":
        return H.calc_by_tem(v_init=state["starts"][0], output_dir=state["out"])
    if kind == "green":
        one, two = state["rows"]
        return {"one": H.expec_green_device(state["v"].data_ptr(), state["vt"], one, 1),
                "two": H.expec_green_device(state["v"].data_ptr(), state["vt"], two, 2)}
    r = state["batch"].lanczos(case["steps"], seed=state["seed"], refine=bool(case["fp32"]))
    return {k: r[k] for k in (["e_lanczos", "e_refined"] if case["fp32"] else ["e_lanczos"])}


def work(case):
    """Each H*v reads its source once and updates its target; HPhi-order conversions, the vector
    reads of the Green's functions; operations are multiply-adds of the matrix elements."""
    kind = case["kind"]
    if kind == "batch":
        es, ms = (4 if case["fp32"] else 8), _members(case)
        return {"bytes": case["steps"] * sum(3 * _dim(m) * es for m in ms),
                "flops": case["steps"] * sum(2 * _dim(m) * (_elements(m) + 3) for m in ms)}
    dim = _dim(case)
    cx = case.get("vec") == "complex" or kind == "tem"
    es, fl = (16, 8 if case.get("twist") or kind == "tem" else 4) if cx else (8, 2)
    if kind == "green":
        one, two = _green_rows(case)
        return {"bytes": dim * es, "flops": fl * dim * 0.25 * (len(one) + len(two))}
    nhv = {"krylov": case.get("steps", 1), "device": 1, "lanczos": case.get("steps", 1),
           "tpq": case.get("steps", 1) * case.get("samples", 1), "tem": 10 * case.get("steps", 1)}[kind]
    per = dim * es * (2 if kind == "device" else 3)
    extra = 4 * dim * es if kind == "krylov" else 0
    return {"bytes": nhv * per + extra, "flops": nhv * fl * dim * (_elements(case) + 2)}


def tolerance(case):
    if case["kind"] == "batch" and case["fp32"]:
        return {"rel": 1e-6, "max": 1e-6}
    return {"rel": 1e-12, "max": 1e-10}  # 64-bit sums; <t|H|t> cancels to a small value


# ------------------------------------------------------------------ 64-bit values in plain torch
def _pop(x):
    x = x - ((x >> 1) & 0x5555555555555555)
    x = (x & 0x3333333333333333) + ((x >> 2) & 0x3333333333333333)
    x = (x + (x >> 4)) & 0x0F0F0F0F0F0F0F0F
    return ((x * 0x0101010101010101) >> 56) & 0x7F


def _words(n, k):
    """All n-bit words with k ones, increasing."""
    w = torch.arange(1 << n, dtype=I64, device=DEV)
    return w[_pop(w) == k]


def _spread(x, n):
    out = torch.zeros_like(x)
    for i in range(n):
        out |= ((x >> i) & 1) << (2 * i)
    return out


class _Spin:
    """Spin-1/2 lattices: rows are configurations in increasing order, found through two half tables."""

    def __init__(self, case):
        n, gc = _sites(case), case["model"] == "kitaev"
        if gc:
            K, J = -1.0, 0.3
            self.terms = [(i, j, J + (K if g == 2 else 0.0), 0.5 * J + (0.25 * K if g != 2 else 0.0),
                           0.25 * K * (1 if g == 0 else -1 if g == 1 else 0)) for i, j, g in _kitaev_bonds(case)]
        else:
            self.terms = [(i, j, J, 0.5 * J, 0.0) for i, j, J in _bonds(case)]
        self.n, self.gc, self.dim = n, gc, _dim(case)
        if gc:
            return
        self.lb, k = (n + 1) // 2, (n + n % 2) // 2
        lo, hi = (torch.arange(1 << b, dtype=I64, device=DEV) for b in (self.lb, n - self.lb))
        pl, ph = _pop(lo), _pop(hi)
        self.lo_rank = torch.zeros_like(lo)
        for q in range(self.lb + 1):
            self.lo_rank[pl == q] = torch.arange(int((pl == q).sum()), device=DEV)
        size = torch.tensor([math.comb(self.lb, k - q) if 0 <= k - q <= self.lb else 0 for q in range(n + 1)],
                            device=DEV)[ph]
        self.hi_off = torch.cumsum(size, 0) - size
        self.c = torch.empty(self.dim, dtype=torch.int32 if n < 32 else I64, device=DEV)
        need = k - ph
        for q in range(self.lb + 1):
            rows, words = hi[need == q], lo[pl == q]
            if len(rows) == 0:
                continue
            for r0 in range(0, len(rows), max(1, CHUNK // len(words))):
                r = rows[r0:r0 + max(1, CHUNK // len(words))]
                at = self.hi_off[r][:, None] + torch.arange(len(words), device=DEV)[None, :]
                self.c[at.reshape(-1)] = ((r[:, None] << self.lb) | words[None, :]).reshape(-1).to(self.c.dtype)

    def words(self, a, b):
        return torch.arange(a, b, dtype=I64, device=DEV) if self.gc else self.c[a:b].to(I64)

    def apply(self, x):
        y = torch.empty_like(x)
        for a in range(0, self.dim, CHUNK):
            b = min(self.dim, a + CHUNK)
            c = self.words(a, b)
            acc, diag = torch.zeros_like(x[a:b]), torch.zeros(b - a, dtype=F64, device=DEV)
            one = torch.ones((), dtype=F64, device=DEV)
            for i, j, jz, jx, jp in self.terms:
                same = ((c >> i) ^ (c >> j)) & 1 == 0
                diag += torch.where(same, 0.25 * jz * one, -0.25 * jz * one)
                t = c ^ ((1 << i) | (1 << j))
                if self.gc:
                    row = t
                else:  # equal spins leave the sector: their row is not used
                    row = torch.where(same, c[0] * 0, self.lo_rank[t & ((1 << self.lb) - 1)] + self.hi_off[t >> self.lb])
                acc += torch.where(same, jp * one, jx * one) * x[row]
            y[a:b] = diag * x[a:b] + acc
        return y

    def hashed(self, seed):
        return _hashed(seed, self.words(0, self.dim).cpu().numpy())


class _Hubbard:
    """(up, down) occupation matrix in the basis with all up modes before all down ones; sigma is
    the sign to HPhi's interleaved modes (bit 2i + s)."""

    def __init__(self, case):
        n = _sites(case)
        self.n, self.dim = n, _dim(case)
        self.u, self.d = _words(n, case["nup"]), _words(n, case["ndown"])
        self.shape = (len(self.u), len(self.d))
        self.hops = _hops(case)
        self.cx = bool(case["twist"])
        su, sd = _spread(self.u, n), _spread(self.d, n) << 1
        self.order = torch.argsort((su[:, None] | sd[None, :]).reshape(-1))
        par = torch.zeros(self.shape, dtype=I64, device=DEV)
        for i in range(n):
            par ^= ((self.d >> i) & 1)[None, :] * (_pop(self.u >> (i + 1)) & 1)[:, None]
        self.sigma = (1.0 - 2.0 * (par & 1)).to(F64)
        self.docc = U_HUBBARD * torch.stack([_pop(r & self.d) for r in self.u]).to(F64)
        self.matrices()

    def matrices(self, phase=0.0):
        self.tu, self.td = (self.hop_matrix(w, [(i, j, -t * complex(math.cos(phase), math.sin(phase if i < j else -phase)))
                                                for i, j, t in self.hops]) for w in (self.u, self.d))

    def one_body(self, words, i, j):
        """(rows, sources, signs) of c+_i c_j on one species."""
        rank = torch.zeros(1 << self.n, dtype=I64, device=DEV)
        rank[words] = torch.arange(len(words), device=DEV)
        if i == j:
            at = torch.nonzero((words >> i) & 1).reshape(-1)
            return at, at, torch.ones(len(at), dtype=F64, device=DEV)
        at = torch.nonzero(((words >> i) & 1 == 0) & ((words >> j) & 1 == 1)).reshape(-1)  # sources
        w = words[at]
        lo, hi = min(i, j), max(i, j)
        sign = 1.0 - 2.0 * (_pop(w & ((1 << hi) - (1 << (lo + 1)))) & 1).to(F64)
        return rank[w ^ ((1 << i) | (1 << j))], at, sign

    def hop_matrix(self, words, hops):
        cx = self.cx or any(t.imag for _, _, t in hops)
        r, c, v = [], [], []
        for i, j, t in hops:
            a, b, s = self.one_body(words, i, j)
            r.append(a), c.append(b), v.append(s * t if cx else s * t.real)
        return torch.sparse_coo_tensor(torch.stack([torch.cat(r), torch.cat(c)]), torch.cat(v),
                                       (len(words), len(words))).coalesce().to_sparse_csr()

    def matrix(self, x):
        m = torch.empty_like(x)
        m[self.order] = x
        return m.reshape(self.shape) * self.sigma

    def vector(self, m):
        return (m * self.sigma).reshape(-1)[self.order]

    def product(self, m):
        def times(t, z):
            if z.is_complex() and not t.is_complex():
                return torch.complex(t @ z.real.contiguous(), t @ z.imag.contiguous())
            return t @ z
        return self.docc * m + times(self.tu, m) + times(self.td, m.T.contiguous()).T

    def apply(self, x):
        return self.vector(self.product(self.matrix(x)))


class _Strings:
    """Kondo chain by ladder operators on bits 2i + s, spin-1 chain by base-3 digits; rows found by search."""

    def __init__(self, case):
        self.spin1, L, n = case["model"] == "spin1", case["L"], _sites(case)
        if self.spin1:
            c, m = torch.zeros(1, dtype=I64, device=DEV), torch.zeros(1, dtype=I64, device=DEV)
            for i in range(n):
                c = torch.cat([c + d * 3 ** i for d in range(3)])
                m = torch.cat([m + d - 1 for d in range(3)])
                keep = m.abs() <= n - 1 - i
                c, m = c[keep], m[keep]
            self.c, self.bonds = torch.sort(c).values, [(i, j) for i, j, _ in _bonds(case)]
        else:
            cond = torch.cat([(_spread4(_words(L, u))[:, None] | (_spread4(_words(L, L - u)) << 1)[None, :]).reshape(-1)
                              for u in range(L + 1)])
            loc = torch.arange(1 << L, dtype=I64, device=DEV)  # bit set: down
            loc = ((_spread4(loc ^ ((1 << L) - 1))) | (_spread4(loc) << 1)) << 2
            c = torch.cat([(loc | x)[_pop((loc | x) & 0x5555555555555555) == L] for x in cond])
            self.c, self.L = torch.sort(c).values, L
        self.dim = len(self.c)

    def string(self, x, y, ops, coef):
        """y += coef * (product of ladder operators, the last one first) x; ops: (mode, creates)."""
        ok, w = torch.ones_like(self.c, dtype=torch.bool), self.c.clone()
        par = torch.zeros_like(w)
        for mode, creates in reversed(ops):
            ok &= ((w >> mode) & 1) == (0 if creates else 1)
            par ^= _pop(w & ((1 << mode) - 1))
            w = w ^ (1 << mode)
        src = torch.nonzero(ok).reshape(-1)
        row = torch.searchsorted(self.c, w[src])
        y.index_add_(0, row, coef * (1.0 - 2.0 * (par[src] & 1)) * x[src])

    def apply(self, x):
        y = torch.zeros_like(x)
        if self.spin1:
            digit = [torch.div(self.c, 3 ** i, rounding_mode="floor") % 3 for i in range(len(self.bonds))]
            for i, j in self.bonds:
                y += ((digit[i] - 1) * (digit[j] - 1)) * x
                for p, q in ((i, j), (j, i)):  # S+_p S-_q / 2, each raising or lowering gives sqrt 2
                    src = torch.nonzero((digit[p] < 2) & (digit[q] > 0)).reshape(-1)
                    y.index_add_(0, torch.searchsorted(self.c, self.c[src] + 3 ** p - 3 ** q), x[src])
            return y
        L = self.L
        for k in range(L):
            a, b = 4 * k, 4 * ((k + 1) % L)
            for s in (0, 1):
                self.string(x, y, [(a + s, 1), (b + s, 0)], -1.0)
                self.string(x, y, [(b + s, 1), (a + s, 0)], -1.0)
            e, l = 4 * k, 4 * k + 2
            sz = [((self.c >> q) & 1) - ((self.c >> (q + 1)) & 1) for q in (e, l)]
            y += (0.25 * J_KONDO) * (sz[0] * sz[1]) * x
            self.string(x, y, [(l, 1), (l + 1, 0), (e + 1, 1), (e, 0)], 0.5 * J_KONDO)
            self.string(x, y, [(l + 1, 1), (l, 0), (e, 1), (e + 1, 0)], 0.5 * J_KONDO)
        return y


def _spread4(x):
    out = torch.zeros_like(x)
    for i in range(12):
        out |= ((x >> i) & 1) << (4 * i)
    return out


def _hamiltonian(case):
    return {"hubbard": _Hubbard, "kondo": _Strings, "spin1": _Strings}.get(case["model"], _Spin)(case)


def _hashed(seed, config):
    """The documented start vector of lanczos_steps and Batch.lanczos: a 64-bit mix of seed and configuration."""
    with np.errstate(over="ignore"):
        x = np.uint64(seed) * np.uint64(0x9E3779B97F4A7C15) + (config.astype(np.uint64) * np.uint64(2) + np.uint64(1)) * np.uint64(0xD1B54A32D192ED03)
        x = (x ^ (x >> np.uint64(30))) * np.uint64(0xBF58476D1CE4E5B9)
        x = (x ^ (x >> np.uint64(27))) * np.uint64(0x94D049BB133111EB)
        x ^= x >> np.uint64(31)
    v = torch.from_numpy((x >> np.uint64(11)).astype(np.float64) / 9007199254740992.0 - 0.5).to(DEV)
    return v / torch.linalg.vector_norm(v)


def _ritz(H, seed, steps):
    """Eigenvalues of the Lanczos matrix after `steps` steps from the hashed start vector."""
    q, p, al, be = H.hashed(seed), None, [], []
    for _ in range(steps):
        w = H.apply(q)
        al.append(float(torch.dot(q, w)))
        w -= al[-1] * q
        if p is not None:
            w -= be[-1] * p
        be.append(float(torch.linalg.vector_norm(w)))
        p, q = q, w / be[-1]
    return np.linalg.eigvalsh(np.diag(al) + np.diag(be[:-1], 1) + np.diag(be[:-1], -1))


def _exact_green(case, H, v):
    """One-body functions from the density matrices of the two species, two-body ones from the
    weights and, for the spin flips, element by element."""
    m = H.matrix(v)
    one, two = _green_rows(case)
    rho = (m.conj() @ m.T, m.T.conj().contiguous() @ m)  # rho[a, b] = sum conj(m_a) m_b
    words, w = (H.u, H.d), (m.conj() * m).real
    g1 = []
    for i, s, j, _ in one:
        r, c, sg = H.one_body(words[s], i, j)
        g1.append((sg * rho[s][r, c]).sum())
    occ = [torch.stack([((x >> i) & 1).to(F64) for i in range(H.n)]) for x in words]
    wu, wd = w.sum(1), w.sum(0)
    nn = [[(occ[0] * wu) @ occ[0].T, occ[0] @ w @ occ[1].T], [None, (occ[1] * wd) @ occ[1].T]]
    nn[1][0] = nn[0][1].T
    g2 = []
    for i, s, j, t, k, x, l, z in two:
        if s == t:
            g2.append(nn[s][x][i, k])
            continue
        # c+_{i up} c_{i dn} c+_{k dn} c_{k up} = - (c+_i c_k)_up (c_i c+_k)_dn; c_i c+_k = -c+_k c_i
        ru, cu, su = H.one_body(H.u, i, k)
        rd, cd, sd = H.one_body(H.d, k, i)
        g2.append((su[:, None] * sd[None, :] * m[ru][:, rd].conj() * m[cu][:, cd]).sum() * -1.0)
    return {k: torch.stack([torch.as_tensor(x, device=DEV).to(C128) for x in g]).cpu().numpy()
            for k, g in (("one", g1), ("two", g2))}


def exact(case, seed):
    kind = case["kind"]
    if kind == "batch":
        if case["fp32"]:  # 32-bit vectors over many steps: the refined values are the converged ones only
            return None
        return {"e_lanczos": np.array([_ritz(_Spin(m), int(seed) % (1 << 31) + 1000003 * i, case["steps"])[0]
                                       for i, m in enumerate(_members(case))])}
    H = _hamiltonian(case)
    if kind == "lanczos":
        return _ritz(H, int(seed) % (1 << 31), case["steps"])[:4]
    if kind == "krylov":
        a, t0 = _norm_bound(case), _start(case, seed, H.dim)
        mu = torch.zeros(case["steps"], 2, dtype=F64, device=DEV)
        prev = None
        for k in range(case["steps"]):
            h = H.apply(t0)
            mu[k, 0] = torch.vdot(t0, h).real
            h *= (2.0 if k else 1.0) / a
            if k:
                h -= prev
            prev, t0 = t0, h
        return {"t": t0, "mu": mu}
    if kind == "device":
        v = _start(case, seed, H.dim)
        h = H.apply(v)
        return {"v0": h, "prdct": [float(torch.vdot(v, h).real), 0.0]}
    if kind == "green":
        return _exact_green(case, H, _start(case, seed, H.dim))
    starts = _host_starts(case, seed, H.dim, case.get("samples", 1))[:, 1:]
    out = []
    if kind == "tpq":  # the energies of the last sample
        v = torch.from_numpy(starts[-1].real.copy()).to(DEV)
        for _ in range(case["steps"]):
            v = v / torch.linalg.vector_norm(v)
            h = H.apply(v)
            out.append(float(torch.dot(v, h)))
            v = 2.0 * v - h / _sites(case)
        return np.array(out)
    # time evolution: the first Taylor term uses the previous index's H psi (zero before the first)
    m = H.matrix(torch.from_numpy(starts[0]).to(DEV))
    hm = torch.zeros_like(m)
    for k in range(case["steps"]):
        H.matrices(0.5 * math.sin(4.0 * 0.01 * k))
        if k:
            acc, t, c = m - 0.01j * hm, hm, -0.01j
            for q in range(2, 11):
                c *= -0.01j / q
                t = H.product(t)
                acc = acc + c * t
            m = acc
        m = m / torch.linalg.vector_norm(m)
        hm = H.product(m)
        out.append(float(torch.vdot(m.reshape(-1), hm.reshape(-1)).real))
    return np.array(out)

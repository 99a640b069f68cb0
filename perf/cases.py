"""Timed cases of the Kohn-Sham hot path, through the public Context calls.

Each case is a dict of plain values: the silicon supercell (r1 x r2 x r3
diamond cells, per-axis strain s1..s3), the wavefunction cutoff (Ry; the
density cutoff is four times that, as in every workload of this repository),
the number of bands, the context precision and the options of its kind:

  hpsi        H|psi> of all bands: the call inside every CG step, and the
              unit in which the hot path is quoted (band applications / s)
  subspace    H_sub, its diagonalisation and the rotation of psi and H psi
  ortho       Gram-Schmidt and the charge density of the new wavefunctions
  cg          one CG eigensolver sweep (all bands at once, or the one-rank
              order of the reference in which each band sees the final ones
              below it)
  scf         one whole SCF iteration from given wavefunctions and density
  batch       one SCF iteration of several independent small cells, each on
              its own stream
  md          the per-geometry work of an MD step: projector tables, local
              potential and forces at the new atom positions

The geometry belongs to the case and is kept for the process; wavefunctions,
densities and displacements come from the seed.
"""
import functools
import math
import random

import numpy as np
import torch

from qxmd_b200 import cell
from qxmd_b200.lib import (CgParm, Context, QX_HPSI_KINETIC, QX_HPSI_NONLOCAL, QX_NL_GSPACE, QX_NL_RSPACE,
                           QX_PREC_FP64, QX_PREC_MIXED)

PP = cell.ModelPP()


def _case(name, kind, reps, ecut, nb, prec="mixed", strain=(1.0, 1.0, 1.0), **kw):
    c = dict(kind=kind, r1=reps[0], r2=reps[1], r3=reps[2], s1=strain[0], s2=strain[1], s3=strain[2], ecut=ecut,
             nb=nb, prec=prec, **kw)
    if name:
        c["name"] = name
    return c


def listed():
    s8, s64, s512 = (1, 1, 1), (2, 2, 2), (4, 4, 4)
    return [
        # the smallest call: a unit cell, where launches and latency count
        _case("hpsi_si8", "hpsi", s8, 12.0, 16, nl="g"),
        # the 64-atom production cell of the benchmark, projectors in G space
        _case("hpsi_si64", "hpsi", s64, 16.0, 160, nl="g"),
        # the same with real-space projectors, QXMD's default for silicon
        _case("hpsi_si64_rspace", "hpsi", s64, 16.0, 160, nl="r"),
        # the plain drop-in: everything in FP64
        _case("hpsi_si64_fp64", "hpsi", s64, 16.0, 160, prec="fp64", nl="g"),
        # the largest: 512 atoms, 1100 bands, 96^3 grid
        _case("hpsi_si512", "hpsi", s512, 12.0, 1100, nl="g"),
        # the dense FP64 part of an iteration: subspace diagonalisation ...
        _case("subspace_si64", "subspace", s64, 16.0, 160),
        # ... and orthonormalisation, with the density that follows it
        _case("ortho_si64", "ortho", s64, 16.0, 160),
        # one CG sweep, all bands at once
        _case("cg_si64", "cg", s64, 16.0, 160, sequential=0),
        # the drop-in's CG in the reference's one-rank band order
        _case("cg_si64_fp64_one_rank", "cg", s64, 16.0, 160, prec="fp64", sequential=1),
        # the headline: a whole SCF iteration of the 64-atom cell
        _case("scf_si64", "scf", s64, 16.0, 160),
        # eight uneven small cells side by side (active-learning batches)
        _case("batch_8_cells", "batch", s8, 12.0, 20, cells=8, first=100),
        # an MD step's geometry tables and forces
        _case("md_si64", "md", s64, 16.0, 160),
    ]


def draw(rng):
    kind = rng.choice(["hpsi", "hpsi", "hpsi", "subspace", "ortho", "cg", "cg", "scf", "batch", "md"])
    reps = rng.choice([(1, 1, 1), (2, 1, 1), (2, 2, 1), (2, 2, 2)])
    strain = tuple(round(rng.uniform(0.97, 1.03), 4) for _ in range(3)) if rng.random() < 0.5 else (1.0, 1.0, 1.0)
    ecut = round(rng.uniform(9.0, 16.0), 2)
    nocc = 16 * reps[0] * reps[1] * reps[2]
    nb = min(160, nocc + rng.randint(0, max(16, nocc // 4)))
    prec = rng.choice(["mixed", "mixed", "fp64"])
    if kind == "hpsi":
        return _case(None, kind, reps, ecut, nb, prec, strain, nl=rng.choice(["g", "g", "r"]))
    if kind == "cg":
        return _case(None, kind, reps, ecut, nb, prec, strain, sequential=1 if prec == "fp64" and rng.random() < 0.7 else 0)
    if kind == "batch":
        return _case(None, kind, (1, 1, 1), 12.0, 20, "mixed", cells=rng.randint(2, 8), first=rng.randint(200, 10000))
    return _case(None, kind, reps, ecut, nb, prec, strain)


# ---- the cell and what a program holds for it ------------------------------

def _cell_key(case):
    return (case["r1"], case["r2"], case["r3"], case["s1"], case["s2"], case["s3"], case["ecut"])


@functools.lru_cache(maxsize=64)
def _sphere(key):
    r, s, ecut = key[:3], key[3:6], key[6]
    c = cell.diamond_si(r, seed=sum(r), strain=s)
    return c, cell.strvec(c.rba, ecut, 4.0 * ecut)


@functools.lru_cache(maxsize=64)
def _tables(key, real):
    """Local potential, G-space projectors (None above Si64, where the device
    builds them) and, when asked for, real-space projectors."""
    c, gs = _sphere(key)
    vloc = cell.vloc_grid(gs, c, PP)
    kb_g, vcl = cell.kb_tables_g(gs, c, PP) if c.natom <= 64 else (None, None)
    if real:
        kb_r = cell.kb_tables_r(gs, c, PP)
    else:
        kb_r = cell.KBReal(off=np.arange(c.natom + 1, dtype=np.int32), mesh=np.zeros(c.natom, dtype=np.int32),
                           vnl=np.zeros((c.natom, 4)), clalp=np.zeros(4), rdelv=gs.rvol / gs.kfft0)
    return vloc, kb_g, vcl, kb_r


def _system(case):
    key = _cell_key(case)
    c, gs = _sphere(key)
    vloc, kb_g, vcl, kb_r = _tables(key, case.get("nl") == "r")
    if kb_g is None:
        kb_g, vcl = np.zeros((gs.nplwex, 1)), np.zeros(1)
    return cell.System(cell=c, gs=gs, pp=PP, nband=case["nb"], occ=cell.occupations(case["nb"], c.nel), vloc=vloc,
                       kb_g=kb_g, vclalp=vcl, kb_r=kb_r, eewald=0.0)


def _context(case, stream=0):
    s = _system(case)
    ctx = Context(s, QX_PREC_FP64 if case["prec"] == "fp64" else QX_PREC_MIXED,
                  QX_NL_RSPACE if case.get("nl") == "r" else QX_NL_GSPACE, stream=stream)
    if s.cell.natom > 64:
        b = cell.kb_builder_tables(s.gs, s.cell, PP)
        ctx.set_kb_builder(b)
        ctx.build_kb_g(b["ityp"], b["satm"])
    return s, ctx


def _dev():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _dtype(case):
    return torch.float64 if case["prec"] == "fp64" else torch.float32


class _Array:
    """A context array for torch; keeps the context alive as long as the tensor."""

    def __init__(self, ctx, ptr, n, dtype):
        self.ctx = ctx
        self.__cuda_array_interface__ = {"shape": (n,), "typestr": "<f8" if dtype == torch.float64 else "<f4",
                                         "data": (int(ptr), False), "version": 3}


def _view(state, which, n, dtype):
    """A context array as a tensor (kept per pointer: psi, H psi and the
    rotation buffer change places)."""
    p = state["ctx"].dev_ptr(which)
    v = state["views"].get(p)
    if v is None or v.numel() != n:
        v = state["views"][p] = torch.as_tensor(_Array(state["ctx"], p, n, dtype), device="cuda")
    return v


def _weights(ne, dev):
    """Gamma-point metric: <x|y> = 2 sum x y - x_0 y_0 (x_1 = 0)."""
    w = torch.full((ne,), 2.0, dtype=torch.float64, device=dev)
    w[0] = 1.0
    return w


def _psi(gs, nb, seed, orthonormal=True):
    """Random wavefunctions that fall off with |G|^2 as those of an SCF run
    do, (nb, nplwex) FP64."""
    dev = _dev()
    g = torch.Generator(device=dev).manual_seed(1000 + int(seed))
    x = torch.rand((nb, gs.nplwex), generator=g, dtype=torch.float64, device=dev) - 0.5
    x[:, 1] = 0.0
    x /= 1.0 + torch.as_tensor(gs.dkgnrm(), device=dev) ** 2 / 4.0
    w = _weights(gs.nplwex, dev)
    if not orthonormal:
        return x / ((x * x) @ w).sqrt()[:, None]
    return torch.linalg.solve_triangular(torch.linalg.cholesky((x * w) @ x.T), x, upper=False).contiguous()


def _batch_cells(case):
    """The uneven cells of a batch: 8, 16 or 32 atoms, strained, cutoffs of 10
    to 16 Ry, 0 to 16 empty bands."""
    out = []
    for i in range(case["cells"]):
        r = random.Random(case["first"] + i)
        reps = r.choice([(1, 1, 1), (2, 1, 1), (2, 2, 1)])
        strain = tuple(round(r.uniform(0.97, 1.03), 4) for _ in range(3))
        nocc = 16 * reps[0] * reps[1] * reps[2]
        out.append(_case(None, "scf", reps, r.choice([10.0, 12.0, 14.0, 16.0]), min(80, nocc + r.randint(0, 16)),
                         "mixed", strain))
    return out


def _noband(s):
    return min(s.nband, int(s.cell.nel // 2))


def _moved(s, seed):
    """Fractional coordinates after a step of about 0.05 bohr."""
    rng = np.random.default_rng(7000 + int(seed))
    pos = s.cell.pos + rng.uniform(-0.05, 0.05, s.cell.pos.shape)
    return pos, np.ascontiguousarray(np.linalg.solve(s.gs.rba, pos.T).T)


def _scf_inputs(s, seed):
    psi = _psi(s.gs, s.nband, seed)
    return psi, _Exact(s).density(psi)


def prepare(case, seed):
    if case["kind"] == "batch":
        parts = []
        for k, c in enumerate(_batch_cells(case)):
            st = torch.cuda.Stream()
            parts.append(_prepare_scf(c, seed + 1000003 * k, st))
        torch.cuda.synchronize()
        return {"kind": "batch", "parts": parts}
    if case["kind"] == "scf":
        st = _prepare_scf(case, seed, None)
        torch.cuda.synchronize()
        return st
    s, ctx = _context(case)
    dt = _dtype(case)
    st = {"kind": case["kind"], "ctx": ctx, "sys": s, "views": {}, "dtype": dt}
    n = s.nband * s.gs.nplwex
    if case["kind"] == "hpsi":
        st["c"] = _psi(s.gs, s.nband, seed).to(dt)
        st["hc"] = torch.empty_like(st["c"])
    elif case["kind"] == "subspace":
        psi = _psi(s.gs, s.nband, seed)
        st["psi"], st["hpsi"] = psi.to(dt).reshape(n), _Exact(s, case).hpsi(psi).to(dt).reshape(n)
    elif case["kind"] == "ortho":
        st["psi"] = _psi(s.gs, s.nband, seed, orthonormal=False).to(dt).reshape(n)
        ctx.softchg()   # allocates the density
    elif case["kind"] == "cg":
        psi, hpsi = _Exact(s, case).ritz(_psi(s.gs, s.nband, seed))
        st["psi"], st["hpsi"] = psi.to(dt).reshape(n), hpsi.to(dt).reshape(n)
        st["parm"] = CgParm.defaults(_noband(s), sequential=case["sequential"])
    elif case["kind"] == "md":
        _view(st, 0, n, dt).copy_(_psi(s.gs, s.nband, seed).to(dt).reshape(n))
        b = cell.kb_builder_tables(s.gs, s.cell, PP)
        ctx.set_kb_builder(b)
        ctx.set_kb_r_builder(cell.kbr_builder_tables(s.gs, s.cell, PP))
        ctx.scf_init()
        ctx.set_force_tables()
        st["ityp"] = b["ityp"]
        st["satm"] = _moved(s, seed)[1]
    torch.cuda.synchronize()
    return st


def _prepare_scf(case, seed, stream):
    s, ctx = _context(case, stream.cuda_stream if stream else 0)
    psi, rho = _scf_inputs(s, seed)
    ctx.scf_init(mixbeta=0.8, kerker_q0=0.8)
    return {"kind": "scf", "ctx": ctx, "sys": s, "views": {}, "dtype": _dtype(case), "stream": stream,
            "psi": psi.to(_dtype(case)).reshape(-1), "rho": rho, "parm": CgParm.defaults(_noband(s))}


# ---- one pass ---------------------------------------------------------------

def _load(st, hpsi=False):
    n = st["psi"].numel()
    _view(st, 0, n, st["dtype"]).copy_(st["psi"])
    if hpsi:
        _view(st, 1, n, st["dtype"]).copy_(st["hpsi"])


def _start_scf(st):
    ctx = st["ctx"]
    if st["stream"] is not None:
        with torch.cuda.stream(st["stream"]):
            _load(st)
            _view(st, 2, st["rho"].numel(), torch.float64).copy_(st["rho"])
    else:
        _load(st)
        _view(st, 2, st["rho"].numel(), torch.float64).copy_(st["rho"])
    ctx.scf_mixing(10, 20.0)   # the reference's Pulay mixing, history restarted
    ctx.scf_launch(st["parm"])


def _end_scf(st):
    out = st["ctx"].scf_result()
    n, nr = st["psi"].numel(), st["rho"].numel()
    return {"energies": np.array([out[k] for k in ("etot", "eband", "ehartree", "exc", "evxc")]), "resid": np.array([out["resid"]]),
            "psi": _view(st, 0, n, st["dtype"]), "eig": _view(st, 4, st["sys"].nband, torch.float64),
            "rho_out": _view(st, 3, nr, torch.float64), "rho_next": _view(st, 2, nr, torch.float64)}


def run(st):
    kind = st["kind"]
    if kind == "batch":
        for p in st["parts"]:
            _start_scf(p)
        return [_end_scf(p) for p in st["parts"]]
    if kind == "scf":
        _start_scf(st)
        return _end_scf(st)
    ctx, nb, dt = st["ctx"], st["sys"].nband, st["dtype"]
    if kind == "hpsi":
        ctx.hpsi_dev(st["c"].data_ptr(), st["hc"].data_ptr(), nb, QX_HPSI_KINETIC | QX_HPSI_NONLOCAL)
        return st["hc"]
    if kind == "md":
        ctx.build_kb_g(st["ityp"], st["satm"])
        ctx.build_kb_r(st["ityp"], st["satm"])
        ctx.build_vloc()
        floc, fnl = ctx.forces()
        return {"vloc": _view(st, 5, st["sys"].gs.kfft0, torch.float64), "floc": floc, "fnl": fnl,
                "fnl_r": ctx.forces_nl_r()}
    n = st["psi"].numel()
    if kind == "subspace":
        _load(st, hpsi=True)
        hm = ctx.hmatrix()
        ev = ctx.untryt()
        ctx.untryhc()
        return {"hsub": hm, "ev": ev, "psi": _view(st, 0, n, dt), "hpsi": _view(st, 1, n, dt)}
    if kind == "ortho":
        _load(st)
        ctx.schmidt()
        ctx.softchg()
        return {"psi": _view(st, 0, n, dt), "rho": _view(st, 3, st["sys"].gs.kfft0, torch.float64)}
    _load(st, hpsi=True)
    ctx.ekinetic()
    iters, _ = ctx.eigen(st["parm"])
    return {"psi": _view(st, 0, n, dt), "hpsi": _view(st, 1, n, dt), "eig": _view(st, 4, nb, torch.float64),
            "iters": iters}


# ---- the same in 64 bits ------------------------------------------------------

class _Exact:
    """The path's equations in plain torch FP64 on the cell's tables."""

    def __init__(self, s, case=None):
        self.s, self.dev = s, _dev()
        t = lambda a: torch.as_tensor(np.ascontiguousarray(a), device=self.dev)   # noqa: E731
        gs = s.gs
        self.n, self.ng = gs.kfft0, gs.nplw + 1
        self.ip, self.im = t(gs.ijk_pos[: self.ng]).long(), t(gs.ijk_neg[1: self.ng]).long()
        self.dk, self.w, self.vloc = t(gs.dkgnrm()), _weights(gs.nplwex, self.dev), t(s.vloc)
        self.real = bool(case) and case.get("nl") == "r"
        if self.real:
            kr = s.kb_r
            self.mesh = t(kr.mesh).long()
            at = np.repeat(np.arange(s.cell.natom), np.diff(kr.off))
            self.at, self.vnl, self.cl, self.rdelv = t(at).long(), t(kr.vnl), t(kr.clalp), kr.rdelv
        elif s.cell.natom <= 64:
            self.kb, self.vcl = t(s.kb_g), t(s.vclalp)
        else:
            self.kb, self.vcl = self.projectors(t(s.cell.pos))

    def projectors(self, pos):
        gs, dev = self.s.gs, self.dev
        g = torch.as_tensor(gs.gvec[: self.ng], device=dev)
        f0, f1 = (torch.as_tensor(f, device=dev) for f in PP.radial_g(np.sqrt(gs.recnrm[: self.ng])))
        ph = g @ pos.T
        c, s = ph.cos(), ph.sin()
        kb = torch.empty((gs.nplwex, pos.shape[0], 4), dtype=torch.float64, device=dev)
        kb[0::2, :, 0], kb[1::2, :, 0] = c * (f0 * cell.Y00)[:, None], -s * (f0 * cell.Y00)[:, None]
        for m in range(3):
            f = (f1 * cell.Y1 * g[:, m])[:, None]
            kb[0::2, :, 1 + m], kb[1::2, :, 1 + m] = -s * f, -c * f
        vcl = torch.tensor([PP.e_s, PP.e_p, PP.e_p, PP.e_p], dtype=torch.float64, device=dev) / gs.rvol
        return kb.reshape(gs.nplwex, -1), vcl.repeat(pos.shape[0])

    def grid(self):
        k1, k2, k3 = self.s.gs.grid
        return k3, k2, k1

    def to_real(self, x):
        c = torch.complex(x[:, 0::2].contiguous(), x[:, 1::2].contiguous())
        z = torch.zeros((x.shape[0], self.n), dtype=torch.complex128, device=self.dev)
        z[:, self.ip] = c
        z[:, self.im] = c[:, 1:].conj()
        return torch.fft.ifftn(z.reshape(-1, *self.grid()), dim=(1, 2, 3)).real.reshape(-1, self.n) * self.n

    def to_g(self, r):
        z = torch.fft.fftn(r.reshape(-1, *self.grid()), dim=(1, 2, 3)).reshape(-1, self.n)[:, self.ip] / self.n
        return torch.view_as_real(z).reshape(r.shape[0], -1)

    def dot(self, x, y):
        return (x * y) @ self.w

    def gram(self, x, y):
        return (x * self.w) @ y.T

    def hpsi(self, x):
        out = self.dk * x
        for b in range(0, x.shape[0], 64):
            r = self.to_real(x[b: b + 64])
            v = r * self.vloc
            if self.real:
                rp = r[:, self.mesh]
                for ch in range(4):
                    p = torch.zeros((r.shape[0], self.s.cell.natom), dtype=torch.float64, device=self.dev)
                    p.index_add_(1, self.at, rp * self.vnl[:, ch])
                    p *= self.rdelv * self.cl[ch]
                    v.index_add_(1, self.mesh, p[:, self.at] * self.vnl[:, ch])
            out[b: b + 64] += self.to_g(v)
        if not self.real:
            p = 2.0 * x @ self.kb - torch.outer(x[:, 0], self.kb[0]) - 2.0 * torch.outer(x[:, 1], self.kb[1])
            out += (p * self.vcl) @ self.kb.T
        return out

    def density(self, x):
        rho = torch.zeros(self.n, dtype=torch.float64, device=self.dev)
        occ = torch.as_tensor(self.s.occ, device=self.dev) / self.s.gs.rvol
        for b in range(0, x.shape[0], 64):
            rho += occ[b: b + 64] @ self.to_real(x[b: b + 64]) ** 2
        return rho

    def orthonormal(self, x):
        return torch.linalg.solve_triangular(torch.linalg.cholesky(self.gram(x, x)), x, upper=False)

    def ritz(self, x):
        hx = self.hpsi(x)
        w, u = torch.linalg.eigh(self.gram(x, hx))
        self.eig = w
        return u.T @ x, u.T @ hx

    def ekib(self, x):
        return 2.0 * self.dot(self.dk * x, x)

    def cg(self, x, hx, ekib, noband, sequential):
        nb = x.shape[0]
        x, hx = x.clone(), hx.clone()
        eig = torch.empty(nb, dtype=torch.float64, device=self.dev)
        iters = torch.zeros(nb, dtype=torch.int32, device=self.dev)
        if not sequential:
            self.cg_bands(x, hx, x.clone(), torch.arange(nb, device=self.dev), ekib, noband, eig, iters)
        else:
            for b in range(nb):
                self.cg_bands(x, hx, x, torch.arange(b, b + 1, device=self.dev), ekib, noband, eig, iters)
        return x, hx, eig, iters

    def cg_bands(self, xa, hxa, snap, idx, ekib, noband, eig, iters):
        """The BKL steps of the bands idx against the vectors of snap below each."""
        x, hx, e = xa[idx], hxa[idx], self.dot(xa[idx], hxa[idx])
        e15 = 1.5 * ekib[idx][:, None]
        q = self.dk / e15
        t = 27.0 + q * (18.0 + q * (12.0 + 8.0 * q))
        prec = t / (t + 16.0 * q ** 4) * 2.0 / e15
        g = e[:, None] * x - hx
        z0 = zb = self.dot(g, g)
        eb, x0 = e.clone(), torch.full_like(e, 1.0e10)
        h, bet = torch.zeros_like(g), torch.ones_like(e)
        below = torch.arange(snap.shape[0], device=self.dev)[None, :] < idx[:, None]
        act = torch.ones_like(idx, dtype=torch.bool)
        it = torch.zeros_like(idx)
        for step in range(1, 5):
            a = act[:, None]
            g = torch.where(a, g * prec, g)
            zp = self.dot(g, g)
            h = torch.where(a, g + (0.0 if step == 1 else (zp / bet)[:, None]) * h, h)
            bet = zp
            if len(idx) == 1:
                lo = snap[: int(idx[0])]
                hn = h - self.gram(h, lo) @ lo
            else:
                hn = h - (self.gram(h, snap) * below) @ snap
            hn = hn - self.dot(x, hn)[:, None] * x
            h = torch.where(a, hn, h)
            cai, gh = self.dot(h, hx), self.hpsi(h)
            cbi, hh = self.dot(h, gh), self.dot(h, h)
            h12, h22 = cai / hh.sqrt(), cbi / hh
            en = 0.5 * (e + h22 - ((e + h22) ** 2 - 4.0 * (e * h22 - h12 * h12)).sqrt())
            dt = (en - e) / h12 / hh.sqrt()
            al = (1.0 / (1.0 + dt * dt * hh)).sqrt()
            xn, hxn = al[:, None] * (x + dt[:, None] * h), al[:, None] * (hx + dt[:, None] * gh)
            x, hx, e = torch.where(a, xn, x), torch.where(a, hxn, hx), torch.where(act, en, e)
            g = torch.where(a, e[:, None] * x - hx, g)
            z, de = self.dot(g, g), (eb - e).abs()
            it = it + act.int()
            stop = (z < 1e-10) | (de < 1e-10) | (z < 0.3 * z0) | (step >= 4)
            if step > 1:
                stop = stop | (de < 0.3 * x0)
            else:
                x0 = de
            eb = torch.where(act, e, eb)
            act = act & ~stop
            if not bool(act.any()):
                break
        xa[idx], hxa[idx], eig[idx], iters[idx] = x, hx, e, it.int()

    def g2(self):
        gs = self.s.gs
        k = [torch.arange(n, device=self.dev, dtype=torch.float64) for n in gs.grid]
        d = [torch.where(x <= n // 2, x, x - n) for x, n in zip(k, gs.grid)]
        d3, d2, d1 = torch.meshgrid(d[2], d[1], d[0], indexing="ij")
        c = gs.cross
        g = [c[i, 0] * d1 + c[i, 1] * d2 + c[i, 2] * d3 for i in range(3)]
        q = (g[0] ** 2 + g[1] ** 2 + g[2] ** 2).reshape(-1)
        return torch.where(q <= gs.ecutdens, q, torch.full_like(q, -1.0))

    def fft(self, r, back=False):
        z = r.reshape(self.grid())
        return (torch.fft.ifftn(z) * self.n if back else torch.fft.fftn(z) / self.n).reshape(-1)

    def lda(self, rho):
        """Perdew-Zunger 1981 unpolarised LDA (Hartree) with QXMD's
        single-precision literals: (e_xc, v_xc)."""
        f = lambda v: float(np.float32(v))   # noqa: E731
        pos = rho >= 1e-30
        rs = (3.0 / (12.56637061436 * torch.where(pos, rho, torch.ones_like(rho)))) ** (1.0 / 3.0)
        ex = -0.4582 / rs
        b2, b3, c2, c3, c4 = f(1.0529), f(0.3334), f(0.0311), f(-0.0116), f(0.0020)
        d = 1.0 + b2 * rs.sqrt() + b3 * rs
        hi = -0.1423 / d
        hv = hi * (1.0 + (b2 * rs.sqrt() / 6.0 + b3 * rs / 3.0) / d)
        ln = rs.log()
        lo = -0.0480 + c2 * ln + c3 * rs + c4 * rs * ln
        lv = lo - (c2 + (c3 + c4) * rs + c4 * rs * ln) / 3.0
        e, v = ex + torch.where(rs >= 1.0, hi, lo), 4.0 * ex / 3.0 + torch.where(rs >= 1.0, hv, lv)
        z = torch.zeros_like(rho)
        return torch.where(pos, e, z), torch.where(pos, v, z)

    def scf(self, psi, rho):
        gs = self.s.gs
        g2 = self.g2()
        m = g2 > 0
        rg = self.fft(rho)
        vg = torch.where(m, 8.0 * math.pi * rg / torch.where(m, g2, torch.ones_like(g2)), torch.zeros_like(rg))
        eh = 0.5 * gs.rvol * float((vg * rg.conj()).real.sum())
        e, v = self.lda(rho)
        dv = gs.rvol / self.n
        exc, evxc = 2.0 * dv * float((e * rho).sum()), 2.0 * dv * float((v * rho).sum())
        self.vloc = self.vloc + self.fft(vg, back=True).real + 2.0 * v
        ekib = self.ekib(psi)
        x, hx = self.ritz(psi)
        eband = float((self.eig * torch.as_tensor(self.s.occ, device=self.dev)).sum())
        x, hx, eig, _ = self.cg(x, hx, ekib, _noband(self.s), False)
        out = self.density(self.orthonormal(x))
        d = out - rho
        dg = torch.where(m, self.fft(out) - rg, torch.zeros_like(rg))
        k = torch.where(m, 0.8 * g2 / (g2 + 0.64), torch.zeros_like(g2))
        return {"energies": np.array([eband - eh + exc - evxc, eband, eh, exc, evxc]), "resid": np.array([dv * float((d * d).sum())]),
                "psi": None, "eig": eig, "rho_out": out, "rho_next": self.fft(rg + k * dg, back=True).real}

    def md(self, psi, seed):
        s, dev = self.s, self.dev
        gs = s.gs
        pos = torch.as_tensor(_moved(s, seed)[0], device=dev)
        occ = torch.as_tensor(s.occ, device=dev)
        # local potential and its force over the density half sphere
        gv = torch.as_tensor(gs.gvec, device=dev)
        ph = gv @ pos.T
        sv = torch.as_tensor(PP.vloc_g(gs.recnrm), device=dev)
        z = torch.zeros(self.n, dtype=torch.complex128, device=dev)
        vg = sv / gs.rvol * torch.complex(ph.cos().sum(1), -ph.sin().sum(1))
        ip, im = (torch.as_tensor(a, device=dev).long() for a in (gs.ijk_pos, gs.ijk_neg))
        z[ip] = vg
        z[im[1:]] = vg[1:].conj()
        vloc = self.fft(z, back=True).real
        rg = self.fft(self.density(psi))[ip]
        floc = 2.0 * ((sv[:, None] * (rg.real[:, None] * ph.sin() + rg.imag[:, None] * ph.cos()))[1:].T @ gv[1:])
        # projectors in G space
        kb, vcl = self.projectors(pos)
        p = 2.0 * psi @ kb - torch.outer(psi[:, 0], kb[0]) - 2.0 * torch.outer(psi[:, 1], kb[1])
        wp = p * vcl * (occ * 2.0)[:, None]
        gw = gv[1: self.ng]
        cr, ci = wp.T @ psi[:, 2::2], wp.T @ psi[:, 3::2]
        fnl = 2.0 * ((kb[2::2].T * ci - kb[3::2].T * cr) @ gw).reshape(-1, 4, 3).sum(1)
        # projectors in real space
        rb = torch.as_tensor(gs.rba, device=dev)
        ib = torch.linalg.inv(rb)
        k1, k2, k3 = gs.grid
        i = torch.arange(self.n, device=dev)
        fr = torch.stack([(i % k1) / k1, (i // k1 % k2) / k2, (i // (k1 * k2)) / k3], 1)
        cl = (PP.e_s, PP.e_p, PP.e_p, PP.e_p)
        rdelv = gs.rvol / self.n
        pts, dis = [], []
        for a in range(pos.shape[0]):
            d = fr - ib @ pos[a]
            d = (d - d.round()) @ rb.T
            sel = torch.nonzero((d * d).sum(1) <= PP.rcut ** 2)[:, 0]
            pts.append(sel)
            dis.append(d[sel])
        fr_ = torch.zeros((pos.shape[0], 3), dtype=torch.float64, device=dev)
        for b in range(0, psi.shape[0], 64):
            r = self.to_real(psi[b: b + 64])
            wb = 2.0 * occ[b: b + 64] / gs.rvol
            for a, (sel, d) in enumerate(zip(pts, dis)):
                ps = r[:, sel]
                ex = torch.exp(-0.5 * (d * d).sum(1) / PP.sig ** 2)
                for ch in range(4):
                    f = ex * (PP.a_s * cell.Y00 if ch == 0 else PP.a_p * cell.Y1)
                    v = f if ch == 0 else f * d[:, ch - 1]
                    gr = -d * (v / PP.sig ** 2)[:, None]
                    if ch:
                        gr[:, ch - 1] += f
                    fr_[a] += (wb * cl[ch] * (ps @ v) * rdelv) @ (ps @ gr) * rdelv
        return {"vloc": vloc, "floc": floc, "fnl": fnl, "fnl_r": fr_}


def _round(case, x):
    """The values the context holds: FP32 in mixed precision."""
    return x.to(_dtype(case)).double()


def _plain(v):
    if isinstance(v, dict):
        return {k: _plain(x) for k, x in v.items()}
    if isinstance(v, list):
        return [_plain(x) for x in v]
    return v.cpu() if isinstance(v, torch.Tensor) else v


def exact(case, seed):
    if case["kind"] == "batch":
        return [exact(c, seed + 1000003 * k) for k, c in enumerate(_batch_cells(case))]
    s = _system(case)
    E = _Exact(s, case)
    kind = case["kind"]
    if kind == "scf":
        psi, rho = _scf_inputs(s, seed)
        return _plain(E.scf(_round(case, psi), rho))
    if kind == "hpsi":
        return E.hpsi(_round(case, _psi(s.gs, s.nband, seed))).cpu()
    psi = _psi(s.gs, s.nband, seed, orthonormal=kind != "ortho")
    if kind == "subspace":
        hx = _round(case, E.hpsi(psi))
        hm = E.gram(_round(case, psi), hx)
        hm = torch.tril(hm.T).T + torch.tril(hm.T, -1)
        # the sign of an eigenvector is free: no value for the rotated bands
        return {"hsub": hm.cpu().numpy(), "ev": torch.linalg.eigvalsh(hm).cpu().numpy(), "psi": None, "hpsi": None}
    if kind == "ortho":
        x = E.orthonormal(_round(case, psi))
        return {"psi": x.reshape(-1).cpu(), "rho": E.density(x).cpu()}
    if kind == "cg":
        x, hx = (_round(case, v) for v in E.ritz(psi))
        x, hx, eig, it = E.cg(x, hx, E.ekib(x), _noband(s), bool(case["sequential"]))
        return {"psi": x.reshape(-1).cpu(), "hpsi": hx.reshape(-1).cpu(), "eig": eig.cpu(), "iters": it.cpu().numpy()}
    out = _plain(E.md(_round(case, psi), seed))
    return {k: v if k == "vloc" else v.numpy() for k, v in out.items()}


# ---- what a pass cannot do without -------------------------------------------

def _work_one(case):
    c, gs = _sphere(_cell_key(case))
    nb, ne, n = case["nb"], gs.nplwex, gs.kfft0
    s = 8 if case["prec"] == "fp64" else 4
    psi, nproj = nb * ne * s, 4 * c.natom
    npts = int(c.natom * 4.0 / 3.0 * math.pi * PP.rcut ** 3 / gs.rvol * n)
    fft = 5.0 * n * math.log2(n)                 # per band: two half-length (real) transforms
    real = case.get("nl") == "r"
    kb_flops = nb * (8.0 * npts * 2 if real else 4.0 * nproj * ne)
    kb_bytes = npts * 4 * s if real else nproj * ne * s
    hpsi = {"bytes": 2 * psi + kb_bytes + n * s, "flops": nb * fft + kb_flops}
    rot = 2.0 * nb * nb * ne
    kind = case["kind"]
    if kind == "hpsi":
        return hpsi
    if kind == "subspace":
        return {"bytes": 4 * psi + nb * nb * 8, "flops": rot + 2 * rot + 6.0 * nb ** 3}
    if kind == "ortho":
        return {"bytes": 2 * psi + n * 8, "flops": 2 * rot + nb ** 3 + nb * fft / 2}
    cg = {"bytes": 4 * psi + hpsi["bytes"], "flops": 2.0 * (hpsi["flops"] + rot)}   # about two steps a band
    if kind == "cg":
        return cg
    if kind == "scf":
        return {"bytes": cg["bytes"] + 2 * psi + 6 * n * 8,
                "flops": cg["flops"] + hpsi["flops"] + 5 * rot + 7.0 * nb ** 3 + nb * fft / 2 + 4 * fft}
    return {"bytes": psi + 2 * nproj * ne * s + 16 * npts * s + 2 * n * 8,
            "flops": nb * fft + nb * (8.0 * nproj * ne + 32.0 * npts)}


def work(case):
    if case["kind"] != "batch":
        return _work_one(case)
    parts = [_work_one(c) for c in _batch_cells(case)]
    return {k: sum(p[k] for p in parts) for k in ("bytes", "flops")}


def tolerance(case):
    """About four times the difference between two orders of summation (other
    tile widths and K splits of the 3xTF32 contractions, FP32 FMA contractions,
    other FFT stages).  The rotated bands of a subspace step carry the rounding
    of H_sub over the gaps between its eigenvalues, which the CG damps again."""
    mixed = case["prec"] != "fp64"
    kind = case["kind"]
    if kind == "hpsi":
        return {"rel": 5e-7} if mixed else {"rel": 2e-15}
    if kind == "ortho":
        return {"rel": 3e-6} if mixed else {"rel": 1e-13}
    if kind == "subspace":
        return {"rel": 1e-3} if mixed else {"rel": 1e-10}
    if kind == "cg":
        return {"rel": 2e-6, "differ": 0.02} if mixed else {"rel": 1e-12, "differ": 0.02}
    if kind == "md":
        return {"rel": 1e-5} if mixed else {"rel": 1e-11}
    return {"rel": 1e-4} if mixed else {"rel": 1e-10}

"""The work that is measured: the kinetic particle loop as a host program
drives it through kaos_b200.lib, from a tube of two thousand ions to one of
1e8, single tubes and batches, every precision mode, 2D and 3D velocity
grids, with and without charge exchange, steps in runs and one by one.

A pass of a "run" case is one stretch of computational steps followed by the
reads that the host makes after it (moments of the last master step, counts,
boundary fluxes, the ion state where the program keeps it).  The first pass
of a new solver holds step 1 and whatever the library sets up on first use.
A pass of a "stats" case is one call of kaos_moments_noalloc.
"""
import ctypes
import dataclasses
import math

import numpy as np
import torch

from kaos_b200 import grids, lib
from kaos_b200.lib import Solver
from kaos_b200.model_input import (GG, KAOS_NMOMENTS, KB, MDIP, ME, MH, MO, RE, ModelInput,
                                   VGrid)

EV = 1.602e-19 / KB  # 1 eV in K
RUN = dict(kind="run", tubes=1, nq=256, L=4.0, ions=1_000_000, n1=48, n2=48, npar=64,
           vmax=30e3, precision=1, dt=0.005, heating=1e-3, neutrals=0.0, cadence=20,
           steps=20, graph=False, host_ions=False, tail=0.0, flux=False, species=1,
           drift=False, hist=False, state=False)


def _case(name=None, **kw):
    c = dict(RUN, **kw)
    return dict(c, name=name) if name else c


def listed():
    return [
        # the smallest calls: a test-sized tube driven master interval by
        # master interval, its state read back each time; launches and
        # synchronisations are all of it
        _case("tiny_mixed", ions=2000, nq=24, n1=16, n2=16, npar=24, vmax=8e3, dt=0.01,
              heating=5.0, cadence=5, steps=5, state=True),
        # the plain FP64 configuration: 1e5 O+, 128 cells, 2D grid, no
        # heating, ions loaded from the host; the full histogram of every
        # master step and the state go to the host (data export)
        _case("plain_fp64", ions=100_000, nq=128, n1=32, n2=0, precision=0, dt=0.01,
              heating=0.0, host_ions=True, hist=True, state=True),
        # a host that couples to the loop at every step: one step per call,
        # every step a master step, all moments read after it
        _case("coupled_mixed", ions=300_000, nq=128, cadence=1, steps=1),
        # a run of five master intervals with a checkpoint of the ions at
        # its end; cells, bins and ions that divide by nothing
        _case("checkpoint_mixed", ions=1_000_003, nq=97, L=5.3, n1=31, n2=29, npar=53,
              steps=100, state=True),
        # the precision A/B tube (the benchmark's headline): 1e7 O+, heating
        # and collisions on, a master step every 20 steps, in each precision
        _case("ab_mixed", ions=10_000_000, neutrals=1e14),
        _case("ab_kick64", ions=10_000_000, neutrals=1e14, precision=2),
        _case("ab_fp64", ions=10_000_000, neutrals=1e14, precision=0),
        # the large single tube: 1e8 O+, kappa tail, flux injection, steps
        # replayed from graphs
        _case("large_mixed", ions=100_000_000, nq=512, L=6.0, n1=64, n2=64, npar=96,
              vmax=40e3, neutrals=1e14, tail=0.1, flux=True, graph=True),
        # a survey of field lines: 256 uneven tubes (64-512 cells, 1e4-1e6
        # ions each) in one handle, graphs
        _case("batch_mixed", tubes=256, nq=512, ions=1_000_000, graph=True),
        # a small FP64 survey on a 2D grid, no heating: 24 uneven tubes
        _case("batch_fp64", tubes=24, nq=300, ions=100_000, n1=40, n2=0, npar=50,
              precision=0, heating=0.0, graph=True),
        # two species with charge exchange to ENAs and the E x B drift: 64
        # tubes x (O+, H+), 2e7 ions, new tables for every entry each interval
        _case("species_ena", tubes=64, ions=312_500, heating=0.0, neutrals=1e16, species=2,
              drift=True, graph=True),
        # start-of-step statistics of ions that another program holds
        dict(kind="stats", name="stats", ions=3_000_000, nq=256, n1=48, n2=48, npar=64,
             vmax=30e3),
    ]


def _log(rng, a, b):
    return int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))


def draw(rng):
    n1, n2, npar = (rng.randint(8, 96) for _ in range(3))
    n2 = n2 if rng.random() < 0.75 else 0
    nq = _log(rng, 12, 512)
    what = rng.random()
    if what < 0.12:
        return dict(kind="stats", ions=_log(rng, 2000, 10_000_000), nq=nq, n1=n1, n2=n2,
                    npar=npar, vmax=30e3)
    c = dict(nq=nq, L=round(rng.uniform(2.5, 7.5), 2), n1=n1, n2=n2, npar=npar,
             precision=rng.choice((0, 1, 1, 2)), heating=rng.choice((0.0, 1e-3, 1e-2)),
             cadence=rng.choice((1, 2, 5, 10, 20, 50)), graph=rng.random() < 0.5)
    c["steps"] = c["cadence"] * rng.choice((1, 1, 2)) if c["cadence"] > 1 else rng.randint(1, 20)
    most = 400_000_000 // (c["steps"] if c["cadence"] > 1 else 3 * c["steps"])  # ions of a pass
    if what < 0.27:
        tubes = rng.randint(1, 32)
        nq = (nq + 3) // 4 * 4  # whole groups of four cells, as every such run here has
        return _case(**dict(c, nq=nq, tubes=tubes, ions=min(_log(rng, 3000, 300_000), most // tubes),
                            species=2, neutrals=1e16, drift=rng.random() < 0.5, steps=c["cadence"]))
    if what < 0.5:
        tubes = rng.randint(2, 64)
        return _case(**dict(c, tubes=tubes, nq=max(nq, 64),
                            ions=min(_log(rng, 20_000, 600_000), most // tubes)))
    ions = min(_log(rng, 2000, 20_000_000), most)
    return _case(**dict(c, ions=ions, host_ions=ions < 1_000_000 and rng.random() < 0.5,
                        tail=rng.choice((0.0, 0.1)), flux=rng.random() < 0.3,
                        hist=nq * n1 * max(n2, 1) * npar < 2_000_000 and rng.random() < 0.5,
                        state=ions < 2_000_000 and rng.random() < 0.6))


# ---- what a program has in hand -----------------------------------------
def _edges(n, vmax, symmetric=True):
    if symmetric and n % 2:  # a geometric symmetric axis has an even count
        return np.linspace(-vmax, vmax, n + 1)
    return grids.geometric_edges(n, vmax, symmetric=symmetric)


def _vgrid(c):
    d3 = c["n2"] > 0
    return VGrid(e1=_edges(c["n1"], c["vmax"], symmetric=d3),
                 e2=_edges(c["n2"], c["vmax"]) if d3 else None, epar=_edges(c["npar"], c["vmax"]))


def _inputs(c, seed):
    """Run parameters, the entries' specifications and tables, the grid."""
    mi = ModelInput(h=c["dt"], ndatfac=c["cadence"], ION2VPERPflag=1 if c["n2"] else 0,
                    ICRflag=1 if c["heating"] else 0, QEXCHANGEflag=1 if c["neutrals"] else 0,
                    FLUXINJECTIONflag=1 if c["flux"] else 0, precision=c["precision"],
                    seed=1 + seed)
    if c["species"] == 2:
        mi.mNeut = MH
    rng = np.random.default_rng(4)  # the survey's field lines
    specs = []
    for _ in range(c["tubes"]):
        sp = grids.TubeSpec(L=c["L"], nq=c["nq"], n_particles=c["ions"], q_ub=1e-3,
                            heat_rate_eV_s=c["heating"], neut_n0=c["neutrals"])
        if c["tubes"] > 1:
            sp.L = float(rng.uniform(2.0, 8.0))
        if c["species"] == 2:  # O+ and H+ at 4:1, an H exosphere
            sp.neut_H = 1000e3
            for ms, frac, n0 in ((MO, 0.8, 1e10), (MH, 0.2, 2.5e9)):
                specs.append(dataclasses.replace(
                    sp, ms=ms, qs=1.602e-19, n0=n0, n_particles=int(round(c["ions"] * frac))))
            continue
        if c["tubes"] > 1:
            sp.nq = int(rng.integers(64, c["nq"] + 1))
            sp.n_particles = int(round(c["ions"] * 10 ** rng.uniform(-2.0, 0.0)))
            sp.n0 = float(10 ** rng.uniform(9.0, 11.0))
            sp.Ti = float(rng.uniform(0.1, 1.0)) * EV
            if c["heating"]:
                sp.heat_rate_eV_s = float(10 ** rng.uniform(-4.0, -2.0))
        specs.append(sp)
    for sp in specs:
        sp.capacity_factor = 1.6
    return mi, specs, [grids.make_tube(sp, mi) for sp in specs], _vgrid(c)


def _moves(c, mi, specs, tubes):
    """The tables of every entry one drift interval out, and back home."""
    if not c["drift"]:
        return []
    dl = grids.conv_c5_dl(c["cadence"], mi.h)
    return [[grids.moved_tube(sp, mi, t, sp.L + d) for sp, t in zip(specs, tubes)]
            for d in (dl, 0.0)]


def _tail(c):
    return dict(tail_fraction=c["tail"], kappa=3.0, tail_T=5.0 * EV if c["tail"] else 0.0)


def _stats_inputs(c, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    sp = grids.TubeSpec(nq=c["nq"], n_particles=c["ions"])
    tube = grids.make_tube(sp, ModelInput())
    q0, q1 = tube.qGL[0], tube.qGH[-1]
    n, d3 = c["ions"], c["n2"] > 0
    u = torch.rand(n, generator=g, device="cuda", dtype=torch.float64)
    # ions crowd towards the lower boundary, as in a stratified tube
    q = q0 + (q1 - q0) * (-torch.log1p(-u) / 6.0).clamp(max=0.999)
    v = torch.randn(3, n, generator=g, device="cuda", dtype=torch.float64) * math.sqrt(KB * 0.3 * EV / MO)
    edges = torch.tensor(np.concatenate([tube.qGL, tube.qGH[-1:]]), device="cuda")
    d3x = torch.tensor(tube.d3xC, device="cuda")
    return tube, edges, d3x, q, v[0].contiguous(), v[1].contiguous(), v[2].contiguous() if d3 else None


def prepare(case, seed):
    c = case
    if c["kind"] == "stats":
        tube, edges, d3x, q, vp, v1, v2 = _stats_inputs(c, seed)
        p = ModelInput(ION2VPERPflag=1 if c["n2"] else 0).to_c()
        vg = _vgrid(c)
        return dict(kind="stats", p=p, vg=vg, vgc=vg.to_c(), nq=c["nq"], w=tube.nsnormfac,
                    arrays=(edges, d3x, q, vp, v1, v2), n=c["ions"],
                    mom=torch.empty(11, c["nq"], dtype=torch.float64, device="cuda"),
                    cnt=torch.empty(c["nq"], dtype=torch.int64, device="cuda"))
    mi, specs, tubes, vg = _inputs(c, seed)
    s = Solver(mi, tubes, vg)
    if c["species"] == 2:
        s.set_ena_grid(VGrid(e1=_edges(48, 30e3), e2=_edges(48, 30e3), epar=_edges(64, 30e3)))
    for k, t in enumerate(tubes):
        if c["host_ions"]:
            s.load(k, *grids.initial_particles(t, specs[k], mi, seed=seed + k))
        else:
            s.init_particles(k, t._counts, seed=seed + 1000 * k, **_tail(c))
    s.set_graph(c["graph"])
    s.set_export(c["hist"])
    # the host's own buffers, pinned: all moments of every entry, the state
    ncell = sum(t.nq for t in tubes)
    flat = torch.zeros(KAOS_NMOMENTS * ncell, dtype=torch.float64, pin_memory=True).numpy()
    views, o = [], 0
    for t in tubes:
        views.append(flat[o:o + KAOS_NMOMENTS * t.nq].reshape(KAOS_NMOMENTS, t.nq))
        o += KAOS_NMOMENTS * t.nq
    st = dict(kind="run", s=s, steps=c["steps"], flat=flat, views=views, hist=c["hist"],
              moves=_moves(c, mi, specs, tubes), passes=0)
    if c["state"]:
        cap = tubes[0].capacity
        st["out"] = {k: torch.zeros(cap, dtype=torch.float64, pin_memory=True).numpy()
                     for k in ("q", "vpar", "vperp1", "vperp2")}
        st["out"]["qind"] = torch.zeros(cap, dtype=torch.int32, pin_memory=True).numpy()
    return st


ROWS = ("M0", "M1Perp1", "M1Perp2", "M1Par", "M2", "M2Perp1", "M2Perp2", "M2Par", "M1Perp",
        "M2Perp", "Nq", "EAmag", "EGmag", "M0Filt", "nuPoi", "enaNq", "enaM0", "enaM1P", "enaM1Q",
        "enaM1Phi", "enaM2", "enaM2P", "enaM2Q", "enaM2Phi")


def run(state):
    st = state
    if st["kind"] == "stats":
        ptr = [None if a is None else a.data_ptr() for a in st["arrays"]]
        rc = lib.load().kaos_moments_noalloc(
            ctypes.addressof(st["p"]), ctypes.addressof(st["vgc"]), st["nq"], ptr[0], ptr[1],
            st["w"], *ptr[2:], st["n"], st["mom"].data_ptr(), st["cnt"].data_ptr(),
            torch.cuda.current_stream().cuda_stream)
        if rc:
            raise RuntimeError("kaos_moments_noalloc: status %d" % rc)
        return {"moments": st["mom"], "counts": st["cnt"]}
    s = st["s"]
    if st["moves"]:
        for k, t in enumerate(st["moves"][st["passes"] % 2]):
            s.update_tube(k, t)
    st["passes"] += 1
    s.step(st["steps"])
    for k, v in enumerate(st["views"]):
        s.moments_all(k, out=v)
    if len(st["views"]) > 1:
        return {"moments": st["flat"]}
    out = {"moments": dict(zip(ROWS, st["views"][0])), "counts": s.counts(0, full=st["hist"]),
           "boundary": s.boundary(0)}
    if "out" in st:
        # the program's buffers, as long as the tube's capacity, and the ions
        # in them (what lies behind is an earlier pass' or zero)
        out["ions"] = dict(st["out"], n=len(s.state(0, out=st["out"])["q"]))
    return out


def work(case):
    c = case
    d3 = c["n2"] > 0
    if c["kind"] == "stats":  # four arrays in; a search per axis and ion
        return {"bytes": c["ions"] * (32 if d3 else 24) + c["nq"] * 12 * 8, "flops": 30 * c["ions"]}
    n = c["ions"] * (c["tubes"] * (0.25 if c["tubes"] > 1 and c["species"] == 1 else 1.0))
    # the state (position, three velocities, two field accelerations, id) in
    # and out once per pass; per ion and step three force points, the
    # combination, the root of the field-line quartic and the heating kick
    state = 56 if c["precision"] == 0 else 48
    out = KAOS_NMOMENTS * 8 * c["nq"] * c["tubes"] * c["species"]
    if c["hist"]:
        out += 8 * c["nq"] * c["n1"] * max(c["n2"], 1) * c["npar"]
    if c["state"]:
        out += 36 * n
    return {"bytes": 2 * state * n + out,
            "flops": n * c["steps"] * (220 + (90 if c["heating"] else 0))}


# ---- the same in 64 bits, with torch and numpy ---------------------------
# Philox4x32-10 and the transforms of the loop's random draws
def _mulhilo(a, b):
    p = a * b  # wraps modulo 2^64: the low word and the shifted high word hold
    return (p >> 32) & 0xFFFFFFFF, p & 0xFFFFFFFF


def _philox(c0, c1, c2, c3, key):
    """Four 32-bit words (int64 tensors) of the counter; c0 a tensor."""
    z = torch.zeros_like(c0)
    c1, c2, c3 = (x if torch.is_tensor(x) else z + x for x in (c1, c2, c3))
    k0, k1 = key & 0xFFFFFFFF, key >> 32
    for _ in range(10):
        h0, l0 = _mulhilo(0xD2511F53, c0)
        h1, l1 = _mulhilo(0xCD9E8D57, c2)
        c0, c1, c2, c3 = h1 ^ c1 ^ k0, l1, h0 ^ c3 ^ k1, l0
        k0, k1 = (k0 + 0x9E3779B9) & 0xFFFFFFFF, (k1 + 0xBB67AE85) & 0xFFFFFFFF
    return c0, c1, c2, c3


def _u01(hi, lo):
    m = (((hi << 32) | lo) >> 11) & ((1 << 53) - 1)
    return (m.double() + 0.5) * 2.0 ** -53


def _pair(i, c1, c2, c3, key):
    w = _philox(i, c1, c2, c3, key)
    r, a = torch.sqrt(-2.0 * torch.log(_u01(w[0], w[1]))), 2.0 * math.pi * _u01(w[2], w[3])
    return r * torch.cos(a), r * torch.sin(a)


HEAT, INJECT, NEUT, POIS, INIT = (k << 24 for k in range(1, 6))


def _root(q, p, u, n=8):
    """u = r/RE > 0 with q^2 u^4 + u/p = 1, by Newton from u."""
    for _ in range(n):
        u = u - (q * q * u ** 4 + u / p - 1.0) / (4.0 * q * q * u ** 3 + 1.0 / p)
    return u


class _Point:
    """Dipole geometry at meridian-plane points."""

    def __init__(self, rho, z):
        r2 = rho * rho + z * z
        self.r = torch.sqrt(r2)
        self.ct, self.st = z / self.r, rho / self.r
        self.q = RE * RE * self.ct / r2
        self.ell = 1.0 + 3.0 * self.ct ** 2
        self.sl = torch.sqrt(self.ell)
        self.er, self.ez = 3.0 * self.ct * self.st / self.sl, (3.0 * self.ct ** 2 - 1.0) / self.sl

    def force(self, vp2, aea, ag):
        s = torch.where(self.ct <= 0.0, -1.0, 1.0)
        m = 1.5 * vp2 * self.ct.abs() / self.r * (2.0 + self.st ** 2 / self.ell) / self.sl
        return s * (m - ag.abs()) + aea


def _bins(e, v, prev=None):
    e = torch.as_tensor(e, device=v.device)
    b = torch.searchsorted(e[1:].contiguous(), v.contiguous()).clamp(max=len(e) - 2)
    return torch.where((v >= e[0]) & (v <= e[-1]), b, -1 if prev is None else prev)


def _filter(a, pt=11):
    """Moving average of pt points, one-sided at the ends (numpy, one tube)."""
    n, H = len(a), (pt - 1) // 2
    up, dn = (lambda q, m: a[q:q + m + 1].sum() / (m + 1)), (lambda q, m: a[q - m:q + 1].sum() / (m + 1))
    up1, dn1 = (lambda q, m: a[q + 1:q + m + 1].sum() / m), (lambda q, m: a[q - m:q].sum() / m)
    out = np.zeros(n)
    for q in range(n):
        if q <= H - 1:
            out[q] = up(q, H) if q == 0 else (up(q, H) + dn1(q, q)) / 2.0
        if H - 1 < q < n - 1 - H:
            out[q] = (up(q, H) + dn1(q, H)) / 2.0
        if q >= n - 1 - H:
            out[q] = dn(q, H) if q == n - 1 else (up1(q, n - 1 - q) + dn(q, H)) / 2.0
    return out


class _Loop:
    """The loop on all entries at once: ions and ENAs as flat arrays with the
    index of their entry, the per-cell tables one after another."""

    def __init__(self, c, seed):
        self.c = c
        self.mi, specs, tubes, self.vg = _inputs(c, seed)
        self.moves = _moves(c, self.mi, specs, tubes)
        self.d3 = c["n2"] > 0
        self.dev = "cuda"
        self.nq = np.array([t.nq for t in tubes])
        self.off = np.concatenate([[0], np.cumsum(self.nq)])
        self.T = len(tubes)
        self.tables(tubes)
        self.Te = self.cells("TeG")
        dev, T = self.dev, self.T
        self.t0, self.tn = self.ten(self.off[:-1]), self.ten(self.nq)
        self.cell_t = self.ten(np.repeat(np.arange(T), self.nq))
        self.key = self.mi.seed
        # initial ions, entry by entry
        parts = []
        for k, t in enumerate(tubes):
            if c["host_ions"]:
                q, *v = (self.ten(a) for a in grids.initial_particles(t, specs[k], self.mi, seed=seed + k))
                s = self.sgn[k] * q
                cell = torch.searchsorted(self.EH[self.off[k]:self.off[k + 1]].contiguous(), s)
            else:
                q, v, cell = self.drawn(t, k, seed + 1000 * k)
            parts.append((torch.full_like(cell, k), cell + int(self.off[k]), q, *v,
                          torch.arange(len(q), device=dev)))
        self.t, self.g, q, self.vpar, self.v1, self.v2, self.id = (torch.cat(x) for x in zip(*parts))
        self.next_id = [len(p[0]) for p in parts]
        del parts
        self.rho, self.z = self.place(q, self.pG[self.t])
        self.qk4, self.rho4, self.z4 = q, self.rho, self.z
        n = len(q)
        self.out = torch.zeros(n, dtype=torch.long, device=dev)  # 0 inside, -1 / -2 escaped
        self.aea = torch.zeros(n, dtype=torch.float64, device=dev)
        self.ag = torch.zeros_like(self.aea)
        self.b1 = self.bp = None
        if not self.d3:
            self.b1 = _bins(self.vg.e1, torch.sqrt(self.v1 ** 2 + self.v2 ** 2))
            self.bp = _bins(self.vg.epar, self.vpar)
        # ENAs: position, velocity, (Vp, Vphi) kept outside the grid, entry,
        # cell, escape, bins
        self.ena = {k: torch.zeros(0, 3, dtype=torch.float64, device=dev) for k in ("x", "v")}
        self.ena.update({k: torch.zeros(0, dtype=torch.float64, device=dev) for k in ("vp", "vh")})
        self.ena.update({k: torch.zeros(0, dtype=torch.long, device=dev)
                         for k in ("t", "g", "out", "bp", "bq", "bh")})
        self.mom = {}
        self.lost = self.gain = np.zeros(2, dtype=np.int64)

    def ten(self, a):
        return torch.as_tensor(np.ascontiguousarray(a), device=self.dev)

    def cells(self, name):
        return self.ten(np.concatenate([getattr(t, name) for t in self.tubes]))

    def tables(self, tubes):
        self.tubes = tubes
        self.sgn = np.array([1.0 if t.qGL[0] <= 0 else -1.0 for t in tubes])
        s = np.repeat(self.sgn, self.nq)
        self.s = self.ten(s)
        self.qC = self.cells("qGC")
        self.EL, self.EH, self.C = self.s * self.cells("qGL"), self.s * self.cells("qGH"), self.s * self.qC
        self.pG = self.ten([t.pG for t in tubes])
        self.ms = self.ten([t.ms or self.mi.ms for t in tubes])
        self.qs = self.ten([t.qs or self.mi.qs for t in tubes])
        self.arc = self.ten([t.sumdsICR for t in tubes])
        self.w = self.ten(np.repeat([t.nsnormfac for t in tubes], self.nq)) / self.cells("d3xC")
        m, q = (x[self.ten(np.repeat(np.arange(len(tubes)), self.nq))] for x in (self.ms, self.qs))
        pre = q * q / (2.0 * m * m) * self.cells("S0") * self.cells("EtaLH") / math.pi
        self.K = [self.mi.h * torch.sqrt(pre * self.cells(x)) for x in ("XiPerp1", "XiPerp2")]
        self.chi, self.Om0 = self.cells("ChiPerp1") * 0.5, self.cells("OmegaG0")
        self.Ts = self.cells("TsG")

    def place(self, q, p):
        u = _root(q, p, p * 0.5, 60)
        return u * RE * torch.sqrt(u / p), u * RE * q * u * u

    def drawn(self, t, k, seed):
        c, dev = self.c, self.dev
        cnt = self.ten(t._counts)
        cell = torch.repeat_interleave(torch.arange(t.nq, device=dev), cnt)
        i = torch.arange(len(cell), device=dev)
        w = _philox(i, 0, 0, INIT, seed)
        pop = _u01(w[2], w[3])
        qL, qH = self.ten(t.qGL)[cell], self.ten(t.qGH)[cell]
        q = qL + (0.02 + 0.96 * _u01(w[0], w[1])) * (qH - qL)
        g0, g1 = _pair(i, 0, 0, INIT | 1, seed)
        g2, g3 = _pair(i, 0, 0, INIT | 2, seed)
        f = torch.sqrt(KB * self.ten(t.TsG)[cell] / self.ms[k])
        if c["tail"]:  # kappa = 3: Student-t of five degrees of freedom
            W = g3 * g3
            for sub in (3, 4):
                for x in _pair(i, 0, 0, INIT | sub, seed):
                    W = W + x * x
            ft = torch.sqrt(KB * 5.0 * EV / self.ms[k] * 3.0 / 5.0) / torch.sqrt(W / 5.0)
            f = torch.where(pop < c["tail"], ft, f)
        return q, (f * g0, f * g1, f * g2), cell

    # -- one step of the ions
    def locate(self, s, g, t):
        lo, hi = self.t0[t], self.t0[t] + self.tn[t] - 1
        while True:
            d = ((s > self.EH[g]) & (g < hi)).long() - ((s <= self.EL[g]) & (g > lo)).long()
            if not bool(d.any()):
                break
            g = g + d
        return g, torch.where(s < self.EL[lo], -1, torch.where(s > self.EH[hi], -2, 0))

    def interpolate(self):
        s = self.sgn_t() * self.qk4
        g, out = self.locate(s, self.g, self.t)
        lo, hi = self.t0[self.t], self.t0[self.t] + self.tn[self.t] - 1
        b = torch.where(s <= self.C[g], g, g + 1).clamp(max=len(self.C))
        a = b - 1
        first, last = b <= lo, b > hi
        a, b = torch.where(first, lo, a), torch.where(last, hi, b)
        x1, x2 = self.qC[a], self.qC[b]
        fr = torch.where(first | last, 0.0, (self.qk4 - x1) / (x2 - x1))
        qm = (self.qs / self.ms)[self.t]
        at = lambda E: torch.where(first, E[b], E[a] + fr * (E[b] - E[a]))  # noqa: E731
        inside = out == 0
        self.aea = torch.where(inside, qm * at(self.EA), self.aea)
        self.ag = torch.where(inside, (qm * at(self.EG).abs()).abs(), self.ag)

    def sgn_t(self):
        return self.ten(self.sgn)[self.t]

    def push(self, n):
        h, P = self.mi.h, _Point(self.rho, self.z)
        vp2 = self.v1 ** 2 + self.v2 ** 2
        a1 = P.force(vp2, self.aea, self.ag)
        if self.c["heating"]:
            m, qs = self.ms[self.t], self.qs[self.t]
            Om = qs / m * MDIP * P.sl / P.r ** 3
            y = Om * self.vpar.abs() / self.arc[self.t]
            G = _pair(self.id, 0, n, HEAT, self.key)
            on = (self.out == 0) & (y <= (2.0 * math.pi / h) ** 2)
            e = torch.exp(-self.chi[self.g] * torch.log(Om / self.Om0[self.g])) * y ** 0.25
            k1, k2 = (torch.where(on, K[self.g] * e * g, 0.0) for K, g in zip(self.K, G))
        Vr, Vz = self.vpar * P.er, self.vpar * P.ez
        P2 = _Point(self.rho + 0.5 * h * Vr, self.z + 0.5 * h * Vz)
        a2 = P2.force(vp2, self.aea, self.ag)
        self.rho4 = self.rho + h * Vr + 0.5 * h * h * a1 * P.er
        self.z4 = self.z + h * Vz + 0.5 * h * h * a1 * P.ez
        P4 = _Point(self.rho4, self.z4)
        a4 = P4.force(vp2, self.aea, self.ag)
        self.qk4 = P4.q
        VN = [V + h / 6.0 * (a1 * d1 + 4.0 * a2 * d2 + a4 * d4) for V, d1, d2, d4 in
              ((Vr, P.er, P2.er, P4.er), (Vz, P.ez, P2.ez, P4.ez))]
        x = [x0 + h / 6.0 * (6.0 * V + 2.0 * h * a1 * d1 + h * a2 * d2) for x0, V, d1, d2 in
             ((self.rho, Vr, P.er, P2.er), (self.z, Vz, P.ez, P2.ez))]
        r = torch.sqrt(x[0] ** 2 + x[1] ** 2)
        q = RE * RE * x[1] / r ** 3
        u = _root(q, self.pG[self.t], r / RE, 3)
        self.rho, self.z = u * RE * torch.sqrt(u / self.pG[self.t]), u * RE * q * u * u
        N = _Point(self.rho, self.z)
        self.vpar = N.er * VN[0] + N.ez * VN[1]
        if self.c["heating"]:
            self.v1, self.v2 = self.v1 + k1, self.v2 + k2
        self.g0, self.out0 = self.g, self.out  # the start-of-step cell
        self.g, self.out = self.locate(self.sgn_t() * q, self.g, self.t)

    # -- a master step's statistics and fields
    def velocity_bins(self):
        if self.d3:
            return _bins(self.vg.e1, self.v1), _bins(self.vg.e2, self.v2), _bins(self.vg.epar, self.vpar)
        self.b1 = _bins(self.vg.e1, torch.sqrt(self.v1 ** 2 + self.v2 ** 2), self.b1)
        self.bp = _bins(self.vg.epar, self.vpar, self.bp)
        return self.b1, None, self.bp

    def count(self, t, g, out, b1, b2, bp):
        """Adds ions at cells g with these bins to the step's counters."""
        nc, vg = int(self.off[-1]), self.vg
        keep = out == 0
        self.cnt += torch.bincount(g[keep], minlength=nc)
        keep = keep & (b1 >= 0) & (bp >= 0) & ((b2 >= 0) if b2 is not None else True)
        g = g[keep]
        for k, b, n in (("1", b1, vg.n1), ("2", b2, vg.n2), ("p", bp, vg.npar)):
            if b is not None:
                self.marg[k] += torch.bincount(g * n + b[keep], minlength=nc * n).reshape(nc, n)
        if self.c["hist"]:
            b = b1[keep] if b2 is None else b1[keep] * vg.n2 + b2[keep]
            nv = vg.nbins(self.d3)
            self.full += torch.bincount(g * nv + b * vg.npar + bp[keep], minlength=nc * nv)

    def clear(self):
        nc, z = int(self.off[-1]), dict(dtype=torch.long, device=self.dev)
        self.cnt = torch.zeros(nc, **z)
        self.marg = {k: torch.zeros(nc, n, **z) for k, n in (("1", self.vg.n1), ("2", self.vg.n2), ("p", self.vg.npar)) if n}
        if self.c["hist"]:
            self.full = torch.zeros(nc * self.vg.nbins(self.d3), **z)

    @staticmethod
    def axis(m, e, w, M0, dev, centred):
        """First moment and second-moment sums (plain, centred, centred with
        the uncentred value where it is zero) of one axis' marginals."""
        v = torch.as_tensor(0.5 * (e[:-1] + e[1:]), device=dev)
        md = m.double()
        single = (m > 0).sum(1) == 1
        M1 = torch.where(single, v[m.argmax(1)], w * (md * v).sum(1) / M0)
        d2 = (v[None, :] - M1[:, None]) ** 2 if centred else (v * v).expand(len(m), -1)
        return M1, (md * v * v).sum(1), (md * d2).sum(1), (md * torch.where(d2 == 0.0, v * v, d2)).sum(1)

    def moments(self):
        vg, w, ms = self.vg, self.w, self.ms[self.cell_t]
        Nq = self.cnt.double() * w
        M0 = w * self.marg["p"].sum(1)
        ok = (Nq != 0) & (M0 != 0)
        Md = torch.where(ok, M0, 1.0)
        a = lambda k, e, cen: self.axis(self.marg[k], e, w, Md, self.dev, cen)  # noqa: E731
        M1p, _, Tq, Tp = a("p", vg.epar, True)
        M1a, Ta, _, _ = a("1", vg.e1, False)
        en = lambda x: ms / 2.0 * (w * x / Md)  # noqa: E731
        m = dict(M0=M0, M1Par=M1p, M2Par=en(Tp))
        if self.d3:
            M1b, Tb, _, _ = a("2", vg.e2, False)
            m.update(M1Perp1=M1a, M1Perp2=M1b, M2=en(Ta + Tb + Tq), M2Perp1=en(Ta), M2Perp2=en(Tb))
        else:
            m.update(M1Perp=M1a, M2=en(Ta + Tq), M2Perp=en(Ta))
        self.mom.update({k: torch.where(ok, v, 0.0) for k, v in m.items()})
        self.mom.update(Nq=Nq)
        self.M0prev = self.mom["M0"]

    def per_tube(self, f, *rows):
        rows = [r.cpu().numpy() for r in rows]
        return self.ten(np.concatenate([f(k, *(r[self.off[k]:self.off[k + 1]] for r in rows))
                                        for k in range(self.T)]))

    def fields(self):
        def ambipolar(k, M0, M0f, Te):
            t, n, M = self.tubes[k], len(M0), M0f
            R1 = KB * Te / ((t.qs or self.mi.qs) * np.where(M0 != 0, M, 1.0)) / np.abs(t.hqC)
            st, den = np.zeros(n), 12.0 * t.dqC
            st[2:-2] = M[:-4] - 8.0 * M[1:-3] + 8.0 * M[3:-1] - M[4:]
            for q in (1, n - 2):
                st[q], den[q] = M[q + 1] - M[q - 1], 2.0 * t.dqC[q]
            st[0] = -25.0 * M[0] + 48.0 * M[1] - 36.0 * M[2] + 16.0 * M[3] - 3.0 * M[4]
            st[-1] = -25.0 * M[-1] + 48.0 * M[-2] - 36.0 * M[-3] + 16.0 * M[-4] - 3.0 * M[-5]
            den[-1] = -12.0 * t.dqC[-1]
            E = np.where(M0 != 0, R1 * (-st / (-self.sgn[k] * den)), 0.0)
            return np.where((np.arange(n) <= 2) & (M0 != 0), E[3], E)
        M0f = self.per_tube(lambda k, a: _filter(a), self.M0prev)
        self.EA = self.per_tube(ambipolar, self.M0prev, M0f, self.Te)
        th, r, el = self.cells("thetaGC"), self.cells("rGC"), self.cells("ellGC")
        m, q = self.ms[self.cell_t], self.qs[self.cell_t]
        self.EG = -2.0 * GG * ME * m * torch.cos(th) / (q * r * r * torch.sqrt(el))
        self.mom.update(EAmag=self.EA, EGmag=self.EG, M0Filt=M0f)

    def inject(self):
        new = []
        for k, t in enumerate(self.tubes):
            n, g = int(np.rint(t.nsnormCLB)), int(self.off[k])
            self.gain = np.array([n, 0])
            if n <= 0:
                continue
            i = self.next_id[k] + torch.arange(n, device=self.dev)
            self.next_id[k] += n
            qc = self.qC[g].expand(n)
            rho, z = self.place(qc, self.pG[k].expand(n))
            P = _Point(rho, z)
            sig = torch.sqrt(KB * self.Ts[g] / self.ms[k])
            x, y, zz = (sig * _pair(i, 0, 0, INJECT | sub, self.key)[0] for sub in range(3))
            hz = x * math.cos(t.phiG) + y * math.sin(t.phiG)
            v1 = (1.0 - 3.0 * P.ct ** 2) / P.sl * hz + 3.0 * zz * P.ct * P.st / P.sl
            vp = P.er * hz + zz * P.ez
            v2 = -x * math.sin(t.phiG) + y * math.cos(t.phiG)
            if self.c["flux"]:
                w = _philox(i, 0, 0, INJECT | 3, self.key)
                vp = sig * torch.sqrt(-2.0 * torch.log(_u01(w[0], w[1])))
            qm = self.qs[k] / self.ms[k]
            c = torch.full((n,), g, device=self.dev)
            e = lambda E: (qm * E[g].abs()).abs().expand(n)  # noqa: E731
            b1 = _bins(self.vg.e1, v1 if self.d3 else torch.sqrt(v1 ** 2 + v2 ** 2))
            b2 = _bins(self.vg.e2, v2) if self.d3 else None
            bp = _bins(self.vg.epar, vp)
            tk, zero = torch.full_like(c, k), torch.zeros_like(c)
            self.count(tk, c, zero, b1, b2, bp)
            new.append(dict(t=tk, g=c, out=zero, g0=c, out0=zero, rho=rho, z=z, vpar=vp, v1=v1, v2=v2,
                            aea=e(self.EA), ag=e(self.EG), qk4=qc, rho4=rho, z4=z, id=i,
                            **({} if self.d3 else dict(b1=b1, bp=bp))))
        for k in (new[0] if new else ()):
            setattr(self, k, torch.cat([getattr(self, k)] + [x[k] for x in new]))

    def keep(self, sel):
        for k in ("t", "g", "out", "g0", "out0", "rho", "z", "vpar", "v1", "v2", "aea", "ag", "qk4",
                  "rho4", "z4", "id") + (() if self.d3 else ("b1", "bp")):
            setattr(self, k, getattr(self, k)[sel])

    # -- charge exchange, ENAs, the drift
    def collisions(self, nn):
        f = {k: self.per_tube(lambda _, a: _filter(a), self.mom[k]) for k in
             (("M1Par", "M1Perp1", "M1Perp2", "M2Par") if self.d3 else ("M1Par", "M1Perp", "M2Par"))}
        f1, f2 = f["M1Par"], f["M1Perp1" if self.d3 else "M1Perp"]
        f3 = f["M1Perp2"] if self.d3 else torch.zeros_like(f1)
        E = 6.242e18 * 1e-3 * f["M2Par"]
        Es = torch.where(E > 0, E, 1.0)
        sigma = torch.where(E > 0, (4.07 - 0.269 * torch.log(Es)) ** 2 * (1.0 - torch.exp(-415.0 / Es)) ** 0.8, 0.0)
        Q = torch.arange(len(E), device=self.dev) - self.t0[self.cell_t]
        G = [_pair(Q, nn, 0, NEUT | s, self.key)[0] * math.sqrt(KB * self.mi.TNeut / self.mi.mNeut) for s in range(3)]
        th, sl = self.cells("thetaGC"), torch.sqrt(self.cells("ellGC"))
        ct, st = torch.cos(th), torch.sin(th)
        ph = self.ten([t.phiG for t in self.tubes])[self.cell_t]
        cp, sp = torch.cos(ph), torch.sin(ph)
        a = (3.0 * f1 * ct * st + f2 * (1.0 - 3.0 * ct * ct)) / sl
        d = (cp * a - f3 * sp - G[0], sp * a + f3 * cp - G[1],
             f1 * (3.0 * ct * ct - 1.0) / sl + 3.0 * f2 * ct * st / sl - G[2])
        mean = self.cells("nsnormCNeut") * sigma * torch.sqrt(sum(x * x for x in d)) * self.mi.h
        lim, prod = torch.exp(-mean), torch.ones_like(mean)
        nu, it = torch.full_like(Q, -1), 0
        while bool((prod > lim).any()):
            w = _philox(Q, nn, it >> 1, POIS, self.key)
            on = prod > lim
            nu += on.long()
            prod = torch.where(on, prod * (_u01(w[2], w[3]) if it & 1 else _u01(w[0], w[1])), prod)
            it += 1
        on = (self.mom["M0"] != 0) & (sigma != 0)
        self.nu = torch.where(on, torch.minimum(nu, self.cnt), 0)
        self.mom["nuPoi"] = self.nu.double()

    @staticmethod
    def frame(ct, st, cp, sp):
        isl = 1.0 / torch.sqrt(1.0 + 3.0 * ct * ct)
        a, b, c = 3.0 * ct * st * isl, (3.0 * ct * ct - 1.0) * isl, (1.0 - 3.0 * ct * ct) * isl
        return (torch.stack((cp * a, sp * a, b), 1), torch.stack((cp * c, sp * c, a), 1),
                torch.stack((-sp, cp, torch.zeros_like(sp)), 1))

    def convert(self):
        """The first nu ions of each cell, by their cell at the start of the
        last push and in index order, become ENAs."""
        key = torch.where(self.out0 == 0, self.g0, len(self.nu))
        order = torch.sort(key, stable=True).indices
        ks = key[order]
        first = torch.searchsorted(ks, torch.arange(len(self.nu) + 1, device=self.dev))
        rank = torch.arange(len(ks), device=self.dev) - first[ks]
        nu = torch.cat([self.nu, self.nu.new_zeros(1)])
        pick = torch.sort(order[rank < nu[ks]]).values
        if not len(pick):
            return
        t = self.t[pick]
        ph = self.ten([x.phiG for x in self.tubes])[t]
        cp, sp = torch.cos(ph), torch.sin(ph)
        P, P4 = _Point(self.rho[pick], self.z[pick]), _Point(self.rho4[pick], self.z4[pick])
        e = self.frame(P.ct, P.st, cp, sp)[0]
        e4, p4, h4 = self.frame(P4.ct, P4.st, cp, sp)
        VN = self.vpar[pick, None] * e
        v = (e4 * VN).sum(1, keepdim=True) * e4 + self.v1[pick, None] * p4 + self.v2[pick, None] * h4
        x = torch.stack((self.rho[pick] * cp, self.rho[pick] * sp, self.z[pick]), 1)
        z = torch.zeros_like(t)
        zv = torch.zeros_like(cp)
        for k, a in dict(x=x, v=v, vp=zv, vh=zv, t=t, g=self.g0[pick], out=z, bp=z - 1, bq=z - 1,
                         bh=z - 1).items():
            self.ena[k] = torch.cat([self.ena[k], a])
        sel = torch.ones(len(self.t), dtype=torch.bool, device=self.dev)
        sel[pick] = False
        self.keep(sel)

    def sphere(self, x):
        rho2 = x[:, 0] ** 2 + x[:, 1] ** 2
        rho, r = torch.sqrt(rho2), torch.sqrt(rho2 + x[:, 2] ** 2)
        ct = x[:, 2] / r
        return ct, rho / r, x[:, 0] / rho, x[:, 1] / rho, RE * RE * ct / (r * r)

    def push_ena(self):
        E, h = self.ena, self.mi.h
        if not len(E["t"]):
            return
        x, t = E["x"], E["t"]
        ct, st, cp, sp, q = self.sphere(x)
        E["g"], E["out"] = self.locate(self.ten(self.sgn)[t] * q, E["g"], t)
        inside = E["out"] == 0
        ep, epp, eph = self.frame(ct, st, cp, sp)
        vq, vp, vh = ((e * E["v"]).sum(1) for e in (ep, epp, eph))
        vp, vh = E["vp"], E["vh"] = torch.where(inside, vp.abs(), E["vp"]), torch.where(inside, vh, E["vh"])
        for k, e, v in (("bp", _edges(48, 30e3), vp), ("bq", _edges(64, 30e3), vq), ("bh", _edges(48, 30e3), vh)):
            E[k] = torch.where(inside, _bins(e, v, E[k]), E[k])
        VR = vq[:, None] * ep + vp[:, None] * epp + vh[:, None] * eph
        acc = lambda y: -GG * ME * y / torch.sqrt((y * y).sum(1, keepdim=True)) ** 3  # noqa: E731
        A1 = acc(x)
        A2, A4 = acc(x + 0.5 * h * VR), acc(x + h * VR + 0.5 * h * h * A1)
        VN = VR + h / 6.0 * (A1 + 4.0 * A2 + A4)
        E["x"] = x + h / 6.0 * (6.0 * VR + 2.0 * h * A1 + h * A2)
        e = self.frame(*self.sphere(E["x"])[:4])
        c = [(d * VN).sum(1, keepdim=True) for d in e]
        E["v"] = c[0] * e[0] + c[1].abs() * e[1] + c[2] * e[2]

    def ena_moments(self):
        E, nc = self.ena, int(self.off[-1])
        on, g = E["out"] == 0, E["g"]
        w, ms = self.w, self.ms[self.cell_t]
        Nq = torch.bincount(g[on], minlength=nc).double() * w
        ok = on & (E["bp"] >= 0) & (E["bq"] >= 0) & (E["bh"] >= 0)
        first, second, M0 = [], [], None
        for k, e in (("bp", _edges(48, 30e3)), ("bq", _edges(64, 30e3)), ("bh", _edges(48, 30e3))):
            v, n = self.ten(0.5 * (e[:-1] + e[1:])), len(e) - 1
            m = torch.bincount(g[ok] * n + E[k][ok], minlength=nc * n).reshape(nc, n).double()
            M0 = torch.where(Nq == 0, 0.0, w * m.sum(1)) if M0 is None else M0
            Md = torch.where(M0 != 0, M0, 1.0)
            M1 = torch.where(M0 != 0, w * (m * v).sum(1) / Md, 0.0)
            d = (M1[:, None] - v[None, :]) ** 2
            first.append(M1)
            second.append(torch.where(M0 != 0, w * (m * d).sum(1) * 6.242e18 * ms / 2.0 / Md, 0.0))
        for k, r in enumerate([Nq, M0] + first + [sum(second)] + second):
            self.mom[ROWS[15 + k]] = r

    def drift(self, tubes):
        g = _Point(self.rho, self.z)
        q, u0 = g.q, g.r / RE
        self.tables(tubes)
        u1 = _root(q, self.pG[self.t], u0)
        b = lambda u: torch.sqrt(1.0 + 3.0 * (q * u * u) ** 2) / u ** 3  # noqa: E731
        f = torch.sqrt(b(u1) / b(u0))
        self.rho, self.z = u1 * RE * torch.sqrt(u1 / self.pG[self.t]), u1 * RE * q * u1 * u1
        self.v1, self.v2 = f * self.v1, f * self.v2

    def step(self, n):
        cx = self.mi.QEXCHANGEflag == 1
        if n == 1:
            b = self.velocity_bins()
            self.clear()
            self.count(self.t, self.g, self.out, *b)
            self.moments()
            if cx:
                self.collisions(1)
            self.fields()
            self.interpolate()
            self.push(1)
            return
        nd = self.mi.ndatfac
        master = n % nd == 0
        if master and self.moves:
            self.drift(self.moves.pop(0))
        if cx:
            self.convert()
        if master:
            self.lost = np.array([int((self.out0 == k).sum()) for k in (-1, -2)])
            self.keep(self.out0 == 0)
            if len(self.ena["t"]):
                sel = self.ena["out"] == 0
                self.ena = {k: v[sel] for k, v in self.ena.items()}
            self.fields()
            self.interpolate()
            self.clear()
            self.count(self.t, self.g, self.out, *self.velocity_bins())
        elif not self.d3:
            self.velocity_bins()
        if cx:
            self.push_ena()
        self.push(n)
        if master:
            self.inject()
            self.moments()
            if cx:
                self.collisions(n // nd + 1)
                self.ena_moments()


def _exact_stats(c, seed):
    L = _Loop.__new__(_Loop)
    tube, edges, d3x, q, vp, v1, v2 = _stats_inputs(c, seed)
    d3, nq = c["n2"] > 0, c["nq"]
    L.c, L.vg, L.d3, L.dev, L.off = dict(hist=False), _vgrid(c), d3, "cuda", np.array([0, nq])
    L.w, L.ms, L.cell_t = tube.nsnormfac / d3x, torch.full((1,), MO, dtype=torch.float64, device="cuda"), torch.zeros(nq, dtype=torch.long, device="cuda")
    L.mom = {}
    L.clear()
    s = -q
    g = torch.searchsorted((-edges[1:]).contiguous(), s).clamp(max=nq - 1)
    out = torch.where((s < -edges[0]) | (s > -edges[-1]), -1, 0)
    b1 = _bins(L.vg.e1, v1 if d3 else v1.abs())
    L.count(None, g, out, b1, _bins(L.vg.e2, v2) if d3 else None, _bins(L.vg.epar, vp))
    L.moments()
    rows = [L.mom.get(k, torch.zeros_like(L.w)) for k in ROWS[:11]]
    return {"moments": torch.stack(rows), "counts": L.cnt}


def exact(case, seed):
    """The first pass of a new state.  Draws of counts (the collision counts)
    and whole numbers are compared as they are: nothing in their place."""
    c = case
    if c["kind"] == "stats":
        return _exact_stats(c, seed)
    L = _Loop(c, seed)
    for n in range(1, c["steps"] + 1):
        L.step(n)
    zero = torch.zeros(int(L.off[-1]), dtype=torch.float64, device="cuda")
    rows = [L.mom.get(k, zero).cpu().numpy() for k in ROWS]
    if L.T > 1:
        return {"moments": np.concatenate([r[L.off[k]:L.off[k + 1]] for k in range(L.T) for r in rows])}
    ions = None
    if c["state"]:
        pad = (0, L.tubes[0].capacity - len(L.vpar))
        ions = {k: torch.nn.functional.pad(v, pad) for k, v in
                dict(q=_Point(L.rho, L.z).q, vpar=L.vpar, vperp1=L.v1, vperp2=L.v2).items()}
        ions.update(qind=None, n=None)
    return {"moments": dict(zip(ROWS, rows), nuPoi=None), "counts": None, "boundary": None, "ions": ions}

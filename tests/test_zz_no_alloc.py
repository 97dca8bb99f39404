"""The allocation-free statistics entry point (kaos_moments_noalloc).

Callers that cannot allocate device memory (a host with its own fixed
device pool, a GPU shared under a memory cap) get the start-of-step counts and moments from this entry point, whose
scratch histograms live in a static device array.  This test drives it
through the C-ABI on device buffers the test owns, twice in a row (the
second call must clear what the first left behind), and checks both results
against the existing path (kaos_step of a handle, then kaos_get_moments /
kaos_get_counts) on the same ions: counts bit-exact, moments within 1e-10
relative, the tolerance of the other GPU parity tests.

It is collected last so that a run stopping at the first failure has already
run every other test.
"""
import ctypes as C

import numpy as np
import pytest

from kaos_b200 import build as kbuild
from kaos_b200 import grids
from kaos_b200 import lib as klib
from kaos_b200.model_input import (KAOS_M0, KAOS_M1PAR, KAOS_M1PERP1, KAOS_M1PERP2, KAOS_NQ,
                                   KAOS_PREC_FP64, KAOS_PREC_MIXED)

pytestmark = pytest.mark.gpu
MOM_TOL = 1e-10


def test_noalloc_matches_handle_path_twice():
    import torch
    kbuild.build()
    L = klib.load()
    mi, spec, tube, vg = grids.config_small(n_particles=5000, three_d=True)
    q, vpar, v1, v2 = grids.initial_particles(tube, spec, mi, seed=17)
    # existing path: first step statistics of a handle
    s = klib.Solver(mi, [tube], vg)
    s.load(0, q, vpar, v1, v2)
    s.step(1)
    ref = np.stack([s.moments(k) for k in range(KAOS_NQ + 1)])
    ref_counts = s.counts()
    s.close()
    # allocation-free path on device buffers owned by the caller (here torch)
    dev = torch.device("cuda:0")
    t = lambda a: torch.as_tensor(np.ascontiguousarray(a), dtype=torch.float64, device=dev)
    edges = t(np.append(tube.qGL, tube.qGH[-1]))
    d3x = t(tube.d3xC)
    dq, dvp, dv1, dv2 = t(q), t(vpar), t(v1), t(v2)
    nq = tube.nq
    pc, vgc = mi.to_c(), vg.to_c()
    for call in range(2):
        out = torch.full((KAOS_NQ + 1, nq), -1.0, dtype=torch.float64, device=dev)
        cnt = torch.full((nq,), -1, dtype=torch.int64, device=dev)
        rc = L.kaos_moments_noalloc(C.addressof(pc), C.addressof(vgc), nq,
                                    edges.data_ptr(), d3x.data_ptr(),
                                    tube.nsnormfac, dq.data_ptr(), dvp.data_ptr(),
                                    dv1.data_ptr(), dv2.data_ptr(), len(q),
                                    out.data_ptr(), cnt.data_ptr(), None)
        assert rc == 0, call
        torch.cuda.synchronize()
        got = out.cpu().numpy()
        np.testing.assert_array_equal(cnt.cpu().numpy(), ref_counts)
        for k in range(KAOS_NQ + 1):
            scale = max(np.max(np.abs(ref[k])), 1e-300)
            assert np.max(np.abs(got[k] - ref[k])) / scale <= MOM_TOL, (call, k)


def test_noalloc_rejects_oversize_grid():
    kbuild.build()
    L = klib.load()
    mi, spec, tube, vg = grids.config_small(n_particles=100, three_d=True)
    pc, vgc = mi.to_c(), vg.to_c()
    dummy = C.c_double(0.0)
    # 513 cells exceed the static array: rejected before any device work
    rc = L.kaos_moments_noalloc(C.addressof(pc), C.addressof(vgc), 513,
                                C.addressof(dummy), C.addressof(dummy), 1.0,
                                None, None, None, None, 0, C.addressof(dummy),
                                None, None)
    assert rc == 2  # KAOS_ERR_CAPACITY
    # a 3D grid needs the Vperp2 array whenever there are ions to bin
    rc = L.kaos_moments_noalloc(C.addressof(pc), C.addressof(vgc), tube.nq,
                                C.addressof(dummy), C.addressof(dummy), 1.0,
                                C.addressof(dummy), C.addressof(dummy),
                                C.addressof(dummy), None, 1, C.addressof(dummy),
                                None, None)
    assert rc == 1  # KAOS_ERR_PARAM


@pytest.mark.parametrize("nq,n1,n2,npar,n", [
    (512, 128, 128, 128, 40_000),  # four parts of cells
    (194, 128, 8, 127, 6_000),     # one cell more than a part holds
    (193, 127, 128, 9, 1025),      # a part exactly full; one ion over a block
    (6, 2, 2, 2, 1),               # the smallest tube, one ion
    (97, 31, 0, 53, 100_003),      # 2D grid, ragged
])
def test_noalloc_matches_handle_sizes(nq, n1, n2, npar, n):
    """Cells and bins around the block-private counters' part sizes, ions
    outside the velocity grid among them (3D): the counts of the handle path
    exactly, its moments within 1e-10."""
    import torch
    kbuild.build()
    L = klib.load()
    d3 = n2 > 0
    mi = grids.ModelInput(ION2VPERPflag=1 if d3 else 0, MOMENTFILTERflag=0)
    spec = grids.TubeSpec(L=4.0, nq=nq, n_particles=n, q_ub=0.15, H=600e3)
    tube = grids.make_tube(spec, mi)
    tube.capacity = n
    vmax = 2.5e3 if d3 else 2e4  # (2D: the handle keeps a first bin outside)
    lin = lambda k, a: np.linspace(a, vmax, k + 1)
    vg = grids.VGrid(e1=lin(n1, -vmax if d3 else 0.0), e2=lin(n2, -vmax) if d3 else None,
                     epar=lin(npar, -vmax))
    rng = np.random.default_rng(nq)
    q = rng.uniform(tube.qGH[-1], tube.qGL[0], n)
    v = rng.normal(size=(3, n)) * 1.3e3
    s = klib.Solver(mi, [tube], vg)
    s.load(0, q, *v)
    s.step(1)
    ref, ref_counts = s.moments_all()[:KAOS_NQ + 1].copy(), s.counts()
    s.close()
    t = lambda a: torch.as_tensor(np.ascontiguousarray(a), dtype=torch.float64, device="cuda")
    arr = [t(np.append(tube.qGL, tube.qGH[-1])), t(tube.d3xC), t(q), t(v[0]), t(v[1]), t(v[2])]
    out = torch.full((KAOS_NQ + 1, nq), -1.0, dtype=torch.float64, device="cuda")
    cnt = torch.full((nq,), -1, dtype=torch.int64, device="cuda")
    pc, vgc = mi.to_c(), vg.to_c()
    ptr = [a.data_ptr() for a in arr]
    rc = L.kaos_moments_noalloc(C.addressof(pc), C.addressof(vgc), nq, ptr[0], ptr[1],
                                tube.nsnormfac, *ptr[2:], n, out.data_ptr(), cnt.data_ptr(), None)
    assert rc == 0
    torch.cuda.synchronize()
    np.testing.assert_array_equal(cnt.cpu().numpy(), ref_counts)
    got = out.cpu().numpy()
    for k in range(KAOS_NQ + 1):
        scale = max(np.max(np.abs(ref[k])), 1e-300)
        assert np.max(np.abs(got[k] - ref[k])) / scale <= MOM_TOL, k


@pytest.mark.parametrize("off,width", [(0.0, 1.0), (1.0, 1e-6), (1.0, 1e-8), (-1.0, 1e-10),
                                       (1e6, 1e-3), (-3e4, 6e4)])
def test_noalloc_bins_at_slot_ends(off, width):
    """Speeds on, and one unit in the last place beside, the velocity edges and
    the ends of the lookup table's slots, for grids far from zero against their
    width: the bin is the smallest k with v <= e[k + 1]."""
    import torch
    kbuild.build()
    L = klib.load()
    nb, nq = 61, 6
    e = off + width * np.linspace(0.0, 1.0, nb + 1)
    e = np.unique(e)
    nb = len(e) - 1
    slots = e[0] + (e[-1] - e[0]) * np.arange(0, 257) / 256.0
    v = np.concatenate([e, slots])
    v = np.concatenate([np.nextafter(v, -np.inf), v, np.nextafter(v, np.inf),
                        [np.nan, np.inf, -np.inf]])
    n = len(v)
    mi = grids.ModelInput(ION2VPERPflag=1)
    vg = grids.VGrid(e1=e.copy(), e2=e.copy(), epar=e.copy())
    want = np.searchsorted(e, v, side="left") - 1
    want[v == e[0]] = 0
    ok = (v >= e[0]) & (v <= e[-1])
    t = lambda a: torch.as_tensor(np.ascontiguousarray(a), dtype=torch.float64, device="cuda")
    qe = np.linspace(0.6, 0.1, nq + 1)
    # each axis in turn takes the values, the others a bin's middle: the first
    # moment of a cell with one ion is its bin's centre
    mid = np.full(n, 0.5 * (e[3] + e[4]))
    for axis, row in ((0, KAOS_M1PAR), (1, KAOS_M1PERP1), (2, KAOS_M1PERP2)):
        arr = [mid, mid, mid]
        arr[axis] = v
        for k0 in range(0, n, nq):
            m = min(nq, n - k0)
            q = 0.5 * (qe[:m] + qe[1:m + 1])
            dev = [t(qe), t(np.ones(nq)), t(q)] + [t(a[k0:k0 + m]) for a in arr]
            out = torch.full((KAOS_NQ + 1, nq), -1.0, dtype=torch.float64, device="cuda")
            pc, vgc = mi.to_c(), vg.to_c()
            ptr = [a.data_ptr() for a in dev]
            rc = L.kaos_moments_noalloc(C.addressof(pc), C.addressof(vgc), nq, ptr[0], ptr[1],
                                        1.0, *ptr[2:], m, out.data_ptr(), None, None)
            assert rc == 0
            got = out.cpu().numpy()
            for i in range(m):
                k = k0 + i
                if ok[k]:
                    b = want[k]
                    assert got[KAOS_M0, i] == 1.0, (axis, v[k])
                    assert got[row, i] == 0.5 * (e[b] + e[b + 1]), (axis, v[k])
                else:
                    assert got[KAOS_M0, i] == 0.0 and got[KAOS_NQ, i] == 1.0, (axis, v[k])


@pytest.mark.parametrize("prec", [KAOS_PREC_FP64, KAOS_PREC_MIXED])
@pytest.mark.parametrize("off,width,nb", [(0.0, 1.0, 64), (1.0, 1e-8, 61), (-3e4, 6e4, 60)])
def test_handle_bins_at_slot_ends(prec, off, width, nb):
    """The same through a handle's full histogram, one axis at a time."""
    e = off + width * np.linspace(0.0, 1.0, nb + 1)
    slots = e[0] + (e[-1] - e[0]) * np.arange(0, 257) / 256.0
    v = np.concatenate([e, slots])
    v = np.concatenate([np.nextafter(v, -np.inf), v, np.nextafter(v, np.inf)])
    v = v[(v >= e[0]) & (v <= e[-1])]
    want = np.maximum(np.searchsorted(e, v, side="left") - 1, 0)
    mi = grids.ModelInput(ION2VPERPflag=1, precision=prec)
    tube = grids.make_tube(grids.TubeSpec(L=4.0, nq=6, n_particles=100, q_ub=0.15, H=600e3), mi)
    mi.MOMENTFILTERflag = 0
    tube.capacity = len(v)
    q = np.full(len(v), tube.qGC[2])
    mid = np.full(len(v), 0.5 * (e[3] + e[4]))
    for axis, along in ((0, 3), (1, 1), (2, 2)):
        arr = [mid, mid, mid]
        arr[axis] = v
        s = klib.Solver(mi, [tube], grids.VGrid(e1=e.copy(), e2=e.copy(), epar=e.copy()))
        s.load(0, q, *arr)
        s.set_export(True)
        s.step(1)
        h = s.counts(full=True).reshape(6, nb, nb, nb)
        s.close()
        got = h.sum(axis=tuple(k for k in range(4) if k != along))
        np.testing.assert_array_equal(got, np.bincount(want, minlength=nb))


def test_noalloc_positions_that_are_no_numbers():
    """Infinite positions lie outside; one that is not a number is in no cell
    by comparison, and counts in the last one (as the cell search ends)."""
    import torch
    kbuild.build()
    L = klib.load()
    nq = 6
    t = lambda a: torch.as_tensor(np.ascontiguousarray(a), dtype=torch.float64, device="cuda")
    q = np.array([np.nan, np.inf, -np.inf, 0.55, 0.6, 0.1, np.nan])
    v = np.zeros(len(q))
    e = np.linspace(-1.0, 1.0, 9)
    mi = grids.ModelInput(ION2VPERPflag=1)
    vg = grids.VGrid(e1=e, e2=e.copy(), epar=e.copy())
    dev = [t(np.linspace(0.6, 0.1, nq + 1)), t(np.ones(nq)), t(q)] + [t(v) for _ in range(3)]
    out = torch.full((KAOS_NQ + 1, nq), -1.0, dtype=torch.float64, device="cuda")
    cnt = torch.full((nq,), -1, dtype=torch.int64, device="cuda")
    pc, vgc = mi.to_c(), vg.to_c()
    ptr = [a.data_ptr() for a in dev]
    rc = L.kaos_moments_noalloc(C.addressof(pc), C.addressof(vgc), nq, ptr[0], ptr[1], 1.0,
                                *ptr[2:], len(q), out.data_ptr(), cnt.data_ptr(), None)
    assert rc == 0
    np.testing.assert_array_equal(cnt.cpu().numpy(), [2, 0, 0, 0, 0, 3])

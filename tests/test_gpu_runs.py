"""Runs of ordinary steps in one launch: the state after kaos_step(n) equals
that of n calls of kaos_step(1) bit for bit, however the run is cut, for
every precision mode, both velocity grids, heating on and off, escaping ions
and speeds that leave the grid."""
import numpy as np
import pytest

from kaos_b200 import build as kbuild
from kaos_b200 import grids
from kaos_b200.grids import TubeSpec, make_tube, make_vgrid
from kaos_b200.lib import Solver
from kaos_b200.model_input import KAOS_PREC_FP64, KAOS_PREC_MIXED, KAOS_PREC_MIXED_K64, ModelInput

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _build():
    kbuild.build()


def _solver(mi, tubes, init, vg, graph=False):
    s = Solver(mi, tubes, vg)
    for k, a in enumerate(init):
        s.load(k, *a)
    s.set_graph(graph)
    return s


def _state(s, n):
    out = []
    for k in range(n):
        p = s.state(k)
        # (a mixed run stores Qindk1 only for the master step that reads it)
        out += [p[x] for x in ("q", "vpar", "vperp1", "vperp2")]
        out += [s.moments_all(k), s.counts(k), s.boundary(k)]
    return out


PRECS = (KAOS_PREC_FP64, KAOS_PREC_MIXED, KAOS_PREC_MIXED_K64)


@pytest.mark.parametrize("prec", PRECS)
@pytest.mark.parametrize("three_d", [True, False])
@pytest.mark.parametrize("heating", [True, False])
def test_runs_equal_single_steps(prec, three_d, heating):
    # two tubes, ion counts around the work-item sizes; a velocity grid that
    # many ions leave (the 2D grid's stale bins matter)
    mi = ModelInput(h=0.5, ndatfac=7, ION2VPERPflag=1 if three_d else 0,
                    ICRflag=1 if heating else 0, precision=prec)
    specs = [TubeSpec(L=3.0, nq=nq, n_particles=n, q_ub=0.5, H=400e3, Ti=5.0 * 1.602e-19 / 138e-25,
                      heat_rate_eV_s=2.0 if heating else 0.0) for nq, n in ((24, 1025), (31, 257))]
    tubes = [make_tube(sp, mi) for sp in specs]
    for t in tubes:
        t.nsnormCLB = 9.0
    vg = make_vgrid(True, 16, 16, 24, 9e3) if three_d else make_vgrid(False, 12, 0, 24, 7e3)
    init = [grids.initial_particles(t, sp, mi, seed=3) for t, sp in zip(tubes, specs)]
    a, b = _solver(mi, tubes, init, vg), _solver(mi, tubes, init, vg)
    g = _solver(mi, tubes, init, vg, graph=True)
    done = 0
    for n in (1, 13, 2, 1, 4, 14, 6):  # cuts inside and at the ends of intervals
        a.step(n)
        g.step(n)
        for _ in range(n):
            b.step(1)
        done += n
        for x, y, z in zip(_state(a, 2), _state(b, 2), _state(g, 2)):
            assert np.array_equal(x, y), done
            assert np.array_equal(x, z), done
    assert a.boundary(0)[:2].sum() > 0  # ions escaped
    for s in (a, b, g):
        s.close()


@pytest.mark.parametrize("n", [1, 255, 256, 257, 5000])
def test_run_ion_counts(n):
    mi = ModelInput(h=0.01, ndatfac=5, ION2VPERPflag=1, ICRflag=1, precision=KAOS_PREC_MIXED)
    spec = TubeSpec(L=4.0, nq=24, n_particles=6000, q_ub=0.15, H=600e3, heat_rate_eV_s=5.0)
    t = make_tube(spec, mi)
    init = [tuple(x[:n] for x in grids.initial_particles(t, spec, mi, seed=2))]
    vg = make_vgrid(True, 16, 16, 24, 8e3)
    a, b = _solver(mi, [t], init, vg), _solver(mi, [t], init, vg)
    a.step(14)
    for _ in range(14):
        b.step(1)
    for x, y in zip(_state(a, 1), _state(b, 1)):
        assert np.array_equal(x, y)
    a.close()
    b.close()


@pytest.mark.parametrize("prec", PRECS)
def test_single_steps_choose_their_shape(prec):
    """A handle above the small-item limit (2^21 slots) stepped one by one
    through a master step: the shape is chosen again after four of them, and
    the state stays that of the runs."""
    mi = ModelInput(h=0.01, ndatfac=9, ION2VPERPflag=1, ICRflag=1, precision=prec)
    spec = TubeSpec(L=3.0, nq=24, n_particles=30000, q_ub=0.5, H=400e3, heat_rate_eV_s=2.0)
    tubes = [make_tube(spec, mi)]
    tubes[0].capacity = (1 << 21) + 1000
    vg = make_vgrid(True, 16, 16, 24, 9e3)
    init = [grids.initial_particles(tubes[0], spec, mi, seed=3)]
    a, b = _solver(mi, tubes, init, vg), _solver(mi, tubes, init, vg)
    for _ in range(12):
        a.step(1)
    b.step(12)
    assert a.launch()[0] in (1024, 2048, 4096) and b.launch()[0] in (1024, 2048, 4096)
    for x, y in zip(_state(a, 1), _state(b, 1)):
        np.testing.assert_array_equal(x, y)


@pytest.mark.parametrize("prec", PRECS)
@pytest.mark.parametrize("slots", [0, (1 << 21) + 1000])
@pytest.mark.parametrize("collisions", [False, True])
def test_counts_hold_between_master_steps(prec, slots, collisions):
    """kaos_get_counts returns the counts of the latest master step whatever
    has been stepped since -- the launch-shape timing among it, which runs at
    the first steps and again after single steps -- and a launch shape set by
    hand (no timing at all) gives the same ones."""
    mi = ModelInput(h=0.01, ndatfac=5, ION2VPERPflag=1, ICRflag=1, precision=prec,
                    QEXCHANGEflag=1 if collisions else 0)
    spec = TubeSpec(L=3.0, nq=24, n_particles=30000, q_ub=0.5, H=400e3, heat_rate_eV_s=2.0,
                    neut_n0=1e18 if collisions else 0.0, neut_H=300e3)
    t = make_tube(spec, mi)
    t.capacity = max(t.capacity, slots)
    vg = make_vgrid(True, 8, 8, 12, 9e3)
    init = [grids.initial_particles(t, spec, mi, seed=3)]
    s, f = _solver(mi, [t], init, vg), _solver(mi, [t], init, vg)
    f.set_launch(2048, 0)
    for x in (s, f):
        x.set_export(True)
    last = None
    for n in range(1, 18):
        s.step(1)
        f.step(1)
        now = [s.counts(), s.counts(full=True)]
        if n == 1 or n % 5 == 0:
            last = now
        for x, y, z in zip(now, last, (f.counts(), f.counts(full=True))):
            np.testing.assert_array_equal(x, y, err_msg=str(n))
            np.testing.assert_array_equal(x, z, err_msg=str(n))
    assert last[0].sum() > 0
    s.set_launch(0, 0)  # timed again, in the middle of an interval
    s.step(1)
    np.testing.assert_array_equal(s.counts(), last[0])
    np.testing.assert_array_equal(s.counts(full=True), last[1])
    s.close()
    f.close()


@pytest.mark.parametrize("drift", [1e-4, 3e-3, 1e-2, 3e-2])
def test_fp64_long_steps_end_on_the_field_line(drift):
    """One FP64 step of a given length over radius: the re-projected point lies
    on the tube's field line, r = RE p sin^2(theta), to rounding -- the radius,
    the root and the two coordinates carry a few units of 2^-53 each, eight in
    all -- however far the Runge-Kutta point had left the line."""
    mi = ModelInput(h=10.0, ndatfac=50, ION2VPERPflag=1)
    spec = TubeSpec(L=4.0, nq=24, n_particles=2000, q_ub=0.15, H=600e3)
    t = make_tube(spec, mi)
    n = 2000
    rng = np.random.default_rng(5)
    q = rng.uniform(t.qGC[-4], t.qGC[3], n)
    r = grids.dipole_q_to_rtheta(q, t.pG)[0]
    v = drift * r / mi.h * rng.choice([-1.0, 1.0], n)
    s = Solver(mi, [t], make_vgrid(True, 8, 8, 8, 1e6))
    s.load(0, q, v, np.zeros(n), np.zeros(n))
    s.step(1)
    p = s.particles()
    s.close()
    rho, z = p["rho"].astype(np.longdouble), p["z"].astype(np.longdouble)
    rr = np.sqrt(rho * rho + z * z)
    off = rr * rr * rr / (grids.RE * t.pG * rho * rho) - 1
    assert np.max(np.abs(off)) < 8 * 2.0 ** -52


@pytest.mark.parametrize("prec", PRECS)
@pytest.mark.parametrize("nq,slots", [(2048, 0), (2048, 600_000), (700, 0), (24, 300_000)])
def test_runs_of_many_cells(prec, nq, slots):
    """Runs of two and of seventeen steps and one-step pushes on both sides of
    the lines where the items grow with the cells, the slots and the run's
    length, and of the small items of one-step pushes: bit for bit."""
    mi = ModelInput(h=0.01, ndatfac=18, ION2VPERPflag=1, ICRflag=1, precision=prec)
    spec = TubeSpec(L=4.0, nq=nq, n_particles=6000, q_ub=0.1, H=600e3, heat_rate_eV_s=5.0)
    t = make_tube(spec, mi)
    t.capacity = max(t.capacity, slots)
    vg = make_vgrid(True, 16, 16, 24, 8e3)
    init = [grids.initial_particles(t, spec, mi, seed=2)]
    a, b = _solver(mi, [t], init, vg), _solver(mi, [t], init, vg)
    for n in (1, 16, 1, 2, 15, 1):
        a.step(n)
        for _ in range(n):
            b.step(1)
    for x, y in zip(_state(a, 1), _state(b, 1)):
        np.testing.assert_array_equal(x, y)
    a.close()
    b.close()

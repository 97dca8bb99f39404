"""Statistical validation of the stochastic terms on the GPU.

The reference draws from gfortran's unseeded random_number
(GaussianRNGSub _3_1_GaussianRNG.f90:27-37, PoissonRNGSub
_3_2_PoissonRNG.f90:27-42, used by WaveHeatingSub
_8_1_1_0_WaveHeating.f90:141-150 and IonNeutralCollisionFrequencyASub
_8_6_6_1_...:275-301), which cannot be reproduced, so the stochastic terms
are checked by their distributions:

* the device Philox4x32-10 against the published known-answer vectors;
* the FP32 Gaussian pair of the mixed push's heating kick and the FP64 pair
  of the FP64 push (kaos_sample_rng evaluates the same device functions):
  mean, variance, tail fractions, independence of the pair, a KS test
  against the normal law, and agreement of the two precisions;
* the collision-count Poisson draw: mean and a chi-square test of its
  distribution for several means;
* a seed ensemble: 20 oracle runs and 20 mixed-precision GPU runs of a
  heated tube with charge exchange, from the same initial ions with
  different random streams -- every moment of every cell agrees between
  the ensembles (difference of means within 3 sigma), and one further GPU
  run lies within 3 sigma of the oracle ensemble;
* two-sample KS tests on the V|| and Vperp marginals of the distribution
  function, pooled and per cell (cells with >= 80 ions), between a GPU
  run and an oracle run with
  different streams (and a heated against an unheated run, which must
  fail: the test has power).
"""
import dataclasses
import math

import numpy as np
import pytest
from scipy import stats

from kaos_b200 import build as kbuild
from kaos_b200 import grids
from kaos_b200 import lib as klib
from kaos_b200.lib import Solver
from kaos_b200.model_input import (KAOS_EAMAG, KAOS_M0, KAOS_M1PAR, KAOS_M1PERP1,
                                   KAOS_M1PERP2, KAOS_M2, KAOS_M2PAR, KAOS_M2PERP1,
                                   KAOS_M2PERP2, KAOS_NQ, KAOS_PREC_MIXED)
from oracle.oracle import Oracle

pytestmark = pytest.mark.gpu

MOMENTS = [KAOS_M0, KAOS_M1PAR, KAOS_M1PERP1, KAOS_M1PERP2, KAOS_M2, KAOS_M2PAR,
           KAOS_M2PERP1, KAOS_M2PERP2, KAOS_NQ, KAOS_EAMAG]
ENSEMBLE = 20
STEPS = 25  # master steps at 5, 10, 15, 20, 25


@pytest.fixture(scope="module", autouse=True)
def _build():
    kbuild.build()


# ---- generators ------------------------------------------------------------
PHILOX_KAT = [
    ((0, 0, 0, 0), (0, 0), (0x6627e8d5, 0xe169c58d, 0xbc57ac4c, 0x9b00dbd8)),
    ((0xffffffff,) * 4, (0xffffffff, 0xffffffff),
     (0x408f276d, 0x41c83b0e, 0xa20bc7c6, 0x6d5451fd)),
    ((0x243f6a88, 0x85a308d3, 0x13198a2e, 0x03707344), (0xa4093822, 0x299f31d0),
     (0xd16cfe09, 0x94fdcceb, 0x5001e420, 0x24126ea1)),
]


@pytest.mark.parametrize("ctr,key,want", PHILOX_KAT)
def test_device_philox_known_answers(ctr, key, want):
    w = klib.sample_rng(klib.SAMPLE_PHILOX, 1, seed=key[0] | (key[1] << 32),
                        id0=ctr[0] | (ctr[1] << 32), step=ctr[2], c3=ctr[3])
    assert [int(x) for x in w[0]] == list(want)


@pytest.fixture(scope="module")
def gauss():
    n = 4_000_000
    g32 = klib.sample_rng(klib.SAMPLE_GAUSS32, n, seed=20261203, id0=1 << 20, step=77)
    g64 = klib.sample_rng(klib.SAMPLE_GAUSS64, n, seed=20261203, id0=1 << 20, step=77)
    return g32, g64


def test_table_reduced_gaussian_pair_equals_fp64_pair(gauss):
    """The Gaussian pair of the KAOS_PREC_MIXED_K64 kick (table-reduced FP64
    logarithm and sine/cosine, kaos_f64.cuh) against the FP64 push's pair
    from the same Philox words: equal to a few units of 2^-52."""
    n = len(gauss[1])
    g64t = klib.sample_rng(klib.SAMPLE_GAUSS64T, n, seed=20261203, id0=1 << 20, step=77)
    assert np.max(np.abs(g64t - gauss[1])) < 1e-14


@pytest.mark.parametrize("which", [0, 1])
def test_gaussian_moments_tails_ks(gauss, which):
    g = gauss[which]
    x = g.ravel()
    n = len(x)
    assert abs(x.mean()) < 5.0 / math.sqrt(n)
    assert abs(x.var() - 1.0) < 5.0 * math.sqrt(2.0 / n)
    for t in (2.0, 3.0, 4.0):
        p = math.erfc(t / math.sqrt(2.0))
        k = np.count_nonzero(np.abs(x) > t)
        assert abs(k - n * p) < 5.0 * math.sqrt(n * p * (1 - p)) + 2, (t, k, n * p)
    # the two members of a pair are independent
    r = np.corrcoef(g[:, 0], g[:, 1])[0, 1]
    assert abs(r) < 5.0 / math.sqrt(len(g))
    assert stats.kstest(x, "norm").pvalue > 1e-4
    if which == 0:
        # 23-bit uniforms: |G| <= sqrt(-2 ln 2^-24) = 5.77 (tail truncated at
        # a probability of 8e-9)
        assert np.max(np.abs(x)) <= 5.78


def test_gaussian_fp32_tracks_fp64(gauss):
    """Same Philox words, 23-bit uniforms and hardware functions against
    53-bit uniforms and FP64 functions: the pairs agree closely except for
    the rare draws whose first uniform lies within 2^-23 of 1."""
    d = np.abs(gauss[0] - gauss[1])
    assert np.median(d) < 1e-6
    assert np.quantile(d, 0.999) < 1e-5


@pytest.mark.parametrize("lam", [0.05, 0.7, 3.0, 12.0])
def test_poisson_draw(lam):
    n = 200_000
    k = klib.sample_rng(klib.SAMPLE_POISSON, n, seed=99, id0=0, step=5, lam=lam)[:, 0]
    assert np.all(k == np.round(k)) and k.min() >= 0
    assert abs(k.mean() - lam) < 5.0 * math.sqrt(lam / n)
    kmax = int(lam + 6 * math.sqrt(lam) + 3)
    obs = np.bincount(k.astype(np.int64), minlength=kmax + 1)
    exp = stats.poisson.pmf(np.arange(len(obs)), lam) * n
    exp[-1] += stats.poisson.sf(len(obs) - 1, lam) * n
    # lump the bins whose expectation is below 5 into their neighbours
    o2, e2, acc_o, acc_e = [], [], 0.0, 0.0
    for a, b in zip(obs, exp):
        acc_o += a
        acc_e += b
        if acc_e >= 5.0:
            o2.append(acc_o)
            e2.append(acc_e)
            acc_o = acc_e = 0.0
    if acc_e > 0:
        o2[-1] += acc_o
        e2[-1] += acc_e
    o2, e2 = np.array(o2), np.array(e2)
    if len(o2) > 1:
        chi2 = float(np.sum((o2 - e2) ** 2 / e2))
        assert stats.chi2.sf(chi2, len(o2) - 1) > 1e-4, (lam, chi2)


# ---- seed ensembles ------------------------------------------------------------
def heated_tube(seed, mixed=False, heating=True):
    mi, spec, tube, vg = grids.config_small(n_particles=4000, three_d=True,
                                            steps_per_master=5, heating=heating,
                                            collisions=True)
    mi = dataclasses.replace(mi, seed=seed)
    if mixed:
        mi = dataclasses.replace(mi, precision=KAOS_PREC_MIXED)
    init = grids.initial_particles(tube, spec, mi, seed=3)
    return mi, tube, vg, init


def run_oracle(seed, heating=True):
    mi, tube, vg, init = heated_tube(seed, heating=heating)
    o = Oracle(mi, tube, vg)
    o.load(*init)
    o.step(STEPS)
    return o


def run_gpu(seed):
    mi, tube, vg, init = heated_tube(seed, mixed=True)
    s = Solver(mi, [tube], vg)
    s.load(0, *init)
    s.step(STEPS)
    return s


def moments(r):
    return np.stack([r.moments(m) for m in MOMENTS])


@pytest.fixture(scope="module")
def ensembles():
    mo = np.stack([moments(run_oracle(1 + k)) for k in range(ENSEMBLE)])
    mg = np.stack([moments(run_gpu(1001 + k)) for k in range(ENSEMBLE)])
    return mo, mg


def _worst(z, live, mu_a, mu_b, sd_a, sd_b, k=5):
    """The k largest deviations: (z, moment, cell, mean a, mean b, sd a, sd b)."""
    idx = np.argwhere(live)
    order = np.argsort(z)[::-1][:k]
    return [(round(float(z[o]), 2), MOMENTS[idx[o][0]], int(idx[o][1]),
             float(mu_a[tuple(idx[o])]), float(mu_b[tuple(idx[o])]),
             float(sd_a[tuple(idx[o])]), float(sd_b[tuple(idx[o])])) for o in order]


def test_ensemble_means_agree(ensembles):
    mo, mg = ensembles
    K = ENSEMBLE
    mu_o, mu_g = mo.mean(0), mg.mean(0)
    sd_o, sd_g = mo.std(0, ddof=1), mg.std(0, ddof=1)
    # standard error of the difference of means, with a floor of 1e-9 of the
    # moment's scale (entries whose spread is rounding noise)
    scale = np.max(np.abs(mu_o), axis=1, keepdims=True)
    se = np.sqrt((sd_o ** 2 + sd_g ** 2) / K + (1e-9 * scale) ** 2)
    live = (sd_o > 0) | (sd_g > 0)
    # entries without spread are deterministic: equal on both sides
    assert np.all(np.abs(mu_g - mu_o)[~live] <= 1e-6 * np.broadcast_to(scale, mu_o.shape)[~live])
    z = np.abs(mu_g - mu_o)[live] / se[live]
    assert live.sum() > 100
    worst = _worst(z, live, mu_o, mu_g, sd_o, sd_g)
    assert np.mean(z > 3.0) <= 0.02, worst
    assert z.max() < 5.0, worst


def test_single_gpu_run_within_3_sigma(ensembles):
    mo, _ = ensembles
    K = ENSEMBLE
    mu, sd = mo.mean(0), mo.std(0, ddof=1)
    m = moments(run_gpu(777))
    live = sd > 0
    scale = np.max(np.abs(mu), axis=1, keepdims=True)
    se = np.sqrt(sd ** 2 * (1.0 + 1.0 / K) + (1e-9 * scale) ** 2)
    z = np.abs(m - mu)[live] / se[live]
    worst = _worst(z, live, mu, m, sd, sd)
    assert np.mean(z > 3.0) <= 0.03, worst
    assert z.max() < 6.0, worst


def ks_samples(r):
    p = r.particles()
    return p["qind"], p["vpar"], p["vperp1"], p["vperp2"]


def test_distribution_function_ks():
    g = ks_samples(run_gpu(4242))
    o = ks_samples(run_oracle(4343))
    cold = ks_samples(run_oracle(4343, heating=False))
    # pooled marginals: same law; a heated run against an unheated one differs
    for a in (1, 2, 3):
        assert stats.ks_2samp(g[a], o[a]).pvalue > 1e-3, a
    assert stats.ks_2samp(g[2], cold[2]).pvalue < 1e-6
    # per cell: V||, Vperp1, Vperp2 of every cell holding >= 80 ions
    pv = []
    for c in np.unique(o[0]):
        if c < 0:
            continue
        mg, mo_ = g[0] == c, o[0] == c
        if mg.sum() < 80 or mo_.sum() < 80:
            continue
        for a in (1, 2, 3):
            pv.append(stats.ks_2samp(g[a][mg], o[a][mo_]).pvalue)
    pv = np.array(pv)
    assert len(pv) >= 30
    assert np.mean(pv < 0.01) <= 0.05, np.sort(pv)[:10]
    assert pv.min() > 1e-5


@pytest.mark.parametrize("lam,chi2", [(0.0, 1.7), (20.0, 0.9), (-20.0, 1.7)])
def test_fp64_kick_against_extended_precision(lam, chi2):
    """One FP64 step's kick, ion by ion, against the reference's formula in
    64-bit mantissas on the same Philox words: the sum of the roundings on its
    way -- the position's two coordinates and the seven operations of Omega
    (times 0.6), the exponent's four, the roots', the product's and the draw's
    eight -- stays below 16 units of 2^-52 of the kick's own size, also where
    the draw's uniform is next to 1 and the radius small.  A negative
    lambdaPerp leaves the Sigma factor out (Sigma < 1)."""
    LD = np.longdouble
    pi = LD("3.14159265358979323846264338327950288")
    mi = grids.ModelInput(h=0.005, ndatfac=50, ION2VPERPflag=1, ICRflag=1, EAMBflag=0, GRAVflag=0)
    spec = grids.TubeSpec(L=4.0, nq=97, n_particles=1000, q_ub=1e-3, heat_rate_eV_s=1e-3)
    t = grids.make_tube(spec, mi)
    t.lambdaPerp, t.ChiPerp2 = np.full(t.nq, lam), np.full(t.nq, chi2)
    n = 1 << 19
    t.capacity = n
    rng = np.random.default_rng(3)
    q = rng.uniform(t.qGC[-2], t.qGC[1], n)
    vpar = rng.normal(size=n) * 2e3 * 10.0 ** rng.uniform(-3, 1, n)
    v = rng.normal(size=(2, n)) * 3e3 if lam else np.zeros((2, n))
    s = Solver(mi, [t], grids.make_vgrid(True, 16, 16, 16, 1e5))
    s.load(0, q, vpar, *v)
    s.step(1)
    got = s.state()
    s.close()
    w = klib.sample_rng(klib.SAMPLE_PHILOX, n, seed=mi.seed, id0=0, step=1,
                        c3=1 << 24).astype(np.uint64)
    u = [(((w[:, k] << np.uint64(32)) | w[:, k + 1]) >> np.uint64(11)).astype(float) + 0.5
         for k in (0, 2)]
    u1, u2 = (x * 2.0 ** -53 for x in u)
    assert np.max(u1) > 1 - 1e-5
    R = np.sqrt(-2 * np.log(u1.astype(LD)))
    k = np.rint(4 * u2)
    a = 2 * pi * (u2.astype(LD) - k.astype(LD) / 4)
    c_, s_ = np.cos(a), np.sin(a)
    k = k.astype(int) & 3
    g = [R * np.choose(k, [c_, -s_, -c_, s_]), R * np.choose(k, [s_, c_, -s_, -c_])]
    Q, pG, r0 = q.astype(LD), LD(t.pG), LD(grids.RE)
    x = np.full(n, LD(1.5))
    for _ in range(20):
        x = x - (Q * Q * x ** 4 + x / pG - 1) / (4 * Q * Q * x ** 3 + 1 / pG)
    ell = 1 + 3 * (Q * x * x) ** 2
    Om = LD(mi.qs) / LD(mi.ms) * LD(8.06e15) * np.sqrt(ell) / (x * r0) ** 3
    cell = np.clip(np.searchsorted(-t.qGH, -q), 0, t.nq - 1)
    y = Om * np.abs(vpar.astype(LD)) / LD(t.sumdsICR)
    on = y <= (2 * pi / LD(mi.h)) ** 2
    amp = np.sqrt(np.sqrt(y))
    if lam > 0:
        sig = 2 * pi * np.sqrt(v[0].astype(LD) ** 2 + v[1].astype(LD) ** 2) / (Om * LD(lam))
        amp = np.where(sig >= 1, amp * sig ** LD(-1.5), amp)
        on &= np.abs(sig - 1) > 1e-12  # (the factor jumps there)
    pre = (LD(mi.qs) ** 2 / (2 * LD(mi.ms) ** 2)) * t.S0[cell] * t.EtaLH[cell]
    for key, v0, xi, chi, gi in (("vperp1", v[0], t.XiPerp1, t.ChiPerp1, g[0]),
                                 ("vperp2", v[1], t.XiPerp2, t.ChiPerp2, g[1])):
        kick = LD(mi.h) * np.sqrt(pre * xi[cell] / LD(np.pi)) * amp * gi * \
            (Om / t.OmegaG0[cell].astype(LD)) ** (-chi[cell].astype(LD) / 2)
        scale = np.abs(v0) + np.abs(kick)
        use = on & (np.abs(gi) > 1e-6 * R)  # (a zero of the sine has no relative error)
        err = (np.abs(got[key] - (v0 + kick)) / scale)[use]
        assert np.max(err) < 16 * 2.0 ** -52, key


def test_fp64_pair_radius_next_to_zero():
    """The radius of the FP64 push's Gaussian pair, relative, against 64-bit
    mantissas on the same Philox words, uniforms next to 1 among them: a
    quarter unit of 2^-52 from the logarithm and half a unit each from the
    root, the products and the sine and cosine."""
    n = 1 << 21
    g = klib.sample_rng(klib.SAMPLE_GAUSS64, n, seed=77, id0=5, step=9).astype(np.longdouble)
    w = klib.sample_rng(klib.SAMPLE_PHILOX, n, seed=77, id0=5, step=9, c3=1 << 24).astype(np.uint64)
    u1 = ((((w[:, 0] << np.uint64(32)) | w[:, 1]) >> np.uint64(11)).astype(float) + 0.5) * 2.0 ** -53
    assert np.max(u1) > 1 - 1e-5
    R = np.sqrt(-2 * np.log(u1.astype(np.longdouble)))
    assert np.max(np.abs(np.sqrt((g ** 2).sum(axis=1)) / R - 1)) < 2 * 2.0 ** -52

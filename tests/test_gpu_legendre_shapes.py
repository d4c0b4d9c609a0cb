"""FP64 Legendre kernels at the edges of their tiles, against the oracle: ring
pair counts around the shapes the launchers choose by (128, 256, 512 pairs) and
around a warp, l ranges around the 16-, 32- and 64-step chunks, spins with
m < s, orders that no ring reaches, several transforms per pass, and rings that
never leave the scaled regime.  Tolerance: 1e-12 relative L2, the FP64 bar of
the parity tests."""
import numpy as np
import pytest

import sharp_b200 as sb
import sht_oracle as so
from helpers import rel_l2, uniform_alm

pytestmark = pytest.mark.gpu


def _geometries(npairs, nphi, theta_max=np.pi / 2, unpaired=False):
    """npairs symmetric ring pairs (the last one a single equator ring if unpaired)."""
    th = (np.arange(npairs) + 0.5) * theta_max / npairs
    if unpaired:
        th[-1] = np.pi / 2
        th = np.concatenate([th, np.pi - th[:-1]])
    else:
        th = np.concatenate([th, np.pi - th])
    n = len(th)
    args = (np.full(n, nphi), np.arange(n) * nphi, np.ones(n, np.int64),
            np.linspace(0.0, 0.3, n), th, np.linspace(0.5, 1.5, n))
    g = sb.Geometry.general(*args)
    assert g.npairs == npairs
    return g, so.make_geom_info(*args), n * nphi


CASES = [(1, 15, 3), (31, 16, 16), (32, 31, 5), (33, 32, 9), (127, 33, 4), (128, 64, 7),
         (129, 63, 6), (255, 40, 3), (256, 65, 5), (257, 17, 3), (511, 47, 2), (512, 48, 3),
         (513, 97, 4), (700, 20, 2), (1025, 34, 2), (40, 200, 200)]


def _check(geo, lmax, mmax, spin, ntrans, seed):
    g, og, npix = geo
    a, oa = sb.AlmInfo.triangular(lmax, mmax), so.triangular_alm_info(lmax, mmax)
    nc = 1 if spin == 0 else 2
    alms = [uniform_alm(lmax, mmax, seed=seed + i, spin=spin) for i in range(nc * ntrans)]
    rng = np.random.default_rng(seed)
    maps = [rng.uniform(-1, 1, npix) for _ in alms]
    got_m, want_m = ([np.zeros(npix) for _ in alms] for _ in range(2))
    got_a, want_a = ([np.full_like(x, 7.0) for x in alms] for _ in range(2))
    sb.execute(sb.SHARP_ALM2MAP, spin, [x.copy() for x in alms], got_m, g, a, ntrans, sb.SHARP_DP)
    sb.execute(sb.SHARP_MAP2ALM, spin, got_a, [x.copy() for x in maps], g, a, ntrans, sb.SHARP_DP)
    so.execute(so.SHARP_ALM2MAP, spin, [x.copy() for x in alms], want_m, og, oa, ntrans, so.SHARP_DP)
    so.execute(so.SHARP_MAP2ALM, spin, want_a, [x.copy() for x in maps], og, oa, ntrans, so.SHARP_DP)
    for x, y in zip(got_m + got_a, want_m + want_a):
        assert rel_l2(x, y) < 1e-12
    if ntrans > 1:   # the last transform alone: the same bits
        m1, a1 = ([np.zeros_like(x) for x in y[-nc:]] for y in (got_m, got_a))
        sb.execute(sb.SHARP_ALM2MAP, spin, [x.copy() for x in alms[-nc:]], m1, g, a, 1, sb.SHARP_DP)
        sb.execute(sb.SHARP_MAP2ALM, spin, a1, [x.copy() for x in maps[-nc:]], g, a, 1, sb.SHARP_DP)
        for x, y in zip(m1 + a1, got_m[-nc:] + got_a[-nc:]):
            assert np.array_equal(x, y)


@pytest.mark.parametrize("spin", [0, 2])
@pytest.mark.parametrize("npairs,lmax,mmax", CASES)
def test_tile_edges(npairs, lmax, mmax, spin):
    _check(_geometries(npairs, 2 * min(mmax, 9) + 1, unpaired=npairs % 2 == 1), lmax, mmax, spin,
           1, 100 * npairs + lmax)


@pytest.mark.parametrize("spin,ntrans", [(0, 2), (0, 4), (0, 7), (1, 3), (3, 2)])
@pytest.mark.parametrize("npairs,lmax,mmax", [(33, 33, 9), (150, 24, 5), (257, 47, 3),
                                              (600, 21, 4)])
def test_several_transforms_per_pass(npairs, lmax, mmax, spin, ntrans):
    _check(_geometries(npairs, 2 * mmax + 2), lmax, mmax, spin, ntrans, 7 * npairs)


@pytest.mark.parametrize("spin", [0, 2])
def test_polar_rings_leave_high_orders_empty(spin):
    # theta < 0.05: no ring takes part above m of about 120, most stay scaled for long
    _check(_geometries(150, 64, theta_max=0.05), 260, 260, spin, 1, 5)


def test_derivatives_at_tile_edges():
    for npairs, lmax in ((129, 33), (513, 18)):
        (g, og, npix), mmax = _geometries(npairs, 9), 4
        a, oa = sb.AlmInfo.triangular(lmax, mmax), so.triangular_alm_info(lmax, mmax)
        alms = [uniform_alm(lmax, mmax, seed=i) for i in range(3)]
        got, want = ([np.zeros(npix) for _ in range(6)] for _ in range(2))
        sb.execute(sb.SHARP_ALM2MAP_DERIV1, 1, [x.copy() for x in alms], got, g, a, 3, sb.SHARP_DP)
        so.execute(so.SHARP_ALM2MAP_DERIV1, 1, [x.copy() for x in alms], want, og, oa, 3, so.SHARP_DP)
        for x, y in zip(got, want):
            assert rel_l2(x, y) < 1e-12


def test_undefined_pixels_stay_out_of_orders_their_ring_does_not_reach():
    # a NaN on a polar ring spoils only the a_lm whose functions are not negligible there
    (g, _, npix), lmax = _geometries(64, 9), 300
    a = sb.AlmInfo.triangular(lmax, lmax)
    for spin in (0, 2):
        nc = 1 if spin == 0 else 2
        maps = [np.ones(npix) for _ in range(nc)]
        out = [np.zeros(sb.nalm_triangular(lmax), np.complex128) for _ in range(nc)]
        maps[0][0] = np.nan
        sb.execute(sb.SHARP_MAP2ALM, spin, out, maps, g, a, 1, sb.SHARP_DP)
        m = np.concatenate([np.full(lmax + 1 - k, k) for k in range(lmax + 1)])
        l = np.concatenate([np.arange(k, lmax + 1) for k in range(lmax + 1)])
        assert np.isnan(out[0][(m == 0) & (l >= spin)]).all()
        assert np.isfinite(out[0][m > 250]).all()

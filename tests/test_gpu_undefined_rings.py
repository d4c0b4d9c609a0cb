"""Undefined pixels in the FP64 analysis: a ring takes part in an a_lm from the l on
where its function leaves the scaled regime, so a NaN on it must reach the later a_lm
of that order and none of the earlier ones, also where its warp holds rings that
are active from the start.

Which a_lm a ring takes part in is read off a map that is zero but for one pixel of
the ring: exactly those that are not zero.  The NaN in the same pixel must then
spoil exactly these."""
import numpy as np
import pytest

import sharp_b200 as sb

pytestmark = pytest.mark.gpu

THETA = 0.0123   # of the spoiled ring
NPHI = 9


def _geometry(npairs):
    """npairs symmetric pairs, THETA first, the others from 0.02 to the equator."""
    th = np.concatenate([[THETA], np.linspace(0.02, 1.57, npairs - 1)])
    th = np.concatenate([th, np.pi - th])
    n = len(th)
    g = sb.Geometry.general(np.full(n, NPHI), np.arange(n) * NPHI, np.ones(n, np.int64),
                            np.linspace(0.1, 0.4, n), th, np.ones(n))
    assert g.npairs == npairs
    return g, n * NPHI


def _analyse(g, npix, spin, lmax, ntrans, value):
    """a_lm of ntrans transforms of zero maps with `value` in the first pixel of the
    first map of the last transform."""
    nc = 1 if spin == 0 else 2
    a = sb.AlmInfo.triangular(lmax, lmax)
    maps = [np.zeros(npix) for _ in range(nc * ntrans)]
    maps[-nc][0] = value
    out = [np.full(sb.nalm_triangular(lmax), 3.0, np.complex128) for _ in maps]
    sb.execute(sb.SHARP_MAP2ALM, spin, out, maps, g, a, ntrans, sb.SHARP_DP)
    return out


# pair counts of each shape of the analysis kernels, one and several transforms
@pytest.mark.parametrize("ntrans", [1, 2])
@pytest.mark.parametrize("npairs", [40, 200, 400, 700])
@pytest.mark.parametrize("spin", [0, 2])
def test_nan_reaches_exactly_the_alm_its_ring_takes_part_in(spin, npairs, ntrans):
    lmax, nc = 300, 1 if spin == 0 else 2
    g, npix = _geometry(npairs)
    unit = _analyse(g, npix, spin, lmax, ntrans, 1.0)
    spoiled = _analyse(g, npix, spin, lmax, ntrans, np.nan)
    m = np.concatenate([np.full(lmax + 1 - k, k) for k in range(lmax + 1)])
    l = np.concatenate([np.arange(k, lmax + 1) for k in range(lmax + 1)])
    for x, y in zip(unit[:-nc], spoiled[:-nc]):    # the other transforms hold no NaN
        assert (x == 0).all() and (y == 0).all()
    for x, y in zip(unit[-nc:], spoiled[-nc:]):
        # at m = 0 the a_lm are real and half of the terms vanish by themselves
        assert np.array_equal((x != 0)[m > 0], np.isnan(y)[m > 0])
        # the orders that matter here are there: some the ring enters after the start
        late = [k for k in range(1, lmax + 1)
                if (x[(m == k) & (l < k + 16)] == 0).all() and (x[m == k][-1] != 0)]
        assert len(late) >= 10
    assert np.isnan(spoiled[-nc][(m == 0) & (l >= spin)]).all()

"""Ring FFT kernels against the oracle: every length of the short-ring kernels
(direct sums, power-of-two passes, Bluestein), odd rings in pairs and alone,
pairs of unequal lengths, alias folding (lengths below 2 mmax), phi0, weights,
strides, SHARP_ADD and single-precision arrays.  Tolerances: 1e-12 relative L2 in
double (the FP64 bar of the parity tests), 1e-6 with float arrays (a float has
2^-24 = 6e-8 per value)."""
import numpy as np
import pytest

import sharp_b200 as sb
import sht_oracle as so
from helpers import rel_l2, uniform_alm

pytestmark = pytest.mark.gpu


def _rings(lengths, mode, stride=1):
    """One ring pair per length ("pair"), one ring ("single"), or a pair whose
    southern ring is longer by two ("unequal")."""
    th, nph = [], []
    for i, n in enumerate(lengths):
        t = 0.2 + 1.3 * (i + 0.5) / len(lengths)
        th.append(t)
        nph.append(n)
        if mode != "single":
            th.append(np.pi - t)
            nph.append(n + (2 if mode == "unequal" else 0))
    nph = np.array(nph)
    ofs = np.concatenate([[0], np.cumsum(nph * stride)[:-1]]) + 1
    k = len(nph)
    args = (nph, ofs, np.full(k, stride), np.linspace(0.0, 1.1, k), np.array(th),
            np.linspace(0.5, 1.5, k))
    return sb.Geometry.general(*args), so.make_geom_info(*args), int(ofs[-1] + nph[-1] * stride) + 3


def _check(lengths, mode, lmax, mmax, spin=0, ntrans=1, dp=True, add=False, stride=1):
    g, og, npix = _rings(lengths, mode, stride)
    a, oa = sb.AlmInfo.triangular(lmax, mmax), so.triangular_alm_info(lmax, mmax)
    nc = (1 if spin == 0 else 2) * ntrans
    real, cpx = (np.float64, np.complex128) if dp else (np.float32, np.complex64)
    rng = np.random.default_rng(lmax + len(lengths))
    alms = [uniform_alm(lmax, mmax, seed=i, spin=spin).astype(cpx) for i in range(nc)]
    maps = [rng.uniform(-1, 1, npix).astype(real) for _ in range(nc)]
    flags = (sb.SHARP_DP if dp else 0) | (sb.SHARP_ADD if add else 0)
    m0 = [rng.uniform(-1, 1, npix).astype(real) for _ in range(nc)]
    a0 = [uniform_alm(lmax, mmax, seed=50 + i, spin=spin).astype(cpx) for i in range(nc)]
    gm, wm, ga, wa = ([x.copy() for x in y] for y in (m0, m0, a0, a0))
    sb.execute(sb.SHARP_ALM2MAP, spin, [x.copy() for x in alms], gm, g, a, ntrans, flags)
    sb.execute(sb.SHARP_MAP2ALM, spin, ga, [x.copy() for x in maps], g, a, ntrans, flags)
    wide = [[x.astype(np.float64 if x.dtype.kind == "f" else np.complex128) for x in y]
            for y in (alms, wm, wa, maps)]
    oflags = so.SHARP_DP | (so.SHARP_ADD if add else 0)
    used = np.zeros(npix, bool)
    for pr in og.pairs:
        for r in pr:
            if r is not None and r.nph > 0:
                used[r.ofs:r.ofs + r.nph * r.stride:r.stride] = True
    if not add:
        for x in wide[1]:
            x[used] = 0.0
        wide[2] = [np.zeros_like(x) for x in wide[2]]
    so.execute(so.SHARP_ALM2MAP, spin, wide[0], wide[1], og, oa, ntrans, oflags)
    so.execute(so.SHARP_MAP2ALM, spin, wide[2], wide[3], og, oa, ntrans, oflags)
    tol = 1e-12 if dp else 1e-6
    for x, y in zip(gm + ga, wide[1] + wide[2]):
        assert rel_l2(x, y) < tol
    for x, y in zip(gm, m0):      # pixels of no ring stay
        assert np.array_equal(x[~used], y[~used])


@pytest.mark.parametrize("mode", ["pair", "single", "unequal"])
@pytest.mark.parametrize("lo,hi", [(1, 40), (40, 70), (70, 140), (250, 270), (500, 530)])
def test_every_length(lo, hi, mode):
    _check(list(range(lo, hi)), mode, 50, 45)


@pytest.mark.parametrize("mode", ["pair", "single"])
def test_folding_of_short_rings(mode):
    _check([2, 3, 4, 5, 6, 8, 12, 16, 30, 31, 32, 33, 34, 62, 64, 66, 90, 128, 130, 200, 256, 257],
           mode, 330, 330)


def test_lengths_at_the_ends_of_the_classes():
    _check([64, 66, 126, 128, 130, 254, 256, 258, 510, 512, 514, 1022, 1024, 1026], "pair", 60, 60)
    _check([127, 129, 255, 257, 511, 513, 1001, 1023, 1025, 2047, 2049, 4095], "pair", 60, 60)
    _check([4097, 1153, 2050], "single", 40, 40)


@pytest.mark.parametrize("spin,ntrans,dp,add,stride", [(2, 2, True, False, 1), (0, 3, False, False, 1),
                                                       (1, 1, True, True, 2), (0, 1, False, True, 3)])
def test_options(spin, ntrans, dp, add, stride):
    _check([4, 7, 12, 31, 64, 65, 100, 128, 201, 256, 333, 512], "pair", 70, 64, spin, ntrans, dp,
           add, stride)

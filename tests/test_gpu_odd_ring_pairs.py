"""Pairs of odd rings, which share one transform: a ring must not see the size of
its partner's pixels beyond what the ring weights let through.  Analysis with an
excluded hemisphere (weight 0) that holds the undefined-pixel value, weights of
very different size, and weighted synthesis.  Tolerances: 1e-12 relative L2 in
double (the FP64 bar of the parity tests), 1e-6 with float arrays; per ring in
the synthesis, where each ring is an output of its own."""
import numpy as np
import pytest

import sharp_b200 as sb
import sht_oracle as so
from helpers import rel_l2, uniform_alm

pytestmark = pytest.mark.gpu

UNDEF = -1.6375e30
LENGTHS = [3, 5, 15, 31, 77, 127, 129, 255, 333, 513, 1001, 1025, 2049]


def _geometry(w_north, w_south):
    th, nph, wgt = [], [], []
    for i, n in enumerate(LENGTHS):
        t = 0.3 + 1.2 * (i + 0.5) / len(LENGTHS)
        th += [t, np.pi - t]
        nph += [n, n]
        wgt += [w_north * (1.0 + 0.1 * i), w_south * (1.0 + 0.1 * i)]
    nph = np.array(nph)
    ofs = np.concatenate([[0], np.cumsum(nph)[:-1]])
    k = len(nph)
    args = (nph, ofs, np.ones(k, np.int64), np.linspace(0.0, 1.1, k), np.array(th), np.array(wgt))
    rings = [slice(o, o + n) for o, n in zip(ofs, nph)]
    return sb.Geometry.general(*args), so.make_geom_info(*args), rings, int(nph.sum())


@pytest.mark.parametrize("dp", [True, False])
@pytest.mark.parametrize("spin", [0, 2])
@pytest.mark.parametrize("w_north,w_south,south", [
    (1.0, 0.0, UNDEF), (0.0, 1.0, 1e-20), (1.0, 1e-9, 1e9), (1e8, 1.0, 1e8)])
def test_analysis(w_north, w_south, south, spin, dp):
    g, og, rings, npix = _geometry(w_north, w_south)
    lmax = 40
    rng = np.random.default_rng(7)
    real, cpx = (np.float64, np.complex128) if dp else (np.float32, np.complex64)
    nc = 1 if spin == 0 else 2
    maps = [rng.uniform(0.5, 1.5, npix) for _ in range(nc)]
    for x in maps:
        for r in rings[1::2]:
            x[r] *= south
    maps = [x.astype(real) for x in maps]
    got = [np.zeros(sb.nalm_triangular(lmax), cpx) for _ in range(nc)]
    want = [x.astype(np.complex128) for x in got]
    sb.execute(sb.SHARP_MAP2ALM, spin, got, [x.copy() for x in maps], g,
               sb.AlmInfo.triangular(lmax), 1, sb.SHARP_DP if dp else 0)
    so.execute(so.SHARP_MAP2ALM, spin, want, [x.astype(np.float64) for x in maps], og,
               so.triangular_alm_info(lmax, lmax), 1, so.SHARP_DP)
    for x, y in zip(got, want):
        assert rel_l2(x, y) < (1e-12 if dp else 1e-6)


@pytest.mark.parametrize("dp", [True, False])
@pytest.mark.parametrize("spin", [0, 2])
@pytest.mark.parametrize("w_north,w_south", [(1.0, 0.0), (0.0, 1e6), (1.0, 1e9), (1e-9, 1.0)])
def test_weighted_synthesis(w_north, w_south, spin, dp):
    g, og, rings, npix = _geometry(w_north, w_south)
    lmax = 40
    real, cpx = (np.float64, np.complex128) if dp else (np.float32, np.complex64)
    alms = [uniform_alm(lmax, lmax, seed=3 + i, spin=spin).astype(cpx)
            for i in range(1 if spin == 0 else 2)]
    got = [np.full(npix, 7.0, real) for _ in alms]
    want = [np.zeros(npix) for _ in alms]
    sb.execute(sb.SHARP_WY, spin, [x.copy() for x in alms], got, g,
               sb.AlmInfo.triangular(lmax), 1, sb.SHARP_DP if dp else 0)
    so.execute(so.SHARP_WY, spin, [x.astype(np.complex128) for x in alms], want, og,
               so.triangular_alm_info(lmax, lmax), 1, so.SHARP_DP)
    for x, y in zip(got, want):
        for i, r in enumerate(rings):
            if (w_south if i % 2 else w_north) == 0.0:
                assert not x[r].any()
            else:
                assert rel_l2(x[r], y[r]) < (1e-12 if dp else 1e-6)

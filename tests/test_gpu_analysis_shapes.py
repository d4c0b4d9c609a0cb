"""Which shape (rings per thread, warps) the FP64 analysis takes for 257 to 512 ring
pairs: eight warps only where they take less time than four (few l).  Read from a
trace; the results at the edges of the rule against those of parts of the grid,
several transforms bit for bit as one."""
import re

import numpy as np
import pytest

import sharp_b200 as sb
from helpers import rel_l2
from test_gpu_legendre_shapes import _geometries

pytestmark = pytest.mark.gpu

NPHI = 8


def _shape(npairs, lmax, spin):
    import torch
    from torch.profiler import ProfilerActivity, profile
    mmax, nc = 3, 2 if spin else 1
    g, _, npix = _geometries(npairs, 8)
    a = sb.AlmInfo.triangular(lmax, mmax)
    alm = [torch.zeros(sb.nalm_triangular(lmax), dtype=torch.complex128, device="cuda")
           for _ in range(nc)]
    mp = [torch.zeros(npix, dtype=torch.float64, device="cuda") for _ in range(nc)]

    def call():
        sb.execute_device(sb.SHARP_MAP2ALM, spin, alm, mp, g, a, 1, sb.SHARP_DP)
        torch.cuda.synchronize()
    call()
    with profile(activities=[ProfilerActivity.CUDA]) as prof:
        for _ in range(5):   # the trace may lack the first kernels
            call()
    for e in prof.key_averages():
        k = re.search(r"anal_spin0?_kernel<1, (\d), (\d)>", e.key)
        if k:
            return int(k[1]), int(k[2])
    pytest.skip("no kernel trace on this machine")


@pytest.mark.parametrize("npairs,lmax,spin0,spin2", [
    (128, 2000, (1, 4), (1, 4)), (256, 2000, (2, 4), (2, 4)), (257, 750, (2, 8), (2, 8)),
    (288, 751, (2, 8), (3, 4)), (289, 751, (4, 4), (3, 4)), (384, 751, (4, 4), (3, 4)),
    (385, 751, (4, 4), (2, 8)), (512, 750, (2, 8), (2, 8)), (512, 2000, (4, 4), (2, 8)),
    (513, 100, (4, 4), (3, 4))])
def test_shape(npairs, lmax, spin0, spin2):
    assert _shape(npairs, lmax, 0) == spin0
    assert _shape(npairs, lmax, 2) == spin2


def _grid(th, rings, n):
    """The pairs (th, pi - th) whose pixels are those of ring numbers `rings` of n."""
    k = 2 * len(th)
    ring = np.concatenate([rings, n + rings])
    g = sb.Geometry.general(np.full(k, NPHI), ring * NPHI, np.ones(k, np.int64), 0.001 * ring,
                            np.concatenate([th, np.pi - th]), 0.5 + 0.001 * ring)
    assert g.npairs == len(th)
    return g


@pytest.mark.parametrize("spin,ntrans", [(0, 1), (2, 1), (0, 3), (2, 3)])
@pytest.mark.parametrize("npairs,lmax", [(257, 751), (288, 751), (289, 751), (384, 770), (385, 751),
                                         (512, 751), (512, 750)])
def test_results(npairs, lmax, spin, ntrans):
    # against the sum of the analyses of up to 128 pairs each, whose shape is another;
    # a ring's terms are the same bits in each, so only the order of at most 512
    # additions differs: 512 2^-53 = 6e-14 of the sum of the terms' sizes
    mmax, nc = 3, 2 if spin else 1
    th, num = (np.arange(npairs) + 0.5) * (np.pi / 2) / npairs, np.arange(npairs)
    a = sb.AlmInfo.triangular(lmax, mmax)
    size = (mmax + 1) * (mmax + 2) // 2 + (mmax + 1) * (lmax - mmax)
    rng = np.random.default_rng(npairs + lmax)
    maps = [rng.uniform(-1, 1, 2 * npairs * NPHI) for _ in range(nc * ntrans)]
    got, want, alone = ([np.zeros(size, np.complex128) for _ in maps] for _ in range(3))
    whole = _grid(th, num, npairs)
    sb.execute(sb.SHARP_MAP2ALM, spin, got, maps, whole, a, ntrans, sb.SHARP_DP)
    for i in range(0, npairs, 128):
        sb.execute(sb.SHARP_MAP2ALM, spin, want, maps, _grid(th[i:i + 128], num[i:i + 128], npairs),
                   a, ntrans, sb.SHARP_DP | sb.SHARP_ADD)
    for x, y in zip(got, want):
        assert rel_l2(x, y) < 1e-13
    for t in range(ntrans):      # one transform alone: the same bits
        k = slice(nc * t, nc * (t + 1))
        sb.execute(sb.SHARP_MAP2ALM, spin, alone[k], maps[k], whole, a, 1, sb.SHARP_DP)
    for x, y in zip(got, alone):
        assert np.array_equal(x, y)

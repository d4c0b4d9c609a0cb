"""Calls enqueued without a synchronisation between them, on one stream and on two
from two threads: kernels of a call may become resident before their predecessors
end, and all calls draw their workspace from one pool.  Each result has to be bit
for bit the one of the call made alone.  The geometry has rings of every ring
kernel: short, power-of-two and Bluestein lengths, odd pairs, pairs of unequal
lengths, single pixels."""
import threading

import numpy as np
import pytest

import sharp_b200 as sb
from helpers import uniform_alm

pytestmark = pytest.mark.gpu

PAIRS = [(1, 1), (3, 3), (4, 4), (7, 9), (31, 31), (64, 64), (100, 100), (128, 130), (333, 333),
         (512, 512), (600, 600), (1001, 1001), (1500, 1500), (2048, 2048), (2500, 2500),
         (4095, 4095), (4096, 4096), (5000, 5000), (8192, 8192), (12000, 12000)]
LMAX, SETS = 60, 12


def _geometry():
    th, nph = [], []
    for i, (a, b) in enumerate(PAIRS):
        t = 0.25 + 1.3 * (i + 0.5) / len(PAIRS)
        th += [t, np.pi - t]
        nph += [a, b]
    nph = np.array(nph)
    ofs = np.concatenate([[0], np.cumsum(nph)[:-1]])
    k = len(nph)
    return sb.Geometry.general(nph, ofs, np.ones(k, np.int64), np.linspace(0.0, 1.1, k),
                               np.array(th), np.linspace(0.5, 1.5, k)), int(nph.sum())


def _round_trip(geom, ainfo, npix, spin, alms, flags):
    """Synthesis and analysis of its maps, enqueued on the current stream."""
    import torch
    maps = [torch.zeros(npix, dtype=torch.float64, device="cuda") for _ in alms]
    back = [torch.zeros_like(a) for a in alms]
    sb.execute_device(sb.SHARP_ALM2MAP, spin, alms, maps, geom, ainfo, 1, flags)
    sb.execute_device(sb.SHARP_MAP2ALM, spin, back, maps, geom, ainfo, 1, flags)
    return maps + back


@pytest.mark.parametrize("spin,flags", [(0, sb.SHARP_DP), (2, sb.SHARP_DP)])
def test_bitwise_as_alone(spin, flags):
    import torch
    geom, npix = _geometry()
    ainfo = sb.AlmInfo.triangular(LMAX)
    sets = [[torch.from_numpy(uniform_alm(LMAX, seed=10 * k + c, spin=spin).view(np.float64)).cuda()
             for c in range(1 if spin == 0 else 2)] for k in range(SETS)]
    alone = []
    for s in sets:
        alone.append(_round_trip(geom, ainfo, npix, spin, s, flags))
        torch.cuda.synchronize()

    def same(k, got):
        assert all(torch.equal(x, y) for x, y in zip(alone[k], got)), k

    got = [_round_trip(geom, ainfo, npix, spin, s, flags) for s in sets * 3]   # one stream
    torch.cuda.synchronize()
    for i, x in enumerate(got):
        same(i % SETS, x)

    results, errors = {}, []

    def work(t):                                                           # two streams
        try:
            st = torch.cuda.Stream()
            with torch.cuda.stream(st):
                results[t] = [_round_trip(geom, ainfo, npix, spin, s, flags) for s in sets[t::2] * 3]
            st.synchronize()
        except Exception as e:   # shown by the main thread
            errors.append(e)

    threads = [threading.Thread(target=work, args=(t,)) for t in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
    for t in range(2):
        own = list(range(SETS))[t::2]
        for i, x in enumerate(results[t]):
            same(own[i % len(own)], x)


@pytest.mark.parametrize("spin", [0, 2])
def test_first_mixed_analyses_share_their_tables(spin):
    # two geometries, one lmax: the batch runs them on two streams, and the first
    # call after an emptied cache builds the coefficients that both use
    import torch
    lmax, flags = 500, sb.SHARP_DP | sb.SHARP_MIXED
    ainfo = sb.AlmInfo.triangular(lmax)
    geoms = [sb.Geometry.healpix(n) for n in (256, 128)]
    rng = np.random.default_rng(spin)
    nc = 1 if spin == 0 else 2
    maps = [[torch.from_numpy(rng.uniform(-1, 1, g.npix())).cuda() for _ in range(nc)] for g in geoms]

    def outputs():
        return [[torch.zeros(2 * sb.nalm_triangular(lmax), dtype=torch.float64, device="cuda")
                 for _ in range(nc)] for _ in geoms]

    alone = outputs()
    for g, m, a in zip(geoms, maps, alone):
        sb.execute_device(sb.SHARP_MAP2ALM, spin, a, m, g, ainfo, 1, flags)
        torch.cuda.synchronize()
    for _ in range(5):
        got = outputs()
        torch.cuda.synchronize()
        sb._lib.sharp_b200_release_cache()
        sb.execute_batch([(sb.SHARP_MAP2ALM, spin, a, m, g, ainfo, 1, flags)
                          for g, m, a in zip(geoms, maps, got)], device=True)
        torch.cuda.synchronize()
        assert all(torch.equal(x, y) for p, q in zip(got, alone) for x, y in zip(p, q))
    sb.check_device_errors()

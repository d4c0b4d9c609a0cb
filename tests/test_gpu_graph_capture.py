"""Device calls captured in a CUDA graph: after one call outside the capture, which
builds the plans, the captured call replays on changed inputs, bit for bit as the
call made directly, also after other calls have used the workspace pool and host
memory in between."""
import numpy as np
import pytest

import sharp_b200 as sb
from helpers import uniform_alm

pytestmark = pytest.mark.gpu

FP64, MIXED = sb.SHARP_DP, sb.SHARP_DP | sb.SHARP_MIXED


@pytest.mark.parametrize("flags", [FP64, MIXED])
@pytest.mark.parametrize("spin,ntrans,lmax,mmax", [(0, 1, 100, 100), (0, 13, 70, 40), (2, 1, 95, 95),
                                                   (2, 4, 64, 33)])
def test_replay(spin, ntrans, lmax, mmax, flags):
    import torch
    geom, ainfo = sb.Geometry.healpix(32), sb.AlmInfo.triangular(lmax, mmax)
    npix = 12 * 32 * 32
    nc = (1 if spin == 0 else 2) * ntrans

    def inputs(seed):
        return [torch.from_numpy(uniform_alm(lmax, mmax, seed=seed + i, spin=spin).view(np.float64)).cuda()
                for i in range(nc)]

    def call(alms, maps, back):
        sb.execute_device(sb.SHARP_ALM2MAP, spin, alms, maps, geom, ainfo, ntrans, flags)
        sb.execute_device(sb.SHARP_MAP2ALM, spin, back, maps, geom, ainfo, ntrans, flags)

    alms = inputs(0)
    maps = [torch.zeros(npix, dtype=torch.float64, device="cuda") for _ in range(nc)]
    back = [torch.zeros_like(a) for a in alms]
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        call(alms, maps, back)
    side.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=side):
        call(alms, maps, back)
    for seed in (100, 200, 300):
        new = inputs(seed)
        want_m, want_b = [torch.zeros_like(m) for m in maps], [torch.zeros_like(b) for b in back]
        call(new, want_m, want_b)
        for a, n in zip(alms, new):
            a.copy_(n)
        graph.replay()
        torch.cuda.synchronize()
        assert all(torch.equal(x, y) for x, y in zip(maps + back, want_m + want_b))
    sb.check_device_errors()

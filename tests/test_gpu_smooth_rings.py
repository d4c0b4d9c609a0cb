"""Rings whose complex length has no factor above 5, between 513 and 1024: on a grid of
such rings alone they take the direct passes (the convolution of the register
kernels was up to 1.5 times as long there), among others, as on a HEALPix grid, the
convolution.  Which kernels ran is read from a trace; the results
are compared with the oracle at 1e-12, the FP64 bar of the parity tests."""
import os
import subprocess

import numpy as np
import pytest

import sharp_b200 as sb
import sht_oracle as so
from conftest import ROOT
from helpers import rel_l2, uniform_alm
from test_launch_contract import CUDA_INCLUDE, needs_toolkit


@needs_toolkit
def test_which_lengths_the_rule_names(tmp_path):
    src, exe = tmp_path / "rule.cc", tmp_path / "rule"
    src.write_text('#include "sht_device.h"\n#include <cstdio>\nint main() {\n'
                   '  for (int n = -2; n <= 4200; ++n)\n'
                   '    if (sht::smooth_ring_length(n)) std::printf("%d ", n);\n}\n')
    subprocess.run(["g++", "-std=c++17", "-I", CUDA_INCLUDE, "-I", os.path.join(ROOT, "include"),
                    "-I", os.path.join(ROOT, "planck-levels_b200", "csrc"), str(src), "-o",
                    str(exe)], check=True)
    got = [int(x) for x in subprocess.run([str(exe)], check=True, capture_output=True,
                                          text=True).stdout.split()]
    smooth = {2**a * 3**b * 5**c for a in range(11) for b in range(7) for c in range(5)}
    assert got == [2 * n for n in range(513, 1025) if n in smooth]


def _kernels(geom, lmax, npix):
    import torch
    from torch.profiler import ProfilerActivity, profile
    a = sb.AlmInfo.triangular(lmax, lmax)
    alm = [torch.zeros(sb.nalm_triangular(lmax), dtype=torch.complex128, device="cuda")]
    mp = [torch.zeros(npix, dtype=torch.float64, device="cuda")]

    def both():
        sb.execute_device(sb.SHARP_ALM2MAP, 0, alm, mp, geom, a, 1, sb.SHARP_DP)
        sb.execute_device(sb.SHARP_MAP2ALM, 0, alm, mp, geom, a, 1, sb.SHARP_DP)
        torch.cuda.synchronize()
    both()
    with profile(activities=[ProfilerActivity.CUDA]) as prof:
        for _ in range(5):   # the trace may lack the first kernels
            both()
    names = [e.key for e in prof.key_averages()]
    if not any("legendre" in n or "spin0" in n for n in names):
        pytest.skip("no kernel trace on this machine")
    return {k for k in ("phase2ring_kernel", "ring2phase_kernel", "phase2ring_blue_kernel",
                        "ring2phase_blue_kernel") if any(k in n for n in names)}


CLASSES, CONVOLUTION = ({"phase2ring_kernel", "ring2phase_kernel"},
                        {"phase2ring_blue_kernel", "ring2phase_blue_kernel"})


@pytest.mark.gpu
@pytest.mark.parametrize("nphi,want", [(1000, CONVOLUTION), (1024, set()), (1026, CONVOLUTION),
                                       (1080, CLASSES), (1120, CONVOLUTION), (1200, CLASSES),
                                       (1536, CLASSES), (2000, CLASSES), (2160, CONVOLUTION)])
def test_route_of_a_grid_of_one_length(nphi, want):
    assert _kernels(sb.Geometry.grid("gauss", 40, nphi), 39, 40 * nphi) == want


@pytest.mark.gpu
@pytest.mark.parametrize("nside,lmax", [(512, 64), (300, 600), (512, 1100)])
def test_route_on_healpix(nside, lmax):
    # 1080, 1200, 1280 ... pixels among the other polar rings; equatorial rings of 1200
    # or (folded) 2048 pixels, more than there are others
    assert _kernels(sb.Geometry.healpix(nside), lmax, 12 * nside**2) == CONVOLUTION


@pytest.mark.gpu
@pytest.mark.parametrize("lengths", [[1080], [1200, 1280, 2000], [1026, 1080], [1080, 1200, 1026],
                                     [2048, 1536, 1250]])
@pytest.mark.parametrize("stride,lmax", [(1, 60), (2, 60), (1, 700)])
def test_results(lengths, stride, lmax):
    mmax = lmax
    th = 0.4 + 1.1 * (np.arange(len(lengths)) + 0.5) / len(lengths)
    th = np.concatenate([th, np.pi - th])
    nph = np.array(lengths * 2)
    ofs = np.concatenate([[0], np.cumsum(nph * stride)[:-1]])
    npix = int(ofs[-1] + nph[-1] * stride)
    args = (nph, ofs, np.full(len(nph), stride), np.linspace(0.0, 1.1, len(nph)), th,
            np.linspace(0.5, 1.5, len(nph)))
    g, og = sb.Geometry.general(*args), so.make_geom_info(*args)
    a, oa = sb.AlmInfo.triangular(lmax, mmax), so.triangular_alm_info(lmax, mmax)
    alm = uniform_alm(lmax, mmax, seed=len(lengths))
    mp = np.random.default_rng(lmax).uniform(-1, 1, npix)
    got_m, want_m, got_a, want_a = np.zeros(npix), np.zeros(npix), alm * 0, alm * 0
    for lib, m, b, geo, lay in ((sb, got_m, got_a, g, a), (so, want_m, want_a, og, oa)):
        lib.execute(lib.SHARP_ALM2MAP, 0, [alm.copy()], [m], geo, lay, 1, lib.SHARP_DP)
        lib.execute(lib.SHARP_MAP2ALM, 0, [b], [mp.copy()], geo, lay, 1, lib.SHARP_DP)
    assert rel_l2(got_m, want_m) < 1e-12
    assert rel_l2(got_a, want_a) < 1e-12

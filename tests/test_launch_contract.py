"""The kernel launches, as far as the sources show it: launch_overlapped takes only
arguments that convert to the kernel's parameters by themselves, as a plain launch
does, and a kernel that may start early waits for its predecessor first of all."""
import glob
import os
import re
import shutil
import subprocess

import pytest

from conftest import ROOT

CUDA_INCLUDE = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include")

SOURCE = """
#include "sht_device.h"
void kernel(const double *, double2 *, long long);
void launch(double *d, const double *cd, double2 *d2, const double2 *cd2, void *v, int n) {
  sht::launch_overlapped(&kernel, dim3(1), 32, 0, nullptr, %s);
}
"""


def _compiles(args, tmp_path):
    src = tmp_path / "launch.cc"
    src.write_text(SOURCE % args)
    cmd = ["g++", "-std=c++17", "-fsyntax-only", "-I", CUDA_INCLUDE, "-I", os.path.join(ROOT, "include"),
           "-I", os.path.join(ROOT, "planck-levels_b200", "csrc"), str(src)]
    return subprocess.run(cmd, capture_output=True, text=True).returncode == 0


needs_toolkit = pytest.mark.skipif(
    shutil.which("g++") is None or not os.path.exists(os.path.join(CUDA_INCLUDE, "cuda_runtime.h")),
    reason="needs g++ and the CUDA headers")


@needs_toolkit
@pytest.mark.parametrize("args", ["cd, d2, 1ll", "d, d2, n"])
def test_matching_arguments_compile(args, tmp_path):
    assert _compiles(args, tmp_path)


@needs_toolkit
@pytest.mark.parametrize("args", ["cd2, d2, 1ll", "cd, cd2, 1ll", "cd, d, 1ll", "v, d2, 1ll",
                                  "cd, d2, d", "n, d2, 1ll", "cd, d2"])
def test_mismatched_arguments_do_not_compile(args, tmp_path):
    assert not _compiles(args, tmp_path)


# what a kernel that may start early does first: wait for its predecessor, or, if it is
# one of a chain, what GridChain does
START = r"(?:grid_wait\(\)|const GridChain chain\(link\))\s*;"


def test_early_kernels_wait_before_anything_else():
    bodies = 0
    for path in glob.glob(os.path.join(ROOT, "planck-levels_b200", "csrc", "*.cu")):
        with open(path) as f:
            text = re.sub(r"//[^\n]*", "", f.read())
        for call in re.finditer(START, text):
            assert re.search(r"\)\s*\{\s*$", text[:call.start()]), (path, text[call.start() - 80:call.end()])
            bodies += 1
        for call in re.finditer(r"grid_release\w*\(\)\s*;", text):
            assert re.search(r"grid_wait\(\)\s*;\s*$", text[:call.start()]), path
    assert bodies >= 14


def test_kernels_of_a_chain_acquire_or_wait_and_end_after_their_predecessor():
    with open(os.path.join(ROOT, "planck-levels_b200", "csrc", "sht_device.h")) as f:
        text = re.sub(r"//[^\n]*", "", f.read())
    chain = re.sub(r"\s+", " ", text[text.index("class GridChain"):])
    chain = chain[:chain.index("bool waited_ = true;")]
    first, later = chain[chain.index("{", 20):chain.index("~GridChain")].split("} else {")
    assert first.index("grid_wait();") < first.index("st.release.gpu")
    assert "if (l.flag == nullptr || l.first)" in first
    steps = ["waited_ = __syncthreads_or(threadIdx.x == 0 && !published(l));",
             "if (waited_) grid_wait();", "fence.proxy.async.global", "grid_release"]
    assert [later.index(x) for x in steps] == sorted(later.index(x) for x in steps)
    assert "~GridChain() { if (!waited_) grid_wait(); }" in chain
    assert "ld.acquire.gpu" in chain


# pointer parameters of the kernels launched early to what an earlier kernel of the
# stream wrote (the coefficients of the staging: by the allocation-free synthesis)
WRITTEN_BEFORE = {"synth_spin0_kernel": "A", "synth_spin_kernel": "A", "anal_spin0_kernel": "phase",
                  "anal_spin_kernel": "phase", "phase2ring_pow2_kernel": "phase",
                  "phase2ring_blue_kernel": "phase", "phase2ring_short_kernel": "phase",
                  "phase2ring_odd_kernel": "phase", "stage_alm_kernel": "cfac",
                  "scatter_alm_kernel": "Aout"}


def test_early_kernels_take_earlier_results_through_plain_pointers():
    text = ""
    for path in glob.glob(os.path.join(ROOT, "planck-levels_b200", "csrc", "*.cu")):
        with open(path) as f:
            text += re.sub(r"//[^\n]*", "", f.read())
    early = re.findall(r"\n(\w+)\(([^{};]*)\)\s*\{\s*" + START, text)
    assert len(early) >= 14
    for name, params in early:
        read = re.findall(r"const double2? \*(__restrict__ )?(A|Aout|phase|cfac)\b", params)
        assert not [p for r, p in read if r and WRITTEN_BEFORE.get(name) == p], name
    assert set(WRITTEN_BEFORE) <= {name for name, _ in early}

"""Device memory that a budget is held against: no clip needs more than when the
first passes worked on 64-bit keys (the bytes below), also with a few voxels per
seed; the first pass's list entries hold every segment, voxel and label."""
import ctypes
import os
import subprocess

import pytest

SRC = r"""
#include "asv_common.cuh"
int main()
{
    for (int seg : { 0, 1, 77, ASV_MAX_CLIPS - 1 })
        for (int v : { 0, 1, 32767, 32768, 1 << 30, 0x7fffffff })
            for (int label : { 0, 1, 12345, 32766 }) {
                const asv_entry_t e = asv_entry(seg, v, label);
                if (asv_entry_seg(e) != seg || asv_entry_voxel(e) != v || asv_entry_label(e) != label) return 1;
            }
    return 0;
}
"""


def test_list_entries(tmp_path):
    from anisotropic_supervoxel_gb300 import _build
    src, exe = tmp_path / "entries.cpp", str(tmp_path / "entries")
    src.write_text(SRC)
    subprocess.run(["g++", "-std=c++17", "-I", _build.CSRC, "-I", _build.INCLUDE,
                    "-I", os.path.join(_build.CUDA_HOME, "include"), str(src), "-o", exe], check=True)
    assert subprocess.run([exe]).returncode == 0


@pytest.mark.parametrize("dims,most", [
    ((64, 48, 12, 60), 1627692), ((320, 240, 85, 1000), 256094760), ((1280, 720, 30, 3000), 1082657444),
    ((32, 32, 32, 32767), 47339508), ((40, 40, 21, 32767), 46386124), ((16, 16, 8, 2000), 2875352),
    ((13, 11, 2, 200), 494104), ((7, 5, 3, 100), 314292), ((2, 2, 2, 8), 224352),
])
def test_bytes_of_a_clip(asv, dims, most):
    assert asv.load().asv_clip_bytes(*dims) <= most


@pytest.mark.gpu
@pytest.mark.parametrize("dims,most", [((32, 32, 32, 32767), 47339508), ((2, 2, 2, 8), 224352)])
def test_a_budget_of_those_bytes_admits_the_clip(asv, dims, most):
    W, H, D, K = dims
    rgb, fwd, bwd = asv.synth_clip(W, H, D, seed=3)
    with asv.Image(lloyd_iters=1, hbm_budget=most) as img:
        assert img.segment(rgb, fwd, bwd, K).shape == (D, H, W)

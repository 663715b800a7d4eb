"""Tiles along an axis of any length that the connectivity and the evaluation take:
volumes of fewer than 2^31 voxels, so up to 2^31 - 1 along one axis."""
import os
import re
import subprocess

SRC = r"""
#include "asv_common.cuh"
#include <climits>
int main()
{
    for (int size : { 8, 32, 64 })
        for (long long n : { 1LL, 7LL, 8LL, 9LL, 63LL, 64LL, 65LL, (long long)INT_MAX - 64, (long long)INT_MAX - 31,
                             (long long)INT_MAX - 1, (long long)INT_MAX }) {
            const long long tiles = asv_tiles_along((int)n, size);
            if (tiles != (n + size - 1) / size) return 1;
            if (tiles * size - 1 > INT_MAX) return 2;                  // coordinates of the last tile's lanes
        }
    return 0;
}
"""


def test_tiles_along_any_axis(tmp_path):
    from anisotropic_supervoxel_gb300 import _build
    src, exe = tmp_path / "tiles.cpp", str(tmp_path / "tiles")
    src.write_text(SRC)
    subprocess.run(["g++", "-std=c++17", "-fsanitize=undefined", "-fno-sanitize-recover=undefined", "-I", _build.CSRC,
                    "-I", _build.INCLUDE, "-I", os.path.join(_build.CUDA_HOME, "include"), str(src), "-o", exe], check=True)
    assert subprocess.run([exe]).returncode == 0


def test_launches_count_their_tiles_so():
    """No int sum of an extent and a tile's size in the launches' tile counts."""
    from anisotropic_supervoxel_gb300 import _build
    for f in ("asv_connect.cu", "asv_eval.cu"):
        src = open(os.path.join(_build.CSRC, f)).read()
        assert "asv_tiles_along" in src
        assert not re.search(r"\(\s*[WHD]\s*\+[^()]*-?[^()]*\)\s*/", src)

"""Grid sizes and indexes over all seed slots of a context, at the largest batch
that asv_batch_init takes."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SRC = r"""
#include "asv_common.cuh"
#include <cstdio>
int main()
{
    const long long most = (long long)ASV_MAX_CLIPS * asv_seed_slots(32767);
    for (long long n : { 1LL, 9LL, 11184811LL, 79536432LL, most }) {
        if (asv_first_blocks((int)n) != (27 * n + 255) / 256) return 1;
        if (256LL * asv_first_blocks((int)n) >= 1LL << 32) return 2;      // a thread's index, 32 bits
        if (asv_ring_tasks((int)n) != ASV_RING * n) return 3;
        if (ASV_RING * n + 2 * 8 * 1216 >= 1LL << 32) return 4;           // the last stride of the ring's tasks
        for (int t = 0; t < ASV_RING; t++)
            if (8 * asv_ring_at((int)n - 1, t) != 8 * (unsigned long long)(ASV_RING * (n - 1) + t)) return 5;
    }
    return most > 1 << 27 ? 0 : 6;
}
"""


def test_indexes_of_the_largest_batch(tmp_path):
    from anisotropic_supervoxel_gb300 import _build
    src, exe = tmp_path / "seeds.cpp", str(tmp_path / "seeds")
    src.write_text(SRC)
    subprocess.run(["g++", "-std=c++17", "-fsanitize=undefined", "-fno-sanitize-recover=undefined", "-I", _build.CSRC,
                    "-I", _build.INCLUDE, "-I", os.path.join(_build.CUDA_HOME, "include"), str(src), "-o", exe], check=True)
    assert subprocess.run([exe]).returncode == 0

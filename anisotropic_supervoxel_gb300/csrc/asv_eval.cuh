// asv_eval.cuh -- supervoxel quality measures on the device (asv_eval.cu).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#define EV_MAX_LABELS 32768     // supervoxel labels -1 .. 32767
#define EV_MAX_TRUTH 4096       // truth ids 0 .. 4095

// meta[0] = largest label, meta[1] = largest truth id, meta[2] = 1 when a
// value is out of range.  All asynchronous on st.
int asv_launch_eval_range_init(int *meta, cudaStream_t st);
int asv_launch_eval_range(const int32_t *lab, const int32_t *gt, long long n, int *meta, cudaStream_t st);

// supervoxel boundary flags of the labels, a bit per voxel
size_t asv_eval_sbound_words(int W, int H, int D);
int asv_launch_eval_sbound(const int32_t *lab, int W, int H, int D, unsigned *sb, cudaStream_t st);

// counts for rows = largest label + 2 (row 0 = label -1) and NG truth ids:
// cnt[rows][NG], zmin/zmax[rows], tot[2] = truth boundary voxels, recalled ones
int asv_launch_eval(const int32_t *lab, const int32_t *gt, int W, int H, int D, int rows, int NG, unsigned *cnt,
                    int *zmin, int *zmax, const unsigned *sb, unsigned long long *tot, cudaStream_t st);

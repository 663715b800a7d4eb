// asv_common.cuh -- device-side layout shared by the kernels and the host
// orchestration of libasv.
//
// A context holds one or more segments (a clip, a streaming window, or the
// clips of a batch).  All volumes of all segments live in single packed
// device arrays; a segment's voxels start at `vox_off` (a multiple of
// ASV_CHUNK) and its seeds at `seed_off`.  Every kernel covers all segments
// in one launch and finds its segment from a prefix table.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#define ASV_MAXP 32          // max JFA passes per Lloyd iteration
#define ASV_CHUNK 2048       // voxels per block in the per-voxel kernels
#define ASV_TILE_X 16        // JFA tile: 16 x 16 columns x SegDesc::zrun chain positions
#define ASV_TILE_Y 16        // (a warp covers 16 x 2 columns: fewer distinct candidates)
#define ASV_BITS_MAXS 6      // largest step of a JFA pass's bit-set form (larger ones: list form)
#define ASV_RING 24          // 8 one-ring + 16 two-ring neighbours of the metric fallback
#define ASV_POST_WORDS 16    // per-segment post-processing record

struct SegDesc {
    int W, H, D, Kp;
    long long vox_off;       // first voxel of the segment in the packed arrays
    long long nvox;          // W*H*D
    int seed_off;            // first seed slot (Kp+1 slots used: slot Kp = label -1)
    int npass;
    int steps[ASV_MAXP];
    float ratio[ASV_MAXP];   // ratio of each pass (base ratio x 1 or x 2)
    int depth[ASV_MAXP];     // chain positions per sub-tile of each pass's bit-set form, 0: list form
    int tiles_x, tiles_y;
    unsigned inv_tiles_x, inv_tiles_y;   // ceil(2^32 / tiles), 0 for one tile (asv_quotient)
    int zrun;                // JFA tile depth: chain positions per column and tile
    int angle_filter;        // plain reseed flow-angle filter
    int wNum, hNum, dNum;    // seed grid (density placement)
    int cell_off;            // x cells at cell_off, y at +W, z at +W+H
    int final_buf;           // 0: last pass wrote buffer A, 1: buffer B
    long long lab_from;      // first voxel whose LAB must be computed (streaming windows keep
                             // the LAB of their overlap frames)
};

// post-processing record per segment (ints), written by k_post_stats
enum {
    POST_DEAD = 0, POST_NEG = 1, POST_VALID = 2, POST_MODE = 3, POST_INVALID = 4,
    POST_L0 = 5, POST_M0 = 6, POST_DEAD0 = 7 /* .. +3: first dead ids */
};

#ifdef __CUDACC__
#define ASV_HD __host__ __device__ __forceinline__
#else
#define ASV_HD inline
#endif

// tiles of `size` along n >= 1 voxels, for any int n
ASV_HD int asv_tiles_along(int n, int size) { return (n - 1) / size + 1; }

// A batch has up to ASV_MAX_CLIPS clips of up to 32767 seeds, each in a run of
// slots rounded up, 134 million in all: 27 or ASV_RING of something per seed
// pass 2^31 and stay below 2^32, bytes and words of them pass that too.
#define ASV_MAX_CLIPS 4096
ASV_HD int asv_seed_slots(int Kp) { return ((Kp + 64 + 31) / 32) * 32; }

// blocks of 256 for a thread per seed slot and voxel around it; solves of the rings
ASV_HD unsigned asv_first_blocks(int slots) { return (27u * (unsigned)slots + 255u) / 256u; }
ASV_HD unsigned asv_ring_tasks(int slots) { return (unsigned)ASV_RING * (unsigned)slots; }

// an entry of AsvDev::tlist: a voxel of a clip (fewer than 2^31) and its label
// (below 32768), in 58 bits
typedef unsigned long long asv_entry_t;
ASV_HD asv_entry_t asv_entry(int seg, int voxel, int label)
{
    return ((asv_entry_t)(unsigned)seg << 46) | ((asv_entry_t)(unsigned)voxel << 15) | (unsigned)label;
}
ASV_HD int asv_entry_seg(asv_entry_t e) { return (int)(e >> 46); }
ASV_HD int asv_entry_voxel(asv_entry_t e) { return (int)((unsigned)(e >> 15) & 0x7fffffffu); }
ASV_HD int asv_entry_label(asv_entry_t e) { return (int)((unsigned)e & 0x7fffu); }

// place of ring neighbour t of seed slot g (of Mring's rows of 8 floats, of ringok)
ASV_HD size_t asv_ring_at(int g, int t) { return (size_t)ASV_RING * g + t; }

#ifdef __CUDACC__
// n / d for n < 2^24, d <= 256, from inv = ceil(2^32 / d) (0 for d = 1): inv * d
// exceeds 2^32 by less than d, so the product's error stays below 1 / d.
__device__ __forceinline__ int asv_quotient(int n, unsigned inv)
{
    return inv ? (int)__umulhi((unsigned)n, inv) : n;
}

// Binary search: largest i in [0, n) with prefix[i] <= v.
__device__ __forceinline__ int asv_find_seg(const int *__restrict__ prefix, int n, int v)
{
    int lo = 0, hi = n - 1;
    while (lo < hi) {
        int mid = (lo + hi + 1) >> 1;
        if (__ldg(prefix + mid) <= v) lo = mid; else hi = mid - 1;
    }
    return lo;
}

__device__ __forceinline__ long long asv_find_seg64(const long long *__restrict__ prefix, int n,
                                                    long long v)
{
    int lo = 0, hi = n - 1;
    while (lo < hi) {
        int mid = (lo + hi + 1) >> 1;
        if (__ldg(prefix + mid) <= v) lo = mid; else hi = mid - 1;
    }
    return lo;
}
#endif

// Host-side launch wrappers (defined in the .cu files, called by asv_api.cpp).
struct AsvDev {
    int nseg;
    const SegDesc *segs;         // device copy
    const int *tile_prefix;      // [nseg+1] JFA tiles
    const int *chunk_prefix;     // [nseg+1] ASV_CHUNK-voxel chunks
    const int *seed_prefix;      // [nseg+1] seed slots (seed_off)
    int total_tiles, total_chunks, total_seeds;
    uint8_t *rgb;                // 3 bytes / voxel
    uchar4 *lab;                 // L, a, b, 0
    float2 *fwd, *bwd;
    int32_t *labA, *labB;
    int32_t *drawn;              // the drawn seeds at their voxels, else -1 (loop: all -1 between its draws; else labA)
    asv_entry_t *tlist;          // voxels labelled by the first pass, 27 per seed
    unsigned *tcount;            // entries of tlist
    float4 *pos0;                // initial seeds (density placement)
    float *M0;                   // initial metric, 8 floats / seed
    float4 *pos, *slab;          // working seeds
    float *M;                    // working metric, 8 floats / seed
    float4 *jtab;                // JFA seed table, 3 float4 / seed
    unsigned long long *sums;    // 8 u64 / slot
    float *Mself; int *neg;      // metric scratch
    float *Mmemo; int *mkey;     // reseed memo: metric of the voxel key of the last solve
    float *Mring; int *ringok;
    int *neglist, *negcount;     // seeds whose own metric is not PSD (empty between solves; the list in rank's place)
    float4 *grid;                // grid seeds
    unsigned long long *dacc;    // density accumulators (2^-24 units)
    int *cells;                  // cell tables
    int *post;                   // ASV_POST_WORDS / segment
    int *rank;                   // per seed: relabel LUT / alive rank
    int *scan;                   // per chunk
    float *srgb;                 // 256-entry sRGB linearisation
    const uchar4 *lablut;        // LAB of every RGB value (per device, shared), or null
    int *err;                    // device error word
};

void asv_launch_srgb_table(const AsvDev &d, cudaStream_t st);
void asv_launch_rgb2lab(const AsvDev &d, cudaStream_t st);
void asv_launch_preprocess(const uint8_t *bgr, uint8_t *rgb, int W, int H, int D, cudaStream_t st);
const uchar4 *asv_lab_table(int device);
void asv_launch_density(const AsvDev &d, cudaStream_t st);
void asv_launch_density_adjust(const AsvDev &d, cudaStream_t st);
void asv_launch_first_init(const AsvDev &d, cudaStream_t st);
void asv_launch_draw(const AsvDev &d, cudaStream_t st);
// (follow: the operation before on st is a kernel, see asv_launch_follow)
void asv_launch_jfa(const AsvDev &d, int pass, int step, bool last, int grid_blocks, bool follow, cudaStream_t st);
void asv_launch_jfa_first(const AsvDev &d, bool filled, bool stale, cudaStream_t st);
void asv_launch_jfa_second_scatter(const AsvDev &d, bool undraw, cudaStream_t st);
// (seg, out: on the device)
void asv_launch_pass_prepare(int32_t *labels, const SegDesc &one, const SegDesc *seg, SegDesc *out, cudaStream_t st);
void asv_launch_centroids(const AsvDev &d, cudaStream_t st);
void asv_launch_finalize(const AsvDev &d, cudaStream_t st);
void asv_launch_post(const AsvDev &d, cudaStream_t st);
void asv_launch_metric(const AsvDev &d, int reseed, cudaStream_t st);
void asv_launch_next_seeds(const AsvDev &d, bool finalize, bool clear_sums, bool follow, cudaStream_t st);
int asv_jfa_grid_blocks(int total_tiles);
int asv_jfa_resident_blocks();
int asv_jfa_slots(int step);   // footprint slots a sub-tile of the step can hold, 0: no bit-set form

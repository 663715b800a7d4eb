// asv_eval.cu -- supervoxel quality measures against a ground-truth
// segmentation (the LIBSVX benchmark the reference is evaluated with,
// README.md:26-28: "3D undersegmentation error", "3D segmentation accuracy",
// "3D boundary recall", mean duration; Xu & Corso, "Evaluation of super-voxel
// methods for early video processing", CVPR 2012).  LIBSVX's own code is not
// available here; the definitions implemented are stated in asv.h.
//
// The device counts: the overlap matrix n[s][g] (supervoxel s, truth segment
// g), each supervoxel's first and last frame, the truth boundary voxels and
// how many of them have a supervoxel boundary within one voxel.  The host
// turns the counts into the measures.
#include "asv_eval.cuh"

#include "asv_common.cuh"
#include "asv_tally.cuh"

#define EV_T 256                    // = TALLY_SLOTS
#define EV_ROWS 8                   // rows of a warp in a tile of 32 x 64 voxels of a frame

#define EV_RANGE_PER_THREAD 8
#define EV_FLAT_PER 8               // voxels per thread of the flat form
#define EV_SPARSE 384               // voxels per tile up to which the flat form is taken

// label ranges and bounds violations: a block reduces EV_T * 8 voxels (warp
// reductions, then the block's warps through shared memory) and issues one
// atomic per quantity, so the three global words see few updates
__global__ void k_ev_range(const int32_t *__restrict__ lab, const int32_t *__restrict__ gt, long long n, int *meta)
{
    __shared__ int red[3][EV_T / 32];
    const long long base = (long long)blockIdx.x * blockDim.x * EV_RANGE_PER_THREAD + threadIdx.x;
    int ls = -1, lg = -1, bad = 0;
#pragma unroll
    for (int k = 0; k < EV_RANGE_PER_THREAD; k++) {
        const long long v = base + (long long)k * blockDim.x;
        if (v < n) {
            const int a = lab[v], b = gt[v];
            ls = max(ls, a);
            lg = max(lg, b);
            bad |= (a < -1 || a >= EV_MAX_LABELS || b < 0 || b >= EV_MAX_TRUTH) ? 1 : 0;
        }
    }
    ls = __reduce_max_sync(0xffffffffu, ls);
    lg = __reduce_max_sync(0xffffffffu, lg);
    bad = __reduce_or_sync(0xffffffffu, bad);
    const int w = threadIdx.x >> 5;
    if ((threadIdx.x & 31) == 0) {
        red[0][w] = ls;
        red[1][w] = lg;
        red[2][w] = bad;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int i = 1; i < EV_T / 32; i++) {
            ls = max(ls, red[0][i]);
            lg = max(lg, red[1][i]);
            bad |= red[2][i];
        }
        atomicMax(meta + 0, ls);
        atomicMax(meta + 1, lg);
        if (bad) atomicOr(meta + 2, 1);
    }
}

// A warp's 32 voxels of a row and the rows after: the voxel's own value, and
// whether it differs from a neighbour along x, y or z
struct EvRows {
    const int32_t *p;
    int W, fr, lane;
    bool in, first, last, zm, zp;
    int cur, up;

    __device__ __forceinline__ EvRows(const int32_t *a, int W_, int H, int D, int x, int y, int z)
    {
        W = W_; fr = W * H;
        lane = threadIdx.x & 31;
        in = x < W; first = x == 0; last = x == W - 1;
        zm = in && z > 0; zp = in && z < D - 1;
        p = a + (size_t)z * fr + (size_t)y * W + x;
        cur = in ? __ldg(p) : 0;
        up = in && y > 0 ? __ldg(p - W) : cur;
    }
    __device__ __forceinline__ bool step(bool more, int *value)
    {
        const int c = cur;
        const int dn = in && more ? __ldg(p + W) : c;
        const int b = zm ? __ldg(p - fr) : c, f = zp ? __ldg(p + fr) : c;
        int l = __shfl_up_sync(0xffffffffu, c, 1), r = __shfl_down_sync(0xffffffffu, c, 1);
        if (lane == 0) l = in && !first ? __ldg(p - 1) : c;
        if (lane == 31) r = in && !last ? __ldg(p + 1) : c;
        if (last) r = c;
        const bool diff = in && (dn != c || up != c || b != c || f != c || l != c || r != c);
        *value = c;
        up = c;
        cur = dn;
        p += W;
        return diff;
    }
};

// Supervoxel boundary flags, a bit per voxel (a voxel with a 6-neighbour of
// another label); a word is 32 voxels of a row
__global__ void __launch_bounds__(EV_T) k_ev_sbound(const int32_t *__restrict__ lab, int W, int H, int D, int tx, int ty,
                                                    unsigned *__restrict__ sb)
{
    const int xt = blockIdx.x % tx, q = blockIdx.x / tx, z = q / ty;
    const int y0 = ((q - z * ty) * (EV_T / 32) + (threadIdx.x >> 5)) * EV_ROWS;
    if (y0 >= H) return;
    EvRows row(lab, W, H, D, xt * 32 + (threadIdx.x & 31), y0, z);
#pragma unroll
    for (int k = 0; k < EV_ROWS; k++) {
        if (y0 + k >= H) break;
        int l;
        const unsigned m = __ballot_sync(0xffffffffu, row.step(y0 + k < H - 1, &l));
        if (row.lane == 0) sb[((size_t)z * H + y0 + k) * tx + xt] = m;
    }
}

// Flags of 32 voxels of one row after the other, those of their neighbours along x
// and z included: lanes 0 to 2 each go down one slice's words
struct EvFlags {
    const unsigned *p;
    int tx;
    bool mine, left, right;

    __device__ __forceinline__ EvFlags(const unsigned *sb, int tx_, int H, int D, int xt, int y, int z)
    {
        const int zz = z + (int)(threadIdx.x & 31) - 1;
        tx = tx_;
        mine = (threadIdx.x & 31) < 3 && zz >= 0 && zz < D;
        left = mine && xt > 0;
        right = mine && xt < tx - 1;
        p = sb + ((long long)zz * H + y) * tx + xt;
    }
    __device__ __forceinline__ unsigned step(bool there)       // the next row (outside the volume: none)
    {
        const unsigned w = mine && there ? __ldg(p) : 0u, a = left && there ? __ldg(p - 1) : 0u;
        const unsigned c = right && there ? __ldg(p + 1) : 0u;
        p += tx;
        return __reduce_or_sync(0xffffffffu, w | __funnelshift_l(a, w, 1) | __funnelshift_r(w, c, 1));
    }
};

// frames z0 to z1 of a supervoxel: the range goes out where it widens the one read
__device__ __forceinline__ void ev_frames(int s, int z0, int z1, int *zmin, int *zmax)
{
    if (z0 < __ldcg(zmin + s)) atomicMin(zmin + s, z0);
    if (z1 > __ldcg(zmax + s)) atomicMax(zmax + s, z1);
}

// hands out c voxels of (supervoxel, truth) key in frame z
__device__ __forceinline__ void ev_out(int key, unsigned c, int z, int NG, unsigned *cnt, int *zmin, int *zmax)
{
    const int s = key / NG;
    atomicAdd(cnt + key, c);
    if (s > 0) ev_frames(s, z, z, zmin, zmax);               // row 0 is label -1
}

// Overlap counts (label -1 is row 0) and per-supervoxel frame range; truth
// boundary voxels, and those with a supervoxel boundary voxel in their 3x3x3
// neighbourhood.  A block counts the (supervoxel, truth) pairs of its tile of one
// frame in shared memory, a run of a row at a time, and keeps the rows' values
// and flags while it goes down them.  (Equal lanes of a warp grouped into three
// global updates, and nine rows of a byte volume per boundary voxel: 135 + 100 us
// on a 320x240x85 volume, now 71 us.)
__global__ void __launch_bounds__(EV_T) k_ev_counts(const int32_t *__restrict__ lab, const int32_t *__restrict__ gt,
                                                    int W, int H, int D, int tx, int ty, int NG,
                                                    unsigned *__restrict__ cnt, int *__restrict__ zmin,
                                                    int *__restrict__ zmax, const unsigned *__restrict__ sb,
                                                    unsigned long long *__restrict__ tot)
{
    __shared__ Tally t;
    __shared__ unsigned red[2][EV_T / 32];
    tally_clear(t);
    __syncthreads();
    const int xt = blockIdx.x % tx, q = blockIdx.x / tx, z = q / ty, w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int y0 = ((q - z * ty) * (EV_T / 32) + w) * EV_ROWS, x = xt * 32 + lane;
    unsigned isb = 0, rec = 0;
    if (y0 < H) {
        EvRows row(gt, W, H, D, x, y0, z);
        const int32_t *pl = lab + (size_t)z * W * H + (size_t)y0 * W + x;
        EvFlags flags(sb, tx, H, D, xt, y0 - 1, z);
        unsigned above = flags.step(y0 > 0), here = flags.step(true);
#pragma unroll
        for (int k = 0; k < EV_ROWS; k++) {
            if (y0 + k >= H) break;
            const int s = row.in ? __ldg(pl + (size_t)k * W) + 1 : 0;
            const unsigned below = flags.step(y0 + k + 1 < H);
            int g;
            const bool b = row.step(y0 + k < H - 1, &g);
            const int key = row.in ? s * NG + g : -1;
            const int before = __shfl_up_sync(0xffffffffu, key, 1);
            const unsigned starts = __ballot_sync(0xffffffffu, lane == 0 || key != before);
            if (row.in && ((starts >> lane) & 1u)) {
                const unsigned next = lane < 31 ? starts & (0xfffffffeu << lane) : 0u;
                const unsigned c = (unsigned)((next ? __ffs(next) - 1 : 32) - lane);
                if (!tally_add(t, key, c)) ev_out(key, c, z, NG, cnt, zmin, zmax);
            }
            if (b) {
                isb++;
                rec += ((above | here | below) >> lane) & 1u;
            }
            above = here;
            here = below;
        }
    }
    isb = __reduce_add_sync(0xffffffffu, isb);
    rec = __reduce_add_sync(0xffffffffu, rec);
    if (lane == 0) {
        red[0][w] = isb;
        red[1][w] = rec;
    }
    __syncthreads();
    if (t.key[threadIdx.x] >= 0) ev_out(t.key[threadIdx.x], t.cnt[threadIdx.x], z, NG, cnt, zmin, zmax);
    if (threadIdx.x == 0) {                                  // one pair of atomics per block
        for (int i = 1; i < EV_T / 32; i++) {
            isb += red[0][i];
            rec += red[1][i];
        }
        if (isb) {
            atomicAdd(tot + 0, (unsigned long long)isb);
            atomicAdd(tot + 1, (unsigned long long)rec);
        }
    }
}

// The same two steps for volumes that would leave most of a tile empty (ev_flat):
// voxels in the order of memory, the flags' words too.
struct EvAt {
    int x, y, z;
    __device__ __forceinline__ EvAt(int v, int W, int H)
    {
        const int row = v / W;
        x = v - row * W;
        z = row / H;
        y = row - z * H;
    }
};

__device__ __forceinline__ bool ev_differs(const int32_t *__restrict__ a, int v, const EvAt &at, int W, int H, int D)
{
    const int l = __ldg(a + v), fr = W * H;
    return (at.x > 0 && __ldg(a + v - 1) != l) || (at.x < W - 1 && __ldg(a + v + 1) != l) ||
           (at.y > 0 && __ldg(a + v - W) != l) || (at.y < H - 1 && __ldg(a + v + W) != l) ||
           (at.z > 0 && __ldg(a + v - fr) != l) || (at.z < D - 1 && __ldg(a + v + fr) != l);
}

__global__ void __launch_bounds__(EV_T) k_ev_sbound_flat(const int32_t *__restrict__ lab, int W, int H, int D, int n,
                                                         unsigned *__restrict__ sb)
{
    const unsigned v = blockIdx.x * EV_T + threadIdx.x;
    const bool in = v < (unsigned)n;
    const unsigned m = __ballot_sync(0xffffffffu, in && ev_differs(lab, (int)v, EvAt((int)v, W, H), W, H, D));
    if (in && (threadIdx.x & 31) == 0) sb[v >> 5] = m;
}

__global__ void __launch_bounds__(EV_T) k_ev_counts_flat(const int32_t *__restrict__ lab, const int32_t *__restrict__ gt,
                                                         int W, int H, int D, int n, int NG, unsigned *__restrict__ cnt,
                                                         int *__restrict__ zmin, int *__restrict__ zmax,
                                                         const unsigned *__restrict__ sb,
                                                         unsigned long long *__restrict__ tot)
{
    __shared__ Tally t;
    __shared__ unsigned red[2];
    tally_clear(t);
    if (threadIdx.x < 2) red[threadIdx.x] = 0u;
    __syncthreads();
    const int lane = threadIdx.x & 31, fr = W * H;
    unsigned isb = 0, rec = 0;
    for (int k = 0; k < EV_FLAT_PER; k++) {
        const unsigned v = (blockIdx.x * EV_FLAT_PER + k) * EV_T + threadIdx.x;
        const bool in = v < (unsigned)n;
        const EvAt at(in ? (int)v : 0, W, H);
        const int s = in ? __ldg(lab + v) + 1 : 0, key = in ? s * NG + __ldg(gt + v) : -1;
        const int before = __shfl_up_sync(0xffffffffu, key, 1);
        const unsigned starts = __ballot_sync(0xffffffffu, lane == 0 || key != before);
        const unsigned next = lane < 31 ? starts & (0xfffffffeu << lane) : 0u;
        const int end = next ? __ffs(next) - 1 : 32;           // of the run that starts here
        const int z1 = __shfl_sync(0xffffffffu, at.z, end - 1);
        if (in && ((starts >> lane) & 1u)) {
            if (!tally_add(t, key, (unsigned)(end - lane))) atomicAdd(cnt + key, (unsigned)(end - lane));
            if (s > 0) ev_frames(s, at.z, z1, zmin, zmax);
        }
        if (in && ev_differs(gt, (int)v, at, W, H, D)) {
            isb++;
            bool near = false;
            for (int dz = at.z > 0 ? -1 : 0; dz <= (at.z < D - 1 ? 1 : 0) && !near; dz++)
                for (int dy = at.y > 0 ? -1 : 0; dy <= (at.y < H - 1 ? 1 : 0) && !near; dy++)
                    for (int dx = at.x > 0 ? -1 : 0; dx <= (at.x < W - 1 ? 1 : 0); dx++) {
                        const int u = (int)v + dz * fr + dy * W + dx;
                        near = near || ((__ldg(sb + (u >> 5)) >> (u & 31)) & 1u);
                    }
            rec += near;
        }
    }
    isb = __reduce_add_sync(0xffffffffu, isb);
    rec = __reduce_add_sync(0xffffffffu, rec);
    if (lane == 0) {
        atomicAdd(&red[0], isb);
        atomicAdd(&red[1], rec);
    }
    __syncthreads();
    if (t.key[threadIdx.x] >= 0) atomicAdd(cnt + t.key[threadIdx.x], t.cnt[threadIdx.x]);
    if (threadIdx.x < 2 && red[0]) atomicAdd(tot + threadIdx.x, (unsigned long long)red[threadIdx.x]);
}

static int ev_tx(int W) { return asv_tiles_along(W, 32); }
static int ev_ty(int H) { return asv_tiles_along(H, EV_T / 32 * EV_ROWS); }

// Whether the volume goes without tiles.  At 384 voxels per tile of 2048 and fewer
// the flat form is the faster one: 1024x1024x6 (x the last) 672 us a call, tiles
// 736; 1024 x 8 rows x 1024 858, 1024; lines along z 0.20 ms, 6.0; at 512, 1024x1024x8
// with noisy labels, 1016 against 844.
static bool ev_flat(int W, int H, int D)
{
    return (long long)W * H * D <= (long long)EV_SPARSE * ev_tx(W) * ev_ty(H) * D;
}

size_t asv_eval_sbound_words(int W, int H, int D)
{
    return ev_flat(W, H, D) ? (size_t)(((long long)W * H * D + 31) / 32) : (size_t)ev_tx(W) * H * D;
}

int asv_launch_eval_range_init(int *meta, cudaStream_t st)
{
    cudaMemsetAsync(meta, 0xff, 2 * sizeof(int), st);       // -1
    return cudaMemsetAsync(meta + 2, 0, sizeof(int), st) == cudaSuccess ? 0 : -1;
}

int asv_launch_eval_range(const int32_t *lab, const int32_t *gt, long long n, int *meta, cudaStream_t st)
{
    k_ev_range<<<(unsigned)((n + EV_T * EV_RANGE_PER_THREAD - 1) / (EV_T * EV_RANGE_PER_THREAD)), EV_T, 0, st>>>(
        lab, gt, n, meta);
    return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

int asv_launch_eval_sbound(const int32_t *lab, int W, int H, int D, unsigned *sb, cudaStream_t st)
{
    const int tx = ev_tx(W), ty = ev_ty(H);
    const long long n = (long long)W * H * D;
    if (ev_flat(W, H, D)) k_ev_sbound_flat<<<(unsigned)((n + EV_T - 1) / EV_T), EV_T, 0, st>>>(lab, W, H, D, (int)n, sb);
    else k_ev_sbound<<<(unsigned)tx * ty * D, EV_T, 0, st>>>(lab, W, H, D, tx, ty, sb);
    return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

int asv_launch_eval(const int32_t *lab, const int32_t *gt, int W, int H, int D, int rows, int NG, unsigned *cnt,
                    int *zmin, int *zmax, const unsigned *sb, unsigned long long *tot, cudaStream_t st)
{
    const int tx = ev_tx(W), ty = ev_ty(H);
    cudaMemsetAsync(cnt, 0, sizeof(unsigned) * (size_t)rows * NG, st);
    cudaMemsetAsync(zmin, 0x7f, sizeof(int) * (size_t)rows, st);      // large
    cudaMemsetAsync(zmax, 0xff, sizeof(int) * (size_t)rows, st);      // -1
    cudaMemsetAsync(tot, 0, 2 * sizeof(unsigned long long), st);
    const long long n = (long long)W * H * D, per = EV_T * EV_FLAT_PER;
    if (ev_flat(W, H, D))
        k_ev_counts_flat<<<(unsigned)((n + per - 1) / per), EV_T, 0, st>>>(lab, gt, W, H, D, (int)n, NG, cnt, zmin, zmax, sb,
                                                                         tot);
    else k_ev_counts<<<(unsigned)tx * ty * D, EV_T, 0, st>>>(lab, gt, W, H, D, tx, ty, NG, cnt, zmin, zmax, sb, tot);
    return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

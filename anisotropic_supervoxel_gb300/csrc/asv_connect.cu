// asv_connect.cu -- 3D connectivity enforcement on the device.
//
// Replaces Image::EnforceLabelConnectivity3D (GPU-AS/Image.cpp:1938-2063,
// called by enforce_connectivity_3d :1808-1837) and Render::label_connected3D
// (streamGPU-AS/Render.cpp:572-695), a sequential raster scan with a flood
// fill per segment.  What the scan computes, restated for a parallel build:
//
//  * segments are the connected components of equal input label under the
//    24-neighbourhood (slices z-1, z, z+1 x the 8 in-plane offsets; the
//    voxel straight above or below is not a neighbour);
//  * segments are numbered in the raster order of their first voxel (the
//    scan's seed), which is the component's smallest voxel index;
//  * a segment of fewer than supsz / 4 voxels takes the label `adj` read at
//    its seed: the label, at that moment, of the last neighbour of the seed
//    (in the reference's loop order) that belongs to an earlier segment; if
//    none does, `adj` keeps the value of the previous segment's scan (0 at
//    the start).  Other segments get consecutive labels.
//
// Build: union-find over voxels (the smaller root always wins, so the root of
// a component is its smallest index = the scan's seed), root compaction by a
// chunked prefix scan, per-root `adj` from the seed's neighbours, and the
// labels of merged segments resolved by pointer jumping over two node kinds:
// F_j (the label of segment j) and A_j (the scan's `adj` after segment j).
// Everything is enqueued at once: the kernels that work on the segments read
// their number from device memory.
//
// Linking follows long serial chains, so most of it is done in shared memory: a
// block first joins its tile of 32 x 8 x 8 voxels by itself, then only the links
// that cross tiles are made in global memory, between sets of known size.  Of its
// 12 earlier neighbours a voxel links only those that the links of others don't
// imply (cc_links), all kinds in one loop, so that the lanes' walks run side by
// side.  Volumes whose tiles would be nearly empty are linked voxel by voxel in
// global memory.  On the 320x240x85 clip's labels: 12 links per voxel, one after the
// other, 543 us; a root walk and an atomic per voxel 113 us, segments numbered by
// few blocks 91 us, 18 jumping rounds 60 us; now 95 us in the tiles
// and 58 between them, 28, 12 and 17 us.
// Integer work only: compiled without -fmad=false.
#include "asv_connect.cuh"

#include "asv_common.cuh"
#include "asv_follow.cuh"

#define CC_CHUNK 2048
#define CC_THREADS 256
#define CC_TZ 8                     // a tile: 32 x 8 (the block's warps) x CC_TZ voxels
#define CC_TILE (CC_THREADS * CC_TZ)
#define CC_SPARSE 64                // voxels per tile up to which the volume goes without tiles
#define CC_SEGS 128                 // segments per group of the rank scan
#define CC_HOPS 256
#define CC_SHOW 4
#define CC_ROUNDS 4
#define CC_MAX_R (1 << 30)
#define CC_SPIN_LIMIT (1 << 24)     // step bound of a union / walk; exceeding it flags an error

__constant__ int c_dx8[8] = { -1, -1, 0, 1, 1, 1, 0, -1 };
__constant__ int c_dy8[8] = { 0, -1, -1, -1, 0, 1, 1, 1 };

// Joins the sets of a and b.  Both walk up together, the one with the larger
// parent first, and its link is moved to the other's smaller parent on the way
// (Rem's algorithm, with compare-and-swap as in Patwary, Refsnes and Manne,
// "Multi-core spanning forest algorithms using the disjoint-set data
// structure", 2012).  A parent is never larger than its voxel and only gets
// smaller, so the root of a component is its smallest voxel in the end.  A link
// that is moved leaves its old parent to be joined by this call's next steps;
// a failed swap means that another call made the parent smaller.
__device__ __forceinline__ void cc_union(int *par, int a, int b, int *err)
{
    for (int it = 0; it < CC_SPIN_LIMIT; it++) {
        int pa = __ldcg(par + a), pb = __ldcg(par + b);
        if (pa == pb) return;
        if (pa < pb) {
            const int t = a, tp = pa;
            a = b; pa = pb;
            b = t; pb = tp;
        }
        const int old = atomicCAS(par + a, pa, pb);
        if (pa == a) {
            if (old == a) return;
        } else a = pa;
    }
    atomicOr(err, 1);
}

// the same in shared memory
__device__ __forceinline__ void cc_union_tile(volatile int *par, int a, int b, int *err)
{
    for (int it = 0; it < CC_SPIN_LIMIT; it++) {
        int pa = par[a], pb = par[b];
        if (pa == pb) return;
        if (pa < pb) {
            const int t = a, tp = pa;
            a = b; pa = pb;
            b = t; pb = tp;
        }
        const int old = atomicCAS((int *)par + a, pa, pb);
        if (pa == a) {
            if (old == a) return;
        } else a = pa;
    }
    atomicOr(err, 1);
}

// Links of a voxel to its earlier neighbours of equal label: N, NW, NE, W in its
// slice and the eight around (x, y) in the slice before (N', NE', ...).  Left out
// are the links that others imply:
//  * neighbours that are neighbours of each other are linked already, so N
//    stands for NW and NE, W for NW, E for NE; N' for NW', NE', W', E'; S' for
//    SW', SE', W', E'; W' and E' for their corners;
//  * where W has the voxel's label and its N (its N', S') has it too, W links
//    the pair of rows, or a voxel further left does.
// As bits: (dy + 1) * 3 + dx + 1, nine further for the slice before.  h*: the
// neighbour exists (west, east, north, south, previous slice); at(dx, dy, dz):
// its label.
template <class F>
__device__ __forceinline__ unsigned cc_links(int l, bool hw, bool he, bool hn, bool hs, bool hp, F at)
{
    const bool w = hw && at(-1, 0, 0) == l, nn = hn && at(0, -1, 0) == l, nw = hw && hn && at(-1, -1, 0) == l;
    unsigned m = w ? 1u << 3 : 0u;
    if (nn) {
        if (!(w && nw)) m |= 1u << 1;
    } else if (hn) {
        if (nw && !w) m |= 1u << 0;
        if (he && at(1, -1, 0) == l && at(1, 0, 0) != l) m |= 1u << 2;
    }
    if (!hp) return m;
    const bool pn = hn && at(0, -1, -1) == l, pnw = hw && hn && at(-1, -1, -1) == l;
    const bool ps = hs && at(0, 1, -1) == l, psw = hw && hs && at(-1, 1, -1) == l;
    if (pn && !(w && pnw)) m |= 1u << 10;
    if (ps && !(w && psw)) m |= 1u << 16;
    if (pn && ps) return m;
    const bool pw = hw && at(-1, 0, -1) == l, pe = he && at(1, 0, -1) == l;
    if (!pn && !ps) m |= (pw ? 1u << 12 : 0u) | (pe ? 1u << 14 : 0u);
    if (!pn && !pw && pnw) m |= 1u << 9;
    if (!ps && !pw && psw) m |= 1u << 15;
    if (he && !pe) {
        if (!pn && hn && at(1, -1, -1) == l) m |= 1u << 11;
        if (!ps && hs && at(1, 1, -1) == l) m |= 1u << 17;
    }
    return m;
}

// A block's links, put down first and then made by all its threads: a few voxels
// in a warp have links, and each link is a chain of dependent accesses.  An entry:
// the voxel's place in the tile and its links' bits, so a tile's voxels have room.
// By whole warps, m = 0 without links.
__device__ __forceinline__ void cc_put(unsigned *queue, int *count, unsigned m, int i)
{
    const unsigned some = __ballot_sync(0xffffffffu, m != 0u);
    if (!some) return;
    const int lane = threadIdx.x & 31, lead = __ffs(some) - 1;
    int at = 0;
    if (lane == lead) at = atomicAdd(count, __popc(some));
    at = __shfl_sync(0xffffffffu, at, lead) + __popc(some & ((1u << lane) - 1u));
    if (m) queue[at] = ((unsigned)i << 18) | m;
}

template <class F>
__device__ __forceinline__ void cc_make(const unsigned *queue, int count, F fn)
{
    for (int j = threadIdx.x; j < count; j += CC_THREADS) {
        const unsigned e = queue[j];
        for (unsigned m = e & 0x3ffffu; m; m &= m - 1) fn((int)(e >> 18), __ffs(m) - 1);
    }
}

struct CcTile {
    int x, y, z, lane, w;                                      // this thread's first voxel, its place in the block
    __device__ __forceinline__ CcTile(int tx, int ty)
    {
        const int q = blockIdx.x / tx, zt = q / ty;
        lane = threadIdx.x & 31;
        w = threadIdx.x >> 5;
        x = (blockIdx.x - q * tx) * 32 + lane;
        y = (q - zt * ty) * (CC_THREADS / 32) + w;
        z = zt * CC_TZ;
    }
};

// The tile's own components: par = the component's smallest voxel, cnt = the
// component's size there, 0 elsewhere.  A row starts as its runs of equal label.
__global__ void __launch_bounds__(CC_THREADS) k_cc_tile(const int32_t *__restrict__ lab, int *par, int *cnt, int W,
                                                        int H, int D, int tx, int ty, int *err)
{
    asv_follow();
    __shared__ int sl[CC_TILE], sp[CC_TILE], sc[CC_TILE];      // sc: the queue, then the sizes
    __shared__ int nq;
    if (threadIdx.x == 0) nq = 0;
    const CcTile t(tx, ty);
    const bool in = t.x < W && t.y < H;
    const int g0 = (t.z * H + t.y - t.w) * W + t.x - t.lane;   // the tile's first voxel
    const int gv = (int)(((unsigned)t.z * H + t.y) * W + t.x), fr = W * H;   // (lanes outside wrap, and use it not)
    unsigned len[CC_TZ];                                       // of the run that starts here, else 0
#pragma unroll
    for (int k = 0; k < CC_TZ; k++) {
        const int i = k * CC_THREADS + threadIdx.x;
        const bool v = in && t.z + k < D;
        const int l = v ? lab[gv + k * fr] : 0, before = __shfl_up_sync(0xffffffffu, l, 1);
        const unsigned starts = __ballot_sync(0xffffffffu, t.lane == 0 || !v || l != before);
        const unsigned next = t.lane < 31 ? starts & (0xfffffffeu << t.lane) : 0u;
        len[k] = v && ((starts >> t.lane) & 1u) ? (next ? __ffs(next) - 1 : 32) - t.lane : 0u;
        sl[i] = l;
        sp[i] = i - t.lane + 31 - __clz((int)(starts & (0xffffffffu >> (31 - t.lane))));
    }
    __syncthreads();
    auto join = [&](int i, int b) {
        const int q = b % 9;
        cc_union_tile(sp, i - (b >= 9 ? CC_THREADS : 0) + (q / 3 - 1) * 32 + q % 3 - 1, i, err);
    };
    if (t.y < H) {
        // cc_links in the tile without its branches: nine labels a slice, of which
        // the next slice's voxel sees eight again
        const bool hw = in && t.lane > 0, he = t.lane < 31 && t.x < W - 1, hn = in && t.w > 0;
        const bool hs = in && t.w < CC_THREADS / 32 - 1 && t.y < H - 1;
        const int ow = hw ? -1 : 0, oe = he ? 1 : 0, on = hn ? -32 : 0, os = hs ? 32 : 0;   // missing: itself, not counted
        int pw = 0, pe = 0, pn = 0, ps = 0, pnw = 0, pne = 0, psw = 0, pse = 0;
#pragma unroll
        for (int k = 0; k < CC_TZ; k++) {
            if (t.z + k >= D) break;
            const int i = k * CC_THREADS + threadIdx.x, l = sl[i];
            const int w = sl[i + ow], e = sl[i + oe], n = sl[i + on], s = sl[i + os];
            const int nw = sl[i + on + ow], ne = sl[i + on + oe], sw = sl[i + os + ow], se = sl[i + os + oe];
            const bool bw = hw && w == l, bn = hn && n == l, bnw = hw && hn && nw == l;
            unsigned m = (bn ? (bw && bnw ? 0u : 1u << 1) : (bnw && !bw ? 1u << 0 : 0u)) |
                         (!bn && hn && he && ne == l && e != l ? 1u << 2 : 0u);
            if (k > 0) {
                const bool qn = hn && pn == l, qs = hs && ps == l, qw = hw && pw == l, qe = he && pe == l;
                const bool qnw = hn && hw && pnw == l, qsw = hs && hw && psw == l;
                m |= (qn ? (bw && qnw ? 0u : 1u << 10) : (qnw && !qw ? 1u << 9 : 0u)) |
                     (qs ? (bw && qsw ? 0u : 1u << 16) : (qsw && !qw ? 1u << 15 : 0u));
                if (!qn && !qs) m |= (qw ? 1u << 12 : 0u) | (qe ? 1u << 14 : 0u);
                if (he && !qe) m |= (!qn && hn && pne == l ? 1u << 11 : 0u) | (!qs && hs && pse == l ? 1u << 17 : 0u);
            }
            cc_put((unsigned *)sc, &nq, m, i);
            pw = w; pe = e; pn = n; ps = s; pnw = nw; pne = ne; psw = sw; pse = se;
        }
    }
    __syncthreads();
    cc_make((const unsigned *)sc, nq, join);
    __syncthreads();
#pragma unroll
    for (int k = 0; k < CC_TZ; k++) sc[k * CC_THREADS + threadIdx.x] = 0;
    __syncthreads();
#pragma unroll
    for (int k = 0; k < CC_TZ; k++) {
        int r = k * CC_THREADS + threadIdx.x;
        if (!in || t.z + k >= D) continue;
        for (int p = sp[r]; p != r; p = sp[r]) r = p;          // ends: parents are smaller
        if (len[k]) atomicAdd(&sc[r], (int)len[k]);
        par[gv + k * fr] = g0 + ((r / CC_THREADS) * H + (r % CC_THREADS) / 32) * W + r % 32;
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < CC_TZ; k++)
        if (in && t.z + k < D) cnt[gv + k * fr] = sc[k * CC_THREADS + threadIdx.x];
}

// The links that cross tiles: 22 rows of a tile have some along y or z (its first
// slice, the first and last row of the others), its 64 rows two voxels along x
__global__ void __launch_bounds__(CC_THREADS) k_cc_union(const int32_t *__restrict__ lab, int *par, int W, int H, int D,
                                                         int tx, int ty, int *err)
{
    asv_follow();
    constexpr unsigned PREV = 0x1ffu << 9, NORTH = 7u | (7u << 9), SOUTH = 7u << 15, WEST = 0x9249u, EAST = WEST << 2;
    constexpr int NW = CC_THREADS / 32, ROWS = NW + 2 * (CC_TZ - 1), TASKS = ROWS + 2 * NW * CC_TZ / 32;
    __shared__ unsigned queue[CC_TILE];
    __shared__ int nq;
    if (threadIdx.x == 0) nq = 0;
    __syncthreads();
    const CcTile t(tx, ty);
    const int fr = W * H, x0 = t.x - t.lane, y0 = t.y - t.w, g0 = (t.z * H + y0) * W + x0;
    auto join = [&](int i, int b) {
        const int q = b % 9, v = g0 + ((i / CC_THREADS) * H + (i % CC_THREADS) / 32) * W + i % 32;
        cc_union(par, v - (b >= 9 ? fr : 0) + (q / 3 - 1) * W + q % 3 - 1, v, err);
    };
    for (int task = t.w; task < TASKS; task += NW) {
        int k, r, lane = t.lane;
        unsigned cross;
        if (task < ROWS) {
            k = task < NW ? 0 : 1 + (task - NW) / 2;
            r = task < NW ? task : (task - NW) % 2 * (NW - 1);
            cross = (k == 0 ? PREV : 0u) | (r == 0 ? NORTH : 0u) | (r == NW - 1 ? SOUTH : 0u);
        } else {
            const int j = (task - ROWS) * 32 + lane;
            k = j / (2 * NW);
            r = j / 2 % NW;
            cross = lane & 1 ? EAST : WEST;
            lane = lane & 1 ? 31 : 0;
        }
        const int x = x0 + lane, y = y0 + r, z = t.z + k;
        unsigned m = 0;
        if (x < W && y < H && z < D) {
            const int32_t *p = lab + z * fr + y * W + x;
            m = cross & cc_links(__ldg(p), x > 0, x < W - 1, y > 0, y < H - 1, z > 0,
                                 [&](int dx, int dy, int dz) { return __ldg(p + dx + dy * W + dz * fr); });
        }
        // an entry per link: two in a row by one thread wait twice as long here
        const int i = k * CC_THREADS + r * 32 + lane;
        int at = m ? atomicAdd(&nq, __popc(m)) : 0;
        for (; m; m &= m - 1, at++) {
            if (at < CC_TILE) queue[at] = ((unsigned)i << 18) | (m & (0u - m));
            else join(i, __ffs(m) - 1);
        }
    }
    __syncthreads();
    cc_make(queue, min(nq, CC_TILE), join);
}

// The same two steps for volumes whose tiles would be nearly empty (lines, columns
// of a few voxels): the runs of equal label along x within a warp, then each
// voxel's links in global memory.  At 64 voxels per tile of 2048 the faster one:
// 131072x2x4 147 us a call, tiles 329; 262144x2x2 192, 567; at 128, 1024x1024x2 with
// noisy labels, 1266 against 634.
__global__ void __launch_bounds__(CC_THREADS) k_cc_runs(const int32_t *__restrict__ lab, int *par, int *cnt, int W, int n)
{
    asv_follow();
    const unsigned v = blockIdx.x * CC_THREADS + threadIdx.x, lane = threadIdx.x & 31;
    const bool in = v < (unsigned)n;
    const int l = in ? __ldg(lab + v) : 0, before = __shfl_up_sync(0xffffffffu, l, 1);
    const unsigned starts = __ballot_sync(0xffffffffu, lane == 0 || !in || l != before || v % (unsigned)W == 0);
    if (!in) return;
    const unsigned next = lane < 31 ? starts & (0xfffffffeu << lane) : 0u;
    par[v] = (int)(v - lane + 31 - __clz((int)(starts & (0xffffffffu >> (31 - lane)))));
    cnt[v] = (starts >> lane) & 1u ? (int)((next ? __ffs(next) - 1 : 32) - lane) : 0;
}

__global__ void __launch_bounds__(CC_THREADS) k_cc_link(const int32_t *__restrict__ lab, int *par, int W, int H, int D,
                                                        int n, int *err)
{
    asv_follow();
    const unsigned u = blockIdx.x * CC_THREADS + threadIdx.x;
    if (u >= (unsigned)n) return;
    const int v = (int)u, fr = W * H, row = v / W, x = v - row * W, z = row / H, y = row - z * H;
    const int32_t *p = lab + v;
    unsigned m = cc_links(__ldg(p), x > 0, x < W - 1, y > 0, y < H - 1, z > 0,
                          [&](int dx, int dy, int dz) { return __ldg(p + dx + dy * W + dz * fr); });
    if (threadIdx.x & 31) m &= ~(1u << 3);                     // W: of the same run
    for (; m; m &= m - 1) {
        const int b = __ffs(m) - 1, q = b % 9;
        cc_union(par, v - (b >= 9 ? fr : 0) + (q / 3 - 1) * W + q % 3 - 1, v, err);
    }
}

// par[v] = root, the tiles' component sizes added up at the roots, roots per
// chunk of CC_CHUNK voxels.  No links change any more, so walks end at the true
// roots, and only thread v writes par[v].  SPARSE: sizes are of runs, so most
// voxels of a warp add to one root, and do it once.
template <bool SPARSE>
__global__ void __launch_bounds__(CC_THREADS) k_cc_flatten(int *par, int *cnt, int n, int *chunk, int *err)
{
    asv_follow();
    constexpr int IT = CC_CHUNK / CC_THREADS;
    __shared__ int tot;
    if (threadIdx.x == 0) tot = 0;
    __syncthreads();
    const int v0 = blockIdx.x * CC_CHUNK + threadIdx.x;        // at most 2^31 - 1, as v0 + k * CC_THREADS
    int r[IT];
#pragma unroll
    for (int k = 0; k < IT; k++) r[k] = v0 + k * CC_THREADS < n ? par[v0 + k * CC_THREADS] : -1;
    bool walk = true;
    for (int it = 0; walk && it < CC_SPIN_LIMIT; it++) {       // the eight walks side by side
        walk = false;
        int p[IT];
#pragma unroll
        for (int k = 0; k < IT; k++) p[k] = r[k] >= 0 ? __ldcg(par + r[k]) : -1;
#pragma unroll
        for (int k = 0; k < IT; k++) { walk |= p[k] != r[k]; r[k] = p[k]; }
    }
    if (walk) atomicOr(err, 1);
    int roots = 0;
#pragma unroll
    for (int k = 0; k < IT; k++) {
        const int v = v0 + k * CC_THREADS;
        const bool child = v < n && r[k] != v;
        roots += v < n && !child;
        int c = child ? cnt[v] : 0;                            // of a tile's component: no one else's to change
        if (SPARSE) {
            const unsigned peers = __match_any_sync(0xffffffffu, child ? r[k] : -1);
            c = __reduce_add_sync(peers, c);
            if ((int)(threadIdx.x & 31) != __ffs(peers) - 1) c = 0;
        }
        if (c) atomicAdd(cnt + r[k], c);
        if (child) par[v] = r[k];
    }
    roots = __reduce_add_sync(0xffffffffu, roots);
    if ((threadIdx.x & 31) == 0 && roots) atomicAdd(&tot, roots);
    __syncthreads();
    if (threadIdx.x == 0) chunk[blockIdx.x] = tot;
}

// exclusive prefix of chunk[0..m) in place, total in *total (one block);
// count: m = ceil(*count / CC_SEGS) instead
__global__ void __launch_bounds__(1024) k_cc_prefix(int *chunk, int m, const int *count, int *total)
{
    asv_follow();
    __shared__ int part[32];
    __shared__ int carry;
    if (count) m = *count > CC_MAX_R ? 0 : (*count + CC_SEGS - 1) / CC_SEGS;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    if (threadIdx.x == 0) carry = 0;
    __syncthreads();
    for (int b0 = 0; b0 < m; b0 += 1024) {
        const int i = b0 + threadIdx.x;
        const int v = i < m ? chunk[i] : 0;
        int incl = v;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int t = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += t;
        }
        if (lane == 31) part[w] = incl;
        __syncthreads();
        if (w == 0) {
            int p = part[lane];
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int t = __shfl_up_sync(0xffffffffu, p, o);
                if (lane >= o) p += t;
            }
            part[lane] = p;
        }
        __syncthreads();
        if (i < m) chunk[i] = carry + (w ? part[w - 1] : 0) + incl - v;
        __syncthreads();
        if (threadIdx.x == 0) carry += part[31];
        __syncthreads();
    }
    if (threadIdx.x == 0) *total = carry;
}

// compact ids of the roots in raster order: rvox[id] = root voxel,
// rsize[id] = its size, cid[root] = id (cid overwrites the size array)
__global__ void __launch_bounds__(CC_THREADS) k_cc_compact(const int *__restrict__ par, int *cnt_cid,
                                                           const int *chunk, int n, int *rvox, int *rsize)
{
    asv_follow();
    constexpr int IT = CC_CHUNK / CC_THREADS, NW = CC_THREADS / 32;
    __shared__ int sum[IT * NW];                               // roots per iteration and warp, then their prefix
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    unsigned bal[IT];
#pragma unroll
    for (int k = 0; k < IT; k++) {
        const int v = blockIdx.x * CC_CHUNK + k * CC_THREADS + threadIdx.x;
        bal[k] = __ballot_sync(0xffffffffu, v < n && par[v] == v);
        if (lane == 0) sum[k * NW + w] = __popc(bal[k]);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        int c = chunk[blockIdx.x];
        for (int i = 0; i < IT * NW; i++) { const int t = sum[i]; sum[i] = c; c += t; }
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < IT; k++)
        if ((bal[k] >> lane) & 1u) {
            const int v = blockIdx.x * CC_CHUNK + k * CC_THREADS + threadIdx.x;
            const int id = sum[k * NW + w] + __popc(bal[k] & ((1u << lane) - 1u));
            rvox[id] = v;
            rsize[id] = cnt_cid[v];
            cnt_cid[v] = id;
        }
}

// kept segments per group of CC_SEGS, for the rank scan
__global__ void __launch_bounds__(CC_SEGS) k_cc_kept_count(const int *rsize, const int *R, int minsz, int *chunk)
{
    asv_follow();
    const int r = *R > CC_MAX_R ? 0 : *R;
    for (int g = blockIdx.x; (long long)g * CC_SEGS < r; g += gridDim.x) {
        const int j = g * CC_SEGS + threadIdx.x;
        const int c = __syncthreads_count(j < r && rsize[j] >= minsz);
        if (threadIdx.x == 0) chunk[g] = c;
    }
}

// Per segment j: its node F_j and the scan's node A_j.  node encoding:
// >= 0 pointer to a node (F_j = j, A_j = R + j), < 0 final value -1 - v.
__global__ void __launch_bounds__(CC_SEGS) k_cc_nodes(const int *__restrict__ par, const int *__restrict__ cid,
                                                      const int *__restrict__ rvox, const int *__restrict__ rsize,
                                                      const int *chunk, const int *R, int minsz, int W,
                                                      int H, int D, int *node)
{
    asv_follow();
    __shared__ int wsum[CC_SEGS / 32];
    const int r = *R > CC_MAX_R ? 0 : *R, lane = threadIdx.x & 31, w = threadIdx.x >> 5, sl = W * H;
    for (int g = blockIdx.x; (long long)g * CC_SEGS < r; g += gridDim.x) {
        const int j = g * CC_SEGS + threadIdx.x;
        const bool kept = j < r && rsize[j] >= minsz;
        const unsigned bal = __ballot_sync(0xffffffffu, kept);
        if (lane == 0) wsum[w] = __popc(bal);
        __syncthreads();
        int before = chunk[g];
        for (int k = 0; k < w; k++) before += wsum[k];
        __syncthreads();
        if (j >= r) continue;
        const int s = rvox[j];
        if (kept) node[j] = -1 - (before + __popc(bal & ((1u << lane) - 1u)));   // its label
        else node[j] = r + j;                                                    // = A_j
        // the scan of segment j: last neighbour of the seed in an earlier segment
        const int row = s / W, x = s - row * W, z = row / H, y = row - z * H;
        int adj = -1;
        for (int dz = -1; dz <= 1; dz++) {
            if (z + dz < 0 || z + dz >= D) continue;
#pragma unroll
            for (int k = 0; k < 8; k++) {
                const int xx = x + c_dx8[k], yy = y + c_dy8[k];
                if (xx < 0 || xx >= W || yy < 0 || yy >= H) continue;
                const int root = par[(z + dz) * sl + yy * W + xx];
                if (root < s) adj = root;
            }
        }
        if (adj >= 0) node[r + j] = cid[adj];        // A_j -> F of that segment
        else if (j > 0) node[r + j] = r + j - 1;     // A_j -> A_{j-1}
        else node[r + j] = -1;                       // initial value 0
    }
}

// One round over the 2R nodes: a node follows its chain up to CC_HOPS nodes
// further (chains point to smaller segments).  A round multiplies the distance
// that a pointer covers by CC_HOPS at least, so CC_ROUNDS rounds (256^4 >= 2^31)
// resolve every node; most end in the first.  On the way a node shows every
// CC_SHOWth place that it has come to, so that walks that come by go on from
// there: the nodes of a long chain walk at once, and every CC_SHOW steps take them
// that many times as far.  (Chains through 0.7 million small segments, 1x1x1048576
// with noisy labels: 427 us a call with the end of a walk shown only, 320 by doubling
// in 22 rounds, 204 so.)  alone: no segment has a neighbour, so every A node leads to
// the A node before, and those walk first (1048576x1x1: 614 us, so 214).
__global__ void __launch_bounds__(CC_THREADS) k_cc_jump(int *node, const int *R, bool alone)
{
    asv_follow();
    const int r = *R > CC_MAX_R ? 0 : *R;
    const unsigned step = gridDim.x * CC_THREADS;
    for (unsigned i = blockIdx.x * CC_THREADS + threadIdx.x; i < 2u * (unsigned)r; i += step) {
        const unsigned t = !alone ? i : (i < (unsigned)r ? i + r : i - r);
        int p = node[t];
        for (int k = 1; k <= CC_HOPS && p >= 0; k++) {
            p = __ldcg(node + p);
            if (p < 0 || k % CC_SHOW == 0) __stcg(node + t, p);
        }
    }
}

__global__ void __launch_bounds__(CC_THREADS) k_cc_output(const int *__restrict__ par, const int *__restrict__ cid,
                                                          const int *node, int n, const int *R, int32_t *out)
{
    asv_follow();
    if (*R > CC_MAX_R) return;
    const long long base = (long long)blockIdx.x * (4 * CC_THREADS) + threadIdx.x;
#pragma unroll
    for (int k = 0; k < 4; k++) {
        const long long v = base + k * CC_THREADS;
        if (v < n) {
            const int f = node[cid[par[v]]];
            out[v] = f < 0 ? -1 - f : 0x7fffffff;            // unresolved cannot happen; marked if it does
        }
    }
}

size_t asv_connect_scratch_bytes(long long n)
{
    const long long chunks = (n + CC_CHUNK - 1) / CC_CHUNK;
    // par, cid/size, rvox, rsize, node (2 per segment), chunk sums (+1), R, error word, labels
    return (size_t)(4 * n * 6 + 4 * (chunks + 2) + 256 * 8);
}

static int *carve(unsigned char *&p, long long count)
{
    int *r = (int *)p;
    p += ((size_t)count * 4 + 255) & ~(size_t)255;
    return r;
}

int asv_launch_connect(const int32_t *lab, int W, int H, int D, int supsz, int32_t *out, void *scratch,
                       cudaStream_t st, int *host_R, int *host_num)
{
    // One voxel wide: its rows as the rows along x of a volume one row high, the same
    // voxels in the same order with the same neighbours, that the tiles' lanes fill
    // (1024x1024x1: 169 us a call, 457 with a voxel per tile row).
    if (W == 1) { W = H; H = 1; }
    const long long n = (long long)W * H * D;
    const long long chunks = (n + CC_CHUNK - 1) / CC_CHUNK;
    unsigned char *p = (unsigned char *)scratch;
    int *par = carve(p, n), *cid = carve(p, n), *rvox = carve(p, n), *rsize = carve(p, n);
    int *node = carve(p, 2 * n), *chunk = carve(p, chunks + 1), *meta = carve(p, 4);
    int *kept = out;                                     // kept per group: read before k_cc_output writes there
    const int minsz = supsz / 4, ni = (int)n;
    const int tx = asv_tiles_along(W, 32), ty = asv_tiles_along(H, CC_THREADS / 32);
    const unsigned tiles = (unsigned)tx * ty * asv_tiles_along(D, CC_TZ);
    int *R = meta, *err = meta + 1, *num = meta + 2;
    cudaMemsetAsync(meta, 0, 16, st);
    const bool sparse = n <= (long long)CC_SPARSE * tiles;
    if (sparse) {
        const unsigned blocks = (unsigned)((n + CC_THREADS - 1) / CC_THREADS);
        asv_launch_follow(false, k_cc_runs, blocks, CC_THREADS, 0, st, lab, par, cid, W, ni);
        asv_launch_follow(true, k_cc_link, blocks, CC_THREADS, 0, st, lab, par, W, H, D, ni, err);
    } else {
        asv_launch_follow(false, k_cc_tile, tiles, CC_THREADS, 0, st, lab, par, cid, W, H, D, tx, ty, err);
        asv_launch_follow(true, k_cc_union, tiles, CC_THREADS, 0, st, lab, par, W, H, D, tx, ty, err);
    }
    asv_launch_follow(true, sparse ? k_cc_flatten<true> : k_cc_flatten<false>, (unsigned)chunks, CC_THREADS, 0, st, par, cid, ni, chunk, err);
    asv_launch_follow(true, k_cc_prefix, 1, 1024, 0, st, chunk, (int)chunks, nullptr, R);
    asv_launch_follow(true, k_cc_compact, (unsigned)chunks, CC_THREADS, 0, st, par, cid, chunk, ni, rvox, rsize);
    // the segments' kernels: enough threads for a few segments per chunk, any
    // number by grid strides
    const unsigned groups = (unsigned)(chunks < 1216 ? chunks : 1216);
    asv_launch_follow(true, k_cc_kept_count, groups, CC_SEGS, 0, st, rsize, R, minsz, kept);
    asv_launch_follow(true, k_cc_prefix, 1, 1024, 0, st, kept, 0, R, num);
    asv_launch_follow(true, k_cc_nodes, groups, CC_SEGS, 0, st, par, cid, rvox, rsize, kept, R, minsz, W, H, D, node);
    for (int k = 0; k < CC_ROUNDS; k++) asv_launch_follow(true, k_cc_jump, groups, CC_THREADS, 0, st, node, R, W * H == 1);
    asv_launch_follow(true, k_cc_output, (unsigned)((n + 4 * CC_THREADS - 1) / (4 * CC_THREADS)), CC_THREADS, 0, st, par, cid,
                      node, ni, R, out);
    int got[3] = { 0, 0, 0 };
    cudaMemcpyAsync(got, meta, sizeof(got), cudaMemcpyDeviceToHost, st);
    if (cudaStreamSynchronize(st) != cudaSuccess) return -1;
    if (cudaGetLastError() != cudaSuccess) return -1;
    if (got[1]) return -2;
    if (got[0] > CC_MAX_R) return -3;                    // node ids (2 per segment) are int
    *host_R = got[0];
    *host_num = got[2];
    return 0;
}

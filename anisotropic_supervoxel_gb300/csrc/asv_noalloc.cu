// asv_noalloc.cu -- check_dead_seeds post-processing over caller-owned
// device buffers, with no device allocation at all.
//
// Some hosts of this library cannot let it call cudaMalloc: a media
// pipeline or inference server that hands every byte of device memory out
// of its own pool (and audits that nothing else allocates), or a
// latency-bound stage where cudaMalloc/cudaFree would synchronize the device
// in the middle of other work.  For them this entry point takes a raw label
// volume and writes the post-processed one, using as scratch a fixed array
// that lives in the library's own device image: it is allocated when the
// library is loaded on a device and held until the process exits.
//
// The scratch is shared by every call on a device and keeps the last call's
// contents; the per-label counts are cleared at the start of each call, the
// other regions are fully rewritten before they are read.  Calls whose work
// overlaps on the GPU (different streams, or host threads without ordering)
// race on the scratch and must be serialized by the caller.
//
// The semantics are those of asv_check_dead_seeds (GPU-AS/Image.cpp:
// 1579-1778): count the voxels of each label, then relabel dead seeds
// (<= 3 dead: label_replace.gs in order; > 3: sequence_label's raster remap)
// and forward-fill label -1.  A label outside [-1, Kp) (which the JFA never
// writes) is read as -1 by every stage: counted in the -1 slot and filled.
#include "asv.h"
#include "asv_follow.cuh"
#include "asv_tally.cuh"

#include <cuda_runtime.h>

#include <mutex>

#define NA_CHUNK 2048
#define NA_GROUP 2                  // chunks per block of the count (1: 38.2 us a call on 320x240x85, 2: 36.8, 4: 38.0)
#define NA_FULL 0xffffffffu
#define NA_MAX_VOXELS (1LL << 25)
#define NA_MAX_SEEDS 32767
#define NA_MAX_CHUNKS (int)(NA_MAX_VOXELS / NA_CHUNK)

// scratch regions (bytes): counts (Kp+1 u32), rank (Kp i32), record, scan carries
#define NA_OFF_COUNTS 0
#define NA_OFF_RANK (NA_OFF_COUNTS + 4 * (NA_MAX_SEEDS + 1))
#define NA_OFF_REC (((NA_OFF_RANK + 4 * NA_MAX_SEEDS) + 255) & ~255)
#define NA_OFF_SCAN (NA_OFF_REC + 256)
#define NA_SCRATCH_BYTES (NA_OFF_SCAN + 4 * NA_MAX_CHUNKS)

static __device__ __align__(256) unsigned char g_asv_noalloc_scratch[NA_SCRATCH_BYTES];

enum { R_DEAD = 0, R_MODE = 1, R_INVALID = 2, R_L0 = 3, R_M0 = 4, R_DEAD0 = 5 };

struct NaScratch {
    unsigned int *counts;
    int *rank;
    int *rec;
    int *scan;
};

// a raw label as every stage reads it: outside [-1, Kp) -> -1
static __device__ __forceinline__ int na_label(const int32_t *__restrict__ raw, long long v, int Kp)
{
    const int l = raw[v];
    return (l >= 0 && l < Kp) ? l : -1;
}

static __device__ __forceinline__ int na_relabel(const int *rec, int Kp, int l)
{
    if (rec[R_MODE] != 1 || l < 0) return l;
    int last = Kp;
    for (int k = 0; k < rec[R_DEAD]; k++) {
        last -= 1;
        if (l == last) l = rec[R_DEAD0 + k];
    }
    return l;
}

static __device__ __forceinline__ bool na_scan_needed(const int *rec)
{
    return rec[R_MODE] == 2 || rec[R_INVALID] != 0;
}

// Voxels per label, and per chunk the last fill source of either rule that the
// label counts will choose between (k_na_scan): a voxel other than the first is
// one when its label is not -1 (up to three dead seeds, where a relabelled
// label never becomes -1), or neither -1 nor voxel 0's (more); voxel 0 always.
// Both in one word: place in the chunk + 1, the second rule's in the upper half.
// Neighbouring voxels mostly share a label: a warp adds each run once, found by
// one ballot, to the block's table (grouping all equal lanes into the global
// counts, and a second kernel for the sources, took 72 + 19 us on a 320x240x85
// volume, this one 20 us).
__global__ void __launch_bounds__(256) k_na_count(NaScratch s, const int32_t *__restrict__ raw, int n, int Kp)
{
    asv_follow();
    __shared__ Tally t;
    __shared__ unsigned last[NA_GROUP][2];
    tally_clear(t);
    if (threadIdx.x < 2 * NA_GROUP) (&last[0][0])[threadIdx.x] = 0u;
    __syncthreads();
    const int lane = threadIdx.x & 31, l0 = na_label(raw, 0, Kp);
    for (int c = 0; c < NA_GROUP; c++) {
        const int v0 = (blockIdx.x * NA_GROUP + c) * NA_CHUNK;
        if (v0 >= n) break;
        unsigned any = 0u, other = 0u;                         // place + 1 of the last source of each rule
        int all[NA_CHUNK / 256];                               // asked for together, before the table's accesses
#pragma unroll
        for (int i = 0; i < NA_CHUNK / 256; i++) {
            const int v = v0 + i * 256 + threadIdx.x;
            all[i] = v < n ? na_label(raw, v, Kp) : -2;
        }
#pragma unroll
        for (int i = 0; i < NA_CHUNK / 256; i++) {
            const int k = i * 256 + threadIdx.x, v = v0 + k, l = all[i];
            const bool in = v < n;
            const int before = __shfl_up_sync(NA_FULL, l, 1);
            const unsigned starts = __ballot_sync(NA_FULL, lane == 0 || before != l);
            if (in && ((starts >> lane) & 1u)) {
                const unsigned next = lane < 31 ? starts & (0xfffffffeu << lane) : 0u;
                const unsigned len = (unsigned)((next ? __ffs(next) - 1 : 32) - lane);
                const int slot = l < 0 ? Kp : l;
                if (!tally_add(t, slot, len)) atomicAdd(s.counts + slot, len);
            }
            if (in && (l >= 0 || v == 0)) {
                any = k + 1;
                if (l != l0 || v == 0) other = k + 1;
            }
        }
        any = __reduce_max_sync(NA_FULL, any);
        other = __reduce_max_sync(NA_FULL, other);
        if (lane == 0) {
            atomicMax(&last[c][0], any);
            atomicMax(&last[c][1], other);
        }
    }
    __syncthreads();
    if (t.key[threadIdx.x] >= 0) atomicAdd(s.counts + t.key[threadIdx.x], t.cnt[threadIdx.x]);
    const int c = blockIdx.x * NA_GROUP + threadIdx.x;
    if (threadIdx.x < NA_GROUP && (long long)c * NA_CHUNK < n)
        s.scan[c] = (int)(last[threadIdx.x][0] | (last[threadIdx.x][1] << 16));
}

// The alive ranks, the record, and where fills are needed every chunk's last
// source in the chunks before it (voxel + 1): one block
__global__ void __launch_bounds__(1024) k_na_scan(NaScratch s, const int32_t *__restrict__ raw, int Kp, int nchunks)
{
    asv_follow();
    __shared__ int warp_tot[32];
    __shared__ int carry;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    if (threadIdx.x == 0) carry = 0;
    __syncthreads();
    // four seeds a thread (the counts and the sources end on multiples of four)
    for (int b0 = 0; b0 < Kp; b0 += 4096) {
        const int i0 = b0 + 4 * threadIdx.x;
        unsigned alive = 0u;
        if (i0 < Kp) {
            const uint4 q = *(const uint4 *)(s.counts + i0);
            alive = (q.x ? 1u : 0u) | (q.y ? 2u : 0u) | (q.z ? 4u : 0u) | (q.w ? 8u : 0u);
            if (Kp - i0 < 4) alive &= (1u << (Kp - i0)) - 1u;
        }
        int incl = __popc(alive);
        for (int o = 1; o < 32; o <<= 1) { const int q = __shfl_up_sync(NA_FULL, incl, o); if (lane >= o) incl += q; }
        if (lane == 31) warp_tot[w] = incl;
        __syncthreads();
        if (threadIdx.x < 32) {
            int ix = warp_tot[threadIdx.x];
            for (int o = 1; o < 32; o <<= 1) { const int q = __shfl_up_sync(NA_FULL, ix, o); if (threadIdx.x >= o) ix += q; }
            warp_tot[threadIdx.x] = ix;
        }
        __syncthreads();
        const int before = carry + (w > 0 ? warp_tot[w - 1] : 0) + incl - __popc(alive);
#pragma unroll
        for (int k = 0; k < 4; k++) {
            const int i = i0 + k, live_before = before + __popc(alive & ((1u << k) - 1u));
            const bool live = (alive >> k) & 1u;
            if (i < Kp) {
                s.rank[i] = live ? live_before : -1;
                const int dead_before = i - live_before;        // the first four dead seeds, in order
                if (!live && dead_before < 4) s.rec[R_DEAD0 + dead_before] = i;
            }
        }
        __syncthreads();
        if (threadIdx.x == 0) carry += warp_tot[31];
        __syncthreads();
    }
    const int dead = Kp - carry;
    __syncthreads();
    if (threadIdx.x == 0) {
        s.rec[R_DEAD] = dead;
        s.rec[R_MODE] = dead == 0 ? 0 : (dead <= 3 ? 1 : 2);
        s.rec[R_INVALID] = s.counts[Kp] > 0 ? 1 : 0;
        const int l0 = na_label(raw, 0, Kp);
        s.rec[R_L0] = l0;
        s.rec[R_M0] = (l0 >= 0 && s.rank[l0] >= 0) ? s.rank[l0] : 0;
        carry = 0;
    }
    __syncthreads();
    if (!na_scan_needed(s.rec)) return;
    const int half = s.rec[R_MODE] == 2 ? 16 : 0;
    for (int b0 = 0; b0 < nchunks; b0 += 4096) {
        const int c0 = b0 + 4 * threadIdx.x;
        int v[4] = { 0, 0, 0, 0 };                             // voxel + 1 of the chunk's last source
        if (c0 < nchunks) {
            const int4 q = *(const int4 *)(s.scan + c0);
            const int p[4] = { q.x, q.y, q.z, q.w };
#pragma unroll
            for (int k = 0; k < 4; k++) {
                const int place = c0 + k < nchunks ? (p[k] >> half) & 0xffff : 0;
                v[k] = place ? (c0 + k) * NA_CHUNK + place : 0;
            }
        }
        int incl = max(max(v[0], v[1]), max(v[2], v[3]));
        for (int o = 1; o < 32; o <<= 1) { int q = __shfl_up_sync(NA_FULL, incl, o); if (lane >= o && q > incl) incl = q; }
        if (lane == 31) warp_tot[w] = incl;
        __syncthreads();
        if (threadIdx.x < 32) {
            int ix = warp_tot[threadIdx.x];
            for (int o = 1; o < 32; o <<= 1) { int q = __shfl_up_sync(NA_FULL, ix, o); if (threadIdx.x >= o && q > ix) ix = q; }
            warp_tot[threadIdx.x] = ix;
        }
        __syncthreads();
        int ew = __shfl_up_sync(NA_FULL, incl, 1);
        if (lane == 0) ew = 0;
        int ex = max(max(carry, w > 0 ? warp_tot[w - 1] : 0), ew);
#pragma unroll
        for (int k = 0; k < 4; k++) {
            if (c0 + k < nchunks) s.scan[c0 + k] = ex;
            ex = max(ex, v[k]);
        }
        __syncthreads();
        if (threadIdx.x == 0) carry = max(carry, warp_tot[31]);
        __syncthreads();
    }
}

// A thread takes eight consecutive voxels (VEC: by two 16-byte loads and
// stores, for buffers aligned to 16 bytes).  A fill carries the source's label
// itself: inside the thread, from the last lane before it that has a source,
// from the warps before, else from the chunk's source in k_na_scan.  (Voxel
// indices as 64-bit maxima and staging through shared memory: 45 us on a
// 320x240x85 volume, now 13 us.)
template <bool VEC>
__global__ void __launch_bounds__(256) k_na_apply(NaScratch s, const int32_t *__restrict__ raw,
                                                  int32_t *__restrict__ out, int n, int Kp)
{
    asv_follow();
    constexpr int PER = NA_CHUNK / 256;
    __shared__ int wlast[8];                                // label of the warp's last source, NONE without
    const int *rec = s.rec;
    const bool scan = na_scan_needed(rec);
    const int mode = rec[R_MODE], l0 = rec[R_L0], lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int NONE = -2;
    const int v0 = blockIdx.x * NA_CHUNK + threadIdx.x * PER;
    const bool full = VEC && v0 + PER <= n;
    int l[PER];
    if (full) {
#pragma unroll
        for (int k = 0; k < PER; k += 4) {
            const int4 q = *(const int4 *)(raw + v0 + k);
            l[k] = q.x; l[k + 1] = q.y; l[k + 2] = q.z; l[k + 3] = q.w;
        }
#pragma unroll
        for (int k = 0; k < PER; k++) l[k] = (l[k] >= 0 && l[k] < Kp) ? l[k] : -1;
    } else {
#pragma unroll
        for (int k = 0; k < PER; k++) l[k] = v0 + k < n ? na_label(raw, v0 + k, Kp) : -1;
    }
    if (scan) {
        // voxel 0 is a source of its own label in either rule, but the value it
        // gives is the rule's own: 0 for mode 2's map and for a -1 there
        auto source = [&](int k) { return (l[k] >= 0 && (mode != 2 || l[k] != l0)) || v0 + k == 0; };
        int mine = NONE;
#pragma unroll
        for (int k = 0; k < PER; k++)
            if (v0 + k < n && source(k)) mine = l[k];
        const unsigned has = __ballot_sync(NA_FULL, mine != NONE);
        const unsigned before = has & ((1u << lane) - 1u);
        const int from = __shfl_sync(NA_FULL, mine, before ? 31 - __clz((int)before) : 0);
        const int last = __shfl_sync(NA_FULL, mine, has ? 31 - __clz((int)has) : 0);
        if (lane == 0) wlast[w] = has ? last : NONE;
        __syncthreads();
        int cur = before ? from : NONE;
        for (int k = w - 1; k >= 0 && cur == NONE; k--) cur = wlast[k];
        if (cur == NONE) {
            const int src = s.scan[blockIdx.x] - 1;          // -1: none (the first chunk's first voxel is one)
            cur = src >= 0 ? na_label(raw, src, Kp) : -1;
        }
#pragma unroll
        for (int k = 0; k < PER; k++) {
            if (source(k)) cur = l[k];
            // mode 2: the source's rank; a source that is voxel 0 gives voxel 0's
            // own (its label is l0, every other source's is not).  Else the
            // source's relabelled label, 0 for a -1 at voxel 0 beyond it.
            if (mode == 2) l[k] = cur == l0 ? rec[R_M0] : ((cur >= 0 && s.rank[cur] >= 0) ? s.rank[cur] : 0);
            else {
                const int r = na_relabel(rec, Kp, cur);
                l[k] = v0 + k == 0 ? r : (r >= 0 ? r : 0);
            }
        }
    } else {
#pragma unroll
        for (int k = 0; k < PER; k++) l[k] = na_relabel(rec, Kp, l[k]);
    }
    if (full) {
#pragma unroll
        for (int k = 0; k < PER; k += 4) *(int4 *)(out + v0 + k) = make_int4(l[k], l[k + 1], l[k + 2], l[k + 3]);
    } else {
#pragma unroll
        for (int k = 0; k < PER; k++)
            if (v0 + k < n) out[v0 + k] = l[k];
    }
}

// Device address of the scratch array, resolved once per device (the first
// call on a device makes this runtime call; do that first call before any
// stream capture).  The array's name in host code is only a host-side
// stand-in, never a device address.
static std::mutex g_na_mu;
static void *g_na_ptr[256];

static cudaError_t na_scratch(int dev, void **out)
{
    std::lock_guard<std::mutex> lk(g_na_mu);
    if (!g_na_ptr[dev]) {
        void *p = nullptr;
        cudaError_t e = cudaGetSymbolAddress(&p, g_asv_noalloc_scratch);
        if (e != cudaSuccess) return e;
        g_na_ptr[dev] = p;
    }
    *out = g_na_ptr[dev];
    return cudaSuccess;
}

extern "C" asv_status asv_check_dead_seeds_noalloc(const int32_t *d_raw, int32_t *d_out, int W, int H,
                                                   int D, int Kp, void *stream)
{
    if (!d_raw || !d_out || W < 1 || H < 1 || D < 1 || Kp < 1) return ASV_ERR_BAD_ARG;
    if ((long long)W * H > NA_MAX_VOXELS || (long long)W * H * D > NA_MAX_VOXELS || Kp > NA_MAX_SEEDS)
        return ASV_ERR_BAD_ARG;
    long long n = (long long)W * H * D;
    // in and out must not overlap: blocks read labels of other chunks (the
    // fill source) while others write theirs
    const uintptr_t r0 = (uintptr_t)d_raw, o0 = (uintptr_t)d_out, nb = 4 * (uintptr_t)n;
    if (r0 < o0 + nb && o0 < r0 + nb) return ASV_ERR_BAD_ARG;
    // an error left pending by earlier work of the caller is returned as
    // ASV_ERR_CUDA and left pending for its owner (not cleared, not mixed
    // with this call's launches)
    if (cudaPeekAtLastError() != cudaSuccess) return ASV_ERR_CUDA;
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 256) { cudaGetLastError(); return ASV_ERR_NO_DEVICE; }
    void *base = nullptr;
    if (na_scratch(dev, &base) != cudaSuccess) { cudaGetLastError(); return ASV_ERR_CUDA; }
    cudaStream_t st = (cudaStream_t)stream;
    unsigned char *b = (unsigned char *)base;
    NaScratch s;
    s.counts = (unsigned int *)(b + NA_OFF_COUNTS);
    s.rank = (int *)(b + NA_OFF_RANK);
    s.rec = (int *)(b + NA_OFF_REC);
    s.scan = (int *)(b + NA_OFF_SCAN);
    int nchunks = (int)((n + NA_CHUNK - 1) / NA_CHUNK);
    if (cudaMemsetAsync(s.counts, 0, sizeof(unsigned int) * (size_t)(Kp + 1), st) != cudaSuccess) {
        cudaGetLastError();
        return ASV_ERR_CUDA;
    }
    k_na_count<<<(nchunks + NA_GROUP - 1) / NA_GROUP, 256, 0, st>>>(s, d_raw, (int)n, Kp);
    asv_launch_follow(true, k_na_scan, 1, 1024, 0, st, s, d_raw, Kp, nchunks);
    asv_launch_follow(true, ((r0 | o0) & 15) == 0 ? k_na_apply<true> : k_na_apply<false>, nchunks, 256, 0, st, s, d_raw, d_out,
                      (int)n, Kp);
    if (cudaGetLastError() != cudaSuccess) return ASV_ERR_CUDA;
    return ASV_OK;
}

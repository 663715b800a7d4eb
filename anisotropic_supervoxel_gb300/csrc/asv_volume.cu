// asv_volume.cu -- per-voxel and per-seed kernels of the supervoxel path.
//
// Compiled with -fmad=false: every float operation is one IEEE operation in
// the order written, so the labels match the CPU restatement bit for bit.
// Reference files (in dongxiao0401/anisotropic_supervoxel): GPU-AS/shaders/*,
// GPU-AS/Image.cpp.
#include "asv_follow.cuh"
#include "asv_seed.cuh"

#include <cuda_fp16.h>

#include <cstddef>
#include <mutex>

#define FULL 0xffffffffu

// ---------------------------------------------------------------------------
// RGB -> LAB (GPU-AS/shaders/RGB2LAB.fs:11-79).  Output bytes are the
// integers the shader writes to its RGB16F target (exact in 8 bits).
// ---------------------------------------------------------------------------
__device__ __forceinline__ float asv_pow_cr(float x, float y)
{
    return (float)pow((double)x, (double)y);
}

__global__ void k_srgb_table(float *__restrict__ tab)
{
    int c = threadIdx.x;
    if (c >= 256) return;
    float v = (float)c / 255.0f;                      // unorm8 texel
    float t;
    if (v <= 0.04045f) t = v / 12.92f;                 // RGB2LAB.fs:27-40
    else t = asv_pow_cr((v + 0.055f) / 1.055f, 2.4f);
    tab[c] = t;
}

// distance of x + 0.5 to the nearest integer (where floor(x + 0.5) can flip)
__device__ __forceinline__ float asv_tie_gap(float x)
{
    float y = x + 0.5f;
    return fabsf(y - rintf(y));
}

// The cube root f = r^(1/3) is first taken in FP32 (exp2/log2, error below
// 1e-6 relative, i.e. below 6e-4 on the scaled L, a, b); only when a scaled
// value lies within 4e-3 of a rounding boundary is the voxel recomputed with
// the correctly rounded FP64 path, so the bytes equal the exact ones.
// asv_lab_of_fp32 is the first part alone: it returns the FP32 bytes and
// whether asv_lab_of would recompute them.
__device__ __forceinline__ bool asv_lab_of_fp32(const float *__restrict__ tab, unsigned r, unsigned g, unsigned b,
                                                uchar4 &out)
{
    float t0 = tab[r], t1 = tab[g], t2 = tab[b];
    float X = (t0 * 0.412453f + t1 * 0.357580f) + t2 * 0.180423f;
    float Y = (t0 * 0.212671f + t1 * 0.715160f) + t2 * 0.072169f;
    float Z = (t0 * 0.019334f + t1 * 0.119193f) + t2 * 0.950227f;
    float rr[3] = { X / 0.950456f, Y / 1.0f, Z / 1.088754f };
    float f[3];
    bool cube[3];
#pragma unroll
    for (int k = 0; k < 3; k++) {
        cube[k] = rr[k] > 0.008856f;
        if (cube[k]) f[k] = exp2f(log2f(rr[k]) * (1.0f / 3.0f));
        else f[k] = (903.3f * rr[k] + 16.0f) / 116.0f;
    }
    float L = 116.0f * f[1] - 16.0f;
    float A = 500.0f * (f[0] - f[1]);
    float B = 200.0f * (f[1] - f[2]);
    L = L * 2.55f; A = A + 128.0f; B = B + 128.0f;
    const bool fix = (cube[0] || cube[1] || cube[2]) &&
                     fminf(asv_tie_gap(L), fminf(asv_tie_gap(A), asv_tie_gap(B))) < 4e-3f;
    float v0 = floorf(L + 0.5f), v1 = floorf(A + 0.5f), v2 = floorf(B + 0.5f);
    v0 = fminf(fmaxf(v0, 0.0f), 255.0f);
    v1 = fminf(fmaxf(v1, 0.0f), 255.0f);
    v2 = fminf(fmaxf(v2, 0.0f), 255.0f);
    out = make_uchar4((unsigned char)v0, (unsigned char)v1, (unsigned char)v2, 0);
    return fix;
}

__device__ __forceinline__ uchar4 asv_lab_of(const float *__restrict__ tab, unsigned r, unsigned g,
                                             unsigned b)
{
    float t0 = tab[r], t1 = tab[g], t2 = tab[b];
    float X = (t0 * 0.412453f + t1 * 0.357580f) + t2 * 0.180423f;   // fs:19-21, 42-44
    float Y = (t0 * 0.212671f + t1 * 0.715160f) + t2 * 0.072169f;
    float Z = (t0 * 0.019334f + t1 * 0.119193f) + t2 * 0.950227f;
    float rr[3] = { X / 0.950456f, Y / 1.0f, Z / 1.088754f };        // fs:54-55
    float f[3];
    bool cube[3];
#pragma unroll
    for (int k = 0; k < 3; k++) {
        cube[k] = rr[k] > 0.008856f;                                   // fs:57-70
        if (cube[k]) f[k] = exp2f(log2f(rr[k]) * (1.0f / 3.0f));
        else f[k] = (903.3f * rr[k] + 16.0f) / 116.0f;
    }
    float L = 116.0f * f[1] - 16.0f;                                  // fs:72
    float A = 500.0f * (f[0] - f[1]);
    float B = 200.0f * (f[1] - f[2]);
    L = L * 2.55f; A = A + 128.0f; B = B + 128.0f;                    // fs:74-76
    if ((cube[0] || cube[1] || cube[2]) &&
        fminf(asv_tie_gap(L), fminf(asv_tie_gap(A), asv_tie_gap(B))) < 4e-3f) {
#pragma unroll
        for (int k = 0; k < 3; k++)
            if (cube[k]) f[k] = asv_pow_cr(rr[k], 1.0f / 3.0f);
        L = 116.0f * f[1] - 16.0f;
        A = 500.0f * (f[0] - f[1]);
        B = 200.0f * (f[1] - f[2]);
        L = L * 2.55f; A = A + 128.0f; B = B + 128.0f;
    }
    float v0 = floorf(L + 0.5f), v1 = floorf(A + 0.5f), v2 = floorf(B + 0.5f);
    v0 = fminf(fmaxf(v0, 0.0f), 255.0f);
    v1 = fminf(fmaxf(v1, 0.0f), 255.0f);
    v2 = fminf(fmaxf(v2, 0.0f), 255.0f);
    return make_uchar4((unsigned char)v0, (unsigned char)v1, (unsigned char)v2, 0);
}

__global__ void __launch_bounds__(256) k_rgb2lab(AsvDev d)
{
    __shared__ float tab[256];
    tab[threadIdx.x] = d.srgb[threadIdx.x];
    __syncthreads();
    int si = asv_find_seg(d.chunk_prefix, d.nseg, blockIdx.x);
    const SegDesc &S = d.segs[si];
    long long base = (long long)(blockIdx.x - d.chunk_prefix[si]) * ASV_CHUNK;
    long long n = S.nvox;
    if (base + ASV_CHUNK <= S.lab_from) return;
    for (int i = 0; i < ASV_CHUNK / 256; i++) {
        long long v = base + i * 256 + threadIdx.x;
        if (v >= n) break;
        const uint8_t *p = d.rgb + 3 * (S.vox_off + v);
        d.lab[S.vox_off + v] = asv_lab_of(tab, p[0], p[1], p[2]);
    }
}

// The LAB bytes of all 2^24 RGB values, indexed r << 16 | g << 8 | b, built
// once per device in two passes: every entry in FP32, the entries near a
// rounding tie listed (about 2 %), then those entries again by asv_lab_of
// itself.  So a lookup returns exactly what the computation would (the
// exhaustive RGB2LAB test covers every entry), and the FP64 recomputations
// run in full warps instead of stalling half of all warps on one lane each.
__global__ void __launch_bounds__(256) k_lab_table(const float *__restrict__ srgb, uchar4 *__restrict__ lut,
                                                   unsigned *__restrict__ fix, unsigned *__restrict__ nfix)
{
    __shared__ float tab[256];
    tab[threadIdx.x] = srgb[threadIdx.x];
    __syncthreads();
    const unsigned c = blockIdx.x * 256u + threadIdx.x;              // 65536 blocks x 256
    uchar4 v;
    const bool again = asv_lab_of_fp32(tab, c >> 16, (c >> 8) & 255u, c & 255u, v);
    lut[c] = v;
    const unsigned m = __ballot_sync(0xffffffffu, again);            // one atomic per warp
    if (!m) return;
    const int lane = threadIdx.x & 31;
    unsigned at = 0;
    if (lane == __ffs(m) - 1) at = atomicAdd(nfix, (unsigned)__popc(m));
    at = __shfl_sync(0xffffffffu, at, __ffs(m) - 1);
    if (again) fix[at + __popc(m & ((1u << lane) - 1u))] = c;
}

__global__ void __launch_bounds__(256) k_lab_table_fix(const float *__restrict__ srgb, uchar4 *__restrict__ lut,
                                                       const unsigned *__restrict__ fix,
                                                       const unsigned *__restrict__ nfix)
{
    __shared__ float tab[256];
    tab[threadIdx.x] = srgb[threadIdx.x];
    __syncthreads();
    const unsigned n = *nfix;
    for (unsigned i = blockIdx.x * 256u + threadIdx.x; i < n; i += gridDim.x * 256u) {
        const unsigned c = fix[i];
        lut[c] = asv_lab_of(tab, c >> 16, (c >> 8) & 255u, c & 255u);
    }
}

// RGB -> LAB through the table: one 4-byte gather per voxel.  A thread takes four
// consecutive voxels: three 4-byte loads, four gathers in flight and one 16-byte
// store (segments start at multiples of ASV_CHUNK); with a voxel at a time, by
// bytes, a batch of 40.5 M voxels took 153 us, now 125: every lane's
// line is a lookup of its own.
__global__ void __launch_bounds__(256) k_rgb2lab_lut(AsvDev d)
{
    int si = asv_find_seg(d.chunk_prefix, d.nseg, blockIdx.x);
    const SegDesc &S = d.segs[si];
    long long base = (long long)(blockIdx.x - d.chunk_prefix[si]) * ASV_CHUNK;
    long long n = S.nvox;
    if (base + ASV_CHUNK <= S.lab_from) return;
    const uchar4 *__restrict__ lut = d.lablut;
#pragma unroll
    for (int i = 0; i < ASV_CHUNK / 1024; i++) {
        const long long v = base + i * 1024 + 4 * threadIdx.x;
        if (v + 4 <= n) {
            const unsigned *q = (const unsigned *)(d.rgb + 3 * (S.vox_off + v));
            const unsigned a = __ldg(q), b = __ldg(q + 1), c = __ldg(q + 2);       // RGBR GBRG BRGB
            const unsigned *t = (const unsigned *)lut;
            uint4 o;
            o.x = __ldg(t + __byte_perm(a, 0, 0x4012));
            o.y = __ldg(t + __byte_perm(__byte_perm(a, b, 0x0543), 0, 0x4012));
            o.z = __ldg(t + __byte_perm(__byte_perm(b, c, 0x0432), 0, 0x4012));
            o.w = __ldg(t + __byte_perm(c, 0, 0x4123));
            *(uint4 *)(d.lab + S.vox_off + v) = o;
        } else {
            for (long long u = v; u < n; u++) {
                const uint8_t *p = d.rgb + 3 * (S.vox_off + u);
                d.lab[S.vox_off + u] = __ldg(lut + (((unsigned)p[0] << 16) | ((unsigned)p[1] << 8) | p[2]));
            }
        }
    }
}

// ---------------------------------------------------------------------------
// Render::cvMat2TexureInput (GPU-AS/Render.cpp:354-359) for raw frames (BGR8,
// top row first): 3x3 Gaussian blur with sigma 0 (the [1,2,1] x [1,2,1] / 16
// kernel, border reflect-101, rounded half up), BGR -> RGB and the vertical
// flip into texture orientation.  One thread per output pixel and frame;
// the same integer arithmetic as the host asv_preprocess_frame.
// ---------------------------------------------------------------------------
__device__ __forceinline__ int asv_reflect101(int i, int n)
{
    if (n == 1) return 0;
    while (i < 0 || i >= n) i = i < 0 ? -i : 2 * n - 2 - i;
    return i;
}

__global__ void k_preprocess(const uint8_t *__restrict__ bgr, uint8_t *__restrict__ rgb, int W, int H, int D)
{
    const long long fr = (long long)W * H;
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= fr * D) return;
    const int z = (int)(t / fr), p = (int)(t - (long long)z * fr);
    const int yo = p / W, x = p - yo * W, y = H - 1 - yo;          // output row yo <- source row y
    const uint8_t *src = bgr + 3 * fr * z;
    int acc[3] = { 0, 0, 0 };
    for (int j = -1; j <= 1; j++) {
        const int yy = asv_reflect101(y + j, H);
        const int wy = j == 0 ? 2 : 1;
        for (int i = -1; i <= 1; i++) {
            const int xx = asv_reflect101(x + i, W);
            const int wgt = wy * (i == 0 ? 2 : 1);
            const uint8_t *q = src + 3 * ((long long)yy * W + xx);
            acc[0] += wgt * q[0];
            acc[1] += wgt * q[1];
            acc[2] += wgt * q[2];
        }
    }
    uint8_t *o = rgb + 3 * t;
    o[0] = (uint8_t)((acc[2] + 8) >> 4);                             // R <- channel 2 of BGR
    o[1] = (uint8_t)((acc[1] + 8) >> 4);
    o[2] = (uint8_t)((acc[0] + 8) >> 4);
}

void asv_launch_preprocess(const uint8_t *bgr, uint8_t *rgb, int W, int H, int D, cudaStream_t st)
{
    const long long n = (long long)W * H * D;
    k_preprocess<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(bgr, rgb, W, H, D);
}

// ---------------------------------------------------------------------------
// Gradient density per grid cell (GPU-AS/Image.cpp:350-620,
// derivative_t.gs:24-49, density_grid.vs:17-43).  Each voxel's gradient is
// rounded to half (RGB16F target) and summed exactly, in units of 2^-24.
// ---------------------------------------------------------------------------
__device__ __forceinline__ float asv_gradient(const uint8_t *__restrict__ rgb, int W, int H, int x,
                                              int y, int z)
{
    long long row = (long long)W;
    long long sl = (long long)W * H;
    long long v = z * sl + y * row + x;
    const uint8_t *c = rgb + 3 * v;
    const uint8_t *nb0 = rgb + 3 * (v - (x > 0 ? 1 : 0));
    const uint8_t *nb1 = rgb + 3 * (v - (y > 0 ? row : 0));
    const uint8_t *nb2 = rgb + 3 * (v - (z > 0 ? sl : 0));
    const uint8_t *nbs[3] = { nb0, nb1, nb2 };
    float g = 0.0f;
#pragma unroll
    for (int k = 0; k < 3; k++) {
        const uint8_t *q = nbs[k];
        float s = (float)abs((int)q[0] - (int)c[0]);
        s = s + (float)abs((int)q[1] - (int)c[1]);
        s = s + (float)abs((int)q[2] - (int)c[2]);
        g = g + 0.33f * s;                                            // gs:36, 43, 49
    }
    return g;
}

// value of a non-negative half in units of 2^-24
__device__ __forceinline__ unsigned long long asv_half_units(__half h)
{
    unsigned short b = __half_as_ushort(h);
    unsigned e = (b >> 10) & 0x1fu, m = b & 0x3ffu;
    if (e == 0) return m;
    return (unsigned long long)(1024u + m) << (e - 1);
}

__global__ void __launch_bounds__(256) k_density(AsvDev d)
{
    int si = asv_find_seg(d.chunk_prefix, d.nseg, blockIdx.x);
    const SegDesc &S = d.segs[si];
    const int W = S.W, H = S.H;
    const int *xc = d.cells + S.cell_off, *yc = xc + W, *zc = yc + H;
    const uint8_t *rgb = d.rgb + 3 * S.vox_off;
    unsigned long long *acc = d.dacc + S.seed_off;
    const int cap = d.seed_prefix[si + 1] - S.seed_off;
    long long base = (long long)(blockIdx.x - d.chunk_prefix[si]) * ASV_CHUNK;
    for (int i = 0; i < ASV_CHUNK / 256; i++) {
        long long v = base + i * 256 + threadIdx.x;
        int key = -1;
        unsigned u32 = 0;
        if (v < S.nvox) {
            int x = (int)(v % W);
            long long r = v / W;
            int y = (int)(r % H), z = (int)(r / H);
            int cx = xc[x], cy = yc[y], cz = zc[z];
            if (cx >= 0 && cy >= 0 && cz >= 0) {
                int k = (cz * S.hNum + cy) * S.wNum + cx;
                // cell id stored in an R16F texture (Image.cpp:474)
                int slot = (int)__half2float(__float2half_rn((float)k));
                unsigned long long units = asv_half_units(__float2half_rn(asv_gradient(rgb, W, H, x, y, z)));
                if (slot < cap) {
                    if ((units & 0xfffull) == 0 && (units >> 12) < (1ull << 26)) {
                        key = slot;
                        u32 = (unsigned)(units >> 12);
                    } else {
                        atomicAdd(acc + slot, units);
                    }
                }
            }
        }
        unsigned grp = __match_any_sync(FULL, key);
        unsigned sum = __reduce_add_sync(grp, u32);
        if (key >= 0 && (threadIdx.x & 31) == __ffs(grp) - 1)
            atomicAdd(acc + key, (unsigned long long)sum << 12);
    }
}

// 1-D redistribution of the seeds along the cells (Image.cpp:549-616).  One
// block per segment: the densities are formed in parallel, the prefix sums
// (sequential float sums in the reference) by one thread, the placement in
// parallel; on shared memory when Kp <= ASV_ADJ_SMEM, else on `scratch`
// (Kp floats).
#define ASV_ADJ_SMEM 12256     // floats: with the kernel's static counter the block stays within 48 KB

__global__ void __launch_bounds__(256) k_density_adjust(AsvDev d, float *scratch)
{
    extern __shared__ float sh_len[];
    int si = blockIdx.x;
    if (si >= d.nseg) return;
    const SegDesc &S = d.segs[si];
    const int Kp = S.Kp;
    const unsigned long long *acc = d.dacc + S.seed_off;
    const int *xl = d.cells + S.cell_off + S.W + S.H + S.D, *xr = xl + S.wNum;
    const float4 *grid = d.grid + S.seed_off;
    float *len = Kp <= ASV_ADJ_SMEM ? sh_len : scratch + S.seed_off;
    for (int i = threadIdx.x; i < Kp; i += blockDim.x) {
        unsigned long long tot = acc[i] + (3ull << 24);               // cleared to 3.0 (:506-507)
        float res = __ull2float_rn(tot) * 0x1p-24f;
        len[i] = (float)(0.001 * (double)res);                        // :554
    }
    __shared__ int placed;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int i = 1; i < Kp; i++) len[i] = len[i] + len[i - 1];    // :558-569 (float order kept)
        placed = 0;
    }
    __syncthreads();
    const float interval = len[Kp - 1] / (float)(Kp + 1);             // :570
    // The reference walks seeds and cells together (:586-616): seed i lands
    // in the first cell j1 with seed_in < len[j1], searching on from the
    // previous seed's cell.  seed_in grows with i and len never decreases,
    // so that cell is the first such cell of the whole array: found here by
    // a binary search per seed.  Once no cell qualifies the walk stops, so
    // the placed seeds are a prefix 0..n-1 of the ids.
    int mine = 0;
    for (int i = threadIdx.x; i < Kp; i += blockDim.x) {
        const float seed_in = (float)(i + 1) * interval;
        int lo = 0, hi = Kp;
        while (lo < hi) {
            const int mid = (lo + hi) >> 1;
            if (seed_in < len[mid]) hi = mid; else lo = mid + 1;
        }
        const int j1 = lo;
        if (j1 == Kp) continue;
        const int c = j1 % S.wNum;
        const int x1 = xl[c], x2 = xr[c];
        const float frac = j1 == 0 ? seed_in / len[j1] : (seed_in - len[j1 - 1]) / (len[j1] - len[j1 - 1]);
        const float ax = floorf((float)x1 + (float)(x2 - x1) * frac);
        const float4 g = grid[j1];
        d.pos0[S.seed_off + i] = make_float4((float)((double)ax + 0.5), g.y, g.z, (float)i);
        mine++;
    }
    atomicAdd(&placed, mine);
    __syncthreads();
    if (threadIdx.x == 0) d.post[si * ASV_POST_WORDS + POST_VALID] = placed;   // checked by the host
}

// ---------------------------------------------------------------------------
// Seeds: first-iteration init (draw_seeds.vs:20-35) and the per-iteration
// draw (draw_next_seeds.vs): seed record at the seed voxel, the later seed
// winning a shared voxel; JFA table packed for the passes.
// ---------------------------------------------------------------------------
__device__ __forceinline__ int asv_seed_seg(const AsvDev &d, int g, int &local)
{
    int si = asv_find_seg(d.seed_prefix, d.nseg, g);
    local = g - d.seed_prefix[si];
    return si;
}

__global__ void k_first_init(AsvDev d)
{
    int g = blockIdx.x * blockDim.x + threadIdx.x;
    if (g >= d.total_seeds) return;
    int i;
    int si = asv_seed_seg(d, g, i);
    const SegDesc &S = d.segs[si];
    if (i >= S.Kp) return;
    float4 p = d.pos0[g];
    d.pos[g] = p;
    d.mkey[g] = -1;   // a new Lloyd run starts without reseed memo
#pragma unroll
    for (int e = 0; e < 8; e++) d.M[8 * g + e] = d.M0[8 * g + e];
    int x = min(max((int)floorf(p.x), 0), S.W - 1);
    int y = min(max((int)floorf(p.y), 0), S.H - 1);
    int z = min(max((int)floorf(p.z), 0), S.D - 1);
    uchar4 l = d.lab[S.vox_off + ((long long)z * S.H + y) * S.W + x];
    d.slab[g] = make_float4((float)l.x, (float)l.y, (float)l.z, 0.0f);
}

__global__ void k_draw(AsvDev d)
{
    int g = blockIdx.x * blockDim.x + threadIdx.x;
    if (g >= d.total_seeds) return;
    int i;
    int si = asv_seed_seg(d, g, i);
    const SegDesc &S = d.segs[si];
    if (i >= S.Kp) return;
    asv_draw_seed(d, S, g, i, d.pos[g], d.slab[g], d.M + 8 * g);
}

// ---------------------------------------------------------------------------
// One JFA pass (GPU-AS/shaders/flood.gs:26-182).  27 candidates per voxel in
// the shader's order: slices z, z-step, z+step; in each slice rows
// y-step..y+step, columns x-step..x+step; clamp to edge.  The winner is the
// first candidate of least distance (strict `<` from 1e8), so any list that
// holds every valid candidate id, each first listed in the order of its first
// occurrence, gives the shader's label: a repeated id has the distance of its
// first occurrence and never wins again.
//
// Work layout: a block owns a tile of ASV_TILE_X x ASV_TILE_Y columns and a
// run of `zrun` voxels of each column, taken in chain order for the
// pass's step: z = r, r+step, r+2*step, ... (residue r = 0, 1, ...).  Along a
// chain the slice z+step of one voxel is the centre slice of the next and its
// centre the minus slice after that, so every slice's 9 labels are loaded
// and reduced to a list of ids once and used by up to three voxels (about
// 1.25 slice reductions per voxel instead of 3).  The voxel's list is the
// centre list, then the ids of the minus and plus lists not already listed
// (asv_merge_lists); a warp evaluates it in one loop, paying for its longest
// list.
// ---------------------------------------------------------------------------
#define ASV_JFA_THREADS 256
#define ASV_SLICE_MAX 9
typedef unsigned short asv_list_t;   // candidate-list entry in shared memory (ids < 32768)

// chain order of the D slices for `step`: position p -> residue r, index j
// in the chain, chain length len (z = r + j * step)
__device__ __forceinline__ void asv_chain_pos(int p, int D, int step, int &r, int &j, int &len)
{
    if (step >= D) { r = p; j = 0; len = 1; return; }
    const int q = D / step, m = D - q * step;       // m chains of q+1 slices, the rest q
    const int big = m * (q + 1);
    if (p < big) { r = p / (q + 1); j = p - r * (q + 1); len = q + 1; }
    else { const int pp = p - big; r = m + pp / q; j = pp - (r - m) * q; len = q; }
}

// valid ids among the 9 labels of one slice (offset zoff) around the
// column, each once, in first-occurrence order: a label is listed unless it
// equals one of the labels before it (compares against the loaded labels,
// all in registers, so nothing is shifted or stored to dedup).  Writes the
// list (stride ASV_JFA_THREADS), returns its length.
__device__ __forceinline__ int asv_slice_list(const int32_t *in, int zoff, const int xs[3],
                                              const int ys[3], int Kp, asv_list_t *__restrict__ lst)
{
    int32_t c[9];
#pragma unroll
    for (int oy = 0; oy < 3; oy++)
#pragma unroll
        for (int ox = 0; ox < 3; ox++) c[oy * 3 + ox] = asv_load_behind(in + zoff + ys[oy] + xs[ox]);
    int n = 0;
#pragma unroll
    for (int k = 0; k < 9; k++) {
        bool fresh = (unsigned)c[k] < (unsigned)Kp;
#pragma unroll
        for (int e = 0; e < k; e++) fresh = fresh && c[k] != c[e];
        if (fresh) {
            lst[n * ASV_JFA_THREADS] = (asv_list_t)c[k];
            n++;
        }
    }
    return n;
}

// The voxel's candidate list: the centre list A, then the ids of the minus
// list B and the plus list C that are not among A's first four entries or
// the last two ids appended (appended to X in order).  Returns X's length.
__device__ __forceinline__ int asv_merge_lists(const asv_list_t *__restrict__ A, int na,
                                               const asv_list_t *__restrict__ B, int nb,
                                               const asv_list_t *__restrict__ C, int nc,
                                               asv_list_t *__restrict__ X)
{
    const int h0 = na > 0 ? A[0] : -1, h1 = na > 1 ? A[ASV_JFA_THREADS] : -1;
    const int h2 = na > 2 ? A[2 * ASV_JFA_THREADS] : -1, h3 = na > 3 ? A[3 * ASV_JFA_THREADS] : -1;
    int nx = 0, r1 = -1, r2 = -1;
    const int n = nb + nc;
    for (int i = 0; i < n; i++) {
        const int l = i < nb ? B[i * ASV_JFA_THREADS] : C[(i - nb) * ASV_JFA_THREADS];
        if (l != h0 && l != h1 && l != h2 && l != h3 && l != r1 && l != r2) {
            X[nx * ASV_JFA_THREADS] = (asv_list_t)l;
            nx++;
            r2 = r1; r1 = l;
        }
    }
    return nx;
}

// flood.gs:72-94: anisotropic distance of the voxel centre to seed l of the
// table, in the shader's operation order: every product and sum of the
// shader on the same operands, each rounded once.  The voxel side comes
// packed as vxy = (x, y), vzl = (z, L), vab = (a, b); the table rows are
// (-x, -y, -z, -L), (M00, M11, 2 M02, 2 M12), (2 M01, M22, -a, -b), so the
// six differences are three two-wide additions (__fadd2_rn: each half
// rounds like the scalar addition, and v + (-s) is v - s) and the products
// pair up two-wide where both operands lie side by side: (dx dx, dy dy),
// (dz dz, eL eL), (ea ea, eb eb), (dx dz, dy dz), then those times
// (M00, M11) and (2 M02, 2 M12).  Every sum stays a scalar addition with
// explicit round-to-nearest (-fmad=false), which the PTX ISA keeps apart
// from the products; a two-wide product feeding a two-wide sum was seen
// fused into a two-wide FMA, so no sum is two-wide.  The bit-exact tests
// against the oracle (millions of distances per run) guard both.
__device__ __forceinline__ float asv_jfa_dist_v(const float4 t0, const float4 t1, const float4 t2, float2 vxy,
                                                float2 vzl, float2 vab, float ratio)
{
    const float2 dxy = __fadd2_rn(vxy, make_float2(t0.x, t0.y));              // (dx, dy)
    const float2 dzl = __fadd2_rn(vzl, make_float2(t0.z, t0.w));              // (dz, eL)
    const float2 eab = __fadd2_rn(vab, make_float2(t2.z, t2.w));              // (ea, eb)
    const float dx = dxy.x, dy = dxy.y, dz = dzl.x;
    const float2 sq = __fmul2_rn(dxy, dxy);
    const float2 zl = __fmul2_rn(dzl, dzl);
    const float2 ab = __fmul2_rn(eab, eab);
    const float2 cz = __fmul2_rn(dxy, make_float2(dz, dz));
    const float2 wa = __fmul2_rn(sq, make_float2(t1.x, t1.y));
    const float2 wc = __fmul2_rn(cz, make_float2(t1.z, t1.w));
    float p1 = wa.x + (dx * dy) * t2.x;
    p1 = p1 + wc.x;
    float p2 = wa.y + wc.y;
    p2 = p2 + zl.x * t2.y;
    float pos = p1 + p2;
    float col = zl.y + ab.x;
    col = col + ab.y;
    pos = (pos < 0.0f) ? 0.0f : pos;                                           // flood.gs:90-93
    return ratio * pos + col;                                                  // flood.gs:94
}

// the same with seed l's row of the table in global memory
__device__ __forceinline__ float asv_jfa_dist(const float4 *__restrict__ tab, int l, float2 vxy, float2 vzl,
                                              float2 vab, float ratio)
{
    return asv_jfa_dist_v(__ldg(tab + 3 * l), __ldg(tab + 3 * l + 1), __ldg(tab + 3 * l + 2), vxy, vzl, vab,
                          ratio);
}

// distance loop over the concatenated lists A (na) and X (nx): the first
// candidate of least distance wins (flood.gs:63, :95-99)
__device__ __forceinline__ int32_t asv_jfa_eval(const asv_list_t *__restrict__ A, int na,
                                                const asv_list_t *__restrict__ X, int nx,
                                                const float4 *__restrict__ tab, uchar4 c, float vx, float vy,
                                                float vz, float ratio)
{
    const float2 vxy = make_float2(vx, vy), vzl = make_float2(vz, (float)c.x);
    const float2 vab = make_float2((float)c.y, (float)c.z);
    float mind = 100000000.0f;
    int32_t best = -1;
    const int n = na + nx;
    int i = 0;
    for (; i + 1 < n; i += 2) {          // two candidates per trip: their loads overlap
        const int32_t la = i < na ? A[i * ASV_JFA_THREADS] : X[(i - na) * ASV_JFA_THREADS];
        const int32_t lb = i + 1 < na ? A[(i + 1) * ASV_JFA_THREADS] : X[(i + 1 - na) * ASV_JFA_THREADS];
        const float da = asv_jfa_dist(tab, la, vxy, vzl, vab, ratio);
        const float db = asv_jfa_dist(tab, lb, vxy, vzl, vab, ratio);
        if (da < mind) { mind = da; best = la; }     // compared in list order
        if (db < mind) { mind = db; best = lb; }
    }
    if (i < n) {
        const int32_t l = i < na ? A[i * ASV_JFA_THREADS] : X[(i - na) * ASV_JFA_THREADS];
        const float dist = asv_jfa_dist(tab, l, vxy, vzl, vab, ratio);
        if (dist < mind) { mind = dist; best = l; }
    }
    return best;
}

// Centroid sums of one voxel in the list form, fused into the last JFA pass
// of a Lloyd iteration (the bit-set form sums runs of equal labels instead,
// asv_run_flush) (centroids.vs:19-54; a label outside [0, Kp) counts in the
// -1 slot, so no slot beyond the segment's is written): the lanes of the warp are grouped by
// destination slot, reduced in the warp, and one u64 atomic per group and
// component is issued.  Every lane of the warp makes this call for every
// voxel of the tile (a lane whose column lies outside the segment passes
// valid = false and joins with key -1, which issues nothing), so the full
// warp mask is exact here whatever path the lanes took through the
// candidate evaluation before it.
__device__ __forceinline__ void asv_accumulate(unsigned long long *__restrict__ sums, int slot0, uchar4 c,
                                               int Kp, int x, int y, int z, int best, bool valid)
{
    const int key = valid ? slot0 + ((unsigned)best < (unsigned)Kp ? best : Kp) : -1;
    const unsigned grp = __match_any_sync(0xffffffffu, key);
    const unsigned q[7] = { 2u * x + 1u, 2u * y + 1u, 2u * z + 1u, 1u, c.x, c.y, c.z };
    unsigned s[7];
#pragma unroll
    for (int k = 0; k < 7; k++) s[k] = __reduce_add_sync(grp, q[k]);
    if (valid && (int)(threadIdx.x & 31) == __ffs(grp) - 1) {
        unsigned long long *dst = sums + 8ull * key;
#pragma unroll
        for (int k = 0; k < 7; k++) atomicAdd(dst + k, (unsigned long long)s[k]);
    }
}

// One column's run of zrun chain positions [p0, p0 + zrun).
// `lists` is this thread's first entry of 3 slice-list rows of ASV_SLICE_MAX
// entries and one merge row of 2 x ASV_SLICE_MAX.  A
// chain continues while z + step < D; the next chain starts at the next
// residue, whose minus slice is slice 0.  A lane whose column lies outside
// the segment runs the same loop on the clamped column (valid = false) and
// stores nothing, so the lanes of a warp stay in the same tile.
template <bool SUMS>
__device__ __forceinline__ void asv_jfa_run(const int32_t *in, int32_t *__restrict__ out,
                                            const uchar4 *__restrict__ lab, const float4 *__restrict__ tab,
                                            unsigned long long *__restrict__ sums, int slot0, int W, int H, int D,
                                            int Kp, int x, int y, int p0, int n, int step,
                                            float ratio, asv_list_t *__restrict__ lists, bool valid)
{
    const int sl = W * H;                       // segments hold < 2^31 voxels
    const int xs[3] = { max(x - step, 0), x, min(x + step, W - 1) };
    const int ys[3] = { max(y - step, 0) * W, y * W, min(y + step, H - 1) * W };
    const int col = y * W + x;
    const float vx = (float)x + 0.5f, vy = (float)y + 0.5f;
    const int row = ASV_SLICE_MAX * ASV_JFA_THREADS;
    int r, j, len;
    asv_chain_pos(p0, D, step, r, j, len);
    int z = r + j * step;
    int sm = 0, sc = 1, sp = 2;                 // list rows of the minus / centre / plus slices
    int nm = asv_slice_list(in, max(z - step, 0) * sl, xs, ys, Kp, lists + sm * row);
    int nc = asv_slice_list(in, z * sl, xs, ys, Kp, lists + sc * row);
    while (true) {
        const bool more = z + step < D;         // the chain goes on
        const int zp = more ? z + step : D - 1;
        const int np = asv_slice_list(in, zp * sl, xs, ys, Kp, lists + sp * row);
        const uchar4 c = __ldg(lab + z * sl + col);
        const int nx = asv_merge_lists(lists + sc * row, nc, lists + sm * row, nm, lists + sp * row, np,
                                       lists + 3 * row);
        const int32_t best = asv_jfa_eval(lists + sc * row, nc, lists + 3 * row, nx, tab, c, vx, vy,
                                          (float)z + 0.5f, ratio);
        if (valid) out[z * sl + col] = best;
        if (SUMS) asv_accumulate(sums, slot0, c, Kp, x, y, z, best, valid);
        if (--n == 0) break;
        if (more) {                             // next voxel of the chain: rotate the rows
            z = zp;
            const int t = sm;
            sm = sc; sc = sp; sp = t;
            nm = nc; nc = np;
        } else {                                // next residue: a new chain
            z = z - (z / step) * step + 1;
            nm = asv_slice_list(in, 0, xs, ys, Kp, lists + sm * row);
            nc = asv_slice_list(in, z * sl, xs, ys, Kp, lists + sc * row);
        }
    }
}

// The same for steps above the bit-set form's, whose chains have few positions
// (one at steps of D and more): the lists of slice 0 and of the last slice, where
// chains start and end, are made once per run, in two more rows, instead of up to
// two of three lists of every voxel (the 240x160x30 clip with its full ladder:
// steps 64 to 8, ten iterations 3.30 ms, so 3.16).  Small steps, whose crowded
// sub-tiles come here too, lose by it (the 64x48x12 clip 0.250 ms, so 0.256).
__device__ __forceinline__ void asv_jfa_run_far(const int32_t *in, int32_t *__restrict__ out,
                                                const uchar4 *__restrict__ lab, const float4 *__restrict__ tab, int W,
                                                int H, int D, int Kp, int x, int y, int p0, int n, int step,
                                                float ratio, asv_list_t *__restrict__ lists, bool valid)
{
    const int sl = W * H;                       // segments hold < 2^31 voxels
    const int xs[3] = { max(x - step, 0), x, min(x + step, W - 1) };
    const int ys[3] = { max(y - step, 0) * W, y * W, min(y + step, H - 1) * W };
    const int col = y * W + x;
    const float vx = (float)x + 0.5f, vy = (float)y + 0.5f;
    const int row = ASV_SLICE_MAX * ASV_JFA_THREADS;
    int r, j, len;
    asv_chain_pos(p0, D, step, r, j, len);
    int z = r + j * step;
    // list rows: 0 to 2 the chain's slices in turn, 3 and 4 the merge's, 5 and 6
    // slice 0 and slice D - 1, where chains start and end
    int rm, rc = 0, nm, n0 = -1, nl = -1;       // minus and centre rows
    auto first = [&]() {
        if (n0 < 0) n0 = asv_slice_list(in, 0, xs, ys, Kp, lists + 5 * row);
        rm = 5;
        nm = n0;
    };
    if (z > step) {
        rm = 2;
        nm = asv_slice_list(in, (z - step) * sl, xs, ys, Kp, lists + rm * row);
    } else first();
    int nc = asv_slice_list(in, z * sl, xs, ys, Kp, lists + rc * row);
    while (true) {
        const bool more = z + step < D;         // the chain goes on
        int rp = 6, np;
        if (more) {
            rp = rc == 2 ? 0 : rc + 1;
            np = asv_slice_list(in, (z + step) * sl, xs, ys, Kp, lists + rp * row);
        } else {
            if (nl < 0) nl = asv_slice_list(in, (D - 1) * sl, xs, ys, Kp, lists + 6 * row);
            np = nl;
        }
        const uchar4 c = __ldg(lab + z * sl + col);
        const int nx = asv_merge_lists(lists + rc * row, nc, lists + rm * row, nm, lists + rp * row, np,
                                       lists + 3 * row);
        const int32_t best = asv_jfa_eval(lists + rc * row, nc, lists + 3 * row, nx, tab, c, vx, vy,
                                          (float)z + 0.5f, ratio);
        if (valid) out[z * sl + col] = best;
        if (--n == 0) break;
        if (more) {                             // next voxel of the chain: rotate the rows
            z += step;
            rm = rc;
            nm = nc;
            rc = rp;
            nc = np;
        } else {                                // next residue: a new chain
            z = z - (z / step) * step + 1;
            first();
            nc = asv_slice_list(in, z * sl, xs, ys, Kp, lists + rc * row);
        }
    }
}

// ---------------------------------------------------------------------------
// Bit-set form of a JFA pass (steps 1..ASV_BITS_MAXS).
//
// The label a voxel takes depends only on the set of distinct valid labels
// among its 27 candidates, except when two of them tie at the least
// distance (then the first in the shader's candidate order wins): the
// distance is a function of the voxel and the label's seed alone.  A
// sub-tile (16 x 16 columns x up to 16 chain positions of the tile) holds
// few distinct labels in its whole footprint (the sub-tile grown by `step`
// on every side; on the benchmarked clips mostly under 32).  So the block
// copies the footprint into shared memory with asynchronous copies (one
// memory latency per sub-tile), numbers the footprint's distinct labels
// 0..T-1 (T <= 32; a sub-tile with more is cut in half, and takes the list form
// below four positions) and turns every footprint entry into its label's bit.  A
// voxel's candidate mask is the OR of the 9 bits of each of its three
// slices (the plus slice's mask becomes the next position's centre mask);
// a voxel with one candidate takes it, the others take the least score of
// their mask's labels (below), and the few whose scores are too close to call
// (1 or 2 in a thousand) the shader's own arithmetic: least distance below
// 1e8, and where two labels tie exactly at it, the shader's ordered scan of
// the voxel's 27 candidates.  So every label equals the shader's.
//
// The passes are bound by instruction issue, so the three steps before the
// walk handle four entries (a quad) per thread and access: a quad is copied
// by one 16-byte cp.async where the width allows it, numbered through a byte
// map that itself says which labels have a number (three instructions per
// entry where a claimed-bits test took about seventeen), and converted with
// one 16-byte load and store.  Each thread numbers the quads it copied, so
// no barrier stands between; with the slot slices worked out by every warp
// and the byte map reset behind the walk, a sub-tile has three barriers
// (six before).  A 1280x720x30 window of 20 iterations: 65.2 -> 53.8 ms, the
// 320x240x85 clip 13.9 -> 12.1 ms.  Widths that are no multiple of four
// copy their quads by four 4-byte cp.async.  A quad whose labels all have
// numbers already is turned into bits at once.
//
// Scores instead of the shader's arithmetic took the evaluation from 44 to 28
// instructions per candidate, and fewer registers: 64, so that with the LAB
// values read straight from global memory (one position ahead) four blocks
// fit an SM, three before.  Passes of a 1280x720x30 window (steps 6, 3, 2, 1,
// 2, 1 + sums) 499, 479, 439, 409, 443, 509 -> 316, 342, 315, 298, 326,
// 425 us.
//
// Then the shared-memory data path bound the passes (103 of its cycles for 32
// voxels of the step-3 pass, 85 % busy): a candidate's fourteen coefficients
// are fourteen words per lane whatever the load's width, and rows of 24 words
// let the two rows of a warp collide in eight banks.  Two positions share a
// candidate's load, a warp walks rows r and r + 2, and runs flush into four
// copies of the sums: 89 -> 59 million cycles at step 3, passes 289, 291, 273, 262, 282, 325 us.
//
// Footprint slices ("slots") of a sub-tile of n chain positions: slot 0 the
// minus slice of position 0, slots 1..n the centre slices, slot n+1 the plus
// slice of position n-1, and where a chain ends inside the sub-tile one for
// slice 0 (the minus slice of every chain start after the first) and one for
// slice D-1 (the clamped plus slice of every chain end), unless slot 0 or n+1
// is that slice already, as for a sub-tile of whole chains.  Along a
// chain the minus slice of a position is the centre of the one before it
// and its plus slice the centre of the one after it.
// ---------------------------------------------------------------------------
#define ASV_JFA_LIST_BYTES (5 * ASV_SLICE_MAX * ASV_JFA_THREADS * (int)sizeof(asv_list_t))
#define ASV_JFA_FAR_BYTES (7 * ASV_SLICE_MAX * ASV_JFA_THREADS * (int)sizeof(asv_list_t))   // asv_jfa_run_far's
#define ASV_BITS_MAXT 32         // labels per sub-tile footprint (one 32-bit mask)
#define ASV_BITS_MAXKP 8192      // segment seed counts up to this use the bit-set form
#define ASV_BITS_TLCAP 256       // claimed labels remembered for the reset
#define ASV_BITS_FREE 255        // map8: label without a number yet
#define ASV_BITS_NOLABEL 254     // map8[ASV_BITS_MAXKP]: no label (shifts to no bit)
#define ASV_BITS_OVER 253        // map8: a label past the 32nd (the sub-tile takes the list form)
#define ASV_ACC_ROW 5            // words per entry of the sub-tile's centroid-sum table (odd: the
                                 // entries' rows start in different shared-memory banks)
#define ASV_BITS_AREA 43264      // shared bytes of the footprint: four blocks per SM

#define ASV_ECO_ROW 5            // float4 per label of the score table (3.5 used; the odd count
                                 // spreads the rows of eight labels over all banks)

struct AsvBitsShared {
    float4 eco[ASV_ECO_ROW * ASV_BITS_MAXT];    // score coefficients per table entry (asv_bits_coefs)
    unsigned claim[ASV_BITS_MAXKP / 32];        // labels numbered in this sub-tile (all zero between)
    int4 slot[20];                              // per footprint slot: offset of its slice, slice relative to the
                                                // sub-tile's middle one (float bits), 2 z + 1 (positions' slots)
    unsigned short tlab[ASV_BITS_TLCAP];        // label of each number
    float magic[3];                             // 2^23 + the colour the scores are relative to
    float margin[2];                            // scores' error margin: [0] + [1] |colour|^2; [0] infinite: no scores
    int tcount;
    unsigned char map8[ASV_BITS_MAXKP + 4];     // number of each claimed label, ASV_BITS_FREE between
};

// The summing variant's centroid sums of the sub-tile, behind AsvBitsShared: per
// table entry (+ label -1) four copies of a row, taken by lanes in turn, so that
// the flushes of neighbouring columns, which mostly end runs of one label
// together, do not queue at one address.
#define ASV_ACC_COPIES 4
#define ASV_ACC_WORDS ((ASV_BITS_MAXT + 1) * ASV_ACC_COPIES * ASV_ACC_ROW)


// The footprint of a slot is kept as rows of 16-byte groups of four entries
// (quads): its left edge is rounded down to four columns, so that for widths
// that are multiples of four a quad is one aligned 16-byte copy, and a thread
// numbers and converts four entries per shared-memory access.
template <int S> struct AsvBitsGeo {
    static constexpr int AL = (S + 3) & ~3;                           // columns kept left and right of the tile
    static constexpr int FW = ASV_TILE_X + 2 * AL;                    // footprint width and height
    static constexpr int FH = ASV_TILE_Y + 2 * S;
    static constexpr int FP = FW * FH;                                // footprint entries per slot
    static constexpr int QW = FW / 4, QPS = FP / 4;                   // quads per row and per slot
    // slots the shared area holds, and chain positions per sub-tile, up to 16:
    // a sub-tile of n positions has n + 2 slots, or up to n + 4 where chains
    // end inside it
    static constexpr int NSLOT = ASV_BITS_AREA / (4 * FP) < 20 ? ASV_BITS_AREA / (4 * FP) : 20;
    static constexpr int SUB = NSLOT - 2 < 16 ? NSLOT - 2 : 16;
    // shared memory: the footprint (or the list rows), AsvBitsShared, sums
    static constexpr int AREA = NSLOT * FP * 4 > ASV_JFA_LIST_BYTES ? NSLOT * FP * 4 : ASV_JFA_LIST_BYTES;
    static constexpr int SMEM = AREA + (int)sizeof(AsvBitsShared);
};

// Slice of chain position p of the D slices for step S (asv_chain_pos's z).
// The quotients by the chain lengths go through FP32: numerators and
// denominators are below 4097, so (p + 0.5) / d is at least 0.5 / 4096 of its
// value away from an integer, far above the division's error.
template <int S>
__device__ __forceinline__ int asv_chain_z(int p, int D)
{
    const int q = D / S, m = D - q * S, big = m * (q + 1);
    const bool lo = p < big || q == 0;
    const int d = lo ? q + 1 : q, pp = lo ? p : p - big;
    const int r = (int)__fdividef((float)pp + 0.5f, (float)d);
    return (lo ? r : m + r) + (pp - r * d) * S;
}

// 4-byte asynchronous copy global -> shared (cp.async, completed by
// asv_cp_async_wait)
__device__ __forceinline__ void asv_cp_async4(void *dst, const void *src)
{
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(d), "l"(src) : "memory");
}
// 16-byte form: both addresses 16-byte aligned (through L2 only: a tile's
// footprint is read once per SM)
__device__ __forceinline__ void asv_cp_async16(void *dst, const void *src)
{
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(d), "l"(src) : "memory");
}
__device__ __forceinline__ void asv_cp_async_wait()
{
    asm volatile("cp.async.commit_group;\ncp.async.wait_all;\n" ::: "memory");
}

// Copies the four entries of one volume row from column x (any, also outside
// the row: clamp to edge) to four shared words.  vec: the row width is a
// multiple of four, so a quad inside the row is 16-byte aligned (x is a
// multiple of four, the volumes start on a 2048-voxel boundary).
__device__ __forceinline__ void asv_copy_quad(void *dst, const int32_t *__restrict__ src, int row, int x, int W,
                                              bool vec)
{
    char *q = (char *)dst;
    if (x >= 0 && x + 3 < W) {
        const int32_t *g = src + row + x;
        if (vec) asv_cp_async16(q, g);
        else {
#pragma unroll
            for (int i = 0; i < 4; i++) asv_cp_async4(q + 4 * i, g + i);
        }
    } else {
#pragma unroll
        for (int i = 0; i < 4; i++) asv_cp_async4(q + 4 * i, src + row + min(max(x + i, 0), W - 1));
    }
}

// index of a label in map8: labels lie in [-1, Kp), no label is the last entry
__device__ __forceinline__ unsigned asv_bits_slot(int v) { return min((unsigned)v, (unsigned)ASV_BITS_MAXKP); }

// 1 << n, 0 for n > 31 (PTX shl clamps the amount)
__device__ __forceinline__ unsigned asv_bit(unsigned n)
{
    unsigned r;
    asm("shl.b32 %0, 1, %1;" : "=r"(r) : "r"(n));
    return r;
}

// a label seen without a number: the thread that claims it gives it the next one
// and starts the copy of its seed table row
__device__ __forceinline__ void asv_bits_claim(AsvBitsShared &b, unsigned v, const float4 *__restrict__ tab)
{
    const unsigned bit = 1u << (v & 31);
    if (atomicOr(&b.claim[v >> 5], bit) & bit) return;
    const int idx = atomicAdd(&b.tcount, 1);
    if (idx < ASV_BITS_TLCAP) b.tlab[idx] = (unsigned short)v;
    if (idx < ASV_BITS_MAXT) {
#pragma unroll
        for (int k = 0; k < 3; k++) asv_cp_async16(b.eco + ASV_ECO_ROW * idx + k, tab + 3 * v + k);
    }
    b.map8[v] = (unsigned char)(idx < ASV_BITS_MAXT ? idx : ASV_BITS_OVER);
}

// the labels and claims of a finished sub-tile: back to unnumbered
__device__ __forceinline__ void asv_bits_reset(AsvBitsShared &b, int T)
{
    if (T <= ASV_BITS_TLCAP) {
        for (int i = threadIdx.x; i < T; i += ASV_JFA_THREADS) {
            b.claim[b.tlab[i] >> 5] = 0u;
            b.map8[b.tlab[i]] = ASV_BITS_FREE;
        }
    } else {
        for (int i = threadIdx.x; i < ASV_BITS_MAXKP / 32; i += ASV_JFA_THREADS) b.claim[i] = 0u;
        for (int i = threadIdx.x; i < ASV_BITS_MAXKP / 4; i += ASV_JFA_THREADS) ((unsigned *)b.map8)[i] = 0xffffffffu;
    }
}

// ---------------------------------------------------------------------------
// Scores.  Which label of a voxel's mask has the least distance is mostly
// decided without the shader's arithmetic: the distance is a quadratic form
// of the voxel's coordinates plus a colour term, so with the coordinates
// (u, v, w) and the colour (l, a, b) taken relative to the sub-tile's middle,
// distance - (l^2 + a^2 + b^2) is
//   max(K0 + ku u + kv v + kw w + kuu u^2 + kvv v^2 + kww w^2 + kuv u v
//       + kuw u w + kvw v w, c0) + cl l + ca a + cb b
// (K0 and c0 hold the colour constant c0 = |seed colour|^2; the max is the
// clamp of a negative form, flood.gs:90-93): fourteen coefficients per label,
// ten fused multiply-adds and additions where the shader's order takes
// twenty-one, nothing between them that must round apart.
//
// Both this score and the shader's rounded distance are off the exact value
// by no more than a bound that follows from the operands' sizes.  With
// e = 2^-24, A = ratio * sum |M_ij| |d_i| |d_j| over the sub-tile's extent and
// C = |s|^2 + 2 sum |s_k| |c_k| for the relative colours s of the seed and c of
// the voxel:
//   shader's distance: 9 e A + 6 e distance (each term passes at most 9
//     roundings, a colour term 6),
//   score: 17 e A + 11 e C (coefficients up to 10 roundings, the sum 7).
// So where the least score is below every other by more than
//   72 e A + 32 e C + 16 e (sum of both distances)
// (the larger label's bounds, twice, with room to spare) it is the strictly
// least shader distance.  With S the largest relative seed colour component
// of the table, q = |(l, a, b)|^2 and |l| + |a| + |b| <= q / 32 + 24, that is
// at most margin[0] + margin[1] q + 16 e (both scores), where
//   margin[0] = max over the labels of 72 e A + 32 e |s|^2, + 64 e S 24,
//   margin[1] = 64 e S / 32 + 32 e.
// Any closer voxel is evaluated in the shader's order (asv_bits_exact), so
// the labels are the shader's in every case.  A label whose A or colour is
// not finite or so large that a distance might reach 1e8 gives an infinite
// margin: that sub-tile takes no scores.  So does a negative ratio (a caller's own
// pass): the shader clamps the form before it is multiplied, and max(ratio * form, 0)
// is that only for ratios of zero and more.
// ---------------------------------------------------------------------------
#define ASV_EPS 5.9604645e-8f    // 2^-24

// One warp, lane = table entry: replaces the entry's seed table row, which the
// claiming thread copied to the entry's place, by its score coefficients
// (ox, oy, oz: the sub-tile's middle, wmax: the largest |w| of its positions).
__device__ __forceinline__ void asv_bits_coefs(AsvBitsShared &b, int T, float ox, float oy, float oz, float wmax,
                                               float ratio)
{
    const int lane = threadIdx.x & 31;
    const bool on = lane < T;
    float4 *e = b.eco + ASV_ECO_ROW * lane;
    float4 r0 = make_float4(0.f, 0.f, 0.f, 0.f), r1 = r0, r2 = r0;
    if (on) { r0 = e[0]; r1 = e[1]; r2 = e[2]; }
    const float col[3] = { -r0.w, -r2.z, -r2.w };
    float s[3], mid[3];
#pragma unroll
    for (int k = 0; k < 3; k++) {                     // middle of the labels' colours
        const int q = min(max(__float2int_rn(col[k]), 0), 255);
        const int lo = __reduce_min_sync(FULL, on ? q : 255), hi = __reduce_max_sync(FULL, on ? q : 0);
        mid[k] = (float)((lo + hi) >> 1);
        s[k] = col[k] - mid[k];
    }
    const float su = -(r0.x + ox), sv = -(r0.y + oy), sw = -(r0.z + oz);
    const float a00 = ratio * r1.x, a11 = ratio * r1.y, a02 = ratio * r1.z, a12 = ratio * r1.w;
    const float a01 = ratio * r2.x, a22 = ratio * r2.y;
    const float c0 = s[0] * s[0] + s[1] * s[1] + s[2] * s[2];
    const float ku = -(2.0f * a00 * su + a01 * sv + a02 * sw);
    const float kv = -(2.0f * a11 * sv + a01 * su + a12 * sw);
    const float kw = -(2.0f * a22 * sw + a02 * su + a12 * sv);
    const float k0 = a00 * su * su + a01 * su * sv + a02 * su * sw + a11 * sv * sv + a12 * sv * sw + a22 * sw * sw;
    const float X = fabsf(su) + 8.0f, Y = fabsf(sv) + 8.0f, Z = fabsf(sw) + wmax;
    const float A = fabsf(a00) * X * X + fabsf(a01) * X * Y + fabsf(a02) * X * Z + fabsf(a11) * Y * Y +
                    fabsf(a12) * Y * Z + fabsf(a22) * Z * Z;
    const float smax = fmaxf(fmaxf(fabsf(s[0]), fabsf(s[1])), fabsf(s[2]));
    const bool ok = ratio >= 0.0f && A < 1e7f && smax < 1000.0f && s[0] == s[0] && s[1] == s[1] && s[2] == s[2];   // false for NaN
    const float mg = ok ? 72.0f * ASV_EPS * A + 32.0f * ASV_EPS * c0 + 1e-30f : __int_as_float(0x7f800000);
    const unsigned top = __reduce_max_sync(FULL, on ? __float_as_uint(mg) : 0u);     // non-negative floats
    const unsigned stop = __reduce_max_sync(FULL, on && ok ? __float_as_uint(smax) : 0u);
    if (on) {
        e[0] = make_float4(ku, kv, a00, a11);
        e[1] = make_float4(a02, a12, a22, a01);
        e[2] = make_float4(kw, k0 + c0, c0, -2.0f * s[0]);
        *(float2 *)(e + 3) = make_float2(-2.0f * s[1], -2.0f * s[2]);
    }
    if (lane == 0) {
        const float S = __uint_as_float(stop);
        b.margin[0] = __uint_as_float(top) + 64.0f * 24.0f * ASV_EPS * S;
        b.margin[1] = 2.0f * ASV_EPS * S + 32.0f * ASV_EPS;
#pragma unroll
        for (int k = 0; k < 3; k++) b.magic[k] = 8388608.0f + mid[k];
    }
}

// The label of mask m for one voxel in the shader's own arithmetic: least
// distance below 1e8 over the mask's labels in any order; where two tie at
// it, the shader's ordered scan of the 27 candidates (slices centre, minus,
// plus; rows y-S, y, y+S; columns x-S, x, x+S) over the footprint's label
// bits, strict '<' from 1e8 (flood.gs:63, :95-99).  Returns the table entry
// or -1.
template <int S>
__device__ __noinline__ int asv_bits_exact(unsigned m, const unsigned *__restrict__ fc, const unsigned *__restrict__ fm,
                                           const unsigned *__restrict__ fp, const AsvBitsShared &b,
                                           const float4 *__restrict__ tab, int x, int y, int z, unsigned c, float ratio)
{
    constexpr int FW = AsvBitsGeo<S>::FW;
    const float2 vxy = make_float2((float)x + 0.5f, (float)y + 0.5f);
    const float2 vzl = make_float2((float)z + 0.5f, (float)(c & 255u));
    const float2 vab = make_float2((float)((c >> 8) & 255u), (float)((c >> 16) & 255u));
    float mind = 100000000.0f;
    int best = -1;
    bool tie = false;
    while (m) {
        const int e = __ffs(m) - 1;
        m &= m - 1;
        const float dist = asv_jfa_dist(tab, b.tlab[e], vxy, vzl, vab, ratio);
        if (dist < mind) { mind = dist; best = e; tie = false; } else if (dist == mind) tie = true;
    }
    if (!tie) return best;
    mind = 100000000.0f;
    best = -1;
    for (int k = 0; k < 3; k++) {
        const unsigned *f = k == 0 ? fc : (k == 1 ? fm : fp);
        for (int a = 0; a < 3; a++)
            for (int o = 0; o < 3; o++) {
                const unsigned bit = f[a * S * FW + o * S];
                if (!bit) continue;
                const int e = __ffs(bit) - 1;
                const float dist = asv_jfa_dist(tab, b.tlab[e], vxy, vzl, vab, ratio);
                if (dist < mind) { mind = dist; best = e; }
            }
    }
    return best;
}

// A thread's run of voxels with one label, added to its table entry's
// centroid sums in shared memory.  A run is its sum of 2 z + 1, its sums of
// L | a << 16 and its sums of b | count << 16; an entry has five words:
// sums of the columns x | y << 16 within the tile, of count << 20 | L, of
// 2 z + 1, of a and of b.  All exact: a summing sub-tile has at most 15 x 256
// = 3840 voxels, so the columns stay below 3840 * 15 < 2^16, L below 3840 *
// 255 < 2^20 and the count below 2^12.  (With seven words, one sum each, the
// summing pass of a 1280x720x30 window took 425 us.)
__device__ __forceinline__ void asv_run_words(unsigned w[ASV_ACC_ROW], unsigned z, unsigned la, unsigned bn, unsigned xy)
{
    w[0] = (bn >> 16) * xy;
    w[1] = ((bn & 0xffff0000u) << 4) | (la & 0xffffu);
    w[2] = z;
    w[3] = la >> 16;
    w[4] = bn & 0xffffu;
}

__device__ __forceinline__ void asv_run_flush(unsigned *__restrict__ a, unsigned z, unsigned la, unsigned bn, unsigned xy)
{
    unsigned w[ASV_ACC_ROW];
    asv_run_words(w, z, la, bn, xy);
#pragma unroll
    for (int k = 0; k < ASV_ACC_ROW; k++) atomicAdd(a + k, w[k]);
}

// One sub-tile of n <= SUB chain positions from p0 in bit-set form; false
// (nothing written) when its footprint holds more than 32 labels.  Called
// by the whole block.
template <int S, bool SUMS>
__device__ bool asv_jfa_bits_sub(const int32_t *in, int32_t *__restrict__ out,
                                 const uchar4 *__restrict__ lab, const float4 *__restrict__ tab,
                                 unsigned long long *__restrict__ sums, int slot0, int W, int H, int D, int Kp,
                                 int tx0, int ty0, int p0, int n, float ratio, unsigned char *smem)
{
    using G = AsvBitsGeo<S>;
    constexpr int FW = G::FW, FP = G::FP;
    int *flab = (int *)smem;                                   // labels, then their bits
    AsvBitsShared &b = *(AsvBitsShared *)(smem + G::AREA);
    unsigned *const acc = (unsigned *)(smem + G::SMEM);           // (summing variant)
    const int tid = threadIdx.x, lane = tid & 31;
    const int sl = W * H;
    // a warp walks rows r and r + 2 of the tile: with footprint rows of 24
    // words their reads fall in different banks (rows r and r + 1 shared eight)
    const int lx = tid % ASV_TILE_X, ly = (tid >> 6) * 4 + ((tid >> 5) & 1) + ((tid >> 3) & 2);
    const int gx = tx0 + lx, gy = ty0 + ly;
    const bool valid = gx < W && gy < H;                       // other lanes run along, store nothing
    const int x = min(gx, W - 1), y = min(gy, H - 1);
    const int col = y * W + x;

    // slices of the footprint slots: every warp works them out and writes
    // the same values, so no barrier is needed before they are read; brk
    // has a bit for each position but the last where a chain ends
    unsigned brk;
    int nf, zslot = 0, lslot;                                  // slots; those of slice 0 and slice D - 1
    int zc;                                                    // middle slice of the positions
    float wmax;                                                // largest distance from it
    {
        const int z = lane < n ? asv_chain_z<S>(p0 + lane, D) : 0;
        const bool end = lane < n - 1 && z + S >= D;
        brk = __ballot_sync(FULL, end);
        const int zf = __shfl_sync(FULL, z, 0), zl = __shfl_sync(FULL, z, n - 1);
        if (zf > S) zslot = n + 2;
        if (zl + S < D - 1) lslot = zslot ? n + 3 : n + 2;
        else lslot = n + 1;
        nf = n + 2 + (brk ? (zslot != 0) + (lslot != n + 1) : 0);
        if (nf > G::NSLOT) return false;
        const int z0 = __reduce_min_sync(FULL, lane < n ? z : D), z1 = __reduce_max_sync(FULL, z);
        zc = (z0 + z1) >> 1;
        wmax = (float)(z1 - zc);                               // z1 - zc >= zc - z0
        if (lane < n) b.slot[1 + lane] = make_int4(z * sl, __float_as_int((float)(z - zc)), 2 * z + 1, 0);
        if (lane == 0) {                                       // (every entry a slice of the volume, used or not)
            b.slot[0].x = max(zf - S, 0) * sl;
            b.slot[n + 1].x = min(zl + S, D - 1) * sl;
            b.slot[n + 2].x = zslot ? 0 : (D - 1) * sl;
            b.slot[n + 3].x = (D - 1) * sl;
        }
        __syncwarp();
    }

    // footprint labels (clamp-to-edge), copied asynchronously a quad at a time
    const bool vec = (W & 3) == 0;
    const int items = nf * G::QPS;
    {
        int slot = tid / G::QPS, q = tid - slot * G::QPS;
        for (int e = tid; e < items; e += ASV_JFA_THREADS) {
            const int fy = q / G::QW, fx = q - fy * G::QW;
            asv_copy_quad(flab + 4 * e, in, b.slot[slot].x + min(max(ty0 - S + fy, 0), H - 1) * W,
                          tx0 - G::AL + 4 * fx, W, vec);
            q += ASV_JFA_THREADS % G::QPS;
            slot += ASV_JFA_THREADS / G::QPS;
            if (q >= G::QPS) { q -= G::QPS; slot++; }
        }
    }
    asv_cp_async_wait();

    // number the distinct labels, each thread those of the quads it copied
    // (its own copies are complete, so no barrier comes first), and turn the
    // quads' entries into their labels' bits in place (0: no label).  A quad
    // with a label that had no number yet is turned after the barrier.
    unsigned pend = 0u;
    for (int e = tid, k = 0; e < items; e += ASV_JFA_THREADS, k++) {
        int4 *q = (int4 *)(flab + 4 * e);
        const int4 v = *q;
        const unsigned i0 = asv_bits_slot(v.x), i1 = asv_bits_slot(v.y), i2 = asv_bits_slot(v.z),
                       i3 = asv_bits_slot(v.w);
        const volatile unsigned char *mp = b.map8;
        const unsigned m0 = mp[i0], m1 = mp[i1], m2 = mp[i2], m3 = mp[i3];
        if (max(max(m0, m1), max(m2, m3)) == ASV_BITS_FREE) {
            if (m0 == ASV_BITS_FREE) asv_bits_claim(b, i0, tab);
            if (m1 == ASV_BITS_FREE && i1 != i0) asv_bits_claim(b, i1, tab);
            if (m2 == ASV_BITS_FREE && i2 != i1) asv_bits_claim(b, i2, tab);
            if (m3 == ASV_BITS_FREE && i3 != i2) asv_bits_claim(b, i3, tab);
            pend |= 1u << k;
        } else {
            *q = make_int4((int)asv_bit(m0), (int)asv_bit(m1), (int)asv_bit(m2), (int)asv_bit(m3));
        }
    }
    asv_cp_async_wait();                                       // the claimed labels' rows
    __syncthreads();
    const int T = b.tcount;
    if (T > ASV_BITS_MAXT) {
        asv_bits_reset(b, T);
        __syncthreads();
        if (tid == 0) b.tcount = 0;
        __syncthreads();
        return false;
    }
    if (SUMS)
        for (int i = tid; i < ASV_ACC_WORDS; i += ASV_JFA_THREADS) acc[i] = 0u;
    while (pend) {
        int4 *q = (int4 *)(flab + 4 * (tid + ASV_JFA_THREADS * (__ffs(pend) - 1)));
        pend &= pend - 1;
        const int4 v = *q;
        const unsigned m0 = b.map8[asv_bits_slot(v.x)], m1 = b.map8[asv_bits_slot(v.y)],
                       m2 = b.map8[asv_bits_slot(v.z)], m3 = b.map8[asv_bits_slot(v.w)];
        *q = make_int4((int)asv_bit(m0), (int)asv_bit(m1), (int)asv_bit(m2), (int)asv_bit(m3));
    }
    if (tid < 32) asv_bits_coefs(b, T, (float)(tx0 + 8), (float)(ty0 + 8), (float)zc + 0.5f, wmax, ratio);
    __syncthreads();
    // the numbers are read no more: unnumbered again for the next sub-tile
    // (which starts after the barrier at the end)
    asv_bits_reset(b, T);
    if (tid == 0) b.tcount = 0;

    // the chain walk of this thread's column
    const unsigned *f0 = (const unsigned *)flab + ly * FW + lx + (G::AL - S);  // candidate (x - S, y - S) of slot 0
    auto smask = [&](const unsigned *f) -> unsigned {             // a slice's 9 candidates
        unsigned m = 0;
#pragma unroll
        for (int a = 0; a < 3; a++)
#pragma unroll
            for (int c = 0; c < 3; c++) m |= f[a * S * FW + c * S];
        return m;
    };
    const float2 uv = make_float2((float)lx - 7.5f, (float)ly - 7.5f);
    const float mg0 = b.margin[0], mg1 = b.margin[1];
    const float mgl = b.magic[0], mga = b.magic[1], mgb = b.magic[2];
    const unsigned m_zero = brk ? smask(f0 + zslot * FP) : 0u, m_last = brk ? smask(f0 + lslot * FP) : 0u;
    unsigned mm = smask(f0), mc = smask(f0 + FP);
    // centroid sums (last pass of an iteration): the thread's current run of
    // equal labels along its column, flushed into the sub-tile's table when
    // the label changes and at the end; the table goes to the global sums
    // once per sub-tile (centroids.vs:19-54; label -1 counts in slot Kp)
    int run_e = -1;
    const unsigned lxy = (unsigned)lx | ((unsigned)ly << 16);
    unsigned run_z = 0u, run_la = 0u, run_bn = 0u;            // L | a << 16, b | count << 16 (16 x 255 < 2^16)
    const unsigned *fn = f0 + 2 * FP;                         // the next slot
    const unsigned *lab32 = (const unsigned *)lab;
    unsigned ends = brk, ca = __ldg(lab32 + (b.slot[1].x + col)), cb = __ldg(lab32 + (b.slot[2].x + col));
    // positions left to the shader's arithmetic: all of them without scores
    unsigned slow = mg0 < 1e30f ? 0u : (1u << n) - 1u;
    // a position's label out and, in a summing pass, into the run
    auto put = [&](int j, const int4 at, unsigned c4, int bt) {
        const int label = bt >= 0 ? b.tlab[bt] : -1;
        if (valid) out[at.x + col] = label;                   // (a slow position's is replaced below)
        if (SUMS && valid && !((slow >> j) & 1u)) {
            const int e = bt >= 0 ? bt : ASV_BITS_MAXT;
            if (e != run_e) {
                if (run_e >= 0) asv_run_flush(acc + ASV_ACC_ROW * (ASV_ACC_COPIES * run_e + lane % ASV_ACC_COPIES), run_z, run_la, run_bn, lxy);
                run_e = e;
                run_z = run_la = run_bn = 0u;
            }
            run_z += (unsigned)at.z;
            run_la += __byte_perm(c4, 0u, 0x4140);
            run_bn += __byte_perm(c4, 1u, 0x7472);            // bytes (b, 0, 1, 0)
        }
    };
    // Two positions at a time: their candidates are mostly the same, so a
    // label's fourteen coefficients are read once for both.  (What bounds the
    // passes is the shared-memory data path, 85 % busy with one position at a
    // time, most of it with coefficients.)
    for (int j = 0; j < n; j += 2, fn += 2 * FP, ends >>= 2) {
        const int4 at0 = b.slot[j + 1], at1 = b.slot[j + 2];
        const unsigned c0 = ca, c1 = cb;
        ca = __ldg(lab32 + (b.slot[j + 3].x + col));          // the next pair's (past the last one: unused)
        cb = __ldg(lab32 + (b.slot[j + 4].x + col));
        const bool end0 = ends & 1u, end1 = ends & 2u;        // the chain ends here and another one starts:
        const unsigned mx = smask(fn), my = smask(fn + FP);   // the next slot is its centre, else this one's plus
        const unsigned ma = mm | mc | (end0 ? m_last : mx);
        const unsigned mb = j + 1 < n ? (end0 ? m_zero : mc) | mx | (end1 ? m_last : my) : 0u;
        mm = end1 ? m_zero : mx;
        mc = my;
        int bta = 31 - __clz((int)ma), btb = 31 - __clz((int)mb);   // the only candidate, or -1
        const bool twoa = ma & (ma - 1), twob = mb & (mb - 1);
        unsigned rest = (twoa ? ma : 0u) | (twob ? mb : 0u);
        if (rest) {
            const float wa = __int_as_float(at0.y), wb = __int_as_float(at1.y);
            // bytes to floats: 2^23 + byte, minus 2^23 + the middle colour
            const float la = __uint_as_float(__byte_perm(c0, 0x4b000000u, 0x7650)) - mgl;
            const float aa = __uint_as_float(__byte_perm(c0, 0x4b000000u, 0x7651)) - mga;
            const float ba = __uint_as_float(__byte_perm(c0, 0x4b000000u, 0x7652)) - mgb;
            const float lb = __uint_as_float(__byte_perm(c1, 0x4b000000u, 0x7650)) - mgl;
            const float ab = __uint_as_float(__byte_perm(c1, 0x4b000000u, 0x7651)) - mga;
            const float bb = __uint_as_float(__byte_perm(c1, 0x4b000000u, 0x7652)) - mgb;
            float besta = 3e38f, seca = 3e38f, bestb = 3e38f, secb = 3e38f;
            do {
                const int t = 31 - __clz((int)rest);
                const unsigned bit = 1u << t;
                rest ^= bit;
                const float4 *e = b.eco + ASV_ECO_ROW * t;
                const float4 e0 = e[0], e1 = e[1], e2 = e[2];
                const float2 e3 = *(const float2 *)(e + 3);
                const float2 g = __ffma2_rn(make_float2(e0.z, e0.w), uv, make_float2(e0.x, e0.y));
                const float k = __fmaf_rn(g.y, uv.y, __fmaf_rn(__fmaf_rn(e1.w, uv.y, g.x), uv.x, e2.y));
                const float h = __fmaf_rn(e1.y, uv.y, __fmaf_rn(e1.x, uv.x, e2.x));
                if (ma & bit) {
                    float p = fmaxf(__fmaf_rn(__fmaf_rn(e1.z, wa, h), wa, k), e2.z);
                    p = __fmaf_rn(e3.y, ba, __fmaf_rn(e3.x, aa, __fmaf_rn(e2.w, la, p)));
                    seca = fminf(seca, fmaxf(besta, p));
                    bta = p < besta ? t : bta;
                    besta = fminf(besta, p);
                }
                if (mb & bit) {
                    float p = fmaxf(__fmaf_rn(__fmaf_rn(e1.z, wb, h), wb, k), e2.z);
                    p = __fmaf_rn(e3.y, bb, __fmaf_rn(e3.x, ab, __fmaf_rn(e2.w, lb, p)));
                    secb = fminf(secb, fmaxf(bestb, p));
                    btb = p < bestb ? t : btb;
                    bestb = fminf(bestb, p);
                }
            } while (rest);
            const float qa = __fmaf_rn(la, la, __fmaf_rn(aa, aa, ba * ba)), qb = __fmaf_rn(lb, lb, __fmaf_rn(ab, ab, bb * bb));
            // (a position whose only candidate also came by keeps it: second stays 3e38)
            if (twoa && !(seca - besta > __fmaf_rn(16.0f * ASV_EPS, seca + besta, __fmaf_rn(mg1, qa, mg0)))) slow |= 1u << j;
            if (twob && !(secb - bestb > __fmaf_rn(16.0f * ASV_EPS, secb + bestb, __fmaf_rn(mg1, qb, mg0)))) slow |= 2u << j;
        }
        put(j, at0, c0, bta);
        if (j + 1 < n) put(j + 1, at1, c1, btb);
    }
    while (slow && valid) {
        const int j = __ffs(slow) - 1;
        slow &= slow - 1;
        const unsigned *fc = f0 + (j + 1) * FP;
        const unsigned *fm = j > 0 && ((brk >> (j - 1)) & 1u) ? f0 + zslot * FP : fc - FP;   // minus slice
        const unsigned *fp = (brk >> j) & 1u ? f0 + lslot * FP : fc + FP;
        const int4 at = b.slot[j + 1];
        const unsigned c4 = __ldg(lab32 + (at.x + col));
        const int bt = asv_bits_exact<S>(smask(fm) | smask(fc) | smask(fp), fc, fm, fp, b, tab, x, y, at.z >> 1, c4, ratio);
        out[at.x + col] = bt >= 0 ? b.tlab[bt] : -1;
        if (SUMS)
            asv_run_flush(acc + ASV_ACC_ROW * ASV_ACC_COPIES * (bt >= 0 ? bt : ASV_BITS_MAXT), (unsigned)at.z, __byte_perm(c4, 0u, 0x4140),
                          __byte_perm(c4, 1u, 0x7472), lxy);
    }
    if (SUMS) {
        // the runs left at the end (straight into the copies: grouping a
        // warp's lanes by entry first took 2 % of the 64x48x12 clip's loop)
        if (run_e >= 0)
            asv_run_flush(acc + ASV_ACC_ROW * (ASV_ACC_COPIES * run_e + lane % ASV_ACC_COPIES), run_z, run_la, run_bn, lxy);
        __syncthreads();
        for (int i = tid; i < (T + 1) * 8; i += ASV_JFA_THREADS) {
            const int e = i >> 3, k = i & 7;
            const int ent = e < T ? e : ASV_BITS_MAXT;           // the -1 entry after the T labels
            if (k == 7) continue;
            unsigned cnt = 0u, v = 0u;
#pragma unroll
            for (int c = 0; c < ASV_ACC_COPIES; c++) {
                const unsigned *a = acc + ASV_ACC_ROW * (ASV_ACC_COPIES * ent + c);
                cnt += a[1] >> 20;
                v += k < 2 ? (a[0] >> (16 * k)) & 0xffffu : (k == 4 ? a[1] & 0xfffffu : (k == 3 ? 0u : a[k == 2 ? 2 : k - 2]));
            }
            if (!cnt) continue;
            if (k < 2) v = 2u * v + cnt * (2u * (unsigned)(k ? ty0 : tx0) + 1u);   // 2 x + 1 = 2 (tx0 + column) + 1
            if (k == 3) v = cnt;
            atomicAdd(sums + 8ull * (slot0 + (ent < ASV_BITS_MAXT ? b.tlab[ent] : Kp)) + k, (unsigned long long)v);
        }
    }
    __syncthreads();                                          // the footprint and table are reused
    return true;
}

// One tile of a pass: bit-set form by sub-tiles (ST the pass's step, 1 to 6),
// else (ST = ASV_JFA_LIST: larger steps; or for a sub-tile whose footprint
// holds too many labels) the list form.
#define ASV_JFA_LIST 7
template <int ST, bool SUMS>
__device__ __forceinline__ void asv_jfa_tile(const int32_t *in, int32_t *__restrict__ out,
                                             const uchar4 *__restrict__ lab, const float4 *__restrict__ tab,
                                             unsigned long long *__restrict__ sums, int slot0, int W, int H, int D,
                                             int Kp, int tx0, int ty0, int p0, int zrun, int depth, int step,
                                             float ratio, unsigned char *smem)
{
    const int n = min(zrun, D - p0);
    const int lx = threadIdx.x % ASV_TILE_X, ly = threadIdx.x / ASV_TILE_X;
    const int gx = tx0 + lx, gy = ty0 + ly;
    const bool valid = gx < W && gy < H;                       // block-uniform loop: every lane runs the tile
    // `todo` has a bit for each position of the tile (32 at a time).  A round
    // cuts the positions to do in sub-tiles of `cap`; the sub-tiles whose
    // labels do not fit go to the next round, half as deep, and below four
    // positions to one inlined copy of the list form.
    for (int c0 = 0; c0 < n; c0 += 32) {
        const int nc = min(n - c0, 32), pc = p0 + c0;
        unsigned todo = 0xffffffffu >> (32 - nc);
        int cap = SUMS ? min(depth, 15) : depth;               // 15: asv_run_words
        if constexpr (ST < ASV_JFA_LIST) {
            cap = Kp > ASV_BITS_MAXKP ? 0 : min(cap, AsvBitsGeo<ST>::SUB);
            while (cap >= 4 && todo) {
                unsigned fail = 0u;
                do {
                    const int q = __ffs(todo) - 1;
                    const unsigned past = ~(todo >> q);
                    const int m = min(cap, past ? __ffs(past) - 1 : 32);
                    const unsigned bits = (0xffffffffu >> (32 - m)) << q;
                    todo &= ~bits;
                    if (!asv_jfa_bits_sub<ST, SUMS>(in, out, lab, tab, sums, slot0, W, H, D, Kp, tx0, ty0, pc + q, m,
                                                    ratio, smem))
                        fail |= bits;
                } while (todo);
                todo = fail;
                cap = (cap + 1) >> 1;
            }
        }
        while (todo) {                                         // runs of positions left
            const int q = __ffs(todo) - 1;
            const unsigned past = ~(todo >> q);
            const int m = past ? __ffs(past) - 1 : 32;
            todo &= ~((0xffffffffu >> (32 - m)) << q);
            if constexpr (ST == ASV_JFA_LIST)
                asv_jfa_run_far(in, out, lab, tab, W, H, D, Kp, min(gx, W - 1), min(gy, H - 1), pc + q, m, step, ratio,
                                (asv_list_t *)smem + threadIdx.x, valid);
            else
                asv_jfa_run<SUMS>(in, out, lab, tab, sums, slot0, W, H, D, Kp, min(gx, W - 1), min(gy, H - 1), pc + q, m,
                                  step, ratio, (asv_list_t *)smem + threadIdx.x, valid);
            __syncthreads();                                   // the list rows alias the footprint
        }
    }
}

__device__ __forceinline__ void asv_jfa_smem_init(AsvBitsShared &b)
{
    for (int i = threadIdx.x; i < ASV_BITS_MAXKP / 32; i += blockDim.x) b.claim[i] = 0u;
    for (int i = threadIdx.x; i < ASV_BITS_MAXKP / 4; i += blockDim.x) ((unsigned *)b.map8)[i] = 0xffffffffu;
    if (threadIdx.x == 0) {
        b.tcount = 0;
        b.map8[ASV_BITS_MAXKP] = ASV_BITS_NOLABEL;
    }
    __syncthreads();
}

// A pass over the tiles (ASV_TILE_X x ASV_TILE_Y columns x S.zrun chain
// positions) of the segments whose step in this pass is ST (ASV_JFA_LIST: larger
// than 6) and, with SUMS, whose last pass it is (always of step 1); a pass of
// segments of different steps is a launch of each.  A variant holds just the
// code of its pass: against one kernel for all, which kept the registers of the
// worst, the 240x160x30 clip with its full ladder took 3.96 instead of 4.39 ms,
// the 640x480x60 one 16.1 instead of 16.7.
template <int ST, bool SUMS>
__global__ void __launch_bounds__(ASV_JFA_THREADS, 4) k_jfa(AsvDev d, int pass,
                                                         const int32_t *in,
                                                         int32_t *__restrict__ out)
{
    extern __shared__ __align__(16) unsigned char asv_jfa_smem[];
    if constexpr (ST < ASV_JFA_LIST) asv_jfa_smem_init(*(AsvBitsShared *)(asv_jfa_smem + AsvBitsGeo<ST>::AREA));
    if constexpr (SUMS) asv_follow();                         // (the seeds' kernels have few blocks)
    else asv_follow_wait();
    for (int t = blockIdx.x; t < d.total_tiles; t += gridDim.x) {
        const int si = asv_find_seg(d.tile_prefix, d.nseg, t);
        const SegDesc &S = d.segs[si];
        if (pass >= S.npass) continue;
        const int step = S.steps[pass];
        if (min(step, ASV_JFA_LIST) != ST || (ST == 1 && (pass == S.npass - 1) != SUMS)) continue;
        const int lt = t - d.tile_prefix[si];
        const int rest = asv_quotient(lt, S.inv_tiles_x), tx = lt - rest * S.tiles_x;
        const int tz = asv_quotient(rest, S.inv_tiles_y), ty = rest - tz * S.tiles_y, p0 = tz * S.zrun;
        asv_jfa_tile<ST, SUMS>(in + S.vox_off, out + S.vox_off, d.lab + S.vox_off, d.jtab + 3 * S.seed_off,
                               SUMS ? d.sums : nullptr, S.seed_off, S.W, S.H, S.D, S.Kp, tx * ASV_TILE_X, ty * ASV_TILE_Y,
                               p0, S.zrun, S.depth[pass], ST < ASV_JFA_LIST ? ST : step, S.ratio[pass], asv_jfa_smem);
    }
}

// ---------------------------------------------------------------------------
// The first pass of a Lloyd iteration from the seeds.  Its input is the drawn
// seed volume: -1 everywhere but at the seed voxels, each holding the seed that
// won its voxel.  At step 1 only the up to 27 voxels around a drawn seed see
// any label, so a thread takes one drawn seed and one of them and gathers that
// voxel's 27 candidates by the shader's own rule (order and clamping of k_jfa's
// list form, strict '<' from 1e8, flood.gs:63, :95-99); nearly all are -1, and
// a candidate is evaluated once per run of equal ids.  Where two seeds reach
// one voxel each of their threads finds the same winner, and the winner's
// thread writes it and lists the voxel for the second pass.  (Two kernels
// before, a 64-bit atomicMin of keys and a take: 5.1 + 5.2 us a pass on the
// 320x240x85 clip.)  The output volume is filled with -1 first.  stale: the seed
// table was replaced after the draw, and only records that stand at their
// seed's position count.
// ---------------------------------------------------------------------------

__global__ void __launch_bounds__(256) k_jfa_first(AsvDev d, bool stale)
{
    asv_follow();
    const unsigned t = blockIdx.x * blockDim.x + threadIdx.x;
    const int g = (int)(t / 27u), o = (int)(t - 27u * (unsigned)g);
    bool won = false;
    int si = 0, label = 0;
    long long vl = 0;
    if (g < d.total_seeds) {
        int i;
        si = asv_seed_seg(d, g, i);
        const SegDesc &S = d.segs[si];
        const float4 p = d.pos[g];
        const int W = S.W, H = S.H, D = S.D;
        const int32_t *in = d.drawn + S.vox_off;
        int sx = -1, sy = -1, sz = -1;
        if (i < S.Kp && p.x >= 0.0f && p.y >= 0.0f && p.z >= 0.0f) { sx = (int)p.x; sy = (int)p.y; sz = (int)p.z; }   // as the draw
        const bool inside = sx >= 0 && sx < W && sy < H && sz < D;
        const int x = sx + (o % 3 - 1), y = sy + ((o / 3) % 3 - 1), z = sz + (o / 9 - 1);
        if (inside && x >= 0 && x < W && y >= 0 && y < H && z >= 0 && z < D &&
            in[((long long)sz * H + sy) * W + sx] == i) {                          // the seed won its voxel
            vl = ((long long)z * H + y) * W + x;
            const uchar4 c = __ldg(d.lab + S.vox_off + vl);
            const float2 vxy = make_float2((float)x + 0.5f, (float)y + 0.5f);
            const float2 vzl = make_float2((float)z + 0.5f, (float)c.x), vab = make_float2((float)c.y, (float)c.z);
            const int zs[3] = { z, max(z - 1, 0), min(z + 1, D - 1) };
            const int ys[3] = { max(y - 1, 0), y, min(y + 1, H - 1) };
            const int xs[3] = { max(x - 1, 0), x, min(x + 1, W - 1) };
            int32_t l[27];
#pragma unroll
            for (int k = 0; k < 27; k++)
                l[k] = in[((long long)zs[k / 9] * H + ys[(k / 3) % 3]) * W + xs[k % 3]];
            if (stale) {
#pragma unroll
                for (int k = 0; k < 27; k++) {
                    if (l[k] < 0 || l[k] >= S.Kp) { l[k] = -1; continue; }
                    const float4 q = d.pos[S.seed_off + l[k]];
                    if ((int)q.x != xs[k % 3] || (int)q.y != ys[(k / 3) % 3] || (int)q.z != zs[k / 9]) l[k] = -1;
                }
            }
            float mind = 100000000.0f;
            int best = -1, prev = -1;
#pragma unroll
            for (int k = 0; k < 27; k++)
                if (l[k] >= 0 && l[k] != prev) {
                    prev = l[k];
                    const float dist = asv_jfa_dist(d.jtab + 3 * S.seed_off, l[k], vxy, vzl, vab, S.ratio[0]);
                    if (dist < mind) { mind = dist; best = l[k]; }
                }
            won = best == i;
            label = i;
            if (won) d.labB[S.vox_off + vl] = i;
        }
    }
    const unsigned m = __ballot_sync(FULL, won);                                   // one addition per warp
    if (!m) return;
    const int lane = threadIdx.x & 31;
    unsigned at = 0;
    if (lane == __ffs(m) - 1) at = atomicAdd(d.tcount, (unsigned)__popc(m));
    at = __shfl_sync(FULL, at, __ffs(m) - 1);
    if (won) d.tlist[at + __popc(m & ((1u << lane) - 1u))] = asv_entry(si, (int)vl, label);
}

// ---------------------------------------------------------------------------
// The second pass (step s = steps[1]) as a scatter: its input, the first
// pass's output, is labelled only at the voxels listed in tlist.  A voxel v
// sees the label at u through offset o when clamp(v + o*s) == u along every
// axis; per axis those v form a range (one voxel inside the volume, up to
// s + 1 next to an edge, where several offsets clamp onto u).  Each (u, o)
// thread visits that box and puts its label into the output, all -1 before, by
// compare-and-swap.  Where a label stands already the two are compared by the
// gather's rule: the least distance, and of equal ones the label met first in
// the shader's order.  Blocks hold one offset of neighbouring entries, whose
// voxels adjoin (an entry's 27 offsets side by side: 36 us a pass on the
// 320x240x85 clip, so 25; with the registers held to 64, four blocks per SM
// instead of three, and the label in the list 22).  Before, 64-bit keys of
// distance, rank and label by atomicMin and a kernel to take the labels out, 8
// bytes more a voxel: 15 iterations of that clip took 9.22 ms, so 8.95, 4 of a
// 64x48x12 one 0.326, so 0.302.
// ---------------------------------------------------------------------------
__device__ __forceinline__ void asv_axis_sources(int u, int o, int s, int n, int &lo, int &hi)
{
    if (o == 0) { lo = hi = u; return; }
    if (o < 0) {                              // clamp(v - s) == u
        if (u > 0) lo = hi = u + s; else { lo = 0; hi = s; }
    } else {                                  // clamp(v + s) == u
        if (u < n - 1) lo = hi = u - s; else { lo = n - 1 - s; hi = n - 1; }
    }
    lo = max(lo, 0);
    hi = min(hi, n - 1);                      // empty when lo > hi
}

// whether voxel (x, y, z) meets label a before label b among its candidates, in the
// shader's order (slices z, z-s, z+s; rows and columns from - to +, clamped)
__device__ __forceinline__ bool asv_met_before(const int32_t *in, int W, int H, int D, int x, int y, int z,
                                               int s, int a, int b)
{
    unsigned ma = 0, mb = 0;
#pragma unroll 1
    for (int i = 0; i < 3; i++) {
        const int zz = i == 0 ? z : (i == 1 ? max(z - s, 0) : min(z + s, D - 1));
#pragma unroll 1
        for (int j = 0; j < 3; j++) {
            const int yy = j == 0 ? max(y - s, 0) : (j == 1 ? y : min(y + s, H - 1)), k = 9 * i + 3 * j;
            const int32_t *row = in + ((long long)zz * H + yy) * W;
            const int l0 = row[max(x - s, 0)], l1 = row[x], l2 = row[min(x + s, W - 1)];
            ma |= (l0 == a ? 1u << k : 0u) | (l1 == a ? 2u << k : 0u) | (l2 == a ? 4u << k : 0u);
            mb |= (l0 == b ? 1u << k : 0u) | (l1 == b ? 2u << k : 0u) | (l2 == b ? 4u << k : 0u);
        }
    }
    return __ffs(ma) < __ffs(mb);       // both are among them
}

// label's claim on one voxel of an entry's box
__device__ __forceinline__ void asv_second_voxel(const AsvDev &d, const SegDesc &S, int label, int x, int y, int z, int s)
{
    const long long v = S.vox_off + ((long long)z * S.H + y) * S.W + x;
    const uchar4 c = __ldg(d.lab + v);
    const float2 vxy = make_float2((float)x + 0.5f, (float)y + 0.5f), vzl = make_float2((float)z + 0.5f, (float)c.x);
    const float2 vab = make_float2((float)c.y, (float)c.z);
    const float4 *tab = d.jtab + 3 * S.seed_off;
    const float dist = asv_jfa_dist(tab, label, vxy, vzl, vab, S.ratio[1]);
    if (!(dist < 100000000.0f)) return;
    int old = -1;
    for (;;) {                          // the voxel's label only gets better: at most its 27 candidates
        const int was = atomicCAS(d.labA + v, old, label);
        if (was == old || was == label) return;
        old = was;
        const float od = asv_jfa_dist(tab, old, vxy, vzl, vab, S.ratio[1]);
        if (od < dist) return;
        if (od == dist && asv_met_before(d.labB + S.vox_off, S.W, S.H, S.D, x, y, z, s, old, label)) return;
    }
}

// A thread per listed voxel and offset.  Inside the volume the box is one
// voxel; next to an edge it has s + 1 to (s + 1)^3 (1728 at step 11), and one
// thread alone made the kernel as long as its largest box (26 to 36 us): boxes
// of more than one voxel are walked by the whole warp, one after another.
// undraw: the threads also take the drawn seeds out of their volume again, so
// that it is all -1 for the next draw without a fill (the first pass has read it).
__global__ void __launch_bounds__(256, 4) k_jfa_second(AsvDev d, bool undraw)
{
    asv_follow_wait();
    const unsigned group = blockIdx.x / 27;
    const int o = (int)(blockIdx.x - 27 * group);              // one offset per block: neighbouring entries' targets
    const long long e = (long long)group * 256 + threadIdx.x, t = (long long)blockIdx.x * 256 + threadIdx.x;   // adjoin
    if (undraw && t < d.total_seeds) {
        int i;
        const SegDesc &S = d.segs[asv_seed_seg(d, (int)t, i)];
        const float4 p = d.pos[t];
        if (i < S.Kp && p.x >= 0.0f && p.y >= 0.0f && p.z >= 0.0f && (int)p.x < S.W && (int)p.y < S.H && (int)p.z < S.D)
            d.drawn[S.vox_off + ((long long)(int)p.z * S.H + (int)p.y) * S.W + (int)p.x] = -1;
    }
    int si = 0, label = 0;
    int x0 = 0, y0 = 0, z0 = 0, nx = 0, ny = 0, nz = 0;
    const asv_entry_t ent = e < 27LL * d.total_seeds ? d.tlist[e] : 0ull;             // asked for beside their number
    if (e < *d.tcount) {
        si = asv_entry_seg(ent);
        const int ul = asv_entry_voxel(ent);
        const SegDesc &S = d.segs[si];
        const int s = S.steps[1];
        const int row = ul / S.W;
        const int ux = ul - row * S.W, uz = row / S.H, uy = row - uz * S.H;
        int x1, y1, z1;
        asv_axis_sources(ux, o % 3 - 1, s, S.W, x0, x1);
        asv_axis_sources(uy, (o / 3) % 3 - 1, s, S.H, y0, y1);
        asv_axis_sources(uz, o / 9 - 1, s, S.D, z0, z1);
        nx = x1 - x0 + 1; ny = y1 - y0 + 1; nz = z1 - z0 + 1;
        if (nx <= 0 || ny <= 0 || nz <= 0) nx = 0;
        else {
            label = asv_entry_label(ent);
            if (nx * ny * nz == 1) {
                asv_second_voxel(d, S, label, x0, y0, z0, s);
                nx = 0;
            }
        }
    }
    unsigned big = __ballot_sync(FULL, nx > 0);
    const int lane = threadIdx.x & 31;
    while (big) {
        const int from = __ffs(big) - 1;
        big &= big - 1;
        const int bsi = __shfl_sync(FULL, si, from), bl = __shfl_sync(FULL, label, from);
        const int bx = __shfl_sync(FULL, x0, from), by = __shfl_sync(FULL, y0, from), bz = __shfl_sync(FULL, z0, from);
        const int bnx = __shfl_sync(FULL, nx, from), bny = __shfl_sync(FULL, ny, from), bnz = __shfl_sync(FULL, nz, from);
        const SegDesc &S = d.segs[bsi];
        for (int k = lane; k < bnx * bny * bnz; k += 32) {
            const int r = k / bnx;
            asv_second_voxel(d, S, bl, bx + k - r * bnx, by + r % bny, bz + r / bny, S.steps[1]);
        }
    }
}

// Before a single pass over a caller's labels: those outside [0, Kp) become -1, as
// the passes' own are, and the pass's descriptor goes to *out.  Kp is the segment's
// on the device, where a streaming window's seeds are counted (k_stream_compose).
__global__ void k_pass_prepare(int32_t *lbl, const __grid_constant__ SegDesc one, const SegDesc *seg, SegDesc *out)
{
    asv_follow();                                             // (the pass may start beside it)
    const long long v = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const int Kp = seg->Kp;
    if (v < one.nvox && (unsigned)lbl[v] >= (unsigned)Kp) lbl[v] = -1;
    if (blockIdx.x) return;
    for (int i = threadIdx.x; i < (int)(sizeof(SegDesc) / 4); i += blockDim.x)
        ((int *)out)[i] = i == (int)(offsetof(SegDesc, Kp) / 4) ? Kp : ((const int *)&one)[i];
}

// ---------------------------------------------------------------------------
// Centroid sums (centroids.vs:19-54): per label slot (label -1 -> slot Kp)
// sum(2x+1), sum(2y+1), sum(2z+1), count, sum L, a, b -- exact integers.
// Lanes with the same label are reduced in the warp, then one u64 atomic per
// group and component.
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(256) k_centroids(AsvDev d)
{
    int si = asv_find_seg(d.chunk_prefix, d.nseg, blockIdx.x);
    const SegDesc &S = d.segs[si];
    const int W = S.W, H = S.H;
    const int32_t *lbl = (S.final_buf ? d.labB : d.labA) + S.vox_off;
    const uchar4 *lab = d.lab + S.vox_off;
    unsigned long long *sums = d.sums + 8ull * S.seed_off;
    long long base = (long long)(blockIdx.x - d.chunk_prefix[si]) * ASV_CHUNK;
    const int lane = threadIdx.x & 31;
    for (int i = 0; i < ASV_CHUNK / 256; i++) {
        long long v = base + i * 256 + threadIdx.x;
        int key = -1;
        unsigned q[7] = { 0, 0, 0, 0, 0, 0, 0 };
        if (v < S.nvox) {
            int l = __ldg(lbl + v);
            key = (l < 0 || l >= S.Kp) ? S.Kp : l;   // out-of-range ids (never produced) count as -1
            int x = (int)(v % W);
            long long r = v / W;
            int y = (int)(r % H), z = (int)(r / H);
            uchar4 c = __ldg(lab + v);
            q[0] = 2 * x + 1; q[1] = 2 * y + 1; q[2] = 2 * z + 1; q[3] = 1;
            q[4] = c.x; q[5] = c.y; q[6] = c.z;
        }
        unsigned grp = __match_any_sync(FULL, key);
        unsigned s[7];
#pragma unroll
        for (int k = 0; k < 7; k++) s[k] = __reduce_add_sync(grp, q[k]);
        if (key >= 0 && lane == __ffs(grp) - 1) {
            unsigned long long *dst = sums + 8ull * key;
#pragma unroll
            for (int k = 0; k < 7; k++) atomicAdd(dst + k, (unsigned long long)s[k]);
        }
    }
}

__global__ void k_finalize(AsvDev d)
{
    int g = blockIdx.x * blockDim.x + threadIdx.x;
    if (g >= d.total_seeds) return;
    int id;
    int si = asv_seed_seg(d, g, id);
    const SegDesc &S = d.segs[si];
    if (id >= S.Kp) return;
    float p[3], c[3];
    asv_reseed(d, S, id, p, c);
    d.pos[g] = make_float4(p[0], p[1], p[2], (float)id);
    d.slab[g] = make_float4(c[0], c[1], c[2], 0.0f);
}

// ---------------------------------------------------------------------------
// Post-processing (GPU-AS/Image.cpp:1579-1778).
//   k_post_stats: one block per segment -- dead seeds, alive ranks, the
//     relabel LUT of the <= 3 dead case, mode and -1 flags.
//   k_post_chunk_max / k_post_prefix / k_post_apply: forward fills of the
//     reference's raster loops as a max-scan of "source" voxel indices.
// The post-processed labels go to the buffer the last pass did not write.
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(1024) k_post_stats(AsvDev d)
{
    asv_follow();
    const int si = blockIdx.x;
    const SegDesc &S = d.segs[si];
    const int Kp = S.Kp;
    const unsigned long long *sums = d.sums + 8ull * S.seed_off;
    int *rank = d.rank + S.seed_off;
    int *rec = d.post + si * ASV_POST_WORDS;
    __shared__ int warp_tot[32];
    __shared__ int carry;
    if (threadIdx.x == 0) carry = 0;
    __syncthreads();
    // alive rank: exclusive scan of (count >= 1) in seed order (:1603-1618)
    for (int b0 = 0; b0 < Kp; b0 += blockDim.x) {
        int i = b0 + threadIdx.x;
        int alive = (i < Kp && sums[8ull * i + 3] >= 1) ? 1 : 0;
        unsigned bal = __ballot_sync(FULL, alive);
        int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
        int pre = __popc(bal & ((1u << lane) - 1u));
        if (lane == 0) warp_tot[w] = __popc(bal);
        __syncthreads();
        if (threadIdx.x < 32) {
            int v = threadIdx.x < (blockDim.x >> 5) ? warp_tot[threadIdx.x] : 0;
            int incl = v;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                int n = __shfl_up_sync(FULL, incl, o);
                if (threadIdx.x >= o) incl += n;
            }
            warp_tot[threadIdx.x] = incl - v;   // exclusive
        }
        __syncthreads();
        if (i < Kp) {
            const int live_before = carry + warp_tot[w] + pre;
            rank[i] = alive ? live_before : -1;
            const int dead_before = i - live_before;        // the first four dead seeds, in order
            if (!alive && dead_before < 4) rec[POST_DEAD0 + dead_before] = i;
        }
        __syncthreads();
        if (threadIdx.x == blockDim.x - 1) carry += warp_tot[w] + pre + alive;
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        int valid = carry, dead = Kp - valid;
        long long negc = (long long)sums[8ull * Kp + 3];
        rec[POST_DEAD] = dead;
        rec[POST_NEG] = negc > 0x7fffffffLL ? 0x7fffffff : (int)negc;
        rec[POST_VALID] = valid;
        rec[POST_INVALID] = negc > 0 ? 1 : 0;
        int mode = dead == 0 ? 0 : (dead <= 3 ? 1 : 2);
        rec[POST_MODE] = mode;
        const int32_t *lbl = (S.final_buf ? d.labB : d.labA) + S.vox_off;
        int l0 = lbl[0];
        rec[POST_L0] = l0;
        rec[POST_M0] = (l0 >= 0 && l0 < Kp && rank[l0] >= 0) ? rank[l0] : 0;
    }
}

// relabelled value of a raw label before the fills (the <= 3 dead relabel
// of label_replace.gs:26-29 applied in order, :1652-1673)
__device__ __forceinline__ int asv_relabel(const int *rec, int Kp, int l)
{
    if (rec[POST_MODE] != 1 || l < 0) return l;
    int last = Kp;
    for (int k = 0; k < rec[POST_DEAD]; k++) {
        last -= 1;
        if (l == last) l = rec[POST_DEAD0 + k];
    }
    return l;
}

// source index of voxel v for the forward fill, or -1
__device__ __forceinline__ long long asv_fill_src(const int *rec, int Kp, long long v, int l)
{
    if (rec[POST_MODE] == 2) {                                  // :1738-1746
        if (v == 0) return 0;
        return (l != rec[POST_L0] && l != -1) ? v : -1;
    }
    int r = asv_relabel(rec, Kp, l);                            // :1763-1775
    if (v == 0) return 0;
    return r != -1 ? v : -1;
}

__device__ __forceinline__ bool asv_needs_scan(const int *rec)
{
    return rec[POST_MODE] == 2 || rec[POST_INVALID] != 0;
}

__global__ void __launch_bounds__(256) k_post_chunk_max(AsvDev d)
{
    asv_follow();
    int si = asv_find_seg(d.chunk_prefix, d.nseg, blockIdx.x);
    const SegDesc &S = d.segs[si];
    const int *rec = d.post + si * ASV_POST_WORDS;
    if (!asv_needs_scan(rec)) return;
    const int32_t *lbl = (S.final_buf ? d.labB : d.labA) + S.vox_off;
    long long base = (long long)(blockIdx.x - d.chunk_prefix[si]) * ASV_CHUNK;
    long long m = -1;
    for (int i = 0; i < ASV_CHUNK / 256; i++) {
        long long v = base + i * 256 + threadIdx.x;
        if (v < S.nvox) { long long s = asv_fill_src(rec, S.Kp, v, lbl[v]); if (s > m) m = s; }
    }
#pragma unroll
    for (int o = 16; o; o >>= 1) { long long n = __shfl_xor_sync(FULL, m, o); if (n > m) m = n; }
    __shared__ long long wm[8];
    if ((threadIdx.x & 31) == 0) wm[threadIdx.x >> 5] = m;
    __syncthreads();
    if (threadIdx.x == 0) {
        long long r = wm[0];
        for (int k = 1; k < 8; k++) if (wm[k] > r) r = wm[k];
        // store +1 so that a chunk without source is 0
        d.scan[blockIdx.x] = (int)(r + 1);
    }
}

// exclusive max-scan of the chunk maxima within each segment (1 block / segment)
__global__ void __launch_bounds__(1024) k_post_prefix(AsvDev d)
{
    asv_follow();
    int si = blockIdx.x;
    const int *rec = d.post + si * ASV_POST_WORDS;
    if (!asv_needs_scan(rec)) return;
    int c0 = d.chunk_prefix[si], c1 = d.chunk_prefix[si + 1];
    __shared__ int carry;
    __shared__ int wmax[32];
    if (threadIdx.x == 0) carry = 0;
    __syncthreads();
    for (int b0 = c0; b0 < c1; b0 += blockDim.x) {
        int c = b0 + threadIdx.x;
        int v = c < c1 ? d.scan[c] : 0;
        int incl = v;
        int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) { int n = __shfl_up_sync(FULL, incl, o); if (lane >= o && n > incl) incl = n; }
        if (lane == 31) wmax[w] = incl;
        __syncthreads();
        if (threadIdx.x < 32) {
            int x = wmax[threadIdx.x];
            int ix = x;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) { int n = __shfl_up_sync(FULL, ix, o); if (threadIdx.x >= o && n > ix) ix = n; }
            wmax[threadIdx.x] = ix;
        }
        __syncthreads();
        int before = w > 0 ? wmax[w - 1] : 0;
        int excl_in_warp = __shfl_up_sync(FULL, incl, 1);
        if (lane == 0) excl_in_warp = 0;
        int ex = max(max(carry, before), excl_in_warp);
        int tot = max(carry, wmax[31]);
        __syncthreads();
        if (c < c1) d.scan[c] = ex;      // max source+1 in earlier chunks of the segment
        if (threadIdx.x == 0) carry = tot;
        __syncthreads();
    }
}

// A thread takes eight consecutive voxels, by two 16-byte loads and stores.  A fill
// carries the source's label itself: inside the thread, from the last lane before
// it that has a source, from the warps before, else from the chunk's source.  (By
// maxima of 64-bit indices and a voxel at a time a batch of 40.5 M voxels took 163
// us, now 47.)
__global__ void __launch_bounds__(256) k_post_apply(AsvDev d)
{
    asv_follow();
    constexpr int PER = ASV_CHUNK / 256, NONE = -2;
    __shared__ int wlast[8];                                // label of the warp's last source, NONE without
    const int si = asv_find_seg(d.chunk_prefix, d.nseg, blockIdx.x);
    const SegDesc &S = d.segs[si];
    const int *rec = d.post + si * ASV_POST_WORDS, *rank = d.rank + S.seed_off;
    const int32_t *lbl = (S.final_buf ? d.labB : d.labA) + S.vox_off;
    int32_t *out = (S.final_buf ? d.labA : d.labB) + S.vox_off;
    const int Kp = S.Kp, mode = rec[POST_MODE], l0 = rec[POST_L0], lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const bool scan = asv_needs_scan(rec);
    const long long v0 = (long long)(blockIdx.x - d.chunk_prefix[si]) * ASV_CHUNK + threadIdx.x * PER;
    const bool full = v0 + PER <= S.nvox;                   // (segments start at multiples of ASV_CHUNK)
    int l[PER];
    if (full) {
#pragma unroll
        for (int k = 0; k < PER; k += 4) {
            const int4 q = *(const int4 *)(lbl + v0 + k);
            l[k] = q.x; l[k + 1] = q.y; l[k + 2] = q.z; l[k + 3] = q.w;
        }
    } else {
#pragma unroll
        for (int k = 0; k < PER; k++) l[k] = v0 + k < S.nvox ? lbl[v0 + k] : -1;
    }
    if (scan) {
        // the sources of asv_fill_src; voxel 0 is one of its own label in either
        // rule, but gives the rule's own value: POST_M0, or 0 for a -1 there
        auto source = [&](int k) { return (l[k] != -1 && (mode != 2 || l[k] != l0)) || v0 + k == 0; };
        int mine = NONE;
#pragma unroll
        for (int k = 0; k < PER; k++)
            if (v0 + k < S.nvox && source(k)) mine = l[k];
        const unsigned has = __ballot_sync(FULL, mine != NONE), before = has & ((1u << lane) - 1u);
        const int from = __shfl_sync(FULL, mine, before ? 31 - __clz((int)before) : 0);
        const int last = __shfl_sync(FULL, mine, has ? 31 - __clz((int)has) : 0);
        if (lane == 0) wlast[w] = has ? last : NONE;
        __syncthreads();
        int cur = before ? from : NONE;
        for (int k = w - 1; k >= 0 && cur == NONE; k--) cur = wlast[k];
        if (cur == NONE) {
            const int src = d.scan[blockIdx.x] - 1;          // -1: none (the first chunk's first voxel is one)
            cur = src >= 0 ? lbl[src] : -1;
        }
#pragma unroll
        for (int k = 0; k < PER; k++) {
            if (source(k)) cur = l[k];
            // mode 2: the source's rank; only voxel 0 as a source has l0.  Else the
            // source's relabelled label, 0 for a -1 at voxel 0 beyond it.
            if (mode == 2) l[k] = cur == l0 ? rec[POST_M0] : ((cur >= 0 && cur < Kp && rank[cur] >= 0) ? rank[cur] : 0);
            else {
                const int r = asv_relabel(rec, Kp, cur);
                l[k] = v0 + k == 0 ? r : (r >= 0 ? r : 0);
            }
        }
    } else {
#pragma unroll
        for (int k = 0; k < PER; k++) l[k] = asv_relabel(rec, Kp, l[k]);
    }
    if (full) {
#pragma unroll
        for (int k = 0; k < PER; k += 4) *(int4 *)(out + v0 + k) = make_int4(l[k], l[k + 1], l[k + 2], l[k + 3]);
    } else {
#pragma unroll
        for (int k = 0; k < PER; k++)
            if (v0 + k < S.nvox) out[v0 + k] = l[k];
    }
}

// ---------------------------------------------------------------------------
// launch wrappers
// ---------------------------------------------------------------------------
static inline int seed_blocks(const AsvDev &d) { return (d.total_seeds + 127) / 128; }

void asv_launch_srgb_table(const AsvDev &d, cudaStream_t st) { k_srgb_table<<<1, 256, 0, st>>>(d.srgb); }
void asv_launch_rgb2lab(const AsvDev &d, cudaStream_t st)
{
    if (d.lablut) k_rgb2lab_lut<<<d.total_chunks, 256, 0, st>>>(d);
    else k_rgb2lab<<<d.total_chunks, 256, 0, st>>>(d);
}

// per-device LAB table (64 MiB), built on first use; nullptr when it cannot
// be allocated (k_rgb2lab then computes every voxel)
const uchar4 *asv_lab_table(int device)
{
    static std::mutex mu;
    static uchar4 *tabs[64] = {};
    static bool tried[64] = {};
    if (device < 0 || device >= 64) return nullptr;
    std::lock_guard<std::mutex> lk(mu);
    if (tried[device]) return tabs[device];
    tried[device] = true;
    float *srgb = nullptr;
    uchar4 *lut = nullptr;
    unsigned *fix = nullptr;                       // entries to recompute, then their count
    cudaStream_t st = nullptr;
    if (cudaMalloc(&srgb, 256 * sizeof(float)) != cudaSuccess ||
        cudaMalloc(&lut, sizeof(uchar4) << 24) != cudaSuccess ||
        cudaMalloc(&fix, (sizeof(unsigned) << 24) + sizeof(unsigned)) != cudaSuccess ||
        cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking) != cudaSuccess) {
        cudaGetLastError();
        if (srgb) cudaFree(srgb);
        if (lut) cudaFree(lut);
        if (fix) cudaFree(fix);
        return nullptr;
    }
    unsigned *nfix = fix + (1u << 24);
    cudaMemsetAsync(nfix, 0, sizeof(unsigned), st);
    k_srgb_table<<<1, 256, 0, st>>>(srgb);
    k_lab_table<<<65536, 256, 0, st>>>(srgb, lut, fix, nfix);
    k_lab_table_fix<<<2048, 256, 0, st>>>(srgb, lut, fix, nfix);
    const bool ok = cudaStreamSynchronize(st) == cudaSuccess && cudaGetLastError() == cudaSuccess;
    cudaStreamDestroy(st);
    cudaFree(srgb);
    cudaFree(fix);
    if (!ok) { cudaFree(lut); return nullptr; }
    tabs[device] = lut;
    return lut;
}
void asv_launch_density(const AsvDev &d, cudaStream_t st) { k_density<<<d.total_chunks, 256, 0, st>>>(d); }
void asv_launch_density_adjust(const AsvDev &d, cudaStream_t st)
{
    k_density_adjust<<<d.nseg, 256, ASV_ADJ_SMEM * sizeof(float), st>>>(d, d.Mring);
}
void asv_launch_first_init(const AsvDev &d, cudaStream_t st) { k_first_init<<<seed_blocks(d), 128, 0, st>>>(d); }
void asv_launch_draw(const AsvDev &d, cudaStream_t st) { k_draw<<<seed_blocks(d), 128, 0, st>>>(d); }

struct AsvJfaVariant {
    void (*kernel)(AsvDev, int, const int32_t *, int32_t *);
    int smem;                                      // dynamic shared memory
};

// k_jfa's variant for a pass of this step (last: the pass that also sums)
static const AsvJfaVariant &asv_jfa_variant(int step, bool last)
{
    static const AsvJfaVariant v[ASV_JFA_LIST + 1] = {
        { k_jfa<1, true>, AsvBitsGeo<1>::SMEM + 4 * ASV_ACC_WORDS },
        { k_jfa<1, false>, AsvBitsGeo<1>::SMEM }, { k_jfa<2, false>, AsvBitsGeo<2>::SMEM },
        { k_jfa<3, false>, AsvBitsGeo<3>::SMEM }, { k_jfa<4, false>, AsvBitsGeo<4>::SMEM },
        { k_jfa<5, false>, AsvBitsGeo<5>::SMEM }, { k_jfa<6, false>, AsvBitsGeo<6>::SMEM },
        { k_jfa<ASV_JFA_LIST, false>, ASV_JFA_FAR_BYTES } };
    return v[last ? 0 : (step < ASV_JFA_LIST ? step : ASV_JFA_LIST)];
}

// the variants' dynamic shared memory exceeds the 48 KiB default: raised once
// per device
static void asv_jfa_attributes()
{
    static std::mutex mu;
    static bool done[64] = {};
    int dev = 0;
    cudaGetDevice(&dev);
    std::lock_guard<std::mutex> lk(mu);
    if (dev >= 0 && dev < 64 && done[dev]) return;
    for (int st = 0; st <= ASV_JFA_LIST; st++) {
        const AsvJfaVariant &v = asv_jfa_variant(st, st == 0);
        cudaFuncSetAttribute((const void *)v.kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, v.smem);
    }
    if (dev >= 0 && dev < 64) done[dev] = true;
}

// resident k_jfa blocks on the device (persistent grid size): the least of
// the variants', computed once per process (thread-safe static initialisation)
int asv_jfa_resident_blocks()
{
    static const int blocks = [] {
        int dev = 0, sms = 0, least = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        asv_jfa_attributes();
        for (int st = 0; st <= ASV_JFA_LIST; st++) {
            const AsvJfaVariant &v = asv_jfa_variant(st, st == 0);
            int per = 0;
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, v.kernel, ASV_JFA_THREADS, v.smem);
            if (per > 0 && (!least || per < least)) least = per;
        }
        const int b = sms * (least > 0 ? least : 1);
        return b > 0 ? b : 1024;
    }();
    return blocks;
}

int asv_jfa_slots(int step)
{
    static const int slots[ASV_BITS_MAXS + 1] = { 0, AsvBitsGeo<1>::NSLOT, AsvBitsGeo<2>::NSLOT, AsvBitsGeo<3>::NSLOT,
                                                  AsvBitsGeo<4>::NSLOT, AsvBitsGeo<5>::NSLOT, AsvBitsGeo<6>::NSLOT };
    return step >= 1 && step <= ASV_BITS_MAXS ? slots[step] : 0;
}

int asv_jfa_grid_blocks(int total_tiles)
{
    const int blocks = asv_jfa_resident_blocks();
    return total_tiles < blocks ? total_tiles : blocks;
}

void asv_launch_jfa(const AsvDev &d, int pass, int step, bool last, int grid_blocks, bool follow, cudaStream_t st)
{
    const int32_t *in = (pass & 1) ? d.labB : d.labA;
    int32_t *out = (pass & 1) ? d.labA : d.labB;
    asv_jfa_attributes();
    const AsvJfaVariant &v = asv_jfa_variant(step, last);
    asv_launch_follow(follow, v.kernel, grid_blocks, ASV_JFA_THREADS, v.smem, st, d, pass, in, out);
}

// filled: the output volume is all -1 and the list empty already
void asv_launch_jfa_first(const AsvDev &d, bool filled, bool stale, cudaStream_t st)
{
    if (!filled) {
        cudaMemsetAsync(d.labB, 0xff, sizeof(int32_t) * (size_t)d.total_chunks * ASV_CHUNK, st);
        cudaMemsetAsync(d.tcount, 0, sizeof(*d.tcount), st);
    }
    k_jfa_first<<<asv_first_blocks(d.total_seeds), 256, 0, st>>>(d, stale);
}

// into labA, which is all -1.  undraw: d.drawn holds nothing but the seeds at
// their current positions, and becomes all -1 again
void asv_launch_jfa_second_scatter(const AsvDev &d, bool undraw, cudaStream_t st)
{
    const unsigned blocks = 27u * (unsigned)((27LL * d.total_seeds + 255) / 256);   // tlist holds <= 27 entries per seed
    asv_launch_follow(undraw, k_jfa_second, blocks, 256, 0, st, d, undraw);      // (undraw: behind the first pass)
}

void asv_launch_pass_prepare(int32_t *labels, const SegDesc &one, const SegDesc *seg, SegDesc *out, cudaStream_t st)
{
    k_pass_prepare<<<(unsigned)((one.nvox + 255) / 256), 256, 0, st>>>(labels, one, seg, out);
}

void asv_launch_centroids(const AsvDev &d, cudaStream_t st) { k_centroids<<<d.total_chunks, 256, 0, st>>>(d); }
void asv_launch_finalize(const AsvDev &d, cudaStream_t st) { k_finalize<<<seed_blocks(d), 128, 0, st>>>(d); }

void asv_launch_post(const AsvDev &d, cudaStream_t st)
{
    k_post_stats<<<d.nseg, 1024, 0, st>>>(d);
    asv_launch_follow(true, k_post_chunk_max, d.total_chunks, 256, 0, st, d);
    asv_launch_follow(true, k_post_prefix, d.nseg, 1024, 0, st, d);
    asv_launch_follow(true, k_post_apply, d.total_chunks, 256, 0, st, d);
}

// asv_flow.cu -- dense optical flow on the device for the clip's metric.
//
// The reference computes the forward and backward flow of every frame with
// OpenCV's CUDA Farneback (GPU-AS/Image.cpp:643-686, cuda::FarnebackOpticalFlow
// with its default configuration: 5 pyramid levels at scale 0.5, polynomial
// neighbourhood 5 with sigma 1.1, a 13x13 averaging window, 10 iterations per
// level) on the grey frames of the preprocessed clip (GPU-AS/Render.cpp:
// 227-243).  OpenCV is not available here, so this is this project's
// implementation of the published method (G. Farneback, "Two-frame motion
// estimation based on polynomial expansion", SCIA 2003) with that
// configuration; its results are not bit-compared with OpenCV's.
//
// Per pyramid level, coarse to fine, for every frame pair of the clip at once
// (frame z -> z+1 and z -> z-1):
//   1. polynomial expansion of each frame: a weighted least-squares fit of
//      f(x+u, y+v) ~ c + b1 u + b2 v + a11 u^2 + a22 v^2 + 2 a12 u v over a
//      5x5 window with Gaussian weights, computed as six separable moment
//      filters and the inverse of the (constant) 6x6 normal matrix;
//   2. per iteration: A = (A_src(x) + A_dst(x + d)) / 2 and
//      db = -(b_dst(x + d) - b_src(x)) / 2 + A d (bilinear samples of the
//      destination expansion), the products A^T A and A^T db averaged over
//      the 13x13 window, and d = (A^T A)^-1 A^T db per pixel;
//   3. the flow is upsampled to the next finer level.
// The grey frames use the integer RGB -> grey of ITU-R BT.601 with 14-bit
// fixed-point weights (4899, 9617, 1868).
#include "asv_follow.cuh"
#include "asv_flow.cuh"

#include <math.h>

#define FL_T 256
#define FL_N 2          // polynomial window half-size (neighbourhood 5)
#define FL_BOX 6        // averaging window half-size (13x13)
#define FL_MAX_LEVELS 5

__constant__ float c_fl_g[3][2 * FL_N + 1];   // g(t), t g(t), t^2 g(t), t = -N..N
__constant__ float c_fl_ginv[5][6];           // rows b1, b2, a11, a22, 2*a12 of the normal-matrix inverse

// ---------------------------------------------------------------------------
__global__ void k_fl_gray(const uint8_t *__restrict__ rgb, float *__restrict__ out, long long n)
{
    asv_follow();
    const long long v = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (v >= n) return;
    const uint8_t *p = rgb + 3 * v;
    out[v] = (float)((p[0] * 4899 + p[1] * 9617 + p[2] * 1868 + 8192) >> 14);
}

// 5x5 binomial blur ([1 4 6 4 1]^2 / 256, clamp to edge) and decimation by 2
__global__ void k_fl_down(const float *in, int Wi, int Hi, float *__restrict__ out, int Wo,
                          int Ho, int D)
{
    asv_follow();
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const long long fo = (long long)Wo * Ho;
    if (t >= fo * D) return;
    const int z = (int)(t / fo), p = (int)(t - z * fo), y = p / Wo, x = p - y * Wo;
    const float w[5] = { 1.f, 4.f, 6.f, 4.f, 1.f };
    const float *src = in + (long long)Wi * Hi * z;
    float acc = 0.f;
    for (int j = -2; j <= 2; j++) {
        const int yy = min(max(2 * y + j, 0), Hi - 1);
        float row = 0.f;
        for (int i = -2; i <= 2; i++) row += w[i + 2] * src[(long long)yy * Wi + min(max(2 * x + i, 0), Wi - 1)];
        acc += w[j + 2] * row;
    }
    out[t] = acc * (1.f / 256.f);
}

// horizontal moments: h_p(x, y) = sum_u t^p g(u) f(x + u, y), p = 0, 1, 2
__global__ void k_fl_poly_h(const float *img, int W, int H, int D, float *__restrict__ h)
{
    asv_follow();
    const long long plane = (long long)W * H * D;
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= plane) return;
    const int x = (int)(t % W);
    const long long row = t - x;
    float s0 = 0.f, s1 = 0.f, s2 = 0.f;
#pragma unroll
    for (int u = -FL_N; u <= FL_N; u++) {
        const float f = img[row + min(max(x + u, 0), W - 1)];
        s0 += c_fl_g[0][u + FL_N] * f;
        s1 += c_fl_g[1][u + FL_N] * f;
        s2 += c_fl_g[2][u + FL_N] * f;
    }
    h[t] = s0;
    h[plane + t] = s1;
    h[2 * plane + t] = s2;
}

// vertical moments and the fit: per pixel (b1, b2, a11, a22) in polyA and
// a12 in polyB, so a bilinear tap of the expansion is two loads
__global__ void k_fl_poly_v(const float *h, int W, int H, int D, float4 *__restrict__ polyA,
                            float *__restrict__ polyB)
{
    asv_follow();
    const long long plane = (long long)W * H * D;
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= plane) return;
    const long long fr = (long long)W * H;
    const int z = (int)(t / fr);
    const int p = (int)(t - z * fr), y = p / W, x = p - y * W;
    float m[6] = { 0.f, 0.f, 0.f, 0.f, 0.f, 0.f };   // 1, u, v, u^2, v^2, uv
#pragma unroll
    for (int v = -FL_N; v <= FL_N; v++) {
        const long long q = fr * z + (long long)min(max(y + v, 0), H - 1) * W + x;
        const float h0 = h[q], h1 = h[plane + q], h2 = h[2 * plane + q];
        const float g = c_fl_g[0][v + FL_N], vg = c_fl_g[1][v + FL_N], vvg = c_fl_g[2][v + FL_N];
        m[0] += g * h0;
        m[1] += g * h1;
        m[2] += vg * h0;
        m[3] += g * h2;
        m[4] += vvg * h0;
        m[5] += vg * h1;
    }
    float r[5];
#pragma unroll
    for (int k = 0; k < 5; k++) {
        r[k] = 0.f;
#pragma unroll
        for (int e = 0; e < 6; e++) r[k] += c_fl_ginv[k][e] * m[e];
    }
    polyA[t] = make_float4(r[0], r[1], r[2], r[3]);
    polyB[t] = 0.5f * r[4];
}

// frame pair p: source and destination frames (forward pairs first)
__device__ __forceinline__ void fl_pair(int p, int D, int &src, int &dst)
{
    if (p < D - 1) { src = p; dst = p + 1; }
    else { src = p - (D - 1) + 1; dst = src - 1; }
}

// the per-pixel products A^T A (g11, g12, g22) and A^T db (h1, h2) at pixel
// (x, y) of the frame with the current flow (dx, dy), from the expansions
// sA/sB of the source frame and dA/dB of the destination frame; zero when
// x + d falls outside the frame.  THIN: the frame may be one pixel wide or high.
template <bool THIN>
__device__ __forceinline__ void fl_matrix(const float4 *__restrict__ sA, const float *__restrict__ sB,
                                          const float4 *__restrict__ dA, const float *__restrict__ dB, int W,
                                          int H, int x, int y, float dx, float dy, float o[5])
{
    // no early exit: the sample indices are clamped into the frame whatever
    // the flow (also NaN), every load is issued, and the result is zeroed by
    // a select, so a thread's evaluations overlap their loads
    const float qx = (float)x + dx, qy = (float)y + dy;
    const bool inside = qx >= 0.f && qy >= 0.f && qx <= (float)(W - 1) && qy <= (float)(H - 1);
    const int x0 = min(max((int)qx, 0), THIN ? max(W - 2, 0) : W - 2), y0 = min(max((int)qy, 0), THIN ? max(H - 2, 0) : H - 2);
    const int right = THIN && W < 2 ? 0 : 1, below = THIN && H < 2 ? 0 : W;   // to the samples at x0 + 1, y0 + 1
    const float fx = qx - (float)x0, fy = qy - (float)y0;
    const float w00 = (1.f - fx) * (1.f - fy), w01 = fx * (1.f - fy), w10 = (1.f - fx) * fy, w11 = fx * fy;
    const int s = y * W + x;                                   // frames hold < 2^31 pixels
    const int i0 = y0 * W + x0, i1 = i0 + below;
    const float4 t00 = __ldg(dA + i0), t01 = __ldg(dA + i0 + right), t10 = __ldg(dA + i1), t11 = __ldg(dA + i1 + right);
    const float u00 = __ldg(dB + i0), u01 = __ldg(dB + i0 + right), u10 = __ldg(dB + i1), u11 = __ldg(dB + i1 + right);
    const float4 sa = __ldg(sA + s);
    const float sb = __ldg(sB + s);
    float q[5];
    q[0] = w00 * t00.x + w01 * t01.x + w10 * t10.x + w11 * t11.x;
    q[1] = w00 * t00.y + w01 * t01.y + w10 * t10.y + w11 * t11.y;
    q[2] = w00 * t00.z + w01 * t01.z + w10 * t10.z + w11 * t11.z;
    q[3] = w00 * t00.w + w01 * t01.w + w10 * t10.w + w11 * t11.w;
    q[4] = w00 * u00 + w01 * u01 + w10 * u10 + w11 * u11;
    const float a11 = 0.5f * (sa.z + q[2]);
    const float a22 = 0.5f * (sa.w + q[3]);
    const float a12 = 0.5f * (sb + q[4]);
    const float db1 = -0.5f * (q[0] - sa.x) + a11 * dx + a12 * dy;
    const float db2 = -0.5f * (q[1] - sa.y) + a12 * dx + a22 * dy;
    o[0] = inside ? a11 * a11 + a12 * a12 : 0.f;
    o[1] = inside ? a11 * a12 + a12 * a22 : 0.f;
    o[2] = inside ? a12 * a12 + a22 * a22 : 0.f;
    o[3] = inside ? a11 * db1 + a12 * db2 : 0.f;
    o[4] = inside ? a12 * db1 + a22 * db2 : 0.f;
}

// One iteration for a strip of FL_TW columns and `rows` rows of one frame pair.
// The block goes down the strip eight rows at a time: it computes the five
// matrix planes of the next rows and their 6-pixel halo in x from the flow
// `fin` (zero outside the frame), sums them over 13 columns into a ring of 20
// rows, and sums the ring over 13 rows for eight finished ones, whose 2x2
// systems it solves into `fout`.  Both sums run in ascending index order, so
// they equal those of separate x and y passes.  fin and fout are separate
// buffers: halo pixels read flow that neighbouring strips overwrite.
//
// The iterations are bound by instruction issue and the shared-memory data path
// (68 % each with a tile of 64 x 32 per block: 1.63 matrices per pixel, 632
// instructions).  Going down a strip leaves the halo in x and twelve rows per
// strip, 1.2 to 1.3 matrices per pixel; the sums of two planes are two-wide
// additions (sums only: no product feeds them); four windows share a thread's
// sixteen loads in both directions.  At 640x480x16, level 0, 240 -> 178 us an
// iteration.
//
// Shared memory: S[5][8][FL_SP], where a column c lies at c + c / 4: the threads
// of a warp, two rows of sixteen windows four columns apart, then read sixteen
// banks five apart and, the row pitch being 16 modulo 32, the other sixteen.
// T[5][20][FL_TW], the ring: row y of the strip is at (y + 6) mod 20.
#define FL_TW 64
#define FL_NT 128
#define FL_RS 8                              // rows per step
#define FL_RING (FL_RS + 2 * FL_BOX)
#define FL_RW (FL_TW + 2 * FL_BOX)
#define FL_PX ((FL_RS * FL_RW + FL_NT - 1) / FL_NT)   // matrices per thread and step
#define FL_SP 112
#define FL_SMEM (4 * 5 * (FL_RS * FL_SP + FL_RING * FL_TW))

template <bool THIN>
__global__ void __launch_bounds__(FL_NT, 5) k_fl_iter(const float4 *__restrict__ polyA, const float *__restrict__ polyB,
                                                   const float *fin, float *__restrict__ fout, int W,
                                                   int H, int D, int P, int rows)
{
    asv_follow();
    extern __shared__ __align__(16) float fl_sm[];
    float *S = fl_sm, *T = fl_sm + 5 * FL_RS * FL_SP;
    const long long fr = (long long)W * H, mplane = fr * P;
    const int strips = (W + FL_TW - 1) / FL_TW, chunks = (H + rows - 1) / rows;
    // blocks take the pairs as z -> z+1, z+1 -> z, z+1 -> z+2, ...: the two
    // pairs of a frame pair read the same two expansions while both are in L2
    const int j = blockIdx.x / (strips * chunks);
    const int pr = (j & 1) ? D - 1 + (j >> 1) : (j >> 1);
    const int rem = blockIdx.x - j * strips * chunks;
    const int x0 = (rem % strips) * FL_TW, yb = (rem / strips) * rows, ye = min(yb + rows, H);
    int src, dst;
    fl_pair(pr, D, src, dst);
    const float4 *sA = polyA + fr * src, *dA = polyA + fr * dst;
    const float *sB = polyB + fr * src, *dB = polyB + fr * dst;
    const float *fx_in = fin + fr * pr, *fy_in = fin + mplane + fr * pr;
    const int t = threadIdx.x;

    // a thread's pixels of a step: the same columns and rows of S every time.
    // Their flow is loaded a step ahead (before the vertical sums), so that a
    // step waits for the samples only, two or three pixels' at a time.
    unsigned px[FL_PX];                                                  // column in the frame, row (3 bits) and place
    unsigned keepx = 0u;
    float fx[FL_PX], fy[FL_PX];
#pragma unroll
    for (int k = 0; k < FL_PX; k++) {
        const int i = min(t + k * FL_NT, FL_RS * FL_RW - 1), r = i / FL_RW, q = i - r * FL_RW, gx = x0 - FL_BOX + q;
        if (gx >= 0 && gx < W) keepx |= 1u << k;                         // zero outside the frame
        px[k] = ((unsigned)min(max(gx, 0), W - 1) << 13) | (r << 10) | (r * FL_SP + q + (q >> 2));   // (10 bits) in S
    }
    auto col_of = [&](int k) { return (int)(px[k] >> 13); };
    auto row_of = [&](int k) { return (int)(px[k] >> 10) & (FL_RS - 1); };
    auto load_flow = [&](int y) {
#pragma unroll
        for (int k = 0; k < FL_PX; k++) {
            const int e = min(max(y + row_of(k), 0), H - 1) * W + col_of(k);
            fx[k] = asv_load_behind(fx_in + e);
            fy[k] = asv_load_behind(fy_in + e);
        }
    };

    // matrices of rows y .. y + n - 1 (their flow loaded) into S, then their
    // window sums along x into the ring from row `slot`
    auto add_rows = [&](int y, int n, int slot) {
#pragma unroll
        for (int k0 = 0; k0 < FL_PX; k0 += 3) {
            float o[3][5];
#pragma unroll
            for (int u = 0; u < 3 && k0 + u < FL_PX; u++) {
                const int k = k0 + u;
                fl_matrix<THIN>(sA, sB, dA, dB, W, H, col_of(k), min(max(y + row_of(k), 0), H - 1), fx[k], fy[k], o[u]);
            }
#pragma unroll
            for (int u = 0; u < 3 && k0 + u < FL_PX; u++) {
                const int k = k0 + u, gy = y + row_of(k);
                if (t + k * FL_NT >= FL_RS * FL_RW) continue;
                const bool keep = (keepx >> k) & 1u && gy >= 0 && gy < H;
#pragma unroll
                for (int c = 0; c < 5; c++) S[c * FL_RS * FL_SP + (px[k] & 1023u)] = keep ? o[u][c] : 0.f;
            }
        }
        __syncthreads();
        const int r = t >> 4, q = t & 15;                                // row, window group (four windows)
        if (r < n) {
            const float *Sr = S + r * FL_SP + 5 * q;
            int d = slot + r;
            d = d >= FL_RING ? d - FL_RING : d;
            float4 *Td = (float4 *)(T + d * FL_TW) + q;
#pragma unroll
            for (int c = 0; c < 4; c += 2) {
                float2 w[16];
#pragma unroll
                for (int k = 0; k < 16; k++)
                    w[k] = make_float2(Sr[c * FL_RS * FL_SP + k + (k >> 2)], Sr[(c + 1) * FL_RS * FL_SP + k + (k >> 2)]);
                float2 v[4];
#pragma unroll
                for (int m = 0; m < 4; m++) {
                    v[m] = make_float2(0.f, 0.f);
#pragma unroll
                    for (int k = 0; k <= 2 * FL_BOX; k++) v[m] = __fadd2_rn(v[m], w[m + k]);
                }
                Td[c * FL_RING * FL_TW / 4] = make_float4(v[0].x, v[1].x, v[2].x, v[3].x);
                Td[(c + 1) * FL_RING * FL_TW / 4] = make_float4(v[0].y, v[1].y, v[2].y, v[3].y);
            }
            float w[16], v[4];
#pragma unroll
            for (int k = 0; k < 16; k++) w[k] = Sr[4 * FL_RS * FL_SP + k + (k >> 2)];
#pragma unroll
            for (int m = 0; m < 4; m++) {
                v[m] = 0.f;
#pragma unroll
                for (int k = 0; k <= 2 * FL_BOX; k++) v[m] += w[m + k];
            }
            Td[4 * FL_RING * FL_TW / 4] = make_float4(v[0], v[1], v[2], v[3]);
        }
        __syncthreads();
    };

    load_flow(yb - FL_BOX);
    add_rows(yb - FL_BOX, FL_RS, 0);                                     // the first twelve rows
    load_flow(yb - FL_BOX + FL_RS);
    add_rows(yb - FL_BOX + FL_RS, 2 * FL_BOX - FL_RS, FL_RS);
    load_flow(yb + FL_BOX);
    int slot = 2 * FL_BOX;                                               // ring row of the next rows
    const int col = t & (FL_TW - 1), h = t / FL_TW;                      // column, half of the eight rows
    for (int y = yb; y < ye; y += FL_RS) {
        add_rows(y + FL_BOX, FL_RS, slot);
        slot += FL_RS;
        slot = slot >= FL_RING ? slot - FL_RING : slot;                  // now the ring row of y - 6
        load_flow(y + FL_RS + FL_BOX);                                   // (clamped into the frame past the strip)
        const float *g[4];                                               // ring rows of y - 6 + 4 h + 0, 4, 8, 12
#pragma unroll
        for (int k = 0; k < 4; k++) {
            int d = slot + 4 * (h + k);
            d = d >= FL_RING ? d - FL_RING : d;
            g[k] = T + d * FL_TW + col;
        }
        float acc[5][4];
#pragma unroll
        for (int c = 0; c < 4; c += 2) {
            float2 w[16];
#pragma unroll
            for (int k = 0; k < 16; k++) {
                const float *e = g[k >> 2] + (k & 3) * FL_TW;
                w[k] = make_float2(e[c * FL_RING * FL_TW], e[(c + 1) * FL_RING * FL_TW]);
            }
#pragma unroll
            for (int m = 0; m < 4; m++) {
                float2 v = make_float2(0.f, 0.f);
#pragma unroll
                for (int k = 0; k <= 2 * FL_BOX; k++) v = __fadd2_rn(v, w[m + k]);
                acc[c][m] = v.x;
                acc[c + 1][m] = v.y;
            }
        }
        {
            float w[16];
#pragma unroll
            for (int k = 0; k < 16; k++) w[k] = g[k >> 2][4 * FL_RING * FL_TW + (k & 3) * FL_TW];
#pragma unroll
            for (int m = 0; m < 4; m++) {
                float v = 0.f;
#pragma unroll
                for (int k = 0; k <= 2 * FL_BOX; k++) v += w[m + k];
                acc[4][m] = v;
            }
        }
        const int x = x0 + col;
#pragma unroll
        for (int m = 0; m < 4; m++) {
            const int yy = y + 4 * h + m;
            if (x >= W || yy >= ye) continue;
            const float g11 = acc[0][m], g12 = acc[1][m], g22 = acc[2][m], h1 = acc[3][m], h2 = acc[4][m];
            const float idet = 1.f / (g11 * g22 - g12 * g12 + 1e-3f);
            const long long e = fr * pr + (long long)yy * W + x;
            fout[e] = (g22 * h1 - g12 * h2) * idet;
            fout[mplane + e] = (g11 * h2 - g12 * h1) * idet;
        }
    }
}

// Rows of a strip per block: a multiple of the eight of a step such that the
// blocks' rounds on the GPU take least, a block costing its rows, the twelve
// before them and about as much as four more to start.  Frames of up to three steps
// go in one strip where that gives every other SM two blocks, which fill it: a
// second strip would do the twelve rows again beside them (500x17x20: 228 us in
// two, 163 in one; 200x20x30 180 and 164; 64x17x40, half a block per SM, 104 and 139).
static int fl_rows(int W, int H, int P, int sms, int resident)
{
    const long long columns = (long long)((W + FL_TW - 1) / FL_TW) * P;
    if (H <= 3 * FL_RS && 2 * columns >= 3 * sms) return (H + FL_RS - 1) / FL_RS * FL_RS;
    int best = FL_RS;
    long long least = 0;
    for (int r = FL_RS; r <= ((H + FL_RS - 1) / FL_RS) * FL_RS; r += FL_RS) {
        const long long blocks = columns * ((H + r - 1) / r);
        const long long cost = (blocks + resident - 1) / resident * (r + 2 * FL_BOX + 4);
        if (!least || cost < least) { least = cost; best = r; }
    }
    return best;
}

// flow of level k from level k+1: bilinear, scaled by the size ratio; a block
// per 256 columns, eight rows and pair (one thread per pixel of a flat index,
// with its 64-bit divisions: 68 us for the 640x480 level of 30 pairs, 39 us now)
#define FL_UP_ROWS 8
__global__ void __launch_bounds__(FL_T) k_fl_up(const float *coarse, int Wc, int Hc, float *__restrict__ fine,
                                                int W, int H, int P)
{
    asv_follow();
    const int x = blockIdx.x * FL_T + threadIdx.x, pr = blockIdx.z;
    if (x >= W) return;
    const long long mplane = (long long)W * H * P, cplane = (long long)Wc * Hc * P;
    const float *F = coarse + (long long)Wc * Hc * pr;
    float *out = fine + (long long)W * H * pr + x;
    const float sx = (float)Wc / (float)W, sy = (float)Hc / (float)H;
    const float cx = fminf(fmaxf(((float)x + 0.5f) * sx - 0.5f, 0.f), (float)(Wc - 1));
    const int x0 = (int)cx, x1 = min(x0 + 1, Wc - 1);
    const float fx = cx - (float)x0;
    const int ye = min((int)(blockIdx.y + 1) * FL_UP_ROWS, H);
    for (int y = blockIdx.y * FL_UP_ROWS; y < ye; y++) {
        const float cy = fminf(fmaxf(((float)y + 0.5f) * sy - 0.5f, 0.f), (float)(Hc - 1));
        const int y0 = (int)cy, y1 = min(y0 + 1, Hc - 1);
        const float fy = cy - (float)y0;
#pragma unroll
        for (int c = 0; c < 2; c++) {
            const float *G = F + c * cplane;
            const float v = (1.f - fx) * (1.f - fy) * G[y0 * Wc + x0] + fx * (1.f - fy) * G[y0 * Wc + x1] +
                            (1.f - fx) * fy * G[y1 * Wc + x0] + fx * fy * G[y1 * Wc + x1];
            out[c * mplane + y * W] = v / (c == 0 ? sx : sy);
        }
    }
}

// level-0 flow of the pairs into the clip's interleaved fwd / bwd volumes
__global__ void k_fl_store(const float *flow, int W, int H, int D, float2 *__restrict__ fwd,
                           float2 *__restrict__ bwd, int keep_first_bwd)
{
    asv_follow();
    const long long fr = (long long)W * H, vox = fr * D, mplane = fr * 2 * (D - 1);
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= vox) return;
    const int z = (int)(t / fr);
    const long long pix = t - z * fr;
    float2 f = make_float2(0.f, 0.f), b = make_float2(0.f, 0.f);
    if (z < D - 1) {
        const long long e = fr * z + pix;
        f = make_float2(flow[e], flow[mplane + e]);
    }
    if (z > 0) {
        const long long e = fr * (D - 1 + z - 1) + pix;
        b = make_float2(flow[e], flow[mplane + e]);
    }
    fwd[t] = f;
    if (z > 0 || !keep_first_bwd) bwd[t] = b;
}

// ---------------------------------------------------------------------------
static int fl_levels(int W, int H, int *Ws, int *Hs)
{
    int L = 0, w = W, h = H;
    while (L < FL_MAX_LEVELS) {
        Ws[L] = w; Hs[L] = h;
        L++;
        const int nw = (w + 1) / 2, nh = (h + 1) / 2;
        if (nw < 16 || nh < 16) break;
        w = nw; h = nh;
    }
    return L;
}

size_t asv_flow_scratch_bytes(int W, int H, int D)
{
    if (D < 2) return 0;
    int Ws[FL_MAX_LEVELS], Hs[FL_MAX_LEVELS];
    const int L = fl_levels(W, H, Ws, Hs);
    const long long P = 2LL * (D - 1);
    size_t b = 0;
    for (int k = 0; k < L; k++) {
        const long long fr = (long long)Ws[k] * Hs[k];
        b += (size_t)fr * D * (1 + 3 + 5) * 4;     // image, horizontal moments, expansion
        b += (size_t)fr * P * 2 * 4;               // flow
    }
    const long long fr0 = (long long)W * H;
    b += (size_t)fr0 * P * 2 * 4;                  // second flow buffer (iterations alternate)
    return b + 64 * 256;
}

struct FlConsts {
    float g[3][2 * FL_N + 1];
    float ginv[5][6];
};

// Gaussian applicability (sigma 1.1) t^p g(t), and rows 1..5 of the inverse
// of the 6x6 normal matrix sum w B B^T of the basis B = (1, u, v, u^2, v^2, uv)
static FlConsts fl_consts()
{
    FlConsts K;
    const double sigma = 1.1;
    double g[2 * FL_N + 1];
    for (int u = -FL_N; u <= FL_N; u++) {
        g[u + FL_N] = exp(-(double)(u * u) / (2.0 * sigma * sigma));
        K.g[0][u + FL_N] = (float)g[u + FL_N];
        K.g[1][u + FL_N] = (float)(u * g[u + FL_N]);
        K.g[2][u + FL_N] = (float)(u * u * g[u + FL_N]);
    }
    double G[6][12] = {};
    for (int v = -FL_N; v <= FL_N; v++)
        for (int u = -FL_N; u <= FL_N; u++) {
            const double w = g[u + FL_N] * g[v + FL_N];
            const double B[6] = { 1.0, (double)u, (double)v, (double)(u * u), (double)(v * v), (double)(u * v) };
            for (int i = 0; i < 6; i++)
                for (int j = 0; j < 6; j++) G[i][j] += w * B[i] * B[j];
        }
    for (int i = 0; i < 6; i++) G[i][6 + i] = 1.0;
    for (int c = 0; c < 6; c++) {                               // Gauss-Jordan, partial pivoting
        int piv = c;
        for (int r = c + 1; r < 6; r++) if (fabs(G[r][c]) > fabs(G[piv][c])) piv = r;
        for (int j = 0; j < 12; j++) { const double tmp = G[c][j]; G[c][j] = G[piv][j]; G[piv][j] = tmp; }
        const double d = G[c][c];
        for (int j = 0; j < 12; j++) G[c][j] /= d;
        for (int r = 0; r < 6; r++)
            if (r != c) {
                const double f = G[r][c];
                for (int j = 0; j < 12; j++) G[r][j] -= f * G[c][j];
            }
    }
    for (int k = 0; k < 5; k++)
        for (int e = 0; e < 6; e++) K.ginv[k][e] = (float)G[k + 1][6 + e];
    return K;
}

static float *fl_carve(unsigned char *&p, size_t floats)
{
    float *r = (float *)p;
    p += (floats * 4 + 255) & ~(size_t)255;
    return r;
}

static unsigned fl_blocks(long long n) { return (unsigned)((n + FL_T - 1) / FL_T); }

int asv_launch_flow(const uint8_t *rgb, int W, int H, int D, float2 *fwd, float2 *bwd, void *scratch,
                    cudaStream_t st, int keep_first_bwd)
{
    if (D < 2) return -1;
    // filter constants: computed once (thread-safe static), copied to this
    // device's constant memory on the stream before the kernels that read them
    static const FlConsts K = fl_consts();
    if (cudaMemcpyToSymbolAsync(c_fl_g, K.g, sizeof(K.g), 0, cudaMemcpyHostToDevice, st) != cudaSuccess ||
        cudaMemcpyToSymbolAsync(c_fl_ginv, K.ginv, sizeof(K.ginv), 0, cudaMemcpyHostToDevice, st) != cudaSuccess)
        return -1;
    int Ws[FL_MAX_LEVELS], Hs[FL_MAX_LEVELS];
    const int L = fl_levels(W, H, Ws, Hs);
    const int P = 2 * (D - 1);
    unsigned char *p = (unsigned char *)scratch;
    float *img[FL_MAX_LEVELS], *hm[FL_MAX_LEVELS], *polyB[FL_MAX_LEVELS], *flow[FL_MAX_LEVELS];
    float4 *polyA[FL_MAX_LEVELS];
    for (int k = 0; k < L; k++) {
        const size_t fr = (size_t)Ws[k] * Hs[k];
        img[k] = fl_carve(p, fr * D);
        hm[k] = fl_carve(p, fr * D * 3);
        polyA[k] = (float4 *)fl_carve(p, fr * D * 4);      // 256-byte aligned
        polyB[k] = fl_carve(p, fr * D);
        flow[k] = fl_carve(p, fr * P * 2);
    }
    const size_t fr0 = (size_t)W * H;
    float *alt = fl_carve(p, fr0 * P * 2);
    int dev = 0, sms = 1, per = 1;
    if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_fl_iter<false>, FL_NT, FL_SMEM) != cudaSuccess)
        return -1;

    k_fl_gray<<<fl_blocks((long long)fr0 * D), FL_T, 0, st>>>(rgb, img[0], (long long)fr0 * D);
    for (int k = 1; k < L; k++)
        asv_launch_follow(true, k_fl_down, fl_blocks((long long)Ws[k] * Hs[k] * D), FL_T, 0, st, img[k - 1], Ws[k - 1],
                          Hs[k - 1], img[k], Ws[k], Hs[k], D);
    for (int k = 0; k < L; k++) {
        const long long n = (long long)Ws[k] * Hs[k] * D;
        asv_launch_follow(true, k_fl_poly_h, fl_blocks(n), FL_T, 0, st, img[k], Ws[k], Hs[k], D, hm[k]);
        asv_launch_follow(true, k_fl_poly_v, fl_blocks(n), FL_T, 0, st, hm[k], Ws[k], Hs[k], D, polyA[k], polyB[k]);
    }
    for (int k = L - 1; k >= 0; k--) {
        const int w = Ws[k], h = Hs[k];
        const long long mplane = (long long)w * h * P;
        if (k == L - 1) cudaMemsetAsync(flow[k], 0, sizeof(float) * mplane * 2, st);
        else
            asv_launch_follow(true, k_fl_up, dim3((w + FL_T - 1) / FL_T, (h + FL_UP_ROWS - 1) / FL_UP_ROWS, P), FL_T, 0, st,
                              flow[k + 1], Ws[k + 1], Hs[k + 1], flow[k], w, h, P);
        const int rows = fl_rows(w, h, P, sms, sms * (per > 0 ? per : 1));
        const unsigned blocks = (unsigned)((w + FL_TW - 1) / FL_TW) * ((h + rows - 1) / rows) * P;
        for (int it = 0; it < 10; it++) {                 // even count: the result ends in flow[k]
            const float *fin = (it & 1) ? alt : flow[k];
            float *fout = (it & 1) ? flow[k] : alt;
            asv_launch_follow(it > 0 || k < L - 1, w > 1 && h > 1 ? k_fl_iter<false> : k_fl_iter<true>, blocks, FL_NT, FL_SMEM,
                              st, polyA[k], polyB[k], fin, fout, w, h, D, P, rows);
        }
    }
    asv_launch_follow(true, k_fl_store, fl_blocks((long long)fr0 * D), FL_T, 0, st, flow[0], W, H, D, fwd, bwd, keep_first_bwd);
    return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

// asv_metric.cu -- per-seed anisotropic metric tensor from the flow field.
//
// Replaces the reference's CPU solve (GPU-AS/Image.cpp:689-1009 seed_matrix /
// matrix_slover, :1300-1534 Ld_next_seeds_matrix) and its GPU->CPU->GPU
// round trip every Lloyd iteration.  For each seed, the 3x3 neighbourhood of
// its voxel gives up to 18 rows d^T M d = b (forward rows d = (dx, dy, 1),
// backward rows d = (dx, dy, -1), b = n^2 + m^2 + 1); M is the min-norm
// least-squares solution in FP32 like the reference's Eigen float solve
// (one-sided Jacobi SVD, rank rule of Eigen's SVD solve: keep
// sigma >= max(sigma_max * min(rows,6) * FLT_EPSILON, FLT_MIN)); the 3x3
// PSD test is exact (principal minors, error-free FP64 expansion) and the
// nearest-PSD projection runs in FP64.  A non-PSD M falls back to the mean of
// the PSD metrics of the 1-ring, then 2-ring neighbours, then to the nearest
// PSD matrix.
//
// Sixteen lanes per solve: two per column of the system, with its even and odd
// rows.  A sweep's rotations of different columns don't touch each other, and the
// pair (p, q) only needs the pairs of p and q before it in the cyclic order, all
// of which have a smaller p + q (6 more per sweep): so the pairs of equal p + q
// modulo 6 rotate together, the last ones of a sweep beside the first of the next,
// in 6 steps a sweep instead of 15, with the same bits.  In step c column i meets
// column c - i (modulo 6): both fetch the other, form the same sums and angle, and
// update themselves.
// Launches: k_metric_self (in a reseed first the seed's new position, then its
// solve and PSD test; the non-PSD seeds are listed), k_metric_ring (a solve per
// listed seed and neighbour) and k_metric_combine (a thread per seed: the
// fallbacks, and the seed's draw where the next flood follows).  A reseed solve is
// skipped when the seed's voxel is the one of its previous reseed solve in this
// Lloyd run: the metric is a function of that voxel and the flow only, so the
// stored result is the solve's result.
// The chain is latency-bound (a few warps per SM, up to some sixty rotations of
// two square roots and three divisions): a warp per solve, a row per lane and one
// pair after the other took 33 us for the seeds of the 320x240x85 clip and 54 us
// for the rings of one with computed flow, now 19 and 35 us.
// Compiled with -fmad=false.
#include "asv_follow.cuh"
#include "asv_seed.cuh"

#include <float.h>

#define SVD_SWEEPS 30
#define FULL 0xffffffffu

#define SVD_ROWS 9                  // rows of a lane: h, h + 2, ... of its column (h = lane & 1)

// Sum over the 32 row slots (rows 0..17, then +0) of products t, of which this lane
// holds slots h + 2k: slot i takes t[i] + t[i + off] for off = 16, 8, 4, 2, 1, the
// order the oracle restates; the last addition is the neighbour lane's (IEEE
// addition commutes, so both end with the same bits).
__device__ __forceinline__ float asv_row_sum(const float t[SVD_ROWS])
{
    const float a0 = (t[0] + t[8]) + t[4], a1 = t[1] + t[5], a2 = t[2] + t[6], a3 = t[3] + t[7];
    const float c = (a0 + a2) + (a1 + a3);
    return c + __shfl_xor_sync(FULL, c, 1);
}

__device__ __forceinline__ float asv_row_dot(const float a[SVD_ROWS], const float b[SVD_ROWS])
{
    float t[SVD_ROWS];
#pragma unroll
    for (int k = 0; k < SVD_ROWS; k++) t[k] = a[k] * b[k];
    return asv_row_sum(t);
}

// |ga| <= FLT_EPSILON * sqrtf(q), the rotation test, mostly without the square
// root, which would stand in the chain of every pair: away from the boundary
// (FLT_EPSILON^2 = 2^-46, all roundings below 2^-21) the squares decide
__device__ __forceinline__ bool asv_orthogonal(float ga, float q)
{
    const float g2 = ga * ga, lim = q * 0x1p-46f;
    if (q > 1e-20f && q < 1e30f) {
        if (g2 > lim * (1.0f + 0x1p-18f)) return false;
        if (g2 < lim * (1.0f - 0x1p-18f)) return true;
    }
    return fabsf(ga) <= FLT_EPSILON * sqrtf(q);
}

// Min-norm least squares in FP32 of m rows, two solves per warp.  Lane 2i + h of
// a half: u = rows h, h + 2, ... of column i (zero beyond m, and for i = 6, 7), bl =
// the right-hand side of those rows.  Returns x[0..5] on every lane.
__device__ void asv_lsq_minnorm(int m, float u[SVD_ROWS], const float bl[SVD_ROWS], float x[6])
{
    const int lane = threadIdx.x & 31, base = lane & 17, i = (lane >> 1) & 7;   // base: the half's lane of column 0, this h
    float v[3];                                                // rows h, h + 2, h + 4 of column i of V
#pragma unroll
    for (int k = 0; k < 3; k++) v[k] = i == (lane & 1) + 2 * k ? 1.0f : 0.0f;
    for (int sw = 0; sw <= SVD_SWEEPS; sw++) {                 // the last sweep's last pairs come in one more
        bool any = false;
        for (int c = 1; c <= 6; c++) {
            int j = c - i;
            j = j < 0 ? j + 6 : j;
            if (i > 5) j = i;
            const int src = base + 2 * j;
            float o[SVD_ROWS], vo[3];
#pragma unroll
            for (int k = 0; k < SVD_ROWS; k++) o[k] = __shfl_sync(FULL, u[k], src);
#pragma unroll
            for (int k = 0; k < 3; k++) vo[k] = __shfl_sync(FULL, v[k], src);
            const float own = asv_row_dot(u, u), ga = asv_row_dot(u, o);
            const float other = __shfl_sync(FULL, own, src);
            const bool now = i + j == c ? sw < SVD_SWEEPS : sw > 0;   // of this sweep, else of the one before
            const bool rot = i != j && now && ga != 0.0f && !asv_orthogonal(ga, own * other);
            any |= rot;
            if (!rot) continue;
            const bool first = i < j;                          // this column is p, the other q
            const float zeta = ((first ? other : own) - (first ? own : other)) / (2.0f * ga);
            float t = 1.0f / (fabsf(zeta) + sqrtf(1.0f + zeta * zeta));
            if (zeta < 0.0f) t = -t;
            const float cs = 1.0f / sqrtf(1.0f + t * t), sn = first ? -(cs * t) : cs * t;
#pragma unroll
            for (int k = 0; k < SVD_ROWS; k++) u[k] = cs * u[k] + sn * o[k];
#pragma unroll
            for (int k = 0; k < 3; k++) v[k] = cs * v[k] + sn * vo[k];
        }
        if (!__any_sync(FULL, any) && sw > 0) break;
    }
    const float sig = sqrtf(asv_row_dot(u, u));
    float smax = sig > 0.0f ? sig : 0.0f;
#pragma unroll
    for (int o = 2; o < 16; o <<= 1) smax = fmaxf(smax, __shfl_xor_sync(FULL, smax, o));
    float thr = smax * ((float)(m < 6 ? m : 6) * FLT_EPSILON);
    if (thr < FLT_MIN) thr = FLT_MIN;
    const float ub = asv_row_dot(u, bl);
    const bool keep = sig >= thr;
    const float coef = (ub / sig) / sig;
    float xr[3] = { 0.0f, 0.0f, 0.0f };                        // x[h], x[h + 2], x[h + 4]
#pragma unroll
    for (int k = 0; k < 3; k++) {
        const float term = keep ? v[k] * coef : 0.0f;
#pragma unroll
        for (int j = 0; j < 6; j++) xr[k] = xr[k] + __shfl_sync(FULL, term, base + 2 * j);
    }
#pragma unroll
    for (int r = 0; r < 6; r++) x[r] = __shfl_sync(FULL, xr[r >> 1], (lane & 16) + (r & 1));
}

// symmetric 3x3 eigen-decomposition, cyclic Jacobi
__device__ void asv_sym3_eig(const float M[6], double w[3], double V[3][3])
{
    double a[3][3] = { { M[0], M[1], M[2] }, { M[1], M[3], M[4] }, { M[2], M[4], M[5] } };
    for (int r = 0; r < 3; r++)
        for (int c = 0; c < 3; c++) V[r][c] = r == c ? 1.0 : 0.0;
    const int P[3] = { 0, 0, 1 }, Q[3] = { 1, 2, 2 };
    for (int sw = 0; sw < 50; sw++) {
        int rot = 0;
        for (int k = 0; k < 3; k++) {
            int p = P[k], q = Q[k];
            double apq = a[p][q];
            if (apq == 0.0) continue;
            if (fabs(apq) <= 1e-18 * (fabs(a[p][p]) + fabs(a[q][q]))) continue;
            double th = (a[q][q] - a[p][p]) / (2.0 * apq);
            double t = 1.0 / (fabs(th) + sqrt(th * th + 1.0));
            if (th < 0.0) t = -t;
            double c = 1.0 / sqrt(t * t + 1.0), s = t * c;
            for (int r = 0; r < 3; r++) {
                double ap = a[r][p], aq = a[r][q];
                a[r][p] = c * ap - s * aq;
                a[r][q] = s * ap + c * aq;
            }
            for (int r = 0; r < 3; r++) {
                double ap = a[p][r], aq = a[q][r];
                a[p][r] = c * ap - s * aq;
                a[q][r] = s * ap + c * aq;
            }
            for (int r = 0; r < 3; r++) {
                double vp = V[r][p], vq = V[r][q];
                V[r][p] = c * vp - s * vq;
                V[r][q] = s * vp + c * vq;
            }
            rot++;
        }
        if (!rot) break;
    }
    for (int k = 0; k < 3; k++) w[k] = a[k][k];
}

// error-free transformations (Knuth's TwoSum, the FMA TwoProduct)
__device__ __forceinline__ void asv_two_sum(double a, double b, double &s, double &e)
{
    s = a + b;
    const double bb = s - a;
    e = (a - (s - bb)) + (b - bb);
}

__device__ __forceinline__ void asv_two_prod(double a, double b, double &p, double &e)
{
    p = a * b;
    e = fma(a, b, -p);
}

// Exact "some eigenvalue is negative" test of the symmetric 3x3 matrix M
// (GPU-AS/Image.cpp:997-1006 asks eigenvalues() for a real part < 0): a
// symmetric matrix has no negative eigenvalue iff all its principal minors
// are >= 0.  Products of two floats are exact in double; the determinant's
// five triple products are split into exact (hi, lo) pairs and summed as a
// nonoverlapping expansion (Shewchuk's Grow-Expansion), whose last non-zero
// component carries the exact sign.  Entries that are not finite count as
// no negative eigenvalue.
__device__ int asv_m6_negative(const float M[6])
{
    const double a = M[0], b = M[1], c = M[2], d = M[3], e = M[4], f = M[5];
    if (!(isfinite(a) && isfinite(b) && isfinite(c) && isfinite(d) && isfinite(e) && isfinite(f)))
        return 0;
    if (a < 0.0 || d < 0.0 || f < 0.0) return 1;
    if (a * d < b * b || a * f < c * c || d * f < e * e) return 1;
    double t[10];
    asv_two_prod(a * d, f, t[0], t[1]);                 // a d f
    asv_two_prod(2.0 * (b * c), e, t[2], t[3]);         // 2 b c e
    asv_two_prod(-(a * e), e, t[4], t[5]);              // - a e e
    asv_two_prod(-(d * c), c, t[6], t[7]);              // - d c c
    asv_two_prod(-(f * b), b, t[8], t[9]);              // - f b b
    double x[10];
    int n = 0;
    for (int k = 0; k < 10; k++) {                      // Grow-Expansion
        double q = t[k];
        for (int i = 0; i < n; i++) {
            double h;
            asv_two_sum(q, x[i], q, h);
            x[i] = h;
        }
        x[n++] = q;
    }
    for (int i = n - 1; i >= 0; i--)
        if (x[i] != 0.0) return x[i] < 0.0 ? 1 : 0;
    return 0;
}

// The same, decided in FP32 where the minors are clear of their rounding
// (a two-by-two minor is off by at most 2^-22 of its terms, the determinant by
// 2^-20 of its terms' sum), as they are for nearly every flow: the FP64 test
// of one matrix takes longer than its solve's last sweep.
__device__ int asv_m6_negative_quick(const float M[6])
{
    const float a = M[0], b = M[1], c = M[2], d = M[3], e = M[4], f = M[5];
    const float ad = a * d, bb = b * b, af = a * f, cc = c * c, df = d * f, ee = e * e;
    const float t1 = ad * f, t2 = 2.0f * b * c * e, t3 = a * ee, t4 = d * cc, t5 = f * bb;
    const float sum = fabsf(t1) + fabsf(t2) + fabsf(t3) + fabsf(t4) + fabsf(t5);
    const float least = fminf(fminf(ad + bb, af + cc), fminf(df + ee, sum));
    const float most = fmaxf(fmaxf(fmaxf(a, d), f), fmaxf(fmaxf(fabsf(b), fabsf(c)), fabsf(e)));
    // (the ranges keep what underflows far below the bounds; NaN fails them)
    if (a > 0.0f && d > 0.0f && f > 0.0f && least > 1e-20f && most < 1e8f && sum < 1e30f) {
        const float m1 = ad - bb, m2 = af - cc, m3 = df - ee, det = (t1 + t2) - (t3 + t4 + t5);
        const float e1 = 0x1p-22f * (ad + bb), e2 = 0x1p-22f * (af + cc), e3 = 0x1p-22f * (df + ee), ed = 0x1p-20f * sum;
        if (m1 > e1 && m2 > e2 && m3 > e3 && det > ed) return 0;
        if (m1 < -e1 || m2 < -e2 || m3 < -e3 || det < -ed) return 1;
    }
    return asv_m6_negative(M);
}

__device__ void asv_m6_nearest_psd(const float M[6], float out[6])
{
    double w[3], V[3][3];
    asv_sym3_eig(M, w, V);
    for (int k = 0; k < 3; k++) if (w[k] < 0.0) w[k] = 0.0;
    const int R[6] = { 0, 0, 0, 1, 1, 2 }, C[6] = { 0, 1, 2, 1, 2, 2 };
    for (int e = 0; e < 6; e++) {
        int i = R[e], j = C[e];
        double acc = (V[i][0] * w[0]) * V[j][0];
        acc = acc + (V[i][1] * w[1]) * V[j][1];
        acc = acc + (V[i][2] * w[2]) * V[j][2];
        out[e] = (float)acc;
    }
}

// floor(f + 0.5) of the reference's round (GPU-AS/Image.cpp:901), exactly:
// f + 0.5 can round in FP32, but f - floorf(f) cannot change which side of
// 0.5 the fraction lies on, and the result is the reference's value for every
// float (the +0.0f turns the -0 of f = -0 into +0, as floor(-0 + 0.5) is +0).
__device__ __forceinline__ float asv_round_half_up(float f)
{
    const float r = floorf(f);
    return (f - r >= 0.5f ? r + 1.0f : r) + 0.0f;
}

// matrix_slover (GPU-AS/Image.cpp:874-1009) by sixteen lanes; M valid on every
// lane (its PSD test, :997-1006, is the caller's).  Rows are numbered in the
// reference's order (neighbour y outer, x inner; forward row, then backward).
// Both halves of a warp call it; with active false one has no rows.
__device__ void asv_metric_solve(bool active, const float2 *__restrict__ fwd, const float2 *__restrict__ bwd, int W,
                                 int H, int D, float sx, float sy, int frame, float M[6])
{
    const int h = threadIdx.x & 1, col = (threadIdx.x >> 1) & 7;
    // rows: each in-bounds neighbour in order gives a forward row (unless the last
    // frame) then a backward row (unless the first frame): with both, this lane's
    // rows are all forward or all backward ones, with one, every other neighbour's
    const bool hf = frame != D - 1, hb = frame != 0;     // D >= 2: at least one
    const bool both = hf && hb;
    unsigned inb = 0;
#pragma unroll
    for (int k = 0; k < 9; k++) {
        const int nx = (int)sx + (k % 3 - 1), ny = (int)sy + (k / 3 - 1);
        if (nx >= 0 && nx < W && ny >= 0 && ny < H) inb |= 1u << k;
    }
    if (!active) inb = 0;
    const int m = (both ? 2 : 1) * __popc(inb);
    const bool back = both ? h != 0 : hb;
    const float2 *flow = back ? bwd : fwd;
    unsigned rest = inb;
    if (!both && h) rest &= rest - 1;
    float u[SVD_ROWS], bl[SVD_ROWS];
    float2 f[SVD_ROWS];
    int at[SVD_ROWS];
#pragma unroll
    for (int k = 0; k < SVD_ROWS; k++) {
        at[k] = __ffs(rest) - 1;
        rest &= rest - 1;
        if (!both) rest &= rest - 1;
        f[k] = make_float2(0.0f, 0.0f);
        if (at[k] >= 0)
            f[k] = __ldg(flow + ((long long)frame * H + ((int)sy + at[k] / 3 - 1)) * W + ((int)sx + at[k] % 3 - 1));
    }
#pragma unroll
    for (int k = 0; k < SVD_ROWS; k++) {
        const int ox = at[k] % 3 - 1, oy = at[k] / 3 - 1;
        const float dx = asv_round_half_up(f[k].x) + (float)ox, dy = asv_round_half_up(f[k].y) + (float)oy;
        const float sgn = back ? -2.0f : 2.0f;
        float r = 0.0f;
        if (col == 0) r = dx * dx;
        if (col == 1) r = 2.0f * dx * dy;
        if (col == 2) r = sgn * dx;
        if (col == 3) r = dy * dy;
        if (col == 4) r = sgn * dy;
        if (col == 5) r = 1.0f;
        u[k] = at[k] >= 0 ? r : 0.0f;
        bl[k] = at[k] >= 0 ? (float)(ox * ox + oy * oy + 1) : 0.0f;   // expected_b of :884: 3 2 3 / 2 1 2 / 3 2 3
    }
    asv_lsq_minnorm(m, u, bl, M);
}

// plain reseed flow-angle filter (GPU-AS/Image.cpp:1406-1409): accept iff
// the float cosine c satisfies T <= c <= 1, T the smallest float with
// float(double(acosf(T)) * (180 / 3.141592653)) < 90 (bits 0x328885a3).
// The last frame's flow is the reference's 4x4 zero Mat: read as zero.
__device__ int asv_angle_ok(const float2 *__restrict__ fwd, int W, int H, int D, int frame, int sx,
                            int sy, int nx, int ny)
{
    float sfx = 0.0f, sfy = 0.0f, nfx = 0.0f, nfy = 0.0f;
    if (frame != D - 1) {
        sx = min(max(sx, 0), W - 1);
        sy = min(max(sy, 0), H - 1);
        float2 a = __ldg(fwd + ((long long)frame * H + sy) * W + sx);
        float2 c = __ldg(fwd + ((long long)frame * H + ny) * W + nx);
        sfx = a.x; sfy = a.y; nfx = c.x; nfy = c.y;
    }
    float num = sfx * nfx + sfy * nfy;
    double den = sqrt((double)sfx * (double)sfx + (double)sfy * (double)sfy) *
                 sqrt((double)nfx * (double)nfx + (double)nfy * (double)nfy);
    float c = (float)((double)num / den);
    return (c >= 1.5893254712295857e-08f && c <= 1.0f) ? 1 : 0;
}

__constant__ int c_ringx[ASV_RING] = { -1, 0, 1, -1, 1, -1, 0, 1,
                                       -2, -1, 0, 1, 2, -2, 2, -2, 2, -2, 2, -2, -1, 0, 1, 2 };
__constant__ int c_ringy[ASV_RING] = { -1, -1, -1, 0, 0, 1, 1, 1,
                                       -2, -2, -2, -2, -2, -1, -1, 0, 0, 1, 1, 2, 2, 2, 2, 2 };

struct SeedRef { int si, i, g; };

__device__ __forceinline__ bool asv_seed_ref(const AsvDev &d, int g, SeedRef &r)
{
    if (g >= d.total_seeds) return false;
    r.g = g;
    r.si = asv_find_seg(d.seed_prefix, d.nseg, g);
    r.i = g - d.seed_prefix[r.si];
    return r.i < d.segs[r.si].Kp;
}

// voxel key of a seed position (the memo key of the reseed solve)
__device__ __forceinline__ int asv_seed_key(const SegDesc &S, float4 p)
{
    int frame = min(max((int)p.z, 0), S.D - 1);
    int x = min(max((int)floorf(p.x), 0), S.W - 1), y = min(max((int)floorf(p.y), 0), S.H - 1);
    return (frame * S.H + y) * S.W + x;
}

// neg[g]: 0 = PSD, 1 = non-PSD (fallbacks run), 2 = memo hit (reseed only).
// Which seed positions: reseed 0 -> pos0 (seed_matrix), 1 -> pos (reseed),
// 2 -> pos formed here from the centroid sums (asv_reseed).
__global__ void __launch_bounds__(128) k_metric_self(AsvDev d, int reseed)
{
    asv_follow();
    const bool writer = (threadIdx.x & 15) == 0;
    SeedRef r;
    bool active = asv_seed_ref(d, (blockIdx.x * blockDim.x + threadIdx.x) >> 4, r);
    if (!__any_sync(FULL, active)) return;
    const SegDesc &S = d.segs[active ? r.si : 0];
    float4 p = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    if (active) {
        if (reseed == 2) {
            float q[3], c[3];
            asv_reseed(d, S, r.i, q, c);              // every lane of the half the same
            p = make_float4(q[0], q[1], q[2], (float)r.i);
            if (writer) {
                d.pos[r.g] = p;
                d.slab[r.g] = make_float4(c[0], c[1], c[2], 0.0f);
            }
        } else {
            p = reseed ? d.pos[r.g] : d.pos0[r.g];
        }
        if (reseed && d.mkey[r.g] == asv_seed_key(S, p)) {
            if (writer) d.neg[r.g] = 2;
            active = false;
        }
    }
    if (!__any_sync(FULL, active)) return;
    float fx = floorf(p.x), fy = floorf(p.y);
    int frame = min(max((int)p.z, 0), S.D - 1);   // positions are inside; keep reads in bounds
    float M[6];
    asv_metric_solve(active, d.fwd + S.vox_off, d.bwd + S.vox_off, S.W, S.H, S.D, fx, fy, frame, M);
    if (active && writer) {
#pragma unroll
        for (int e = 0; e < 6; e++) d.Mself[8 * r.g + e] = M[e];
        const int neg = asv_m6_negative_quick(M);
        d.neg[r.g] = neg;
        if (neg) d.neglist[atomicAdd(d.negcount, 1)] = r.g;
    }
}

// a solve per listed seed and ring neighbour
__global__ void __launch_bounds__(128) k_metric_ring(AsvDev d, int reseed)
{
    asv_follow();
    const bool writer = (threadIdx.x & 15) == 0;
    const unsigned step = (gridDim.x * blockDim.x) >> 4, tasks = asv_ring_tasks(*d.negcount);
    for (unsigned task0 = ((blockIdx.x * blockDim.x + threadIdx.x) >> 5) * 2; task0 < tasks; task0 += step) {
        const unsigned task = task0 + ((threadIdx.x >> 4) & 1);   // of this half
        bool active = task < tasks;
        const int g = d.neglist[active ? task / ASV_RING : 0], t = active ? (int)(task % ASV_RING) : 0;
        SeedRef r;
        asv_seed_ref(d, g, r);
        int *ok = d.ringok + asv_ring_at(g, t);
        const SegDesc &S = d.segs[r.si];
        float4 p = reseed ? d.pos[g] : d.pos0[g];
        float fx = floorf(p.x), fy = floorf(p.y);
        int frame = min(max((int)p.z, 0), S.D - 1);
        float nx = fx + (float)c_ringx[t], ny = fy + (float)c_ringy[t];
        const float2 *fwd = d.fwd + S.vox_off, *bwd = d.bwd + S.vox_off;
        if (active && (!(nx >= 0 && nx < S.W && ny >= 0 && ny < S.H) ||
                       (reseed && S.angle_filter &&
                        !asv_angle_ok(fwd, S.W, S.H, S.D, frame, (int)fx, (int)fy, (int)nx, (int)ny)))) {
            if (writer) *ok = 0;
            active = false;
        }
        if (!__any_sync(FULL, active)) continue;
        float M[6];
        asv_metric_solve(active, fwd, bwd, S.W, S.H, S.D, nx, ny, frame, M);
        if (active && writer) {
            float *dst = d.Mring + 8 * asv_ring_at(g, t);
#pragma unroll
            for (int e = 0; e < 6; e++) dst[e] = M[e];
            *ok = asv_m6_negative_quick(M) ? 0 : 1;
        }
    }
}

// the metric of seed g: its own, the mean of a ring's PSD ones, or the nearest
// PSD matrix
__device__ __forceinline__ void asv_metric_result(const AsvDev &d, int g, int neg, float res[6])
{
    float self[6];
    for (int e = 0; e < 6; e++) self[e] = d.Mself[8 * g + e];
    bool done = false;
    if (!neg) {
        for (int e = 0; e < 6; e++) res[e] = self[e];
        done = true;
    }
    // eight neighbours at a time (the 1-ring, then the 2-ring's halves): their
    // flags in two loads, their matrices side by side, summed in order
    float sum[6] = { 0, 0, 0, 0, 0, 0 };
    int n = 0;
    for (int t0 = 0; t0 < ASV_RING && !done; t0 += 8) {
        const int4 *fl = (const int4 *)(d.ringok + asv_ring_at(g, t0));
        const int4 f0 = fl[0], f1 = fl[1];
        const int ok[8] = { f0.x, f0.y, f0.z, f0.w, f1.x, f1.y, f1.z, f1.w };
        float m[8][6];
#pragma unroll
        for (int t = 0; t < 8; t++)
            if (ok[t]) {
                const float *q = d.Mring + 8 * asv_ring_at(g, t0 + t);
                const float4 a = *(const float4 *)q;
                const float2 b = *(const float2 *)(q + 4);
                m[t][0] = a.x; m[t][1] = a.y; m[t][2] = a.z; m[t][3] = a.w; m[t][4] = b.x; m[t][5] = b.y;
            }
#pragma unroll
        for (int t = 0; t < 8; t++)
            if (ok[t]) {
                n++;
                for (int e = 0; e < 6; e++) sum[e] = sum[e] + m[t][e];
            }
        if (t0 != 8 && n > 0) {                      // a whole ring
            for (int e = 0; e < 6; e++) res[e] = sum[e] / (float)n;
            done = true;
        }
    }
    if (!done) asv_m6_nearest_psd(self, res);
}

// Writes M0 (reseed 0) or M (reseed 1, and the memo) and empties the list of
// non-PSD seeds.  draw: also draws the seed for the next flood (d.drawn is
// all -1) and empties the list of the first pass's voxels; clear: and zeroes the
// seed slot's centroid sums.
__global__ void k_metric_combine(AsvDev d, int reseed, bool draw, bool clear)
{
    asv_follow();
    const int g = blockIdx.x * blockDim.x + threadIdx.x;
    if (g == 0) {
        *d.negcount = 0;
        if (draw) *d.tcount = 0;
    }
    if (clear && g < d.total_seeds) {
        ulonglong2 *q = (ulonglong2 *)(d.sums + 8ull * g);
#pragma unroll
        for (int k = 0; k < 4; k++) q[k] = make_ulonglong2(0ull, 0ull);
    }
    SeedRef r;
    if (!asv_seed_ref(d, g, r)) return;
    const SegDesc &S = d.segs[r.si];
    const float4 p = reseed ? d.pos[g] : d.pos0[g];
    const int neg = d.neg[g];
    float res[6];
    if (neg == 2) {
        for (int e = 0; e < 6; e++) res[e] = d.Mmemo[8 * g + e];
    } else {
        asv_metric_result(d, g, neg, res);
        if (reseed) {
            for (int e = 0; e < 6; e++) d.Mmemo[8 * g + e] = res[e];
            d.mkey[g] = asv_seed_key(S, p);
        }
    }
    float *out = (reseed ? d.M : d.M0) + 8 * g;
    for (int e = 0; e < 6; e++) out[e] = res[e];
    if (draw) asv_draw_seed(d, S, g, r.i, p, d.slab[g], res);
}

static void metric_solves(const AsvDev &d, int reseed, bool follow, cudaStream_t st)
{
    const long long solves = d.total_seeds, ring = solves * ASV_RING;             // 8 per block
    asv_launch_follow(follow, k_metric_self, (unsigned)((solves + 7) / 8), 128, 0, st, d, reseed);
    const long long blocks = (ring + 7) / 8;
    asv_launch_follow(true, k_metric_ring, (unsigned)(blocks < 1216 ? blocks : 1216), 128, 0, st, d, reseed);   // 8 blocks per SM at most
}


void asv_launch_metric(const AsvDev &d, int reseed, cudaStream_t st)
{
    metric_solves(d, reseed, false, st);
    asv_launch_follow(true, k_metric_combine, (d.total_seeds + 63) / 64, 64, 0, st, d, reseed, false, false);
}

// The next iteration's seeds: positions from the centroid sums (finalize),
// metrics, draw
void asv_launch_next_seeds(const AsvDev &d, bool finalize, bool clear_sums, bool follow, cudaStream_t st)
{
    metric_solves(d, finalize ? 2 : 1, follow, st);
    asv_launch_follow(true, k_metric_combine, (d.total_seeds + 63) / 64, 64, 0, st, d, 1, true, clear_sums);
}

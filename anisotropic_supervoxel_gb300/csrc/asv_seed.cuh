// asv_seed.cuh -- per-seed steps shared by the volume and the metric kernels:
// the reseed from the centroid sums and the seed draw.  Compiled with
// -fmad=false in both.
#pragma once

#include "asv_common.cuh"

#ifdef __CUDACC__

// ---------------------------------------------------------------------------
// Reseed (aver_exception.vs:22-81).  Alive seed: position floor(mean)+0.5,
// colour = mean LAB.  Dead seed: midpoint of the means of slots id-1 and
// id+1 (id 0 reads texel (W-1, 0); slot Kp is the -1 slot), colour sampled
// at the new position.
// ---------------------------------------------------------------------------
__device__ __forceinline__ void asv_slot_mean(const unsigned long long *sums, int Kp, int slot,
                                              float q[3])
{
    if (slot < 0 || slot > Kp) { q[0] = q[1] = q[2] = 0.0f; return; }
    const unsigned long long *s = sums + 8ull * slot;
    float cnt = __ull2float_rn(s[3]);
#pragma unroll
    for (int a = 0; a < 3; a++) {
        float sf = __ull2float_rn(s[a]) * 0.5f;
        q[a] = ((int)cnt != 0) ? sf / cnt : sf;
    }
}

// position p and colour c of seed `id` of segment S
__device__ __forceinline__ void asv_reseed(const AsvDev &d, const SegDesc &S, int id, float p[3], float c[3])
{
    const unsigned long long *sums = d.sums + 8ull * S.seed_off;
    const unsigned long long *s = sums + 8ull * id;
    if (s[3] != 0) {
        float cnt = __ull2float_rn(s[3]);
#pragma unroll
        for (int a = 0; a < 3; a++) {
            float sf = __ull2float_rn(s[a]) * 0.5f;
            p[a] = floorf(sf / cnt) + 0.5f;
            c[a] = __ull2float_rn(s[4 + a]) / cnt;
        }
    } else {
        float q1[3], q2[3];
        asv_slot_mean(sums, S.Kp, id == 0 ? S.W - 1 : id - 1, q1);
        asv_slot_mean(sums, S.Kp, id + 1, q2);
#pragma unroll
        for (int a = 0; a < 3; a++) p[a] = floorf(0.5f * (q1[a] + q2[a])) + 0.5f;
        int x = min(max((int)floorf(p[0]), 0), S.W - 1);
        int y = min(max((int)floorf(p[1]), 0), S.H - 1);
        int z = min(max((int)floorf(p[2]), 0), S.D - 1);
        uchar4 l = d.lab[S.vox_off + ((long long)z * S.H + y) * S.W + x];
        c[0] = l.x; c[1] = l.y; c[2] = l.z;
    }
}

// The seed's row of the JFA table from its position, colour and metric, and
// the seed record at its voxel (draw_next_seeds.vs), the later seed winning a
// shared one.
__device__ __forceinline__ void asv_draw_seed(const AsvDev &d, const SegDesc &S, int g, int i, float4 p, float4 c,
                                              const float *m)
{
    // table: (-x, -y, -z, -L) (M00, M11, 2M02, 2M12) (2M01, M22, -a, -b),
    // laid out for asv_jfa_dist's paired operations.  v - s == v + (-s) in
    // IEEE arithmetic, and doubling is exact, so
    // (dx*dy)*(2*M01) == ((2*dx)*dy)*M01 (flood.gs:85).
    d.jtab[3 * g + 0] = make_float4(-p.x, -p.y, -p.z, -c.x);
    d.jtab[3 * g + 1] = make_float4(m[0], m[3], 2.0f * m[2], 2.0f * m[4]);
    d.jtab[3 * g + 2] = make_float4(2.0f * m[1], m[5], -c.y, -c.z);
    if (!(p.x >= 0.0f && p.y >= 0.0f && p.z >= 0.0f)) return;
    int x = (int)p.x, y = (int)p.y, z = (int)p.z;
    if (x >= S.W || y >= S.H || z >= S.D) return;
    atomicMax(d.drawn + S.vox_off + ((long long)z * S.H + y) * S.W + x, i);
}

#endif

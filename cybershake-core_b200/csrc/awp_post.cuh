/*
 * awp_post.cuh -- the serial work that ends a time step: source insertion,
 * the fstr redo for moment sources near the surface, the CHKJ sample and the
 * step counter (source.f:812-913, pmcl3d.f:1379-1385, 1478-1479).  Called by
 * k_post and by the last warp of a staged stress sweep, which reads what other
 * SMs have just written: wavefield loads bypass L1 (__ldcg).  Products that
 * feed a sum are rounded on their own in every build (__fmul_rn).
 */
#ifndef AWP_POST_CUH
#define AWP_POST_CUH

#include "awp_stencil.cuh"

__device__ __forceinline__ void fstr_column(const AwpGeom &g, const AwpComp &cp, int i, int j)
{
    const int nz = g.nz, sz = g.plane;
    const int c = g.idx(i, j, nz);
    float *zz = cp.f[AF_ZZ], *xz = cp.f[AF_XZ], *yz = cp.f[AF_YZ];
    zz[c + sz] = -__ldcg(&zz[c]);
    zz[c + 2 * sz] = -__ldcg(&zz[c - sz]);
    xz[c + sz] = -__ldcg(&xz[c - sz]);
    xz[c + 2 * sz] = -__ldcg(&xz[c - 2 * sz]);
    yz[c + sz] = -__ldcg(&yz[c - sz]);
    yz[c + 2 * sz] = -__ldcg(&yz[c - 2 * sz]);
    xz[c] = 0.0f;
    yz[c] = 0.0f;
}

__device__ __forceinline__ float d1_at(const AwpPostArgs &a, int c)
{
    switch (a.media_type) {
    case 1: return __bfloat162float(((const __nv_bfloat16 *)a.d1)[c]);
    case 2: return __half2float(((const __half *)a.d1)[c]) * a.d1_inv;
    default: return ((const float *)a.d1)[c];
    }
}

/* One warp; lane q handles component q and walks its sources in order,
 * as the Fortran loop over j=1,npsrc does.
 * initial != 0: addsrc(1) before the time loop (pmcl3d.f:966-988).
 * otherwise: step n = *step + 1 just finished its stress update:
 *   addsrc(n+1) [and fstr again where a moment source sits in the top three
 *   layers, since pmcl3d.f:1383-1384 inserts before fstr], CHKJ sample,
 *   then *step = n. */
static __device__ __noinline__ void step_post(const AwpPostArgs &a, int initial)
{
    const int q = threadIdx.x & 31;
    const int n = initial ? 0 : (*a.step + 1);
    const int sample = initial ? 1 : n + 1;
    if (q < a.ncomp && sample <= a.nst && !a.kinematic) {
        const AwpSrcDev &s = a.src[q];
        const AwpComp &cp = a.comp[q];
        const AwpGeom &g = a.g;
        const int nz = g.nz, sz = g.plane;
        for (int m = 0; m < s.nsrc; ++m) {
            const int i = s.ijk[3 * m], j = s.ijk[3 * m + 1], k = s.ijk[3 * m + 2];
            const float *t = s.stf + ((int64_t)m * a.nst + (sample - 1)) * 6;
            const float axx = t[0], ayy = t[1], azz = t[2], axz = t[3], ayz = t[4], axy = t[5];
            const int c = g.idx(i, j, k);
            const int ct = g.idx(i, j, nz);
            switch (s.igreen) {
            case -1:
                cp.f[AF_XX][c] = __ldcg(&cp.f[AF_XX][c]) - __fmul_rn(a.vtst, axx);
                cp.f[AF_YY][c] = __ldcg(&cp.f[AF_YY][c]) - __fmul_rn(a.vtst, ayy);
                cp.f[AF_ZZ][c] = __ldcg(&cp.f[AF_ZZ][c]) - __fmul_rn(a.vtst, azz);
                cp.f[AF_XZ][c] = __ldcg(&cp.f[AF_XZ][c]) - __fmul_rn(a.vtst, axz);
                cp.f[AF_YZ][c] = __ldcg(&cp.f[AF_YZ][c]) - __fmul_rn(a.vtst, ayz);
                cp.f[AF_XY][c] = __ldcg(&cp.f[AF_XY][c]) - __fmul_rn(a.vtst, axy);
                break;
            case 1:
                cp.f[AF_U][c] = __ldcg(&cp.f[AF_U][c]) + axx * a.vtst / d1_at(a, c);
                break;
            case 2:
                cp.f[AF_V][c] = __ldcg(&cp.f[AF_V][c]) + ayy * a.vtst / d1_at(a, c);
                break;
            case 3:
                cp.f[AF_W][c] = __ldcg(&cp.f[AF_W][c]) + azz * a.vtst / d1_at(a, c);
                break;
            case -2:
                cp.f[AF_U][c] = __ldcg(&cp.f[AF_U][c]) + axx * a.vtst / d1_at(a, c);
                cp.f[AF_V][c] = __ldcg(&cp.f[AF_V][c]) + ayy * a.vtst / d1_at(a, c);
                cp.f[AF_W][c] = __ldcg(&cp.f[AF_W][c]) + azz * a.vtst / d1_at(a, c);
                break;
            case 4: {
                float *F = cp.f[AF_XZ];
                F[ct] = axx * a.vtst1;
                F[ct + sz] = __fmul_rn(2.0f * axx, a.vtst1) - __ldcg(&F[ct - sz]);
                F[ct + 2 * sz] = __fmul_rn(2.0f * axx, a.vtst1) - __ldcg(&F[ct - 2 * sz]);
            } break;
            case 5: {
                float *F = cp.f[AF_YZ];
                F[ct] = ayy * a.vtst1;
                F[ct + sz] = __fmul_rn(2.0f * ayy, a.vtst1) - __ldcg(&F[ct - sz]);
                F[ct + 2 * sz] = __fmul_rn(2.0f * ayy, a.vtst1) - __ldcg(&F[ct - 2 * sz]);
            } break;
            case 6: {
                float *F = cp.f[AF_ZZ];
                F[ct + sz] = __fmul_rn(2.0f * azz, a.vtst1) - __ldcg(&F[ct]);
                F[ct + 2 * sz] = __fmul_rn(2.0f * azz, a.vtst1) - __ldcg(&F[ct - sz]);
            } break;
            default:
                break;
            }
        }
        if (!initial && s.igreen == -1) {
            for (int m = 0; m < s.nsrc; ++m)
                if (s.ijk[3 * m + 2] >= nz - 2) fstr_column(g, cp, s.ijk[3 * m], s.ijk[3 * m + 1]);
        }
    }
    if (initial) return;
    __syncwarp();
    if (q < a.ncomp && a.probe > 0 && n >= 1 && n <= a.nt) {
        const int c = a.g.idx(a.probe, a.probe, a.probe);
        a.chkj[q][3 * (n - 1)] = __ldcg(&a.comp[q].f[AF_U][c]);
        a.chkj[q][3 * (n - 1) + 1] = __ldcg(&a.comp[q].f[AF_V][c]);
        a.chkj[q][3 * (n - 1) + 2] = __ldcg(&a.comp[q].f[AF_W][c]);
    }
    __syncwarp();
    if (q == 0) *a.step = n;
}

#endif

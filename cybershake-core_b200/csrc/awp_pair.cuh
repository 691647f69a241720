/*
 * awp_pair.cuh -- the staged velocity sweep, two x-adjacent cells per thread.
 *
 * Included by awp_staged.cu inside its anonymous namespace (both builds, with
 * and without multiply-add contraction).  The tile of a block is 32 cells in
 * x and 2 * CW rows: a consumer warp owns two rows, 16 lanes of two cells
 * each, so every tile and array access moves 64 bits per lane and the loop,
 * barrier and address work is shared by two cells (146 M instead of 182 M
 * instructions on 256x256x128 with three components).
 *   - Every value comes through the ring: the planes k+1 / k+2 that the z
 *     differences need arrive as point tiles of their own with level k, so no
 *     consumer waits for a global load inside the level loop.
 *   - A stencil tile has only the rows and columns its differences use.
 *   - Lanes outside the grid compute nothing: their density is zero, and the
 *     slow path of a division by zero would hold up the whole tile.
 * What bounds it: DRAM (5.5 TB/s of algorithmic bytes on 400x400x200 with
 * three components).  Bytes in flight beyond about 110 KB per SM make it
 * slower, not faster: with two blocks of 28 KB slots per SM, three slots a
 * block took 0.87 ms a launch there, four 1.04, two 1.02.  Against one cell
 * per thread (three blocks of a 32 x 8 tile, column values by global loads):
 * 0.99 -> 0.86 ms on 400x400x200 fx+fy+fz, 1.26 -> 1.13 on 500x500x250 fx+fy,
 * 0.113 -> 0.096 on 251x187x93 fx+fy.
 * The per-cell arithmetic is awp_stencil.cuh's, in the same order.
 */

#define PR_X 32                       /* tile width: 16 lanes x 2 cells          */
#define PR_W 40                       /* stencil tile row: 4 + 32 + 4 cells      */

__host__ __device__ constexpr int pr_pad(int n) { return (n + 31) / 32 * 32; }   /* 128-byte tiles */

/* three consecutive media values */
__device__ __forceinline__ void med3(const float *p, float, float m[3])
{
    const float2 a = *(const float2 *)p, b = *(const float2 *)(p + 2);
    m[0] = a.x; m[1] = a.y; m[2] = b.x;
}

__device__ __forceinline__ void med3(const __nv_bfloat16 *p, float, float m[3])
{
    const __nv_bfloat162 a = *(const __nv_bfloat162 *)p;
    m[0] = __low2float(a); m[1] = __high2float(a); m[2] = __bfloat162float(p[2]);
}
__device__ __forceinline__ void med3(const __half *p, float inv, float m[3])
{
    const __half2 a = *(const __half2 *)p;
    m[0] = __low2float(a) * inv; m[1] = __high2float(a) * inv; m[2] = __half2float(p[2]) * inv;
}

__device__ __forceinline__ float2 ld2(const float *p) { return *(const float2 *)p; }

/* the lanes' two cells to global memory (m: how many of them are inside) */
__device__ __forceinline__ void st2(float *p, float a, float b, int m)
{
    if (m == 2) __stwb((float2 *)p, make_float2(a, b));
    else if (m) __stwb(p, a);
}

/* ---- velocity sweep ------------------------------------------------------ */

template <class TM, int CW>
struct PairVelL {
    static constexpr int ROWS = 2 * CW, PT = PR_X * ROWS;
    static constexpr int XX = 0, YY = XX + pr_pad(PR_W * ROWS), XY = YY + PR_X * (ROWS + 3);
    static constexpr int XZ = XY + pr_pad(PR_W * (ROWS + 3)), YZ = XZ + pr_pad(PR_W * ROWS);
    static constexpr int D1 = YZ + PR_X * (ROWS + 3);
    static constexpr int P = D1 + pr_pad((int)(MedRow<TM>::W * (ROWS + 1) * sizeof(TM) + 3) / 4), SLOT = P + 6 * PT;
    static constexpr uint32_t TXB = (uint32_t)((2 * PR_W * ROWS + (PR_W + 2 * PR_X) * (ROWS + 3) + 6 * PT) * 4 +
                                               MedRow<TM>::W * (ROWS + 1) * sizeof(TM));
    static size_t smem(int s) { return 128 + (size_t)s * SLOT * 4 + 2 * 8 * s; }
};

/* stresses around both cells: x rows -2 .. 1 (xx) and -1 .. 2 (xy, xz) from
 * each cell, y rows, and the column */
struct PairStrVals {
    float xx[6], xy[6], xz[6];                   /* offsets -2 .. 3 from the first cell            */
    float2 yy[4], xyy[4], yz[4];                 /* rows -1 0 1 2 | -2 -1 0 1 (0 unused) | -2 -1 0 1 */
    float2 xz_m2, xz_m1, xz_p1, yz_m2, yz_m1, yz_p1, zz_m1, zz_0, zz_p1, zz_p2;
};
template <int S>
struct PairStrCell {
    const PairStrVals &p;
    static __device__ __forceinline__ float pick2(const float2 &a) { return S ? a.y : a.x; }
    __device__ __forceinline__ float s(int a, int dx, int dy, int dz) const
    {
        if (a == S_ZZ) return pick2(dz == -1 ? p.zz_m1 : (dz == 0 ? p.zz_0 : (dz == 1 ? p.zz_p1 : p.zz_p2)));
        if (a == S_XZ && dz) return pick2(dz == -2 ? p.xz_m2 : (dz == -1 ? p.xz_m1 : p.xz_p1));
        if (a == S_YZ && dz) return pick2(dz == -2 ? p.yz_m2 : (dz == -1 ? p.yz_m1 : p.yz_p1));
        if (a == S_XX) return p.xx[2 + S + dx];
        if (a == S_XZ) return p.xz[2 + S + dx];
        if (a == S_YY) return pick2(p.yy[1 + dy]);
        if (a == S_YZ) return pick2(p.yz[2 + dy]);
        return dy ? pick2(p.xyy[2 + dy]) : p.xy[2 + S + dx];
    }
};

__device__ __forceinline__ void ld6(const float *t, float x[6])
{
#pragma unroll
    for (int n = 0; n < 3; ++n) {
        const float2 b = ld2(t + 2 * n - 2);
        x[2 * n] = b.x; x[2 * n + 1] = b.y;
    }
}

template <class TM, int CW, int S, int MINB>
__global__ void __launch_bounds__(32 * (CW + 1), MINB)
k_vel_tma(const __grid_constant__ AwpStagedVelMaps maps, AwpGeom g, AwpCompSet<AWP_MAX_COMP> cs, int ncomp, int qslow,
           const TM *__restrict__ d1, float inv, const float *__restrict__ cx, const float *__restrict__ cy,
           const float *__restrict__ cz, float dth, AwpWork w, int *err, AwpWait wt)
{
    typedef PairVelL<TM, CW> L;
    constexpr int ROWS = L::ROWS, MW = MedRow<TM>::W;
    extern __shared__ unsigned char st_smem[];
    float *ring = ring_base(st_smem);
    uint64_t *full = (uint64_t *)(ring + S * L::SLOT), *empty = full + S;
    __shared__ volatile int abort_s;
    ring_init<S>(full, empty, &abort_s, CW);
    const int tx = threadIdx.x, ty = threadIdx.y;

    if (ty == CW) {                   /* producer warp */
        if (tx != 0) return;
        uint32_t use = 0;
        bool ok = true;
        for (int item = blockIdx.x; ok && item < w.nitems; item += gridDim.x) {
            int q, t;
            split_item(item, ncomp, w.nitems / ncomp, qslow, q, t);
            int bx, by, k0, k1;
            staged_item(g, w, t, bx, by, k0, k1);
            const int j0 = by * ROWS + 1, xp = bx * PR_X + AWP_XO, x = xp - 4;
            for (int k = k0; k <= k1; ++k, ++use) {
                ok = ring_acquire<S>(empty, use, &abort_s, wt.ns);
                if (!ok) break;
                float *sl = ring + (use % S) * L::SLOT;
                uint64_t *b = &full[use % S];
                fence_async_smem();
                mb_expect(b, L::TXB);
                tma_3d(sl + L::XX, &maps.xx[q], b, x, j0 + 1, k + 1);
                tma_3d(sl + L::YY, &maps.yy[q], b, xp, j0, k + 1);
                tma_3d(sl + L::XY, &maps.xy[q], b, x, j0 - 1, k + 1);
                tma_3d(sl + L::XZ, &maps.xz[q], b, x, j0 + 1, k + 1);
                tma_3d(sl + L::YZ, &maps.yz[q], b, xp, j0 - 1, k + 1);
                tma_3d(sl + L::D1, &maps.d1, b, xp, j0, k + 1);
#pragma unroll
                for (int a = 0; a < 6; ++a)
                    tma_3d(sl + L::P + a * L::PT, &maps.p[q][a], b, xp, j0 + 1, k + (a < 3 ? 1 : (a == 3 ? 3 : 2)));
            }
        }
        if (!ok) {
            abort_s = 1;
            atomicOr(err, AWP_KERR_TMA_WAIT);
        }
        ring_drain<S>(full, use, wt.ns);
        return;
    }

    const int sy = g.px, sz = g.plane;
    const int lx = 2 * (tx & 15), row = 2 * ty + (tx >> 4);
    const int cw = row * PR_W + 4 + lx, cp = row * PR_X + lx, cm = (row + 1) * MW + lx;
    uint32_t use = 0;
    for (int item = blockIdx.x; item < w.nitems; item += gridDim.x) {
        int q, t;
        split_item(item, ncomp, w.nitems / ncomp, qslow, q, t);
        int bx, by, k0, k1;
        staged_item(g, w, t, bx, by, k0, k1);
        const int i = bx * PR_X + 1 + lx, j = by * ROWS + 1 + row;
        const int live = j <= g.ny ? max(0, min(2, g.nx - i + 1)) : 0;
        float *U = pick(cs, q, AF_U), *V = pick(cs, q, AF_V), *W = pick(cs, q, AF_W);
        int c = g.idx(i, j, k0);
        const float cyj = live ? cy[j] : 0.f, cxy0 = live ? cx[i] * cyj : 0.f, cxy1 = live == 2 ? cx[i + 1] * cyj : 0.f;
        PairStrVals A;
        float dp[3], dm[2];           /* d1 of plane k-1: the cell's row, the row below */
        A.xz_m2 = A.xz_m1 = A.yz_m2 = A.yz_m1 = A.zz_m1 = A.zz_0 = A.zz_p1 = make_float2(0.f, 0.f);
        dp[0] = dp[1] = dp[2] = dm[0] = dm[1] = 0.f;
        if (live) {
            const float *XZ = pick(cs, q, AF_XZ) + c, *YZ = pick(cs, q, AF_YZ) + c, *ZZ = pick(cs, q, AF_ZZ) + c;
            A.xz_m2 = __ldg((const float2 *)(XZ - 2 * sz)); A.xz_m1 = __ldg((const float2 *)(XZ - sz));
            A.yz_m2 = __ldg((const float2 *)(YZ - 2 * sz)); A.yz_m1 = __ldg((const float2 *)(YZ - sz));
            A.zz_m1 = __ldg((const float2 *)(ZZ - sz)); A.zz_0 = __ldg((const float2 *)ZZ);
            A.zz_p1 = __ldg((const float2 *)(ZZ + sz));
            const TM *d = d1 + c - sz;
#pragma unroll
            for (int n = 0; n < 3; ++n) dp[n] = Store<TM>::ld(d, n, inv);
            dm[0] = Store<TM>::ld(d, -sy, inv); dm[1] = Store<TM>::ld(d, 1 - sy, inv);
        }
#pragma unroll 1
        for (int k = k0; k <= k1; ++k, c += sz, ++use) {
            const float czk = cz[k];
            /* warp-uniform outcome, so a warp leaves together or not at all */
            if (!__all_sync(0xffffffffu, mb_wait_or_abort(&full[use % S], (use / S) & 1, &abort_s, wt.ns))) {
                abort_s = 1;
                atomicOr(err, AWP_KERR_TMA_WAIT);
                return;
            }
            const float *sl = ring + (use % S) * L::SLOT;
            if (live) {               /* lanes outside the grid hold zero density: their divisions would be slow */
            float p0[3], m0[3];
            med3((const TM *)(sl + L::D1) + cm, inv, p0);
            med3((const TM *)(sl + L::D1) + cm - MW, inv, m0);
            float fu[2], fv[2], fw[2];
            vel_factors7(p0[0], m0[0], dp[0], dm[0], p0[1], dp[1], m0[1], dth, fu[0], fv[0], fw[0]);
            vel_factors7(p0[1], m0[1], dp[1], dm[1], p0[2], dp[2], m0[2], dth, fu[1], fv[1], fw[1]);
            ld6(sl + L::XX + cw, A.xx);
            ld6(sl + L::XY + cw + 2 * PR_W, A.xy);
            ld6(sl + L::XZ + cw, A.xz);
#pragma unroll
            for (int n = 0; n < 4; ++n) {
                A.yy[n] = ld2(sl + L::YY + cp + n * PR_X);
                A.yz[n] = ld2(sl + L::YZ + cp + n * PR_X);
            }
            A.xyy[0] = ld2(sl + L::XY + cw); A.xyy[1] = ld2(sl + L::XY + cw + PR_W);
            A.xyy[3] = ld2(sl + L::XY + cw + 3 * PR_W);
            const float *P = sl + L::P + cp;
            const float2 u0 = ld2(P), v0 = ld2(P + L::PT), w0 = ld2(P + 2 * L::PT);
            A.zz_p2 = ld2(P + 3 * L::PT); A.xz_p1 = ld2(P + 4 * L::PT); A.yz_p1 = ld2(P + 5 * L::PT);
            float u[2], v[2], w_[2];
            vel_one_t(PairStrCell<0>{A}, u0.x, v0.x, w0.x, fu[0], fv[0], fw[0], u[0], v[0], w_[0]);
            vel_one_t(PairStrCell<1>{A}, u0.y, v0.y, w0.y, fu[1], fv[1], fw[1], u[1], v[1], w_[1]);
            const float crj0 = cxy0 * czk, crj1 = cxy1 * czk;
            st2(U + c, u[0] * crj0, u[1] * crj1, live);
            st2(V + c, v[0] * crj0, v[1] * crj1, live);
            st2(W + c, w_[0] * crj0, w_[1] * crj1, live);
            A.xz_m2 = A.xz_m1; A.xz_m1 = make_float2(A.xz[2], A.xz[3]);
            A.yz_m2 = A.yz_m1; A.yz_m1 = A.yz[2];
            A.zz_m1 = A.zz_0; A.zz_0 = A.zz_p1; A.zz_p1 = A.zz_p2;
#pragma unroll
            for (int n = 0; n < 3; ++n) dp[n] = p0[n];
            dm[0] = m0[0]; dm[1] = m0[1];
            }
            __syncwarp();
            if (tx == 0) mb_arrive(&empty[use % S]);
        }
    }
}

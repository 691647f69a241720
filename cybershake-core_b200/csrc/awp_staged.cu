/*
 * awp_staged.cu -- the two-sweep stepper with TMA-staged xy tiles (2.5D blocking).
 *
 * A thread block owns a 32 x 8 column tile (the velocity sweep, awp_pair.cuh:
 * 32 x 16) and marches up a chunk of z levels, of one component or (stress
 * sweep) of all of them.  A producer warp issues, for every level, TMA tile
 * loads (cp.async.bulk.tensor over 3D tensor maps of the padded volume) into a
 * ring of shared-memory slots ahead of the level being computed: stencil tiles
 * with a halo, media tiles with the row below, and the point-wise state
 * without.  A "full" mbarrier per slot counts the bytes in; the consumer warps
 * release a slot through its "empty" mbarrier.  The stress sweep's values
 * along the cell's own column (z neighbours) travel in per-thread register
 * queues, loaded one level ahead; the velocity sweep's come through the ring.
 * Results are written with coalesced stores.  The bytes in flight per SM are set by the
 * ring depth, not by registers or resident warps.
 *
 * Work items (x tile, y tile, z chunk, component) are spread over a
 * persistent grid, one component after the other or the components of a
 * tile side by side (split_item).
 *
 * The per-cell arithmetic is the shared code of awp_stencil.cuh, evaluated in
 * the same order as the other steppers (bit-identical results), for every
 * storage of the media (FP32, bf16, scaled binary16) and of the memory
 * variables (FP32, bf16, block floating point).
 *
 * Every wait on an mbarrier is bounded (2 s of %globaltimer); on expiry the
 * block records AWP_KERR_TMA_WAIT in the error word and its warps leave; the
 * producer first waits (bounded again) for its own copies in flight.
 */
#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>
#include <stdlib.h>
#include <string.h>

#include "../../include/awp_sgt.h"
#include "awp_internal.h"
#include "awp_kernels.h"
#include "awp_stencil.cuh"
#include "awp_post.cuh"

#define ST_X 32                      /* tile width: one warp along x            */
#define ST_Y 8                       /* tile rows                               */
#define ST_W 40                      /* staged row: 4 halo + 32 + 4 halo        */
#define ST_HR (ST_Y + 4)             /* stencil tile rows: 2 below, 2 above     */
#define ST_MR (ST_Y + 1)             /* media tile rows: 1 below                */
#define ST_VT (ST_W * ST_HR)         /* floats of a stencil tile (1920 B)       */
#define ST_MP 384                    /* floats reserved per media tile (1536 B) */
#define ST_PT (ST_X * ST_Y)          /* floats of a point tile (no halo)        */

/* bound of every barrier wait (the solver's setting, 2 s by default) and the
 * test-only injection of AwpStepArgs::withhold */
struct AwpWait {
    unsigned long long ns;
    int withhold;
};

struct AwpStagedStrMaps {
    CUtensorMap v[AWP_MAX_COMP][3];  /* u v w, box 40 x 12                     */
    CUtensorMap med[4];              /* lam mu qp qs, box W x 9 (MedRow)       */
    CUtensorMap s[AWP_MAX_COMP][6];  /* xx yy zz xy xz yz, box 32 x 8          */
    CUtensorMap r[AWP_MAX_COMP][6];  /* r1..r6 (FP32, bf16 or int16), box 32 x 8 */
    CUtensorMap rx[AWP_MAX_COMP];    /* exponent words of block floating point r */
};
/* tensor maps of the velocity sweep with two cells per thread (awp_pair.cuh) */
struct AwpStagedVelMaps {
    CUtensorMap xx[AWP_MAX_COMP];     /* box 40 x rows                           */
    CUtensorMap yy[AWP_MAX_COMP];     /* box 32 x (rows + 3)                     */
    CUtensorMap xy[AWP_MAX_COMP];     /* box 40 x (rows + 3)                     */
    CUtensorMap xz[AWP_MAX_COMP];     /* box 40 x rows                           */
    CUtensorMap yz[AWP_MAX_COMP];     /* box 32 x (rows + 3)                     */
    CUtensorMap d1;                   /* box W x (rows + 1)                      */
    CUtensorMap p[AWP_MAX_COMP][6];   /* u v w (plane k), zz xz yz (planes k+2 k+1 k+1), box 32 x rows */
};
#define PR_VEL_CW 8                  /* its consumer warps                      */

struct AwpStaged {
    AwpStagedStrMaps sm;
    AwpStagedVelMaps vm;
};

/* The kernels live in an anonymous namespace: this file is compiled twice,
 * without (the bit-exact stepper) and with multiply-add contraction
 * (AWP_STAGED_FMA: AWP_KERNEL_STAGED_FMA), and the two sets must not merge. */
namespace {

/* ------------------------------------------------------------------ */
/* mbarrier / TMA primitives (PTX ISA: mbarrier, cp.async.bulk.tensor) */
/* ------------------------------------------------------------------ */

__device__ __forceinline__ uint32_t s_addr(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mb_init(uint64_t *b, uint32_t count)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(s_addr(b)), "r"(count) : "memory");
}

__device__ __forceinline__ void mb_fence_init() { asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory"); }

__device__ __forceinline__ void mb_expect(uint64_t *b, uint32_t bytes)
{
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(s_addr(b)), "r"(bytes) : "memory");
}

__device__ __forceinline__ bool mb_try(uint64_t *b, uint32_t parity)
{
    uint32_t ok;
    asm volatile("{\n\t.reg .pred p;\n\t"
                 "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
                 "selp.u32 %0, 1, 0, p;\n\t}"
                 : "=r"(ok)
                 : "r"(s_addr(b)), "r"(parity)
                 : "memory");
    return ok != 0;
}

__device__ __forceinline__ uint64_t global_ns()
{
    uint64_t t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

/* true once the phase of the given parity has completed; false after the bound */
__device__ __forceinline__ bool mb_wait(uint64_t *b, uint32_t parity, uint64_t limit_ns)
{
    if (mb_try(b, parity)) return true;
    const uint64_t t0 = global_ns();
    for (uint32_t n = 0; n < (1u << 26); ++n) {
        if (mb_try(b, parity)) return true;
        if ((n & 63) == 63 && global_ns() - t0 > limit_ns) return false;
    }
    return false;
}

/* generic-proxy accesses to a slot are ordered before the async-proxy refill */
__device__ __forceinline__ void fence_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

__device__ __forceinline__ void tma_3d(void *dst, const CUtensorMap *map, uint64_t *b, int x, int y, int z)
{
    asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes"
                 " [%0], [%1, {%2, %3, %4}], [%5];" ::"r"(s_addr(dst)),
                 "l"((uint64_t)map), "r"(x), "r"(y), "r"(z), "r"(s_addr(b))
                 : "memory");
}

/* memory coordinates of a tile: column of cell i0 - 4 (a multiple of 4, so
 * the copy starts on a 16-byte boundary), row of cell j0 - 2 (stencil) or
 * j0 - 1 (media), level k */
__device__ __forceinline__ int tile_x(int i0) { return i0 + AWP_XO - 1 - 4; }

/* tile and levels of a work item: nzc chunks that differ by a level at most */
__device__ __forceinline__ void staged_item(const AwpGeom &g, const AwpWork &w, int item, int &bx, int &by, int &k0,
                                            int &k1)
{
    bx = item % w.ntx;
    const int t = item / w.ntx;
    by = t % w.nty;
    const int bz = t / w.nty;
    k0 = bz * g.nz / w.nzc + 1;
    k1 = (bz + 1) * g.nz / w.nzc;
}

/* component q and tile item t of work item `item`: the components of one
 * tile side by side (qslow = 0; their common media tiles come from L2) or one
 * component over all tiles at a time (qslow = 1; fewer arrays streamed at once) */
__device__ __forceinline__ void split_item(int item, int ncomp, int ntile, int qslow, int &q, int &t)
{
    if (qslow) {
        q = item / ntile;
        t = item - q * ntile;
    } else {
        q = item % ncomp;
        t = item / ncomp;
    }
}

__device__ __forceinline__ float *pick(const AwpCompSet<AWP_MAX_COMP> &cs, int q, int f)
{
    return q == 0 ? cs.c[0].f[f] : (q == 1 ? cs.c[1].f[f] : cs.c[2].f[f]);
}

/* ------------------------------------------------------------------ */
/* warp roles and the ring                                             */
/* ------------------------------------------------------------------ */

/* media tile row of storage type TM, from cell i0 on (the averages reach one
 * cell up in x, none down): a multiple of 16 bytes */
template <class TM> struct MedRow { static constexpr int W = 40; };
template <> struct MedRow<float> { static constexpr int W = 36; };
template <class TM>
__host__ __device__ constexpr int med_bytes(int rows) { return MedRow<TM>::W * rows * (int)sizeof(TM); }

/* Eight consumer warps (one tile row each) and one producer warp whose lane
 * 0 issues the copies.  Ring slot s has a "full" barrier (the producer's
 * expect_tx arrival plus the bytes) and an "empty" barrier (one arrival per
 * consumer warp once it is done with the slot's level); the producer refills
 * a slot only after its empty phase completes, so no block-wide barrier
 * stands in the level loop and warps drift within the ring depth. */
#define ST_CW 8
#define ST_THREADS (32 * (ST_CW + 1))

__device__ __forceinline__ void mb_arrive(uint64_t *b)
{
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(s_addr(b)) : "memory");
}

/* bounded wait that also gives up once another thread has flagged an abort */
__device__ __forceinline__ bool mb_wait_or_abort(uint64_t *b, uint32_t parity, const volatile int *abort,
                                                 uint64_t limit_ns)
{
    if (mb_try(b, parity)) return true;
    const uint64_t t0 = global_ns();
    for (uint32_t n = 0; n < (1u << 26); ++n) {
        if (mb_try(b, parity)) return true;
        if ((n & 63) == 63 && (*abort || global_ns() - t0 > limit_ns)) return false;
    }
    return false;
}

/* the ring starts at the first 128-byte boundary of the dynamic shared
 * memory; the pad is added to the shared pointer itself (no round trip
 * through an integer), so the compiler keeps knowing the ring is shared
 * memory and reads its tiles with shared-memory loads, not generic ones */
__device__ __forceinline__ float *ring_base(unsigned char *raw)
{
    const unsigned pad = (unsigned)(-(uintptr_t)raw) & 127u;
    return (float *)(raw + pad);
}

template <int S>
__device__ __forceinline__ void ring_init(uint64_t *full, uint64_t *empty, volatile int *abort, int consumers = ST_CW)
{
    if (threadIdx.x == 0 && threadIdx.y == 0) {
        for (int s = 0; s < S; ++s) {
            mb_init(&full[s], 1);
            mb_init(&empty[s], consumers);
        }
        mb_fence_init();
        *abort = 0;
    }
    __syncthreads();
}

/* the producer's last act: the most recent use of every slot has landed, so
 * no copy into this block's shared memory is still in flight when it exits
 * (`skip`: a use it issued nothing for) */
template <int S>
__device__ __forceinline__ void ring_drain(uint64_t *full, uint32_t uses, uint64_t limit_ns, uint32_t skip = 0xffffffffu)
{
    for (uint32_t u = uses > (uint32_t)S ? uses - S : 0; u < uses; ++u)
        if (u != skip && !mb_wait(&full[u % S], (u / S) & 1, limit_ns)) return;
}

/* the ring use block 0's producer withholds under the test injection */
__device__ __forceinline__ uint32_t withheld_use(const AwpWait &wt)
{
    return blockIdx.x == 0 && wt.withhold >= 0 ? (uint32_t)wt.withhold : 0xffffffffu;
}

/* producer: wait until use `use` of its slot may be refilled */
template <int S>
__device__ __forceinline__ bool ring_acquire(uint64_t *empty, uint32_t use, const volatile int *abort,
                                             uint64_t limit_ns)
{
    return use < (uint32_t)S || mb_wait_or_abort(&empty[use % S], ((use / S) - 1) & 1, abort, limit_ns);
}

/* ------------------------------------------------------------------ */
/* stress sweep                                                        */
/* ------------------------------------------------------------------ */

/* Slot layout (floats): u v w stencil tiles, lam mu qp qs media tiles, the
 * six stresses and the six memory variables of the tile (32 x 8 each; the
 * memory variables in their storage type).  Levels k-1 and k are in use
 * while level k+1 is in flight. */
#define STR_D 1
#define STR_ST (3 * ST_VT + 4 * ST_MP)           /* first stress tile        */
#define STR_SLOT (STR_ST + 12 * ST_PT)           /* r tiles fit in 6 x 256   */

/* the six stresses of a cell, times the sponge factor, to global memory
 * (the array pointers come from a shared-memory table) */
__device__ __forceinline__ void gst6(const AwpComp &o, int c, const Stress6 &s, float crj)
{
    __stwb(o.f[AF_XX] + c, s.xx * crj); __stwb(o.f[AF_YY] + c, s.yy * crj); __stwb(o.f[AF_ZZ] + c, s.zz * crj);
    __stwb(o.f[AF_XY] + c, s.xy * crj); __stwb(o.f[AF_XZ] + c, s.xz * crj); __stwb(o.f[AF_YZ] + c, s.yz * crj);
}

template <class TM>
struct TMed {
    const float *p0, *pm; /* media tiles (lam first) of planes k and k-1 */
    int c;                /* the cell in a tile */
    const AwpMediaScale &sc;
    __device__ __forceinline__ float m(int a, int dx, int dy, int dz) const
    {
        const int n = a == AM_LAM ? 0 : (a == AM_MU ? 1 : (a == AM_QP ? 2 : 3));
        return Store<TM>::ld((const TM *)((dz == 0 ? p0 : pm) + n * ST_MP), c + dy * MedRow<TM>::W + dx, sc.inv[a]);
    }
};

/* velocities: plane k from the slot, the column from registers */
struct TVel {
    const float *t;   /* u tile of plane k at the cell; v and w tiles follow */
    float um1, vm1, wm1, up1, up2, vp1, vp2, wm2, wp1;
    __device__ __forceinline__ float u(int dx, int dy, int dz) const
    {
        return dz == 0 ? t[dy * ST_W + dx] : (dz == -1 ? um1 : (dz == 1 ? up1 : up2));
    }
    __device__ __forceinline__ float v(int dx, int dy, int dz) const
    {
        return dz == 0 ? t[ST_VT + dy * ST_W + dx] : (dz == -1 ? vm1 : (dz == 1 ? vp1 : vp2));
    }
    __device__ __forceinline__ float w(int dx, int dy, int dz) const
    {
        return dz == 0 ? t[2 * ST_VT + dy * ST_W + dx] : (dz == -1 ? wm1 : (dz == -2 ? wm2 : wp1));
    }
};

/* the memory-variable tiles of a slot by storage type: element size, tile
 * count (block floating point adds the tile of exponent words) and the six
 * values of the cell at point-tile offset cp */
template <class TR>
struct RTile {
    static constexpr int size = (int)sizeof(TR), ntiles = 6;
    static __device__ __forceinline__ void ld(const unsigned char *base, int cp, float r[6])
    {
#pragma unroll
        for (int a = 0; a < 6; ++a) r[a] = Store<TR>::ld((const TR *)base + cp, a * ST_PT, 1.0f);
    }
};
template <>
struct RTile<RBfp> {
    static constexpr int size = 2, ntiles = 7;
    static __device__ __forceinline__ void ld(const unsigned char *base, int cp, float r[6])
    {
        bfp_load6((const short *)base + cp, ST_PT, ((const unsigned short *)base)[6 * ST_PT + cp], r);
    }
};

/* bytes one level brings in (rtile_bytes: its r tiles) */
template <class TM>
__host__ __device__ __forceinline__ uint32_t str_txb(int nve, int rtile_bytes)
{
    return (uint32_t)((3 * ST_VT + 6 * ST_PT) * 4 + (nve == 1 ? 4 : 2) * med_bytes<TM>(ST_MR) + (nve == 1 ? rtile_bytes : 0));
}

/* issues the r tiles of component q at a point-tile position */
template <class TR>
__device__ __forceinline__ void r_issue(const AwpStagedStrMaps &maps, int q, unsigned char *rb, uint64_t *b, int xp,
                                        int y, int z)
{
#pragma unroll
    for (int a = 0; a < 6; ++a) tma_3d(rb + a * ST_PT * RTile<TR>::size, &maps.r[q][a], b, xp, y, z);
    if (RTile<TR>::ntiles == 7) tma_3d(rb + 6 * ST_PT * RTile<TR>::size, &maps.rx[q], b, xp, y, z);
}

template <int S, class TM, class TR>
__device__ __forceinline__ void str_issue(const AwpStagedStrMaps &maps, int q, int nve, float *ring, uint64_t *full,
                                          uint32_t use, int i0, int j0, int k)
{
    float *sl = ring + (use % S) * STR_SLOT;
    uint64_t *b = &full[use % S];
    fence_async_smem();
    mb_expect(b, str_txb<TM>(nve, RTile<TR>::ntiles * ST_PT * RTile<TR>::size));
    const int x = tile_x(i0);
#pragma unroll
    for (int a = 0; a < 3; ++a) tma_3d(sl + a * ST_VT, &maps.v[q][a], b, x, j0 - 1, k + 1);
    const int nmed = nve == 1 ? 4 : 2;
    /* media and point tiles start at cell i0: memory column i0 + 7 (a multiple of 8) */
    const int xp = i0 + AWP_XO - 1;
    for (int a = 0; a < nmed; ++a) tma_3d(sl + 3 * ST_VT + a * ST_MP, &maps.med[a], b, xp, j0, k + 1);
#pragma unroll
    for (int a = 0; a < 6; ++a) tma_3d(sl + STR_ST + a * ST_PT, &maps.s[q][a], b, xp, j0 + 1, k + 1);
    if (nve == 1) r_issue<TR>(maps, q, (unsigned char *)(sl + STR_ST + 6 * ST_PT), b, xp, j0 + 1, k + 1);
}

/* ---- the ends of a stress sweep ------------------------------------------ */

/* Free-surface velocities of one column (fvelxy and fvelz, operator.f:246-306;
 * k_fsvel's expressions).  Only the column's own stress update reads them (the
 * z differences at k = nz-2 .. nz), so the thread that owns the column in the
 * top chunk writes them before its levels and reads them back itself; a launch
 * of their own cost about 3 us a step. */
template <class TM>
__device__ __forceinline__ void fs_velocity(const AwpGeom &g, float *u1, float *v1, float *w1, const TM *lam, const TM *mu,
                                            const AwpMediaScale &sc, int i, int j)
{
    const int c = g.idx(i, j, g.nz), sy = g.px, sz = g.plane;
    const float xl = 1.0f / Store<TM>::ld(lam, c, sc.inv[AM_LAM]);
    const float xl2m = 2.0f / Store<TM>::ld(mu, c, sc.inv[AM_MU]) + xl;
    const float u_fs = u1[c] - (w1[c] - w1[c - 1]);
    const float v_fs = v1[c] - (w1[c + sy] - w1[c]);
    const float u_fs_e = (i + 1 <= g.nx) ? (u1[c + 1] - (w1[c + 1] - w1[c])) : 0.0f;
    const float v_fs_s = (j - 1 >= 1) ? (v1[c - sy] - (w1[c] - w1[c - sy])) : 0.0f;
    const float w_fs = w1[c - sz] - __fmul_rn(xl / xl2m, (u_fs_e - u_fs) + (u1[c + 1] - u1[c]) + (v_fs - v_fs_s) + (v1[c] - v1[c - sy]));
    u1[c + sz] = u_fs;
    v1[c + sz] = v_fs;
    w1[c + sz] = w_fs;
}

/* What a stress sweep does besides: the media arrays of fs_velocity, and the
 * step's serial work once all its warps are done (done: their count, back at
 * zero for the next launch; NULL: left to k_post). */
struct StrEnds {
    const void *lam, *mu;
    int *done;
    AwpPostArgs post;
};

/* the last of the grid's `warps` consumer warps runs step_post */
__device__ __forceinline__ void str_finish(const StrEnds &e, int warps)
{
    if (!e.done) return;
    __threadfence();                  /* this lane's stores before the count */
    __syncwarp();
    int n = 0;
    if ((threadIdx.x & 31) == 0) n = atomicAdd(e.done, 1);
    if (__shfl_sync(0xffffffffu, n, 0) != warps - 1) return;
    __syncwarp();                     /* lane 0's count before every lane's loads (a shuffle orders no memory) */
    __threadfence();
    step_post(e.post, 0);
    if ((threadIdx.x & 31) == 0) *e.done = 0;
}

/* work items: (x tile, y tile, z chunk, component); see split_item for the order.
 * RPT rows of the tile per consumer thread (ST_Y / RPT consumer warps): with
 * RPT = 2 a thread carries two independent cells per level. */
template <class TM, class TR, int UNR, int RPT>
__global__ void __launch_bounds__(32 * (ST_Y / RPT + 1), 3)
k_str_tma(const __grid_constant__ AwpStagedStrMaps maps, AwpGeom g, AwpCompSet<AWP_MAX_COMP> cs, int ncomp, int qslow,
          const float *__restrict__ cx, const float *__restrict__ cy, const float *__restrict__ cz,
          const float *__restrict__ tau, float dth, float dt, float dh1, AwpWork w, int nve, const __grid_constant__ AwpMediaScale sc, int *err, AwpWait wt,
          const __grid_constant__ StrEnds ends)
{
    constexpr int S = 2 + STR_D;      /* levels k-1 and k in use, STR_D in flight */
    constexpr int CW = ST_Y / RPT;    /* consumer warps */
    extern __shared__ unsigned char st_smem[];
    float *ring = ring_base(st_smem);
    uint64_t *full = (uint64_t *)(ring + S * STR_SLOT), *empty = full + S;
    __shared__ volatile int abort_s;
    __shared__ AwpComp tab[AWP_MAX_COMP];
    if (threadIdx.y == 0 && threadIdx.x < AWP_MAX_COMP) {
#pragma unroll
        for (int f = 0; f < AWP_NF_ARRAYS; ++f) tab[threadIdx.x].f[f] = pick(cs, threadIdx.x, f);
    }
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
            for (int k = k0 - 1; k <= k1; ++k, ++use) {
                ok = ring_acquire<S>(empty, use, &abort_s, wt.ns);
                if (!ok) break;
                if (use == withheld_use(wt)) continue;   /* test injection: nothing issued, no arrival */
                str_issue<S, TM, TR>(maps, q, nve, ring, full, use, bx * ST_X + 1, by * ST_Y + 1, k);
            }
        }
        if (!ok) {
            abort_s = 1;
            atomicOr(err, AWP_KERR_TMA_WAIT);
        }
        ring_drain<S>(full, use, wt.ns, withheld_use(wt));
        return;
    }

    const int sz = g.plane, sy = g.px;
    uint32_t use0 = 0;                /* ring use of the item's first level */
    for (int item = blockIdx.x; item < w.nitems; item += gridDim.x) {
        int q, t;
        split_item(item, ncomp, w.nitems / ncomp, qslow, q, t);
        int bx, by, k0, k1;
        staged_item(g, w, t, bx, by, k0, k1);
        const int i = bx * ST_X + 1 + tx;
        const int np = k1 - k0 + 2;   /* levels k0-1 .. k1 */
        float *U = tab[q].f[AF_U], *V = tab[q].f[AF_V], *W = tab[q].f[AF_W];
        /* per row: column queues u, v at k+1, k+2 (k+3 loaded one level ahead), w at k-2, k+1 (k+2 ahead) */
        float up1[RPT], up2[RPT], vp1[RPT], vp2[RPT], wm2[RPT], wp1[RPT], cxy[RPT];
        bool live[RPT];
        int itxy[RPT];
        const int c0 = g.idx(i, by * ST_Y + 1 + ty, k0);
#pragma unroll
        for (int r = 0; r < RPT; ++r) {
            const int j = by * ST_Y + 1 + ty + r * CW, c = c0 + r * CW * sy;
            live[r] = i <= g.nx && j <= g.ny;
            itxy[r] = ((j & 1) << 1) | (i & 1);
            up1[r] = up2[r] = vp1[r] = vp2[r] = wm2[r] = wp1[r] = cxy[r] = 0.f;
            if (live[r]) {
                if (k1 == g.nz)
                    fs_velocity(g, U, V, W, (const TM *)ends.lam, (const TM *)ends.mu, sc, i, j);
                up1[r] = __ldg(&U[c + sz]); up2[r] = __ldg(&U[c + 2 * sz]);
                vp1[r] = __ldg(&V[c + sz]); vp2[r] = __ldg(&V[c + 2 * sz]);
                wm2[r] = __ldg(&W[c - 2 * sz]); wp1[r] = __ldg(&W[c + sz]);
                cxy[r] = cx[i] * cy[j];
            }
        }
        int cc = c0;
#pragma unroll (UNR)
        for (int k = k0; k <= k1; ++k, cc += sz) {
            const uint32_t use = use0 + (uint32_t)(k - k0 + 1), usem = use - 1;
            float up3[RPT], vp3[RPT], wp2[RPT];
            const float czk = cz[k];
#pragma unroll
            for (int r = 0; r < RPT; ++r) {
                const int c = cc + r * CW * sy;
                up3[r] = vp3[r] = wp2[r] = 0.f;
                if (live[r] && k < k1) { up3[r] = __ldcg(&U[c + 3 * sz]); vp3[r] = __ldcg(&V[c + 3 * sz]); wp2[r] = __ldcg(&W[c + 2 * sz]); }
            }
            bool ok = true;
            if (k == k0) ok = mb_wait_or_abort(&full[usem % S], (usem / S) & 1, &abort_s, wt.ns);
            if (ok) ok = mb_wait_or_abort(&full[use % S], (use / S) & 1, &abort_s, wt.ns);
            if (!__all_sync(0xffffffffu, ok)) {   /* warp-uniform outcome */
                abort_s = 1;
                atomicOr(err, AWP_KERR_TMA_WAIT);
                return;
            }
            const float *sk = ring + (use % S) * STR_SLOT, *sm = ring + (usem % S) * STR_SLOT;
            const int ipar = ((g.nz + 1 - k) & 1) << 2;                    /* viscoop.f:93-101 */
#pragma unroll
            for (int r = 0; r < RPT; ++r) {
                const int row = ty + r * CW, c = cc + r * CW * sy;
                const int cv = (row + 2) * ST_W + tx + 4, cm = (row + 1) * MedRow<TM>::W + tx, cp = row * ST_X + tx;
                const float wm1 = sm[2 * ST_VT + cv];
                if (live[r]) {
                    const int it = ipar | itxy[r];
                    const TMed<TM> M{sk + 3 * ST_VT, sm + 3 * ST_VT, cm, sc};
                    const StrCoef kc = str_coef_t(M, nve, tau[it], tau[8 + it]);
                    const float *ps = sk + STR_ST + cp;
                    const Stress6 s0{ps[0], ps[ST_PT], ps[2 * ST_PT], ps[3 * ST_PT], ps[4 * ST_PT], ps[5 * ST_PT]};
                    const TVel Vq{sk + cv, sm[cv], sm[ST_VT + cv], wm1, up1[r], up2[r], vp1[r], vp2[r], wm2[r], wp1[r]};
                    Stress6 o;
                    if (nve == 1) {
                        float rr[6];
                        RTile<TR>::ld((const unsigned char *)(sk + STR_ST + 6 * ST_PT), cp, rr);
                        const VelDiff dd = vel_diff(Vq);
                        o = str_visco(kc, dd, s0, rr, dth, dt, dh1);
                        RVars<TR>::st(tab[q], c, rr);
                    } else {
                        o = str_elastic(kc, Vq, s0, dth);
                    }
                    const float crj = cxy[r] * czk;
                    gst6(tab[q], c, o, crj);
                }
                up1[r] = up2[r]; up2[r] = up3[r];
                vp1[r] = vp2[r]; vp2[r] = vp3[r];
                wm2[r] = wm1; wp1[r] = wp2[r];
            }
            __syncwarp();
            if (tx == 0) mb_arrive(&empty[usem % S]);
        }
        __syncwarp();
        if (tx == 0) mb_arrive(&empty[(use0 + np - 1) % S]);
        use0 += np;
        if (k1 == g.nz) {
#pragma unroll
            for (int r = 0; r < RPT; ++r) {
                if (!live[r]) continue;
                /* fstr (operator.f:594-606) on this thread's own column; the top
                 * chunk holds at least levels nz-2..nz, all written by this thread */
                const int ct = g.idx(i, by * ST_Y + 1 + ty + r * CW, g.nz);
                float *ZZ = tab[q].f[AF_ZZ], *XZ = tab[q].f[AF_XZ], *YZ = tab[q].f[AF_YZ];
                ZZ[ct + sz] = -__ldcg(&ZZ[ct]);
                ZZ[ct + 2 * sz] = -__ldcg(&ZZ[ct - sz]);
                XZ[ct + sz] = -__ldcg(&XZ[ct - sz]);
                XZ[ct + 2 * sz] = -__ldcg(&XZ[ct - 2 * sz]);
                YZ[ct + sz] = -__ldcg(&YZ[ct - sz]);
                YZ[ct + 2 * sz] = -__ldcg(&YZ[ct - 2 * sz]);
                XZ[ct] = 0.0f;
                YZ[ct] = 0.0f;
            }
        }
    }
    str_finish(ends, gridDim.x * CW);
}

/* ---- components side by side in one work item -------------------------- */

/* A work item is (x tile, y tile, z chunk) with every component.  The media
 * tiles of a level, and the cell coefficients computed from them (the 8-cell
 * sums and the five divisions), serve all components: the media ring (levels
 * k-1 and k in use, k+1 in flight) is filled once per level.  The components'
 * tiles follow in a ring of their own, one sub-slot per (level, component);
 * a component's plane k-1 values at the cell (u, v, w) travel in registers,
 * so a sub-slot is released as soon as its level is done. */
#define STB_MS 3                                  /* media slots              */
#define STB_MSLOT (4 * ST_MP)
#define STB_CST (3 * ST_VT)                       /* first stress tile        */
#define STB_CSLOT (STB_CST + 12 * ST_PT)          /* r tiles fit in 6 x 256   */

__host__ __device__ __forceinline__ uint32_t strb_comp_txb(int nve, int rtile_bytes)
{
    return (uint32_t)((3 * ST_VT + 6 * ST_PT) * 4 + (nve == 1 ? rtile_bytes : 0));
}

/* RPT tile rows per consumer thread (ST_Y / RPT consumer warps) */
template <class TM, class TR, int NCB, int STB_CS, int RPT>
__global__ void __launch_bounds__(32 * (ST_Y / RPT + 1), 2)
k_str_tmab(const __grid_constant__ AwpStagedStrMaps maps, AwpGeom g, AwpCompSet<AWP_MAX_COMP> cs,
           const float *__restrict__ cx, const float *__restrict__ cy, const float *__restrict__ cz,
           const float *__restrict__ tau, float dth, float dt, float dh1, AwpWork w, int nve, const __grid_constant__ AwpMediaScale sc, int *err, AwpWait wt,
          const __grid_constant__ StrEnds ends)
{
    constexpr int CW = ST_Y / RPT;    /* consumer warps */
    extern __shared__ unsigned char st_smem[];
    float *mring = ring_base(st_smem);
    float *cring = mring + STB_MS * STB_MSLOT;
    uint64_t *mfull = (uint64_t *)(cring + STB_CS * STB_CSLOT), *mempty = mfull + STB_MS;
    uint64_t *cfull = mempty + STB_MS, *cempty = cfull + STB_CS;
    __shared__ volatile int abort_s;
    __shared__ AwpComp tab[AWP_MAX_COMP];
    if (threadIdx.y == 0 && threadIdx.x < AWP_MAX_COMP) {
#pragma unroll
        for (int f = 0; f < AWP_NF_ARRAYS; ++f) tab[threadIdx.x].f[f] = pick(cs, threadIdx.x, f);
    }
    ring_init<STB_MS>(mfull, mempty, &abort_s, CW);
    ring_init<STB_CS>(cfull, cempty, &abort_s, CW);
    const int tx = threadIdx.x, ty = threadIdx.y;

    if (ty == CW) {                   /* producer warp */
        if (tx != 0) return;
        uint32_t um = 0, uc = 0;
        bool ok = true;
        const int nmed = nve == 1 ? 4 : 2;
        for (int item = blockIdx.x; ok && item < w.nitems; item += gridDim.x) {
            int bx, by, k0, k1;
            staged_item(g, w, item, bx, by, k0, k1);
            const int i0 = bx * ST_X + 1, j0 = by * ST_Y + 1;
            const int x = tile_x(i0), xp = i0 + AWP_XO - 1;
            for (int k = k0 - 1; ok && k <= k1; ++k) {
                ok = ring_acquire<STB_MS>(mempty, um, &abort_s, wt.ns);
                if (!ok) break;
                if (um != withheld_use(wt)) {                 /* test injection: nothing issued, no arrival */
                    float *sl = mring + (um % STB_MS) * STB_MSLOT;
                    uint64_t *b = &mfull[um % STB_MS];
                    fence_async_smem();
                    mb_expect(b, (uint32_t)(nmed * med_bytes<TM>(ST_MR)));
                    for (int a = 0; a < nmed; ++a) tma_3d(sl + a * ST_MP, &maps.med[a], b, xp, j0, k + 1);
                }
                ++um;
                if (k < k0) continue;
#pragma unroll
                for (int q = 0; q < NCB; ++q) {
                    ok = ring_acquire<STB_CS>(cempty, uc, &abort_s, wt.ns);
                    if (!ok) break;
                    float *sl = cring + (uc % STB_CS) * STB_CSLOT;
                    uint64_t *b = &cfull[uc % STB_CS];
                    fence_async_smem();
                    mb_expect(b, strb_comp_txb(nve, RTile<TR>::ntiles * ST_PT * RTile<TR>::size));
#pragma unroll
                    for (int a = 0; a < 3; ++a) tma_3d(sl + a * ST_VT, &maps.v[q][a], b, x, j0 - 1, k + 1);
#pragma unroll
                    for (int a = 0; a < 6; ++a) tma_3d(sl + STB_CST + a * ST_PT, &maps.s[q][a], b, xp, j0 + 1, k + 1);
                    if (nve == 1) r_issue<TR>(maps, q, (unsigned char *)(sl + STB_CST + 6 * ST_PT), b, xp, j0 + 1, k + 1);
                    ++uc;
                }
            }
        }
        if (!ok) {
            abort_s = 1;
            atomicOr(err, AWP_KERR_TMA_WAIT);
        }
        ring_drain<STB_MS>(mfull, um, wt.ns, withheld_use(wt));
        ring_drain<STB_CS>(cfull, uc, wt.ns);
        return;
    }

    const int sz = g.plane, sy = g.px;
    uint32_t um0 = 0, uc = 0;         /* media use of the item's level k0 - 1; next component use */
    for (int item = blockIdx.x; item < w.nitems; item += gridDim.x) {
        int bx, by, k0, k1;
        staged_item(g, w, item, bx, by, k0, k1);
        const int i = bx * ST_X + 1 + tx;
        const int c0 = g.idx(i, by * ST_Y + 1 + ty, k0);
        /* per row and component: column queues u, v at k+1, k+2 and w at k+1,
         * fed by loads one level ahead (pu, pv, pw) that rotate in when the
         * component comes up at the next level, a full level after their
         * issue; w at k-2, k-1 and u, v at k-1 come from earlier tiles */
        float up1[RPT][NCB], up2[RPT][NCB], pu[RPT][NCB], vp1[RPT][NCB], vp2[RPT][NCB], pv[RPT][NCB];
        float wp1[RPT][NCB], pw[RPT][NCB], wm2[RPT][NCB], wm1[RPT][NCB], um1[RPT][NCB], vm1[RPT][NCB];
        bool live[RPT];
        int itxy[RPT];
        float cxy[RPT];
#pragma unroll
        for (int r = 0; r < RPT; ++r) {
            const int j = by * ST_Y + 1 + ty + r * CW, c = c0 + r * CW * sy;
            live[r] = i <= g.nx && j <= g.ny;
            itxy[r] = ((j & 1) << 1) | (i & 1);
            cxy[r] = live[r] ? cx[i] * cy[j] : 0.f;
#pragma unroll
            for (int q = 0; q < NCB; ++q) {
                up1[r][q] = up2[r][q] = pu[r][q] = vp1[r][q] = vp2[r][q] = pv[r][q] = wp1[r][q] = pw[r][q] = 0.f;
                wm2[r][q] = wm1[r][q] = um1[r][q] = vm1[r][q] = 0.f;
                if (live[r]) {
                    float *U = tab[q].f[AF_U], *V = tab[q].f[AF_V], *W = tab[q].f[AF_W];
                    if (k1 == g.nz)
                        fs_velocity(g, U, V, W, (const TM *)ends.lam, (const TM *)ends.mu, sc, i, j);
                    up2[r][q] = __ldg(&U[c + sz]); pu[r][q] = __ldg(&U[c + 2 * sz]);
                    vp2[r][q] = __ldg(&V[c + sz]); pv[r][q] = __ldg(&V[c + 2 * sz]);
                    pw[r][q] = __ldg(&W[c + sz]);
                    wm2[r][q] = __ldg(&W[c - 2 * sz]); wm1[r][q] = __ldg(&W[c - sz]);
                    um1[r][q] = __ldg(&U[c - sz]); vm1[r][q] = __ldg(&V[c - sz]);
                }
            }
        }
        int cc = c0;
#pragma unroll 1
        for (int k = k0; k <= k1; ++k, cc += sz) {
            const uint32_t mk = um0 + (uint32_t)(k - k0 + 1), mm = mk - 1;
            const float czk = cz[k];
            bool ok = true;
            if (k == k0) ok = mb_wait_or_abort(&mfull[mm % STB_MS], (mm / STB_MS) & 1, &abort_s, wt.ns);
            if (ok) ok = mb_wait_or_abort(&mfull[mk % STB_MS], (mk / STB_MS) & 1, &abort_s, wt.ns);
            if (!__all_sync(0xffffffffu, ok)) {   /* warp-uniform outcome */
                abort_s = 1;
                atomicOr(err, AWP_KERR_TMA_WAIT);
                return;
            }
            const int ipar = ((g.nz + 1 - k) & 1) << 2;                        /* viscoop.f:93-101 */
            StrCoef kc[RPT];
#pragma unroll
            for (int r = 0; r < RPT; ++r) {
                const int cm = (ty + r * CW + 1) * MedRow<TM>::W + tx;
                const int it = ipar | itxy[r];
                const TMed<TM> M{mring + (mk % STB_MS) * STB_MSLOT, mring + (mm % STB_MS) * STB_MSLOT, cm, sc};
                if (live[r])          /* lanes outside the grid hold zero media: their divisions would be slow */
                    kc[r] = str_coef_t(M, nve, tau[it], tau[8 + it]);
            }
            __syncwarp();
            if (tx == 0) mb_arrive(&mempty[mm % STB_MS]);
#pragma unroll
            for (int q = 0; q < NCB; ++q, ++uc) {
#pragma unroll
                for (int r = 0; r < RPT; ++r) {
                    /* rotate this component's queues, then load one level ahead */
                    const int c = cc + r * CW * sy;
                    up1[r][q] = up2[r][q]; up2[r][q] = pu[r][q];
                    vp1[r][q] = vp2[r][q]; vp2[r][q] = pv[r][q];
                    wp1[r][q] = pw[r][q];
                    pu[r][q] = pv[r][q] = pw[r][q] = 0.f;
                    if (live[r] && k < k1) {
                        pu[r][q] = __ldcg(&tab[q].f[AF_U][c + 3 * sz]);
                        pv[r][q] = __ldcg(&tab[q].f[AF_V][c + 3 * sz]);
                        pw[r][q] = __ldcg(&tab[q].f[AF_W][c + 2 * sz]);
                    }
                }
                ok = mb_wait_or_abort(&cfull[uc % STB_CS], (uc / STB_CS) & 1, &abort_s, wt.ns);
                if (!__all_sync(0xffffffffu, ok)) {
                    abort_s = 1;
                    atomicOr(err, AWP_KERR_TMA_WAIT);
                    return;
                }
                const float *sk = cring + (uc % STB_CS) * STB_CSLOT;
#pragma unroll
                for (int r = 0; r < RPT; ++r) {
                    const int row = ty + r * CW, c = cc + r * CW * sy;
                    const int cv = (row + 2) * ST_W + tx + 4, cp = row * ST_X + tx;
                    const float nu = sk[cv], nv = sk[ST_VT + cv], nw = sk[2 * ST_VT + cv];
                    if (live[r]) {
                        const float *ps = sk + STB_CST + cp;
                        const Stress6 s0{ps[0], ps[ST_PT], ps[2 * ST_PT], ps[3 * ST_PT], ps[4 * ST_PT], ps[5 * ST_PT]};
                        const TVel Vq{sk + cv, um1[r][q], vm1[r][q], wm1[r][q], up1[r][q], up2[r][q], vp1[r][q],
                                      vp2[r][q], wm2[r][q], wp1[r][q]};
                        Stress6 o;
                        if (nve == 1) {
                            float rr[6];
                            RTile<TR>::ld((const unsigned char *)(sk + STB_CST + 6 * ST_PT), cp, rr);
                            const VelDiff dd = vel_diff(Vq);
                            o = str_visco(kc[r], dd, s0, rr, dth, dt, dh1);
                            RVars<TR>::st(tab[q], c, rr);
                        } else {
                            o = str_elastic(kc[r], Vq, s0, dth);
                        }
                        const float crj = cxy[r] * czk;
                        gst6(tab[q], c, o, crj);
                    }
                    wm2[r][q] = wm1[r][q];
                    um1[r][q] = nu; vm1[r][q] = nv; wm1[r][q] = nw;
                }
                __syncwarp();
                if (tx == 0) mb_arrive(&cempty[uc % STB_CS]);
            }
        }
        __syncwarp();
        if (tx == 0) mb_arrive(&mempty[(um0 + (uint32_t)(k1 - k0 + 1)) % STB_MS]);
        um0 += (uint32_t)(k1 - k0 + 2);
        if (k1 == g.nz) {
#pragma unroll
            for (int r = 0; r < RPT; ++r) {
                if (!live[r]) continue;
#pragma unroll
                for (int q = 0; q < NCB; ++q) {
                    /* fstr (operator.f:594-606) on this thread's own column */
                    const int ct = g.idx(i, by * ST_Y + 1 + ty + r * CW, g.nz);
                    float *ZZ = tab[q].f[AF_ZZ], *XZ = tab[q].f[AF_XZ], *YZ = tab[q].f[AF_YZ];
                    ZZ[ct + sz] = -__ldcg(&ZZ[ct]);
                    ZZ[ct + 2 * sz] = -__ldcg(&ZZ[ct - sz]);
                    XZ[ct + sz] = -__ldcg(&XZ[ct - sz]);
                    XZ[ct + 2 * sz] = -__ldcg(&XZ[ct - 2 * sz]);
                    YZ[ct + sz] = -__ldcg(&YZ[ct - sz]);
                    YZ[ct + 2 * sz] = -__ldcg(&YZ[ct - 2 * sz]);
                    XZ[ct] = 0.0f;
                    YZ[ct] = 0.0f;
                }
            }
        }
    }
    str_finish(ends, gridDim.x * CW);
}

#include "awp_pair.cuh"

}  // namespace

/* ------------------------------------------------------------------ */
/* host side                                                           */
/* ------------------------------------------------------------------ */

#ifdef AWP_STAGED_FMA
#define AWP_STAGED_ENTRY(name) name##_fma
#else
#define AWP_STAGED_ENTRY(name) name
#endif

#ifndef AWP_STAGED_FMA
typedef CUresult (*EncodeTiledFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
                                  const cuuint64_t *, const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static EncodeTiledFn encode_fn()
{
    static EncodeTiledFn fn = NULL;
    if (!fn) {
        void *p = NULL;
        cudaDriverEntryPointQueryResult qr;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &qr) == cudaSuccess &&
            qr == cudaDriverEntryPointSuccess)
            fn = (EncodeTiledFn)p;
    }
    return fn;
}

/* tensor map of one padded volume (pitch, ny + 4, nz + 4) of 4- or 2-byte
 * elements, box w x rows x 1 */
static bool make_map(CUtensorMap *m, const AwpGeom &g, const void *base, int w, int rows, int esize = 4)
{
    EncodeTiledFn fn = encode_fn();
    if (!fn || !base || ((uintptr_t)base & 15) || (g.px * esize) % 16 || (w * esize) % 16) return false;
    const cuuint64_t dim[3] = {(cuuint64_t)g.px, (cuuint64_t)g.py, (cuuint64_t)g.nz + 4};
    const cuuint64_t stride[2] = {(cuuint64_t)g.px * esize, (cuuint64_t)g.plane * esize};
    const cuuint32_t box[3] = {(cuuint32_t)w, (cuuint32_t)rows, 1};
    const cuuint32_t es[3] = {1, 1, 1};
    const CUtensorMapDataType t = esize == 4 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16;
    return fn(m, t, 3, (void *)base, dim, stride, box, es, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
              CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

cudaError_t awp_staged_create(AwpStaged **out, const AwpGeom &g, int ncomp, const AwpComp *comp, const AwpMediaT &md,
                              int rtype)
{
    *out = NULL;
    if (ncomp < 1 || ncomp > AWP_MAX_COMP) return cudaErrorInvalidValue;
    const int msize = md.type == AWP_STORE_F32 ? 4 : 2, mw = md.type == AWP_STORE_F32 ? MedRow<float>::W : MedRow<__half>::W;
    if (g.px % 8 != 0) return cudaErrorInvalidValue;
    AwpStaged *s = (AwpStaged *)aligned_alloc(64, sizeof(AwpStaged));
    if (!s) return cudaErrorMemoryAllocation;
    memset(s, 0, sizeof *s);
    static const int med_f[4] = {AM_LAM, AM_MU, AM_QP, AM_QS};
    const int rsize = rtype == AWP_STORE_F32 ? 4 : 2;
    bool ok = true;
    for (int q = 0; q < ncomp; ++q) {
        for (int a = 0; a < 3; ++a) ok = ok && make_map(&s->sm.v[q][a], g, comp[q].f[AF_U + a], ST_W, ST_HR);
        for (int a = 0; a < 6; ++a) ok = ok && make_map(&s->sm.s[q][a], g, comp[q].f[AF_XX + a], ST_X, ST_Y);
        for (int a = 0; a < 6; ++a)     /* absent in the elastic scheme, which never loads them */
            if (comp[q].f[AF_R1 + a]) ok = ok && make_map(&s->sm.r[q][a], g, comp[q].f[AF_R1 + a], ST_X, ST_Y, rsize);
        if (rtype == AWP_STORE_BFP && comp[q].f[AF_R1])
            ok = ok && comp[q].f[AF_RX] && make_map(&s->sm.rx[q], g, comp[q].f[AF_RX], ST_X, ST_Y, 2);
    }
    for (int a = 0; a < 4; ++a) ok = ok && make_map(&s->sm.med[a], g, md.m[med_f[a]], mw, ST_MR, msize);
    const int vr = 2 * PR_VEL_CW;
    ok = ok && make_map(&s->vm.d1, g, md.m[AM_D1], mw, vr + 1, msize);
    for (int q = 0; q < ncomp; ++q) {
        const AwpComp &o = comp[q];
        static const int pf[6] = {AF_U, AF_V, AF_W, AF_ZZ, AF_XZ, AF_YZ};
        ok = ok && make_map(&s->vm.xx[q], g, o.f[AF_XX], PR_W, vr) && make_map(&s->vm.yy[q], g, o.f[AF_YY], PR_X, vr + 3) &&
             make_map(&s->vm.xy[q], g, o.f[AF_XY], PR_W, vr + 3) && make_map(&s->vm.xz[q], g, o.f[AF_XZ], PR_W, vr) &&
             make_map(&s->vm.yz[q], g, o.f[AF_YZ], PR_X, vr + 3);
        for (int a = 0; a < 6; ++a) ok = ok && make_map(&s->vm.p[q][a], g, o.f[pf[a]], PR_X, vr);
    }
    if (!ok) {
        free(s);
        return cudaErrorInvalidValue;
    }
    *out = s;
    return cudaSuccess;
}

void awp_staged_destroy(AwpStaged *s) { free(s); }
#endif

static AwpWait awp_wait_of(const AwpStepArgs &s)
{
    AwpWait w;
    w.ns = s.wait_ns ? s.wait_ns : 2000000000ull;
    w.withhold = s.withhold;
    return w;
}

/* SMs a launch may use and resident blocks of the kernel on one of them */
struct StagedSlots {
    int nsm, per;
};

template <class K>
static cudaError_t staged_slots(K kernel, size_t smem, int sm_limit, int threads, StagedSlots *o)
{
    int dev = 0;
    o->nsm = 148;
    o->per = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&o->nsm, cudaDevAttrMultiProcessorCount, dev);
    if (sm_limit > 0 && sm_limit < o->nsm) o->nsm = sm_limit;
    if (e == cudaSuccess) e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&o->per, kernel, threads, smem);
    if (e != cudaSuccess) return e;
    return o->per < 1 ? cudaErrorInvalidConfiguration : cudaSuccess;
}

/* z chunks of a sweep over `tiles` column tiles.  An item costs
 * its levels plus about `extra` for its prologue (the planes below its first
 * level, column values from global memory, the first copies).  Items run in
 * rounds of nsm * per; a full SM works through them at one level per unit of
 * time and block, and an SM with fewer blocks is bound by the latency of a
 * level, about 0.65 * per units.  The split with the least time by that count
 * is taken: on a grid that fills the device it keeps the last round full, on
 * a small one it spreads the columns over all SMs (100x100x50, one component:
 * chunks of 7 levels instead of 25).  At least five levels: the prologue must
 * not outweigh them, and the top chunk's threads mirror the levels nz-2 .. nz
 * themselves.  Steps, fixed 25 .. 40 levels before -> this rule: 100x100x50 one
 * component 0.052 -> 0.037 ms, 160x160x80 0.114 -> 0.084, 120x110x60 two
 * components 0.114 -> 0.072, 400x400x200 three 3.18 -> 3.11.
 * The constants are measured, not derived.  On twelve grids from 64x64x48 to
 * 640x500x150 with one to three components, 0.65 up to 1.0 gave the same step
 * to 0.6 %, 0.5 and less cost up to 11 %; extra halved or doubled moved single
 * grids by 3 %, halved 10 % on one, none at all cost up to 6 %.  Against
 * explicit chunks of 8, 10, 13, 17, 20, 25, 32 and 40 levels the rule was
 * within 1.3 % of the best one on every grid; the best single one of them, 8,
 * was up to 13 % slower. */
static int pick_chunks(int nz, int tiles, const StagedSlots &sl, double extra)
{
    const int slots = sl.nsm * sl.per, kmin = nz < 5 ? nz : 5;
    int best = 1;
    double best_t = 1e30;
    for (int n = 1; n * kmin <= nz; ++n) {
        const long long items = (long long)tiles * n;
        const int rem = (int)(items % slots), on_sm = (rem + sl.nsm - 1) / sl.nsm;
        const double tail = rem ? (on_sm > 0.65 * sl.per ? on_sm : 0.65 * sl.per) : 0.0;
        const double t = ((double)nz / n + extra) * ((double)(items / slots) * sl.per + tail);
        if (t < best_t) {
            best_t = t;
            best = n;
        }
    }
    return best;
}

/* work items of a sweep over 32 x rows tiles; kchunk: most levels of an item, 0: pick_chunks */
static AwpWork staged_work(const AwpGeom &g, int rows, int kchunk, int ncomp, const StagedSlots &sl, double extra)
{
    AwpWork w;
    w.ntx = (g.nx + ST_X - 1) / ST_X;
    w.nty = (g.ny + rows - 1) / rows;
    w.kchunk = kchunk;
    w.nzc = kchunk > 0 ? (g.nz + kchunk - 1) / kchunk : pick_chunks(g.nz, w.ntx * w.nty * ncomp, sl, extra);
    w.nitems = w.ntx * w.nty * w.nzc * ncomp;
    return w;
}

static int staged_grid(const StagedSlots &sl, const AwpWork &w)
{
    const int n = sl.nsm * sl.per;
    return n < w.nitems ? n : w.nitems;
}

static StrEnds str_ends(const AwpStepArgs &s)
{
    StrEnds e;
    memset(&e, 0, sizeof e);
    e.lam = s.md.m[AM_LAM];
    e.mu = s.md.m[AM_MU];
    if (s.post) {
        e.post = *s.post;
        e.done = s.post_done;
    }
    return e;
}

static AwpCompSet<AWP_MAX_COMP> comp_set3(const AwpStepArgs &s)
{
    AwpCompSet<AWP_MAX_COMP> cs;
    memset(&cs, 0, sizeof cs);
    for (int q = 0; q < s.ncomp; ++q) cs.c[q] = s.comp[q];
    return cs;
}

template <class TM>
static cudaError_t launch_vel(const AwpStaged *st, const AwpStepArgs &s, cudaStream_t stream)
{
    constexpr int CW = PR_VEL_CW, S = 3;
    const size_t smem = PairVelL<TM, CW>::smem(S);
    StagedSlots sl;
    cudaError_t e = staged_slots(k_vel_tma<TM, CW, S, 2>, smem, s.sm_limit, 32 * (CW + 1), &sl);
    if (e != cudaSuccess) return e;
    const AwpWork w = staged_work(s.g, 2 * CW, s.kchunk_staged, s.ncomp, sl, 1.0);
    k_vel_tma<TM, CW, S, 2><<<staged_grid(sl, w), dim3(32, CW + 1), smem, stream>>>(
        st->vm, s.g, comp_set3(s), s.ncomp, s.staged_qslow, (const TM *)s.md.m[AM_D1], s.md.sc.inv[AM_D1], s.cx, s.cy,
        s.cz, s.dth, w, s.kerr, awp_wait_of(s));
    return cudaGetLastError();
}

/* dynamic shared memory of a ring: alignment slack, slots, full + empty barriers */
static size_t ring_bytes(int slots, int slot_floats) { return 128 + (size_t)slots * slot_floats * 4 + 2 * 8 * slots; }

template <class TM, class TR, int UNR, int RPT>
static cudaError_t launch_str_rpt(const AwpStaged *st, const AwpStepArgs &s, cudaStream_t stream)
{
    constexpr int CW = ST_Y / RPT;
    const size_t smem = ring_bytes(2 + STR_D, STR_SLOT);
    StagedSlots sl;
    cudaError_t e = staged_slots(k_str_tma<TM, TR, UNR, RPT>, smem, s.sm_limit, 32 * (CW + 1), &sl);
    if (e != cudaSuccess) return e;
    const AwpWork w = staged_work(s.g, ST_Y, s.kchunk_staged, s.ncomp, sl, 1.5);
    k_str_tma<TM, TR, UNR, RPT><<<staged_grid(sl, w), dim3(32, CW + 1), smem, stream>>>(st->sm, s.g, comp_set3(s), s.ncomp,
                                                                       s.staged_qslow, s.cx, s.cy, s.cz, s.tau,
                                                                       s.dth, s.dt, s.dh1, w, s.nve, s.md.sc, s.kerr, awp_wait_of(s), str_ends(s));
    return cudaGetLastError();
}

/* CS component sub-slots: CS - 1 (level, component) tiles in flight */
template <class TM, class TR, int NCB, int CS, int RPT>
static cudaError_t launch_str_bc(const AwpStaged *st, const AwpStepArgs &s, cudaStream_t stream)
{
    constexpr int CW = ST_Y / RPT;
    const size_t smem = 128 + (size_t)(STB_MS * STB_MSLOT + CS * STB_CSLOT) * 4 + 2 * 8 * (STB_MS + CS);
    StagedSlots sl;
    cudaError_t e = staged_slots(k_str_tmab<TM, TR, NCB, CS, RPT>, smem, s.sm_limit, 32 * (CW + 1), &sl);
    if (e != cudaSuccess) return e;
    const AwpWork w = staged_work(s.g, ST_Y, s.kchunk_staged, 1, sl, 1.0);
    k_str_tmab<TM, TR, NCB, CS, RPT><<<staged_grid(sl, w), dim3(32, CW + 1), smem, stream>>>(
        st->sm, s.g, comp_set3(s), s.cx, s.cy, s.cz, s.tau, s.dth, s.dt, s.dh1, w, s.nve, s.md.sc, s.kerr, awp_wait_of(s), str_ends(s));
    return cudaGetLastError();
}

/* five sub-slots (109 KB with the media ring, two blocks per SM) measured
 * slightly ahead of four on the 400 x 400 x 200 three-component grid; one
 * row per thread: with two (161 registers) a launch took 3.00 ms against
 * 2.39 ms there, so staged_rpt applies to the one-component-per-item form only */
template <class TM, class TR, int NCB>
static cudaError_t launch_str_b(const AwpStaged *st, const AwpStepArgs &s, cudaStream_t stream)
{
    return launch_str_bc<TM, TR, NCB, 5, 1>(st, s, stream);
}

/* 16-bit media go through the same sweeps: their tiles are half as large and
 * widened when the coefficients are formed.  640x640x256 fx+fy in binary16:
 * 8.87 ms a step with the plain two-sweep kernels, 6.30 this way.
 * Two rows per thread carry twice the live state already: that variant keeps
 * its level loop rolled (unrolled twice it needs 128 registers and runs slower) */
template <class TM, class TR>
static cudaError_t launch_str_tr(const AwpStaged *st, const AwpStepArgs &s, cudaStream_t stream)
{
    if ((s.staged_batch & 1) && s.ncomp == 3) return launch_str_b<TM, TR, 3>(st, s, stream);
    if ((s.staged_batch & 1) && s.ncomp == 2) return launch_str_b<TM, TR, 2>(st, s, stream);
    if constexpr (sizeof(TM) == 4) {
        if (s.staged_rpt == 2) return launch_str_rpt<TM, TR, 1, 2>(st, s, stream);
        if (s.unroll == 1) return launch_str_rpt<TM, TR, 1, 1>(st, s, stream);
    }
    return launch_str_rpt<TM, TR, 2, 1>(st, s, stream);
}

cudaError_t AWP_STAGED_ENTRY(awp_launch_vel_staged)(const AwpStaged *st, const AwpStepArgs &s, cudaStream_t stream)
{
    if (!st) return cudaErrorInvalidValue;
    if (s.md.type == AWP_STORE_BF16) return launch_vel<__nv_bfloat16>(st, s, stream);
    if (s.md.type == AWP_STORE_F16) return launch_vel<__half>(st, s, stream);
    return launch_vel<float>(st, s, stream);
}

cudaError_t AWP_STAGED_ENTRY(awp_launch_str_staged)(const AwpStaged *st, const AwpStepArgs &s, cudaStream_t stream)
{
    if (!st) return cudaErrorInvalidValue;
    if (s.md.type == AWP_STORE_BF16) return launch_str_tr<__nv_bfloat16, __nv_bfloat16>(st, s, stream);
    if (s.md.type == AWP_STORE_F16) return launch_str_tr<__half, __nv_bfloat16>(st, s, stream);
    if (s.rtype == AWP_STORE_BF16) return launch_str_tr<float, __nv_bfloat16>(st, s, stream);
    if (s.rtype == AWP_STORE_BFP) return launch_str_tr<float, RBfp>(st, s, stream);
    return launch_str_tr<float, float>(st, s, stream);
}

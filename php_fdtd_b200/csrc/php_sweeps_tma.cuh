/*
 * php_sweeps_tma.cuh -- the two sweeps with a TMA plane pipeline (sm_100a).
 *
 * A block owns a 32 x 8 (x, y) tile of a z chunk.  One thread streams whole
 * planes of the tile into a ring of shared-memory stages with
 * cp.async.bulk.tensor (tile mode, no multicast: every byte comes from this
 * GPU's own memory), each stage completed on its own mbarrier; all 256
 * threads compute from shared memory.  The bytes in flight are set by the
 * ring depth instead of by registers, which is what a streaming stencil on
 * HBM needs.
 *
 *   h_sweep_tma: per plane, Ex/Ey/Ez with a +1 halo in x and y (the box is
 *     widened to 16 bytes in x) and Hx/Hy/Hz of the tile; the update at k
 *     reads E planes k and k+1.
 *   e_sweep_tma: per plane, Hx/Hy/Hz with a -1 halo in x and y (the box starts
 *     16 bytes left of the tile so that its x offset stays 16-byte aligned),
 *     Ex/Ey/Ez (strict mode: Dx/Dy/Dz) of the tile; the update at k reads H
 *     planes k and k-1.
 * Out-of-range parts of a box read the tensor map's zero fill; those values
 * are only used by cells the reference never updates there (i = nx-1 or
 * j = ny-1 for H, the x/y border for D).
 *
 * Waits on the mbarriers are bounded: after kWaitLimit polls the block sets
 * a device error flag and leaves the loop (the decision is made uniform
 * across the block with __syncthreads_or), and the host reports
 * PHP_ERR_TIMEOUT.
 */
#pragma once

#include <cuda.h>

namespace phpdev {

constexpr uint32_t kWaitLimit = 1u << 24;

/* Ring depths.  A plane's load takes about 1.8 us from its issue to the
 * barrier (one block per SM, everything in L2: 0.94 us per plane of the H
 * sweep with two planes in flight, 1.68 us of the fused sweep with one), so
 * an SM needs some 80 KB in flight for the copy bandwidth; the depths fill
 * the shared memory that the resident blocks share. */
#ifndef PHP_TMA_ES64
#define PHP_TMA_ES64 3
#endif
#ifndef PHP_TMA_ES32
#define PHP_TMA_ES32 4
#endif
#ifndef PHP_TMA_HS64
#define PHP_TMA_HS64 4
#endif
#ifndef PHP_TMA_HS32
#define PHP_TMA_HS32 4
#endif
/* resident blocks the fused sweep is compiled for (register budget), FP64
 * and FP32 */
#ifndef PHP_E_MINBLOCKS
#define PHP_E_MINBLOCKS 4
#endif
#ifndef PHP_E_MINBLOCKS32
#define PHP_E_MINBLOCKS32 4
#endif
/* the same for its launches over the blocks of one kind: plain and tensor
 * blocks, atom blocks, the rest */
#ifndef PHP_EP_MINBLOCKS64
#define PHP_EP_MINBLOCKS64 4
#endif
#ifndef PHP_EP_MINBLOCKS32
#define PHP_EP_MINBLOCKS32 5
#endif
#ifndef PHP_EA_MINBLOCKS64
#define PHP_EA_MINBLOCKS64 3
#endif
#ifndef PHP_EA_MINBLOCKS32
#define PHP_EA_MINBLOCKS32 4
#endif
#ifndef PHP_EG_MINBLOCKS64
#define PHP_EG_MINBLOCKS64 3
#endif
#ifndef PHP_EG_MINBLOCKS32
#define PHP_EG_MINBLOCKS32 4
#endif
/* When the CPML state of the planes after a block's first is read.  FP32: a
 * plane ahead, into registers (256^3 tip workload, fused sweep of the rest 114
 * -> 110 us); where r and v sit in registers too, and in the strict mode, after
 * the plane before it is done (two-atom fused sweep, 512 x 512 x 256: 480 ->
 * 450 us).  FP64: before the plane's wait, its lines requested a plane
 * ahead (the same sweep 785 us; after the plane before it 851 us). */
enum : int { kPsiAhead = 0, kPsiAfter = 1, kPsiTop = 2 };
template <typename R, bool STRICT, bool VREG>
constexpr int kPsiMode = STRICT ? kPsiAfter : sizeof(R) == 8 ? kPsiTop : VREG ? kPsiAfter : kPsiAhead;

/* Tensor maps of the device arrays: 4-D (x, y, plane, component), planes
 * counted from the low halo plane; the three components of a field are one
 * allocation, so that one load brings a plane of all three. */
struct TmaMaps {
    CUtensorMap e_halo; /* E: box (32 + 16/s) x 9 at (i0, j0) */
    CUtensorMap h_own;  /* H: box 32 x 8 */
    CUtensorMap h_halo; /* H: box (32 + 16/s) x 9 at (i0 - 16/s, j0 - 1) */
    CUtensorMap own;    /* E (strict mode: D): box 32 x 8 */
    /* he_sweep_tma's and interior_sweep_tma's boxes (FusedGeom), at (i0 - 16/s, j0 - 1) */
    CUtensorMap e_wide; /* E: box EX x EY */
    CUtensorMap h_wide; /* H: box HX x HY */
};

__device__ __forceinline__ uint32_t smem_addr(const void* p)
{
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(bar)), "r"(count) : "memory");
}

__device__ __forceinline__ void mbar_arrive_expect_tx(uint64_t* bar, uint32_t bytes)
{
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(bar)), "r"(bytes) : "memory");
}

__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity)
{
    uint32_t done;
    asm volatile(
        "{\n"
        "  .reg .pred p;\n"
        "  mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
        "  selp.u32 %0, 1, 0, p;\n"
        "}\n"
        : "=r"(done)
        : "r"(smem_addr(bar)), "r"(parity)
        : "memory");
    return done != 0;
}

/* bounded wait: false after `limit` polls (kWaitLimit by default) */
__device__ __forceinline__ bool mbar_wait_n(uint64_t* bar, uint32_t parity, uint32_t limit)
{
    for (uint32_t n = 0; n < limit; ++n)
        if (mbar_try_wait(bar, parity)) return true;
    return false;
}
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity)
{
    return mbar_wait_n(bar, parity, kWaitLimit);
}

/* After a bounded wait gave up: waits (bounded again) for the block's plane
 * loads that may still be in flight -- at most the last S of the `issued`
 * loads, load g in stage g % S with phase parity (g / S) & 1, since a load
 * is only issued into a stage whose previous load every thread has
 * consumed -- so that none lands in shared memory after the block left. */
__device__ __forceinline__ void ring_drain(uint64_t* full, int S, uint32_t issued)
{
    const uint32_t first = issued > (uint32_t)S ? issued - (uint32_t)S : 0u;
    for (uint32_t g = first; g < issued; ++g) mbar_wait(&full[g % S], (g / S) & 1u);
}

/* Loads a block has issued when it stops after plane k: the H sweep loads
 * planes k0..k1 (the first S at once, then plane j + S after plane j), the
 * fused sweep planes k0-1..k1-1 (then plane j - 1 + S after plane j). */
__device__ __forceinline__ uint32_t h_loads_issued(int k, int k0, int k1, int S)
{
    return (uint32_t)(min(k1, k + S - 1) - k0 + 1);
}
__device__ __forceinline__ uint32_t e_loads_issued(int k, int k0, int k1, int S)
{
    return (uint32_t)(min(k1 - 1, k + S - 2) - k0 + 2);
}

/* polls of the failure-path test's wait on a barrier nothing arrives on */
constexpr uint32_t kStallPolls = 1u << 12;

__device__ __forceinline__ void fence_barrier_init()
{
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

/* orders this thread's generic-proxy accesses to shared memory before the
 * async-proxy (TMA) writes it issues next */
__device__ __forceinline__ void fence_proxy_async_smem()
{
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

__device__ __forceinline__ void tma_load_3d(void* dst, const CUtensorMap* map, uint64_t* bar, int x, int y, int z)
{
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
        ::"r"(smem_addr(dst)), "l"(map), "r"(smem_addr(bar)), "r"(x), "r"(y), "r"(z)
        : "memory");
}

/* plane z of the box at (x, y), all three components */
__device__ __forceinline__ void tma_load_plane(void* dst, const CUtensorMap* map, uint64_t* bar, int x, int y, int z)
{
    asm volatile(
        "cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6}], [%2];"
        ::"r"(smem_addr(dst)), "l"(map), "r"(smem_addr(bar)), "r"(x), "r"(y), "r"(z), "r"(0)
        : "memory");
}

template <typename R>
struct TmaGeom {
    static constexpr int TX = kBlockX, TY = kBlockY;
    static constexpr int HALO = 16 / (int)sizeof(R);      /* x halo widened to 16 bytes */
    static constexpr int BX = TX + HALO, BY = TY + 1;      /* halo box */
    static constexpr int HALO_ELEMS = BX * BY, OWN_ELEMS = TX * TY;
    /* three components each */
    static constexpr uint32_t HALO3_BYTES = 3 * HALO_ELEMS * sizeof(R), OWN3_BYTES = 3 * OWN_ELEMS * sizeof(R);
    __host__ __device__ static constexpr uint32_t align128(uint32_t b) { return (b + 127u) / 128u * 128u; }
    /* a stage of either sweep: a halo box (H sweep: E, E sweep: H), then an
     * own box (H; old E, strict mode D) */
    static constexpr uint32_t OWN_AT = align128(HALO3_BYTES), STAGE = OWN_AT + align128(OWN3_BYTES);
    static constexpr int HS = sizeof(R) == 8 ? PHP_TMA_HS64 : PHP_TMA_HS32;
    static constexpr int ES = sizeof(R) == 8 ? PHP_TMA_ES64 : PHP_TMA_ES32;
    /* dynamic shared memory: 128 bytes of alignment slack, the stages, then
     * the stage barriers */
    /* H sweep: the failure-path test's barrier, then (both) the CPML table */
    static constexpr uint32_t TAB = align128(pml_table_len(TY) * sizeof(R));
    static constexpr uint32_t H_SMEM = 128 + HS * STAGE + 128 + TAB;
    static constexpr uint32_t E_SMEM = 128 + ES * STAGE + 128 + TAB;
};

/* A block's tile, planes [k0, k1) and class: from the launch's list, or from
 * the grid of z chunks with the per-block classes `cls` (none: dflt). */
struct SweepJob {
    int bx, by, k0, k1, cls;
};
template <bool LIST, typename R>
__device__ __forceinline__ SweepJob sweep_job(const StepArgs<R>& a, const uint8_t* cls, int dflt)
{
    if constexpr (LIST) {
        const int4 e = a.list[blockIdx.x];
        return SweepJob{e.x & 0xffff, e.x >> 16, e.y, e.z, e.w};
    }
    const int bz = blockIdx.z + a.zc0, k0 = bz * a.zchunk;
    return SweepJob{(int)blockIdx.x, (int)blockIdx.y, k0, min(k0 + a.zchunk, a.nz),
                    cls ? cls[((size_t)bz * gridDim.y + blockIdx.y) * gridDim.x + blockIdx.x] : dflt};
}

/* 128-byte aligned start of the stage ring inside dynamic shared memory */
__device__ __forceinline__ unsigned char* ring_base(unsigned char* dyn)
{
    const uint32_t a = smem_addr(dyn);
    return dyn + ((128u - (a & 127u)) & 127u);
}

/* ================================================================ H sweep */

/* fdtd.c:3123-3231: cells i < nx-1, j < ny-1, all k.  Compiled for the
 * resident blocks per SM that shared memory allows: six in FP32, four in
 * FP64. */
#ifndef PHP_H_MINBLOCKS32
#define PHP_H_MINBLOCKS32 6
#endif
template <typename R, bool STRICT, bool LIST>
__global__ void __launch_bounds__(kBlockX * kBlockY, sizeof(R) == 4 ? PHP_H_MINBLOCKS32 : 4) h_sweep_tma(const __grid_constant__ StepArgs<R> a,
                                                                 const __grid_constant__ TmaMaps tm)
{
    using G = TmaGeom<R>;
    extern __shared__ __align__(128) unsigned char dyn_smem[];
    unsigned char* smem = ring_base(dyn_smem);
    uint64_t* full = reinterpret_cast<uint64_t*>(smem + G::HS * G::STAGE);
    R* const tab = reinterpret_cast<R*>(smem + G::HS * G::STAGE + 128);

    const int tx = threadIdx.x, ty = threadIdx.y, tid = ty * G::TX + tx;
    const SweepJob job = sweep_job<LIST>(a, a.plain_h, 0);
    const int i0 = job.bx * G::TX, j0 = job.by * G::TY;
    const int i = i0 + tx, j = j0 + ty;
    const int k0 = job.k0, k1 = job.k1;
    if (k0 >= k1) return; /* uniform over the block */

    constexpr int EBW = G::HALO_ELEMS, HBW = G::OWN_ELEMS; /* one component in a box */
    auto stage = [&](int p) -> unsigned char* { return smem + (uint32_t)((p - k0) % G::HS) * G::STAGE; };
    /* plane p = k0..k1: E (halo boxes) of every plane, H of planes < k1 */
    auto issue = [&](int p) {
        uint64_t* bar = &full[(p - k0) % G::HS];
        unsigned char* b = stage(p);
        const bool with_h = p < k1;
        mbar_arrive_expect_tx(bar, G::HALO3_BYTES + (with_h ? G::OWN3_BYTES : 0u));
        tma_load_plane(b, &tm.e_halo, bar, i0, j0, p + 1);
        if (with_h) tma_load_plane(b + G::OWN_AT, &tm.h_own, bar, i0, j0, p + 1);
    };

    if (tid == 0) {
        for (int s = 0; s < G::HS + 1; ++s) mbar_init(&full[s], 1);
        fence_barrier_init();
    }
    const bool plain = !STRICT && job.cls;
    if (!plain) pml_table<R, STRICT, true>(a, tab, i0, j0, G::TY, tid);
    chain_enter(a.beside);
    if (tid == 0)
        for (int p = k0; p <= min(k1, k0 + G::HS - 1); ++p) issue(p);
    const bool active = (i < a.nx - 1) && (j < a.ny - 1);
    const int L2 = 2 * a.L;
    const int nxp = a.nxp, ny = a.ny;
    const int sx = active ? pml_slot(i, a.nx, a.L) : -1;
    const int sy = active ? pml_slot(j, a.ny, a.L) : -1;
    /* CPML state and per-plane values do not depend on the staged planes:
     * the first plane's are read beside the coefficient table and the first
     * stages, the next ones' as kPsiMode says */
    struct Psi6 {
        int sz;
        R xy, xz, yx, yz, zx, zy;
        ZCoef<R> z;
    };
    auto load_psi = [&](int k, Psi6& p) {
        p.sz = z_slot(a, k);
        p.z = z_coef<R, STRICT, true>(a, p.sz, k);
        p.xy = p.xz = p.yx = p.yz = p.zx = p.zy = R(0);
        if (!active) return;
        const int qx = (k * ny + j) * L2 + sx, qy = (k * L2 + sy) * nxp + i, qz = (p.sz * ny + j) * nxp + i;
        if (sx >= 0) { p.xy = ld_state<LIST>(a.psi.hxy + qx); p.xz = ld_state<LIST>(a.psi.hxz + qx); }
        if (sy >= 0) { p.yx = ld_state<LIST>(a.psi.hyx + qy); p.yz = ld_state<LIST>(a.psi.hyz + qy); }
        if (p.sz >= 0) { p.zx = ld_state<LIST>(a.psi.hzx + qz); p.zy = ld_state<LIST>(a.psi.hzy + qz); }
    };
    Psi6 ps;
    if (!plain) load_psi(k0, ps);
    __syncthreads();
    if (a.stall_test && blockIdx.x == 0 && blockIdx.y == 0 && blockIdx.z == 0) {
        /* failure-path test (StepArgs::stall_test): a bounded wait on the
         * barrier after the ring's, on which nothing ever arrives, gives up
         * like a wait for a plane that never lands */
        const bool ok = mbar_wait_n(&full[G::HS], 0, kStallPolls);
        if (__syncthreads_or(!ok)) {
            if (tid == 0) {
                atomicExch(a.err, 1);
                ring_drain(full, G::HS, h_loads_issued(k0, k0, k1, G::HS));
            }
            chain_leave(a.beside, tid);
            return;
        }
    }

    const int eo = ty * G::BX + tx; /* own cell in a halo box */
    const int ho = ty * G::TX + tx; /* own cell in an own box */

    /* a plain block (no CPML cell, every cell updated; marked on the host):
     * the stencil with the kappa = 1 factors only, the same arithmetic as the
     * general path below takes for such cells */
    if (plain) {
        const R khx = a.khp[0], khy = a.khp[1], khz = a.khp[2];
        for (int k = k0; k < k1; ++k) {
            bool ok = true;
            if (k == k0) ok = mbar_wait(&full[0], 0);
            ok = ok && mbar_wait(&full[(k + 1 - k0) % G::HS], ((k + 1 - k0) / G::HS) & 1);
            if (ok) {
                const R* Ex0 = reinterpret_cast<const R*>(stage(k));
                const R* Ey0 = Ex0 + EBW;
                const R* Ez0 = Ex0 + 2 * EBW;
                const R* Ex1 = reinterpret_cast<const R*>(stage(k + 1));
                const R* Ey1 = Ex1 + EBW;
                const R* Hs = reinterpret_cast<const R*>(stage(k) + G::OWN_AT);
                const R ex0 = Ex0[eo], ey0 = Ey0[eo], ez0 = Ez0[eo];
                const R dEyz = Ey1[eo] - ey0, dEzy = Ez0[eo + G::BX] - ez0, dEzx = Ez0[eo + 1] - ez0;
                const R dExz = Ex1[eo] - ex0, dExy = Ex0[eo + G::BX] - ex0, dEyx = Ey0[eo + 1] - ey0;
                const int c = (k * a.ny + j) * a.nxp + i;
                R hx = Hs[ho], hy = Hs[HBW + ho], hz = Hs[2 * HBW + ho];
                h_update(khx, khy, khz, dEyz, dEzy, dEzx, dExz, dExy, dEyx, R(0), R(0), R(0), R(0), R(0), R(0), hx, hy, hz);
                a.hnew[0][c] = hx;
                a.hnew[1][c] = hy;
                a.hnew[2][c] = hz;
            }
            if (__syncthreads_or(!ok)) {
                if (tid == 0) {
                    atomicExch(a.err, 1);
                    ring_drain(full, G::HS, h_loads_issued(k, k0, k1, G::HS));
                }
                break;
            }
            if (tid == 0 && k + G::HS <= k1) {
                fence_proxy_async_smem();
                issue(k + G::HS);
            }
        }
        chain_leave(a.beside, tid);
        return;
    }

    const R* const xt = tab + 3 * tx;
    const R* const yt = tab + 3 * (32 + ty);
    R* __restrict__ hxg = a.hnew[0];
    R* __restrict__ hyg = a.hnew[1];
    R* __restrict__ hzg = a.hnew[2];

    constexpr int mode = kPsiMode<R, STRICT, false>;
    for (int k = k0; k < k1; ++k) {
        Psi6 pn;
        if (mode == kPsiAhead && k + 1 < k1) load_psi(k + 1, pn);
        if (mode == kPsiTop) {
            if (k > k0) load_psi(k, ps);
            if (active && k + 1 < k1) {
                const int sz1 = z_slot(a, k + 1);
                if (sx >= 0) {
                    const int q = ((k + 1) * ny + j) * L2 + sx;
                    prefetch_state<LIST>(a.psi.hxy + q);
                    prefetch_state<LIST>(a.psi.hxz + q);
                }
                if (sy >= 0) {
                    const int q = ((k + 1) * L2 + sy) * nxp + i;
                    prefetch_state<LIST>(a.psi.hyx + q);
                    prefetch_state<LIST>(a.psi.hyz + q);
                }
                if (sz1 >= 0) {
                    const int q = (sz1 * ny + j) * nxp + i;
                    prefetch_state<LIST>(a.psi.hzx + q);
                    prefetch_state<LIST>(a.psi.hzy + q);
                }
            }
        }
        const int sz = ps.sz;
        const R pxy = ps.xy, pxz = ps.xz, pyx = ps.yx, pyz = ps.yz, pzx = ps.zx, pzy = ps.zy;
        const int qx = (k * ny + j) * L2 + sx, qy = (k * L2 + sy) * nxp + i, qz = (sz * ny + j) * nxp + i;

        bool ok = true;
        if (k == k0) ok = mbar_wait(&full[0], 0);
        ok = ok && mbar_wait(&full[(k + 1 - k0) % G::HS], ((k + 1 - k0) / G::HS) & 1);
        if (ok && active) {
            const R* Ex0 = reinterpret_cast<const R*>(stage(k));
            const R* Ey0 = Ex0 + EBW;
            const R* Ez0 = Ex0 + 2 * EBW;
            const R* Ex1 = reinterpret_cast<const R*>(stage(k + 1));
            const R* Ey1 = Ex1 + EBW;
            const R* Hx0 = reinterpret_cast<const R*>(stage(k) + G::OWN_AT);
            const R* Hy0 = Hx0 + HBW;
            const R* Hz0 = Hx0 + 2 * HBW;
            const R ex0 = Ex0[eo], ey0 = Ey0[eo], ez0 = Ez0[eo];
            const R ex1 = Ex1[eo], ey1 = Ey1[eo];
            const R ezi = Ez0[eo + 1], eyi = Ey0[eo + 1];
            const R ezj = Ez0[eo + G::BX], exj = Ex0[eo + G::BX];
            const R hx0 = Hx0[ho], hy0 = Hy0[ho], hz0 = Hz0[ho];
            const int c = (k * ny + j) * nxp + i;
            if constexpr (STRICT) {
                const double mu0 = a.mu0;
                /* fdtd.c:3132-3137 */
                const double dEy_dz = SOp::div(SOp::sub(ey1, ey0), a.dzs);
                const double dEz_dy = SOp::div(SOp::sub(ezj, ez0), a.dys);
                const double dEz_dx = SOp::div(SOp::sub(ezi, ez0), a.dxs);
                const double dEx_dz = SOp::div(SOp::sub(ex1, ex0), a.dzs);
                const double dEx_dy = SOp::div(SOp::sub(exj, ex0), a.dys);
                const double dEy_dx = SOp::div(SOp::sub(eyi, ey0), a.dxs);
                double kappa_x = 1.0, kappa_y = 1.0, kappa_z = 1.0;
                if (sx >= 0) { /* fdtd.c:3143-3170 */
                    kappa_x = xt[0];
                    const double bb = xt[1], cc = xt[2];
                    a.psi.hxy[qx] = SOp::add(SOp::mul(bb, pxy), SOp::mul(cc, SOp::div(dEz_dx, mu0)));
                    a.psi.hxz[qx] = SOp::add(SOp::mul(bb, pxz), SOp::mul(cc, SOp::div(-dEy_dx, mu0)));
                }
                if (sy >= 0) { /* fdtd.c:3173-3200 */
                    kappa_y = yt[0];
                    const double bb = yt[1], cc = yt[2];
                    a.psi.hyx[qy] = SOp::add(SOp::mul(bb, pyx), SOp::mul(cc, SOp::div(-dEz_dy, mu0)));
                    a.psi.hyz[qy] = SOp::add(SOp::mul(bb, pyz), SOp::mul(cc, SOp::div(dEx_dy, mu0)));
                }
                kappa_z = ps.z.k; /* fdtd.c:3203-3219 */
                /* fdtd.c:3222-3224 */
                const double ux = SOp::add(SOp::add(SOp::add(SOp::div(SOp::div(-dEz_dy, mu0), kappa_y), pyx),
                                                    SOp::div(SOp::div(dEy_dz, mu0), kappa_z)), pzx);
                const double uy = SOp::add(SOp::add(SOp::add(SOp::div(SOp::div(dEz_dx, mu0), kappa_x), pxy),
                                                    SOp::div(SOp::div(-dEx_dz, mu0), kappa_z)), pzy);
                const double uz = SOp::add(SOp::add(SOp::add(SOp::div(SOp::div(-dEy_dx, mu0), kappa_x), pxz),
                                                    SOp::div(SOp::div(dEx_dy, mu0), kappa_y)), pyz);
                hxg[c] = SOp::add(hx0, SOp::mul(a.dt, ux));
                hyg[c] = SOp::add(hy0, SOp::mul(a.dt, uy));
                hzg[c] = SOp::add(hz0, SOp::mul(a.dt, uz));
                if (sz >= 0) { /* fdtd.c:3225-3228 */
                    const double bb = ps.z.b, cc = ps.z.c;
                    a.psi.hzx[qz] = SOp::add(SOp::mul(bb, pzx), SOp::mul(cc, SOp::div(dEy_dz, mu0)));
                    a.psi.hzy[qz] = SOp::add(SOp::mul(bb, pzy), SOp::mul(cc, SOp::div(-dEx_dz, mu0)));
                }
            } else {
                const R dEyz = ey1 - ey0, dEzy = ezj - ez0, dEzx = ezi - ez0;
                const R dExz = ex1 - ex0, dExy = exj - ex0, dEyx = eyi - ey0;
                /* psi terms enter as zeros outside the PML */
                R hx = hx0, hy = hy0, hz = hz0;
                h_update(xt[0], yt[0], ps.z.k, dEyz, dEzy, dEzx, dExz, dExy, dEyx, pxy, pxz, pyx, pyz, pzx, pzy, hx, hy, hz);
                hxg[c] = hx;
                hyg[c] = hy;
                hzg[c] = hz;
                if (sx >= 0) {
                    a.psi.hxy[qx] = curl2(xt[1], pxy, -xt[2], dEzx);
                    a.psi.hxz[qx] = curl2(xt[1], pxz, xt[2], dEyx);
                }
                if (sy >= 0) {
                    a.psi.hyx[qy] = curl2(yt[1], pyx, yt[2], dEzy);
                    a.psi.hyz[qy] = curl2(yt[1], pyz, -yt[2], dExy);
                }
                if (sz >= 0) {
                    a.psi.hzx[qz] = curl2(ps.z.b, pzx, -ps.z.c, dEyz);
                    a.psi.hzy[qz] = curl2(ps.z.b, pzy, ps.z.c, dExz);
                }
            }
        }
        if (mode == kPsiAhead) ps = pn;
        if (mode == kPsiAfter && k + 1 < k1) load_psi(k + 1, ps);
        /* every thread is done with plane k: its stage takes plane k + stages */
        if (__syncthreads_or(!ok)) {
            if (tid == 0) {
                atomicExch(a.err, 1);
                ring_drain(full, G::HS, h_loads_issued(k, k0, k1, G::HS));
            }
            break;
        }
        if (tid == 0 && k + G::HS <= k1) {
            fence_proxy_async_smem();
            issue(k + G::HS);
        }
    }
    chain_leave(a.beside, tid);
}

/* ================================================================ E sweep */

/* fdtd.c:3238-3528 fused, with H and the old E (strict mode: D) streamed
 * through the stage ring; material ids and pool slots are read a plane ahead.
 * Bound by HBM: 9 words per cell (read H, E; write E) plus the CPML and pool
 * state; with D kept for every cell it was 12, and 15 in lossy cells. */
/* The classes of blocks an instantiation holds: a launch over a list of
 * blocks of one kind gets the registers that kind needs. */
enum : int { kEAll = 0, kEPlain = 1, kEAtoms = 2, kEGeneral = 3 };

template <typename R, int NAMAX, int CLS>
constexpr int kEBlocks = CLS == kEPlain ? (sizeof(R) == 4 ? PHP_EP_MINBLOCKS32 : PHP_EP_MINBLOCKS64)
                         : NAMAX > 4 ? 1
                         : CLS == kEAtoms ? (sizeof(R) == 4 ? PHP_EA_MINBLOCKS32 : PHP_EA_MINBLOCKS64)
                         : CLS == kEGeneral ? (sizeof(R) == 4 ? PHP_EG_MINBLOCKS32 : PHP_EG_MINBLOCKS64)
                         : sizeof(R) == 4 ? (kIonVReg<R, NAMAX> ? PHP_E_MINBLOCKS32_ATOMS : PHP_E_MINBLOCKS32)
                         : kIonVReg<R, NAMAX> ? PHP_E_MINBLOCKS64_ATOMS : PHP_E_MINBLOCKS;

template <typename R, bool STRICT, int NAMAX, int CLS>
__global__ void __launch_bounds__(kBlockX * kBlockY, (kEBlocks<R, NAMAX, CLS>))
    e_sweep_tma(const __grid_constant__ StepArgs<R> a, const __grid_constant__ TmaMaps tm)
{
    using G = TmaGeom<R>;
    extern __shared__ __align__(128) unsigned char dyn_smem[];
    unsigned char* smem = ring_base(dyn_smem);
    uint64_t* full = reinterpret_cast<uint64_t*>(smem + G::ES * G::STAGE);
    R* const tab = reinterpret_cast<R*>(smem + G::ES * G::STAGE + 128);

    const int tx = threadIdx.x, ty = threadIdx.y, tid = ty * G::TX + tx;
    constexpr bool CG = CLS == kEPlain || CLS == kEAtoms; /* launches beside others */
    const SweepJob job = sweep_job<CLS != kEAll>(a, a.plain_blk, 255);
    const int i0 = job.bx * G::TX, j0 = job.by * G::TY;
    const int i = i0 + tx, j = j0 + ty;
    const int k0 = job.k0, k1 = job.k1;
    if (k0 >= k1) return; /* uniform over the block */
    const int pm = STRICT || CLS == kEGeneral ? 255 : CLS == kEAtoms ? kPlainAtoms : job.cls; /* StepArgs::plain_blk */
    /* atom blocks without loss do not read the old E */
    const bool with_own = STRICT || pm != kPlainAtoms || (a.amc.flags & kLossy);
    constexpr int HBW = G::HALO_ELEMS, OBW = G::OWN_ELEMS; /* one component in a box */
    /* plane p = k0-1 .. k1-1 into stage (p - k0 + 1) % stages */
    auto stage = [&](int p) -> unsigned char* { return smem + (uint32_t)((p - k0 + 1) % G::ES) * G::STAGE; };
    auto issue = [&](int p) {
        uint64_t* bar = &full[(p - k0 + 1) % G::ES];
        unsigned char* b = stage(p);
        const bool own = p >= k0 && with_own;
        mbar_arrive_expect_tx(bar, G::HALO3_BYTES + (own ? G::OWN3_BYTES : 0u));
        tma_load_plane(b, &tm.h_halo, bar, i0 - G::HALO, j0 - 1, p + 1);
        if (own) tma_load_plane(b + G::OWN_AT, &tm.own, bar, i0, j0, p + 1);
    };

    if (tid == 0) {
        for (int s = 0; s < G::ES; ++s) mbar_init(&full[s], 1);
        fence_barrier_init();
    }
    const bool more = CLS == kEAtoms || CLS == kEGeneral || pm >= kPlainCpml; /* than the stencil */
    if (more) pml_table<R, STRICT, false>(a, tab, i0, j0, G::TY, tid);
    chain_enter(a.beside);
    if (tid == 0)
        for (int p = k0 - 1; p <= min(k1 - 1, k0 - 1 + G::ES - 1); ++p) issue(p);
    const bool active = (i < a.nx) && (j < a.ny);
    const bool interior = (i >= 1 && i < a.nx - 1 && j >= 1 && j < a.ny - 1);
    const int sx = active ? pml_slot(i, a.nx, a.L) : -1;
    const int sy = active ? pml_slot(j, a.ny, a.L) : -1;
    /* what does not come with the stages (CPML state; general path: the
     * material id and the pool slot of ADE, atom and D cells): the first
     * plane's is read beside the coefficient table and the first stages, the
     * next ones' CPML state as kPsiMode says, the rest after the plane before */
    constexpr int mode = kPsiMode<R, STRICT, kIonVReg<R, NAMAX>>;
    /* (not in the FP64 launches of plain and of general blocks: it spills) */
    constexpr bool first = mode != kPsiTop || CLS == kEAll || CLS == kEAtoms;
    const bool slots = !STRICT && a.slot != nullptr && active && (CLS == kEAtoms || CLS == kEGeneral || pm >= kPlainAtoms);
    CellPsi<R> ps;
    int slot = -1, mid = 0;
    if (more) {
        if (first) load_psi_d<R, STRICT, CG>(a, i, j, k0, sx, sy, interior, ps);
        if (slots) slot = ldg(a.slot + (k0 * a.ny + j) * a.nxp + i);
        if (pm == 255 && active) mid = ldg(a.mat + (k0 * a.ny + j) * a.nxp + i);
    }
    __syncthreads();

    const int ho = (ty + 1) * G::BX + tx + G::HALO; /* own cell in a halo box */
    const int oo = ty * G::TX + tx;                 /* own cell in an own box */
    const R* const xt = tab + 3 * tx;
    const R* const yt = tab + 3 * (32 + ty);

    auto wait = [&](int k) -> bool {
        bool ok = true;
        if (k == k0) ok = mbar_wait(&full[0], 0);
        return ok && mbar_wait(&full[(k - k0 + 1) % G::ES], ((k - k0 + 1) / G::ES) & 1);
    };
    /* every thread is done with plane k-1: its stage takes plane k-1 + stages;
     * false when the block gave up */
    auto next = [&](int k, bool ok) -> bool {
        if (__syncthreads_or(!ok)) {
            if (tid == 0) {
                atomicExch(a.err, 1);
                ring_drain(full, G::ES, e_loads_issued(k, k0, k1, G::ES));
            }
            return false;
        }
        if (tid == 0 && k - 1 + G::ES <= k1 - 1) {
            fence_proxy_async_smem();
            issue(k - 1 + G::ES);
        }
        return true;
    };
    /* the cell's H values of planes k and k-1 and its old E (or D) */
    struct Cell {
        R hx0, hy0, hz0, hxk, hyk, hz_jm, hx_jm, hz_im, hy_im;
    };
    auto cell_h = [&](int k) -> Cell {
        const R* Hp = reinterpret_cast<const R*>(stage(k - 1));
        const R* Hx = reinterpret_cast<const R*>(stage(k));
        const R* Hy = Hx + HBW;
        const R* Hz = Hx + 2 * HBW;
        return Cell{Hx[ho], Hy[ho], Hz[ho], Hp[ho], Hp[HBW + ho], Hz[ho - G::BX], Hx[ho - G::BX], Hz[ho - 1], Hy[ho - 1]};
    };
    auto own = [&](int k) -> const R* { return reinterpret_cast<const R*>(stage(k) + G::OWN_AT) + oo; };

    if constexpr (!STRICT) {
        if ((CLS == kEAll || CLS == kEPlain) && pm < kPlainCpml) {
            /* a plain block (one plain isotropic material, no CPML, edge or
             * source cell; marked on the host): E += iso dt curl H with the
             * kappa = 1 factors, nothing per cell beyond the stencil (the same
             * arithmetic as the general path below takes for such cells) */
            const R iso = a.iso[pm];
            const R kdx = a.kdp[0], kdy = a.kdp[1], kdz = a.kdp[2];
            for (int k = k0; k < k1; ++k) {
                const bool ok = wait(k);
                if (ok) {
                    const Cell h = cell_h(k);
                    const R* Es = own(k);
                    R ex = Es[0], ey = Es[OBW], ez = Es[2 * OBW];
                    iso_add(iso, curl2(kdy, h.hz0 - h.hz_jm, kdz, h.hy0 - h.hyk), curl2(kdz, h.hx0 - h.hxk, kdx, h.hz0 - h.hz_im),
                            curl2(kdx, h.hy0 - h.hy_im, kdy, h.hx0 - h.hx_jm), ex, ey, ez);
                    const int c = (k * a.ny + j) * a.nxp + i;
                    a.enew[0][c] = ex;
                    a.enew[1][c] = ey;
                    a.enew[2][c] = ez;
                }
                if (!next(k, ok)) break;
            }
        } else {
            if (CLS != kEGeneral && (CLS != kEAll || pm != 255)) {
                /* one material without a source: plain with CPML or domain-edge
                 * cells, the tensor material of StepArgs::tns_* or (few atoms, or
                 * the ion pass apart) the atom material of StepArgs::amc; its
                 * record comes from the kernel parameters, and what does not
                 * depend on the stages (CPML state, the cell's pool slot) is
                 * read before the wait */
                const bool atoms = CLS == kEAtoms || (CLS == kEAll && pm == kPlainAtoms);
                const R iso = CLS != kEAtoms && pm < kPlainTensor ? a.iso[pm - kPlainCpml] : R(0);
                for (int k = k0; k < k1; ++k) {
                    CellPsi<R> pn;
                    if (mode == kPsiAhead && k + 1 < k1) load_psi_d<R, false, CG>(a, i, j, k + 1, sx, sy, interior, pn);
                    if (mode == kPsiTop) {
                        if (!first || k > k0) load_psi_d<R, false, CG>(a, i, j, k, sx, sy, interior, ps);
                        if (interior && k + 1 < k1) prefetch_psi_d<CG>(a, i, j, k + 1, sx, sy);
                    }
                    const int c = (k * a.ny + j) * a.nxp + i;
                    IonPre ip;
                    ip.slot = slot;
                    if constexpr (NAMAX <= 4 && CLS != kEPlain) {
                        if (atoms && active) {
                            /* its D, and r and v (or P_ion), requested ahead of their reads */
                            constexpr int QN = 3 * NAMAX;
                            const int n3 = 3 * a.amc.natom;
                            if (a.Dc) prefetch_state<CG>(a.Dc + ip.slot);
#pragma unroll
                            for (int q = 0; q < 3; ++q) {
                                prefetch_state<CG>(a.Dp + q * a.nslot + ip.slot);
                                if (NAMAX == 0 && a.pr) prefetch_state<CG>(a.pr + q * a.nslot + ip.slot);
                            }
#pragma unroll
                            for (int q = 0; q < QN; ++q) {
                                const int64_t o = (int64_t)q * a.nslot + ip.slot;
                                if (q < n3) {
                                    prefetch_state<CG>(a.r + o);
                                    prefetch_state<CG>(a.v + o);
                                }
                            }
                        }
                    }
                    const bool ok = wait(k);
                    if (ok && active) {
                        const Cell h = cell_h(k);
                        const R* Es = own(k);
                        R ex = R(0), ey = R(0), ez = R(0);
                        if (with_own) {
                            ex = Es[0];
                            ey = Es[OBW];
                            ez = Es[2 * OBW];
                        }
                        R ux = R(0), uy = R(0), uz = R(0);
                        if (interior) {
                            d_update<R, false>(a, i, j, k, sx, sy, h.hx0, h.hy0, h.hz0, h.hxk, h.hyk, h.hz_jm, h.hx_jm,
                                               h.hz_im, h.hy_im, ps, xt, yt, ux, uy, uz);
                            if (CLS != kEAtoms && pm == kPlainTensor && (a.tns_flags & kLossy)) loss_sub(a.tns_im, ex, ey, ez, ux, uy, uz);
                            if (atoms && (a.amc.flags & kLossy)) loss_sub(a.amc.eps_im, ex, ey, ez, ux, uy, uz);
                        }
                        if (CLS != kEAtoms && pm < kPlainTensor) {
                            iso_add(iso, ux, uy, uz, ex, ey, ez);
                        } else if (CLS == kEPlain || (CLS == kEAll && pm == kPlainTensor)) {
                            e_only_add(a.tns_em, ux, uy, uz, ex, ey, ez);
                        } else if constexpr (NAMAX <= 4 && CLS != kEPlain) {
                            const int64_t ns = a.nslot;
                            R* __restrict__ dp = a.Dp + ip.slot;
                            R dx, dy, dz;
                            pool_add<R, CG>(a, ip.slot, ux, uy, uz, dx, dy, dz);
                            e_update<R, false, NAMAX, CG>(a, a.amc, c, dx, dy, dz, ux, uy, uz, ex, ey, ez, &ip);
                            dp[0] = dx;
                            dp[ns] = dy;
                            dp[2 * ns] = dz;
                        }
                        a.enew[0][c] = ex;
                        a.enew[1][c] = ey;
                        a.enew[2][c] = ez;
                    }
                    if (mode == kPsiAhead) ps = pn;
                    if (mode == kPsiAfter && k + 1 < k1) load_psi_d<R, false, CG>(a, i, j, k + 1, sx, sy, interior, ps);
                    if (atoms && slots && k + 1 < k1) slot = ldg(a.slot + ((k + 1) * a.ny + j) * a.nxp + i);
                    if (!next(k, ok)) break;
                }
            } else if (CLS == kEAll || CLS == kEGeneral) {
                /* the general path: the lines of a cell's pool state are
                 * requested before the stage wait */
                for (int k = k0; k < k1; ++k) {
                    CellPsi<R> pn;
                    if (mode == kPsiAhead && k + 1 < k1) load_psi_d<R, false, CG>(a, i, j, k + 1, sx, sy, interior, pn);
                    if (mode == kPsiTop) {
                        if (!first || k > k0) load_psi_d<R, false, CG>(a, i, j, k, sx, sy, interior, ps);
                        if (interior && k + 1 < k1) prefetch_psi_d<CG>(a, i, j, k + 1, sx, sy);
                    }
                    if (slot >= 0) {
                        const int64_t ns = a.nslot;
#pragma unroll
                        for (int q = 0; q < 3; ++q) {
                            prefetch_state<CG>(a.Dp + q * ns + slot);
                            if (a.P) {
                                prefetch_state<CG>(a.P + q * ns + slot);
                                prefetch_state<CG>(a.Po + q * ns + slot);
                            }
                            if (NAMAX == 0 && a.pr) prefetch_state<CG>(a.pr + q * ns + slot);
                        }
                    }
                    const bool ok = wait(k);
                    if (ok && active) {
                        const Cell h = cell_h(k);
                        const R* Es = own(k);
                        const int c = (k * a.ny + j) * a.nxp + i;
                        R ex = Es[0], ey = Es[OBW], ez = Es[2 * OBW];
                        e_cell_fast<R, NAMAX>(a, i, j, k, c, interior, sx, sy, h.hx0, h.hy0, h.hz0, h.hxk, h.hyk, h.hz_jm,
                                              h.hx_jm, h.hz_im, h.hy_im, mid, ps, xt, yt, ex, ey, ez, slot);
                        a.enew[0][c] = ex;
                        a.enew[1][c] = ey;
                        a.enew[2][c] = ez;
                    }
                    if (mode == kPsiAhead) ps = pn;
                    if (mode == kPsiAfter && k + 1 < k1) load_psi_d<R, false, CG>(a, i, j, k + 1, sx, sy, interior, ps);
                    if (slots && k + 1 < k1) slot = ldg(a.slot + ((k + 1) * a.ny + j) * a.nxp + i);
                    if (active && k + 1 < k1) mid = ldg(a.mat + ((k + 1) * a.ny + j) * a.nxp + i);
                    if (!next(k, ok)) break;
                }
            }
        }
    } else {
        for (int k = k0; k < k1; ++k) {
            const bool ok = wait(k);
            if (ok && active) {
                const Cell h = cell_h(k);
                const R* Ds = own(k);
                e_cell_strict<NAMAX>(a, i, j, k, (k * a.ny + j) * a.nxp + i, interior, sx, sy, h.hx0, h.hy0, h.hz0, h.hxk,
                                     h.hyk, h.hz_jm, h.hx_jm, h.hz_im, h.hy_im, Ds[0], Ds[OBW], Ds[2 * OBW], mid, ps, xt, yt);
            }
            if (k + 1 < k1) {
                load_psi_d<R, true>(a, i, j, k + 1, sx, sy, interior, ps);
                if (active) mid = ldg(a.mat + ((k + 1) * a.ny + j) * a.nxp + i);
            }
            if (!next(k, ok)) break;
        }
    }
    /* after the march: the running DFT samples and the monitor row of this
     * chunk's planes */
    if (a.ndft) dft_fold<CG>(a, a.enew, i, j, k0, k1);
    if (a.probe_rows) probe_fold<CG>(a, a.enew, a.hnew, i, j, k0, k1);
    chain_leave(a.beside, tid);
}

} // namespace phpdev

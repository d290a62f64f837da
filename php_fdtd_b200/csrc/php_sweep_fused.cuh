/*
 * php_sweep_fused.cuh -- the time step of fdtd.c:3116-3528 in one launch
 * (sm_100a): the H sweep and the fused D / source / E / ADE / ion sweep of
 * php_sweeps_tma.cuh in a single z march per block.
 *
 * The two sweeps read H and E twice per step.  Here the block of an
 * (x, y) tile and z range computes, plane by plane, the new H of its tile and
 * of the cells one below it in x and y (its D update needs their H; they
 * belong to the neighbouring tiles and are computed twice), and updates E
 * from it: E and H cross HBM once per step in each direction (12 words per
 * cell; the two sweeps move 18), and one launch replaces two.
 *
 * Two rings of shared-memory stages are fed by TMA (tile mode, no multicast,
 * this GPU's own memory only): E^n on the tile widened by one cell on every
 * side (x widened to 16 bytes), and H^{n-1/2} on the tile and the cells
 * below it.  What bounds the march is the latency of those loads, so the
 * stages come free as early as the data allow:
 *   - the own cell's E of plane p is carried in registers from its load at
 *     plane p - 1, and its neighbours' E is only read by the H part, so the
 *     stage of E plane p takes plane p + SE at the barrier between the two
 *     parts of plane p (loads 2 planes ahead with three stages);
 *   - the new H overwrites the old one in its stage (nobody else reads the
 *     old H of a cell), so no second H tile is needed, and the stage of H
 *     plane p - 1 takes plane p - 1 + SH at the barrier of plane p.
 * With one E and H stage freed only a full plane later (and D staged beside
 * them) an earlier form of this kernel ran at half the copy bandwidth.
 *
 * The march starts one plane below the block's range (the E update of plane
 * k0 needs the new H of plane k0 - 1, computed again here) and reads E one
 * plane above it, so ranges are long (StepArgs::zstep, chosen on the host so
 * that the blocks fill whole waves), and block classes are kept per plane
 * (StepArgs::pcls) so that a long range keeps the short paths.
 *
 * The cells below the tile are updated by their own blocks during the same
 * launch, so their old E, H and H CPML state must stay readable: those are
 * double buffered (the launch reads StepArgs::f and psi, and writes the new
 * level to enew, hnew and psin_h; the host swaps the buffers after the
 * launch).  The D CPML state and the pools belong to one cell each and are
 * updated in place.  The arithmetic per cell is that of the two sweeps,
 * operation for operation, so both paths give the same fields.
 *
 * Waits are bounded as in the two sweeps (kWaitLimit polls, error flag,
 * drain of the loads in flight).
 */
#pragma once

namespace phpdev {

/* he_sweep_tma: rows of the tile per thread and resident blocks per SM the
 * kernel is compiled for.  Its paths for CPML, ADE and atom cells want 80
 * registers and more: at 64 they spill, and with the stages taking nearly all
 * of an SM's shared memory the spilled values miss L1. */
#ifndef PHP_STEP_ROWS64
#define PHP_STEP_ROWS64 1
#endif
#ifndef PHP_STEP_ROWS32
#define PHP_STEP_ROWS32 2
#endif
#ifndef PHP_STEP_MINB64
#define PHP_STEP_MINB64 3
#endif
#ifndef PHP_STEP_MINB32
#define PHP_STEP_MINB32 3
#endif
/* interior_sweep_tma: the same */
#ifndef PHP_INNER_ROWS64
#define PHP_INNER_ROWS64 2
#endif
#ifndef PHP_INNER_ROWS32
#define PHP_INNER_ROWS32 2
#endif
#ifndef PHP_INNER_MINB64
#define PHP_INNER_MINB64 2
#endif
#ifndef PHP_INNER_MINB32
#define PHP_INNER_MINB32 4
#endif
/* ring depths of E and H */
#ifndef PHP_STEP_SE
#define PHP_STEP_SE 3
#endif
#ifndef PHP_STEP_SH
#define PHP_STEP_SH 3
#endif

__host__ __device__ constexpr uint32_t align128u(uint32_t b) { return (b + 127u) / 128u * 128u; }

/* INNER: interior_sweep_tma, else he_sweep_tma */
template <typename R, bool INNER>
struct FusedGeom {
    static constexpr int ROWS = INNER ? (sizeof(R) == 8 ? PHP_INNER_ROWS64 : PHP_INNER_ROWS32)
                                      : (sizeof(R) == 8 ? PHP_STEP_ROWS64 : PHP_STEP_ROWS32);
    static constexpr int TX = kBlockX, TY = kBlockY * ROWS;
    static constexpr int HALO = 16 / (int)sizeof(R);
    static constexpr int EX = TX + 2 * HALO, EY = TY + 2; /* E box: x from i0 - HALO, y from j0 - 1 */
    static constexpr int HX = TX + HALO, HY = TY + 1;     /* H box: x from i0 - HALO, y from j0 - 1 */
    static constexpr int NHALO = TX + 1 + TY;             /* cells below the tile: row j0 - 1, column i0 - 1 */
    static constexpr int EBW = EX * EY, HBW = HX * HY;    /* one component in a box */
    static constexpr uint32_t E3_BYTES = 3 * EBW * sizeof(R), H3_BYTES = 3 * HBW * sizeof(R);
    static constexpr uint32_t EB = align128u(E3_BYTES), HB = align128u(H3_BYTES); /* a stage of each ring */
    static constexpr int SE = PHP_STEP_SE, SH = PHP_STEP_SH;
    /* the H part of plane p reads E planes p and p + 1, and H plane p - 1 is
     * still read while plane p's is staged */
    static_assert(SE >= 2 && SH >= 2, "he_sweep_tma needs two stages of each ring");
    static_assert(NHALO <= kBlockX * kBlockY, "one cell below the tile per thread");
    /* alignment slack, the stages, their barriers and the failure-path test's */
    static constexpr uint32_t SMEM = 128 + SE * EB + SH * HB + 128 + (INNER ? 0u : align128u(pml_table_len(TY) * sizeof(R)));
};

/* per-plane block classes (StepArgs::pcls): the fused sweep's plain-block
 * code, plus kHPlain where the H part needs no CPML term and updates every
 * cell of the tile and of the cells below it */
constexpr uint32_t kHPlain = 256;

/* the old H CPML state of cell (i, j) of plane k into psi[6]: xy xz yx yz zx zy */
template <typename R>
__device__ __forceinline__ void h_psi_load(const StepArgs<R>& a, int sx, int sy, int sz, int i, int j, int k, R* psi)
{
    const int L2 = 2 * a.L;
    if (sx >= 0) {
        const int q = (k * a.ny + j) * L2 + sx;
        psi[0] = a.psi.hxy[q];
        psi[1] = a.psi.hxz[q];
    }
    if (sy >= 0) {
        const int q = (k * L2 + sy) * a.nxp + i;
        psi[2] = a.psi.hyx[q];
        psi[3] = a.psi.hyz[q];
    }
    if (sz >= 0) {
        const int q = (sz * a.ny + j) * a.nxp + i;
        psi[4] = a.psi.hzx[q];
        psi[5] = a.psi.hzy[q];
    }
}

/* the lines h_psi_load reads, requested into L1 */
template <typename R>
__device__ __forceinline__ void h_psi_prefetch(const StepArgs<R>& a, int sx, int sy, int sz, int i, int j, int k)
{
    const int L2 = 2 * a.L;
    if (sx >= 0) {
        const int q = (k * a.ny + j) * L2 + sx;
        asm volatile("prefetch.global.L1 [%0];" ::"l"(a.psi.hxy + q));
        asm volatile("prefetch.global.L1 [%0];" ::"l"(a.psi.hxz + q));
    }
    if (sy >= 0) {
        const int q = (k * L2 + sy) * a.nxp + i;
        asm volatile("prefetch.global.L1 [%0];" ::"l"(a.psi.hyx + q));
        asm volatile("prefetch.global.L1 [%0];" ::"l"(a.psi.hyz + q));
    }
    if (sz >= 0) {
        const int q = (sz * a.ny + j) * a.nxp + i;
        asm volatile("prefetch.global.L1 [%0];" ::"l"(a.psi.hzx + q));
        asm volatile("prefetch.global.L1 [%0];" ::"l"(a.psi.hzy + q));
    }
}

/* the six E differences of the curl in the H update (fdtd.c:3132-3137) */
template <typename R>
struct HCurl {
    R dEyz, dEzy, dEzx, dExz, dExy, dEyx;
};

/* H of one cell with its CPML terms (the general path of h_sweep_tma); with
 * `store` the new CPML state goes to StepArgs::psin_h (the block's own cells;
 * the cells below the tile are only read) */
template <typename R>
__device__ __forceinline__ void h_cpml(const StepArgs<R>& a, const HCurl<R>& d, int sx, int sy, int sz, int i, int j, int k,
                                       R& hx, R& hy, R& hz, bool store)
{
    R psi[6] = {R(0), R(0), R(0), R(0), R(0), R(0)};
    h_psi_load(a, sx, sy, sz, i, j, k, psi);
    /* psi terms enter as zeros outside the PML */
    h_update(ldg(a.tx.kh + i), ldg(a.ty.kh + j), ldg_nh(a.tz.kh + k), d.dEyz, d.dEzy, d.dEzx, d.dExz, d.dExy, d.dEyx, psi[0],
             psi[1], psi[2], psi[3], psi[4], psi[5], hx, hy, hz);
    if (!store) return;
    const int L2 = 2 * a.L;
    if (sx >= 0) {
        const R bb = ldg_nh(a.tx.b + i), ch = ldg_nh(a.tx.ch + i);
        const int q = (k * a.ny + j) * L2 + sx;
        a.psin_h[0][q] = curl2(bb, psi[0], -ch, d.dEzx);
        a.psin_h[1][q] = curl2(bb, psi[1], ch, d.dEyx);
    }
    if (sy >= 0) {
        const R bb = ldg_nh(a.ty.b + j), ch = ldg_nh(a.ty.ch + j);
        const int q = (k * L2 + sy) * a.nxp + i;
        a.psin_h[2][q] = curl2(bb, psi[2], ch, d.dEzy);
        a.psin_h[3][q] = curl2(bb, psi[3], -ch, d.dExy);
    }
    if (sz >= 0) {
        const R bb = ldg_nh(a.tz.b + k), ch = ldg_nh(a.tz.ch + k);
        const int q = (sz * a.ny + j) * a.nxp + i;
        a.psin_h[4][q] = curl2(bb, psi[4], -ch, d.dEyz);
        a.psin_h[5][q] = curl2(bb, psi[5], ch, d.dExz);
    }
}

template <typename R, int NAMAX>
constexpr int kStepBlocks = NAMAX > 4 ? 1
                            : sizeof(R) == 8 ? (kIonVReg<R, NAMAX> ? 2 : PHP_STEP_MINB64)
                                             : PHP_STEP_MINB32;

template <typename R, int NAMAX>
__global__ void __launch_bounds__(kBlockX * kBlockY, (kStepBlocks<R, NAMAX>))
    he_sweep_tma(const __grid_constant__ StepArgs<R> a, const __grid_constant__ TmaMaps tm)
{
    using G = FusedGeom<R, false>;
    constexpr int SE = G::SE, SH = G::SH, ROWS = G::ROWS;
    constexpr int EBW = G::EBW, HBW = G::HBW, ES = G::EB / (int)sizeof(R), HS = G::HB / (int)sizeof(R);
    extern __shared__ __align__(128) unsigned char dyn_smem[];
    unsigned char* smem = ring_base(dyn_smem);
    R* const ering = reinterpret_cast<R*>(smem);              /* [SE] stages of [3][EBW] */
    R* const hring = reinterpret_cast<R*>(smem + SE * G::EB); /* [SH] stages of [3][HBW] */
    uint64_t* const ebar = reinterpret_cast<uint64_t*>(smem + SE * G::EB + SH * G::HB);
    uint64_t* const hbar = ebar + SE;
    R* const tab = reinterpret_cast<R*>(smem + SE * G::EB + SH * G::HB + 128);

    const int tx = threadIdx.x, ty = threadIdx.y, tid = ty * G::TX + tx;
    const int i0 = blockIdx.x * G::TX, j0 = blockIdx.y * G::TY;
    const int i = i0 + tx, j = j0 + ty * ROWS; /* the thread's first row */
    const int k0 = blockIdx.z * a.zstep;
    const int k1 = min(k0 + a.zstep, a.nz);
    if (k0 >= k1) return; /* uniform over the block */
    const int nE = k1 - k0 + 2, nH = k1 - k0 + 1; /* planes k0-1 .. k1 of E, k0-1 .. k1-1 of H */

    /* plane k0 - 1 + g into stage g % S of its ring (the field arrays have a
     * zero halo plane on either end) */
    auto issue_e = [&](int g) {
        uint64_t* bar = &ebar[g % SE];
        R* b = ering + (g % SE) * ES;
        mbar_arrive_expect_tx(bar, G::E3_BYTES);
        tma_load_plane(b, &tm.e_wide, bar, i0 - G::HALO, j0 - 1, k0 + g);
    };
    auto issue_h = [&](int g) {
        uint64_t* bar = &hbar[g % SH];
        R* b = hring + (g % SH) * HS;
        mbar_arrive_expect_tx(bar, G::H3_BYTES);
        tma_load_plane(b, &tm.h_wide, bar, i0 - G::HALO, j0 - 1, k0 + g);
    };
    /* after a wait gave up at plane g: the loads issued so far */
    auto drain = [&](int g) {
        ring_drain(ebar, SE, (uint32_t)min(nE, SE + g));
        ring_drain(hbar, SH, (uint32_t)min(nH, SH + max(0, g - 1)));
    };

    if (tid == 0) {
        for (int s = 0; s < SE + SH + 1; ++s) mbar_init(&ebar[s], 1);
        fence_barrier_init();
    }
    pml_table<R, false, false>(a, tab, i0, j0, G::TY, tid);
    chain_enter(a.beside);
    __syncthreads();
    if (tid == 0) {
        for (int g = 0; g < max(SE, SH); ++g) {
            if (g < SE && g < nE) issue_e(g);
            if (g < SH && g < nH) issue_h(g);
        }
    }
    if (a.stall_test && blockIdx.x == 0 && blockIdx.y == 0 && blockIdx.z == 0) {
        /* failure-path test (StepArgs::stall_test), as in h_sweep_tma */
        const bool ok = mbar_wait_n(&hbar[SH], 0, kStallPolls);
        if (__syncthreads_or(!ok)) {
            if (tid == 0) {
                atomicExch(a.err, 1);
                drain(0);
            }
            return;
        }
    }

    const uint16_t* pcls = a.pcls + ((size_t)k0 * gridDim.y + blockIdx.y) * gridDim.x + blockIdx.x;
    const size_t pstride = (size_t)gridDim.x * gridDim.y;

    const bool icol = i < a.nx, iin = i >= 1 && i < a.nx - 1, ih = i < a.nx - 1;
    const int slot_i = icol ? pml_slot(i, a.nx, a.L) : -1;
    int slot_j[ROWS];
#pragma unroll
    for (int r = 0; r < ROWS; ++r) slot_j[r] = j + r < a.ny ? pml_slot(j + r, a.ny, a.L) : -1;
    /* the cell below the tile this thread computes H of as well (tid < NHALO):
     * the row j0 - 1 from i0 - 1, then the column i0 - 1 */
    const int ci = tid <= G::TX ? i0 - 1 + tid : i0 - 1;
    const int cj = tid <= G::TX ? j0 - 1 : j0 + tid - G::TX - 1;
    const bool halo = tid < G::NHALO && ci >= 0 && cj >= 0 && ci < a.nx && cj < a.ny;
    const bool halo_upd = halo && ci < a.nx - 1 && cj < a.ny - 1;

    /* offsets of the own cell (row 0) in the boxes, of the cell below the tile */
    const int eo = (ty * ROWS + 1) * G::EX + tx + G::HALO;
    const int ho = (ty * ROWS + 1) * G::HX + tx + G::HALO;
    const int ce = (cj - j0 + 1) * G::EX + (ci - i0 + G::HALO);
    const int ch = (cj - j0 + 1) * G::HX + (ci - i0 + G::HALO);

    R e0[ROWS][3];   /* E of the own cells at plane p */
    R hk[ROWS][2];   /* new Hx, Hy of the own cells at plane p - 1 */
#pragma unroll
    for (int r = 0; r < ROWS; ++r) {
        e0[r][0] = e0[r][1] = e0[r][2] = R(0);
        hk[r][0] = hk[r][1] = R(0);
    }
    /* class of the plane, read a plane ahead (plane k0 - 1: only its H part) */
    uint32_t cls_next = k0 > 0 ? pcls[-(ptrdiff_t)pstride] : kHPlain;

    for (int g = 0; g < nH; ++g) {
        const int p = k0 - 1 + g;
        const bool eph = g > 0; /* E of plane p this pass */
        const uint32_t cls = cls_next;
        if (g + 1 < nH) cls_next = pcls[(size_t)g * pstride];
        const int pm = (int)(cls & 255u);
        const bool hplain = (cls & kHPlain) != 0;
        const int c0 = (p * a.ny + j) * a.nxp + i;
        const R* const Eb0 = ering + (g % SE) * ES;
        const R* const Eb1 = ering + ((g + 1) % SE) * ES;
        R* const Hb = hring + (g % SH) * HS;

        /* per-cell state that does not come with the stages: requested a
         * plane ahead (CPML lines) or read before the wait (pool slots) */
        int szp = -1;
        if (!hplain && p >= 0) {
            szp = z_slot(a, p);
            if (p + 1 < k1) {
                const int sz1 = z_slot(a, p + 1);
#pragma unroll
                for (int r = 0; r < ROWS; ++r) {
                    if (ih && j + r < a.ny - 1) h_psi_prefetch(a, slot_i, slot_j[r], sz1, i, j + r, p + 1);
                    if (iin && j + r >= 1 && j + r < a.ny - 1) prefetch_psi_d<false>(a, i, j + r, p + 1, slot_i, slot_j[r]);
                }
                if (halo_upd) h_psi_prefetch(a, pml_slot(ci, a.nx, a.L), pml_slot(cj, a.ny, a.L), sz1, ci, cj, p + 1);
            }
        }
        int slot[ROWS], mid[ROWS];
#pragma unroll
        for (int r = 0; r < ROWS; ++r) {
            slot[r] = -1;
            mid[r] = 0;
            if (eph && pm >= kPlainAtoms && icol && j + r < a.ny) {
                const int c = c0 + r * a.nxp;
                if (pm == 255) mid[r] = a.mat[c];
                if (a.slot) slot[r] = a.slot[c];
                if (slot[r] >= 0) {
                    const int64_t ns = a.nslot;
#pragma unroll
                    for (int q = 0; q < 3; ++q) {
                        asm volatile("prefetch.global.L1 [%0];" ::"l"(a.Dp + q * ns + slot[r]));
                        if (a.P) {
                            asm volatile("prefetch.global.L1 [%0];" ::"l"(a.P + q * ns + slot[r]));
                            asm volatile("prefetch.global.L1 [%0];" ::"l"(a.Po + q * ns + slot[r]));
                        }
                        if (NAMAX == 0 && a.pr) asm volatile("prefetch.global.L1 [%0];" ::"l"(a.pr + q * ns + slot[r]));
                    }
                    if (NAMAX > 0 && NAMAX <= 4 && pm == kPlainAtoms) {
                        const int n3 = 3 * a.amc.natom;
#pragma unroll
                        for (int q = 0; q < 3 * NAMAX; ++q) {
                            if (q < n3) {
                                asm volatile("prefetch.global.L1 [%0];" ::"l"(a.r + q * ns + slot[r]));
                                asm volatile("prefetch.global.L1 [%0];" ::"l"(a.v + q * ns + slot[r]));
                            }
                        }
                    }
                }
            }
        }

        bool ok = true;
        if (g == 0) ok = mbar_wait(&ebar[0], 0);
        ok = ok && mbar_wait(&hbar[g % SH], (g / SH) & 1);
        ok = ok && mbar_wait(&ebar[(g + 1) % SE], ((g + 1) / SE) & 1);

        /* ---- H of plane p: the own cells, and the cell below the tile */
        R h[ROWS][3], e1[ROWS][3];
#pragma unroll
        for (int r = 0; r < ROWS; ++r) {
            h[r][0] = h[r][1] = h[r][2] = R(0); /* plane -1: the zero halo plane */
            e1[r][0] = e1[r][1] = e1[r][2] = R(0);
        }
        if (ok) {
            const R khx = a.khp[0], khy = a.khp[1], khz = a.khp[2];
            if (g == 0) {
#pragma unroll
                for (int r = 0; r < ROWS; ++r)
#pragma unroll
                    for (int q = 0; q < 3; ++q) e0[r][q] = Eb0[q * EBW + eo + r * G::EX];
            }
#pragma unroll
            for (int r = 0; r < ROWS; ++r)
#pragma unroll
                for (int q = 0; q < 3; ++q) e1[r][q] = Eb1[q * EBW + eo + r * G::EX];
            if (p >= 0) {
#pragma unroll
                for (int r = 0; r < ROWS; ++r) {
                    const int er = eo + r * G::EX, hr = ho + r * G::HX;
                    R hx = Hb[hr], hy = Hb[HBW + hr], hz = Hb[2 * HBW + hr];
                    HCurl<R> d;
                    d.dEyz = e1[r][1] - e0[r][1];
                    d.dExz = e1[r][0] - e0[r][0];
                    d.dEzx = Eb0[2 * EBW + er + 1] - e0[r][2];
                    d.dEyx = Eb0[EBW + er + 1] - e0[r][1];
                    d.dEzy = (r + 1 < ROWS ? e0[r + 1 < ROWS ? r + 1 : r][2] : Eb0[2 * EBW + er + G::EX]) - e0[r][2];
                    d.dExy = (r + 1 < ROWS ? e0[r + 1 < ROWS ? r + 1 : r][0] : Eb0[er + G::EX]) - e0[r][0];
                    if (hplain) {
                        h_update(khx, khy, khz, d.dEyz, d.dEzy, d.dEzx, d.dExz, d.dExy, d.dEyx, R(0), R(0), R(0), R(0), R(0),
                                 R(0), hx, hy, hz);
                    } else if (ih && j + r < a.ny - 1) {
                        h_cpml(a, d, slot_i, slot_j[r], szp, i, j + r, p, hx, hy, hz, eph);
                    }
                    h[r][0] = hx;
                    h[r][1] = hy;
                    h[r][2] = hz;
                    if (eph) {
                        if (hplain || (icol && j + r < a.ny)) {
                            const int c = c0 + r * a.nxp;
                            a.hnew[0][c] = hx;
                            a.hnew[1][c] = hy;
                            a.hnew[2][c] = hz;
                        }
                        Hb[hr] = hx;
                        Hb[HBW + hr] = hy;
                        Hb[2 * HBW + hr] = hz;
                    }
                }
                if (eph && halo) {
                    R qx = Hb[ch], qy = Hb[HBW + ch], qz = Hb[2 * HBW + ch];
                    const R cx = Eb0[ce], cy = Eb0[EBW + ce], cz = Eb0[2 * EBW + ce];
                    HCurl<R> d;
                    d.dEyz = Eb1[EBW + ce] - cy;
                    d.dExz = Eb1[ce] - cx;
                    d.dEzx = Eb0[2 * EBW + ce + 1] - cz;
                    d.dEyx = Eb0[EBW + ce + 1] - cy;
                    d.dEzy = Eb0[2 * EBW + ce + G::EX] - cz;
                    d.dExy = Eb0[ce + G::EX] - cx;
                    if (hplain) {
                        h_update(khx, khy, khz, d.dEyz, d.dEzy, d.dEzx, d.dExz, d.dExy, d.dEyx, R(0), R(0), R(0), R(0), R(0),
                                 R(0), qx, qy, qz);
                    } else if (halo_upd) {
                        h_cpml(a, d, pml_slot(ci, a.nx, a.L), pml_slot(cj, a.ny, a.L), szp, ci, cj, p, qx, qy, qz, false);
                    }
                    Hb[ch] = qx;
                    Hb[HBW + ch] = qy;
                    Hb[2 * HBW + ch] = qz;
                }
            }
        }
        /* the new H of plane p is in its stage; every thread is done with the
         * E stage of plane p and with H plane p - 1 (whose stage this block
         * wrote: ordered before the loads that overwrite it) */
        fence_proxy_async_smem();
        if (__syncthreads_or(!ok)) {
            if (tid == 0) {
                atomicExch(a.err, 1);
                drain(g);
            }
            break;
        }
        if (tid == 0) {
            fence_proxy_async_smem();
            if (g + SE < nE) issue_e(g + SE);
            if (g >= 1 && g - 1 + SH < nH) issue_h(g - 1 + SH);
        }

        /* ---- E of plane p */
        if (eph) {
#pragma unroll
            for (int r = 0; r < ROWS; ++r) {
                const int hr = ho + r * G::HX;
                const R hx = h[r][0], hy = h[r][1], hz = h[r][2];
                const R hz_jm = r > 0 ? h[r > 0 ? r - 1 : 0][2] : Hb[2 * HBW + hr - G::HX];
                const R hx_jm = r > 0 ? h[r > 0 ? r - 1 : 0][0] : Hb[hr - G::HX];
                const R hz_im = Hb[2 * HBW + hr - 1], hy_im = Hb[HBW + hr - 1];
                const int c = c0 + r * a.nxp;
                R ex = e0[r][0], ey = e0[r][1], ez = e0[r][2];
                if (pm < kPlainCpml) {
                    /* one plain material, no CPML, edge or source cell */
                    const R kdx = a.kdp[0], kdy = a.kdp[1], kdz = a.kdp[2];
                    iso_add(a.iso[pm], curl2(kdy, hz - hz_jm, kdz, hy - hk[r][1]), curl2(kdz, hx - hk[r][0], kdx, hz - hz_im),
                            curl2(kdx, hy - hy_im, kdy, hx - hx_jm), ex, ey, ez);
                    a.enew[0][c] = ex;
                    a.enew[1][c] = ey;
                    a.enew[2][c] = ez;
                } else if (icol && j + r < a.ny) {
                    const bool interior = iin && j + r >= 1 && j + r < a.ny - 1;
                    CellPsi<R> ps;
                    load_psi_d(a, i, j + r, p, slot_i, slot_j[r], interior, ps);
                    const R* const xt = tab + 3 * tx;
                    const R* const yt = tab + 3 * (32 + ty * ROWS + r);
                    if (pm == 255) {
                        e_cell_fast<R, NAMAX>(a, i, j + r, p, c, interior, slot_i, slot_j[r], hx, hy, hz, hk[r][0], hk[r][1],
                                              hz_jm, hx_jm, hz_im, hy_im, mid[r], ps, xt, yt, ex, ey, ez, slot[r]);
                    } else {
                        /* one material without a source, as in e_sweep_tma */
                        const bool atoms = pm == kPlainAtoms;
                        R ux = R(0), uy = R(0), uz = R(0);
                        if (interior) {
                            d_update<R, false>(a, i, j + r, p, slot_i, slot_j[r], hx, hy, hz, hk[r][0], hk[r][1], hz_jm, hx_jm,
                                               hz_im, hy_im, ps, xt, yt, ux, uy, uz);
                            if (pm == kPlainTensor && (a.tns_flags & kLossy)) loss_sub(a.tns_im, ex, ey, ez, ux, uy, uz);
                            if (atoms && (a.amc.flags & kLossy)) loss_sub(a.amc.eps_im, ex, ey, ez, ux, uy, uz);
                        }
                        if (pm < kPlainTensor) {
                            iso_add(a.iso[pm - kPlainCpml], ux, uy, uz, ex, ey, ez);
                        } else if (pm == kPlainTensor) {
                            e_only_add(a.tns_em, ux, uy, uz, ex, ey, ez);
                        } else if constexpr (NAMAX <= 4) {
                            const int64_t ns = a.nslot;
                            IonPre ip;
                            ip.slot = slot[r];
                            R* __restrict__ dp = a.Dp + ip.slot;
                            R dx, dy, dz;
                            pool_add(a, ip.slot, ux, uy, uz, dx, dy, dz);
                            e_update<R, false, NAMAX>(a, a.amc, c, dx, dy, dz, ux, uy, uz, ex, ey, ez, &ip);
                            dp[0] = dx;
                            dp[ns] = dy;
                            dp[2 * ns] = dz;
                        }
                    }
                    a.enew[0][c] = ex;
                    a.enew[1][c] = ey;
                    a.enew[2][c] = ez;
                }
            }
        }
#pragma unroll
        for (int r = 0; r < ROWS; ++r) {
            hk[r][0] = h[r][0];
            hk[r][1] = h[r][1];
#pragma unroll
            for (int q = 0; q < 3; ++q) e0[r][q] = e1[r][q];
        }
    }
#pragma unroll 1
    for (int r = 0; r < ROWS; ++r) {
        if (a.ndft) dft_fold<false>(a, a.enew, i, j + r, k0, k1); /* the new E */
        if (a.probe_rows) probe_fold<false>(a, a.enew, a.hnew, i, j + r, k0, k1);
    }
}

/* The interior of a domain in one launch: blocks of one plain or tensor
 * material (kEOnly), no CPML cell in the tile or one below it, no domain
 * edge, no source.  The same march as he_sweep_tma with nothing but the
 * stencil: two words of curl state per cell in registers, no spills.  The
 * other blocks of the domain take the two sweeps (their CPML, pool and
 * source handling need the registers this march does not), the H sweep
 * beside this kernel and the E sweep after both: on a 1024 x 512 x 64 vacuum
 * grid the whole step in he_sweep_tma took 0.83 ms in FP64 (64 registers,
 * spills), the two sweeps 0.78 ms.
 * Bound by HBM: reads E, H and writes E, H once, 12 words per cell, plus
 * about 2 planes of a block's range. */
template <typename R>
__global__ void __launch_bounds__(kBlockX * kBlockY, (sizeof(R) == 8 ? PHP_INNER_MINB64 : PHP_INNER_MINB32))
    interior_sweep_tma(const __grid_constant__ StepArgs<R> a, const __grid_constant__ TmaMaps tm)
{
    using G = FusedGeom<R, true>;
    constexpr int SE = G::SE, SH = G::SH, ROWS = G::ROWS;
    constexpr int EBW = G::EBW, HBW = G::HBW, ES = G::EB / (int)sizeof(R), HS = G::HB / (int)sizeof(R);
    extern __shared__ __align__(128) unsigned char dyn_smem[];
    unsigned char* smem = ring_base(dyn_smem);
    R* const ering = reinterpret_cast<R*>(smem);              /* [SE] stages of [3][EBW] */
    R* const hring = reinterpret_cast<R*>(smem + SE * G::EB); /* [SH] stages of [3][HBW] */
    uint64_t* const ebar = reinterpret_cast<uint64_t*>(smem + SE * G::EB + SH * G::HB);
    uint64_t* const hbar = ebar + SE;

    const int tx = threadIdx.x, ty = threadIdx.y, tid = ty * G::TX + tx;
    const int4 job = a.list[blockIdx.x];
    const int i0 = (job.x & 0xffff) * G::TX, j0 = (job.x >> 16) * G::TY;
    const int i = i0 + tx, j = j0 + ty * ROWS; /* the thread's first row */
    const int k0 = job.y, k1 = job.z, cls = job.w;
    const int nE = k1 - k0 + 2, nH = k1 - k0 + 1; /* planes k0-1 .. k1 of E, k0-1 .. k1-1 of H */

    /* plane k0 - 1 + g into stage s of its ring */
    auto issue_e = [&](int g, int s) {
        R* b = ering + s * ES;
        mbar_arrive_expect_tx(&ebar[s], G::E3_BYTES);
        tma_load_plane(b, &tm.e_wide, &ebar[s], i0 - G::HALO, j0 - 1, k0 + g);
    };
    auto issue_h = [&](int g, int s) {
        R* b = hring + s * HS;
        mbar_arrive_expect_tx(&hbar[s], G::H3_BYTES);
        tma_load_plane(b, &tm.h_wide, &hbar[s], i0 - G::HALO, j0 - 1, k0 + g);
    };

    if (tid == 0) {
        for (int s = 0; s < SE + SH; ++s) mbar_init(&ebar[s], 1);
        fence_barrier_init();
    }
    chain_enter(a.beside);
    __syncthreads();
    if (tid == 0) {
        for (int g = 0; g < max(SE, SH); ++g) {
            if (g < SE && g < nE) issue_e(g, g);
            if (g < SH && g < nH) issue_h(g, g);
        }
    }

    /* the cell below the tile this thread computes H of as well (tid < NHALO):
     * the row j0 - 1 from i0 - 1, then the column i0 - 1 (the tile has no
     * domain edge cell, so both are in the grid) */
    const int cx_ = tid <= G::TX ? tid - 1 : -1, cy_ = tid <= G::TX ? -1 : tid - G::TX - 1;
    const bool halo = tid < G::NHALO;
    /* offsets of the own cell (row 0) in the boxes, of the cell below the tile */
    const int eo = (ty * ROWS + 1) * G::EX + tx + G::HALO;
    const int ho = (ty * ROWS + 1) * G::HX + tx + G::HALO;
    const int ce = (cy_ + 1) * G::EX + (cx_ + G::HALO);
    const int ch = (cy_ + 1) * G::HX + (cx_ + G::HALO);
    const R khx = a.khp[0], khy = a.khp[1], khz = a.khp[2];
    const R kdx = a.kdp[0], kdy = a.kdp[1], kdz = a.kdp[2];
    const bool tensor = cls == kPlainTensor;
    const bool lossy = tensor && (a.tns_flags & kLossy);
    const R iso = tensor ? R(0) : a.iso[cls];
    const R z0 = R(0);

    R e0[ROWS][3];   /* E of the own cells at plane p */
    R hk[ROWS][2];   /* new Hx, Hy of the own cells at plane p - 1 */
    int se = 0, sh = 0;             /* stages of E plane p and H plane p */
    uint32_t pe = 0, ph = 0;        /* phases of E plane p + 1's stage and of H plane p's */
    int c0 = ((k0 - 1) * a.ny + j) * a.nxp + i;
    bool ok = mbar_wait(&ebar[0], 0);
#pragma unroll
    for (int r = 0; r < ROWS; ++r) {
#pragma unroll
        for (int q = 0; q < 3; ++q) e0[r][q] = ok ? ering[q * EBW + eo + r * G::EX] : z0;
        hk[r][0] = hk[r][1] = z0;
    }

    for (int g = 0; g < nH; ++g) {
        const int se1 = se + 1 == SE ? 0 : se + 1;
        const uint32_t pe1 = se1 == 0 ? pe ^ 1u : pe;
        const R* const Eb0 = ering + se * ES;
        const R* const Eb1 = ering + se1 * ES;
        R* const Hb = hring + sh * HS;
        ok = ok && mbar_wait(&hbar[sh], ph);
        ok = ok && mbar_wait(&ebar[se1], pe1);

        /* ---- H of plane p = k0 - 1 + g: the own cells, and the cell below
         * the tile (plane -1 is the zero halo plane) */
        R h[ROWS][3], e1[ROWS][3];
        const bool upd = k0 + g > 0;
        if (ok) {
#pragma unroll
            for (int r = 0; r < ROWS; ++r)
#pragma unroll
                for (int q = 0; q < 3; ++q) {
                    e1[r][q] = Eb1[q * EBW + eo + r * G::EX];
                    h[r][q] = Hb[q * HBW + ho + r * G::HX];
                }
            if (upd) {
#pragma unroll
                for (int r = 0; r < ROWS; ++r) {
                    const int er = eo + r * G::EX;
                    const R dEzx = Eb0[2 * EBW + er + 1] - e0[r][2], dEyx = Eb0[EBW + er + 1] - e0[r][1];
                    const R dEzy = (r + 1 < ROWS ? e0[r + 1 < ROWS ? r + 1 : r][2] : Eb0[2 * EBW + er + G::EX]) - e0[r][2];
                    const R dExy = (r + 1 < ROWS ? e0[r + 1 < ROWS ? r + 1 : r][0] : Eb0[er + G::EX]) - e0[r][0];
                    h_update(khx, khy, khz, e1[r][1] - e0[r][1], dEzy, dEzx, e1[r][0] - e0[r][0], dExy, dEyx, z0, z0, z0, z0, z0,
                             z0, h[r][0], h[r][1], h[r][2]);
                }
            }
            if (g > 0) {
#pragma unroll
                for (int r = 0; r < ROWS; ++r)
#pragma unroll
                    for (int q = 0; q < 3; ++q) Hb[q * HBW + ho + r * G::HX] = h[r][q];
                if (halo) {
                    R qx = Hb[ch], qy = Hb[HBW + ch], qz = Hb[2 * HBW + ch];
                    const R cx = Eb0[ce], cy = Eb0[EBW + ce], cz = Eb0[2 * EBW + ce];
                    h_update(khx, khy, khz, Eb1[EBW + ce] - cy, Eb0[2 * EBW + ce + G::EX] - cz, Eb0[2 * EBW + ce + 1] - cz,
                             Eb1[ce] - cx, Eb0[ce + G::EX] - cx, Eb0[EBW + ce + 1] - cy, z0, z0, z0, z0, z0, z0, qx, qy, qz);
                    Hb[ch] = qx;
                    Hb[HBW + ch] = qy;
                    Hb[2 * HBW + ch] = qz;
                }
            }
        }
        /* the new H of plane p is in its stage; every thread is done with the
         * E stage of plane p and with H plane p - 1 (whose stage this block
         * wrote: ordered before the loads that overwrite it) */
        fence_proxy_async_smem();
        if (__syncthreads_or(!ok)) {
            if (tid == 0) {
                atomicExch(a.err, 1);
                ring_drain(ebar, SE, (uint32_t)min(nE, SE + g));
                ring_drain(hbar, SH, (uint32_t)min(nH, SH + max(0, g - 1)));
            }
            break;
        }
        if (tid == 0) {
            fence_proxy_async_smem();
            if (g + SE < nE) issue_e(g + SE, se);
            if (g >= 1 && g - 1 + SH < nH) issue_h(g - 1 + SH, sh == 0 ? SH - 1 : sh - 1);
        }

        /* ---- E of plane p */
        if (g > 0) {
#pragma unroll
            for (int r = 0; r < ROWS; ++r) {
                const int hr = ho + r * G::HX, c = c0 + r * a.nxp;
                const R hx = h[r][0], hy = h[r][1], hz = h[r][2];
                const R hz_jm = r > 0 ? h[r > 0 ? r - 1 : 0][2] : Hb[2 * HBW + hr - G::HX];
                const R hx_jm = r > 0 ? h[r > 0 ? r - 1 : 0][0] : Hb[hr - G::HX];
                const R hz_im = Hb[2 * HBW + hr - 1], hy_im = Hb[HBW + hr - 1];
                R ex = e0[r][0], ey = e0[r][1], ez = e0[r][2];
                R ux = curl2(kdy, hz - hz_jm, kdz, hy - hk[r][1]);
                R uy = curl2(kdz, hx - hk[r][0], kdx, hz - hz_im);
                R uz = curl2(kdx, hy - hy_im, kdy, hx - hx_jm);
                if (tensor) {
                    if (lossy) loss_sub(a.tns_im, ex, ey, ez, ux, uy, uz);
                    e_only_add(a.tns_em, ux, uy, uz, ex, ey, ez);
                } else {
                    iso_add(iso, ux, uy, uz, ex, ey, ez);
                }
                a.hnew[0][c] = hx;
                a.hnew[1][c] = hy;
                a.hnew[2][c] = hz;
                a.enew[0][c] = ex;
                a.enew[1][c] = ey;
                a.enew[2][c] = ez;
            }
        }
#pragma unroll
        for (int r = 0; r < ROWS; ++r) {
            hk[r][0] = h[r][0];
            hk[r][1] = h[r][1];
#pragma unroll
            for (int q = 0; q < 3; ++q) e0[r][q] = e1[r][q];
        }
        se = se1;
        pe = pe1;
        if (++sh == SH) {
            sh = 0;
            ph ^= 1u;
        }
        c0 += (int)a.plane;
    }
#pragma unroll 1
    for (int r = 0; r < ROWS; ++r) {
        if (a.ndft) dft_fold<false>(a, a.enew, i, j + r, k0, k1); /* the new E */
        if (a.probe_rows) probe_fold<false>(a, a.enew, a.hnew, i, j + r, k0, k1);
    }
    chain_leave(a.beside, tid);
}

} // namespace phpdev

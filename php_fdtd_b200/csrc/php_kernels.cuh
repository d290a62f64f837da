/*
 * php_kernels.cuh -- device types and the small kernels of the PhP_FDTD
 * time step on sm_100a (the sweeps are in php_sweeps*.cuh and
 * php_sweep_fused.cuh, the ion pass in php_ions.cuh).
 *
 * Device layout (one domain per GPU):
 *   field arrays  R[(nz + 2) planes][ny][nxp]   x fastest, nxp = nx rounded up
 *                 to 32 elements; plane -1 and plane nz are zero halos that
 *                 are never written, so the z stencils need no branch
 *                 (the reference's k = -1 / k = local_nz halo, fdtd.c:2006-2056,
 *                 holds zeros on a single rank).
 *   mat           uint8 [nz][ny][nxp] material id
 *   slot          int32 [nz][ny][nxp] index into the ADE / ion pools, -1 else
 *   psi x-slab    [nz][ny][2L]   (low side s = i, high side s = L + nx-1-i)
 *   psi y-slab    [nz][2L][nxp]
 *   psi z-slab    [2L][ny][nxp]
 *   pools         SoA: P[3][nslot], Po[3][nslot], r[3*natom_max][nslot], v[...]
 *   D             strict mode: field arrays like E and H.  Fast modes: only
 *                 where E is not a fixed linear map of D (ADE and atom
 *                 cells) or the map would lose digits: Dp[3][nslot] beside
 *                 the other state of those cells.  Every other cell keeps E
 *                 alone and advances it by M (D^{n+1} - D^n), M the material's
 *                 3 x 3 map from D to E (e_only_add): the two sweeps move 18
 *                 field words per cell instead of 21 (E is read in place of
 *                 D and D not written; 24 where a lossy cell read both).
 *                 Read-outs of D form M^-1 E (d_at).
 *
 * Arithmetic modes:
 *   Strict (double): every operation of the reference in its order, with
 *     IEEE division and no contraction (__dadd_rn & co. are never fused),
 *     on coefficient tables derived on the host exactly as fdtd.c derives
 *     them per cell.  Reproduces the reference bit for bit.
 *   Fast (double or float): the same update with host-folded coefficients
 *     (reciprocal spacings, psi stored pre-multiplied by dt, eps^-1 folded
 *     with the loss factors) and FMA.
 */
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

namespace phpdev {

constexpr int kMaxSources = 16;
constexpr int kBlockX = 32;
constexpr int kBlockY = 8;

/* ----------------------------------------------------------------- tables */

/* Per material coefficients.  Strict and fast variants share the layout;
 * fields not used by a mode are zero. */
template <typename R>
struct MatCoef {
    int32_t flags;     /* kLossy | kAde | kRotZ | kRotX | kAtoms | kIso | kEOnly */
    int32_t natom;
    int32_t ion_off;   /* offset of QeZV (9N), QeZM (9N), DMM (9N^2) in ion_coef */
    int32_t pad;
    R eps_inv[9];      /* strict: Re eps^-1; fast: (1-lt)*lf/eps0 * Re eps^-1 */
    R eps_im[9];       /* strict: eps''; fast: c1*eps0*eps'' */
    R lf, lt;          /* loss factor and loss term (strict) */
    R cs, sn;          /* rotation cosine / sine */
    R gp_inv[9];       /* ADE (I + gamma dt/2)^-1 */
    R gm[9];           /* ADE (I - gamma dt/2) */
    R wp2[9];          /* strict: wp2; fast: eps0 dt^2 wp2 */
    R ade_scale;       /* fast: (1-lt)/(eps0*EPS_INF) */
    R pad2;
    R em[9];           /* fast: E = em D in the lab frame (rotations folded in) */
};

/* kIso (fast modes only): no rotation, loss, ADE or atoms and eps^-1 a
 * multiple of the identity, so E = eps_inv[0] * D.
 * kEOnly (fast modes only): no ADE or atoms, and em is well conditioned, so
 * the cell keeps E alone (kIso implies it); the other cells have a pool slot. */
enum : int32_t { kLossy = 1, kAde = 2, kRotZ = 4, kRotX = 8, kAtoms = 16, kIso = 32, kEOnly = 64 };

/* Per-axis CPML tables, indexed by the cell index along the axis.  slot < 0
 * outside the PML (pml_slot).  Strict uses kappa, b, c (fdtd.c:3146-3151 evaluated on
 * the host); fast uses kh = dt/(mu0 d kappa), kd = dt/(d kappa),
 * ch = dt c/(mu0 d), cd = dt c/d. */
template <typename R>
struct AxisTab {
    const R* kappa;
    const R* b;
    const R* c;
    const R* kh;
    const R* kd;
    const R* ch;
    const R* cd;
};

template <typename R>
struct Fields {
    R *ex, *ey, *ez, *dx, *dy, *dz, *hx, *hy, *hz;
};

/* Where D is in the fast modes (Fields::dx is null): the pool of the cells
 * with a slot, M^-1 E (dm, 9 doubles per material) in the others. */
template <typename R>
struct DView {
    const R* dp;
    const uint8_t* mat;
    const int32_t* slot;       /* null: no cell has one */
    const double* dm;
    int64_t nslot, ncell;
};

template <typename R>
struct Psi {
    R *hxy, *hxz, *hyx, *hyz, *hzx, *hzy;
    R *dxy, *dxz, *dyx, *dyz, *dzx, *dzy;
};

/* The fused sweep's copy of one few-atom material's ion coefficients in the
 * kernel parameters (constant bank): QeZV [9 N], QeZM [9 N] and DMM with row
 * stride kIonKQ, for N <= 4 */
constexpr int kIonKQ = 12;
constexpr int kIonKM = 36;
constexpr int kIonKD = 72;
constexpr int kIonK = kIonKD + kIonKQ * kIonKQ;
constexpr int kIsoMats = 32;
/* running DFT planes the E sweep can sample itself (StepArgs::dft_*) */
constexpr int kDftFold = 4;
/* plain-block codes of the fused sweep: id, or kPlainCpml + id for blocks of
 * one plain material with CPML or domain-edge cells, kPlainTensor for blocks
 * of the tensor material in StepArgs::tns_*, kPlainAtoms for blocks of the
 * few-atom material in StepArgs::amc; 255 = general path */
constexpr int kPlainCpml = 64;
constexpr int kPlainTensor = 128;
constexpr int kPlainAtoms = 129;

template <typename R>
struct StepArgs {
    Fields<R> f;
    Psi<R> psi;
    AxisTab<R> tx, ty, tz;
    const uint8_t* mat;
    const int32_t* slot;
    const MatCoef<R>* mc;
    const R* ion_coef;
    R *P, *Po, *r, *v;         /* pools */
    R* Dp;                     /* D of the cells with a slot [3][nslot] (fast modes) */
    uint32_t* Dc;              /* FP32 with atoms: what Dp's sums rounded off (pool_add) [nslot], else null */
    DView<R> dv;
    const R* pr;               /* QeZV . r [3][nslot] when the ion pass runs apart (php_ions.cuh), else null */
    int32_t ion_k_off;         /* ion_coef offset of the material copied in ion_k, -1 for none */
    R ion_k[kIonK];
    /* dE = iso[id] * dD for the plain isotropic materials (kIso) among the
     * first kIsoMats ids, 0 for the others: the fused sweep's common case
     * without a load of the material record */
    R iso[kIsoMats];
    /* per block of the fused sweep: the material id of a plain block (one
     * plain isotropic material, no CPML or domain-edge cell, no source), 255
     * for the others; nullptr = no plain blocks.  kdp: dt / d of the axes
     * outside the CPML (kappa = 1) */
    const uint8_t* plain_blk;
    R kdp[3];
    /* per block of the H sweep: 1 for a tile and z chunk with no CPML cell
     * and every cell updated (i < nx-1, j < ny-1); kh of kappa = 1 */
    const uint8_t* plain_h;
    R khp[3];
    /* the material record of one lossy or anisotropic material without ADE
     * or ions (the one filling most blocks): blocks of that material alone
     * (kPlainTensor) read it as constant-bank operands */
    R tns_em[9], tns_im[9];
    int32_t tns_flags;
    /* the material record of the few-atom material whose ion coefficients
     * are in ion_k (or of the lattice of the ion pass, or, in a domain without
     * atoms, of a material that keeps D), for blocks of that material alone
     * (kPlainAtoms) */
    MatCoef<R> amc;
    /* the record of the material with pool cells but no atoms (ADE, or D kept
     * beside E) that fills the most cells, -1 for none: the general path reads
     * some 30 of its values per cell as constant-bank operands instead of loads */
    MatCoef<R> dmc;
    int32_t dmc_id;
    int64_t nslot;
    int32_t nx, ny, nz, nxp, L, zchunk;
    int32_t z_off, nzg;        /* global index of plane 0 and plane count (z slabs) */
    int32_t zc0;                /* first z chunk of the launch (blockIdx.z + zc0 is the chunk) */
    int64_t plane;             /* nxp * ny */
    /* strict scalars */
    double dt, dxs, dys, dzs, mu0, eps0, c1, e0dt2;
    /* sources of this step */
    int32_t nsrc;
    int64_t src_cell[kMaxSources];
    int32_t src_comp[kMaxSources];
    const double* src_val;     /* nsrc values of this step */
    /* FP32: E of the source cells that keep E alone, summed in double [nsrc][3].
     * A point source's own cell holds some 1e4 times the field of the
     * radiation zone, so the rounding of its sum is the largest error there. */
    double* src_acc;
    /* programmatic launch chain: 1 when the launch before this one is one it
     * does not depend on (it waits for it at its end; see chain_enter) */
    int32_t beside;
    int32_t* err;              /* set to 1 by a block whose bounded wait gave up */
    int32_t stall_test;        /* failure-path test: the first H sweep block's wait gives up */
    /* where the sweeps write the new E, H and H CPML state.  The two sweeps of
     * a domain in place: the arrays of f and psi.  Double buffered (the
     * one-launch step, and the interior / rest split): f's E and H hold the
     * old time level, read only during the step (the one-launch step's H CPML
     * state likewise).  The D CPML state and the pools are updated in place. */
    R *enew[3], *hnew[3];
    R* psin_h[6];              /* hxy hxz hyx hyz hzx hzy */
    /* blocks of a launch over part of the domain (blockIdx.x indexes it):
     * x = tile x | tile y << 16, y .. z the planes [k0, k1), w the class (H
     * sweep: 1 for a plain block; fused sweep: its plain-block code);
     * nullptr: the whole grid in z chunks */
    const int4* list;
    /* he_sweep_tma: planes per block, and per plane and tile (of its own
     * height) the class of the fused sweep's plain blocks, plus kHPlain
     * [nz][tiles y][tiles x] */
    int32_t zstep;
    const uint16_t* pcls;
    /* running DFT planes of E or D components that the E sweep samples
     * after its z march (dft_fold), instead of a dft_sample launch: plane,
     * component (0-5), frequencies, the float32 cast flag, the offset of the
     * plane's flag and phasors in the step's input row (src_val), and the
     * accumulators [nfreq][ny][nx][2] */
    int32_t ndft;
    int32_t dft_z[kDftFold], dft_comp[kDftFold], dft_nfreq[kDftFold], dft_cast[kDftFold], dft_off[kDftFold];
    double* dft_acc[kDftFold];
    /* the monitor row the sweeps record after their z march (probe_fold),
     * instead of a probe_record_counted launch: its index is the value at
     * probe_off of the step's input row (src_val), the fields are those of
     * (i, j, kf), r and v those of slot, the cell (i, j, ka); probe_rows null:
     * no such row */
    double* probe_rows;
    int32_t* probe_count;      /* [rows written, overflow flag] */
    int32_t probe_i, probe_j, probe_kf, probe_ka, probe_n3, probe_cap, probe_off;
    int64_t probe_slot;
    double rv_unit;            /* physical r, v per stored unit */
};

/* ------------------------------------------------------------ arithmetic */

/* The fast modes' updates are written with explicit fused multiply-adds, so
 * that every kernel and block path that contains them rounds alike (slabs,
 * the one-launch step and the two sweeps give the same fields, bit for bit). */
__device__ __forceinline__ double fma_(double a, double b, double c) { return __fma_rn(a, b, c); }
__device__ __forceinline__ float fma_(float a, float b, float c) { return __fmaf_rn(a, b, c); }
/* ka a - kb b: one component of a scaled curl */
template <typename R>
__device__ __forceinline__ R curl2(R ka, R a, R kb, R b) { return fma_(ka, a, -(kb * b)); }

struct SOp {
    static __device__ __forceinline__ double add(double a, double b) { return __dadd_rn(a, b); }
    static __device__ __forceinline__ double sub(double a, double b) { return __dsub_rn(a, b); }
    static __device__ __forceinline__ double mul(double a, double b) { return __dmul_rn(a, b); }
    static __device__ __forceinline__ double div(double a, double b) { return __ddiv_rn(a, b); }
};

template <typename T>
__device__ __forceinline__ T ldg(const T* p) { return __ldg(p); }

/* Read-only loads the compiler may not hoist out of the z loop: PML and
 * material coefficients are only needed inside rare branches, and keeping
 * them live across the loop would cost the registers that hold the next
 * plane in flight. */
__device__ __forceinline__ double ldg_nh(const double* p)
{
    double v;
    asm volatile("ld.global.nc.f64 %0, [%1];" : "=d"(v) : "l"(p));
    return v;
}
__device__ __forceinline__ float ldg_nh(const float* p)
{
    float v;
    asm volatile("ld.global.nc.f32 %0, [%1];" : "=f"(v) : "l"(p));
    return v;
}

/* The launches of recorded steps form a chain of programmatic launches: a
 * launch may start once every block of the one before it has passed
 * chain_enter, so its blocks fill the SMs that the last blocks of that one
 * leave idle, and its set-up runs meanwhile.  A launch that depends on the one
 * before waits in chain_enter for its completion, and only then lets the next
 * one start.  One that does not (StepArgs::beside: its inputs come from
 * launches further back, complete since the launch before it entered) waits at
 * its end instead, in chain_leave, so that its own completion still implies
 * that of all before it.  Only a grid that waited is promised a view of what
 * earlier ones wrote, its L1 included.  What one beside another reads is in L2
 * before it starts (the launch before it entered after a wait for its writers,
 * and started it after that), but a line of an earlier step may still be in an
 * L1: the kernels that run so read what earlier launches wrote through L2
 * (ld_state, prefetch_state, TMA); with these reads through L1 an interval of
 * 256^3 took 23.2 ms FP64 and 14.7 ms FP32, through L2 23.3 and 15.0.  Launched
 * without the attribute, both return at once.  Per step, plain launches and the chain: 32^3 7.6 -> 6.4 us, 96^3
 * two-atom slab FP64 55 -> 50 us, FP32 34.4 -> 34.0 us; 256^3 unchanged. */
__device__ __forceinline__ void chain_enter(int beside)
{
    if (!beside) asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}
__device__ __forceinline__ void chain_leave(int beside, int tid)
{
    if (beside && blockIdx.x == 0 && blockIdx.y == 0 && blockIdx.z == 0 && tid == 0) asm volatile("griddepcontrol.wait;" ::: "memory");
}

/* State that an earlier launch wrote and this one does not before the read;
 * CG: through L2, past the L1 (see chain_enter). */
template <bool CG>
__device__ __forceinline__ double ld_state(const double* p)
{
    if constexpr (!CG) return *p;
    double v;
    asm volatile("ld.global.cg.f64 %0, [%1];" : "=d"(v) : "l"(p));
    return v;
}
template <bool CG>
__device__ __forceinline__ float ld_state(const float* p)
{
    if constexpr (!CG) return *p;
    float v;
    asm volatile("ld.global.cg.f32 %0, [%1];" : "=f"(v) : "l"(p));
    return v;
}
template <bool CG>
__device__ __forceinline__ uint32_t ld_state(const uint32_t* p)
{
    if constexpr (!CG) return *p;
    uint32_t v;
    asm volatile("ld.global.cg.u32 %0, [%1];" : "=r"(v) : "l"(p));
    return v;
}
/* its line, requested ahead of the read */
template <bool CG>
__device__ __forceinline__ void prefetch_state(const void* p)
{
    if constexpr (CG) asm volatile("prefetch.global.L2 [%0];" ::"l"(p));
    else asm volatile("prefetch.global.L1 [%0];" ::"l"(p));
}

/* CPML slot of cell i of an axis of n cells: i at the low side, L + n - 1 - i
 * at the high one, -1 between */
__host__ __device__ __forceinline__ int pml_slot(int i, int n, int L)
{
    return i < L ? i : i >= n - L ? L + n - 1 - i : -1;
}

/* ========================================================== small kernels */

/* one row of M^-1 E, rounded as a stored D would be; a component that does not
 * enter stays out even where it overflowed */
template <typename R>
__device__ __forceinline__ double d_of_e(const double* m, R ex, R ey, R ez)
{
    const double x = m[0] != 0.0 ? (double)ex : 0.0, y = m[1] != 0.0 ? (double)ey : 0.0, z = m[2] != 0.0 ? (double)ez : 0.0;
    return (double)(R)__fma_rn(m[0], x, __fma_rn(m[1], y, m[2] * z));
}

/* D component q of device cell c, halo planes included (zero) */
template <typename R>
__device__ __forceinline__ double d_at(const Fields<R>& f, const DView<R>& v, int q, int64_t c)
{
    if (f.dx) return (double)(q == 0 ? f.dx : q == 1 ? f.dy : f.dz)[c];
    if (c < 0 || c >= v.ncell) return 0.0;
    const int32_t s = v.slot ? v.slot[c] : -1;
    if (s >= 0) return (double)v.dp[(int64_t)q * v.nslot + s];
    return d_of_e<R>(v.dm + 9 * (int)v.mat[c] + 3 * q, f.ex[c], f.ey[c], f.ez[c]);
}

/* field component comp (0-8) of device cell c */
template <typename R>
__device__ __forceinline__ double field_at(const Fields<R>& f, const DView<R>& v, int comp, int64_t c)
{
    switch (comp) {
    case 0: return (double)f.ex[c];
    case 1: return (double)f.ey[c];
    case 2: return (double)f.ez[c];
    case 6: return (double)f.hx[c];
    case 7: return (double)f.hy[c];
    case 8: return (double)f.hz[c];
    default: return d_at(f, v, comp - 3, c);
    }
}

/* Gathers one plane of a component into out (float or double).
 * axis 0: z plane kk -> [i][j]; axis 1: x plane -> [j][k]; axis 2: y plane
 * -> [i][k].  comp 9 is |E|. */
template <typename R, typename O>
__global__ void gather_plane(const Fields<R> f, const DView<R> dv, int comp, int axis, int pos, int nx, int ny, int nz,
                             int nxp, O* out)
{
    int A, B;
    if (axis == 0) { A = nx; B = ny; }
    else if (axis == 1) { A = ny; B = nz; }
    else { A = nx; B = nz; }
    const int64_t n = (int64_t)A * B;
    for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < n; t += (int64_t)gridDim.x * blockDim.x) {
        const int u = (int)(t / B), w = (int)(t % B);
        int i, j, k;
        if (axis == 0) { i = u; j = w; k = pos; }
        else if (axis == 1) { i = pos; j = u; k = w; }
        else { i = u; j = pos; k = w; }
        const int64_t c = ((int64_t)k * ny + j) * nxp + i;
        double val;
        if (comp < 9) {
            val = field_at(f, dv, comp, c);
        } else {
            const double x = (double)f.ex[c], y = (double)f.ey[c], z = (double)f.ez[c];
            val = __dsqrt_rn(__dadd_rn(__dadd_rn(__dmul_rn(x, x), __dmul_rn(y, y)), __dmul_rn(z, z)));
        }
        out[t] = (O)val;
    }
}

/* The nine field values of one cell. */
template <typename R>
__global__ void point_gather(const Fields<R> f, const DView<R> dv, int64_t c, double* out9)
{
    if (threadIdx.x < 9) out9[threadIdx.x] = field_at(f, dv, threadIdx.x, c);
}

/* Whole component to file order [i][j][k]. */
template <typename R>
__global__ void gather_volume(const Fields<R> f, const DView<R> dv, int comp, int nx, int ny, int nz, int nxp, double* out)
{
    const int64_t n = (int64_t)nx * ny * nz;
    for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < n; t += (int64_t)gridDim.x * blockDim.x) {
        const int k = (int)(t % nz);
        const int64_t ij = t / nz;
        const int j = (int)(ij % ny), i = (int)(ij / ny);
        out[t] = field_at(f, dv, comp, ((int64_t)k * ny + j) * nxp + i);
    }
}

/* Where D of one cell is: its pool slot, else M^-1 (fast modes) */
struct DCell {
    int32_t slot;
    double dm[9];
};

/* Probe row appended at count[0]: 9 fields at cf, then r and v of pool slot
 * (3*natom each, times rv_unit: the stored state is scaled in FP32).
 * count[1] is raised instead of writing past cap. */
template <typename R>
__global__ void probe_record_counted(const Fields<R> f, const R* dp, const DCell dc, int64_t cf, const R* r, const R* v, double rv_unit,
                                     int64_t nslot, int64_t slot, int n3, double* rows, int32_t* count, int cap,
                                     int row_len)
{
    __shared__ int row;
    if (threadIdx.x == 0) row = count[0];
    __syncthreads();
    if (row >= cap) {
        if (threadIdx.x == 0) count[1] = 1;
        return;
    }
    double* out = rows + (int64_t)row * row_len;
    const int t = threadIdx.x;
    if (t < 9) {
        if (t < 3 || t > 5) {
            out[t] = (double)(t == 0 ? f.ex : t == 1 ? f.ey : t == 2 ? f.ez : t == 6 ? f.hx : t == 7 ? f.hy : f.hz)[cf];
        } else if (f.dx) {
            out[t] = (double)(t == 3 ? f.dx : t == 4 ? f.dy : f.dz)[cf];
        } else {
            const double* m = dc.dm + 3 * (t - 3);
            out[t] = dc.slot >= 0 ? (double)dp[(int64_t)(t - 3) * nslot + dc.slot] : d_of_e<R>(m, f.ex[cf], f.ey[cf], f.ez[cf]);
        }
    } else if (t < 9 + 2 * n3) {
        const int q = t - 9;
        out[t] = rv_unit * ((q < n3) ? (double)r[(int64_t)q * nslot + slot] : (double)v[(int64_t)(q - n3) * nslot + slot]);
    }
    __syncthreads();
    if (threadIdx.x == 0) count[0] = row + 1;
}

/* One cell's running-DFT samples: acc[f][t] += x * (cos, sin) for the
 * phasors of this step (ph[2f], ph[2f+1]), t = j * nx + i of n = nx * ny
 * (x fastest, so that a warp's cells along x update adjacent accumulators;
 * php_dft_read hands them out in [f][i][j] order). */
template <bool CG>
__device__ __forceinline__ void dft_accumulate(double x, const double* ph, int nfreq, double* acc, int64_t n, int64_t t)
{
    for (int f = 0; f < nfreq; ++f) {
        double* a = acc + ((int64_t)f * n + t) * 2;
        const double re = ld_state<CG>(a), im = ld_state<CG>(a + 1);
        a[0] = re + x * ld_state<CG>(ph + 2 * f);
        a[1] = im + x * ld_state<CG>(ph + 2 * f + 1);
    }
}

/* Running DFT sample of one plane; skipped when flag == 0. */
template <typename R>
__global__ void dft_sample(const Fields<R> fld, const DView<R> dv, int comp, int64_t plane_off, int nx, int ny, int nxp, int nfreq,
                           int cast_f32, const double* step_in, int flag_off, int phasor_off,
                           double* acc)
{
    if (step_in[flag_off] == 0.0) return;
    const int64_t n = (int64_t)nx * ny;
    const double* ph = step_in + phasor_off;
    for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < n; t += (int64_t)gridDim.x * blockDim.x) {
        const int j = (int)(t / nx), i = (int)(t % nx);
        double x = field_at(fld, dv, comp, plane_off + (int64_t)j * nxp + i);
        if (cast_f32) x = (double)(float)x;
        dft_accumulate<false>(x, ph, nfreq, acc, n, t);
    }
}

/* Accumulators [nfreq][ny][nx] to elements o0 .. o0+n-1 of the caller's order
 * [nfreq][nx][ny].  A plane's accumulators fit the L2, so the strided 16-byte
 * reads cost no more than a tiled transpose would; the copy out bounds it. */
__global__ void __launch_bounds__(256) dft_reorder(const double2* acc, int nx, int ny, int64_t o0, int64_t n, double2* out)
{
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < n; t += stride) {
        const int64_t fi = (o0 + t) / ny, f = fi / nx;
        const int j = (int)(o0 + t - fi * ny), i = (int)(fi - f * nx);
        out[t] = acc[(f * ny + j) * nx + i];
    }
}

/* The same samples taken by the E sweep (StepArgs::dft_*): after a block's z
 * march over planes k0 .. k1-1, each of its threads reads back the E or D
 * values it stored at cell (i, j) of every registered plane in that range
 * that this step samples (e3: the E arrays the sweep wrote).  A cell's
 * accumulators belong to the one thread that updates the cell; no register
 * is held for this inside the march. */
template <bool CG, typename R>
__device__ __forceinline__ void dft_fold(const StepArgs<R>& a, R* const* e3, int i, int j, int k0, int k1)
{
    if (i >= a.nx || j >= a.ny) return;
    for (int q = 0; q < a.ndft; ++q) {
        const int k = a.dft_z[q];
        if (k < k0 || k >= k1 || ld_state<CG>(a.src_val + a.dft_off[q]) == 0.0) continue;
        const int cp = a.dft_comp[q];
        const int c = (k * a.ny + j) * a.nxp + i;
        double x;
        if (cp < 3) {
            x = (double)(cp == 0 ? e3[0] : cp == 1 ? e3[1] : e3[2])[c];
        } else {
            Fields<R> f = a.f;
            f.ex = e3[0];
            f.ey = e3[1];
            f.ez = e3[2];
            x = d_at(f, a.dv, cp - 3, c);
        }
        if (a.dft_cast[q]) x = (double)(float)x;
        dft_accumulate<CG>(x, a.src_val + a.dft_off[q] + 1, a.dft_nfreq[q], a.dft_acc[q], (int64_t)a.nx * a.ny,
                       (int64_t)j * a.nx + i);
    }
}

/* The monitor row of probe_record_counted taken by the sweeps
 * (StepArgs::probe_*): after its z march over planes k0 .. k1-1, the thread of
 * column (i, j) reads back the E, D and H of the field cell (e3, h3: the arrays
 * the step's launches wrote), and the one whose planes hold the atom cell its r
 * and v. */
template <bool CG, typename R>
__device__ __forceinline__ void probe_fold(const StepArgs<R>& a, R* const* e3, R* const* h3, int i, int j, int k0, int k1)
{
    if (i != a.probe_i || j != a.probe_j) return;
    const bool fields = a.probe_kf >= k0 && a.probe_kf < k1, atoms = a.probe_n3 && a.probe_ka >= k0 && a.probe_ka < k1;
    if (!fields && !atoms) return;
    const int row = (int)ld_state<CG>(a.src_val + a.probe_off);
    if (row >= a.probe_cap) {
        if (fields) a.probe_count[1] = 1;
        return;
    }
    double* out = a.probe_rows + (int64_t)row * (9 + 2 * a.probe_n3);
    if (fields) {
        const int64_t c = ((int64_t)a.probe_kf * a.ny + j) * a.nxp + i;
        Fields<R> f = a.f;
        f.ex = e3[0];
        f.ey = e3[1];
        f.ez = e3[2];
        for (int q = 0; q < 6; ++q) out[q] = field_at(f, a.dv, q, c);
        for (int q = 0; q < 3; ++q) out[6 + q] = (double)ld_state<CG>(h3[q] + c);
        a.probe_count[0] = row + 1;
    }
    for (int q = 0; atoms && q < a.probe_n3; ++q) {
        out[9 + q] = a.rv_unit * (double)a.r[(int64_t)q * a.nslot + a.probe_slot];
        out[9 + a.probe_n3 + q] = a.rv_unit * (double)a.v[(int64_t)q * a.nslot + a.probe_slot];
    }
}

/* ------------------------------------------------------------ diagnostics */

struct DiagPartial {
    double max_e, max_ex, max_r;
    int64_t key_r; /* reference loop-order key of the first max_r */
};

/* The reference keeps the first strictly larger |r| starting from 0
 * (fdtd.c:3567-3586): ties go to the smaller loop-order key and zeros never
 * set an argmax. */
__device__ __forceinline__ void diag_merge(DiagPartial& a, const DiagPartial& b)
{
    a.max_e = fmax(a.max_e, b.max_e);
    a.max_ex = fmax(a.max_ex, b.max_ex);
    if (b.max_r > a.max_r || (b.max_r == a.max_r && b.max_r > 0.0 && b.key_r < a.key_r)) {
        a.max_r = b.max_r;
        a.key_r = b.key_r;
    }
}

/* The reference's loop-order key of coordinate q of pool slot s */
__device__ __forceinline__ int64_t diag_key(const int64_t* slot_cell, int64_t s, int q, int ny, int nz, int nxp, int n3max)
{
    const int64_t c = slot_cell[s], jk = c / nxp;
    const int i = (int)(c % nxp), j = (int)(jk % ny), k = (int)(jk / ny);
    return (((int64_t)i * ny + j) * nz + k) * (int64_t)n3max + q;
}

/* Pass 1 over cells (|E|, |Ex|) and pool slots (|r|, times rv_unit); one
 * partial per block into scratch.  slot_cell maps a pool slot to its device
 * cell index.  Bound by HBM: E once and r once.  The square root is taken of
 * the largest sum (it rounds monotonically), the pool's cell is decoded only
 * where a new maximum or a tie needs its key, rows are read 16 bytes per
 * lane, and a slot's coordinates eight loads at a time: 1.6 GB of E (512 x 512
 * x 256, FP64) or of r (16 atoms) took 0.8 ms with a root, a division by the
 * row length and one load in flight per cell; a frame of 256 x 256 x 128 with
 * 16 atoms in half the cells (1.8 GB FP64) takes 0.45 ms now, 0.04 of it
 * without the diagnostics. */
template <typename R>
__global__ void __launch_bounds__(256) diag_pass1(const Fields<R> f, int nx, int ny, int nz, int nxp,
                                                  const R* r, double rv_unit, int64_t nslot, const int64_t* slot_cell,
                                                  const int32_t* slot_n3, int n3max, DiagPartial* scratch)
{
    DiagPartial acc{0.0, 0.0, 0.0, INT64_MAX};
    constexpr int V = 16 / (int)sizeof(R);
    struct alignas(16) Vec { R v[V]; };
    const int lane = threadIdx.x & 31;
    const int64_t rows = (int64_t)ny * nz, warps = (int64_t)gridDim.x * (blockDim.x / 32);
    for (int64_t row = (int64_t)blockIdx.x * (blockDim.x / 32) + threadIdx.x / 32; row < rows; row += warps) {
        const Vec* x = reinterpret_cast<const Vec*>(f.ex + row * nxp);
        const Vec* y = reinterpret_cast<const Vec*>(f.ey + row * nxp);
        const Vec* z = reinterpret_cast<const Vec*>(f.ez + row * nxp);
#pragma unroll 2
        for (int t = lane; t < nxp / V; t += 32) {
            const Vec a = x[t], b = y[t], c = z[t];
#pragma unroll
            for (int q = 0; q < V; ++q) {
                if (t * V + q >= nx) continue; /* padding */
                const double u = (double)a.v[q], v = (double)b.v[q], w = (double)c.v[q];
                acc.max_e = fmax(acc.max_e, __dadd_rn(__dadd_rn(__dmul_rn(u, u), __dmul_rn(v, v)), __dmul_rn(w, w)));
                acc.max_ex = fmax(acc.max_ex, fabs(u));
            }
        }
    }
    acc.max_e = __dsqrt_rn(acc.max_e);
    R best = R(0); /* |r| as stored */
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t s = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; s < nslot; s += stride) {
        const int n3 = slot_n3[s];
        for (int q0 = 0; q0 < n3; q0 += 8) {
            R v[8];
#pragma unroll
            for (int q = 0; q < 8; ++q) v[q] = q0 + q < n3 ? r[(int64_t)(q0 + q) * nslot + s] : R(0);
#pragma unroll
            for (int q = 0; q < 8; ++q) {
                const R m = v[q] < R(0) ? -v[q] : v[q];
                if (m >= best && m > R(0)) {
                    const int64_t key = diag_key(slot_cell, s, q0 + q, ny, nz, nxp, n3max);
                    if (m > best || key < acc.key_r) acc.key_r = key;
                    best = m;
                }
            }
        }
    }
    acc.max_r = rv_unit * (double)best;
    __shared__ DiagPartial sh[256];
    sh[threadIdx.x] = acc;
    __syncthreads();
    for (int w = blockDim.x / 2; w > 0; w >>= 1) {
        if ((int)threadIdx.x < w) diag_merge(sh[threadIdx.x], sh[threadIdx.x + w]);
        __syncthreads();
    }
    if (threadIdx.x == 0) scratch[blockIdx.x] = sh[0];
}

/* the partials of pass 1 reduced by one block of 256 threads; every thread
 * gets the result */
__device__ __forceinline__ DiagPartial diag_reduce(const DiagPartial* scratch, int n)
{
    DiagPartial acc{0.0, 0.0, 0.0, INT64_MAX};
    for (int t = threadIdx.x; t < n; t += blockDim.x) diag_merge(acc, scratch[t]);
    __shared__ DiagPartial sh[256];
    sh[threadIdx.x] = acc;
    __syncthreads();
    for (int w = blockDim.x / 2; w > 0; w >>= 1) {
        if ((int)threadIdx.x < w) diag_merge(sh[threadIdx.x], sh[threadIdx.x + w]);
        __syncthreads();
    }
    return sh[0];
}

__global__ void __launch_bounds__(256) diag_pass2(const DiagPartial* scratch, int n, DiagPartial* out)
{
    const DiagPartial d = diag_reduce(scratch, n);
    if (threadIdx.x == 0) *out = d;
}

/* ---------------------------------------------------------- output frames */

constexpr int kFrameMaxN3 = 192; /* 3 N for N <= 64 atoms */

/* The small part of an output frame (php_frame_begin), written by the device
 * into page-locked host memory. */
struct FrameHead {
    DiagPartial diag;                                       /* diagnostics */
    double diag_point[9];                                   /* fields at the max |r| cell */
    double diag_r[kFrameMaxN3], diag_v[kFrameMaxN3];        /* r, v there */
    double point[9];                                        /* fields at the requested point */
    double cell_r[kFrameMaxN3], cell_v[kFrameMaxN3];        /* r, v of the requested cell */
    int32_t diag_natom, cell_natom;
    int32_t probe_count[2];                                 /* rows recorded, overflow flag */
    int32_t err;                                            /* a sweep's bounded wait gave up */
    int32_t pad_;
};

/* Field values (Ex Ey Ez Dx Dy Dz Hx Hy Hz) at device cell cf, and r, v of the
 * atom cell ca (none when its material has no atoms, or ca < 0), zeros past
 * them: the head's memory is not cleared between frames. */
template <typename R>
__device__ __forceinline__ void frame_cell(const Fields<R>& f, const DView<R>& dv, const uint8_t* mat, const int32_t* slot,
                                           const MatCoef<R>* mc, const R* r, const R* v, double rv_unit,
                                           int64_t nslot, int64_t cf, int64_t ca, double* point9, double* rr,
                                           double* vv, int32_t* natom)
{
    const int t = threadIdx.x;
    if (point9 && t < 9) {
        point9[t] = field_at(f, dv, t, cf);
    }
    if (!rr) return;
    const int na = ca >= 0 ? mc[mat[ca]].natom : 0;
    const int64_t s = (na > 0 && slot) ? slot[ca] : -1;
    if (t == 0) *natom = s >= 0 ? na : 0;
    for (int q = t; q < kFrameMaxN3; q += blockDim.x) {
        const bool live = s >= 0 && q < 3 * na;
        rr[q] = live ? rv_unit * (double)r[(int64_t)q * nslot + s] : 0.0;
        vv[q] = live ? rv_unit * (double)v[(int64_t)q * nslot + s] : 0.0;
    }
}

/* One block of 256 threads.  parts: the partials of this frame's diagnostics
 * (nullptr: none); the point's device index (k may be -1 or nz, the halo
 * planes; has_point 0: none) and the cell's (-1: none); probe_count: the probe
 * row counter (nullptr: no probe), reset where `rows` (nrows of them) go with
 * the frame.  head and rows_out are page-locked host memory, written over
 * PCIe: a frame of a small grid is a few launches, and a copy or a memset
 * costs as much as one (32^3 grid: frame 69 us with three copies, a memset and
 * the reduction in a launch of its own).  Thread 0 writes every natom field. */
template <typename R>
__global__ void __launch_bounds__(256) frame_gather(const Fields<R> f, const DView<R> dv, const uint8_t* mat, const int32_t* slot,
                             const MatCoef<R>* mc, const R* r, const R* v, double rv_unit, int64_t nslot, int nx, int ny, int nz,
                             int nxp, int n3max, const DiagPartial* parts, int nparts, int has_point, int64_t point_c,
                             int64_t cell_c, int32_t* probe_count, const double* rows, int64_t nrows, int row_len, double* rows_out,
                             const int32_t* err, FrameHead* head)
{
    const int t = threadIdx.x;
    if (parts) {
        const DiagPartial d = diag_reduce(parts, nparts);
        if (t == 0) head->diag = d;
        if (d.max_r > 0.0 && d.key_r != INT64_MAX) {
            /* reference loop order (i, j, k, coordinate), as php_diagnostics decodes it */
            const int64_t n3 = n3max > 1 ? n3max : 1;
            int64_t cell = d.key_r / n3;
            const int k = (int)(cell % nz);
            cell /= nz;
            const int j = (int)(cell % ny);
            const int i = (int)(cell / ny);
            const int64_t c = ((int64_t)k * ny + j) * nxp + i;
            frame_cell(f, dv, mat, slot, mc, r, v, rv_unit, nslot, c, c, head->diag_point, head->diag_r, head->diag_v,
                       &head->diag_natom);
        } else {
            if (t < 9) head->diag_point[t] = 0.0;
            frame_cell<R>(f, dv, mat, slot, mc, r, v, rv_unit, nslot, 0, -1, nullptr, head->diag_r, head->diag_v, &head->diag_natom);
        }
    }
    if (has_point)
        frame_cell<R>(f, dv, mat, slot, mc, r, v, rv_unit, nslot, point_c, -1, head->point, nullptr, nullptr, nullptr);
    if (cell_c >= 0)
        frame_cell<R>(f, dv, mat, slot, mc, r, v, rv_unit, nslot, cell_c, cell_c, nullptr, head->cell_r, head->cell_v,
                      &head->cell_natom);
    if (rows_out)
        for (int64_t q = t; q < nrows * row_len; q += blockDim.x) rows_out[q] = rows[q];
    if (t == 0) {
        head->probe_count[0] = probe_count ? probe_count[0] : 0;
        head->probe_count[1] = probe_count ? probe_count[1] : 0;
        if (rows) probe_count[0] = probe_count[1] = 0;
        head->err = *err;
    }
}

} // namespace phpdev

#include "php_sweeps.cuh"
#include "php_sweeps_tma.cuh"
#include "php_sweep_fused.cuh"
#include "php_ions.cuh"

/*
 * php_fdtd.cu -- libphpfdtd: the C ABI of include/php_fdtd.h on one B200.
 *
 * Host side of the device path: derives every per-material and per-axis
 * coefficient once (where the reference recomputes them per cell and step),
 * lays the domain out in HBM (see php_kernels.cuh), records one CUDA graph
 * per distinct step count and replays it, and serves the read-outs.
 *
 * Coefficients used by the strict mode are computed with the reference's
 * expressions and evaluation order (this file is compiled with host FP
 * contraction off), so the device sees the same doubles fdtd.c computes.
 */
#include "php_fdtd.h"
#include "php_internal.h"
#include "php_kernels.cuh"

#include <cuda_runtime.h>
#include <cudaTypedefs.h>

#include <algorithm>
#include <array>
#include <atomic>
#include <chrono>
#include <cmath>
#include <cstdarg>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>
#include <string>
#include <thread>
#include <vector>

using namespace phpdev;

namespace {

constexpr int kMaxChunk = 256;      /* steps per recorded graph */
/* steps per graph where a step is three to five sweep launches: recording and
 * instantiating one takes some 35 us per step then (a launch without the
 * programmatic attribute takes 4 us); php_step calls of more steps replay it,
 * their input rows in page-locked slots of this many steps, so that the same
 * 512 steps are enqueued ahead */
constexpr int kListChunk = 64;
constexpr int kProfKinds = PHP_PROFILE_KINDS; /* H sweep, E sweep, probe, DFT, ion pass, one-launch step */
/* Bytes of a slice that its gather writes to page-locked host memory itself,
 * and of monitor rows that frame_gather does; more go by a copy.  Frame with a
 * slice, by copy and direct: 16 KB 34 and 29 us, 64 KB 37 and 34, 256 KB 49
 * and 46, 512 KB 61 and 55, 1 MB 110 and 108, 4 MB 378 and 415.  Frame with
 * rows (one block writes them): 1 KB 27 and 26, 16 KB 29 and 28, 64 KB 40 and
 * 39, 131 KB 45 and 48, 262 KB 50 and 73. */
constexpr size_t kDirectSlice = 256 << 10;
constexpr int64_t kDirectRows = 64 << 10;
constexpr int kProbeCap = 8192;     /* probe rows held on the device */
constexpr double kEpsInf = 20.0;    /* EPS_INF, fdtd.c:202 */
/* The FP32 path keeps the lattice state as 2^48 r and 2^48 v: early in a
 * pulse the reference's displacements are 1e-42 m and below, under FP32's
 * normal range (1.2e-38), where subnormals keep only a few bits; scaled,
 * every displacement from 1e-52 m to the 1e-10 m divergence guard is a
 * normal number.  The factor is folded into QeZM (times 2^48) and QeZV
 * (times 2^-48), so a = QeZM E - DMM r and P_ion = QeZV r need no extra
 * operation, and a power of two changes no rounding.  Read-outs multiply
 * by rv_unit = 2^-48. */
constexpr double kIonScale32 = 281474976710656.0; /* 2^48 */

thread_local std::string g_create_error; /* errors of php_create, per calling thread */

struct DftPlane {
    int comp, z, first, interval, nfreq, cast_f32;
    std::vector<double> freq;
    double* acc = nullptr; /* [nfreq][ny][nx][2], x fastest (php_dft_read reorders) */
    int nsamples = 0;
    int in_off = 0;        /* offset of this plane's flag in a step-input row */
};

} // namespace

struct php_ctx {
    php_desc d{};
    int prec = 0;
    int nx = 0, ny = 0, nz = 0, nxp = 0, L = 0;
    int64_t plane = 0, ncell_dev = 0;
    int zchunk = 1;
    int n3max = 0, namax_tpl = 0;
    int64_t nslot = 0;           /* pool slots, padded to a multiple of 32 */
    int z_off = 0, nz_glob = 0;  /* z slab: global index of local plane 0, global nz */
    int step_part = 7;           /* launches of a step: 1 H sweep, 2 fused E sweep, 4 the rest (ions, probe, DFT) */
    int zc_first = 0, zc_count = -1; /* z chunks the sweeps launch over (-1: all) */
    bool part_staged = false;    /* php_step_part: this step's inputs are on the device */
    int num_sms = 148;
    double rv_unit = 1.0;        /* physical r, v per stored unit (FP32: 2^-48, kIonScale32) */
    /* failure-path test (PHP_TEST_STALL_WAIT=1 at php_create): the first
     * block of every H sweep gives up a bounded wait on a barrier nothing
     * arrives on, so the error flag and PHP_ERR_TIMEOUT can be checked
     * without a fault */
    int32_t stall_test = 0;
    bool any_ade = false, any_atoms = false;
    cudaStream_t stream = nullptr;
    /* php_create's own work (allocation, zeroing, uploads) runs on a stream
     * of the highest priority, so that a context built while others keep the
     * device busy does not queue behind their sweeps; `stream` (default
     * priority) takes over at the end of php_create */
    cudaStream_t setup = nullptr;
    /* launches recorded in the graph being captured (launch_chained), -1 when
     * none is */
    int chain = -1;
    /* page-locked staging of host -> device uploads (upload()) */
    void* up_buf[2] = {};
    cudaEvent_t up_ev[2] = {};
    bool up_used[2] = {};
    int up_cur = 0;              /* the buffer being filled, up to up_off */
    size_t up_off = 0;
    /* last error text: a fixed buffer, so that php_last_error's pointer stays
     * valid while another thread (php_frame_wait) records an error */
    char err[1024] = "";
    std::mutex err_mu;
    uint64_t bytes = 0;
    std::vector<void*> allocs;

    /* device state */
    void* f[9] = {};            /* field bases (plane 0) */
    void* psi[12] = {};
    /* one-launch step (he_sweep_tma): the second buffers of E, H (fo[0..2],
     * fo[6..8]) and of the H CPML state, which the
     * launch writes the new level to; swap_levels exchanges them with f and
     * psi after it.  level: how many swaps since php_create, mod 2 */
    bool fused = false;
    /* the interior of the domain in one launch (interior_sweep_tma), the rest
     * in the two sweeps: E and H double buffered like the one-launch step's,
     * the H CPML state in place (the interior has none).  Block lists
     * (StepArgs::list): interior, H sweep, E sweep */
    bool split = false;
    /* the E sweep's blocks in a launch per kind (lists[2..4]), in place */
    bool by_class = false;
    bool allow_split = true;     /* php_create_buffers */
    int4* lists[5] = {};         /* interior, H sweep, E sweep: plain, atom, general blocks */
    int nlist[5] = {};
    void* fo[9] = {};
    void* psio[6] = {};
    int level = 0;
    uint16_t* pcls = nullptr;    /* StepArgs::pcls */
    int zstep = 0;               /* planes per block of he_sweep_tma */
    uint8_t* mat = nullptr;
    uint8_t* plain_blk = nullptr; /* plain blocks of the fused sweep (StepArgs::plain_blk) */
    double kdp[3] = {};
    uint8_t* plain_h = nullptr;   /* plain blocks of the H sweep (StepArgs::plain_h) */
    double khp[3] = {};
    int32_t* slot = nullptr;
    int64_t* slot_cell = nullptr;
    uint8_t* slot_mat = nullptr;
    int32_t* slot_n3 = nullptr;
    void *P = nullptr, *Po = nullptr, *r = nullptr, *v = nullptr;
    void* Dp = nullptr;          /* D of the cells with a slot (fast modes; the strict mode keeps D in f[3..5]) */
    uint32_t* Dc = nullptr;      /* StepArgs::Dc */
    double* dmat = nullptr;      /* M^-1 per material, for D of the cells that keep E alone */
    void* mc = nullptr;          /* MatCoef<R>[nmat] */
    void* ion_coef = nullptr;
    void* axis_tab[3][7] = {};   /* kappa b c kh kd ch cd per axis */
    /* per-step inputs (source values, DFT flags and phasors), double
     * buffered so that the host fills one while the GPU runs the other */
    double* step_in = nullptr;   /* buffer the graph being recorded reads */
    double* step_in_dev[2] = {};  /* [kMaxChunk][row] each */
    double* step_in_host[2] = {}; /* pinned */
    int max_chunk = kMaxChunk;    /* steps per graph: kMaxChunk or kListChunk */
    /* copy out of a page-locked slot (max_chunk rows; 2 kMaxChunk rows in all) finished */
    cudaEvent_t staged[2 * kMaxChunk / kListChunk] = {};
    int chunk_no = 0;
    int step_row = 0;
    int probe_off = 0;           /* offset of the monitor row's index in a step-input row */
    double* src_acc = nullptr;   /* StepArgs::src_acc */
    void* scratch = nullptr;     /* plane gathers, diagnostics */
    size_t scratch_bytes = 0;
    void* host_stage = nullptr;  /* pinned */
    size_t host_stage_bytes = 0;

    /* host copies kept for reads */
    std::vector<int> mat_natom, mat_ade, mat_flags;
    std::vector<double> mat_cs, mat_sn;
    std::vector<int32_t> slot_host_dummy;

    /* sources */
    std::vector<php_source_desc> src;
    int64_t src_cell[kMaxSources] = {};
    int32_t src_comp[kMaxSources] = {};
    int nsrc_active = 0;
    std::vector<int> src_active_index;

    /* stepping */
    int32_t t = 0;
    std::map<int, cudaGraphExec_t> graphs; /* key: 4 * steps + 2 * level + input buffer */
    int last_launches = 0;

    /* probe */
    bool probe = false;
    int64_t probe_cf = 0, probe_slot = -1;
    DCell probe_d{};             /* where D of the field cell is */
    int probe_ka = 0;            /* plane of the atom cell */
    int probe_n3 = 0;
    double* probe_rows = nullptr;
    int32_t* probe_count = nullptr;

    std::vector<DftPlane> dft;
    /* the E sweep samples E and D planes itself (dft_folded); PHP_DFT_FOLD=0
     * at create keeps a dft_sample launch per plane; likewise it records the
     * monitor row (probe_folded; PHP_PROBE_FOLD=0) */
    bool dft_fold = true, probe_fold = true;

    /* TMA maps of the sweep kernels; maps_o those of the second buffers */
    TmaMaps maps, maps_o;
    int64_t census[PHP_CENSUS_LEN] = {}; /* php_block_census */
    int32_t* err_flag = nullptr;

    /* per-kernel timing (php_profile_enable) */
    bool profile = false;
    std::vector<cudaEvent_t> prof_ev;   /* [kMaxChunk][kProfKinds][begin, end] */
    double prof_ms[kProfKinds] = {};
    int64_t prof_n[kProfKinds] = {};

    /* many-atom cells: ion pass apart from the E sweep (php_ions.cuh) */
    bool ion_split = false, ion_tc = false;
    int ion_np = 0;              /* 3N padded to 16 */
    void* Pr = nullptr;          /* [3][nslot] */
    void* ion_dmm = nullptr;     /* CUDA-core kernel: [np][np] R */
    void* ion_dfrag = nullptr;   /* FP64 ring: m8n8k4 B fragments */
    void* ion_bsplit = nullptr;  /* tensor kernel: DMM hi, lo bf16 images */
    bool ion_pipe = false;       /* TMA-fed pass (ion_pipe) */
    IonMaps ion_maps;
    int n3_ion = 0;
    int ion_off_ref = 0;
    /* the few-atom material (N <= 4) with the most cells: its coefficients
     * ride in the sweep's kernel parameters (StepArgs::ion_k) */
    int ion_k_off = -1;
    std::vector<double> ion_k;
    std::vector<double> iso_scale;   /* StepArgs::iso, per material */
    /* per material: em and eps_im of the packed record; the chosen one rides
     * in StepArgs::tns_* */
    std::vector<std::array<double, 18>> mat_tns;
    int tns_id = -1;
    /* the few-atom material of ion_k (with the ion pass apart: the atom
     * material with the most cells; without atoms: one that keeps D beside E)
     * and its packed record (MatCoef<R> bytes),
     * for StepArgs::amc; atom_blocks: kPlainAtoms blocks exist */
    int atom_id = -1;
    std::vector<unsigned char> atom_mc;
    bool atom_blocks = false;
    int pool_id = -1;             /* StepArgs::dmc */
    std::vector<unsigned char> pool_mc;

    /* output frames (php_frame_begin): page-locked slots taken in ticket
     * order; state 0 free, 1 taken (begun and not released) */
    struct FrameSlot {
        std::atomic<int> state{0};
        int32_t ticket = -1, step = 0;
        php_frame_req req{};
        int64_t rows_copied = 0, slice_len = 0;
        int32_t row_len = 0;
        cudaEvent_t done = nullptr;
        FrameHead* head = nullptr;   /* pinned */
        float* slice = nullptr;      /* pinned */
        double* rows = nullptr;      /* pinned */
        size_t rows_bytes = 0;
    };
    FrameSlot frames[PHP_FRAME_SLOTS];
    int32_t frame_next = 0;
    int32_t probe_t0 = 0;        /* step of the last probe read (rows pending = t - probe_t0) */
};

/* ------------------------------------------------------------------ utils */

static int fail(php_ctx* c, int code, const char* fmt, ...)
{
    char buf[1024];
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(buf, sizeof(buf), fmt, ap);
    va_end(ap);
    if (c) {
        std::lock_guard<std::mutex> g(c->err_mu);
        memcpy(c->err, buf, sizeof(buf));
    } else {
        g_create_error = buf;
    }
    return code;
}

#define CK(call)                                                                                   \
    do {                                                                                           \
        cudaError_t e_ = (call);                                                                   \
        if (e_ != cudaSuccess)                                                                     \
            return fail(ctx, PHP_ERR_CUDA, "%s failed: %s (%s:%d)", #call, cudaGetErrorString(e_), \
                        __FILE__, __LINE__);                                                       \
    } while (0)

/* Device buffers come from the device's stream-ordered pool, allocated and
 * freed on the context's stream: destroying one context never waits for the
 * work of the others (cudaFree would synchronise the whole device), which
 * the serving loop relies on. */
static int dalloc(php_ctx* ctx, void** p, size_t bytes, bool clear = true)
{
    *p = nullptr;
    if (bytes == 0) bytes = 16;
    cudaError_t e = cudaMallocAsync(p, bytes, ctx->stream);
    if (e != cudaSuccess) {
        *p = nullptr;
        cudaGetLastError();
        return fail(ctx, PHP_ERR_OOM, "cudaMallocAsync(%zu) failed: %s", bytes, cudaGetErrorString(e));
    }
    ctx->allocs.push_back(*p);
    ctx->bytes += bytes;
    if (!clear) return PHP_OK;
    e = cudaMemsetAsync(*p, 0, bytes, ctx->stream);
    if (e != cudaSuccess) return fail(ctx, PHP_ERR_CUDA, "cudaMemset failed: %s", cudaGetErrorString(e));
    return PHP_OK;
}

static int upload(php_ctx* ctx, void* dst, const void* src, size_t bytes);

static size_t rsize(int prec) { return prec == PHP_PREC_FP32 ? sizeof(float) : sizeof(double); }

/* --------------------------------------------------- coefficient derivation */

/* Real part of inverse_dielectric_tensor (fdtd.c:555-625). */
static int complex_inverse_re(const double* e, const double* ei, double* out)
{
    const double xx = e[0], xy = e[1], xz = e[2], yx = e[3], yy = e[4], yz = e[5], zx = e[6], zy = e[7], zz = e[8];
    const double xxi = ei[0], xyi = ei[1], xzi = ei[2], yxi = ei[3], yyi = ei[4], yzi = ei[5], zxi = ei[6],
                 zyi = ei[7], zzi = ei[8];
    double det_real = xx * (yy * zz - yz * zy) - xy * (yx * zz - yz * zx) + xz * (yx * zy - yy * zx);
    double det_imag = xxi * (yyi * zzi - yzi * zyi) - xyi * (yxi * zzi - yzi * zxi) + xzi * (yxi * zyi - yyi * zxi);
    double det_magnitude = sqrt(det_real * det_real + det_imag * det_imag);
    if (fabs(det_magnitude) < 1e-12) return -1;
    double idr = det_real / (det_real * det_real + det_imag * det_imag);
    double idi = -det_imag / (det_real * det_real + det_imag * det_imag);
    out[0] = idr * (yy * zz - yz * zy) - idi * (yyi * zzi - yzi * zyi);
    out[1] = idr * (xz * zy - xy * zz) - idi * (xzi * zyi - xyi * zzi);
    out[2] = idr * (xy * yz - xz * yy) - idi * (xyi * yzi - xzi * yyi);
    out[3] = idr * (yz * zx - yx * zz) - idi * (yzi * zxi - yxi * zzi);
    out[4] = idr * (xx * zz - xz * zx) - idi * (xxi * zzi - xzi * zxi);
    out[5] = idr * (xz * yx - xx * yz) - idi * (xzi * yxi - xxi * yzi);
    out[6] = idr * (yx * zy - yy * zx) - idi * (yxi * zyi - yyi * zxi);
    out[7] = idr * (xy * zx - xx * zy) - idi * (xyi * zxi - xxi * zyi);
    out[8] = idr * (xx * yy - xy * yx) - idi * (xxi * yyi - xyi * yxi);
    return 0;
}

/* 3x3 inverse by the adjugate (fdtd.c:205-258); -1 when |det| < 1e-12. */
static int inverse3(const double m[3][3], double inv[3][3])
{
    double det = m[0][0] * (m[1][1] * m[2][2] - m[1][2] * m[2][1]) - m[0][1] * (m[1][0] * m[2][2] - m[1][2] * m[2][0]) +
                 m[0][2] * (m[1][0] * m[2][1] - m[1][1] * m[2][0]);
    if (fabs(det) < 1e-12) return -1;
    double adj[3][3];
    adj[0][0] = (m[1][1] * m[2][2] - m[1][2] * m[2][1]);
    adj[0][1] = -(m[1][0] * m[2][2] - m[1][2] * m[2][0]);
    adj[0][2] = (m[1][0] * m[2][1] - m[1][1] * m[2][0]);
    adj[1][0] = -(m[0][1] * m[2][2] - m[0][2] * m[2][1]);
    adj[1][1] = (m[0][0] * m[2][2] - m[0][2] * m[2][0]);
    adj[1][2] = -(m[0][0] * m[2][1] - m[0][1] * m[2][0]);
    adj[2][0] = (m[0][1] * m[1][2] - m[0][2] * m[1][1]);
    adj[2][1] = -(m[0][0] * m[1][2] - m[0][2] * m[1][0]);
    adj[2][2] = (m[0][0] * m[1][1] - m[0][1] * m[1][0]);
    for (int i = 0; i < 3; i++)
        for (int j = 0; j < 3; j++) inv[i][j] = adj[j][i] / det;
    return 0;
}

/* Double-precision per-material coefficients in the reference's order. */
struct MatD {
    int flags = 0, natom = 0;
    double eps_inv[9] = {}, eps_im[9] = {};
    double lf = 1.0, lt = 0.0, cs = 1.0, sn = 0.0;
    double gp_inv[9] = {}, gm[9] = {}, wp2[9] = {};
    /* fast modes, materials without ADE and atoms: E = em D in the lab frame
     * and D = dm E; e_only: both well conditioned, the cells keep E alone */
    double em[9] = {}, dm[9] = {};
    bool e_only = false;
    /* whether a cell of the material has a pool slot */
    bool slotted(bool strict) const { return (flags & (kAde | kAtoms)) || (!strict && !e_only); }
};

/* em = R^T eps^-1 R lf (1 - lt) / eps0, the map from D to E that the fast
 * modes apply (fdtd.c:3429-3503), and its inverse.  Where eps^-1 is close to
 * singular (its real part can be, for complex eps) the increment form would
 * lose digits, and D has no read-out from E: those materials keep D.  So do
 * those whose D would be read out with fewer correct digits than it was held
 * in: M^-1 of a rounded E has up to kDSpread = max over rows of |M^-1| |M|
 * (Skeel's condition number) roundings.  It is 1 for a diagonal M of any
 * contrast and the contrast of eps for one turned by 45 degrees.  Error of D
 * over that of a stored D, and of E over E = M D (one cell, 1000 oscillating
 * increments, single precision, largest of 2 axes x 3 angles): 1.8 and 1.4 at a
 * contrast of 2, 3.1 and 1.2 at 4, 8.5 and 1.5 at 8, 33 and 1.7 at 32, 170 and
 * 1.8 at 250.  The limit admits the first of these; both precisions alike. */
constexpr double kDSpread = 2.0;
static void derive_e_only(const php_desc& d, MatD& o)
{
    double rot[3][3] = {{1, 0, 0}, {0, 1, 0}, {0, 0, 1}}, m[3][3], inv[3][3];
    if (o.flags & kRotZ) {
        rot[0][0] = rot[1][1] = o.cs;
        rot[0][1] = -o.sn;
        rot[1][0] = o.sn;
    } else if (o.flags & kRotX) {
        rot[1][1] = rot[2][2] = o.cs;
        rot[1][2] = -o.sn;
        rot[2][1] = o.sn;
    }
    double big = 0.0, big_inv = 0.0;
    for (int a = 0; a < 3; a++)
        for (int b = 0; b < 3; b++) {
            double v = 0.0;
            for (int p = 0; p < 3; p++)
                for (int q = 0; q < 3; q++) v += rot[p][a] * (o.eps_inv[p * 3 + q] * (o.lf * (1.0 - o.lt))) * rot[q][b];
            m[a][b] = v;
            big = std::max(big, fabs(v));
        }
    if (!(big > 0.0) || !std::isfinite(big)) return;
    double s[3][3]; /* scaled to order one, for inverse3's absolute bound on the determinant */
    for (int a = 0; a < 3; a++)
        for (int b = 0; b < 3; b++) s[a][b] = m[a][b] / big;
    if (inverse3(s, inv)) return;
    for (int a = 0; a < 9; a++) big_inv = std::max(big_inv, fabs(inv[a / 3][a % 3]));
    if (!(big_inv < 256.0)) return;
    double spread = 0.0;
    for (int a = 0; a < 3; a++) {
        double row = 0.0;
        for (int b = 0; b < 3; b++)
            for (int c = 0; c < 3; c++) row += fabs(inv[a][b] * s[b][c]);
        spread = std::max(spread, row);
    }
    if (!(spread <= kDSpread * (1.0 + 1e-9))) return;
    for (int a = 0; a < 9; a++) {
        o.em[a] = m[a / 3][a % 3] / d.epsilon0;
        o.dm[a] = inv[a / 3][a % 3] / big * d.epsilon0;
    }
    o.e_only = true;
}

static int derive_material(php_ctx* ctx, int id, const php_material_desc& m, MatD& o)
{
    const php_desc& d = ctx->d;
    if (complex_inverse_re(m.eps_re, m.eps_im, o.eps_inv))
        return fail(ctx, PHP_ERR_INPUT, "Error: Singular dielectric tensor! (material %d)", id);
    memcpy(o.eps_im, m.eps_im, sizeof(o.eps_im));
    /* fdtd.c:3414-3415 */
    o.lf = 1.0 / (1.0 + m.sigma * d.dt / (2 * d.epsilon0));
    o.lt = (m.sigma * d.dt / (2 * d.epsilon0)) * o.lf;
    if (fabs(m.anglez) > 1e-10) {
        o.flags |= kRotZ;
        o.cs = cos(m.anglez);
        o.sn = sin(m.anglez);
    } else if (fabs(m.anglex) > 1e-10) {
        o.flags |= kRotX;
        o.cs = cos(-m.anglex);
        o.sn = sin(-m.anglex);
    }
    if (m.use_ade != 0 && m.use_ade != 1) return fail(ctx, PHP_ERR_INPUT, "Error: use_ADE must be 0 or 1 (material %d)", id);
    if (m.use_ade == 1) {
        o.flags |= kAde;
        const double f = d.source_frequency;
        double epsr1[3][3], epsr1_inv[3][3], gama[3][3], gdt2p1[3][3], gdt2m1[3][3], gp_inv[3][3];
        for (int a = 0; a < 3; a++)
            for (int b = 0; b < 3; b++) epsr1[a][b] = m.eps_re[a * 3 + b];
        epsr1[0][0] = m.eps_re[0] - kEpsInf;
        epsr1[1][1] = m.eps_re[4] - kEpsInf;
        epsr1[2][2] = m.eps_re[8] - kEpsInf;
        if (epsr1[0][0] >= 0 || epsr1[1][1] >= 0 || epsr1[2][2] >= 0)
            return fail(ctx, PHP_ERR_INPUT, "Error: EPS_INF is too small for material %d", id);
        if (inverse3(epsr1, epsr1_inv)) return fail(ctx, PHP_ERR_INPUT, "Error: epsr1 can not be inversed (material %d)", id);
        const double* ei = m.eps_im;
        /* fdtd.c:2490-2498 */
        for (int a = 0; a < 3; a++)
            for (int b = 0; b < 3; b++)
                gama[a][b] = -(ei[a * 3 + 0] * epsr1_inv[0][b] + ei[a * 3 + 1] * epsr1_inv[1][b] + ei[a * 3 + 2] * epsr1_inv[2][b]) *
                             f * 2.0 * M_PI;
        /* fdtd.c:2499-2507 */
        for (int a = 0; a < 3; a++)
            for (int b = 0; b < 3; b++)
                o.wp2[a * 3 + b] = -f * f * 4.0 * M_PI * M_PI * epsr1[a][b] +
                                   f * 2.0 * M_PI * (gama[a][0] * ei[0 * 3 + b] + gama[a][1] * ei[1 * 3 + b] + gama[a][2] * ei[2 * 3 + b]);
        /* fdtd.c:2508-2517 */
        for (int a = 0; a < 3; a++)
            for (int b = 0; b < 3; b++) {
                gdt2p1[a][b] = +gama[a][b] * d.dt / 2.0;
                gdt2m1[a][b] = -gama[a][b] * d.dt / 2.0;
                if (a == b) {
                    gdt2p1[a][b] += 1.0;
                    gdt2m1[a][b] += 1.0;
                }
            }
        if (inverse3(gdt2p1, gp_inv)) return fail(ctx, PHP_ERR_INPUT, "Error: gdt2p1 can not be inversed (material %d)", id);
        for (int a = 0; a < 3; a++)
            for (int b = 0; b < 3; b++) {
                o.gp_inv[a * 3 + b] = gp_inv[a][b];
                o.gm[a * 3 + b] = gdt2m1[a][b];
            }
    } else {
        bool lossy = false;
        for (int q = 0; q < 9; q++) lossy |= (m.eps_im[q] != 0.0);
        if (lossy) o.flags |= kLossy;
    }
    if (m.natom < 0) return fail(ctx, PHP_ERR_INPUT, "negative natom (material %d)", id);
    if (m.natom > 0) {
        if (!m.qezv || !m.qezm || !m.dmm) return fail(ctx, PHP_ERR_INPUT, "material %d: natom > 0 needs QeZV, QeZM and DMM", id);
        o.flags |= kAtoms;
        o.natom = m.natom;
    }
    if (!(o.flags & (kAde | kAtoms))) derive_e_only(d, o);
    return PHP_OK;
}

static bool is_iso(const MatD& s);

template <typename R>
static MatCoef<R> pack_material(const php_ctx* ctx, const MatD& s, int ion_off)
{
    MatCoef<R> o;
    memset(&o, 0, sizeof(o));
    o.flags = s.flags;
    o.natom = s.natom;
    o.ion_off = ion_off;
    const php_desc& d = ctx->d;
    const bool strict = ctx->prec == PHP_PREC_FP64_STRICT;
    const double c1 = d.dt * d.source_frequency * 2.0 * 3.14159265;
    const double e0dt2 = d.epsilon0 * d.dt * d.dt;
    for (int q = 0; q < 9; q++) {
        if (strict) {
            o.eps_inv[q] = (R)s.eps_inv[q];
            o.eps_im[q] = (R)s.eps_im[q];
            o.wp2[q] = (R)s.wp2[q];
        } else {
            o.eps_inv[q] = (R)(s.eps_inv[q] * (s.lf * (1.0 - s.lt) / d.epsilon0));
            o.eps_im[q] = (R)(s.eps_im[q] * c1 * d.epsilon0);
            o.wp2[q] = (R)(s.wp2[q] * e0dt2);
        }
        o.gp_inv[q] = (R)s.gp_inv[q];
        o.gm[q] = (R)s.gm[q];
    }
    if (ctx->prec == PHP_PREC_FP32 && (s.flags & kAde)) {
        /* increment form of the ADE recurrence (see e_update):
         * A = (I + G)^-1 2G with G = I - gm, B = (I + G)^-1 eps0 dt^2 wp2,
         * formed in double before rounding */
        for (int r = 0; r < 3; r++)
            for (int q = 0; q < 3; q++) {
                double av = 0.0, bv = 0.0;
                for (int t = 0; t < 3; t++) {
                    const double g2 = 2.0 * ((t == q ? 1.0 : 0.0) - s.gm[t * 3 + q]); /* 2G[t][q] */
                    av += s.gp_inv[r * 3 + t] * g2;
                    bv += s.gp_inv[r * 3 + t] * s.wp2[t * 3 + q] * e0dt2;
                }
                o.gm[r * 3 + q] = (R)av;
                o.wp2[r * 3 + q] = (R)bv;
            }
    }
    o.lf = (R)s.lf;
    o.lt = (R)s.lt;
    o.cs = (R)s.cs;
    o.sn = (R)s.sn;
    o.ade_scale = (R)((1.0 - s.lt) / (d.epsilon0 * kEpsInf));
    if (!strict && s.e_only) {
        o.flags |= kEOnly;
        for (int q = 0; q < 9; q++) o.em[q] = (R)s.em[q];
    }
    if (!strict && is_iso(s)) o.flags |= kIso;
    return o;
}

/* init_pml (fdtd.c:962-989) and the per-cell b, c of fdtd.c:3146-3151. */
struct AxisD {
    std::vector<int32_t> slot;
    std::vector<double> kappa, b, c, kh, kd, ch, cd;
};

static void derive_axis(const php_desc& d, int n, double delta, bool is_z, AxisD& ax)
{
    const int L = d.pml_thickness;
    ax.slot.assign(n, -1);
    ax.kappa.assign(n, 1.0);
    ax.b.assign(n, 1.0);
    ax.c.assign(n, 0.0);
    ax.kh.assign(n, 0.0);
    ax.kd.assign(n, 0.0);
    ax.ch.assign(n, 0.0);
    ax.cd.assign(n, 0.0);
    std::vector<double> sigma(L > 0 ? L : 0), kappa(L > 0 ? L : 0), alpha(L > 0 ? L : 0);
    if (L > 0) {
        double m = 3.0, kappa_max = 7.0, alpha_max = 0.05;
        double eta0 = sqrt(d.mu0 / d.epsilon0);
        double sigma_max = -(m + 1) * log(d.pml_reflection) / (2.0 * eta0 * delta * L);
        for (int i = 0; i < L; i++) {
            double r = (double)(L - i) / L;
            sigma[i] = sigma_max * pow(r, m);
            kappa[i] = 1.0 + (kappa_max - 1.0) * pow(r, m);
            alpha[i] = alpha_max * (1.0 - r);
        }
    }
    for (int i = 0; i < n; i++) {
        int idx = -1, s = -1;
        if (is_z) {
            if (i < L || i >= n - L) {
                idx = (i < L) ? i : n - 1 - i;
                s = (i < L) ? i : L + idx;
            }
        } else if (L > 0 && i < L) {
            idx = i;
            s = i;
        } else if (L > 0 && i >= n - L) {
            idx = n - 1 - i;
            s = L + idx;
        }
        double kap = 1.0, bb = 1.0, cc = 0.0;
        if (idx >= 0) {
            double sx = sigma[idx];
            kap = kappa[idx];
            double ax_ = alpha[idx];
            double aw = sx / (kap * d.epsilon0) + ax_ / d.epsilon0;
            bb = exp(-aw * d.dt);
            cc = (aw > 1e-30) ? sx / (kap * kap * d.epsilon0) * (bb - 1.0) / aw : 0.0;
        }
        ax.slot[i] = s;
        ax.kappa[i] = kap;
        ax.b[i] = bb;
        ax.c[i] = cc;
        ax.kh[i] = d.dt / (d.mu0 * delta * kap);
        ax.kd[i] = d.dt / (delta * kap);
        ax.ch[i] = d.dt * cc / (d.mu0 * delta);
        ax.cd[i] = d.dt * cc / delta;
    }
}

#ifndef M_PI
#define M_PI 3.14159265358979323846
#endif

/* calculate_source_value, fdtd.c:1923-1947 */
static double source_value(const php_source_desc* s, double time)
{
    if (time < s->start_time || time > s->end_time) return 0.0;
    switch (s->type) {
    case 0: return s->amplitude * exp(-pow((time - s->t0) / s->tau, 2));
    case 1: return s->amplitude * sin(2 * M_PI * s->frequency * time);
    case 2: {
        double t_shift = time - s->t0;
        double arg = M_PI * M_PI * s->frequency * s->frequency * t_shift * t_shift;
        return s->amplitude * (1.0 - 2.0 * arg) * exp(-arg);
    }
    case 3: return s->amplitude * sin(2 * M_PI * s->frequency * time) * exp(-pow((time - s->t0) / s->tau, 2));
    default: return 0.0;
    }
}

/* fdtd.c:3375-3393: sources outside the grid or with an unknown component are
 * skipped (their value still goes to source.txt) */
static bool source_cell(const php_desc& d, const php_source_desc& S, int (&c)[3], int& comp)
{
    c[0] = S.x, c[1] = S.y, c[2] = S.z;
    comp = S.component == 'x' ? 0 : S.component == 'y' ? 1 : S.component == 'z' ? 2 : -1;
    return c[0] >= 0 && c[0] < d.nx && c[1] >= 0 && c[1] < d.ny && c[2] >= 0 && c[2] < d.nz && comp >= 0;
}

/* ------------------------------------------------------------ kernel args */

/* Whether the E sweep samples DFT plane q itself (StepArgs::dft_*): the first
 * kDftFold planes of E or D components; H planes and the rest take a
 * dft_sample launch after the step. */
static bool dft_folded(const php_ctx* ctx, size_t q)
{
    if (!ctx->dft_fold || ctx->dft[q].comp > PHP_DZ) return false;
    int before = 0;
    for (size_t r = 0; r < q; r++) before += ctx->dft[r].comp <= PHP_DZ;
    return before < kDftFold;
}

/* Whether the sweeps record the monitor row themselves (StepArgs::probe_*):
 * the field cell is a plane of the grid (not a halo plane) and a sweep
 * updates the atom cell's r and v (no ion pass apart).  A caller that sets the
 * z chunks keeps the launches it had with them: the row is folded where field
 * and atom cell lie in one chunk. */
static bool probe_folded(const php_ctx* ctx)
{
    if (!ctx->probe || !ctx->probe_fold || ctx->ion_split) return false;
    const int kf = (int)(ctx->probe_cf / ctx->plane);
    if (ctx->probe_cf < 0 || kf >= ctx->nz) return false;
    return ctx->probe_n3 == 0 || ctx->d.z_chunk <= 0 || kf / ctx->zchunk == ctx->probe_ka / ctx->zchunk;
}

/* dft_sample launches per step */
static int dft_launched(const php_ctx* ctx)
{
    int n = 0;
    for (size_t q = 0; q < ctx->dft.size(); q++) n += !dft_folded(ctx, q);
    return n;
}

template <typename R>
static Fields<R> make_fields(const php_ctx* ctx)
{
    R* const* fp = reinterpret_cast<R* const*>(ctx->f);
    return Fields<R>{fp[0], fp[1], fp[2], fp[3], fp[4], fp[5], fp[6], fp[7], fp[8]};
}

template <typename R>
static DView<R> make_dview(const php_ctx* ctx)
{
    return DView<R>{(const R*)ctx->Dp, ctx->mat, ctx->slot, ctx->dmat, ctx->nslot, ctx->ncell_dev};
}

template <typename R>
static StepArgs<R> make_args(php_ctx* ctx, int s_local)
{
    StepArgs<R> a;
    memset(&a, 0, sizeof(a));
    a.f = make_fields<R>(ctx);
    a.Dp = (R*)ctx->Dp;
    a.Dc = ctx->Dc;
    a.dv = make_dview<R>(ctx);
    R* const* pp = reinterpret_cast<R* const*>(ctx->psi);
    a.psi = Psi<R>{pp[0], pp[1], pp[2], pp[3], pp[4], pp[5], pp[6], pp[7], pp[8], pp[9], pp[10], pp[11]};
    AxisTab<R>* tabs[3] = {&a.tx, &a.ty, &a.tz};
    for (int ax = 0; ax < 3; ax++) {
        AxisTab<R>& t = *tabs[ax];
        t.kappa = (const R*)ctx->axis_tab[ax][0];
        t.b = (const R*)ctx->axis_tab[ax][1];
        t.c = (const R*)ctx->axis_tab[ax][2];
        t.kh = (const R*)ctx->axis_tab[ax][3];
        t.kd = (const R*)ctx->axis_tab[ax][4];
        t.ch = (const R*)ctx->axis_tab[ax][5];
        t.cd = (const R*)ctx->axis_tab[ax][6];
    }
    a.mat = ctx->mat;
    a.slot = ctx->slot;
    a.mc = (const MatCoef<R>*)ctx->mc;
    a.ion_coef = (const R*)ctx->ion_coef;
    a.P = (R*)ctx->P;
    a.Po = (R*)ctx->Po;
    a.r = (R*)ctx->r;
    a.v = (R*)ctx->v;
    a.pr = ctx->ion_split ? (const R*)ctx->Pr : nullptr;
    a.ion_k_off = ctx->ion_k_off;
    for (size_t q = 0; q < ctx->ion_k.size() && q < (size_t)kIonK; q++) a.ion_k[q] = (R)ctx->ion_k[q];
    for (size_t q = 0; q < ctx->iso_scale.size() && q < (size_t)kIsoMats; q++) a.iso[q] = (R)ctx->iso_scale[q];
    a.plain_blk = ctx->plain_blk;
    for (int q = 0; q < 3; q++) a.kdp[q] = (R)ctx->kdp[q];
    a.plain_h = ctx->plain_h;
    for (int q = 0; q < 3; q++) a.khp[q] = (R)ctx->khp[q];
    a.tns_flags = 0;
    if (ctx->tns_id >= 0) {
        const std::array<double, 18>& t = ctx->mat_tns[ctx->tns_id];
        a.tns_flags = ctx->mat_flags[ctx->tns_id];
        for (int q = 0; q < 9; q++) {
            a.tns_em[q] = (R)t[q];
            a.tns_im[q] = (R)t[9 + q];
        }
    }
    memset(&a.amc, 0, sizeof(a.amc));
    if (ctx->atom_blocks && ctx->atom_mc.size() == sizeof(MatCoef<R>)) memcpy(&a.amc, ctx->atom_mc.data(), sizeof(MatCoef<R>));
    a.dmc_id = -1;
    if (ctx->pool_id >= 0 && ctx->pool_mc.size() == sizeof(MatCoef<R>)) {
        a.dmc_id = ctx->pool_id;
        memcpy(&a.dmc, ctx->pool_mc.data(), sizeof(MatCoef<R>));
    }
    a.nslot = ctx->nslot;
    a.nx = ctx->nx;
    a.ny = ctx->ny;
    a.nz = ctx->nz;
    a.nxp = ctx->nxp;
    a.L = ctx->L;
    a.zchunk = ctx->zchunk;
    a.z_off = ctx->z_off;
    a.nzg = ctx->nz_glob;
    a.plane = ctx->plane;
    const php_desc& d = ctx->d;
    a.dt = d.dt;
    a.dxs = d.dx;
    a.dys = d.dy;
    a.dzs = d.dz;
    a.mu0 = d.mu0;
    a.eps0 = d.epsilon0;
    a.c1 = d.dt * d.source_frequency * 2.0 * 3.14159265;
    a.e0dt2 = d.epsilon0 * d.dt * d.dt;
    a.nsrc = ctx->nsrc_active;
    for (int s = 0; s < ctx->nsrc_active; s++) {
        a.src_cell[s] = ctx->src_cell[s];
        a.src_comp[s] = ctx->src_comp[s];
    }
    a.src_val = ctx->step_in + (size_t)s_local * ctx->step_row;
    a.src_acc = ctx->src_acc;
    a.err = ctx->err_flag;
    a.stall_test = ctx->stall_test;
    a.ndft = 0;
    for (size_t q = 0; q < ctx->dft.size(); q++) {
        if (!dft_folded(ctx, q)) continue;
        const DftPlane& p = ctx->dft[q];
        a.dft_z[a.ndft] = p.z;
        a.dft_comp[a.ndft] = p.comp;
        a.dft_nfreq[a.ndft] = p.nfreq;
        a.dft_cast[a.ndft] = p.cast_f32;
        a.dft_off[a.ndft] = p.in_off;
        a.dft_acc[a.ndft] = p.acc;
        a.ndft++;
    }
    a.probe_rows = nullptr;
    if (probe_folded(ctx)) {
        const int64_t cf = ctx->probe_cf;
        a.probe_rows = ctx->probe_rows;
        a.probe_count = ctx->probe_count;
        a.probe_kf = (int32_t)(cf / ctx->plane);
        a.probe_ka = ctx->probe_ka;
        a.probe_off = ctx->probe_off;
        a.probe_j = (int32_t)((cf % ctx->plane) / ctx->nxp);
        a.probe_i = (int32_t)(cf % ctx->nxp);
        a.probe_n3 = ctx->probe_n3;
        a.probe_slot = ctx->probe_slot;
        a.probe_cap = kProbeCap;
    }
    a.rv_unit = ctx->rv_unit;
    const bool dbl = ctx->fused || ctx->split;
    for (int q = 0; q < 3; q++) {
        a.enew[q] = (R*)(dbl ? ctx->fo : ctx->f)[PHP_EX + q];
        a.hnew[q] = (R*)(dbl ? ctx->fo : ctx->f)[PHP_HX + q];
    }
    for (int q = 0; q < 6; q++) a.psin_h[q] = (R*)(ctx->fused ? ctx->psio : ctx->psi)[q];
    a.pcls = ctx->pcls;
    a.zstep = ctx->zstep;
    return a;
}

/* After a double-buffered step: the buffers it wrote hold the current E, H and H
 * CPML state (on the host side, for every later launch and read). */
static void swap_levels(php_ctx* ctx)
{
    for (int q = 0; q < 3; q++) {
        std::swap(ctx->f[PHP_EX + q], ctx->fo[PHP_EX + q]);
        std::swap(ctx->f[PHP_HX + q], ctx->fo[PHP_HX + q]);
    }
    if (ctx->fused)
        for (int q = 0; q < 6; q++) std::swap(ctx->psi[q], ctx->psio[q]);
    std::swap(ctx->maps, ctx->maps_o);
    ctx->level ^= 1;
}

/* sweep launches of a step with the interior apart */
static int split_launches(const php_ctx* ctx)
{
    int n = 0;
    for (int c : ctx->nlist) n += c > 0;
    return n;
}

static inline void prof_mark(php_ctx* ctx, int s_local, int kind, int end)
{
    if (ctx->profile)
        cudaEventRecordWithFlags(ctx->prof_ev[((size_t)s_local * kProfKinds + kind) * 2 + end], ctx->stream,
                                 cudaEventRecordExternal);
}

template <typename R>
static void launch_ions(php_ctx* ctx)
{
    IonArgs<R> a;
    memset(&a, 0, sizeof(a));
    R* const* fp = reinterpret_cast<R* const*>(ctx->f);
    a.ex = fp[0];
    a.ey = fp[1];
    a.ez = fp[2];
    a.r = (R*)ctx->r;
    a.v = (R*)ctx->v;
    a.pr = (R*)ctx->Pr;
    a.slot_cell = ctx->slot_cell;
    a.slot_n3 = ctx->slot_n3;
    a.slot_mat = ctx->slot_mat;
    a.ion_off_ref = ctx->ion_off_ref;
    a.mat = ctx->mat;
    a.mc = (const MatCoef<R>*)ctx->mc;
    a.ion_coef = (const R*)ctx->ion_coef;
    a.dmm = (const R*)ctx->ion_dmm;
    a.dfrag = (const double*)ctx->ion_dfrag;
    a.bsplit = (const uint32_t*)ctx->ion_bsplit;
    a.nslot = ctx->nslot;
    const int tile = ctx->ion_pipe ? ion_tile<R>() : kIonTile;
    a.ntiles = (int32_t)((ctx->nslot + tile - 1) / tile);
    a.dt = ctx->d.dt;
    a.err = ctx->err_flag;
    a.stall_test = ctx->stall_test;
    cudaStream_t st = ctx->stream;
    if (ctx->ion_pipe) {
        /* one persistent CTA per SM */
        const int grid = (int)std::min<int64_t>(a.ntiles, ctx->num_sms);
        const int n3 = ctx->n3_ion;
#define PHP_ION_PIPE(NP, S) \
    ion_pipe<R, NP, S><<<grid, IonPipe<R, NP, S>::THREADS, IonPipe<R, NP, S>::SMEM, st>>>(a, ctx->ion_maps, n3)
        if constexpr (sizeof(R) == 4) {
            switch (ctx->ion_np) {
            case 16: PHP_ION_PIPE(16, 6); break;
            case 32: PHP_ION_PIPE(32, 6); break;
            case 48: PHP_ION_PIPE(48, 4); break;
            default: PHP_ION_PIPE(64, 3); break;
            }
        } else {
            switch (ctx->ion_np) {
            case 16: PHP_ION_PIPE(16, 6); break;
            case 32: PHP_ION_PIPE(32, 6); break;
            default: PHP_ION_PIPE(48, 4); break;
            }
        }
#undef PHP_ION_PIPE
        return;
    }
    const int grid = (int)std::min<int64_t>(a.ntiles, 148 * 4);
    ion_update_cc<R, 64><<<grid, kIonTile, 0, st>>>(a);
}

/* A sweep launch.  While a graph is recorded each one but the first is a
 * programmatic launch behind the one before it (chain_enter; not under
 * php_profile_enable, whose events stand between the launches); beside: it
 * does not depend on that one. */
template <typename R, typename F>
static void launch_chained(php_ctx* ctx, F kernel, dim3 grid, uint32_t smem, StepArgs<R>& a, const TmaMaps& maps, bool beside = false)
{
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(kBlockX, kBlockY, 1);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = ctx->stream;
    cudaLaunchAttribute at = {};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    const bool chained = ctx->chain > 0 && !ctx->profile;
    if (chained) {
        cfg.attrs = &at;
        cfg.numAttrs = 1;
    }
    if (ctx->chain >= 0) ctx->chain++;
    a.beside = chained && beside;
    cudaLaunchKernelEx(&cfg, kernel, a, maps);
}

/* The E sweep's launches over the block lists of its three kinds, beside each
 * other (the first behind the launches before); a.f and maps as for one
 * launch. */
template <typename R, int NA>
static void launch_e_lists(php_ctx* ctx, int s_local, StepArgs<R>& a, const TmaMaps& maps)
{
    const uint32_t smem = TmaGeom<R>::E_SMEM;
    bool beside = false;
    prof_mark(ctx, s_local, 1, 0);
    if (ctx->nlist[4]) { /* few blocks with long chains: first */
        a.list = ctx->lists[4];
        launch_chained(ctx, e_sweep_tma<R, false, NA, kEGeneral>, dim3(ctx->nlist[4]), smem, a, maps, beside);
        beside = true;
    }
    if constexpr (NA <= 4) /* more atoms in the sweep: no atom blocks */
        if (ctx->nlist[3]) {
            a.list = ctx->lists[3];
            launch_chained(ctx, e_sweep_tma<R, false, NA, kEAtoms>, dim3(ctx->nlist[3]), smem, a, maps, beside);
            beside = true;
        }
    if (ctx->nlist[2]) {
        a.list = ctx->lists[2];
        launch_chained(ctx, e_sweep_tma<R, false, 0, kEPlain>, dim3(ctx->nlist[2]), smem, a, maps, beside);
    }
    prof_mark(ctx, s_local, 1, 1);
    a.list = nullptr;
}

template <typename R, bool STRICT, int NA>
static void launch_step_t(php_ctx* ctx, int s_local, int& launches)
{
    StepArgs<R> a = make_args<R>(ctx, s_local);
    const int nchunk = (ctx->nz + ctx->zchunk - 1) / ctx->zchunk;
    a.zc0 = ctx->zc_count < 0 ? 0 : ctx->zc_first;
    dim3 grid((ctx->nx + kBlockX - 1) / kBlockX, (ctx->ny + kBlockY - 1) / kBlockY,
              ctx->zc_count < 0 ? nchunk : ctx->zc_count);
    bool do_h = ctx->step_part & 1, do_e = ctx->step_part & 2;
    const bool do_rest = ctx->step_part & 4;
    if constexpr (!STRICT) {
        if (ctx->split && do_h && do_e && grid.z > 0) {
            /* the interior and the H sweep of the rest read this level and
             * write the other; then the E sweep of the rest, whose H is the new
             * one */
            StepArgs<R> in = a;
            in.list = ctx->lists[0];
            prof_mark(ctx, s_local, 5, 0);
            launch_chained(ctx, interior_sweep_tma<R>, dim3(ctx->nlist[0]), FusedGeom<R, true>::SMEM, in, ctx->maps);
            prof_mark(ctx, s_local, 5, 1);
            a.list = ctx->lists[1];
            prof_mark(ctx, s_local, 0, 0);
            launch_chained(ctx, h_sweep_tma<R, STRICT, true>, dim3(ctx->nlist[1]), TmaGeom<R>::H_SMEM, a, ctx->maps, true);
            prof_mark(ctx, s_local, 0, 1);
            TmaMaps me = ctx->maps;
            me.h_halo = ctx->maps_o.h_halo;
            launch_e_lists<R, NA>(ctx, s_local, a, me);
            launches += split_launches(ctx);
            swap_levels(ctx);
            do_h = do_e = false;
        }
        if (ctx->fused && do_h && do_e && grid.z > 0) {
            /* the one-launch step: reads this level, writes the other */
            prof_mark(ctx, s_local, 5, 0);
            const dim3 fgrid((ctx->nx + FusedGeom<R, false>::TX - 1) / FusedGeom<R, false>::TX, (ctx->ny + FusedGeom<R, false>::TY - 1) / FusedGeom<R, false>::TY,
                             (ctx->nz + ctx->zstep - 1) / ctx->zstep);
            launch_chained(ctx, he_sweep_tma<R, NA>, fgrid, FusedGeom<R, false>::SMEM, a, ctx->maps);
            prof_mark(ctx, s_local, 5, 1);
            launches++;
            swap_levels(ctx);
            do_h = do_e = false;
        }
    }
    if (grid.z == 0) { /* an empty part: no sweep blocks */
    } else if (do_h) {
        prof_mark(ctx, s_local, 0, 0);
        launch_chained(ctx, h_sweep_tma<R, STRICT, false>, grid, TmaGeom<R>::H_SMEM, a, ctx->maps);
        prof_mark(ctx, s_local, 0, 1);
        launches++;
    }
    if constexpr (!STRICT) {
        if (ctx->by_class && do_e && ctx->zc_count < 0) {
            launch_e_lists<R, NA>(ctx, s_local, a, ctx->maps);
            launches += split_launches(ctx);
            do_e = false;
        }
    }
    if (do_e && grid.z > 0) {
        prof_mark(ctx, s_local, 1, 0);
        launch_chained(ctx, e_sweep_tma<R, STRICT, NA, kEAll>, grid, TmaGeom<R>::E_SMEM, a, ctx->maps);
        prof_mark(ctx, s_local, 1, 1);
        launches++;
    }
    if (!do_rest) return;
    if constexpr (!STRICT && NA == 0) {
        if (ctx->ion_split) {
            prof_mark(ctx, s_local, 4, 0);
            launch_ions<R>(ctx);
            prof_mark(ctx, s_local, 4, 1);
            launches++;
        }
    }
    if (ctx->probe && !probe_folded(ctx)) {
        prof_mark(ctx, s_local, 2, 0);
        const int threads = (9 + 2 * ctx->probe_n3 + 31) / 32 * 32;
        probe_record_counted<R><<<1, threads, 0, ctx->stream>>>(
            make_fields<R>(ctx), (const R*)ctx->Dp, ctx->probe_d, ctx->probe_cf, (const R*)ctx->r, (const R*)ctx->v, ctx->rv_unit, ctx->nslot, ctx->probe_slot,
            ctx->probe_n3, ctx->probe_rows, ctx->probe_count, kProbeCap, 9 + 2 * ctx->probe_n3);
        prof_mark(ctx, s_local, 2, 1);
        launches++;
    }
    const bool dft_kernels = dft_launched(ctx) > 0;
    if (dft_kernels) prof_mark(ctx, s_local, 3, 0);
    for (size_t q = 0; q < ctx->dft.size(); q++) {
        if (dft_folded(ctx, q)) continue; /* sampled by the E sweep */
        const DftPlane& p = ctx->dft[q];
        const int64_t n = (int64_t)ctx->nx * ctx->ny;
        int blocks = (int)std::min<int64_t>((n + 255) / 256, 148 * 8);
        dft_sample<R><<<blocks, 256, 0, ctx->stream>>>(make_fields<R>(ctx), make_dview<R>(ctx), p.comp, (int64_t)p.z * ctx->plane, ctx->nx, ctx->ny, ctx->nxp,
                                                       p.nfreq, p.cast_f32, ctx->step_in + (size_t)s_local * ctx->step_row,
                                                       p.in_off, p.in_off + 1, p.acc);
        launches++;
    }
    if (dft_kernels) prof_mark(ctx, s_local, 3, 1);
}

typedef void (*step_fn)(php_ctx*, int, int&);
typedef int (*prep_fn)(php_ctx*);

/* Planes per block of he_sweep_tma: a block pays about two planes more than
 * its range (the H of the plane below it, the E above, the first loads), and
 * blocks run in waves of `slots`, the last one partly empty: the range with
 * the shortest waves x (planes + 2). */
static int fused_zstep(int tiles, int nz, int slots)
{
    int best = std::max(1, nz);
    double cost = 1e300;
    for (int n = 1; n <= nz; n++) {
        const int64_t blocks = (int64_t)tiles * ((nz + n - 1) / n);
        const double waves = std::max(1.0, blocks <= 4 * (int64_t)slots ? std::ceil((double)blocks / slots) : (double)blocks / slots + 0.5);
        const double t = waves * (n + 2.0);
        if (t < cost) {
            cost = t;
            best = n;
        }
    }
    return best;
}

/* the TMA sweeps need more than the default 48 KB of dynamic shared memory */
template <typename R, bool STRICT, int NA>
static int prepare_t(php_ctx* ctx)
{
    cudaError_t e = cudaFuncSetAttribute(h_sweep_tma<R, STRICT, false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)TmaGeom<R>::H_SMEM);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(e_sweep_tma<R, STRICT, NA, kEAll>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)TmaGeom<R>::E_SMEM);
    if constexpr (!STRICT)
        if (e == cudaSuccess && (ctx->split || ctx->by_class)) {
            const cudaFuncAttribute at = cudaFuncAttributeMaxDynamicSharedMemorySize;
            e = cudaFuncSetAttribute(e_sweep_tma<R, STRICT, 0, kEPlain>, at, (int)TmaGeom<R>::E_SMEM);
            if constexpr (NA <= 4)
                if (e == cudaSuccess) e = cudaFuncSetAttribute(e_sweep_tma<R, STRICT, NA, kEAtoms>, at, (int)TmaGeom<R>::E_SMEM);
            if (e == cudaSuccess) e = cudaFuncSetAttribute(e_sweep_tma<R, STRICT, NA, kEGeneral>, at, (int)TmaGeom<R>::E_SMEM);
        }
    if constexpr (!STRICT)
        if (e == cudaSuccess && ctx->split)
            e = cudaFuncSetAttribute(interior_sweep_tma<R>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)FusedGeom<R, true>::SMEM);
    if constexpr (!STRICT)
        if (e == cudaSuccess && ctx->split)
            e = cudaFuncSetAttribute(h_sweep_tma<R, STRICT, true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)TmaGeom<R>::H_SMEM);
    if constexpr (!STRICT)
        if (e == cudaSuccess && ctx->fused)
            e = cudaFuncSetAttribute(he_sweep_tma<R, NA>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)FusedGeom<R, false>::SMEM);
    if constexpr (!STRICT) {
        if (e == cudaSuccess && ctx->fused) { /* planes per block */
            int nb = 0;
            e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, he_sweep_tma<R, NA>, kBlockX * kBlockY, FusedGeom<R, false>::SMEM);
            const int tiles = ((ctx->nx + FusedGeom<R, false>::TX - 1) / FusedGeom<R, false>::TX) *
                              ((ctx->ny + FusedGeom<R, false>::TY - 1) / FusedGeom<R, false>::TY);
            ctx->zstep = ctx->d.z_chunk > 0 ? ctx->d.z_chunk : fused_zstep(tiles, ctx->nz, std::max(1, nb) * ctx->num_sms);
        }
    }
    if (e != cudaSuccess) return fail(ctx, PHP_ERR_CUDA, "cudaFuncSetAttribute: %s", cudaGetErrorString(e));
    return PHP_OK;
}

struct StepKernels {
    step_fn launch;
    prep_fn prepare;
};

template <typename R, bool STRICT>
static StepKernels pick_na(int namax)
{
    switch (namax) {
    case 0: return {launch_step_t<R, STRICT, 0>, prepare_t<R, STRICT, 0>};
    case 2: return {launch_step_t<R, STRICT, 2>, prepare_t<R, STRICT, 2>};
    case 4: return {launch_step_t<R, STRICT, 4>, prepare_t<R, STRICT, 4>};
    case 8: return {launch_step_t<R, STRICT, 8>, prepare_t<R, STRICT, 8>};
    case 16: return {launch_step_t<R, STRICT, 16>, prepare_t<R, STRICT, 16>};
    default: return {launch_step_t<R, STRICT, 64>, prepare_t<R, STRICT, 64>};
    }
}

static StepKernels pick_step(const php_ctx* ctx)
{
    /* with the ion pass apart, the E sweep carries no per-atom state */
    const int na = ctx->ion_split ? 0 : ctx->namax_tpl;
    if (ctx->prec == PHP_PREC_FP64_STRICT) return pick_na<double, true>(ctx->namax_tpl);
    if (ctx->prec == PHP_PREC_FP64) return pick_na<double, false>(na);
    return pick_na<float, false>(na);
}

/* ------------------------------------------------------------ tensor maps */

/* d3, s3: size and byte stride of a fourth dimension, all of it in the box
 * (0: three dimensions) */
static int encode_map(php_ctx* ctx, CUtensorMap* m, void* base, CUtensorMapDataType dt, size_t esize, uint64_t d0,
                      uint64_t d1, uint64_t d2, uint32_t b0, uint32_t b1, uint32_t d3 = 0, uint64_t s3 = 0)
{
    static PFN_cuTensorMapEncodeTiled_v12000 encode = nullptr;
    if (!encode) {
        void* fn = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &q) != cudaSuccess || !fn ||
            q != cudaDriverEntryPointSuccess)
            return fail(ctx, PHP_ERR_CUDA, "cuTensorMapEncodeTiled is not available from the driver");
        encode = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(fn);
    }
    const cuuint64_t dims[4] = {d0, d1, d2, d3};
    const cuuint64_t strides[3] = {d0 * esize, d0 * d1 * esize, s3};
    const cuuint32_t box[4] = {b0, b1, 1, d3};
    const cuuint32_t estr[4] = {1, 1, 1, 1};
    CUresult r = encode(m, dt, d3 ? 4 : 3, base, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                        CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return fail(ctx, PHP_ERR_CUDA, "cuTensorMapEncodeTiled failed (%d)", (int)r);
    return PHP_OK;
}

/* Maps of the field arrays (planes -1..nz) with the boxes of
 * php_sweeps_tma.cuh and php_sweep_fused.cuh. */
template <typename R>
static int make_maps(php_ctx* ctx)
{
    using G = TmaGeom<R>;
    using F = FusedGeom<R, false>;
    using I = FusedGeom<R, true>;
    const CUtensorMapDataType dt = sizeof(R) == 8 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT64 : CU_TENSOR_MAP_DATA_TYPE_FLOAT32;
    const uint64_t nxp = ctx->nxp, ny = ctx->ny, nzh = ctx->nz + 2;
    const uint64_t comp = (uint64_t)ctx->plane * nzh * sizeof(R); /* bytes from one component to the next */
    int rc = PHP_OK;
    /* maps of the current buffers, then of the second ones */
    for (int set = 0; set < (ctx->fused || ctx->split ? 2 : 1) && !rc; ++set) {
        TmaMaps& m = set ? ctx->maps_o : ctx->maps;
        void* const* fb = set ? ctx->fo : ctx->f;
        auto map = [&](CUtensorMap& t, int field, uint32_t bx, uint32_t by) {
            if (!rc)
                rc = encode_map(ctx, &t, (char*)fb[field] - (size_t)ctx->plane * sizeof(R), dt, sizeof(R), nxp, ny, nzh, bx, by, 3, comp);
        };
        map(m.e_halo, PHP_EX, G::BX, G::BY);
        map(m.h_own, PHP_HX, G::TX, G::TY);
        map(m.h_halo, PHP_HX, G::BX, G::BY);
        map(m.own, ctx->prec == PHP_PREC_FP64_STRICT ? PHP_DX : PHP_EX, G::TX, G::TY);
        map(m.e_wide, PHP_EX, ctx->split ? I::EX : F::EX, ctx->split ? I::EY : F::EY);
        map(m.h_wide, PHP_HX, ctx->split ? I::HX : F::HX, ctx->split ? I::HY : F::HY);
    }
    return rc;
}

/* --------------------------------------------------------------- creation */

template <typename R>
static int upload_tables(php_ctx* ctx, const std::vector<MatD>& mats, const std::vector<int>& ion_off,
                         const std::vector<double>& ion_coef, const AxisD* axes)
{
    std::vector<MatCoef<R>> mc(mats.size());
    ctx->iso_scale.assign(mats.size(), 0.0);
    ctx->mat_tns.assign(mats.size(), {});
    for (size_t i = 0; i < mats.size(); i++) {
        mc[i] = pack_material<R>(ctx, mats[i], ion_off[i]);
        if (mc[i].flags & kIso) ctx->iso_scale[i] = (double)mc[i].eps_inv[0];
        for (int q = 0; q < 9; q++) {
            ctx->mat_tns[i][q] = (double)mc[i].em[q];
            ctx->mat_tns[i][9 + q] = (double)mc[i].eps_im[q];
        }
        if ((int)i == ctx->atom_id) {
            const unsigned char* p = reinterpret_cast<const unsigned char*>(&mc[i]);
            ctx->atom_mc.assign(p, p + sizeof(MatCoef<R>));
        }
        if ((int)i == ctx->pool_id) {
            const unsigned char* p = reinterpret_cast<const unsigned char*>(&mc[i]);
            ctx->pool_mc.assign(p, p + sizeof(MatCoef<R>));
        }
    }
    int rc = dupload(ctx, &ctx->mc, mc.data(), mc.size() * sizeof(MatCoef<R>));
    if (rc) return rc;
    std::vector<R> ic(ion_coef.size() ? ion_coef.size() : 1);
    for (size_t i = 0; i < ion_coef.size(); i++) ic[i] = (R)ion_coef[i];
    if ((rc = dupload(ctx, &ctx->ion_coef, ic.data(), ic.size() * sizeof(R)))) return rc;
    for (int ax = 0; ax < 3; ax++) {
        const AxisD& A = axes[ax];
        const std::vector<double>* cols[7] = {&A.kappa, &A.b, &A.c, &A.kh, &A.kd, &A.ch, &A.cd};
        for (int q = 0; q < 7; q++) {
            std::vector<R> h(cols[q]->size());
            for (size_t i = 0; i < h.size(); i++) h[i] = (R)(*cols[q])[i];
            if ((rc = dupload(ctx, &ctx->axis_tab[ax][q], h.data(), h.size() * sizeof(R)))) return rc;
        }
    }
    return PHP_OK;
}

/* Page-locked host buffers, kept for reuse by later contexts: freeing one
 * (cudaFreeHost) can wait for the whole device, which would stall the other
 * contexts a serving loop runs beside it. */
static std::mutex g_pinned_mu;
static std::multimap<size_t, void*> g_pinned_free;
static std::map<void*, size_t> g_pinned_size;

static void* pinned_get(size_t bytes)
{
    {
        std::lock_guard<std::mutex> g(g_pinned_mu);
        auto it = g_pinned_free.lower_bound(bytes);
        if (it != g_pinned_free.end() && it->first <= 2 * bytes) {
            void* p = it->second;
            g_pinned_free.erase(it);
            return p;
        }
    }
    void* p = nullptr;
    if (cudaMallocHost(&p, bytes) != cudaSuccess) {
        cudaGetLastError();
        return nullptr;
    }
    std::lock_guard<std::mutex> g(g_pinned_mu);
    g_pinned_size[p] = bytes;
    return p;
}

static void pinned_put(void* p)
{
    if (!p) return;
    std::lock_guard<std::mutex> g(g_pinned_mu);
    g_pinned_free.emplace(g_pinned_size[p], p);
}

/* Host -> device copy through page-locked staging.  A copy from pageable
 * memory is staged by the driver in small synchronous pieces; while other
 * contexts kept the device busy that took up to seconds per context.  Here the
 * pieces are laid one behind the other into two pooled page-locked buffers,
 * one filled while the other's copies run, and the host waits for the device
 * only when both are full: in a process of many streams each wait may last as
 * long as the work that other contexts have queued (16 running jobs, creation
 * with a wait every second upload and between stages 1.6 s, this way 1.2; 0.03
 * with CUDA_DEVICE_MAX_CONNECTIONS=32, which gives more streams a hardware
 * queue of their own).  The source may be freed on return. */
constexpr size_t kUploadChunk = (size_t)4 << 20;
static int upload(php_ctx* ctx, void* dst, const void* src, size_t bytes)
{
    for (size_t off = 0; off < bytes;) {
        if (ctx->up_off == kUploadChunk) { /* to the other buffer, once its copies have left */
            CK(cudaEventRecord(ctx->up_ev[ctx->up_cur], ctx->stream));
            ctx->up_used[ctx->up_cur] = true;
            ctx->up_cur ^= 1;
            ctx->up_off = 0;
            if (ctx->up_used[ctx->up_cur]) CK(cudaEventSynchronize(ctx->up_ev[ctx->up_cur]));
        }
        const int b = ctx->up_cur;
        if (!ctx->up_buf[b]) {
            ctx->up_buf[b] = pinned_get(kUploadChunk);
            if (!ctx->up_buf[b]) return fail(ctx, PHP_ERR_OOM, "page-locked host allocation failed");
        }
        if (!ctx->up_ev[b]) CK(cudaEventCreateWithFlags(&ctx->up_ev[b], cudaEventDisableTiming));
        const size_t n = std::min(kUploadChunk - ctx->up_off, bytes - off);
        char* stage = (char*)ctx->up_buf[b] + ctx->up_off;
        memcpy(stage, (const char*)src + off, n);
        CK(cudaMemcpyAsync((char*)dst + off, stage, n, cudaMemcpyHostToDevice, ctx->stream));
        ctx->up_off = std::min(kUploadChunk, (ctx->up_off + n + 255) / 256 * 256);
        off += n;
    }
    return PHP_OK;
}

/* a buffer and its contents (not cleared first) */
static int dupload(php_ctx* ctx, void** p, const void* src, size_t bytes)
{
    int rc = dalloc(ctx, p, bytes, bytes == 0);
    return rc ? rc : upload(ctx, *p, src, bytes);
}

/* returns the staging buffers to the pool once their copies are done */
static void upload_release(php_ctx* ctx)
{
    if (ctx->up_buf[0] && ctx->stream) cudaStreamSynchronize(ctx->stream);
    for (int b = 0; b < 2; ++b) {
        pinned_put(ctx->up_buf[b]);
        ctx->up_buf[b] = nullptr;
        ctx->up_used[b] = false;
    }
    ctx->up_cur = 0;
    ctx->up_off = 0;
}

static void ctx_free(php_ctx* ctx)
{
    if (!ctx) return;
    for (auto& g : ctx->graphs) cudaGraphExecDestroy(g.second);
    ctx->graphs.clear();
    for (void* p : ctx->allocs) cudaFreeAsync(p, ctx->stream);
    ctx->allocs.clear();
    if (ctx->stream) cudaStreamSynchronize(ctx->stream);
    for (cudaEvent_t e : ctx->prof_ev) cudaEventDestroy(e);
    ctx->prof_ev.clear();
    pinned_put(ctx->host_stage);
    for (int b = 0; b < 2; ++b) {
        pinned_put(ctx->step_in_host[b]);
    }
    for (cudaEvent_t e : ctx->staged)
        if (e) cudaEventDestroy(e);
    upload_release(ctx);
    for (int b = 0; b < 2; ++b)
        if (ctx->up_ev[b]) cudaEventDestroy(ctx->up_ev[b]);
    for (auto& f : ctx->frames) {
        if (f.done) cudaEventDestroy(f.done);
        pinned_put(f.head);
        pinned_put(f.slice);
        pinned_put(f.rows);
    }
    if (ctx->stream) cudaStreamDestroy(ctx->stream);
    if (ctx->setup && ctx->setup != ctx->stream) {
        cudaStreamSynchronize(ctx->setup);
        cudaStreamDestroy(ctx->setup);
    }
    delete ctx;
}

/* (Re)allocates both per-step input buffers for rows of `row` doubles; the
 * stream must be idle.  Replaced device buffers stay allocated until
 * destroy. */
static int alloc_step_inputs(php_ctx* ctx, int row)
{
    ctx->step_row = row;
    for (int b = 0; b < 2; ++b) {
        int rc = dalloc(ctx, (void**)&ctx->step_in_dev[b], (size_t)kMaxChunk * row * sizeof(double));
        if (rc) return rc;
        pinned_put(ctx->step_in_host[b]);
        ctx->step_in_host[b] = (double*)pinned_get((size_t)kMaxChunk * row * sizeof(double));
        if (!ctx->step_in_host[b]) return fail(ctx, PHP_ERR_OOM, "page-locked host allocation failed");
    }
    for (int q = 0; q < 2 * kMaxChunk / ctx->max_chunk; q++)
        if (!ctx->staged[q]) CK(cudaEventCreateWithFlags(&ctx->staged[q], cudaEventDisableTiming));
    ctx->step_in = ctx->step_in_dev[0];
    return PHP_OK;
}

template <typename R, int NP, int S>
static cudaError_t ion_pipe_attr()
{
    return cudaFuncSetAttribute(ion_pipe<R, NP, S>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)IonPipe<R, NP, S>::SMEM);
}

/* bf16 bits of x, rounded to nearest even (finite inputs) */
static uint16_t bf16_bits(float x)
{
    uint32_t u;
    memcpy(&u, &x, 4);
    u += 0x7FFFu + ((u >> 16) & 1u);
    return (uint16_t)(u >> 16);
}

static double bf16_value(uint16_t b)
{
    const uint32_t u = (uint32_t)b << 16;
    float f;
    memcpy(&f, &u, 4);
    return (double)f;
}

/* Many-atom cells (3N >= 24, one DMM shared by every atom material) get the
 * ion pass of php_ions.cuh in the fast FP64 and FP32 paths; PHP_IONS=fused
 * keeps the update inside the E sweep and PHP_IONS=pass moves few-atom cells
 * to the pass too (both for A/B timing). */
static int setup_ion_pass(php_ctx* ctx, const std::vector<MatD>& mats, const std::vector<int>& ion_off, const php_desc& d)
{
    const char* iv = getenv("PHP_IONS");
    const bool force = iv && !strcmp(iv, "pass");
    if ((iv && !strcmp(iv, "fused")) || ctx->prec == PHP_PREC_FP64_STRICT || (ctx->n3max < 24 && !force) ||
        ctx->n3max == 0 || ctx->n3max > 64)
        return PHP_OK;
    int ref = -1;
    for (int i = 0; i < d.num_materials; i++) {
        if (mats[i].natom == 0) continue;
        if (ref < 0) {
            ref = i;
            continue;
        }
        const int N = mats[i].natom;
        if (N != mats[ref].natom || memcmp(d.materials[i].dmm, d.materials[ref].dmm, sizeof(double) * 9 * N * N))
            return PHP_OK; /* several lattices: keep the fused update */
    }
    if (ref < 0) return PHP_OK;
    const int n3 = 3 * mats[ref].natom, np = (n3 + 15) / 16 * 16;
    const double* D = d.materials[ref].dmm;
    const size_t rs = rsize(ctx->prec);
    int rc = dalloc(ctx, &ctx->Pr, 3 * (size_t)ctx->nslot * rs);
    if (rc) return rc;
    if (ctx->prec == PHP_PREC_FP32) {
        /* B operand of D = r DMM^T: row n = output coordinate q, k = p */
        std::vector<uint16_t> img(2 * (size_t)np * np, 0);
        for (int q = 0; q < n3; q++)
            for (int p = 0; p < n3; p++) {
                const double x = D[(size_t)q * n3 + p];
                const uint16_t hi = bf16_bits((float)x);
                const uint16_t lo = bf16_bits((float)(x - bf16_value(hi)));
                const size_t off = umma_kmajor_off(q, p, np) / 2;
                img[off] = hi;
                img[(size_t)np * np + off] = lo;
            }
        if ((rc = dupload(ctx, &ctx->ion_bsplit, img.data(), img.size() * 2))) return rc;
        ctx->ion_tc = true;
    } else {
        std::vector<double> pad((size_t)np * np, 0.0);
        for (int q = 0; q < n3; q++)
            for (int p = 0; p < n3; p++) pad[(size_t)q * np + p] = D[(size_t)q * n3 + p];
        if ((rc = dupload(ctx, &ctx->ion_dmm, pad.data(), pad.size() * sizeof(double)))) return rc;
        /* the same matrix as B fragments of the m8n8k4 FP64 MMA (B[k][n] =
         * DMM[n][k]): lane l of fragment (ks, nt) holds B[4 ks + l % 4][8 nt + l / 4];
         * then the E step, B[t][q] = -QeZM(q, t) (t < 3), and P_ion's B[p][c] =
         * QeZV(c, p) (c < 3), both of the lattice (fdtd.c:3418-3427, 3507-3528) */
        const double* zv = d.materials[ref].qezv;
        const double* zm = d.materials[ref].qezm;
        std::vector<double> frag((size_t)np * np + (size_t)(np / 8) * 32 + (size_t)(np / 4) * 32, 0.0);
        for (int ks = 0; ks < np / 4; ks++)
            for (int nt = 0; nt < np / 8; nt++)
                for (int l = 0; l < 32; l++) {
                    const int q = nt * 8 + l / 4, p = ks * 4 + l % 4;
                    frag[((size_t)ks * (np / 8) + nt) * 32 + l] = (q < n3 && p < n3) ? D[(size_t)q * n3 + p] : 0.0;
                }
        const size_t fe = (size_t)np * np, fp = fe + (size_t)(np / 8) * 32;
        for (int nt = 0; nt < np / 8; nt++)
            for (int l = 0; l < 32; l++) {
                const int t = l % 4, q = nt * 8 + l / 4;
                frag[fe + (size_t)nt * 32 + l] = (t < 3 && q < n3) ? -zm[(q / 3) * 9 + t * 3 + q % 3] : 0.0;
            }
        for (int ks = 0; ks < np / 4; ks++)
            for (int l = 0; l < 32; l++) {
                const int p = ks * 4 + l % 4, c = l / 4;
                frag[fp + (size_t)ks * 32 + l] = (c < 3 && p < n3) ? zv[(p / 3) * 9 + c * 3 + p % 3] : 0.0;
            }
        if ((rc = dupload(ctx, &ctx->ion_dfrag, frag.data(), frag.size() * sizeof(double)))) return rc;
    }
    ctx->ion_np = np;
    ctx->ion_split = true;
    ctx->n3_ion = n3;
    ctx->ion_off_ref = ion_off[ref];
    ctx->ion_pipe = ctx->prec == PHP_PREC_FP32 ? np <= 64 : np <= 48;
    if (ctx->ion_pipe) {
        const CUtensorMapDataType dt = ctx->prec == PHP_PREC_FP32 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_FLOAT64;
        const uint32_t cells = ctx->prec == PHP_PREC_FP32 ? ion_tile<float>() : ion_tile<double>();
        rc = encode_map(ctx, &ctx->ion_maps.r, ctx->r, dt, rs, (uint64_t)ctx->nslot, (uint64_t)n3, 1, cells, (uint32_t)n3);
        if (!rc) rc = encode_map(ctx, &ctx->ion_maps.v, ctx->v, dt, rs, (uint64_t)ctx->nslot, (uint64_t)n3, 1, cells, (uint32_t)n3);
        if (rc) return rc;
        cudaError_t e;
        if (ctx->prec == PHP_PREC_FP32)
            e = np == 16 ? ion_pipe_attr<float, 16, 6>() : np == 32 ? ion_pipe_attr<float, 32, 6>()
              : np == 48 ? ion_pipe_attr<float, 48, 4>() : ion_pipe_attr<float, 64, 3>();
        else
            e = np == 16 ? ion_pipe_attr<double, 16, 6>() : np == 32 ? ion_pipe_attr<double, 32, 6>()
                         : ion_pipe_attr<double, 48, 4>();
        if (e != cudaSuccess) return fail(ctx, PHP_ERR_CUDA, "cudaFuncSetAttribute: %s", cudaGetErrorString(e));
    }
    return PHP_OK;
}

/* E = em D with em a multiple of the identity and no loss (kIso) */
static bool is_iso(const MatD& s)
{
    const double* e = s.eps_inv;
    return s.e_only && !(s.flags & (kLossy | kRotZ | kRotX)) && e[1] == 0.0 && e[2] == 0.0 && e[3] == 0.0 && e[5] == 0.0 &&
           e[6] == 0.0 && e[7] == 0.0 && e[0] == e[4] && e[0] == e[8];
}

/* Sizes from which the interior runs in a launch of its own, and the share of
 * the cells it has to hold.  Gain of a step over the two sweeps, FP64 and FP32,
 * vacuum / two-atom slab / metal tip over a tensor slab, CPML of 8 cells:
 *   96^3  0.86 0.88 0.98, 0.79 0.60 0.82     128^3 1.05 0.98 1.22, 0.96 0.91 0.99
 *   160^3 1.09 1.03 1.18, 1.07 1.09 1.20     192^3 1.11 1.04 1.17, 1.07 1.02 1.14
 *   256 x 256 x 128 1.14 1.05 1.21, 1.07 1.04 1.16
 *   256^3 1.15 1.05 1.19, 1.04 1.04 1.11; with a CPML of 56 cells (a quarter of
 *   the domain inside) 1.11 and 1.06 in vacuum
 * It pays from some 4 M cells on and down to small interiors.  Both lines are
 * well inside: a second field level is memory that the domain could be stepped
 * without, taken where a step gains several per cent by it. */
constexpr int64_t kSplitCells = 8 << 20;
constexpr double kSplitShare = 0.4;

/* Whether the E sweep in place takes a launch per kind of block, where atom
 * blocks want other registers than the rest: from about 74^3 cells (two-atom
 * slab: step of 64^3 21.4 -> 19.7 us FP64, 17.4 -> 17.5 us FP32; 80^3 34.8 ->
 * 32.1, 28.5 -> 25.9; 128^3 112.9 -> 104.5, 78.1 -> 72.0; 192^3 319 -> 296,
 * 215 -> 192). */
constexpr int64_t kByClassCells = 400000;
static bool by_class_size(const php_ctx* ctx)
{
    return (int64_t)ctx->nx * ctx->ny * ctx->nz >= kByClassCells;
}

/* Block classes of a domain in the fast modes, from the one material id (or
 * -1) of each plane and 32 x 8 tile. */
struct BlockPlan {
    int nx = 0, ny = 0, nz = 0, gx = 0, gy = 0;
    const AxisD* axes = nullptr;
    std::vector<int> pml_before[3]; /* CPML cells of the axis below each index */
    const int16_t* uni = nullptr;
    bool on = false;
    bool forced = false;            /* the interior launch whatever the domain's size (PHP_FUSED=2) */
    int atom_id = -1, tns_id = -1;
    std::vector<std::array<int, 3>> src;
    std::vector<char> iso;
    /* the interior launch's blocks (tiles of inner_ty rows), and the planes and
     * 32 x 8 tiles they cover */
    std::vector<int4> inner;
    std::vector<uint8_t> inner_cell;
    int64_t inner_cells = 0;

    /* no CPML cell in [lo, hi) of the axis */
    bool no_pml(int ax, int lo, int hi) const
    {
        const std::vector<int>& n = pml_before[ax];
        const int last = (int)n.size() - 1;
        return n[std::min(hi, last)] == n[std::min(std::max(lo, 0), last)];
    }
    void set_axes(const AxisD* a)
    {
        axes = a;
        for (int ax = 0; ax < 3; ax++) {
            pml_before[ax].assign(1, 0);
            for (int32_t s : a[ax].slot) pml_before[ax].push_back(pml_before[ax].back() + (s >= 0));
        }
    }
    bool source_in(int i0, int j0, int ty, int k0, int k1) const
    {
        for (const auto& q : src)
            if (q[0] >= i0 && q[0] < i0 + kBlockX && q[1] >= j0 && q[1] < j0 + ty && q[2] >= k0 && q[2] < k1) return true;
        return false;
    }
    /* the one material of plane k over the tile's rows j0 .. j0+ty-1, or -1 */
    int tile_id(int bx, int j0, int ty, int k) const
    {
        int id = uni[((size_t)k * gy + j0 / kBlockY) * gx + bx];
        for (int q = j0 / kBlockY + 1; q < std::min(gy, (j0 + ty) / kBlockY) && id >= 0; q++)
            if (uni[((size_t)k * gy + q) * gx + bx] != id) id = -1;
        return id;
    }
    /* class of a block of one material id; inner: no CPML cell and no domain
     * edge cell */
    uint8_t code(int id, bool inner_blk) const
    {
        if (id < 0) return 255;
        if (id < kIsoMats && iso[id]) return (uint8_t)(inner_blk ? id : kPlainCpml + id);
        if (id == atom_id) return (uint8_t)kPlainAtoms;
        return (uint8_t)(id == tns_id ? kPlainTensor : 255);
    }
    bool full(int i0, int j0, int ty) const { return i0 + kBlockX <= nx - 1 && j0 + ty <= ny - 1; } /* all i < nx-1, j < ny-1 */
    /* H sweep: no CPML cell, every cell updated */
    bool h_plain(int bx, int by, int k0, int k1) const
    {
        const int i0 = bx * kBlockX, j0 = by * kBlockY;
        return full(i0, j0, kBlockY) && no_pml(0, i0, i0 + kBlockX) && no_pml(1, j0, j0 + kBlockY) && no_pml(2, k0, k1);
    }
    uint8_t e_class(int bx, int by, int k0, int k1) const
    {
        const int i0 = bx * kBlockX, j0 = by * kBlockY;
        if (source_in(i0, j0, kBlockY, k0, k1)) return 255;
        int id = tile_id(bx, j0, kBlockY, k0);
        for (int k = k0 + 1; k < k1 && id >= 0; k++)
            if (tile_id(bx, j0, kBlockY, k) != id) id = -1;
        return code(id, i0 >= 1 && j0 >= 1 && h_plain(bx, by, k0, k1));
    }
    /* The interior: tiles of ty rows whose cells, and those one below in x and
     * y, lie outside the CPML and off the domain edge; of them, runs of at
     * least min_run planes of one plain or tensor material without a source,
     * outside the z CPML with the plane below (the march starts with that
     * plane's H).  Runs are cut into ranges: a range costs about two planes
     * more than it holds, and the blocks run in waves of `slots`. */
    void find_interior(int ty, int slots, int min_run)
    {
        struct Run { int bx, j0, k0, k1, cls; };
        std::vector<Run> runs;
        inner_cell.assign((size_t)nz * gy * gx, 0);
        std::vector<char> ztop(nz + 1, 0); /* plane k and the one below it outside the CPML */
        for (int k = 0; k < nz; k++) ztop[k] = axes[2].slot[k] < 0 && (k == 0 || axes[2].slot[k - 1] < 0);
        for (int j0 = 0; j0 + ty <= ny - 1; j0 += ty)
            for (int bx = 0; bx < gx; bx++) {
                const int i0 = bx * kBlockX;
                if (i0 < 1 || j0 < 1 || !full(i0, j0, ty) || !no_pml(0, i0 - 1, i0 + kBlockX) || !no_pml(1, j0 - 1, j0 + ty)) continue;
                const bool s = source_in(i0, j0, ty, 0, nz);
                int start = 0, cur = 255;
                for (int k = 0; k <= nz; k++) {
                    int c = 255;
                    if (ztop[k] && !(s && source_in(i0, j0, ty, k, k + 1)))
                        c = code(tile_id(bx, j0, ty, k), true);
                    if (c == kPlainAtoms) c = 255;
                    if (c == cur) continue;
                    if (cur != 255 && k - start >= min_run) runs.push_back({bx, j0, start, k, cur});
                    start = k;
                    cur = c;
                }
            }
        int best = 8;
        double cost = 1e300;
        for (int n = 8; n <= 64; n++) {
            int64_t blocks = 0;
            for (const Run& r : runs) blocks += (r.k1 - r.k0 + n - 1) / n;
            const double w = (double)blocks / slots, waves = w <= 4.0 ? std::ceil(w) : w + 0.5;
            if (waves * (n + 2.0) < cost) {
                cost = waves * (n + 2.0);
                best = n;
            }
        }
        for (const Run& r : runs) {
            const int m = (r.k1 - r.k0 + best - 1) / best;
            for (int q = 0; q < m; q++) {
                const int a = r.k0 + (int)((int64_t)(r.k1 - r.k0) * q / m), b = r.k0 + (int)((int64_t)(r.k1 - r.k0) * (q + 1) / m);
                inner.push_back(make_int4(r.bx | (r.j0 / ty) << 16, a, b, r.cls));
            }
            inner_cells += (int64_t)kBlockX * ty * (r.k1 - r.k0);
            for (int k = r.k0; k < r.k1; k++)
                for (int by = r.j0 / kBlockY; by < (r.j0 + ty) / kBlockY; by++) inner_cell[((size_t)k * gy + by) * gx + r.bx] = 1;
        }
        /* neighbouring tiles of one range run together: their halos meet in L2 */
        std::stable_sort(inner.begin(), inner.end(), [](const int4& a, const int4& b) { return a.y < b.y; });
    }
    /* The blocks of the two sweeps over the rest: planes outside the interior
     * in chunks of at most zc, cut where the class changes once half a chunk
     * is full. */
    void rest(int zc, std::vector<int4>& hj, std::vector<int4>& ej) const
    {
        for (int by = 0; by < gy; by++)
            for (int bx = 0; bx < gx; bx++)
                for (int sweep = 0; sweep < 2; sweep++) {
                    auto cls = [&](int k0, int k1) { return sweep ? (int)e_class(bx, by, k0, k1) : (int)h_plain(bx, by, k0, k1); };
                    for (int k = 0; k < nz;) {
                        if (inner_cell[((size_t)k * gy + by) * gx + bx]) {
                            k++;
                            continue;
                        }
                        int e = k + 1;
                        const int c = cls(k, k + 1);
                        while (e < nz && e - k < zc && !inner_cell[((size_t)e * gy + by) * gx + bx] &&
                               !(2 * (e - k) >= zc && cls(e, e + 1) != c))
                            e++;
                        (sweep ? ej : hj).push_back(make_int4(bx | by << 16, k, e, cls(k, e)));
                        k = e;
                    }
                }
        auto order = [](const int4& a, const int4& b) { return a.y < b.y; };
        std::stable_sort(hj.begin(), hj.end(), order);
        std::stable_sort(ej.begin(), ej.end(), order);
    }
};

/* The plan of a whole domain or a slab: what the classes are chosen from. */
static void plan_classes(const php_desc& d, const std::vector<MatD>& mats, const AxisD* axes, const std::vector<int16_t>& uni,
                         BlockPlan& plan)
{
    const bool strict = d.precision == PHP_PREC_FP64_STRICT;
    plan.nx = d.nx, plan.ny = d.ny, plan.nz = d.nz;
    plan.gx = (d.nx + kBlockX - 1) / kBlockX, plan.gy = (d.ny + kBlockY - 1) / kBlockY;
    plan.set_axes(axes);
    plan.uni = uni.data();
    const char* pv = getenv("PHP_PLAIN");
    const char* tv = getenv("PHP_PLAIN_TENSOR");
    plan.on = !strict && !(pv && !strcmp(pv, "0"));
    for (int s = 0; s < d.num_sources; s++) {
        int c[3], comp;
        if (source_cell(d, d.sources[s], c, comp)) plan.src.push_back({c[0], c[1], c[2]});
    }
    for (const MatD& m : mats) plan.iso.push_back(!strict && is_iso(m));
    /* the lossy or anisotropic material filling the most tiles */
    std::vector<size_t> count(mats.size(), 0);
    if (plan.on && !(tv && !strcmp(tv, "0")))
        for (int16_t id : uni)
            if (id >= 0 && mats[id].e_only && !plan.iso[id]) count[id]++;
    for (size_t id = 0; id < count.size(); id++)
        if (count[id] && (plan.tns_id < 0 || count[id] > count[plan.tns_id])) plan.tns_id = (int)id;
}

/* PHP_FUSED at create: the interior launch at any size ("2"), the one-launch
 * step ("1"), neither (another value); unset: by size and share */
static bool interior_wanted(const php_desc& d)
{
    const char* fv = getenv("PHP_FUSED");
    return d.precision != PHP_PREC_FP64_STRICT && (fv ? !strcmp(fv, "2") : (int64_t)d.nx * d.ny * d.nz >= kSplitCells);
}

/* A list entry holds the tile's x in 16 bits and its y in 15 (int4::x); longer
 * domains keep the grid launches, whose z chunks carry no such bound. */
static bool listable(const BlockPlan& plan) { return plan.gx <= 0xffff && plan.gy <= 0x7fff; }

/* Finds the interior of a whole domain; whether it is worth its launch. */
static bool plan_interior(const php_desc& d, BlockPlan& plan, int sms)
{
    if (!plan.on || !interior_wanted(d)) return false;
    if (!listable(plan)) return false;
    plan.forced = getenv("PHP_FUSED") != nullptr;
    const bool f32 = d.precision == PHP_PREC_FP32;
    plan.find_interior(kBlockY * (f32 ? FusedGeom<float, true>::ROWS : FusedGeom<double, true>::ROWS),
                       sms * (f32 ? PHP_INNER_MINB32 : PHP_INNER_MINB64), plan.forced ? 2 : 8);
    return !plan.inner.empty() && (plan.forced || plan.inner_cells >= kSplitShare * (double)d.nx * d.ny * d.nz);
}

/* Bytes of one field level (E and H), and whether the second one may be had:
 * it makes a step faster and no domain possible, so half of the device's
 * memory has to stay free beside it for the contexts that come after. */
static uint64_t level_bytes(const php_desc& d)
{
    return 6 * (uint64_t)((d.nx + 31) / 32 * 32) * d.ny * (d.nz + 2) * rsize(d.precision);
}
static bool second_buffers_fit(const php_desc& d, uint64_t free_b, uint64_t total_b)
{
    return 2 * level_bytes(d) + total_b / 2 <= free_b;
}
/* What the device's stream-ordered pool holds and no buffer uses (of contexts
 * destroyed, where a release threshold keeps it): free for the next context,
 * though cudaMemGetInfo does not say so. */
static uint64_t pool_reusable(int device)
{
    cudaMemPool_t pool;
    uint64_t reserved = 0, used = 0;
    if (cudaDeviceGetMemPool(&pool, device) != cudaSuccess ||
        cudaMemPoolGetAttribute(pool, cudaMemPoolAttrReservedMemCurrent, &reserved) != cudaSuccess ||
        cudaMemPoolGetAttribute(pool, cudaMemPoolAttrUsedMemCurrent, &used) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    return reserved > used ? reserved - used : 0;
}
constexpr uint64_t kDeviceBytes = (uint64_t)183359 << 20; /* of a B200: the most that cudaMemGetInfo reports */

static int create_impl(const php_desc* desc, php_ctx* ctx)
{
    const php_desc& d = *desc;
    if (d.abi_version != PHP_ABI_VERSION) return fail(ctx, PHP_ERR_INPUT, "abi_version %d, library %d", d.abi_version, PHP_ABI_VERSION);
    if (d.nx < 2 || d.ny < 2 || d.nz < 1) return fail(ctx, PHP_ERR_INPUT, "grid %dx%dx%d too small", d.nx, d.ny, d.nz);
    if (!(d.dt > 0) || !(d.dx > 0) || !(d.dy > 0) || !(d.dz > 0))
        return fail(ctx, PHP_ERR_INPUT, "dt and cell sizes must be positive");
    if (d.precision < 0 || d.precision > 2) return fail(ctx, PHP_ERR_INPUT, "unknown precision %d", d.precision);
    if (d.pml_thickness < 0) return fail(ctx, PHP_ERR_INPUT, "negative pml_thickness");
    if (d.num_materials < 1 || d.num_materials > 256 || !d.materials)
        return fail(ctx, PHP_ERR_INPUT, "num_materials must be 1..256 (got %d)", d.num_materials);
    if (!d.medium) return fail(ctx, PHP_ERR_INPUT, "medium is NULL");
    if (d.num_sources < 0 || (d.num_sources > 0 && !d.sources)) return fail(ctx, PHP_ERR_INPUT, "bad sources");
    ctx->d = d;
    if (ctx->nz_glob == 0) ctx->nz_glob = d.nz;
    ctx->prec = d.precision;
    ctx->nx = d.nx;
    ctx->ny = d.ny;
    ctx->nz = d.nz;
    ctx->nxp = (d.nx + 31) / 32 * 32;
    ctx->L = d.pml_thickness;
    ctx->plane = (int64_t)ctx->nxp * d.ny;
    ctx->ncell_dev = ctx->plane * d.nz;

    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) return fail(ctx, PHP_ERR_NODEVICE, "no CUDA device visible");
    if (d.device < 0 || d.device >= ndev) return fail(ctx, PHP_ERR_INPUT, "device %d not present", d.device);
    CK(cudaSetDevice(d.device));
    CK(cudaDeviceGetAttribute(&ctx->num_sms, cudaDevAttrMultiProcessorCount, d.device));
    {
        int least = 0, greatest = 0;
        CK(cudaDeviceGetStreamPriorityRange(&least, &greatest));
        CK(cudaStreamCreateWithPriority(&ctx->setup, cudaStreamNonBlocking, greatest));
        ctx->stream = ctx->setup;
    }

    /* materials */
    std::vector<MatD> mats(d.num_materials);
    std::vector<int> ion_off(d.num_materials, 0);
    std::vector<double> ion_coef;
    const double ion_scale = ctx->prec == PHP_PREC_FP32 ? kIonScale32 : 1.0;
    ctx->rv_unit = 1.0 / ion_scale;
    for (int i = 0; i < d.num_materials; i++) {
        int rc = derive_material(ctx, i, d.materials[i], mats[i]);
        if (rc) return rc;
        if (mats[i].natom > 0) {
            const int N = mats[i].natom;
            ion_off[i] = (int)ion_coef.size();
            for (int q = 0; q < 9 * N; q++) ion_coef.push_back(d.materials[i].qezv[q] / ion_scale);
            for (int q = 0; q < 9 * N; q++) ion_coef.push_back(d.materials[i].qezm[q] * ion_scale);
            ion_coef.insert(ion_coef.end(), d.materials[i].dmm, d.materials[i].dmm + 9 * N * N);
        }
        ctx->mat_natom.push_back(mats[i].natom);
        ctx->mat_ade.push_back(mats[i].flags & kAde ? 1 : 0);
        ctx->mat_flags.push_back(mats[i].flags);
        ctx->mat_cs.push_back(mats[i].cs);
        ctx->mat_sn.push_back(mats[i].sn);
    }

    /* medium census, slots, device material map */
    const int nx = d.nx, ny = d.ny, nz = d.nz, nxp = ctx->nxp;
    std::vector<uint8_t> mat_dev((size_t)ctx->ncell_dev, 0);
    std::vector<int32_t> slot_dev;
    std::vector<int64_t> slot_cell;
    std::vector<int32_t> slot_n3;
    int n3max = 0;
    std::vector<int64_t> mat_cells(d.num_materials, 0);
    /* per plane and 32 x 8 tile: the one material id of its cells, or -1 */
    const int gx = (nx + kBlockX - 1) / kBlockX, gy = (ny + kBlockY - 1) / kBlockY;
    std::vector<int16_t> uni((size_t)gx * gy * nz, -1);
    const bool strict = ctx->prec == PHP_PREC_FP64_STRICT;
    {
        /* the medium from file order (z fastest) into the device layout (x
         * fastest), with the pool slots of ADE and atom cells in device cell
         * order: z-plane ranges on host threads (a 1024 x 1024 x 512 medium
         * is 537 M strided reads), joined in plane order */
        struct Part {
            std::vector<int64_t> cell;
            std::vector<int32_t> n3;
            std::vector<int64_t> count;
            int n3max = 0;
            bool ade = false, atoms = false;
            int bad = 0, bad_id = 0, bi = 0, bj = 0, bk = 0;
        };
        const int nt = (int)std::max<int64_t>(1, std::min<int64_t>({(int64_t)std::thread::hardware_concurrency(), 32,
                                                                    (int64_t)nz, (int64_t)nx * ny * nz / (1 << 20) + 1}));
        std::vector<Part> parts(nt);
        auto work = [&](int t) {
            Part& P = parts[t];
            P.count.assign(d.num_materials, 0);
            const int k0 = (int)((int64_t)nz * t / nt), k1 = (int)((int64_t)nz * (t + 1) / nt);
            for (int k = k0; k < k1; k++) {
                for (int j = 0; j < ny; j++)
                    for (int i = 0; i < nx; i++) {
                        const int32_t id = d.medium[((size_t)i * ny + j) * nz + k];
                        if (id < 0 || id >= d.num_materials) {
                            P.bad = 1;
                            P.bad_id = id;
                            P.bi = i, P.bj = j, P.bk = k;
                            return;
                        }
                        const int64_t c = ((int64_t)k * ny + j) * nxp + i;
                        mat_dev[c] = (uint8_t)id;
                        P.count[id]++;
                        if (mats[id].slotted(strict)) {
                            P.cell.push_back(c);
                            P.n3.push_back(3 * mats[id].natom);
                            P.n3max = std::max(P.n3max, 3 * mats[id].natom);
                            if (mats[id].flags & kAde) P.ade = true;
                            if (mats[id].flags & kAtoms) P.atoms = true;
                        }
                    }
                for (int by = 0; by < gy && !strict; by++)
                    for (int bx = 0; bx < gx; bx++) {
                        const int i0 = bx * kBlockX, w = std::min(kBlockX, nx - i0), j1 = std::min((by + 1) * kBlockY, ny);
                        const uint8_t* first = &mat_dev[((int64_t)k * ny + by * kBlockY) * nxp + i0];
                        bool same = w < 2 || !memcmp(first, first + 1, w - 1);
                        for (int j = by * kBlockY + 1; j < j1 && same; j++) same = !memcmp(first, first + (int64_t)(j - by * kBlockY) * nxp, w);
                        if (same) uni[((size_t)k * gy + by) * gx + bx] = *first;
                    }
            }
        };
        std::vector<std::thread> th;
        for (int t = 1; t < nt; t++) th.emplace_back(work, t);
        work(0);
        for (auto& x : th) x.join();
        for (const Part& P : parts) /* the first bad id in the reference's plane order */
            if (P.bad)
                return fail(ctx, PHP_ERR_INPUT, "medium id %d at (%d,%d,%d) outside the material table (0..%d)", P.bad_id,
                            P.bi, P.bj, P.bk, d.num_materials - 1);
        size_t total = 0;
        for (const Part& P : parts) total += P.cell.size();
        slot_cell.reserve(total);
        slot_n3.reserve(total);
        for (const Part& P : parts) {
            slot_cell.insert(slot_cell.end(), P.cell.begin(), P.cell.end());
            slot_n3.insert(slot_n3.end(), P.n3.begin(), P.n3.end());
            for (int m = 0; m < d.num_materials; m++) mat_cells[m] += P.count[m];
            n3max = std::max(n3max, P.n3max);
            ctx->any_ade = ctx->any_ade || P.ade;
            ctx->any_atoms = ctx->any_atoms || P.atoms;
        }
    }
    /* pad the pool to a multiple of 32 slots (16-byte rows for the tensor
     * maps of the ion pass); padding slots have no atoms */
    const int64_t nreal = (int64_t)slot_cell.size();
    while (nreal > 0 && slot_cell.size() % 32) {
        slot_cell.push_back(slot_cell.back());
        slot_n3.push_back(0);
    }
    ctx->nslot = (int64_t)slot_cell.size();
    ctx->n3max = n3max;
    {
        int best = -1;
        for (int i = 0; i < d.num_materials; i++)
            if ((mats[i].flags & kAtoms) && mats[i].natom <= 4 && mat_cells[i] > 0 && (best < 0 || mat_cells[i] > mat_cells[best]))
                best = i;
        if (best >= 0) {
            const int N = mats[best].natom, n3 = 3 * N;
            const php_material_desc& M = d.materials[best];
            ctx->ion_k.assign(kIonK, 0.0);
            for (int q = 0; q < 9 * N; q++) {
                ctx->ion_k[q] = M.qezv[q] / ion_scale;
                ctx->ion_k[kIonKM + q] = M.qezm[q] * ion_scale;
            }
            for (int q = 0; q < n3; q++)
                for (int p = 0; p < n3; p++) ctx->ion_k[kIonKD + q * kIonKQ + p] = M.dmm[(size_t)q * n3 + p];
            ctx->ion_k_off = ion_off[best];
            ctx->atom_id = best;
        }
    }
    for (int i = 0; i < d.num_materials; i++)
        if (!strict && mats[i].slotted(false) && !(mats[i].flags & kAtoms) && mat_cells[i] > 0 &&
            (ctx->pool_id < 0 || mat_cells[i] > mat_cells[ctx->pool_id]))
            ctx->pool_id = i;
    const int namax = n3max / 3;
    ctx->namax_tpl = namax == 0 ? 0 : namax <= 2 ? 2 : namax <= 4 ? 4 : namax <= 8 ? 8 : namax <= 16 ? 16 : 64;
    if (namax > 64) return fail(ctx, PHP_ERR_UNSUPPORTED, "natom %d above the supported 64", namax);
    /* the two-atom update holds r, v in registers and indexes its pools with
     * 32-bit offsets (both precisions) */
    if (ctx->namax_tpl == 2 && (uint64_t)ctx->nslot * 6u >= ((uint64_t)1 << 32))
        return fail(ctx, PHP_ERR_UNSUPPORTED, "%lld atom / ADE cells exceed the 2^32-element pools of the two-atom update",
                    (long long)ctx->nslot);

    /* sources */
    if (d.num_sources > kMaxSources) return fail(ctx, PHP_ERR_UNSUPPORTED, "at most %d sources", kMaxSources);
    ctx->src.assign(d.sources, d.sources + d.num_sources);
    for (int s = 0; s < d.num_sources; s++) {
        const php_source_desc& S = d.sources[s];
        int c[3], comp;
        if (!source_cell(d, S, c, comp)) continue;
        ctx->src_cell[ctx->nsrc_active] = ((int64_t)c[2] * ny + c[1]) * nxp + c[0];
        ctx->src_comp[ctx->nsrc_active] = comp;
        ctx->src_active_index.push_back(s);
        ctx->nsrc_active++;
    }

    /* z chunking: long marches while they leave at least 2 waves of 4 blocks on
     * 148 SMs, in the strict mode 4 (its marches are bound by the divisions of
     * a cell, so a longer one saves nothing), and for 8 planes 4.  Step in us
     * with 1, 2, 4, 8 planes per block:
     *   vacuum 80^3    FP64 24.4 22.8 25.7 36.3  FP32 19.8 17.9 20.3 25.4  strict 56.5 61.7 77.5 124
     *   vacuum 128^3   FP64 87.2 73.2 70.6 75.5  FP32 55.8 44.6 41.9 44.7  strict 169 165 177 201
     *   two-atom 128^3 FP64 113 98.2 95.6 97.8   FP32 76.7 66.4 67.1 75.7  strict 254 253 268 306
     *   two-atom 160^3 FP64 209 177 167 171      FP32 143 118 115 124      strict 467 453 462 496
     *   vacuum 192^3   FP64 268 216 195 200      FP32 195 141 124 121      strict 508 472 465 482
     * (within 3 % of the best of the four on cubes of 80 to 192 of vacuum, a
     * two-atom slab or a metal tip, 48^3 and 64^3 within 6 %, 101 x 67 x 53
     * FP32 13 %; with 2 waves throughout the strict mode was up to 10 % off, FP32
     * at 160^3 8 %; with 4 FP64 and FP32 up to 11 % at 80^3) */
    {
        const int tiles = ((nx + kBlockX - 1) / kBlockX) * ((ny + kBlockY - 1) / kBlockY);
        int zc = std::min(ctx->prec == PHP_PREC_FP32 ? 8 : 4, nz);
        while (zc > 1 && (int64_t)tiles * ((nz + zc - 1) / zc) < 148 * 4 * (strict || zc == 8 ? 4 : 2)) zc /= 2;
        ctx->zchunk = d.z_chunk > 0 ? d.z_chunk : zc;
    }
    AxisD axes[3];
    derive_axis(d, nx, d.dx, false, axes[0]);
    derive_axis(d, ny, d.dy, false, axes[1]);
    derive_axis(d, ctx->nz_glob, d.dz, true, axes[2]);
    if (ctx->nz_glob != nz) { /* a z slab: its planes of the global profile */
        AxisD& z = axes[2];
        auto cut = [&](auto& v) { v = std::vector<typename std::decay_t<decltype(v)>::value_type>(
                                      v.begin() + ctx->z_off, v.begin() + ctx->z_off + nz); };
        cut(z.slot); cut(z.kappa); cut(z.b); cut(z.c); cut(z.kh); cut(z.kd); cut(z.ch); cut(z.cd);
    }
    /* block classes of the fast modes */
    BlockPlan plan;
    plan_classes(d, mats, axes, uni, plan);
    ctx->tns_id = plan.tns_id;
    /* the interior in a launch of its own (interior_sweep_tma) */
    if (ctx->z_off == 0 && ctx->nz_glob == nz && ctx->allow_split && plan_interior(d, plan, ctx->num_sms)) {
        size_t free_b = 0, total_b = 0;
        CK(cudaMemGetInfo(&free_b, &total_b));
        free_b += pool_reusable(d.device);
        ctx->split = plan.forced || second_buffers_fit(d, free_b, total_b);
    }

    /* 32-bit cell offsets inside the sweeps */
    if ((int64_t)ctx->plane * (nz + 2) >= ((int64_t)1 << 31))
        return fail(ctx, PHP_ERR_UNSUPPORTED, "grid of %lld padded cells exceeds the 2^31 cell limit of one domain",
                    (long long)ctx->plane * (nz + 2));

    /* allocations */
    const size_t rs = rsize(ctx->prec);
    const size_t field_bytes = (size_t)ctx->plane * (nz + 2) * rs;
    /* the three components of a field in one allocation (TmaMaps); in the fast
     * modes Dp and E hold D */
    auto alloc_field = [&](void** f3) -> int {
        void* p;
        int rc = dalloc(ctx, &p, 3 * field_bytes);
        for (int q = 0; q < 3 && !rc; q++) f3[q] = (char*)p + q * field_bytes + (size_t)ctx->plane * rs; /* plane 0; plane -1 is the low halo */
        return rc;
    };
    for (int f : {PHP_EX, PHP_DX, PHP_HX}) {
        if (!strict && f == PHP_DX) continue;
        int rc = alloc_field(&ctx->f[f]);
        if (rc) return rc;
    }
    const int L = ctx->L;
    const size_t xs = (size_t)nz * ny * 2 * L, ys = (size_t)nz * 2 * L * nxp, zs = (size_t)2 * L * ny * nxp;
    const size_t psz[12] = {xs, xs, ys, ys, zs, zs, xs, xs, ys, ys, zs, zs};
    for (int q = 0; q < 12; q++) {
        int rc = dalloc(ctx, &ctx->psi[q], psz[q] * rs);
        if (rc) return rc;
    }
    /* the one-launch step (he_sweep_tma) on a whole domain in the fast
     * modes, with PHP_FUSED=1 at create: it moves a third fewer field words
     * than the two sweeps but measured slower (all classes in one kernel
     * spill: 256^3 tip 517-680 us FP64 against 495), so the two sweeps, with
     * the interior launch on large domains, are the default */
    {
        const char* fv = getenv("PHP_FUSED");
        ctx->fused = ctx->prec != PHP_PREC_FP64_STRICT && ctx->z_off == 0 && ctx->nz_glob == nz && fv && !strcmp(fv, "1");
        if (ctx->fused) ctx->split = false;
    }
    int rc = dupload(ctx, (void**)&ctx->mat, mat_dev.data(), mat_dev.size());
    if (rc) return rc;
    if (ctx->nslot > 0) {
        slot_dev.assign((size_t)ctx->ncell_dev, -1);
        for (int64_t s = 0; s < nreal; s++) slot_dev[slot_cell[s]] = (int32_t)s;
        if ((rc = dupload(ctx, (void**)&ctx->slot, slot_dev.data(), slot_dev.size() * sizeof(int32_t)))) return rc;
        if ((rc = dupload(ctx, (void**)&ctx->slot_cell, slot_cell.data(), slot_cell.size() * sizeof(int64_t)))) return rc;
        if ((rc = dupload(ctx, (void**)&ctx->slot_n3, slot_n3.data(), slot_n3.size() * sizeof(int32_t)))) return rc;
        std::vector<uint8_t> slot_mat(slot_cell.size(), 0);
        for (int64_t s = 0; s < nreal; s++) slot_mat[s] = mat_dev[slot_cell[s]];
        if ((rc = dupload(ctx, (void**)&ctx->slot_mat, slot_mat.data(), slot_mat.size()))) return rc;
    }
    if (!strict) {
        if (ctx->nslot > 0 && (rc = dalloc(ctx, &ctx->Dp, 3 * (size_t)ctx->nslot * rs))) return rc;
        if (ctx->prec == PHP_PREC_FP32 && ctx->any_atoms && (rc = dalloc(ctx, (void**)&ctx->Dc, (size_t)ctx->nslot * 4))) return rc;
        std::vector<double> dm(9 * mats.size());
        for (size_t i = 0; i < mats.size(); i++) memcpy(&dm[9 * i], mats[i].dm, sizeof(mats[i].dm));
        if ((rc = dupload(ctx, (void**)&ctx->dmat, dm.data(), dm.size() * sizeof(double)))) return rc;
    }
    if (ctx->any_ade) {
        if ((rc = dalloc(ctx, &ctx->P, 3 * (size_t)ctx->nslot * rs))) return rc;
        if ((rc = dalloc(ctx, &ctx->Po, 3 * (size_t)ctx->nslot * rs))) return rc;
    }
    if (ctx->any_atoms) {
        if ((rc = dalloc(ctx, &ctx->r, (size_t)n3max * ctx->nslot * rs))) return rc;
        if ((rc = dalloc(ctx, &ctx->v, (size_t)n3max * ctx->nslot * rs))) return rc;
    }
    if ((rc = setup_ion_pass(ctx, mats, ion_off, d))) return rc;
    /* the second field level, after everything the domain cannot do without;
     * the interior launch's is given up where it does not fit after all (the
     * pools may take more than half of the device, or another context may have
     * been created meanwhile) */
    if (ctx->split || ctx->fused) {
        const size_t held = ctx->allocs.size();
        for (int f : {PHP_EX, PHP_HX})
            if (!rc) rc = alloc_field(&ctx->fo[f]);
        if (!rc && ctx->split && getenv("PHP_TEST_NO_SECOND_LEVEL")) rc = PHP_ERR_OOM; /* failure-path test */
        for (int q = 0; q < 6 && ctx->fused && !rc; q++) rc = dalloc(ctx, &ctx->psio[q], psz[q] * rs);
        if (rc == PHP_ERR_OOM && ctx->split) {
            for (; ctx->allocs.size() > held; ctx->allocs.pop_back()) {
                cudaFreeAsync(ctx->allocs.back(), ctx->stream);
                ctx->bytes -= 3 * field_bytes;
            }
            for (void*& p : ctx->fo) p = nullptr;
            ctx->split = false;
            ctx->err[0] = 0;
            rc = PHP_OK;
        }
        if (rc) return rc;
    }
    if (ctx->ion_split) { /* the atom material whose blocks read their record from the kernel parameters */
        ctx->atom_id = -1;
        for (int i = 0; i < d.num_materials; i++)
            if ((mats[i].flags & kAtoms) && (ctx->atom_id < 0 || mat_cells[i] > mat_cells[ctx->atom_id])) ctx->atom_id = i;
    } else if (!ctx->any_atoms && !strict) {
        /* no atoms: the material that keeps D beside E takes the atom blocks'
         * path, pool state and a record from the parameters.  Step of 192^3,
         * half of it such a material: by the general path FP64 251 us, FP32
         * 163, this one 235 and 153 */
        for (int i = 0; i < d.num_materials; i++)
            if (mats[i].slotted(false) && !(mats[i].flags & kAde) && mat_cells[i] > 0 &&
                (ctx->atom_id < 0 || mat_cells[i] > mat_cells[ctx->atom_id]))
                ctx->atom_id = i;
    }

    if (ctx->prec == PHP_PREC_FP32) rc = upload_tables<float>(ctx, mats, ion_off, ion_coef, axes);
    else rc = upload_tables<double>(ctx, mats, ion_off, ion_coef, axes);
    if (rc) return rc;

    /* plain blocks of the fused sweep: a 32 x 8 tile and z chunk of cells of
     * one plain isotropic material (id < kIsoMats), none in the CPML, none
     * on the domain's x/y edge, no source.  The sweep updates them without
     * the per-cell material, CPML and source handling; PHP_PLAIN=0 turns it
     * off (A/B timing and tests).  Blocks without a source of the one lossy
     * or anisotropic material (no ADE, no ions) that fills the most blocks
     * take its coefficients from the kernel parameters (kPlainTensor;
     * PHP_PLAIN_TENSOR=0 turns that class off), and so do blocks of the
     * few-atom material whose ions the sweep updates (kPlainAtoms;
     * PHP_PLAIN_ATOMS=0). */
    {
        const int gz = (nz + ctx->zchunk - 1) / ctx->zchunk;
        std::vector<uint8_t> pm((size_t)gx * gy * gz, 255), ph(pm.size(), 0);
        size_t nplain = 0, nplain_h = 0;
        /* blocks of one atom material: the fused sweep updates its ions (two
         * or four atoms), or the ion pass runs apart */
        const char* av = getenv("PHP_PLAIN_ATOMS");
        if (!(av && !strcmp(av, "0")) && ctx->atom_id >= 0 && (ctx->ion_split || ctx->namax_tpl <= 4) &&
            !(ctx->mat_flags[ctx->atom_id] & kAde) && ctx->atom_mc.size() > 0)
            plan.atom_id = ctx->atom_id;
        for (int bz = 0; bz < gz && plan.on; bz++)
            for (int by = 0; by < gy; by++)
                for (int bx = 0; bx < gx; bx++) {
                    const int k0 = bz * ctx->zchunk, k1 = std::min(k0 + ctx->zchunk, nz);
                    const size_t b = ((size_t)bz * gy + by) * gx + bx;
                    ph[b] = plan.h_plain(bx, by, k0, k1);
                    nplain_h += ph[b];
                    pm[b] = plan.e_class(bx, by, k0, k1);
                    nplain += pm[b] != 255;
                }
        ctx->atom_blocks = plan.atom_id >= 0;
        if (ctx->fused) {
            /* the one-launch step's classes, per plane and tile of its height;
             * its H part also computes the cells one below the tile in x and y */
            const int ty = kBlockY * (ctx->prec == PHP_PREC_FP32 ? FusedGeom<float, false>::ROWS : FusedGeom<double, false>::ROWS);
            const int fy = (ny + ty - 1) / ty;
            std::vector<uint16_t> pc((size_t)gx * fy * nz, 255);
            for (int by = 0; by < fy && plan.on; by++)
                for (int bx = 0; bx < gx; bx++) {
                    const int i0 = bx * kBlockX, j0 = by * ty;
                    const bool full = i0 + kBlockX <= nx - 1 && j0 + ty <= ny - 1;
                    const bool inner = full && i0 >= 1 && j0 >= 1 && plan.no_pml(0, i0, i0 + kBlockX) && plan.no_pml(1, j0, j0 + ty);
                    const bool ring = full && plan.no_pml(0, i0 - 1, i0 + kBlockX) && plan.no_pml(1, j0 - 1, j0 + ty);
                    const bool src = plan.source_in(i0, j0, ty, 0, nz);
                    for (int k = 0; k < nz; k++) {
                        const bool zfree = axes[2].slot[k] < 0;
                        const int id = src && plan.source_in(i0, j0, ty, k, k + 1) ? -1 : plan.tile_id(bx, j0, ty, k);
                        pc[((size_t)k * fy + by) * gx + bx] = (uint16_t)(plan.code(id, inner && zfree) | (ring && zfree ? kHPlain : 0u));
                    }
                }
            if ((rc = dupload(ctx, (void**)&ctx->pcls, pc.data(), pc.size() * sizeof(uint16_t)))) return rc;
        }
        ctx->by_class = !ctx->split && !ctx->fused && plan.on && plan.atom_id >= 0 && by_class_size(ctx) && listable(plan);
        if (ctx->split || ctx->by_class) {
            ctx->max_chunk = kListChunk;
            std::vector<int4> hj, ej_all;
            if (ctx->split) {
                plan.rest(ctx->prec == PHP_PREC_FP32 ? 8 : 4, hj, ej_all);
            } else {
                for (int bz = 0; bz < gz; bz++)
                    for (int by = 0; by < gy; by++)
                        for (int bx = 0; bx < gx; bx++)
                            ej_all.push_back(make_int4(bx | by << 16, bz * ctx->zchunk, std::min((bz + 1) * ctx->zchunk, nz),
                                                       pm[((size_t)bz * gy + by) * gx + bx]));
            }
            std::vector<int4> ej[3];
            for (const int4& e : ej_all) ej[e.w == 255 ? 2 : e.w == kPlainAtoms ? 1 : 0].push_back(e);
            if (!ctx->split) plan.inner.clear(); /* found, but too small a share or no memory */
            const std::vector<int4>* jobs[5] = {&plan.inner, &hj, &ej[0], &ej[1], &ej[2]};
            for (int q = 0; q < 5; q++) {
                ctx->nlist[q] = (int)jobs[q]->size();
                if (jobs[q]->empty()) continue;
                if ((rc = dupload(ctx, (void**)&ctx->lists[q], jobs[q]->data(), jobs[q]->size() * sizeof(int4)))) return rc;
            }
        }
        for (size_t b = 0; b < pm.size(); b++) {
            const int c = pm[b] == 255 ? 4 : pm[b] == kPlainAtoms ? 3 : pm[b] == kPlainTensor ? 2
                        : pm[b] >= kPlainCpml ? 1 : 0;
            ctx->census[c]++;
            ctx->census[ph[b] ? 5 : 6]++;
        }
        ctx->census[7] = (int64_t)pm.size();
        if (nplain) {
            if ((rc = dupload(ctx, (void**)&ctx->plain_blk, pm.data(), pm.size()))) return rc;
        }
        if (nplain_h) {
            if ((rc = dupload(ctx, (void**)&ctx->plain_h, ph.data(), ph.size()))) return rc;
        }
        ctx->khp[0] = d.dt / (d.mu0 * d.dx * 1.0);
        ctx->khp[1] = d.dt / (d.mu0 * d.dy * 1.0);
        ctx->khp[2] = d.dt / (d.mu0 * d.dz * 1.0);
        ctx->kdp[0] = d.dt / (d.dx * 1.0);
        ctx->kdp[1] = d.dt / (d.dy * 1.0);
        ctx->kdp[2] = d.dt / (d.dz * 1.0);
    }

    if (const char* st = getenv("PHP_TEST_STALL_WAIT")) ctx->stall_test = !strcmp(st, "1");
    if (const char* dv = getenv("PHP_DFT_FOLD")) ctx->dft_fold = strcmp(dv, "0") != 0;
    if (const char* pv = getenv("PHP_PROBE_FOLD")) ctx->probe_fold = strcmp(pv, "0") != 0;
    /* sweep kernels: the TMA plane pipeline */
    if ((rc = dalloc(ctx, (void**)&ctx->err_flag, sizeof(int32_t)))) return rc;
    rc = ctx->prec == PHP_PREC_FP32 ? make_maps<float>(ctx) : make_maps<double>(ctx);
    if (!rc) rc = pick_step(ctx).prepare(ctx);
    if (rc) return rc;

    /* per-step inputs, scratch, staging */
    ctx->probe_off = ctx->nsrc_active;
    if ((rc = alloc_step_inputs(ctx, ctx->probe_off + 1))) return rc;
    if ((rc = dalloc(ctx, (void**)&ctx->src_acc, 3 * kMaxSources * sizeof(double)))) return rc;
    const size_t maxplane = std::max({(size_t)nx * ny, (size_t)ny * nz, (size_t)nx * nz});
    ctx->scratch_bytes = std::max(maxplane * sizeof(double), (size_t)4096 * sizeof(DiagPartial));
    if ((rc = dalloc(ctx, &ctx->scratch, ctx->scratch_bytes))) return rc;
    ctx->host_stage_bytes = ctx->scratch_bytes;
    ctx->host_stage = pinned_get(ctx->host_stage_bytes);
    if (!ctx->host_stage) return fail(ctx, PHP_ERR_OOM, "page-locked host allocation failed");
    CK(cudaStreamSynchronize(ctx->stream));
    upload_release(ctx);
    /* hand over to the context's stream (everything above is complete) */
    cudaStream_t work = nullptr;
    CK(cudaStreamCreateWithFlags(&work, cudaStreamNonBlocking));
    ctx->stream = work;
    cudaStreamDestroy(ctx->setup);
    ctx->setup = nullptr;
    return PHP_OK;
}

/* Whether php_create takes the interior launch for a description where memory
 * allows, as create_impl finds it. */
static bool interior_expected(const php_desc& d, const std::vector<MatD>& mats)
{
    if (!interior_wanted(d)) return false;
    const int gx = (d.nx + kBlockX - 1) / kBlockX, gy = (d.ny + kBlockY - 1) / kBlockY;
    std::vector<int16_t> col((size_t)gx * gy * d.nz, -2), uni(col.size()); /* [tile][plane], -2: none seen */
    for (int i = 0; i < d.nx; i++)
        for (int j = 0; j < d.ny; j++) {
            const int32_t* m = d.medium + ((size_t)i * d.ny + j) * d.nz;
            int16_t* u = &col[((size_t)(j / kBlockY) * gx + i / kBlockX) * d.nz];
            for (int k = 0; k < d.nz; k++) u[k] = u[k] == -2 || u[k] == m[k] ? (int16_t)m[k] : (int16_t)-1;
        }
    for (size_t t = 0; t < (size_t)gx * gy; t++)
        for (int k = 0; k < d.nz; k++) uni[(size_t)k * gx * gy + t] = col[t * d.nz + k];
    AxisD axes[3];
    derive_axis(d, d.nx, d.dx, false, axes[0]);
    derive_axis(d, d.ny, d.dy, false, axes[1]);
    derive_axis(d, d.nz, d.dz, true, axes[2]);
    BlockPlan plan;
    plan_classes(d, mats, axes, uni, plan);
    return plan_interior(d, plan, 148) && (plan.forced || second_buffers_fit(d, kDeviceBytes, kDeviceBytes));
}

/* Device bytes php_create will allocate for a description (the buffers of
 * create_impl, without DFT planes or the probe ring), and what the interior
 * launch's second buffers may add; no device needed. */
static int estimate_bytes(const php_desc& d, uint64_t* out, uint64_t* more)
{
    if (d.nx < 2 || d.ny < 2 || d.nz < 1 || d.num_materials < 1 || !d.materials || !d.medium || d.pml_thickness < 0 ||
        d.precision < 0 || d.precision > 2)
        return PHP_ERR_INPUT;
    const uint64_t rs = d.precision == PHP_PREC_FP32 ? 4 : 8;
    const bool strict = d.precision == PHP_PREC_FP64_STRICT;
    const uint64_t nxp = (uint64_t)(d.nx + 31) / 32 * 32, plane = nxp * d.ny, ncell = plane * d.nz;
    std::vector<int> n3(d.num_materials, 0);
    std::vector<char> slotted(d.num_materials, 0);
    std::vector<MatD> mats(d.num_materials);
    bool any_ade = false, any_atoms = false, usable = true; /* php_create refuses what is not */
    for (int m = 0; m < d.num_materials; m++) {
        n3[m] = 3 * std::max(0, (int)d.materials[m].natom);
        slotted[m] = d.materials[m].use_ade == 1 || d.materials[m].natom > 0;
        if (!strict) {
            php_ctx probe;
            probe.d = d;
            usable = derive_material(&probe, m, d.materials[m], mats[m]) == PHP_OK && usable;
            /* a material that keeps D although it has no ADE and no atoms */
            if (!slotted[m]) slotted[m] = usable && mats[m].slotted(false);
        }
    }
    uint64_t nslot = 0;
    int n3max = 0;
    const size_t V = (size_t)d.nx * d.ny * d.nz;
    for (size_t c = 0; c < V; c++) {
        const int id = d.medium[c];
        if (id < 0 || id >= d.num_materials) return PHP_ERR_INPUT;
        if (slotted[id]) {
            nslot++;
            n3max = std::max(n3max, n3[id]);
            if (d.materials[id].use_ade == 1) any_ade = true;
            if (d.materials[id].natom > 0) any_atoms = true;
        }
    }
    const uint64_t L = d.pml_thickness;
    uint64_t b = (strict ? 9 : 6) * plane * (d.nz + 2) * rs;
    const uint64_t tiles = nxp / kBlockX * (((uint64_t)d.ny + kBlockY - 1) / kBlockY);
    if (!strict) b += 16 * tiles * d.nz; /* class launches: their lists */
    /* second E and H buffers of the interior launch, its list and the sweeps' */
    *more = usable && d.num_materials <= 256 && interior_expected(d, mats) ? level_bytes(d) + 32 * tiles * d.nz : 0;
    b += 4 * ((uint64_t)d.nz * d.ny * 2 * L + (uint64_t)d.nz * 2 * L * nxp + 2 * L * d.ny * nxp) * rs;
    const char* fv = getenv("PHP_FUSED");
    if (d.precision != PHP_PREC_FP64_STRICT && fv && !strcmp(fv, "1")) { /* second E, H and H CPML buffers */
        b += 6 * plane * (d.nz + 2) * rs;
        b += 2 * ((uint64_t)d.nz * d.ny * 2 * L + (uint64_t)d.nz * 2 * L * nxp + 2 * L * d.ny * nxp) * rs;
    }
    b += ncell; /* material ids */
    if (nslot) b += ncell * 4 + nslot * 13;
    if (nslot && !strict) b += 3 * nslot * rs + (any_atoms && rs == 4 ? 4 * nslot : 0);
    if (any_ade) b += 6 * nslot * rs;
    if (any_atoms) b += 2 * (uint64_t)n3max * nslot * rs;
    if (n3max >= 24 && d.precision != PHP_PREC_FP64_STRICT) b += 3 * nslot * rs + 64 * 64 * 8; /* ion pass */
    b += 7 * (uint64_t)(d.nx + d.ny + d.nz) * (rs + 4);
    b += 2 * (uint64_t)kMaxChunk * (std::max(1, (int)d.num_sources) + 8) * 8;
    b += std::max((uint64_t)std::max({(uint64_t)d.nx * d.ny, (uint64_t)d.ny * d.nz, (uint64_t)d.nx * d.nz}) * 8,
                  (uint64_t)4096 * sizeof(DiagPartial));
    b += (uint64_t)d.num_materials * 512 + (1u << 20); /* tables, pool granularity */
    *out = b;
    return PHP_OK;
}

/* ---------------------------------------------------------------- stepping */

static int record_graph(php_ctx* ctx, int n, int b, cudaGraphExec_t* out);

/* graph of n steps reading per-step input buffer b; a new chunk length
 * records the graphs of both buffers at once, so that a repeated step
 * pattern instantiates nothing after its first pass */
static int graph_key(const php_ctx* ctx, int n, int b) { return 4 * n + 2 * ctx->level + b; }

static int ensure_graph(php_ctx* ctx, int n, int b, cudaGraphExec_t* out)
{
    auto it = ctx->graphs.find(graph_key(ctx, n, b));
    if (it != ctx->graphs.end()) {
        *out = it->second;
        return PHP_OK;
    }
    cudaGraphExec_t other;
    int rc = record_graph(ctx, n, b ^ 1, &other);
    if (rc) return rc;
    return record_graph(ctx, n, b, out);
}

/* The graph of n steps from the current level; each one-launch step of the
 * recording swaps the levels on the host as the step will on the device, so
 * the recording ends by restoring the level it started from. */
static int record_graph(php_ctx* ctx, int n, int b, cudaGraphExec_t* out)
{
    const int key = graph_key(ctx, n, b);
    const int level = ctx->level;
    ctx->step_in = ctx->step_in_dev[b];
    step_fn fn = pick_step(ctx).launch;
    cudaGraph_t g = nullptr;
    CK(cudaStreamBeginCapture(ctx->stream, cudaStreamCaptureModeThreadLocal));
    ctx->chain = 0;
    int launches = 0;
    for (int s = 0; s < n; s++) fn(ctx, s, launches);
    if (ctx->level != level) swap_levels(ctx);
    cudaError_t le = cudaGetLastError();
    cudaError_t ce = cudaStreamEndCapture(ctx->stream, &g);
    ctx->chain = -1;
    if (le != cudaSuccess) {
        if (g) cudaGraphDestroy(g);
        return fail(ctx, PHP_ERR_CUDA, "kernel launch during capture failed: %s", cudaGetErrorString(le));
    }
    if (ce != cudaSuccess) return fail(ctx, PHP_ERR_CUDA, "graph capture failed: %s", cudaGetErrorString(ce));
    cudaGraphExec_t ge = nullptr;
    cudaError_t ie = cudaGraphInstantiate(&ge, g, 0);
    cudaGraphDestroy(g);
    if (ie != cudaSuccess) return fail(ctx, PHP_ERR_CUDA, "graph instantiate failed: %s", cudaGetErrorString(ie));
    ctx->graphs[key] = ge;
    *out = ge;
    return PHP_OK;
}

static void drop_graphs(php_ctx* ctx)
{
    if (ctx->stream) cudaStreamSynchronize(ctx->stream);
    for (auto& g : ctx->graphs) cudaGraphExecDestroy(g.second);
    ctx->graphs.clear();
}

/* The caller holds the addresses of planes, or orders the sweeps itself: the
 * context's E and H stay where they are from now on (the buffers current at
 * this point), stepped by the two sweeps. */
static void step_in_place(php_ctx* ctx)
{
    if (!ctx->split) return;
    drop_graphs(ctx);
    ctx->split = false;
}

static int relayout_step_inputs(php_ctx* ctx)
{
    int row = ctx->probe_off + 1;
    for (auto& p : ctx->dft) {
        p.in_off = row;
        row += 1 + 2 * p.nfreq;
    }
    if (row == ctx->step_row) return PHP_OK;
    drop_graphs(ctx);
    return alloc_step_inputs(ctx, row);
}

template <typename R>
static void launch_gather_plane(php_ctx* ctx, int comp, int axis, int pos, bool f32, void* out)
{
    const Fields<R> f = make_fields<R>(ctx);
    const DView<R> dv = make_dview<R>(ctx);
    if (f32) gather_plane<R, float><<<296, 256, 0, ctx->stream>>>(f, dv, comp, axis, pos, ctx->nx, ctx->ny, ctx->nz, ctx->nxp, (float*)out);
    else gather_plane<R, double><<<296, 256, 0, ctx->stream>>>(f, dv, comp, axis, pos, ctx->nx, ctx->ny, ctx->nz, ctx->nxp, (double*)out);
}

/* Fills pinned buffer b with the per-step inputs (source values, DFT
 * sample flags and phasors) of steps t .. t+n-1 and copies it to device
 * buffer b on the stream. */
static int stage_step_inputs(php_ctx* ctx, int n, int b)
{
    const double dt = ctx->d.dt;
    /* the last copy out of this page-locked slot must be done; the chunks in
     * between keep the GPU busy meanwhile */
    const int slots = 2 * kMaxChunk / ctx->max_chunk, slot = ctx->chunk_no % slots;
    CK(cudaEventSynchronize(ctx->staged[slot]));
    double* h = ctx->step_in_host[slot * 2 / slots] + (size_t)(slot % (slots / 2)) * ctx->max_chunk * ctx->step_row;
    for (int s = 0; s < n; s++) {
        const int t = ctx->t + s;
        double* row = h + (size_t)s * ctx->step_row;
        const double current_time = t * dt; /* fdtd.c:3117 */
        for (int q = 0; q < ctx->nsrc_active; q++)
            row[q] = source_value(&ctx->src[ctx->src_active_index[q]], current_time);
        row[ctx->probe_off] = t - ctx->probe_t0;
        for (auto& p : ctx->dft) {
            const bool take = t >= p.first && ((t - p.first) % p.interval) == 0;
            row[p.in_off] = take ? 1.0 : 0.0;
            for (int f = 0; f < p.nfreq; f++) {
                const double ph = -2.0 * M_PI * p.freq[f] * (t * dt);
                row[p.in_off + 1 + 2 * f] = take ? cos(ph) : 0.0;
                row[p.in_off + 2 + 2 * f] = take ? sin(ph) : 0.0;
            }
            if (take) p.nsamples++;
        }
    }
    /* the device buffer b was last read by the work of two chunks back,
     * which precedes this copy on the stream */
    CK(cudaMemcpyAsync(ctx->step_in_dev[b], h, (size_t)n * ctx->step_row * sizeof(double), cudaMemcpyHostToDevice,
                       ctx->stream));
    CK(cudaEventRecord(ctx->staged[slot], ctx->stream));
    return PHP_OK;
}

/* ------------------------------------------------------------- public API */

/* frame gathers (php_frame_begin) */

static int64_t point_index(const php_ctx* ctx, const int32_t* p)
{
    return ((int64_t)p[2] * ctx->ny + p[1]) * ctx->nxp + p[0];
}

template <typename R>
static void launch_frame_gather(php_ctx* ctx, const DiagPartial* parts, int nparts, int has_point, int64_t pc, int64_t cc,
                                const double* rows, int64_t nrows, int row_len, double* rows_out, FrameHead* head)
{
    frame_gather<R><<<1, 256, 0, ctx->stream>>>(make_fields<R>(ctx), make_dview<R>(ctx), ctx->mat, ctx->slot, (const MatCoef<R>*)ctx->mc, (const R*)ctx->r,
                                                 (const R*)ctx->v, ctx->rv_unit, ctx->nslot, ctx->nx, ctx->ny, ctx->nz, ctx->nxp,
                                                 ctx->n3max, parts, nparts, has_point, pc, cc,
                                                 ctx->probe ? ctx->probe_count : nullptr, rows, nrows, row_len, rows_out,
                                                 ctx->err_flag, head);
}

extern "C" {

int php_create(const php_desc* desc, php_ctx** out)
{
    return php_create_buffers(desc, true, out);
}

int php_create_buffers(const php_desc* desc, bool split, php_ctx** out)
{
    if (!desc || !out) return fail(nullptr, PHP_ERR_INPUT, "null argument");
    *out = nullptr;
    php_ctx* ctx = new (std::nothrow) php_ctx();
    if (!ctx) return fail(nullptr, PHP_ERR_OOM, "host allocation failed");
    ctx->allow_split = split;
    int rc = create_impl(desc, ctx);
    if (rc) {
        g_create_error = ctx->err;
        ctx_free(ctx);
        return rc;
    }
    *out = ctx;
    return PHP_OK;
}

int php_create_slab(const php_desc* desc, int32_t z0, int32_t nz_local, php_ctx** out)
{
    if (!desc || !out) return fail(nullptr, PHP_ERR_INPUT, "null argument");
    *out = nullptr;
    if (!desc->medium || desc->nz < 1 || z0 < 0 || nz_local < 1 || z0 + nz_local > desc->nz)
        return fail(nullptr, PHP_ERR_INPUT, "slab [%d, %d) outside the grid of %d planes", z0, z0 + nz_local, desc->nz);
    if (desc->num_sources < 0 || (desc->num_sources > 0 && !desc->sources))
        return fail(nullptr, PHP_ERR_INPUT, "bad sources");
    /* the slab's medium and sources in local z */
    const size_t nx = desc->nx, ny = desc->ny, nzg = desc->nz;
    std::vector<int32_t> med(nx * ny * (size_t)nz_local);
    for (size_t i = 0; i < nx; i++)
        for (size_t j = 0; j < ny; j++)
            memcpy(&med[(i * ny + j) * nz_local], desc->medium + (i * ny + j) * nzg + z0, sizeof(int32_t) * nz_local);
    std::vector<php_source_desc> src(desc->sources, desc->sources + std::max(0, desc->num_sources));
    for (auto& x : src) x.z -= z0; /* sources outside the slab are skipped like those outside the grid */
    php_desc d = *desc;
    d.nz = nz_local;
    d.medium = med.data();
    d.sources = src.empty() ? nullptr : src.data();
    php_ctx* ctx = new (std::nothrow) php_ctx();
    if (!ctx) return fail(nullptr, PHP_ERR_OOM, "host allocation failed");
    ctx->z_off = z0;
    ctx->nz_glob = desc->nz;
    int rc = create_impl(&d, ctx);
    if (rc) {
        g_create_error = ctx->err;
        ctx_free(ctx);
        return rc;
    }
    ctx->d.medium = nullptr; /* the local copies go out of scope */
    ctx->d.sources = nullptr;
    *out = ctx;
    return PHP_OK;
}

int php_halo_planes(php_ctx* ctx, int32_t which, void** ptrs, uint64_t* plane_bytes)
{
    if (!ctx || !ptrs || which < 0 || which > 3) return PHP_ERR_INPUT;
    step_in_place(ctx);
    /* E plane 0 | E halo above | H top plane | H halo below */
    const int64_t plane_idx[4] = {0, ctx->nz, ctx->nz - 1, -1};
    const int first[4] = {PHP_EX, PHP_EX, PHP_HX, PHP_HX};
    const size_t rs = rsize(ctx->prec);
    for (int q = 0; q < 3; q++)
        ptrs[q] = (char*)ctx->f[first[which] + q] + plane_idx[which] * ctx->plane * (int64_t)rs;
    if (plane_bytes) *plane_bytes = (uint64_t)ctx->plane * rs;
    return PHP_OK;
}

int php_step_half(php_ctx* ctx, int32_t half)
{
    if (!ctx || (half != 0 && half != 1)) return PHP_ERR_INPUT;
    step_in_place(ctx);
    ctx->last_launches = 0;
    int launches = 0;
    const int b = ctx->chunk_no & 1;
    if (half == 1) {
        int rc = stage_step_inputs(ctx, 1, b);
        if (rc) return rc;
    }
    ctx->step_in = ctx->step_in_dev[b];
    ctx->step_part = half == 0 ? 1 : 6;
    pick_step(ctx).launch(ctx, 0, launches);
    ctx->step_part = 7;
    CK(cudaGetLastError());
    if (half == 1) {
        ctx->chunk_no++;
        ctx->t++;
    }
    ctx->last_launches = launches;
    return PHP_OK;
}

int php_step_part(php_ctx* ctx, int32_t part, void* stream)
{
    if (!ctx || part < 0 || part > 4) return PHP_ERR_INPUT;
    step_in_place(ctx);
    ctx->last_launches = 0;
    int launches = 0;
    const int b = ctx->chunk_no & 1;
    const int nchunk = (ctx->nz + ctx->zchunk - 1) / ctx->zchunk;
    cudaStream_t own = ctx->stream;
    if (stream) ctx->stream = static_cast<cudaStream_t>(stream);
    int rc = PHP_OK;
    if (part <= 1 && !ctx->part_staged) { /* the first H part stages the step's source values and DFT phasors */
        rc = stage_step_inputs(ctx, 1, b);
        ctx->part_staged = rc == PHP_OK;
    }
    if (rc == PHP_OK && part != 0 && !ctx->part_staged)
        rc = fail(ctx, PHP_ERR_STATE, "php_step_part %d before an H part (0 or 1) of the step", part);
    if (rc == PHP_OK) {
        ctx->step_in = ctx->step_in_dev[b];
        /* H: part 0 the top chunk, part 1 the others; E: part 2 the bottom
         * chunk, part 3 the others; part 4 the rest of the step */
        static const int kPartBits[5] = {1, 1, 2, 2, 4};
        ctx->step_part = kPartBits[part];
        ctx->zc_first = part == 0 ? nchunk - 1 : part == 3 ? 1 : 0;
        ctx->zc_count = part == 0 || part == 2 ? 1 : part == 4 ? 0 : nchunk - 1;
        pick_step(ctx).launch(ctx, 0, launches);
        ctx->step_part = 7;
        ctx->zc_first = 0;
        ctx->zc_count = -1;
        const cudaError_t e = cudaGetLastError();
        if (e != cudaSuccess) rc = fail(ctx, PHP_ERR_CUDA, "%s", cudaGetErrorString(e));
    }
    ctx->stream = own;
    if (rc == PHP_OK && part == 4) {
        ctx->part_staged = false;
        ctx->chunk_no++;
        ctx->t++;
    }
    ctx->last_launches = launches;
    return rc;
}

int php_destroy(php_ctx* ctx)
{
    ctx_free(ctx);
    return PHP_OK;
}

const char* php_last_error(const php_ctx* ctx)
{
    if (!ctx) return g_create_error.c_str();
    return ctx->err;
}

int php_step(php_ctx* ctx, int32_t nsteps)
{
    if (!ctx) return PHP_ERR_INPUT;
    if (nsteps < 0) return fail(ctx, PHP_ERR_INPUT, "negative step count");
    ctx->last_launches = 0;
    while (nsteps > 0) {
        const int n = std::min(nsteps, ctx->max_chunk);
        const int b = ctx->chunk_no & 1;
        int rc = stage_step_inputs(ctx, n, b);
        if (rc) return rc;
        cudaGraphExec_t g;
        rc = ensure_graph(ctx, n, b, &g);
        if (rc) return rc;
        CK(cudaGraphLaunch(g, ctx->stream));
        if ((ctx->fused || ctx->split) && (n & 1)) swap_levels(ctx); /* the level the graph leaves current */
        ctx->chunk_no++;
        if (ctx->profile) {
            CK(cudaStreamSynchronize(ctx->stream));
            for (int s = 0; s < n; s++)
                for (int kind = 0; kind < kProfKinds; kind++) {
                    if ((kind == 2 && (!ctx->probe || probe_folded(ctx))) || (kind == 3 && dft_launched(ctx) == 0) ||
                        (kind == 4 && !ctx->ion_split) ||
                        (kind <= 1 && ctx->fused) || (kind == 5 && !ctx->fused && !ctx->split))
                        continue;
                    float ms = 0.f;
                    CK(cudaEventElapsedTime(&ms, ctx->prof_ev[((size_t)s * kProfKinds + kind) * 2],
                                            ctx->prof_ev[((size_t)s * kProfKinds + kind) * 2 + 1]));
                    ctx->prof_ms[kind] += ms;
                    ctx->prof_n[kind] += kind == 3 ? (int64_t)dft_launched(ctx) : 1;
                }
        }
        ctx->last_launches += n * ((ctx->fused ? 1 : ctx->split ? split_launches(ctx) : ctx->by_class ? 1 + split_launches(ctx) : 2) + (ctx->ion_split ? 1 : 0) + (ctx->probe && !probe_folded(ctx) ? 1 : 0) +
                                   dft_launched(ctx));
        ctx->t += n;
        nsteps -= n;
    }
    return PHP_OK;
}

int php_prepare(php_ctx* ctx, int32_t nsteps)
{
    if (!ctx) return PHP_ERR_INPUT;
    if (nsteps < 0) return fail(ctx, PHP_ERR_INPUT, "negative step count");
    cudaGraphExec_t g;
    /* double buffered, a chunk of odd length leaves the other level current:
     * the graphs of both levels */
    int rc = PHP_OK;
    for (int lv = 0; lv < (ctx->fused || ctx->split ? 2 : 1) && rc == PHP_OK; lv++) {
        if (lv) swap_levels(ctx);
        if (nsteps >= ctx->max_chunk) rc = ensure_graph(ctx, ctx->max_chunk, 0, &g);
        if (rc == PHP_OK && nsteps % ctx->max_chunk) rc = ensure_graph(ctx, nsteps % ctx->max_chunk, 0, &g);
        if (lv) swap_levels(ctx);
    }
    return rc;
}

int php_sync(php_ctx* ctx)
{
    if (!ctx) return PHP_ERR_INPUT;
    CK(cudaStreamSynchronize(ctx->stream));
    CK(cudaGetLastError());
    int32_t flag = 0;
    CK(cudaMemcpy(&flag, ctx->err_flag, sizeof(flag), cudaMemcpyDeviceToHost));
    if (flag) return fail(ctx, PHP_ERR_TIMEOUT, "a sweep kernel gave up waiting for its plane loads");
    return PHP_OK;
}

int php_get_step(const php_ctx* ctx, int32_t* t)
{
    if (!ctx || !t) return PHP_ERR_INPUT;
    *t = ctx->t;
    return PHP_OK;
}

/* Gather geometry of a slice, with the reference's messages for bad ones. */
static int slice_geom(php_ctx* ctx, int32_t comp, char axis, int32_t position, int& ax, int& pos, size_t& n)
{
    if (comp < 0 || comp > 9) return fail(ctx, PHP_ERR_INPUT, "bad component %d", comp);
    if (axis == 'z') {
        if (position < 0 || position >= ctx->nz) return fail(ctx, PHP_ERR_INPUT, "Error: No process contains slice z=%d", position);
        ax = 0;
        pos = position + 1; /* fdtd.c:1029 with the halo already in the pointers (fdtd.c:274) */
        n = (size_t)ctx->nx * ctx->ny;
    } else if (axis == 'x') {
        if (position < 0 || position >= ctx->nx)
            return fail(ctx, PHP_ERR_INPUT, "Error: Invalid x slice position %d (range: 0-%d)", position, ctx->nx - 1);
        ax = 1;
        pos = position;
        n = (size_t)ctx->ny * ctx->nz;
    } else if (axis == 'y') {
        if (position < 0 || position >= ctx->ny)
            return fail(ctx, PHP_ERR_INPUT, "Error: Invalid y slice position %d (range: 0-%d)", position, ctx->ny - 1);
        ax = 2;
        pos = position;
        n = (size_t)ctx->nx * ctx->nz;
    } else {
        return fail(ctx, PHP_ERR_INPUT, "Error: Invalid slice axis '%c'. Must be 'x', 'y', or 'z'.", axis);
    }
    return PHP_OK;
}

static int read_slice_impl(php_ctx* ctx, int32_t comp, char axis, int32_t position, void* out, bool f32)
{
    if (!ctx || !out) return PHP_ERR_INPUT;
    int ax, pos;
    size_t n;
    int rc = slice_geom(ctx, comp, axis, position, ax, pos, n);
    if (rc) return rc;
    if (ctx->prec == PHP_PREC_FP32) launch_gather_plane<float>(ctx, comp, ax, pos, f32, ctx->scratch);
    else launch_gather_plane<double>(ctx, comp, ax, pos, f32, ctx->scratch);
    CK(cudaGetLastError());
    const size_t bytes = n * (f32 ? sizeof(float) : sizeof(double));
    CK(cudaMemcpyAsync(ctx->host_stage, ctx->scratch, bytes, cudaMemcpyDeviceToHost, ctx->stream));
    CK(cudaStreamSynchronize(ctx->stream));
    memcpy(out, ctx->host_stage, bytes);
    return PHP_OK;
}

int php_read_slice(php_ctx* ctx, int32_t comp, char axis, int32_t position, float* out)
{
    return read_slice_impl(ctx, comp, axis, position, out, true);
}

int php_read_slice_f64(php_ctx* ctx, int32_t comp, char axis, int32_t position, double* out)
{
    return read_slice_impl(ctx, comp, axis, position, out, false);
}

int php_read_volume(php_ctx* ctx, int32_t comp, double* out)
{
    if (!ctx || !out) return PHP_ERR_INPUT;
    if (comp < 0 || comp > 8) return fail(ctx, PHP_ERR_INPUT, "bad component %d", comp);
    const size_t n = (size_t)ctx->nx * ctx->ny * ctx->nz;
    void* dbuf = nullptr;
    CK(cudaMallocAsync(&dbuf, n * sizeof(double), ctx->stream));
    if (ctx->prec == PHP_PREC_FP32)
        gather_volume<float><<<592, 256, 0, ctx->stream>>>(make_fields<float>(ctx), make_dview<float>(ctx), comp, ctx->nx, ctx->ny, ctx->nz, ctx->nxp, (double*)dbuf);
    else
        gather_volume<double><<<592, 256, 0, ctx->stream>>>(make_fields<double>(ctx), make_dview<double>(ctx), comp, ctx->nx, ctx->ny, ctx->nz, ctx->nxp, (double*)dbuf);
    CK(cudaGetLastError());
    CK(cudaMemcpyAsync(out, dbuf, n * sizeof(double), cudaMemcpyDeviceToHost, ctx->stream));
    CK(cudaFreeAsync(dbuf, ctx->stream));
    CK(cudaStreamSynchronize(ctx->stream));
    return PHP_OK;
}

int php_read_point(php_ctx* ctx, int32_t i, int32_t j, int32_t k, double* out9)
{
    if (!ctx || !out9) return PHP_ERR_INPUT;
    if (i < 0 || i >= ctx->nx || j < 0 || j >= ctx->ny || k < -1 || k > ctx->nz)
        return fail(ctx, PHP_ERR_INPUT, "point (%d,%d,%d) outside the grid", i, j, k);
    const int64_t c = ((int64_t)k * ctx->ny + j) * ctx->nxp + i;
    double* pt = (double*)ctx->scratch;
    if (ctx->prec == PHP_PREC_FP32) point_gather<float><<<1, 32, 0, ctx->stream>>>(make_fields<float>(ctx), make_dview<float>(ctx), c, pt);
    else point_gather<double><<<1, 32, 0, ctx->stream>>>(make_fields<double>(ctx), make_dview<double>(ctx), c, pt);
    CK(cudaGetLastError());
    CK(cudaMemcpyAsync(ctx->host_stage, pt, 9 * sizeof(double), cudaMemcpyDeviceToHost, ctx->stream));
    CK(cudaStreamSynchronize(ctx->stream));
    memcpy(out9, ctx->host_stage, 9 * sizeof(double));
    return PHP_OK;
}

int php_read_cell_state(php_ctx* ctx, int32_t i, int32_t j, int32_t k, int32_t* natom, double* r, double* v,
                        double* p_ade, double* p_ade_old)
{
    if (!ctx) return PHP_ERR_INPUT;
    if (i < 0 || i >= ctx->nx || j < 0 || j >= ctx->ny || k < 0 || k >= ctx->nz)
        return fail(ctx, PHP_ERR_INPUT, "cell (%d,%d,%d) outside the grid", i, j, k);
    const int64_t c = ((int64_t)k * ctx->ny + j) * ctx->nxp + i;
    CK(cudaStreamSynchronize(ctx->stream));
    uint8_t mid = 0;
    CK(cudaMemcpy(&mid, ctx->mat + c, 1, cudaMemcpyDeviceToHost));
    const int na = ctx->mat_natom[mid];
    if (natom) *natom = na;
    int32_t s = -1;
    if (ctx->slot) CK(cudaMemcpy(&s, ctx->slot + c, sizeof(int32_t), cudaMemcpyDeviceToHost));
    const size_t rs = rsize(ctx->prec);
    auto fetch = [&](void* base, int q, double* dst) -> int {
        char tmp[8];
        cudaError_t e = cudaMemcpy(tmp, (const char*)base + ((int64_t)q * ctx->nslot + s) * (int64_t)rs, rs, cudaMemcpyDeviceToHost);
        if (e != cudaSuccess) return fail(ctx, PHP_ERR_CUDA, "cudaMemcpy: %s", cudaGetErrorString(e));
        *dst = rs == 4 ? (double)*(float*)tmp : *(double*)tmp;
        return PHP_OK;
    };
    for (int q = 0; q < 3 * na; q++) {
        if (r) { int rc = fetch(ctx->r, q, &r[q]); if (rc) return rc; r[q] *= ctx->rv_unit; }
        if (v) { int rc = fetch(ctx->v, q, &v[q]); if (rc) return rc; v[q] *= ctx->rv_unit; }
    }
    if (ctx->mat_ade[mid] && s >= 0) {
        double pq[3], poq[3];
        for (int q = 0; q < 3; q++) {
            double p = 0.0, po = 0.0;
            int rc = fetch(ctx->P, q, &p);
            if (!rc) rc = fetch(ctx->Po, q, &po);
            if (rc) return rc;
            pq[q] = p;
            poq[q] = po;
        }
        if (ctx->prec == PHP_PREC_FP32) {
            /* FP32 keeps Q = D - P (lab frame) in the P pool and
             * J = P - P_old (crystal frame) in the P_old pool */
            double dl[3];
            for (int q = 0; q < 3; q++) {
                double dv = 0.0;
                int rc = fetch(ctx->Dp, q, &dv);
                if (rc) return rc;
                dl[q] = dv - pq[q];
            }
            const int fl = ctx->mat_flags[mid];
            const double cs = ctx->mat_cs[mid], sn = ctx->mat_sn[mid];
            if (fl & kRotZ) {
                const double u = dl[0] * cs - dl[1] * sn, w = dl[0] * sn + dl[1] * cs;
                dl[0] = u; dl[1] = w;
            } else if (fl & kRotX) {
                const double u = dl[1] * cs - dl[2] * sn, w = dl[1] * sn + dl[2] * cs;
                dl[1] = u; dl[2] = w;
            }
            for (int q = 0; q < 3; q++) {
                poq[q] = dl[q] - poq[q];
                pq[q] = dl[q];
            }
        }
        for (int q = 0; q < 3; q++) {
            if (p_ade) p_ade[q] = pq[q];
            if (p_ade_old) p_ade_old[q] = poq[q];
        }
    } else {
        for (int q = 0; q < 3; q++) {
            if (p_ade) p_ade[q] = 0.0;
            if (p_ade_old) p_ade_old[q] = 0.0;
        }
    }
    return PHP_OK;
}

/* Enqueues the first diagnostics pass; *blocks_out partials in *part_out (scratch). */
static int enqueue_diag(php_ctx* ctx, DiagPartial** part_out, int* blocks_out)
{
    const int blocks = (int)std::min<int64_t>(148 * 8, std::max<int64_t>(((int64_t)ctx->ny * ctx->nz + 15) / 16, (ctx->nslot + 1023) / 1024));
    DiagPartial* part = (DiagPartial*)ctx->scratch;
    *part_out = part;
    *blocks_out = blocks;
    if (ctx->prec == PHP_PREC_FP32) {
        diag_pass1<float><<<blocks, 256, 0, ctx->stream>>>(make_fields<float>(ctx), ctx->nx, ctx->ny, ctx->nz, ctx->nxp, (const float*)ctx->r,
                                                           ctx->rv_unit, ctx->any_atoms ? ctx->nslot : 0, ctx->slot_cell, ctx->slot_n3,
                                                           std::max(ctx->n3max, 1), part);
    } else {
        diag_pass1<double><<<blocks, 256, 0, ctx->stream>>>(make_fields<double>(ctx), ctx->nx, ctx->ny, ctx->nz, ctx->nxp, (const double*)ctx->r,
                                                            ctx->rv_unit, ctx->any_atoms ? ctx->nslot : 0, ctx->slot_cell, ctx->slot_n3,
                                                            std::max(ctx->n3max, 1), part);
    }
    CK(cudaGetLastError());
    return PHP_OK;
}

/* php_diag from the reduced partial (argmax in the reference's loop order) */
static void decode_diag(const php_ctx* ctx, const DiagPartial& h, php_diag* out)
{
    out->max_e = h.max_e;
    out->max_ex = h.max_ex;
    out->max_r = h.max_r;
    if (h.max_r > 0.0 && h.key_r != INT64_MAX) {
        const int64_t n3 = std::max(ctx->n3max, 1);
        int64_t cell = h.key_r / n3;
        const int q = (int)(h.key_r % n3);
        out->argmax_r[2] = (int)(cell % ctx->nz);
        cell /= ctx->nz;
        out->argmax_r[1] = (int)(cell % ctx->ny);
        out->argmax_r[0] = (int)(cell / ctx->ny);
        out->argmax_r[3] = q / 3;
        out->argmax_r[4] = q % 3;
    } else {
        for (int q = 0; q < 5; q++) out->argmax_r[q] = -1;
    }
}

int php_diagnostics(php_ctx* ctx, php_diag* out)
{
    if (!ctx || !out) return PHP_ERR_INPUT;
    DiagPartial* part = nullptr;
    int blocks = 0;
    int rc = enqueue_diag(ctx, &part, &blocks);
    if (rc) return rc;
    DiagPartial* fin = part + blocks;
    diag_pass2<<<1, 256, 0, ctx->stream>>>(part, blocks, fin);
    CK(cudaGetLastError());
    DiagPartial h;
    CK(cudaMemcpyAsync(ctx->host_stage, fin, sizeof(DiagPartial), cudaMemcpyDeviceToHost, ctx->stream));
    CK(cudaStreamSynchronize(ctx->stream));
    memcpy(&h, ctx->host_stage, sizeof(h));
    decode_diag(ctx, h, out);
    return PHP_OK;
}

int php_probe_set(php_ctx* ctx, int32_t i, int32_t j, int32_t k_field, int32_t k_atom)
{
    if (!ctx) return PHP_ERR_INPUT;
    if (i < 0 || i >= ctx->nx || j < 0 || j >= ctx->ny || k_field < -1 || k_field > ctx->nz || k_atom < 0 || k_atom >= ctx->nz)
        return fail(ctx, PHP_ERR_INPUT, "probe (%d,%d,%d/%d) outside the grid", i, j, k_field, k_atom);
    drop_graphs(ctx);
    ctx->probe_cf = ((int64_t)k_field * ctx->ny + j) * ctx->nxp + i;
    const int64_t ca = ((int64_t)k_atom * ctx->ny + j) * ctx->nxp + i;
    ctx->probe_ka = k_atom;
    uint8_t mid = 0;
    CK(cudaMemcpy(&mid, ctx->mat + ca, 1, cudaMemcpyDeviceToHost));
    ctx->probe_n3 = 3 * ctx->mat_natom[mid];
    int32_t s = -1;
    if (ctx->slot) CK(cudaMemcpy(&s, ctx->slot + ca, sizeof(int32_t), cudaMemcpyDeviceToHost));
    ctx->probe_slot = s;
    DCell& pd = ctx->probe_d;
    pd.slot = -1;
    for (double& m : pd.dm) m = 0.0;
    if (k_field >= 0 && k_field < ctx->nz) {
        if (ctx->slot) CK(cudaMemcpy(&pd.slot, ctx->slot + ctx->probe_cf, sizeof(int32_t), cudaMemcpyDeviceToHost));
        if (ctx->dmat) {
            uint8_t fm = 0;
            CK(cudaMemcpy(&fm, ctx->mat + ctx->probe_cf, 1, cudaMemcpyDeviceToHost));
            CK(cudaMemcpy(pd.dm, ctx->dmat + 9 * (int)fm, sizeof(pd.dm), cudaMemcpyDeviceToHost));
        }
    }
    if (ctx->probe_n3 == 0) ctx->probe_slot = 0;
    if (!ctx->probe_rows) {
        int rc = dalloc(ctx, (void**)&ctx->probe_rows, (size_t)kProbeCap * (9 + 2 * std::max(ctx->n3max, 1)) * sizeof(double));
        if (rc) return rc;
        rc = dalloc(ctx, (void**)&ctx->probe_count, 2 * sizeof(int32_t));
        if (rc) return rc;
    }
    CK(cudaMemsetAsync(ctx->probe_count, 0, 2 * sizeof(int32_t), ctx->stream));
    ctx->probe = true;
    ctx->probe_t0 = ctx->t;
    return PHP_OK;
}

int php_probe_read(php_ctx* ctx, double* rows, int32_t max_rows, int32_t* nrows, int32_t* row_len)
{
    if (!ctx || !nrows) return PHP_ERR_INPUT;
    if (!ctx->probe) return fail(ctx, PHP_ERR_STATE, "no probe set");
    int32_t cnt[2];
    CK(cudaMemcpyAsync(cnt, ctx->probe_count, 2 * sizeof(int32_t), cudaMemcpyDeviceToHost, ctx->stream));
    CK(cudaStreamSynchronize(ctx->stream));
    const int rl = 9 + 2 * ctx->probe_n3;
    if (row_len) *row_len = rl;
    if (cnt[1]) return fail(ctx, PHP_ERR_STATE, "probe buffer overflowed (more than %d rows between reads)", kProbeCap);
    if (cnt[0] > max_rows) return fail(ctx, PHP_ERR_STATE, "%d probe rows pending, buffer holds %d", cnt[0], max_rows);
    if (cnt[0] > 0 && rows)
        CK(cudaMemcpyAsync(rows, ctx->probe_rows, (size_t)cnt[0] * rl * sizeof(double), cudaMemcpyDeviceToHost, ctx->stream));
    CK(cudaMemsetAsync(ctx->probe_count, 0, 2 * sizeof(int32_t), ctx->stream));
    CK(cudaStreamSynchronize(ctx->stream));
    *nrows = cnt[0];
    ctx->probe_t0 = ctx->t;
    return PHP_OK;
}

/* ------------------------------------------------------------ output frames */

int php_frame_begin(php_ctx* ctx, const php_frame_req* req, int32_t* ticket)
{
    if (!ctx || !req || !ticket) return PHP_ERR_INPUT;
    int ax = 0, pos = 0;
    size_t slice_n = 0;
    if (req->slice_comp >= 0) {
        int rc = slice_geom(ctx, req->slice_comp, (char)req->slice_axis, req->slice_pos, ax, pos, slice_n);
        if (rc) return rc;
    }
    const bool has_point = req->point[0] >= 0;
    if (has_point && (req->point[0] >= ctx->nx || req->point[1] < 0 || req->point[1] >= ctx->ny || req->point[2] < -1 ||
                      req->point[2] > ctx->nz))
        return fail(ctx, PHP_ERR_INPUT, "point (%d,%d,%d) outside the grid", req->point[0], req->point[1], req->point[2]);
    const bool has_cell = req->cell[0] >= 0;
    if (has_cell && (req->cell[0] >= ctx->nx || req->cell[1] < 0 || req->cell[1] >= ctx->ny || req->cell[2] < 0 ||
                     req->cell[2] >= ctx->nz))
        return fail(ctx, PHP_ERR_INPUT, "cell (%d,%d,%d) outside the grid", req->cell[0], req->cell[1], req->cell[2]);
    if (req->probe && !ctx->probe) return fail(ctx, PHP_ERR_STATE, "no probe set");
    const int32_t tk = ctx->frame_next;
    php_ctx::FrameSlot& F = ctx->frames[tk % PHP_FRAME_SLOTS];
    /* the oldest frame must have been released (bounded wait) */
    const auto t0 = std::chrono::steady_clock::now();
    while (F.state.load(std::memory_order_acquire) != 0) {
        if (std::chrono::steady_clock::now() - t0 > std::chrono::seconds(60))
            return fail(ctx, PHP_ERR_TIMEOUT, "frame %d was not released within 60 s", F.ticket);
        std::this_thread::sleep_for(std::chrono::microseconds(50));
    }
    if (!F.done) CK(cudaEventCreateWithFlags(&F.done, cudaEventDisableTiming));
    if (!F.head) F.head = (FrameHead*)pinned_get(sizeof(FrameHead));
    const size_t slice_cap = std::max({(size_t)ctx->nx * ctx->ny, (size_t)ctx->ny * ctx->nz, (size_t)ctx->nx * ctx->nz});
    if (!F.slice) F.slice = (float*)pinned_get(slice_cap * sizeof(float));
    const int32_t row_len = 9 + 2 * ctx->probe_n3;
    int64_t rows = 0;
    if (req->probe) {
        rows = std::min<int64_t>((int64_t)ctx->t - ctx->probe_t0, kProbeCap);
        const size_t need = (size_t)std::max<int64_t>(rows, 1) * row_len * sizeof(double);
        if (F.rows_bytes < need) {
            pinned_put(F.rows);
            F.rows = (double*)pinned_get(need);
            F.rows_bytes = F.rows ? need : 0;
        }
        if (!F.rows) return fail(ctx, PHP_ERR_OOM, "page-locked host allocation failed");
    }
    if (!F.head || !F.slice) return fail(ctx, PHP_ERR_OOM, "page-locked host allocation failed");

    DiagPartial* part = nullptr;
    int nparts = 0;
    if (req->diag) {
        int rc = enqueue_diag(ctx, &part, &nparts);
        if (rc) return rc;
    }
    const int64_t pc = has_point ? point_index(ctx, req->point) : 0;
    const int64_t cc = has_cell ? point_index(ctx, req->cell) : -1;
    /* many rows (a long interval, a large lattice) by a copy, ahead of the
     * gather that resets their counter */
    const double* rows_dev = req->probe ? ctx->probe_rows : nullptr;
    const bool copy_rows = rows * row_len * (int64_t)sizeof(double) > kDirectRows;
    if (req->probe && copy_rows)
        CK(cudaMemcpyAsync(F.rows, rows_dev, (size_t)rows * row_len * sizeof(double), cudaMemcpyDeviceToHost, ctx->stream));
    double* rows_out = req->probe && !copy_rows ? F.rows : nullptr;
    if (ctx->prec == PHP_PREC_FP32) launch_frame_gather<float>(ctx, part, nparts, has_point, pc, cc, rows_dev, rows, row_len, rows_out, F.head);
    else launch_frame_gather<double>(ctx, part, nparts, has_point, pc, cc, rows_dev, rows, row_len, rows_out, F.head);
    CK(cudaGetLastError());
    if (req->probe) ctx->probe_t0 = ctx->t;
    if (req->slice_comp >= 0) {
        /* a small slice straight into the page-locked buffer, a large one by a copy */
        const bool direct = slice_n * sizeof(float) <= kDirectSlice;
        float* dst = direct ? F.slice : (float*)ctx->scratch;
        if (ctx->prec == PHP_PREC_FP32) launch_gather_plane<float>(ctx, req->slice_comp, ax, pos, true, dst);
        else launch_gather_plane<double>(ctx, req->slice_comp, ax, pos, true, dst);
        CK(cudaGetLastError());
        if (!direct) CK(cudaMemcpyAsync(F.slice, ctx->scratch, slice_n * sizeof(float), cudaMemcpyDeviceToHost, ctx->stream));
    }
    CK(cudaEventRecord(F.done, ctx->stream));
    F.ticket = tk;
    F.step = ctx->t;
    F.req = *req;
    F.rows_copied = rows;
    F.row_len = row_len;
    F.slice_len = req->slice_comp >= 0 ? (int64_t)slice_n : 0;
    F.state.store(1, std::memory_order_release);
    ctx->frame_next++;
    *ticket = tk;
    return PHP_OK;
}

int php_frame_wait(php_ctx* ctx, int32_t ticket, php_frame* out)
{
    if (!ctx || !out || ticket < 0) return PHP_ERR_INPUT;
    php_ctx::FrameSlot& F = ctx->frames[ticket % PHP_FRAME_SLOTS];
    if (F.state.load(std::memory_order_acquire) != 1 || F.ticket != ticket)
        return fail(ctx, PHP_ERR_STATE, "frame %d is not taken", ticket);
    CK(cudaEventSynchronize(F.done));
    const FrameHead& h = *F.head;
    if (h.err) return fail(ctx, PHP_ERR_TIMEOUT, "a sweep kernel gave up waiting for its plane loads");
    memset(out, 0, sizeof(*out));
    out->step = F.step;
    if (F.req.diag) {
        decode_diag(ctx, h.diag, &out->diag);
        out->diag_natom = h.diag_natom;
        memcpy(out->diag_point, h.diag_point, sizeof(out->diag_point));
        memcpy(out->diag_r, h.diag_r, sizeof(out->diag_r));
        memcpy(out->diag_v, h.diag_v, sizeof(out->diag_v));
    }
    if (F.req.point[0] >= 0) memcpy(out->point, h.point, sizeof(out->point));
    if (F.req.cell[0] >= 0) {
        out->cell_natom = h.cell_natom;
        memcpy(out->cell_r, h.cell_r, sizeof(out->cell_r));
        memcpy(out->cell_v, h.cell_v, sizeof(out->cell_v));
    }
    out->slice = F.slice_len ? F.slice : nullptr;
    out->slice_len = F.slice_len;
    out->row_len = F.row_len;
    if (F.req.probe) {
        if (h.probe_count[1])
            return fail(ctx, PHP_ERR_STATE, "probe buffer overflowed (more than %d rows between reads)", kProbeCap);
        out->nrows = (int32_t)std::min<int64_t>(h.probe_count[0], F.rows_copied);
        out->rows = F.rows;
    }
    return PHP_OK;
}

int php_frame_release(php_ctx* ctx, int32_t ticket)
{
    if (!ctx || ticket < 0) return PHP_ERR_INPUT;
    php_ctx::FrameSlot& F = ctx->frames[ticket % PHP_FRAME_SLOTS];
    if (F.ticket != ticket) return fail(ctx, PHP_ERR_STATE, "frame %d is not taken", ticket);
    F.state.store(0, std::memory_order_release);
    return PHP_OK;
}

int php_dft_add(php_ctx* ctx, int32_t comp, int32_t z_plane, int32_t first_step, int32_t sample_interval, int32_t nfreq,
                const double* freq_hz, int32_t cast_f32, int32_t* id)
{
    if (!ctx || !freq_hz || !id) return PHP_ERR_INPUT;
    if (comp < 0 || comp > 8) return fail(ctx, PHP_ERR_INPUT, "DFT component must be 0..8");
    if (z_plane < -1 || z_plane > ctx->nz) return fail(ctx, PHP_ERR_INPUT, "DFT plane %d outside -1..nz", z_plane);
    if (sample_interval < 1 || nfreq < 1 || nfreq > 64 || first_step < 0) return fail(ctx, PHP_ERR_INPUT, "bad DFT arguments");
    DftPlane p;
    p.comp = comp;
    p.z = z_plane;
    p.first = first_step;
    p.interval = sample_interval;
    p.nfreq = nfreq;
    p.cast_f32 = cast_f32 ? 1 : 0;
    p.freq.assign(freq_hz, freq_hz + nfreq);
    int rc = dalloc(ctx, (void**)&p.acc, (size_t)nfreq * ctx->nx * ctx->ny * 2 * sizeof(double));
    if (rc) return rc;
    ctx->dft.push_back(p);
    rc = relayout_step_inputs(ctx);
    if (rc) return rc;
    drop_graphs(ctx);
    *id = (int32_t)ctx->dft.size() - 1;
    return PHP_OK;
}

int php_dft_read(php_ctx* ctx, int32_t id, double* out, int32_t* nsamples)
{
    if (!ctx || !out) return PHP_ERR_INPUT;
    if (id < 0 || id >= (int)ctx->dft.size()) return fail(ctx, PHP_ERR_INPUT, "no DFT plane %d", id);
    const DftPlane& p = ctx->dft[id];
    /* the device keeps [nfreq][ny][nx][2] (x fastest for the samplers); the
     * caller gets [nfreq][nx][ny][2], transposed on the device (three planes
     * of 512 x 512: 5 ms on the host) */
    const int64_t total = (int64_t)p.nfreq * ctx->nx * ctx->ny, chunk = (int64_t)(ctx->scratch_bytes / sizeof(double2));
    for (int64_t o = 0; o < total; o += chunk) {
        const int64_t n = std::min(chunk, total - o);
        dft_reorder<<<(unsigned)std::min<int64_t>((n + 255) / 256, 148 * 8), 256, 0, ctx->stream>>>((const double2*)p.acc, ctx->nx, ctx->ny, o, n,
                                                                                      (double2*)ctx->scratch);
        CK(cudaGetLastError());
        CK(cudaMemcpyAsync(out + 2 * o, ctx->scratch, (size_t)n * sizeof(double2), cudaMemcpyDeviceToHost, ctx->stream));
    }
    CK(cudaStreamSynchronize(ctx->stream));
    if (nsamples) *nsamples = p.nsamples;
    return PHP_OK;
}

int php_memory_bytes(const php_ctx* ctx, uint64_t* bytes)
{
    if (!ctx || !bytes) return PHP_ERR_INPUT;
    *bytes = ctx->bytes;
    return PHP_OK;
}

bool php_holds_second_level(const php_ctx* ctx) { return ctx->split; }

int php_estimate_buffers(const php_desc* desc, uint64_t* bytes, uint64_t* more)
{
    return estimate_bytes(*desc, bytes, more);
}

int php_estimate_bytes(const php_desc* desc, uint64_t* bytes)
{
    if (!desc || !bytes) return PHP_ERR_INPUT;
    uint64_t more = 0;
    const int rc = estimate_bytes(*desc, bytes, &more);
    if (rc == PHP_OK) *bytes += more;
    return rc;
}

int php_last_launch_count(const php_ctx* ctx, int32_t* launches)
{
    if (!ctx || !launches) return PHP_ERR_INPUT;
    *launches = ctx->last_launches;
    return PHP_OK;
}

int php_block_census(const php_ctx* ctx, int64_t* counts)
{
    if (!ctx || !counts) return PHP_ERR_INPUT;
    for (int q = 0; q < PHP_CENSUS_LEN; q++) counts[q] = ctx->census[q];
    return PHP_OK;
}

int php_stream(const php_ctx* ctx, void** stream)
{
    if (!ctx || !stream) return PHP_ERR_INPUT;
    *stream = (void*)ctx->stream;
    return PHP_OK;
}

int php_profile_enable(php_ctx* ctx, int32_t enable)
{
    if (!ctx) return PHP_ERR_INPUT;
    drop_graphs(ctx);
    if (enable && ctx->prof_ev.empty()) {
        ctx->prof_ev.resize((size_t)kMaxChunk * kProfKinds * 2);
        for (auto& e : ctx->prof_ev) CK(cudaEventCreate(&e));
    }
    ctx->profile = enable != 0;
    for (int q = 0; q < kProfKinds; q++) {
        ctx->prof_ms[q] = 0.0;
        ctx->prof_n[q] = 0;
    }
    return PHP_OK;
}

int php_profile_read(php_ctx* ctx, double* ms, int64_t* launches)
{
    if (!ctx) return PHP_ERR_INPUT;
    CK(cudaStreamSynchronize(ctx->stream));
    for (int q = 0; q < kProfKinds; q++) {
        if (ms) ms[q] = ctx->prof_ms[q];
        if (launches) launches[q] = ctx->prof_n[q];
    }
    return PHP_OK;
}

} // extern "C"

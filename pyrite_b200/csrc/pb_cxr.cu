// Incoherent PXR + CBS line scoring of a segment list (sm_100a).
//
// For every (segment, reflection row, detector direction) the kernels follow
// the reference's batched line chain (src/pyrite/montecarlo/spectrum/cxr/
// _batched.py:461-931): exact-recoil vacuum root, three fixed-point passes
// of the first-order Snell resonance (cxr/_kernels.py:702-765), the shared
// interpolation bracket for chi/U/mu (cxr/_kernels.py:482-620), the exact
// second-order PXR+CBS amplitude of both polarisations (cxr/_recoil.py:35),
// the segment-mean Beer-Lambert escape (segment_escape.py:276) and the
// line weight and width (cxr/_kernels.py:658, cxr/_batched.py:702-730).
//
// Reductions:
//  * bin-mean (production): each kept line is integrated exactly over the
//    bins within ``exact_widths`` sinc widths of its centre (FP64 sine
//    integral), and its far field -- the cycle-averaged envelope
//    1/(2 a^2 (E_lo - E_r)(E_hi - E_r)) -- is carried by three moments per
//    centre bin in global memory and spread onto the grid by one convolution
//    (cxr/_bin_quadrature.py:280-560 for the exact and far forms).
//    Lines never leave the SM: warp work -> shared-memory spectrum -> one
//    global atomic per bin per block.
//  * node sampling: kept lines are appended to a line buffer and reduced
//    against the grid nodes by a separate kernel (cxr/_cpu_reduce.py:26-50).
//
// PB_FP64 evaluates the chain and the bins in double; PB_MIXED in float, with
// the node phase a (E - E_r) formed and range-reduced in double and every
// spectrum sum in double.
#include <algorithm>
#include <climits>
#include <type_traits>
#include <cstdint>
#include <cstdio>
#include <cuda.h>
#include <mutex>

#include "pb_common.cuh"
#include "pb_internal.h"
#include "pb_layers.cuh"

namespace pb {

constexpr int kSegTile = 16;
constexpr int kCxrThreads = 256;
// Two blocks an SM (128 registers). Three of the float instances fit 80 registers
// and 75 KB, but the kernel is bound by issue, not latency: 8192 histories of the
// 50 MeV Si scene took 95.9 ms with three and 82.7 with two, whose passes are
// larger.
constexpr int kCxrBlocks = 2;
// Reflection rows per pass: 120 on the float path (a pass's prefilter survivors
// then fill the block's threads about one and a half times), 48 on the FP64 path,
// whose queues and tables take twice the room.
template <class Real>
constexpr int row_chunk() { return sizeof(Real) == 4 ? 120 : 48; }
template <class Real>
constexpr int pair_queue() { return kSegTile * row_chunk<Real>(); }  // every pair of a pass may keep a line
// The prefilter's survivors and the kept lines wait until a whole round of
// kCxrThreads is there.
template <class Real>
constexpr int surv_queue() { return pair_queue<Real>() + kCxrThreads; }
template <class Real>
constexpr int line_queue() { return surv_queue<Real>() + kCxrThreads; }
constexpr int kStripBins = 31;  // bins a warp owns in the whole-axis phase (32 edges)
// Window lines collected before the window phase runs; one more round of
// kCxrThreads lines always fits.
constexpr int kWideCap = 2 * kCxrThreads;
constexpr int kWideRun = kWideCap - kCxrThreads;
// Classes of window lines: 4, 8, 16 or 32 lanes a line (two edges a lane), or
// the block's warps together over strips of the axis (kWinStrip: windows of more
// than kStripSpan bins a side; kWinAxis: no moments, every bin).
enum WinClass { kWin4 = 0, kWin8, kWin16, kWin32, kWinStrip, kWinAxis, kWinClasses };
constexpr int kStripSpan = 124;
// Strip lines wait for one another over several window phases.
constexpr int kStripRun = kCxrThreads / 2;
// The list's lines by class: two classes share an index array, one from each end
// (a line is in one class, so the ends cannot meet).
__device__ __forceinline__ int win_slot(int cls, int k) {
    return (cls >> 1) * kWideCap + ((cls & 1) ? kWideCap - 1 - k : k);
}
constexpr int kMaxTab = 4096;   // E_tab / delta staged in shared memory up to this size

// Math of the line chain. FP64 uses IEEE operations throughout (parity with
// the reference's FP64 chain); the float path uses the SFU approximations
// (division by reciprocal, sqrt by reciprocal square root, base-2 exp/log),
// each within a few ulp, which the 1 % spectrum tolerance of the mixed path
// absorbs many times over.
// A rounded product the compiler does not contract into the following addition.
__device__ __forceinline__ float r_mul(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ double r_mul(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ double r_sqrt(double x) { return sqrt(x); }
__device__ __forceinline__ float r_sqrt(float x) { return x > 0.0f ? x * rsqrtf(x) : sqrtf(x); }
__device__ __forceinline__ double r_exp(double x) { return exp(x); }
__device__ __forceinline__ float r_exp(float x) { return __expf(x); }
__device__ __forceinline__ double r_expm1(double x) { return expm1(x); }
__device__ __forceinline__ float r_expm1(float x) { return expm1f(x); }
__device__ __forceinline__ double r_log1p(double x) { return log1p(x); }
__device__ __forceinline__ float r_log1p(float x) { return log1pf(x); }
__device__ __forceinline__ double rdiv(double a, double b) { return a / b; }
__device__ __forceinline__ float rdiv(float a, float b) { return __fdividef(a, b); }

// Per (segment, direction) quantities shared by every reflection row.
template <class Real>
struct SegPre {
    Real vx, vy, vz;        // beta v_hat
    Real gamma;
    Real denom_row;         // 1 - beta v_hat.n, cancellation free
    Real t_L;               // L / beta
    Real path0, path1;      // escape paths at the segment ends
    Real gx, gy, gz;        // grad L
    Real grad2;
    Real v_dot_grad;
    Real inv_E;             // hbar c / E
    int radiates;           // elec_id < Ne
};

template <class Real>
struct RowPre {
    Real G[3];
    Real ES[3];
    Real EP[3];
    Real g2, n_dot_g, g_dot_es, g_dot_ep, wm;
    int row;
};

template <class Real>
__device__ __forceinline__ Real slab_path(Real z, Real thickness, Real nz) {
    const Real inv_nz = (Real)1 / fmax(fabs(nz), (Real)1.0e-12);
    const Real depth = fmin(fmax(z, (Real)0), thickness);
    return nz < (Real)0 ? depth * inv_nz : (thickness - depth) * inv_nz;
}

template <class Real>
__device__ void seg_precompute(SegPre<Real> &sp, const pb_cxr_args &a, int64_t s, const double *nh) {
    const double E = a.E_keV[s];
    const Real Er = (Real)E;
    const Real vhx = (Real)a.v_hat[3 * s], vhy = (Real)a.v_hat[3 * s + 1], vhz = (Real)a.v_hat[3 * s + 2];
    const Real nx = (Real)nh[0], ny = (Real)nh[1], nz = (Real)nh[2];
    // cxr/_setup.py:945-1005; kinematics.py:151-154
    const Real g0 = (Real)1 + Er / (Real)510.99895;
    const Real beta = r_sqrt((Real)1 - (Real)1 / (g0 * g0));
    sp.vx = beta * vhx;
    sp.vy = beta * vhy;
    sp.vz = beta * vhz;
    // cxr/_kernels.py:678-699
    const Real gamma = (Real)1 + Er / (Real)(kMeEv / 1e3);
    const Real omb = (Real)1 / (gamma * gamma * ((Real)1 + beta));
    const Real dvx = vhx - nx, dvy = vhy - ny, dvz = vhz - nz;
    const Real omc = (Real)0.5 * (dvx * dvx + dvy * dvy + dvz * dvz);
    sp.gamma = gamma;
    sp.denom_row = omb + beta * omc;
    sp.t_L = (Real)a.L[s] / beta;
    // segment_escape.py:239-270, single slab
    const Real T = (Real)a.thickness;
    const Real half = (Real)0.5 * (Real)a.L[s];
    const Real z_mid = (Real)a.r_mid[3 * s + 2];
    sp.path0 = slab_path<Real>(z_mid - half * vhz, T, nz);
    sp.path1 = slab_path<Real>(z_mid + half * vhz, T, nz);
    // segment_escape.py:95-131
    Real gx = (Real)-0.0 / nz, gy = (Real)-0.0 / nz, gz = (Real)-1 / nz;
    if (z_mid < (Real)0 || z_mid > T) { gx = 0; gy = 0; gz = 0; }
    sp.gx = gx; sp.gy = gy; sp.gz = gz;
    sp.grad2 = gx * gx + gy * gy + gz * gz;
    sp.v_dot_grad = sp.vx * gx + sp.vy * gy + sp.vz * gz;
    sp.inv_E = (Real)kHbarcEvAng / (gamma * (Real)kMeEv);
    sp.radiates = a.elec_id[s] < a.Ne && (a.seg_layer == nullptr || a.seg_layer[s] == a.emit_layer);
}

// searchsorted(grid, x, side="left") clipped to [1, n-1] and the blend
// fraction (cxr/_kernels.py:328-349).
// Geometric tabulation grids (grid[i] = exp(log0 + i h)) are indexed in
// closed form and then corrected to the exact searchsorted answer, which
// replaces ~log2(n) dependent shared-memory loads by one logarithm.
struct TabIndex {
    bool geometric;
    double log0;
    double inv_h;
};

__device__ __forceinline__ double t_log(double x) { return log(x); }
__device__ __forceinline__ float t_log(float x) { return __logf(x); }

template <class Real>
__device__ __forceinline__ void bracket(const Real *grid, int n, Real x, int &idx, Real &frac,
                                        bool &below, bool &above, const TabIndex &ti) {
    int i;
    if (isnan(x)) {
        i = n;
    } else if (ti.geometric) {
        int c = 0;
        if (x > grid[0]) {
            const Real f = (t_log(x) - (Real)ti.log0) * (Real)ti.inv_h;
            c = f >= (Real)(n - 1) ? n : (int)ceil(f);
            if (c < 0) c = 0;
        }
        // searchsorted(side="left"): first index with grid[i] >= x
        while (c > 0 && !(grid[c - 1] < x)) --c;
        while (c < n && grid[c] < x) ++c;
        i = c;
    } else {
        int lo = 0, hi = n;
        while (lo < hi) {
            const int mid = (lo + hi) >> 1;
            if (grid[mid] < x) lo = mid + 1; else hi = mid;
        }
        i = lo;
    }
    i = i < 1 ? 1 : (i > n - 1 ? n - 1 : i);
    idx = i;
    frac = rdiv(x - grid[i - 1], grid[i] - grid[i - 1]);
    below = x <= grid[0];
    above = x >= grid[n - 1];
}

// A bracket kept with its cell's bounds: the passes of one pair move the
// energy by parts in 1e5, so most land in the cell already found and cost a
// comparison instead of a search (the same index and fraction either way).
template <class Real>
struct Cell {
    Real x0, x1, frac;
    int idx;
    bool below, above;
};

template <class Real>
__device__ __forceinline__ void locate(Cell<Real> &c, const Real *grid, int n, Real x, const TabIndex &ti) {
    if (x > c.x0 && x < c.x1) {
        c.frac = rdiv(x - c.x0, c.x1 - c.x0);
        c.below = c.above = false;
    } else {
        bracket<Real>(grid, n, x, c.idx, c.frac, c.below, c.above, ti);
        c.x0 = grid[c.idx - 1];
        c.x1 = grid[c.idx];
    }
}

// The value at a bracket; off the table's ends the bracket is the end cell, whose
// outer value is held.
template <class Real, class T>
__device__ __forceinline__ Real gather(const T *f, int idx, Real frac, bool below, bool above) {
    const Real f0 = (Real)f[idx - 1], f1 = (Real)f[idx];
    const Real y = f0 + frac * (f1 - f0);
    return below ? f0 : above ? f1 : y;
}

// cxr/_recoil.py:35-76
template <class Real>
__device__ __forceinline__ void quantum_line_factors(Real h, Real gamma, Real vdg, Real k_dot_v,
                                                     Real k_dot_g, Real g2, Real k2, Real v_dot_e,
                                                     Real g_dot_e, Real k_dot_e, Real &pxr_num,
                                                     Real &f_cbs) {
    const Real gg = gamma * gamma;
    const Real n_1 = h * g2 - (Real)2 * gamma * vdg;
    const Real n_2 = n_1 + (Real)2 * h * k_dot_g;
    const Real n_f = h * (g2 + (Real)2 * k_dot_g + k2) - (Real)2 * gamma * (vdg + k_dot_v);
    const Real e_1 = r_sqrt(gg + h * n_1);
    const Real e_2 = r_sqrt(gg + h * (h * k2 - (Real)2 * gamma * k_dot_v));
    const Real e_f = r_sqrt(gg + h * n_f);
    const Real s_if = gamma + e_f;
    const Real ge_ke = g_dot_e + k_dot_e;
    pxr_num = rdiv(-n_f * ge_ke - k2 * ((Real)2 * gamma * v_dot_e - h * ge_ke), s_if);
    const Real s_1 = e_1 + gamma;
    const Real s_3 = e_1 + e_f;
    const Real s_4 = gamma + e_2;
    const Real x = (Real)2 * gamma * v_dot_e - h * k_dot_e;
    const Real sigma = s_if + e_1 + e_2;
    f_cbs = rdiv((Real)2 * g_dot_e * s_1, s_3 * n_1) +
            rdiv(x * (n_1 * rdiv(n_f, s_if) * sigma - (Real)2 * s_1 * s_4 * k_dot_g), s_3 * s_4 * n_1 * n_2);
}

// segment_escape.py:276-289. The float path switches to the series below
// d = 0.01, where 1 - exp(-d) in float would lose digits.
template <class Real>
__device__ __forceinline__ Real mean_transmission(Real t0, Real t1) {
    const Real lo = fmin(t0, t1);
    const Real d = fabs(t1 - t0);
    if constexpr (sizeof(Real) == 8) {
        const Real safe = d > (Real)1.0e-4 ? d : (Real)1;
        const Real ratio = d > (Real)1.0e-4 ? -r_expm1(-safe) / safe
                                             : (Real)1 - (Real)0.5 * d + d * d / (Real)6;
        return r_exp(-lo) * ratio;
    } else {
        const float ratio = d > 0.01f ? rdiv(1.0f - __expf(-d), d)
                                      : 1.0f - d * (0.5f - d * (1.0f / 6.0f - d * (1.0f / 24.0f)));
        return __expf(-lo) * ratio;
    }
}

// Layered escape of one (segment, direction): its pieces (pb_layers.cuh)
// with the exit-side depth inside the piece's layer at both ends, already
// divided by |n_z|.
template <class Real>
struct EscSeg {
    int np;
    int up;                 // exits through the entrance face (n_z < 0)
    Real inv_nz;
    int m[kMaxEscLayers];
    Real f[kMaxEscLayers], w0[kMaxEscLayers], w1[kMaxEscLayers];
};

template <class Real>
__device__ void esc_precompute(EscSeg<Real> &es, const pb_cxr_args &a, int64_t s, const double *nh,
                               const double *zt, const double *zb) {
    const double nz = nh[2];
    const double inv_nz = 1.0 / fmax(fabs(nz), 1.0e-12);
    const double half = 0.5 * a.L[s];
    const double z = a.r_mid[3 * s + 2], vz = a.v_hat[3 * s + 2];
    EscPiece pp[kMaxEscLayers];
    const int np = esc_pieces(z - half * vz, z + half * vz, a.n_layer, zt, zb, pp);
    es.np = np;
    es.up = nz < 0.0;
    es.inv_nz = (Real)inv_nz;
    for (int p = 0; p < np; ++p) {
        const double t = zb[pp[p].m] - zt[pp[p].m];
        es.m[p] = pp[p].m;
        es.f[p] = (Real)pp[p].f;
        es.w0[p] = (Real)((nz < 0.0 ? pp[p].u0 : t - pp[p].u0) * inv_nz);
        es.w1[p] = (Real)((nz < 0.0 ? pp[p].u1 : t - pp[p].u1) * inv_nz);
    }
}

// piece_mean_transmission (segment_escape.py:335-355) with every layer's
// exact mu at the line energy (cxr/_batched.py:702-720): the layers between
// a piece's layer and the exit face are crossed whole.
template <class Real>
__device__ Real esc_transmission(const EscSeg<Real> &es, const pb_cxr_args &a, const Real *lay_t, double E_eV) {
    Real mu[kMaxEscLayers], c[kMaxEscLayers];
    const int nl = a.n_layer;
#pragma unroll
    for (int k = 0; k < kMaxEscLayers; ++k) {
        mu[k] = 0;
        if (k < nl) {
            const int o = a.mu_off[k];
            mu[k] = (Real)esc_mu_at(a.mu_knot + o, a.mu_value + o, a.mu_slope + o, a.mu_off[k + 1] - o, E_eV);
        }
    }
    Real run = 0;
    if (es.up) {
#pragma unroll
        for (int k = 0; k < kMaxEscLayers; ++k) {
            c[k] = run;
            if (k < nl) run += mu[k] * lay_t[k];
        }
    } else {
#pragma unroll
        for (int k = kMaxEscLayers - 1; k >= 0; --k) {
            c[k] = run;
            if (k < nl) run += mu[k] * lay_t[k];
        }
    }
    Real T = 0;
    for (int p = 0; p < es.np; ++p) {
        const int m = es.m[p];
        const Real mm = esc_pick<Real>(mu, m), cm = esc_pick<Real>(c, m) * es.inv_nz;
        T += es.f[p] * mean_transmission<Real>(cm + mm * es.w0[p], cm + mm * es.w1[p]);
    }
    return T;
}

template <class Real>
struct Line {
    Real E_res, a_width, weight;
    bool good;
};

// Cheap test of whether a pair's resonance can reach the keep window under
// any refraction the table allows: omega <= 0 is never kept (denom > 0 is
// required); above the window, with D the largest |delta| the table holds at
// or above E_vac / 1.5, D |grad L| <= denom_vac / 2 keeps every root iterate
// (and so the root) at or above E_vac / 1.5, by induction over the passes.
template <class Real>
__device__ __forceinline__ bool pair_may_keep(const SegPre<Real> &sp, const RowPre<Real> &rw,
                                              const Real *E_tab, const Real *dtail, int n_tab,
                                              const pb_cxr_tables &t, const TabIndex &ti) {
    const Real r_num = (Real)0.5 * rw.g2 * sp.inv_E;
    const Real r_den = rw.n_dot_g * sp.inv_E;
    const Real num = (sp.vx * rw.G[0] + sp.vy * rw.G[1] + sp.vz * rw.G[2]) - r_num;
    const Real denom_vac = sp.denom_row + r_den;
    if (!sp.radiates || !(num > (Real)0) || !(denom_vac > (Real)0)) return false;
    if (dtail == nullptr) return true;
    const Real E_low = (Real)kHbarcEvAng * rdiv(num, denom_vac) * (Real)(1.0 / 1.5);
    if (E_low < (Real)t.hi_keep) return true;
    int ix = n_tab - 1;  // the tabulation usually ends at the window: the last cell
    if (!(E_low >= E_tab[n_tab - 1])) {
        Real fr;
        bool bl, ab;
        bracket<Real>(E_tab, n_tab, E_low, ix, fr, bl, ab, ti);
    }
    return !(dtail[ix - 1] * r_sqrt(sp.grad2) <= (Real)0.5 * denom_vac);
}

// The per-pair chain up to the complex PXR+CBS amplitude of both
// polarisations (cxr/_batched.py:461-559 and 789-826): the resonance (three
// Snell passes), the keep decision, the line's slope, the attenuation at the
// line energy and the amplitudes. Shared by the incoherent line (pair_line)
// and the coherent route's records (coh_records_kernel). ``E_tab`` /
// ``delta_tab`` / ``log_mu`` point at the shared-memory staging (or global
// memory for a large FP64 grid). The float path stops after the keep
// decision for dropped pairs.
template <class Real>
struct PairAmps {
    Real omega, E_res, slope, mu, v_dot_g, r_num, r_den;
    Real A_re[2], A_im[2];
    bool keep;
};

// The resonance of a pair: three Snell passes for the refraction at the line
// energy and the keep decision (delta and denom carry what the amplitude part
// needs; denom is NaN when the passes did not settle).
template <class Real>
struct Resonance {
    Real delta, denom;
    Cell<Real> cell;
    bool keep;
};

template <class Real>
__device__ __forceinline__ Resonance<Real> pair_resonance(const SegPre<Real> &sp, const RowPre<Real> &rw,
                                                          const Real *E_tab, const Real *delta_tab, int n_tab,
                                                          const pb_cxr_tables &t, const TabIndex &ti) {
    const Real Gx = rw.G[0], Gy = rw.G[1], Gz = rw.G[2];
    const Real g2 = rw.g2, n_dot_g = rw.n_dot_g;
    const Real hbarc = (Real)kHbarcEvAng;
    // cxr/_block_prologue.py:18-38, cxr/_recoil.py:79-97
    const Real r_num = (Real)0.5 * g2 * sp.inv_E;
    const Real r_den = n_dot_g * sp.inv_E;
    const Real v_dot_g = sp.vx * Gx + sp.vy * Gy + sp.vz * Gz;
    const Real v_dot_g_exact = v_dot_g - r_num;
    // (rounded as written, so that a float line lies at the same energy in the slab
    // and the layered instance: one ulp is 4e-3 eV at 40 keV)
    const Real denom_vac = sp.denom_row + r_mul(n_dot_g, sp.inv_E);
    // cxr/_kernels.py:702-765
    Real denom = denom_vac, previous = denom, delta = (Real)NAN;
    Cell<Real> cell;
    cell.x0 = cell.x1 = (Real)0;
    for (int pass = 0; pass < 3; ++pass) {
        const Real Er = hbarc * rdiv(v_dot_g_exact, denom);
        locate<Real>(cell, E_tab, n_tab, Er, ti);
        delta = gather<Real>(delta_tab, cell.idx, cell.frac, cell.below, cell.above);
        previous = denom;
        denom = denom_vac - delta * sp.v_dot_grad;
    }
    bool settled = fabs(denom - previous) <= (Real)1e-3 * fabs(denom);
    settled = settled && ((Real)2 * fabs(delta) * sp.grad2 < (Real)1);
    if (!settled) denom = (Real)NAN;
    const Real omega = rdiv(v_dot_g - r_num, denom);
    const Real E_res = hbarc * omega;
    bool keep = sp.radiates && (E_res > (Real)t.lo_keep) && (E_res > (Real)10) && (E_res < (Real)t.hi_keep);
    keep = keep && (denom > (Real)0) && (omega * sp.inv_E <= (Real)1 - rdiv((Real)1, sp.gamma));
    return Resonance<Real>{delta, denom, cell, keep};
}

// The rest of the chain from the resonance: the line's slope, the attenuation
// at the line energy and the complex amplitudes. The chain stops after the
// resonance for dropped pairs, unless ``all_pairs`` asks for the values of every
// pair (FP64 with per-pair output, which matches the reference's arrays).
template <class Real, bool kLayered>
__device__ __forceinline__ PairAmps<Real> pair_amps_from(const SegPre<Real> &sp, const RowPre<Real> &rw,
                                                         const Resonance<Real> &res, const Real *E_tab,
                                                         const Real *log_mu, int n_tab, int n_mu,
                                                         const pb_cxr_tables &t, const TabIndex &ti, bool all_pairs) {
    const Real Gx = rw.G[0], Gy = rw.G[1], Gz = rw.G[2];
    const Real g2 = rw.g2, n_dot_g = rw.n_dot_g;
    const Real hbarc = (Real)kHbarcEvAng;
    PairAmps<Real> o;
    const Real r_num = (Real)0.5 * g2 * sp.inv_E;
    const Real r_den = n_dot_g * sp.inv_E;
    const Real v_dot_g = sp.vx * Gx + sp.vy * Gy + sp.vz * Gz;
    o.r_num = r_num;
    o.r_den = r_den;
    o.v_dot_g = v_dot_g;
    const Real delta = res.delta, denom = res.denom;
    const Real n_dot_g_blk = n_dot_g + delta * (sp.gx * Gx + sp.gy * Gy + sp.gz * Gz);
    // cxr/_kernels.py:624-655
    const Real omega = rdiv(v_dot_g - r_num, denom);
    const Real k_dot_v = omega * (((Real)1 - denom) + r_den);
    const Real k_dot_g = omega * n_dot_g_blk;
    const Real detuning = g2 + (Real)2 * k_dot_g;
    // cxr/_batched.py:435-458
    const Real k_mag = omega * r_sqrt(sp.grad2 == (Real)0 ? (Real)1
                                                           : (Real)1 - (Real)2 * delta + delta * delta * sp.grad2);
    const Real E_res = hbarc * omega;
    o.omega = omega;
    o.E_res = E_res;
    o.mu = (Real)0;
    // cxr/_block_prologue.py:53-62, cxr/_recoil.py:100-118
    o.slope = denom * rdiv((Real)1, (Real)1 - omega * sp.inv_E);
    o.keep = res.keep;
    if (!res.keep && !(sizeof(Real) == 8 && all_pairs)) return o;
    Cell<Real> cell = res.cell;
    locate<Real>(cell, E_tab, n_tab, E_res, ti);
    const int ix = cell.idx;
    const Real fr = cell.frac;
    const bool bl = cell.below, ab = cell.above;
    Real lfr;
    {
        const Real x0 = cell.x0, x1 = cell.x1;
        Real bx = fmin(fmax(E_res, x0), x1);
        if (isnan(E_res)) bx = E_res;
        if constexpr (sizeof(Real) == 8) {
            lfr = r_log1p((bx - x0) / x0) / r_log1p((x1 - x0) / x0);
        } else {
            // cxr/_kernels.py:352-366 on a geometric grid: log(bx/x0)/h.
            lfr = ti.geometric ? __logf(rdiv(bx, x0)) * (float)ti.inv_h
                               : rdiv(log1pf(rdiv(bx - x0, x0)), log1pf(rdiv(x1 - x0, x0)));
        }
    }
    // cxr/_kernels.py:482-506 couplings, 369-388 attenuation
    const int64_t base = (int64_t)rw.row * n_tab;
    const Real chi_re = gather<Real>(t.chi_re + base, ix, fr, bl, ab);
    const Real chi_im = gather<Real>(t.chi_im + base, ix, fr, bl, ab);
    const Real u_re = gather<Real>(t.u_re + base, ix, fr, bl, ab);
    const Real u_im = gather<Real>(t.u_im + base, ix, fr, bl, ab);
    Real mu = 0;
    for (int el = 0; el < (kLayered ? 0 : n_mu); ++el) {
        const Real *lm = log_mu + (int64_t)el * n_tab;
        const Real f0 = lm[ix - 1], f1 = lm[ix];
        mu += r_exp(bl ? f0 : ab ? f1 : f0 + lfr * (f1 - f0));
    }
    o.mu = mu;
    // cxr/_batched.py:789-826, cxr/_line_amplitude.py:14-37
    const Real h = (Real)(kHbarcEvAng / kMeEv);
    const Real k2 = k_mag * k_mag;
#pragma unroll
    for (int pol = 0; pol < 2; ++pol) {
        const Real *Ev = pol == 0 ? rw.ES : rw.EP;
        const Real g_dot_e = pol == 0 ? rw.g_dot_es : rw.g_dot_ep;
        const Real v_dot_e = sp.vx * Ev[0] + sp.vy * Ev[1] + sp.vz * Ev[2];
        const Real k_dot_e = omega * delta * (sp.gx * Ev[0] + sp.gy * Ev[1] + sp.gz * Ev[2]);
        Real pxr_num, f_cbs;
        quantum_line_factors<Real>(h, sp.gamma, v_dot_g, k_dot_v, k_dot_g, g2, k2, v_dot_e, g_dot_e,
                                   k_dot_e, pxr_num, f_cbs);
        const Real f_pxr = rdiv(pxr_num, detuning);
        o.A_re[pol] = chi_re * f_pxr + u_re * f_cbs;
        o.A_im[pol] = chi_im * f_pxr + u_im * f_cbs;
    }
    return o;
}

template <class Real, bool kLayered>
__device__ __forceinline__ PairAmps<Real> pair_amps(const SegPre<Real> &sp, const RowPre<Real> &rw,
                                                    const Real *E_tab, const Real *delta_tab, const Real *log_mu,
                                                    int n_tab, int n_mu, const pb_cxr_tables &t,
                                                    const TabIndex &ti) {
    const Resonance<Real> res = pair_resonance<Real>(sp, rw, E_tab, delta_tab, n_tab, t, ti);
    return pair_amps_from<Real, kLayered>(sp, rw, res, E_tab, log_mu, n_tab, n_mu, t, ti, false);
}

// The incoherent line of a pair: resonance, width and weight
// (cxr/_batched.py:702-730, cxr/_kernels.py:658-668).
template <class Real, bool kLayered>
__device__ Line<Real> pair_line_from(const SegPre<Real> &sp, const RowPre<Real> &rw, const Resonance<Real> &res,
                                     const Real *E_tab, const Real *log_mu, int n_tab, int n_mu,
                                     const pb_cxr_tables &t, const TabIndex &ti, const EscSeg<Real> *es,
                                     const pb_cxr_args &a, const Real *lay_t) {
    const bool all_pairs = a.pair_E != nullptr;
    const PairAmps<Real> p = pair_amps_from<Real, kLayered>(sp, rw, res, E_tab, log_mu, n_tab, n_mu, t, ti, all_pairs);
    Line<Real> out;
    out.good = false;
    out.E_res = p.E_res;
    out.a_width = (Real)NAN;
    out.weight = (Real)NAN;
    if (!p.keep && !(sizeof(Real) == 8 && all_pairs)) return out;
    const Real A2 = (p.A_re[0] * p.A_re[0] + p.A_im[0] * p.A_im[0]) + (p.A_re[1] * p.A_re[1] + p.A_im[1] * p.A_im[1]);
    Real T_abs;
    if constexpr (kLayered) T_abs = esc_transmission<Real>(*es, a, lay_t, (double)p.E_res);
    else T_abs = mean_transmission<Real>(sp.path0 * p.mu, sp.path1 * p.mu);
    const Real pref_c1 = (Real)(4.0 * (kPi * kPi) * kHbarcEvAng);
    const Real pref = rdiv((Real)kAlphaFs * p.omega, pref_c1) * (sp.t_L * sp.t_L) * T_abs;
    out.a_width = rdiv(p.slope * sp.t_L, (Real)2 * (Real)kHbarcEvAng) * (Real)1;
    out.weight = pref * A2 * rw.wm;
    out.good = p.keep && isfinite(out.weight) && (out.weight > (Real)0);
    return out;
}

template <class Real, bool kLayered>
__device__ __forceinline__ Line<Real> pair_line(const SegPre<Real> &sp, const RowPre<Real> &rw, const Real *E_tab,
                                                const Real *delta_tab, const Real *log_mu, int n_tab, int n_mu,
                                                const pb_cxr_tables &t, const TabIndex &ti, const EscSeg<Real> *es,
                                                const pb_cxr_args &a, const Real *lay_t) {
    const Resonance<Real> res = pair_resonance<Real>(sp, rw, E_tab, delta_tab, n_tab, t, ti);
    return pair_line_from<Real, kLayered>(sp, rw, res, E_tab, log_mu, n_tab, n_mu, t, ti, es, a, lay_t);
}

// ---- the sinc^2 antiderivative ---------------------------------------------
// R(x) = F(x) - sign(x)/2, F the integral of sinc^2 from 0, for |x| < 8 in FP64:
// a Taylor polynomial of degree 23 about the middle c_k = 1/4 + k/2 of each half
// unit. With h = x - c_k, 1 - cos 2 pi x = 1 + (-1)^k sin 2 pi h exactly, so
// sinc^2(x) = (1 - cos 2 pi x) / (2 pi^2 (c_k + h)^2) has its coefficients from
// the recurrence of a division by (c_k + h)^2; integrated term by term and
// matched at the interval ends from R(0) = -1/2. Truncation: the n-th term is
// below (pi/2)^n / n! at |h| = 1/4, 1e-19 for n = 24; the recurrence's rounding
// stays below 1e-14 (it grows as n (h / c_k)^n). 23 multiply-adds replace a
// 31-term series of the sine integral below |x| = 2.1 and a continued fraction
// with two divisions a step above.
constexpr int kSincParts = 16, kSincDeg = 23;
struct SincTable {
    double c[kSincParts][kSincDeg + 1];
};
__host__ __device__ constexpr SincTable make_sinc_table() {
    SincTable t{};
    double left = -0.5;  // R at the left end of the interval
    for (int k = 0; k < kSincParts; ++k) {
        const double c = 0.25 + 0.5 * k, sg = (k & 1) ? -1.0 : 1.0;
        double s[kSincDeg + 1] = {}, f = 1.0;  // f = (2 pi)^n / n!
        for (int n = 0; n <= kSincDeg; ++n) {
            double num = n == 0 ? 1.0 : 0.0;
            if (n > 0) {
                f *= 2.0 * kPi / n;
                if (n & 1) num = ((n >> 1) & 1) ? -sg * f : sg * f;
            }
            num /= 2.0 * kPi * kPi;
            s[n] = (num - (n > 0 ? 2.0 * c * s[n - 1] : 0.0) - (n > 1 ? s[n - 2] : 0.0)) / (c * c);
        }
        double lo = 0.0, hi = 0.0;  // the polynomial without its constant at h = -1/4, 1/4
        for (int n = kSincDeg; n > 0; --n) {
            t.c[k][n] = s[n - 1] / n;
            lo = (lo + t.c[k][n]) * -0.25;
            hi = (hi + t.c[k][n]) * 0.25;
        }
        t.c[k][0] = left - lo;
        left = t.c[k][0] + hi;
    }
    return t;
}
__device__ const SincTable kSincTable = make_sinc_table();

__device__ __forceinline__ double sincsq_tail(double x) {
    const double u = fabs(x);
    const int k = min((int)(2.0 * u), kSincParts - 1);
    const double h = u - (0.25 + 0.5 * k);
    const double *c = kSincTable.c[k];
    double r = c[kSincDeg];
#pragma unroll
    for (int n = kSincDeg - 1; n >= 0; --n) r = fma(r, h, c[n]);
    return x >= 0.0 ? r : -r;
}

// sin and cos of 2 pi x: the quarter turn nearest to x is taken off (adding and
// subtracting 1.5 2^52 rounds 4 x, |x| < 2^48), the rest, within an eighth of a
// turn, goes to the Taylor series (terms to g^15 and g^16: truncation 5e-17),
// about half the issue slots of the library's sincospi, whose argument is not
// limited to a few thousand turns.
struct TurnSeries {
    double s[8], c[9];
};
__host__ __device__ constexpr TurnSeries make_turn_series() {
    TurnSeries t{};
    double f = 1.0;  // (2 pi)^n / n!
    for (int n = 0; n <= 16; ++n) {
        if (n > 0) f *= 2.0 * kPi / n;
        const double v = ((n >> 1) & 1) ? -f : f;
        if (n & 1) t.s[n >> 1] = v;
        else t.c[n >> 1] = v;
    }
    return t;
}
__device__ __forceinline__ void sincos_turns(double x, double &sn, double &cs) {
    constexpr TurnSeries t = make_turn_series();
    constexpr double kRound = 6755399441055744.0;  // 1.5 2^52
    const double m = __dadd_rn(4.0 * x, kRound);
    const int q = __double2loint(m);
    const double g = fma(__dsub_rn(m, kRound), -0.25, x);
    const double y = g * g;
    double s = t.s[7], c = t.c[8];
#pragma unroll
    for (int k = 6; k >= 0; --k) s = fma(s, y, t.s[k]);
#pragma unroll
    for (int k = 7; k >= 0; --k) c = fma(c, y, t.c[k]);
    s *= g;
    const double a = (q & 1) ? c : s, b = (q & 1) ? s : c;
    sn = (q & 2) ? -a : a;
    cs = ((q + 1) & 2) ? -b : b;
}

constexpr double kInvPi = 1.0 / kPi;
constexpr double kInv2Pi2 = 1.0 / (2.0 * kPi * kPi);

struct BinAxis {
    const double *edges;
    int n;
    double lo, w, inv_w;  // uniform axis: edges[b] = lo + b w
    bool uniform;
    int pad;              // virtual centre bins on each side (uniform axes)
};

__device__ __forceinline__ int bin_of(const BinAxis &ax, double E) {
    if (ax.uniform) return (int)floor((E - ax.lo) * ax.inv_w);
    if (E < ax.edges[0]) return -1;
    if (E >= ax.edges[ax.n]) return ax.n;
    int lo = 0, hi = ax.n;  // last edge index with edges[b] <= E
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (ax.edges[mid] <= E) lo = mid; else hi = mid;
    }
    return lo;
}

__device__ __forceinline__ double centre_of(const BinAxis &ax, int c) {
    if (ax.uniform) return ax.lo + ((double)c + 0.5) * ax.w;
    return 0.5 * (ax.edges[c] + ax.edges[c + 1]);
}

// Oscillatory part of the sinc^2 antiderivative beyond the asymptotic
// threshold (Abramowitz & Stegun 5.2.8, 5.2.34-35): with u = 2 pi |x|,
//   int sinc^2 = (1/(2 pi^2)) (1/x_a - 1/x_b) + (1/pi) [Q(u)]_a^b,
//   Q(u) = cos u (1/u - f(u)) - g(u) sin u,
// where 1/u - f(u) ~ (1/u) sum_{k>=1} (-1)^(k+1) (2k)!/u^2k and
// g(u) ~ (1/u^2) sum_{k>=0} (-1)^k (2k+1)!/u^2k. The envelope term carries
// the mass without the cancellation of a difference of antiderivatives.
constexpr int kOscTerms = 13;  // the first omitted one at u = 48 is below 1e-17 of the leading
struct OscSeries {
    double c1[kOscTerms], c2[kOscTerms];  // (-1)^k (2k+2)!, (-1)^k (2k+1)!
};
__host__ __device__ constexpr OscSeries make_osc_series() {
    OscSeries s{};
    double f = 1.0;
    for (int k = 0; k < kOscTerms; ++k) {
        f *= 2.0 * k + 1.0;
        s.c2[k] = (k & 1) ? -f : f;
        f *= 2.0 * k + 2.0;
        s.c1[k] = (k & 1) ? -f : f;
    }
    return s;
}

// Far limit of an edge: |x| past u = 2 pi |x| = 24 (float) or 48 (FP64).
template <class R>
__device__ __forceinline__ constexpr R far_limit() { return (R)((sizeof(R) == 4 ? 24.0 : 48.0) / (2.0 * kPi)); }

// sign(x) Q(2 pi |x|) with iu = 1 / (2 pi x) given (Q is odd in x and iu).
__device__ __forceinline__ double q_osc(double x, double iu) {
    constexpr OscSeries c = make_osc_series();
    const double y = iu * iu;
    double p1, p2;
    if (fabs(iu) < 1.0 / 200.0) {
        // u > 200: six terms reach 14!/200^12 < 3e-17 of the leading one,
        // three of them 8!/3000^6 < 6e-17 past u = 3000.
        p1 = c.c1[2];
        p2 = c.c2[2];
        if (fabs(iu) > 1.0 / 3000.0) {
            p1 = c.c1[5];
            p2 = c.c2[5];
#pragma unroll
            for (int k = 4; k >= 2; --k) { p1 = fma(p1, y, c.c1[k]); p2 = fma(p2, y, c.c2[k]); }
        }
#pragma unroll
        for (int k = 1; k >= 0; --k) { p1 = fma(p1, y, c.c1[k]); p2 = fma(p2, y, c.c2[k]); }
    } else {
        p1 = c.c1[kOscTerms - 1];
        p2 = c.c2[kOscTerms - 1];
#pragma unroll
        for (int k = kOscTerms - 2; k >= 0; --k) { p1 = fma(p1, y, c.c1[k]); p2 = fma(p2, y, c.c2[k]); }
    }
    double sn, cs;
    sincos_turns(x, sn, cs);
    return y * (cs * p1 * iu - sn * p2);
}
__device__ __forceinline__ float q_osc(float x, float iu) {
    const float y = iu * iu;
    const float p1 = 2.0f + y * (-24.0f + y * (720.0f + y * (-40320.0f + y * 3628800.0f)));
    const float p2 = 1.0f + y * (-6.0f + y * (120.0f + y * (-5040.0f + y * 362880.0f)));
    // x to [-1/2, 1/2] turns by adding and taking off 1.5 2^23 (an FADD each
    // where the rounding instruction runs at the SFU's rate).
    constexpr float kRound = 12582912.0f;
    float sn, cs;
    __sincosf(6.28318530717958648f * (x - __fsub_rn(__fadd_rn(x, kRound), kRound)), &sn, &cs);
    return y * (cs * p1 * iu - sn * p2);
}

// Bin-mean deposit of a line: exact bin integrals within the line's window
// (``exact_widths`` first-zero widths, at least K_far bins); beyond it the far
// envelope w/(2 a^2) / ((E_lo - E_r)(E_hi - E_r)) is carried by three moments
// about the centre bin and spread by far_field_conv_kernel onto every bin more
// than K_far bins away. A line whose window is wider than K_far removes the
// envelope again from its extra exact bins, so each bin takes exactly one of
// the two forms. Lines centred off a non-uniform axis, or too wide for a
// window, are integrated exactly over the whole axis.
struct LineWindow {
    int c;        // centre bin (may lie off the axis)
    int b0, nb;   // first exact bin and count
    int K;        // half width of the window [bins]
    bool mom;     // far field through the moments
};

__device__ __forceinline__ LineWindow line_window(double E_r, double inv_a, const BinAxis &ax,
                                                  double exact_widths, int K_far, bool moments) {
    const int n = ax.n;
    LineWindow lw;
    lw.c = bin_of(ax, E_r);
    lw.mom = moments && K_far > 0 && lw.c >= -ax.pad && lw.c < n + ax.pad;
    int K;
    if (!lw.mom) {
        K = n + (lw.c < 0 ? -lw.c : (lw.c >= n ? lw.c - n + 1 : 0));
    } else {
        const double kk = ceil(exact_widths * kPi * (inv_a * ax.inv_w));
        K = kk > (double)(2 * n) ? 2 * n : (kk < (double)K_far ? K_far : (int)kk);
    }
    int b0 = lw.c - K, b1 = lw.c + K;
    if (b0 < 0) b0 = 0;
    if (b1 > n - 1) b1 = n - 1;
    lw.b0 = b0;
    lw.K = K;
    lw.nb = b1 >= b0 ? b1 - b0 + 1 : 0;
    return lw;
}

// Mean of sinc^2 over [xc - dx/2, xc + dx/2] by its midpoint Taylor series
// f + f2 dx^2/24 + f4 dx^4/1920 + f6 dx^6/322560, f = (1 - cos 2 pi x)/(2 pi^2 x^2),
// with the derivatives by the Leibniz rule on (1 - cos 2 pi x) and x^-2
// (montecarlo/spectrum/cxr/_bin_quadrature.py:179-221, the reference's
// device bin mean, on by default there). Valid for dx <= 0.1 and |xc| >= 2, where the omitted term is below
// 2.5e-9 of the envelope 1/(2 pi^2 xc^2).
__device__ __forceinline__ double sincsq_midpoint_mean(double xc, double dx) {
    double sp, cp;  // of pi xc
    sincos_turns(0.5 * xc, sp, cp);
    const double om = 2.0 * kPi;
    const double a0 = 2.0 * sp * sp;
    const double s2 = 2.0 * sp * cp;
    const double c2 = (cp - sp) * (cp + sp);
    const double a1 = om * s2, a2 = om * om * c2;
    const double om3 = om * om * om;
    const double a3 = -om3 * s2, a4 = -om3 * om * c2;
    const double a5 = om3 * om * om * s2, a6 = om3 * om3 * c2;
    const double q = 1.0 / xc;
    const double h0 = q * q;
    const double h1 = -2.0 * h0 * q;
    const double h2 = -3.0 * h1 * q;
    const double h3 = -4.0 * h2 * q;
    const double h4 = -5.0 * h3 * q;
    const double h5 = -6.0 * h4 * q;
    const double h6 = -7.0 * h5 * q;
    const double f0 = a0 * h0;
    const double f2 = a2 * h0 + 2.0 * a1 * h1 + a0 * h2;
    const double f4 = a4 * h0 + 4.0 * a3 * h1 + 6.0 * a2 * h2 + 4.0 * a1 * h3 + a0 * h4;
    const double f6 = a6 * h0 + 6.0 * a5 * h1 + 15.0 * a4 * h2 + 20.0 * a3 * h3 + 15.0 * a2 * h4 + 6.0 * a1 * h5 +
                      a0 * h6;
    const double d2 = dx * dx;
    const double series = f0 + d2 * (f2 * (1.0 / 24.0) + d2 * (f4 * (1.0 / 1920.0) + d2 * (f6 * (1.0 / 322560.0))));
    return series * kInv2Pi2;
}

// Reciprocal on the SFU alone (rcp.approx, about 1 ulp): the mixed path's
// bin forms carry float rounding far below their tolerance.
__device__ __forceinline__ float rcp_fast(float x) {
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ double rcp_fast(double x) { return 1.0 / x; }

// R(x) of sincsq_tail in float:
// Si(t) - pi/2 = -f(t) cos t - g(t) sin t with t = 2 pi |x| and the rational
// auxiliary functions of Abramowitz & Stegun 5.2.38-5.2.39 (|error| < 5e-7 for
// t >= 1); its Maclaurin series below t = 1.
__device__ __forceinline__ float sincsq_tail_f32(float x) {
    const float u = fabsf(x);
    const float red = u - rintf(u);
    float sp, cp;
    __sincosf(3.14159265358979324f * red, &sp, &cp);  // sin(pi u) up to sign
    const float t = 6.28318530717958648f * u;
    const float t2 = t * t;
    float si_m;  // Si(t) - pi/2
    if (t < 1.0f) {
        si_m = t * (1.0f + t2 * (-1.0f / 18.0f + t2 * (1.0f / 600.0f + t2 * (-1.0f / 35280.0f + t2 * (1.0f / 3265920.0f))))) -
               1.57079632679489662f;
    } else {
        const float f = __fdividef(t2 * (t2 * (t2 * (t2 + 38.027264f) + 265.187033f) + 335.677320f) + 38.102495f,
                                   (t2 * (t2 * (t2 * (t2 + 40.021433f) + 322.624911f) + 570.236280f) + 157.105423f) * t);
        const float g = __fdividef(t2 * (t2 * (t2 * (t2 + 42.242855f) + 302.757865f) + 352.018498f) + 21.821899f,
                                   (t2 * (t2 * (t2 * (t2 + 48.196927f) + 482.485984f) + 1114.978885f) + 449.690326f) * t2);
        const float sin_t = 2.0f * sp * cp, cos_t = (cp - sp) * (cp + sp);
        si_m = -f * cos_t - g * sin_t;
    }
    const float lobe = u > 0.0f ? __fdividef(sp * sp, 9.86960440108935862f * u) : 0.0f;
    const float r = si_m * (float)kInvPi - lobe;
    return x >= 0.0f ? r : -r;
}

// Mean of sinc^2 over a bin of width dx in first-zero units centred on xc
// (the midpoint series of sincsq_midpoint_mean), in float.
__device__ __forceinline__ float sincsq_midpoint_mean_f32(float xc, float dx) {
    const float red = xc - 2.0f * rintf(0.5f * xc);
    float sp, cp;
    __sincosf(3.14159265358979324f * red, &sp, &cp);
    const float om = 6.28318530717958648f;
    const float a0 = 2.0f * sp * sp;
    const float s2 = 2.0f * sp * cp;
    const float c2 = (cp - sp) * (cp + sp);
    const float a1 = om * s2, a2 = om * om * c2;
    const float om3 = om * om * om;
    const float a3 = -om3 * s2, a4 = -om3 * om * c2;
    const float a5 = om3 * om * om * s2, a6 = om3 * om3 * c2;
    const float q = __frcp_rn(xc);
    const float h0 = q * q;
    const float h1 = -2.0f * h0 * q;
    const float h2 = -3.0f * h1 * q;
    const float h3 = -4.0f * h2 * q;
    const float h4 = -5.0f * h3 * q;
    const float h5 = -6.0f * h4 * q;
    const float h6 = -7.0f * h5 * q;
    const float f0 = a0 * h0;
    const float f2 = a2 * h0 + 2.0f * a1 * h1 + a0 * h2;
    const float f4 = a4 * h0 + 4.0f * a3 * h1 + 6.0f * a2 * h2 + 4.0f * a1 * h3 + a0 * h4;
    const float f6 = a6 * h0 + 6.0f * a5 * h1 + 15.0f * a4 * h2 + 20.0f * a3 * h3 + 15.0f * a2 * h4 +
                     6.0f * a1 * h5 + a0 * h6;
    const float d2 = dx * dx;
    const float series = f0 + d2 * (f2 * (1.0f / 24.0f) + d2 * (f4 * (1.0f / 1920.0f) + d2 * (f6 * (1.0f / 322560.0f))));
    return series * (float)kInv2Pi2;
}

__device__ __forceinline__ float tail_of(float x) { return sincsq_tail_f32(x); }
__device__ __forceinline__ double tail_of(double x) { return sincsq_tail(x); }
__device__ __forceinline__ float midpoint_mean(float xc, float dx) { return sincsq_midpoint_mean_f32(xc, dx); }
__device__ __forceinline__ double midpoint_mean(double xc, double dx) { return sincsq_midpoint_mean(xc, dx); }

// ---- the deposit as a function of bin edges --------------------------------
// pi times the mass of sinc^2 in a bin is a difference of one function of its
// edges, pi R(x) = pi (F(x) - sign(x)/2) (plus pi in the bin that holds x = 0).
// Past the far limit pi R(x) = Q(x) - 1/(2 pi x), both odd in x, which float
// keeps without cancellation for bins wider than 0.1 first-zero widths; narrower
// ones take the midpoint series away from the centre.
//
// Where the moments spread the far envelope of the line (bins more than K_far
// from its centre bin c), the exact window takes that envelope back out. Its
// expansion about the centre is itself a difference over the bin's edges: with
// Dm the edge's distance from the centre of bin c in bins, d = (E_r - E_c) / w
// and A = s w Dm (first-zero units), the spread f0 + f1 d + f2 d^2 is
// [T(A) - T(B)] / (B - A) with T(A) = (1 + t + t^2) / A, t = d / Dm. So
//   pi R(x) + T(A) / (2 pi)
// is the edge function there, and past the far limit, since x = A (1 - t),
// 1/x - T(A) = t^3 / x makes it Q(x) - t^3 / (2 pi x): the envelope and its
// expansion never meet as two large numbers.
template <class R>
__device__ __forceinline__ R edge_near_bins(R x) {
    if (fabs(x) >= far_limit<R>()) {
        const R iu = rcp_fast((R)(2.0 * kPi) * x);
        return q_osc(x, iu) - iu;
    }
    return (R)kPi * tail_of(x);
}

// x and Dm of one sign (an edge outside the centre bin).
template <class R>
__device__ __forceinline__ R edge_window_far(R x, R Dm, R d) {
    const R ux = (R)(2.0 * kPi) * x;
    const R r = rcp_fast(ux * Dm);  // one reciprocal for 1/(2 pi x) and 1/Dm
    const R iu = r * Dm;
    const R t = d * (r * ux);
    return q_osc(x, iu) - (iu * t) * (t * t);
}

// sw: the bin width in first-zero units.
template <class R>
__device__ __forceinline__ R edge_window_near(R x, R Dm, R d, R sw) {
    const R iD = rcp_fast(Dm);
    const R t = d * iD;
    return (R)kPi * tail_of(x) + (R)(0.5 / kPi) * (iD * rcp_fast(sw)) * fma(t, t, (R)1 + t);
}

// The edge function of a window edge.
template <class R>
__device__ __forceinline__ R edge_window_bins(R x, R Dm, R d, R sw) {
    if (fabs(x) >= far_limit<R>()) return edge_window_far<R>(x, Dm, d);
    return edge_window_near<R>(x, Dm, d, sw);
}

// What the moments spread into a bin whose left edge is Dm from the centre bin's
// centre, [T(A) - T(B)] / (2 pi), as a product: a line far wider than the axis
// spreads an envelope as large as an ordinary line's although its own mass is
// next to nothing, and a difference of T over the edges would leave 1e-7 Dm of
// that envelope behind in float (1e-4 at 1,000 bins; the product 5e-7). Powers of
// the distance in bins stay in float's range however short the segment is.
template <class R>
__device__ __forceinline__ R spread_envelope(R Dm, R d, R sw) {
    const R ra = rcp_fast(Dm), rb = rcp_fast(Dm + (R)1);
    const R sum = ra + rb;
    return (R)(0.5 / kPi) * rcp_fast(sw) * (ra * rb) * ((R)1 + d * (sum + d * fma(ra, sum, rb * rb)));
}

// pi times the mass of a bin of at most 0.1 first-zero widths, |xc| >= 2, by the
// midpoint series, less the spread envelope: Dm its left edge, xc its centre.
template <class R>
__device__ __forceinline__ R window_midpoint(R xc, R Dm, R d, R sw) {
    return sw * (R)kPi * midpoint_mean(xc, sw) - spread_envelope<R>(Dm, d, sw);
}

// One line of the window list, read back as broadcasts.
template <class R>
struct alignas(16) WinLine {
    R s, scale, d, E_r;   // a / pi, w / a, (E_r - E_c) / bin width
    int c, D0, D1;        // centre bin, window bins D0 <= |b - c| <= D1 on the axis
    int pad;
};

__device__ __forceinline__ void smem_add(double *p, double v) {
    asm volatile("red.shared.add.f64 [%0], %1;" ::"r"((uint32_t)__cvta_generic_to_shared(p)), "d"(v) : "memory");
}

// A kept line's three far-field moments about its centre bin, added to the
// direction's moments in global memory (L2 reductions: a few per kept line,
// so the block keeps no on-chip copy of the moment array).
__device__ __forceinline__ void line_moments(double E_r, double inv_a, double w, const LineWindow &lw,
                                             const BinAxis &ax, double *mom) {
    const int slot = lw.c + ax.pad;
    const double m = 0.5 * w * (inv_a * inv_a);
    const double dd = E_r - centre_of(ax, lw.c);
    atomicAdd(&mom[3 * slot + 0], m);
    atomicAdd(&mom[3 * slot + 1], m * dd);
    atomicAdd(&mom[3 * slot + 2], m * dd * dd);
}

// Persistent blocks over the flattened (direction, row chunk, segment tile) work,
// in contiguous ranges, so the grid is an exact multiple of the SM count; a
// block flushes its on-chip spectrum whenever its direction changes.
// Per pass (a segment tile x a chunk of reflection rows):
//   A0  a cheap prefilter drops pairs whose resonance cannot reach the keep
//       window and compacts the survivors into a shared queue (warp ballots);
//   A1  the full chain runs over the survivors in whole rounds of one per thread
//       (the rest waits for the next tile's; its own tile stays staged until
//       then) and pushes kept lines onto a second shared queue. (Rounds of each
//       tile alone: 2.27 -> 2.14 ms for 14,500 segments, 16 directions, 238 rows
//       with two-width windows, 78.2 -> 75.9 for 8,192 histories with 64.)
//   B1  lines leave the queue in whole rounds of one per thread (the rest
//       waits for the next pass): the owner thread adds the line's far-field
//       moments and the bins within K_far of its centre, and passes lines
//       whose exact window is wider on to a window list;
//   B2  when the window list is full, groups of 4 to 32 lanes (by the window's
//       width) take a line each: a lane holds two bin edges, evaluates the edge
//       function once each and gets the third from the next lane. The widest
//       windows wait for more of their kind and are summed strip by strip.
// B is bound by FP32/FP64 issue and the SFU (one reciprocal, one sine, one
// cosine per edge).
template <class Real, bool kLayered>
__global__ void __launch_bounds__(kCxrThreads, kCxrBlocks) cxr_kernel(const pb_cxr_args a, int K_far, int far_pad,
                                                                         bool tab_smem) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    constexpr bool kMixed = sizeof(Real) == 4;
    const int n_g = a.tables.n_g;
    const int n_tab = a.tables.n_tab;
    const int n_mu = a.tables.n_mu;
    const bool binmean = a.quadrature == PB_QUAD_BINMEAN;
    const int n_E = a.n_E;
    int64_t n_seg = a.n_seg;
    if (a.n_seg_device) n_seg = (int64_t)*a.n_seg_device;
    if (n_seg > a.n_seg && a.n_seg > 0) n_seg = a.n_seg;

    // Shared layout: [rows][segs][queues][tables][spec][float edges][escape pieces]
    unsigned char *cur = smem_raw;
    RowPre<Real> *rows = reinterpret_cast<RowPre<Real> *>(cur);
    constexpr int kRowChunk = row_chunk<Real>();
    constexpr int kQueue = surv_queue<Real>();
    constexpr int kPairs = pair_queue<Real>();
    cur += sizeof(RowPre<Real>) * kRowChunk;
    SegPre<Real> *segs = reinterpret_cast<SegPre<Real> *>(cur);
    cur += sizeof(SegPre<Real>) * 2 * kSegTile;  // this tile and the last one
    cur = (unsigned char *)(((uintptr_t)cur + 15) & ~(uintptr_t)15);
    constexpr int kLineQueue = line_queue<Real>();
    Real *qE = reinterpret_cast<Real *>(cur);
    Real *qA = qE + kLineQueue;
    Real *qW = qA + kLineQueue;
    cur = (unsigned char *)(((uintptr_t)(qW + kLineQueue) + 15) & ~(uintptr_t)15);
    WinLine<Real> *wLine = reinterpret_cast<WinLine<Real> *>(cur);  // window list
    uint16_t *wIdx = reinterpret_cast<uint16_t *>(wLine + kWideCap);  // its lines by class
    int *scratch = reinterpret_cast<int *>(wIdx + kWinClasses / 2 * kWideCap);  // counters
    uint16_t *pq = reinterpret_cast<uint16_t *>(scratch + 64);  // surviving pair ids
    cur = reinterpret_cast<unsigned char *>(pq + kQueue);
    cur = (unsigned char *)(((uintptr_t)cur + 15) & ~(uintptr_t)15);
    Real *E_tab_s = reinterpret_cast<Real *>(cur);
    Real *delta_s = E_tab_s + (tab_smem ? n_tab : 0);
    Real *logmu_s = delta_s + (tab_smem ? n_tab : 0);
    Real *dtail_s = logmu_s + (tab_smem ? n_tab * n_mu : 0);
    const bool has_dtail = tab_smem && a.tables.delta_tail_absmax != nullptr && a.pair_E == nullptr;
    cur = reinterpret_cast<unsigned char *>(dtail_s + (tab_smem ? n_tab : 0));
    cur = (unsigned char *)(((uintptr_t)cur + 15) & ~(uintptr_t)15);
    double *spec_s = reinterpret_cast<double *>(cur);
    const int n_mom = n_E + 2 * far_pad;
    float *edges_f = reinterpret_cast<float *>(spec_s + (binmean ? n_E : 0));  // mixed path: float bin edges
    // Layered absorber: per-segment escape pieces, layer thicknesses and bounds.
    unsigned char *esc_raw = reinterpret_cast<unsigned char *>(edges_f + (binmean && kMixed ? n_E + 1 : 0));
    esc_raw = (unsigned char *)(((uintptr_t)esc_raw + 15) & ~(uintptr_t)15);
    EscSeg<Real> *esc = reinterpret_cast<EscSeg<Real> *>(esc_raw);
    double *lay_zt = reinterpret_cast<double *>(esc + (kLayered ? 2 * kSegTile : 0));
    double *lay_zb = lay_zt + (kLayered ? kMaxEscLayers : 0);
    Real *lay_t = reinterpret_cast<Real *>(lay_zb + (kLayered ? kMaxEscLayers : 0));
    int &q_count = scratch[40];
    int &p_count = scratch[42];
    int &w_count = scratch[43];
    int *w_class = scratch + 48;  // lines per class
    int &strip_next = scratch[44];

    const int tid = threadIdx.x;
    const unsigned lane = tid & 31u;
    const int warp = tid >> 5, n_warps = kCxrThreads / 32;
    if (tab_smem) {
        for (int j = tid; j < n_tab; j += blockDim.x) {
            E_tab_s[j] = (Real)a.tables.E_tab[j];
            delta_s[j] = (Real)a.tables.delta[j];
            if (has_dtail) dtail_s[j] = (Real)a.tables.delta_tail_absmax[j];
        }
        for (int j = tid; j < n_tab * n_mu; j += blockDim.x) logmu_s[j] = (Real)a.tables.log_mu[j];
    }
    const Real *dtail = has_dtail ? dtail_s : nullptr;
    if (binmean) {
        for (int j = tid; j < n_E; j += blockDim.x) spec_s[j] = 0.0;
        if (kMixed)
            for (int j = tid; j <= n_E; j += blockDim.x) edges_f[j] = (float)a.edges[j];
    }
    if (tid == 0) { q_count = 0; p_count = 0; w_count = 0; strip_next = 0; }
    if (tid < kWinClasses) w_class[tid] = 0;
    if constexpr (kLayered) {
        if (tid < a.n_layer) {
            lay_zt[tid] = a.z_top[tid];
            lay_zb[tid] = a.z_bot[tid];
            lay_t[tid] = (Real)(a.z_bot[tid] - a.z_top[tid]);
        }
        if (tid == 0) {
            // Contiguous layers in depth order, as the pieces assume.
            int bad = 0;
            for (int k = 0; k < a.n_layer; ++k) {
                if (!(a.z_bot[k] > a.z_top[k])) bad = 1;
                if (k + 1 < a.n_layer && fabs(a.z_bot[k] - a.z_top[k + 1]) > 1e-9 * fmax(1.0, fabs(a.z_bot[k])))
                    bad = 1;
            }
            scratch[46] = bad;
            if (bad && a.status) atomicOr(a.status, PB_DEV_BAD_INPUT);
        }
    }
    const Real *E_tab = tab_smem ? E_tab_s : reinterpret_cast<const Real *>(a.tables.E_tab);
    const Real *delta_tab = tab_smem ? delta_s : reinterpret_cast<const Real *>(a.tables.delta);
    const Real *log_mu = tab_smem ? logmu_s : reinterpret_cast<const Real *>(a.tables.log_mu);

    TabIndex ti{};
    ti.geometric = a.tables.tab_log_step > 0.0;
    ti.log0 = a.tables.tab_log0;
    ti.inv_h = ti.geometric ? 1.0 / a.tables.tab_log_step : 0.0;

    BinAxis ax{};
    if (binmean) {
        ax.edges = a.edges;
        ax.n = n_E;
        ax.uniform = K_far > 0;  // the launcher enables moments on uniform axes only
        ax.lo = a.edges[0];
        ax.w = (a.edges[n_E] - a.edges[0]) / n_E;
        ax.inv_w = 1.0 / ax.w;
        ax.pad = far_pad;
    }
    __syncthreads();
    if (kLayered && scratch[46]) return;

    const int n_chunks = (n_g + kRowChunk - 1) / kRowChunk;
    int seg_tile = kSegTile;
    while (seg_tile > 4 && (n_seg + seg_tile - 1) / seg_tile * a.n_dir * n_chunks < 4 * (int64_t)gridDim.x)
        seg_tile >>= 1;
    const int64_t n_tiles = (n_seg + seg_tile - 1) / seg_tile;
    const int64_t n_work = n_tiles * a.n_dir * n_chunks;
    const int64_t w_begin = n_work * blockIdx.x / gridDim.x;
    const int64_t w_end = n_work * (blockIdx.x + 1) / gridDim.x;
    const bool pairs_out = a.pair_E != nullptr;
    const bool lines_out = a.line_E != nullptr;
    const double exact_widths = K_far > 0 ? a.exact_widths : 0.0;
    const Real w_r = (Real)ax.w, inv_w_r = (Real)ax.inv_w;
    const Real s_narrow = (Real)(0.1 * ax.inv_w);  // uniform axis: bins of 0.1 first-zero widths
    // Bin edge j, clamped to the axis (a clamped edge bounds no bin).
    const auto edge_at = [&](int j) {
        j = min(max(j, 0), n_E);
        if constexpr (kMixed) return edges_f[j];
        else return ax.edges[j];
    };
    int d_cur = -1;

    // B1: the line in queue slot j, if any, by this thread.
    auto near_round = [&](int j, int d) {
        int cls = kWinClasses;
        WinLine<Real> wl{};
        if (j >= 0) {
            const double Ed = (double)qE[j], wd = (double)qW[j], inv_a = 1.0 / (double)qA[j];
            const LineWindow lw = line_window(Ed, inv_a, ax, exact_widths, K_far, K_far > 0);
            const Real sx = (Real)(kMixed ? (float)qA[j] * (float)kInvPi : (double)qA[j] * kInvPi);
            wl.E_r = qE[j];
            wl.s = sx;
            wl.scale = (Real)(wd * inv_a);
            if (a.counters) {
                atomicAdd(&a.counters[0], 1ULL);
                atomicAdd(&a.counters[1], (unsigned long long)lw.nb);
            }
            if (lw.mom) {
                line_moments(Ed, inv_a, wd, lw, ax, a.far_moments + (int64_t)d * n_mom * 3);
                const Real sw = sx * w_r;
                wl.d = (Real)((Ed - centre_of(ax, lw.c)) * ax.inv_w);
                wl.c = lw.c;
                if (lw.nb > 0) {
                    // window bins on the axis, by distance from the centre bin
                    const int left = lw.c - lw.b0, right = lw.b0 + lw.nb - 1 - lw.c;
                    wl.D0 = max(K_far + 1, max(-left, -right));
                    wl.D1 = max(left, right);
                    const int span = wl.D1 - wl.D0 + 1;
                    if (span > 0)
                        cls = span <= 3 ? kWin4 : span <= 7 ? kWin8 : span <= 15 ? kWin16 : span <= kStripSpan ? kWin32 : kWinStrip;
                    // bins narrower than 0.1 first-zero widths take the midpoint series
                    if (span > 0 && sx <= s_narrow) cls = kWinStrip;
                }
                // the bins c - K_far .. c + K_far, left to right
                const Real out = wl.scale * (Real)ax.inv_w;
                const int eb = lw.c - K_far;
                Real x_lo = sx * (edge_at(eb) - wl.E_r);
                Real f_lo = edge_near_bins<Real>(x_lo);
                for (int k = 0; k <= 2 * K_far; ++k) {
                    const int bin = eb + k;
                    const Real x_hi = sx * (edge_at(bin + 1) - wl.E_r);
                    const Real f_hi = edge_near_bins<Real>(x_hi);
                    Real mass = f_hi - f_lo + ((x_lo < (Real)0 && x_hi >= (Real)0) ? (Real)kPi : (Real)0);
                    const Real xc = (Real)0.5 * (x_lo + x_hi);
                    if (sx <= s_narrow && fabs(xc) >= (Real)2) mass = (Real)kPi * sw * midpoint_mean(xc, sw);
                    if (bin >= 0 && bin < n_E) smem_add(&spec_s[bin], (double)(out * mass));
                    x_lo = x_hi;
                    f_lo = f_hi;
                }
            } else {
                if (lw.nb > 0) cls = kWinAxis;
            }
        }
        const unsigned mask = __ballot_sync(0xffffffffu, cls < kWinClasses);
        int base = 0;
        if (lane == 0 && mask) base = atomicAdd(&w_count, __popc(mask));
        base = __shfl_sync(0xffffffffu, base, 0);
        if (cls < kWinClasses) {
            const int k = base + __popc(mask & ((1u << lane) - 1u));
            wLine[k] = wl;
            wIdx[win_slot(cls, atomicAdd(&w_class[cls], 1))] = (uint16_t)k;
        }
    };

    // B2: window bins outside the near bins. A group of G lanes takes one line:
    // its lower half the bins right of the centre, its upper half those left of
    // it. A lane holds two neighbouring edges from bin distance D on outwards and
    // the bins outside of each (G - 1 edges, G - 1 bins a side and visit), the
    // outer edge of its second bin from the next lane.
    auto visit = [&](const WinLine<Real> &l, int D, int G, bool live) {
        const int h = (int)lane & (G / 2 - 1);
        const bool left = (lane & (unsigned)(G / 2)) != 0;
        const Real sgn = left ? (Real)-1 : (Real)1;
        const int Dh = D + 2 * h;                      // distance of this lane's first bin
        const Real Dm = sgn * ((Real)Dh - (Real)0.5);  // its inner edge
        const int bin = left ? l.c - Dh : l.c + Dh;
        const int edge = left ? bin + 1 : bin;
        const Real x0 = l.s * (edge_at(edge) - l.E_r);
        const Real x1 = l.s * (edge_at(left ? edge - 1 : edge + 1) - l.E_r);
        const Real sw = l.s * w_r;
        const Real f0 = edge_window_bins<Real>(x0, Dm, l.d, sw);
        const Real f1 = edge_window_bins<Real>(x1, Dm + sgn, l.d, sw);
        const Real f2 = __shfl_down_sync(0xffffffffu, f0, 1);
        const Real out = sgn * l.scale * inv_w_r;
        const int next = left ? bin - 1 : bin + 1;
        if (live && Dh <= l.D1 && bin >= 0 && bin < n_E) smem_add(&spec_s[bin], (double)(out * (f1 - f0)));
        if (live && h < G / 2 - 1 && Dh < l.D1 && next >= 0 && next < n_E) smem_add(&spec_s[next], (double)(out * (f2 - f1)));
    };

    auto window_phase = [&]() {
        for (int cls = kWin4; cls <= kWin16; ++cls) {  // one visit a line
            const int G = 4 << cls, per = 32 / G, n = w_class[cls];
            for (int i = warp * per; i < n; i += n_warps * per) {
                const int k = i + (int)lane / G;
                const WinLine<Real> &l = wLine[wIdx[win_slot(cls, min(k, n - 1))]];
                visit(l, l.D0, G, k < n);
            }
        }
        for (int i = warp; i < w_class[kWin32]; i += n_warps) {
            const WinLine<Real> &l = wLine[wIdx[win_slot(kWin32, i)]];
            for (int D = l.D0; D <= l.D1; D += 31) visit(l, D, 32, true);
        }
    };

    // Wide windows: a warp takes strips of 31 bins in turn, a lane holds one edge
    // of the strip and sums its bin over the lines in a register (no atomics).
    auto strip_phase = [&]() {
        const int nw = w_class[kWinStrip];
        for (int first = warp * kStripBins; first < n_E; first += n_warps * kStripBins) {
            const int last = min(first + kStripBins, n_E) - 1;
            const int bin = first + (int)lane;
            const Real e = edge_at(bin);
            Real acc = 0;
            for (int k0 = 0; k0 < nw; k0 += 32) {
                int idx = 0;
                bool hit = false;
                if (k0 + (int)lane < nw) {
                    idx = wIdx[win_slot(kWinStrip, k0 + (int)lane)];
                    const int c = wLine[idx].c, D1 = wLine[idx].D1;
                    hit = first <= c + D1 && last >= c - D1;
                }
                for (unsigned todo = __ballot_sync(0xffffffffu, hit); todo; todo &= todo - 1) {
                    const WinLine<Real> &l = wLine[__shfl_sync(0xffffffffu, idx, __ffs(todo) - 1)];
                    const Real sw = l.s * w_r, D = (Real)(bin - l.c), Dm = D - (Real)0.5;
                    const bool on = fabs(D) >= (Real)l.D0 && fabs(D) <= (Real)l.D1;
                    const Real x = l.s * (e - l.E_r);
                    Real mass;
                    if (l.s > s_narrow) {
                        const Real f = edge_window_bins<Real>(x, Dm, l.d, sw);
                        mass = __shfl_down_sync(0xffffffffu, f, 1) - f;
                    } else {
                        const Real f = fabs(x) < (Real)2.2 ? (Real)kPi * tail_of(x) : (Real)0;
                        mass = __shfl_down_sync(0xffffffffu, f, 1) - f;
                        const Real xc = fma((Real)0.5, sw, x);
                        if (fabs(xc) >= (Real)2) mass = window_midpoint<Real>(xc, Dm, l.d, sw);
                        else mass -= spread_envelope<Real>(Dm, l.d, sw);
                    }
                    if (on) acc = fma(l.scale, mass, acc);
                }
            }
            if (lane < kStripBins && bin < n_E) spec_s[bin] += (double)acc * ax.inv_w;
        }
    };

    // Lines integrated over the whole axis (no moments): every line reaches
    // every bin, so a warp takes strips of 31 bins in turn, a lane holds one
    // edge of the strip and sums its bin over the lines in a register.
    auto axis_phase = [&]() {
        const int n_strips = (n_E + kStripBins - 1) / kStripBins, nw = w_class[kWinAxis];
        while (true) {
            int strip = 0;
            if (lane == 0) strip = atomicAdd(&strip_next, 1);
            strip = __shfl_sync(0xffffffffu, strip, 0);
            if (strip >= n_strips) break;
            const int bin = strip * kStripBins + (int)lane;
            const double e_lo = a.edges[min(bin, n_E)];
            const Real e = (Real)e_lo;
            // The width between the edges as they are held here: a bin's mass divided by
            // it is right to the rounding of the mass, while by the FP64 width it would
            // carry that of the float edges (5e-4 of 0.8 eV at 8 keV), and a difference
            // of phases loses a narrow bin's width far from its line.
            const Real width = __shfl_down_sync(0xffffffffu, e, 1) - e;
            Real acc = 0;
            for (int k = 0; k < nw; ++k) {
                const WinLine<Real> &l = wLine[wIdx[win_slot(kWinAxis, k)]];
                const Real x = l.s * (e - l.E_r);
                const Real x_hi = __shfl_down_sync(0xffffffffu, x, 1);
                const Real sw = l.s * width, xc = (Real)0.5 * (x + x_hi);
                // (lane 31 holds the strip's last edge and no bin)
                const bool narrow = sw <= (Real)0.1 && fabs(xc) >= (Real)2 && lane < kStripBins;
                const unsigned wide_bins = __ballot_sync(0xffffffffu, !narrow && lane < kStripBins);
                const bool need = ((wide_bins | (wide_bins << 1)) >> lane) & 1u;
                const Real f = need ? edge_near_bins<Real>(x) : (Real)0;
                Real mass = __shfl_down_sync(0xffffffffu, f, 1) - f +
                            ((x < (Real)0 && x_hi >= (Real)0) ? (Real)kPi : (Real)0);
                if (narrow) mass = (Real)kPi * sw * midpoint_mean(xc, sw);
                acc = fma(l.scale, mass, acc);
            }
            if (lane < kStripBins && bin < n_E) {
                // this warp owns the strip's bins until the phase ends
                spec_s[bin] += (double)acc / (double)width;
            }
        }
    };

    // Lines leave the queue in whole rounds; ``flush`` takes what is left too
    // (before the direction changes). Every condition is uniform over the block.
    auto deposit = [&](bool flush) {
        int nq = q_count;
        bool more = flush ? nq > 0 || w_count > 0 : nq >= kCxrThreads;
        if (flush) __syncthreads();  // every thread has read w_count
        while (more) {
            const int take = min(nq, kCxrThreads);
            near_round(tid < take ? nq - take + tid : -1, d_cur);
            nq -= take;
            __syncthreads();
            const int nw = w_count;
            const bool leave = flush && nq == 0;
            if (nw > kWideRun || (leave && nw > 0)) {
                window_phase();
                const int n_strip = w_class[kWinStrip], n_axis = w_class[kWinAxis];
                const bool strips = n_strip > kStripRun || (leave && n_strip > 0);
                // the window's adds and the strips' sums share spec_s
                __syncthreads();
                if (strips) strip_phase();
                if (n_axis > 0) {
                    if (strips) __syncthreads();
                    axis_phase();
                }
                // strip lines that wait move to the front of the list
                WinLine<Real> wl;
                const bool keep = !strips && tid < n_strip;
                if (keep) wl = wLine[wIdx[win_slot(kWinStrip, tid)]];
                __syncthreads();
                if (keep) {
                    wLine[tid] = wl;
                    wIdx[win_slot(kWinStrip, tid)] = (uint16_t)tid;
                }
                if (tid < kWinClasses) w_class[tid] = tid == kWinStrip && !strips ? n_strip : 0;
                if (tid == 0) { w_count = strips ? 0 : n_strip; strip_next = 0; }
            }
            more = flush ? nq > 0 : nq >= kCxrThreads;
            __syncthreads();
        }
        if (tid == 0) q_count = nq;
    };

    auto publish = [&](int d) {
        // Publish (and clear) the block's spectrum of direction d.
        __syncthreads();
        double *gspec = a.spec + (int64_t)d * n_E;
        for (int j = tid; j < n_E; j += blockDim.x) {
            if (spec_s[j] != 0.0) atomicAdd(&gspec[j], spec_s[j]);
            spec_s[j] = 0.0;
        }
        __syncthreads();
    };

    // Work units: (direction, row chunk, segment tile), tiles innermost, so a
    // block stages its rows once per run of tiles. Chunk k holds rows k,
    // k + n_chunks, ...: neighbouring rows of a reflection list radiate alike, so
    // the chunks carry equal work. Fewer than four units a block: halve the tile, so that a short
    // segment list still reaches every SM (a tile below four segments leaves
    // most threads of a pass idle).
    int64_t d_ch = -1, win = -1;
    // The staged chunk's rows, the two staged tiles (tile ``par`` is the newer), and
    // the survivors that wait for the next tile's.
    int ng = 1, par = 0, n_wait = 0, g0 = 0, n_pairs = 0;
    unsigned ng_magic = 0;
    int64_t s0_of[2] = {0, 0};
    // q / ng for the pass's pair ids q < kSegTile * ng by a multiply-high:
    // magic = floor((2^32 - 1) / ng) + 1 is at least 2^32 / ng and
    // exceeds it by under one, so q magic / 2^32 lies in
    // [q / ng, q / ng + q / 2^32) and its floor is exact for q < 2^32 / ng
    // (one row: magic does not fit 32 bits, and the quotient is q).
    const auto seg_of = [&](int q) { return ng == 1 ? q : (int)__umulhi((unsigned)q, ng_magic); };
    // A1: the full chain of pair ``id`` (tile parity x kPairs + pair of the tile;
    // -1: none), by this thread. All threads call it.
    const auto chain = [&](int id, int d) {
        Line<Real> ln;
        ln.good = false;
        if (id >= 0) {
            const int t = id >= kPairs ? 1 : 0;
            const int q = id - t * kPairs;
            const int si = seg_of(q);
            const int gi = q - si * ng;
            ln = pair_line<Real, kLayered>(segs[t * kSegTile + si], rows[gi], E_tab, delta_tab, log_mu, n_tab, n_mu,
                                           a.tables, ti, esc + t * kSegTile + si, a, lay_t);
            if (pairs_out) {
                const int64_t o = ((int64_t)d * n_seg + s0_of[t] + si) * n_g + g0 + gi * n_chunks;
                a.pair_E[o] = (double)ln.E_res;
                a.pair_a[o] = (double)ln.a_width;
                a.pair_w[o] = (double)ln.weight;
                a.pair_good[o] = ln.good ? 1 : 0;
            }
            if (ln.good && lines_out) {
                const unsigned long long slot = atomicAdd(a.line_count, 1ULL);
                if (slot < (unsigned long long)a.line_capacity) {
                    a.line_E[slot] = (double)ln.E_res;
                    a.line_a[slot] = (double)ln.a_width;
                    a.line_w[slot] = (double)ln.weight;
                    a.line_dir[slot] = d;
                    if (a.line_seg) a.line_seg[slot] = s0_of[t] + si;
                } else {
                    set_status(a.status, PB_DEV_QUEUE_OVERFLOW);
                }
            }
        }
        if (binmean) {
            const unsigned mask = __ballot_sync(0xffffffffu, ln.good);
            int base = 0;
            if (lane == 0 && mask) base = atomicAdd(&q_count, __popc(mask));
            base = __shfl_sync(0xffffffffu, base, 0);
            if (ln.good) {
                const int kk = base + __popc(mask & ((1u << lane) - 1u));
                qE[kk] = ln.E_res;
                qA[kk] = ln.a_width;
                qW[kk] = ln.weight;
            }
        }
    };
    // Tiles without a radiating segment are passed over a window of kCxrThreads
    // segments at a time: one flag word per warp, a tile is 4, 8 or 16 of its bits.
    unsigned *const rad_words = reinterpret_cast<unsigned *>(scratch);
    const int per_win = kCxrThreads / seg_tile;
    int64_t wk = w_begin, dc = n_work > 0 ? w_begin / n_tiles : 0, tile = w_begin - dc * n_tiles;
    const auto next_unit = [&]() {
        ++wk;
        if (++tile == n_tiles) { tile = 0; ++dc; }
    };
    for (;; next_unit()) {
        for (; wk < w_end && !pairs_out; next_unit()) {
            if (tile / per_win != win) {
                win = tile / per_win;
                const int64_t sg = win * kCxrThreads + tid;
                const bool rad = sg < n_seg && a.elec_id[sg] < a.Ne &&
                                 (a.seg_layer == nullptr || a.seg_layer[sg] == a.emit_layer);
                const unsigned mask = __ballot_sync(0xffffffffu, rad);
                __syncthreads();  // the last window's flags have been read
                if (lane == 0) rad_words[warp] = mask;
                __syncthreads();
            }
            const int bit = (int)(tile % per_win) * seg_tile;
            if ((rad_words[bit >> 5] >> (bit & 31)) & ((1u << seg_tile) - 1u)) break;
        }
        const bool end = wk >= w_end;
        const int d = (int)dc / n_chunks;
        // The lines the last unit queued: whole rounds, or all of them before
        // the direction changes or the block ends.
        const bool leave = end || d != d_cur;
        __syncthreads();
        // A1 over whole rounds of the last tile's survivors (every pair without the
        // prefilter), oldest first. The rest waits for the next tile's, but not beyond
        // it (its segments are staged until then), and not for other rows.
        {
            const int n_surv = dtail != nullptr ? p_count : n_pairs;
            const bool all = dtail == nullptr || end || dc != d_ch;
            int done = 0;
            while (n_surv - done >= kCxrThreads || (done < n_surv && (all || (done == 0 && n_wait > 0)))) {
                const int k = done + tid;
                chain(k < n_surv ? (dtail != nullptr ? (int)pq[k] : par * kPairs + k) : -1, d_cur);
                done = min(done + kCxrThreads, n_surv);
            }
            n_wait = n_surv - done;
            const uint16_t w = tid < n_wait ? pq[done + tid] : (uint16_t)0;
            __syncthreads();
            if (tid < n_wait) pq[tid] = w;
            if (tid == 0) p_count = n_wait;
        }
        if (binmean && d_cur >= 0) {
            deposit(leave);
            if (leave) publish(d_cur);
        }
        if (end) break;
        d_cur = d;
        const double *nh = a.n_hat + 3 * d;
        const int64_t s0 = tile * seg_tile;
        const int nst = (int)((n_seg - s0) < seg_tile ? (n_seg - s0) : seg_tile);
        par ^= 1;
        s0_of[par] = s0;
        __syncthreads();  // before the staged rows and segments are replaced
        SegPre<Real> *const seg_t = segs + par * kSegTile;
        if (tid < nst) seg_precompute<Real>(seg_t[tid], a, s0 + tid, nh);
        if constexpr (kLayered) {
            if (tid < nst) esc_precompute<Real>(esc[par * kSegTile + tid], a, s0 + tid, nh, lay_zt, lay_zb);
        }
        {
            if (dc != d_ch) {
                g0 = (int)dc - d * n_chunks;
                ng = (n_g - g0 + n_chunks - 1) / n_chunks;
                ng_magic = (unsigned)(0xFFFFFFFFull / (unsigned)ng) + 1u;
            }
            for (int j = tid; j < (dc != d_ch ? ng : 0); j += blockDim.x) {
                const int g = g0 + j * n_chunks;
                RowPre<Real> &r = rows[j];
                const double *G = a.tables.G + 3 * g;
                const double *ES = a.tables.ES + 3 * ((int64_t)d * n_g + g);
                const double *EP = a.tables.EP + 3 * ((int64_t)d * n_g + g);
                for (int c = 0; c < 3; ++c) {
                    r.G[c] = (Real)G[c];
                    r.ES[c] = (Real)ES[c];
                    r.EP[c] = (Real)EP[c];
                }
                r.g2 = r.G[0] * r.G[0] + r.G[1] * r.G[1] + r.G[2] * r.G[2];
                r.n_dot_g = r.G[0] * (Real)nh[0] + r.G[1] * (Real)nh[1] + r.G[2] * (Real)nh[2];
                r.g_dot_es = r.G[0] * r.ES[0] + r.G[1] * r.ES[1] + r.G[2] * r.ES[2];
                r.g_dot_ep = r.G[0] * r.EP[0] + r.G[1] * r.EP[1] + r.G[2] * r.EP[2];
                r.wm = (Real)a.tables.WM[g];
                r.row = a.tables.row_table[g];
            }
            d_ch = dc;
            __syncthreads();
            // ---- A0: prefilter and compact the surviving pairs ----
            n_pairs = nst * ng;
            if (dtail == nullptr) continue;
            // Lane ``it`` keeps the survivors' mask of the warp's iteration
            // ``it`` (at most pair_queue / kCxrThreads = 8 of them): one
            // shared counter update a warp and pass.
            const int n_it0 = (n_pairs + (int)blockDim.x - 1) / (int)blockDim.x;
            unsigned mine = 0;
            for (int it = 0; it < n_it0; ++it) {
                const int q = it * blockDim.x + tid;
                bool ok = false;
                if (q < n_pairs) {
                    const int si = seg_of(q);
                    ok = pair_may_keep<Real>(seg_t[si], rows[q - si * ng], E_tab, dtail, n_tab, a.tables, ti);
                }
                const unsigned mask = __ballot_sync(0xffffffffu, ok);
                if ((int)lane == it) mine = mask;
            }
            int incl = __popc(mine);
            for (int o = 1; o < 32; o <<= 1) {
                const int v = __shfl_up_sync(0xffffffffu, incl, o);
                if ((int)lane >= o) incl += v;
            }
            int base = 0;
            if (lane == 31 && incl) base = atomicAdd(&p_count, incl);
            base = __shfl_sync(0xffffffffu, base, 31) + incl - __popc(mine);  // of iteration ``lane``
            for (int it = 0; it < n_it0; ++it) {
                const unsigned mask = __shfl_sync(0xffffffffu, mine, it);
                const int at = __shfl_sync(0xffffffffu, base, it);
                if ((mask >> lane) & 1u)
                    pq[at + __popc(mask & ((1u << lane) - 1u))] = (uint16_t)(par * kPairs + it * blockDim.x + tid);
            }
        }
    }
}

// Far field: spec[d][b] += sum_c M[d][c] . envelope(b, c) over the (padded)
// centre bins c farther than K_far bins from b. The moments sit on a uniform
// axis, so this is a convolution: with the bins a distance D = b - c apart,
// A = (D - 1/2) w and B = (D + 1/2) w, and the three expansion coefficients are
//   f0 = r / w^2, f1 = 2 D r^2 / w^3, f2 = (3 D^2 + 1/4) r^3 / w^4,
//   r = 1 / (D^2 - 1/4),
// r a function of the integer D alone. 3 D^2 + 1/4 = 3 / r + 1, so a pair is
//   w^2 f = r (m0 + r (2 D m1 / w + (3 + r) m2 / w^2)):
// four FMAs, one step of D and two shared loads (the moment of the centre,
// broadcast to the warp, serves kFarPer bins; r is consecutive over the lanes
// and zero within K_far). The first form took the moments from L2 in FP64, a
// conversion and nine products a pair (2,048 bins x 2,872 centres, mixed: 4
// directions 90 -> 15 us, 16 directions 153 -> 42 us).
// A block takes kFarBins bins of one direction and walks the centres in chunks
// staged with the chunk's r; its 16 warps split each chunk. Sums leave Acc for
// FP64 after each chunk, and the warps' sums are added in warp order, so the
// result does not depend on the launch.
constexpr int kFarPer = 2;             // output bins per thread, 32 apart
constexpr int kFarBins = 32 * kFarPer;
constexpr int kFarSlices = 16;
constexpr int kFarChunk = 512;         // most centres staged at a time

template <class Acc>
struct __align__(16) FarMoment {
    Acc m0, m1, m2, m2x3;
};

// Acc is the type of a chunk's products and sums: double on the FP64 path,
// float on the mixed one (a bin's far field is a sum of positive envelope terms
// and two small corrections; a chunk's share of a thread is at most 32 terms).
template <class Acc>
__global__ void __launch_bounds__(32 * kFarSlices) far_field_conv_kernel(const double *edges, int n_E, int pad,
                                                                         const double *mom, double *spec, int K_far) {
    __shared__ FarMoment<Acc> sM[kFarChunk];
    __shared__ Acc sR[kFarChunk + kFarBins];  // r(D) at D - D_lo
    __shared__ double part[kFarSlices][kFarBins];
    const int d = blockIdx.y;
    const int n_mom = n_E + 2 * pad;
    const int n_chunk = (n_mom + kFarChunk - 1) / kFarChunk;
    // equal chunks, whole rounds of the warps
    const int per = ((n_mom + n_chunk - 1) / n_chunk + kFarSlices - 1) / kFarSlices;
    const int len = per * kFarSlices;
    const double iw = 1.0 / ((edges[n_E] - edges[0]) / n_E);
    const double iw2 = iw * iw;
    const int lane = threadIdx.x & 31, slice = threadIdx.x >> 5;
    const int b0 = blockIdx.x * kFarBins;
    const double *m = mom + (int64_t)d * n_mom * 3;
    double sum[kFarPer];
#pragma unroll
    for (int j = 0; j < kFarPer; ++j) sum[j] = 0.0;
    for (int c0 = 0; c0 < n_mom; c0 += len) {
        const int n = min(len, n_mom - c0);
        // r at the distances b0 + t - (c0 - pad + i), t < kFarBins, i < n
        const int D_lo = b0 - (c0 - pad + n - 1);
        __syncthreads();  // the last chunk has been read
        for (int i = threadIdx.x; i < n; i += blockDim.x) {
            const double *mi = m + 3 * (int64_t)(c0 + i);
            const double m0 = mi[0], m1 = m0 != 0.0 ? mi[1] * iw : 0.0, m2 = m0 != 0.0 ? mi[2] * iw2 : 0.0;
            sM[i] = {(Acc)m0, (Acc)(2.0 * m1), (Acc)m2, (Acc)(3.0 * m2)};
        }
        for (int i = threadIdx.x; i < n + kFarBins - 1; i += blockDim.x) {
            const int D = D_lo + i;
            sR[i] = D >= -K_far && D <= K_far ? (Acc)0 : (Acc)(1.0 / ((double)D * (double)D - 0.25));
        }
        __syncthreads();
        const int i0 = min(slice * per, n), i1 = min(i0 + per, n);
        const Acc *r_at = sR + lane + (n - 1);  // r of bin b0 + lane + 32 j and centre i: r_at[32 j - i]
        Acc D = (Acc)(b0 + lane - (c0 - pad + i0));
        Acc acc[kFarPer];
#pragma unroll
        for (int j = 0; j < kFarPer; ++j) acc[j] = 0;
#pragma unroll 4
        for (int i = i0; i < i1; ++i) {
            const FarMoment<Acc> q = sM[i];
#pragma unroll
            for (int j = 0; j < kFarPer; ++j) {
                const Acc r = r_at[32 * j - i];
                const Acc u = fma(D + (Acc)(32 * j), q.m1, fma(q.m2, r, q.m2x3));
                acc[j] = fma(fma(u, r, q.m0), r, acc[j]);
            }
            D -= (Acc)1;
        }
#pragma unroll
        for (int j = 0; j < kFarPer; ++j) sum[j] += (double)acc[j];
    }
#pragma unroll
    for (int j = 0; j < kFarPer; ++j) part[slice][lane + 32 * j] = sum[j];
    __syncthreads();
    const int b = b0 + threadIdx.x;
    if (threadIdx.x < kFarBins && b < n_E) {
        double t = 0.0;
#pragma unroll
        for (int k = 0; k < kFarSlices; ++k) t += part[k][threadIdx.x];
        spec[(int64_t)d * n_E + b] += t * iw2;
    }
}

// Node reduction of buffered lines: spec[d][e] += sum_j w_j sinc^2(x_je),
// x = a (E_e - E_j) / pi, formed in FP64. sinc^2 needs sin^2 alone, so the phase
// is reduced to half a turn about the nearest integer x (no quadrants) and the
// sine is one Taylor series to (pi f)^21 (FP64, truncation 1e-18) or the SFU's
// (mixed). Lines are staged in shared memory with a / pi and w / pi^2 ready, and
// four lines are in flight per thread: the loop is bound by the latency of its
// division otherwise (300 segments x 144 rows x 781 nodes: 130 -> 65 us).
constexpr int kNodeTile = 128;

__device__ __forceinline__ double sin_pi_series(double f) {
    constexpr int kTerms = 11;
    struct C {
        double c[kTerms];
    };
    constexpr C t = [] {
        C r{};
        double v = 1.0;  // pi^n / n!
        for (int n = 1; n <= 2 * kTerms - 1; ++n) {
            v *= kPi / n;
            if (n & 1) r.c[n >> 1] = ((n >> 1) & 1) ? -v : v;
        }
        return r;
    }();
    const double y = f * f;
    double s = t.c[kTerms - 1];
#pragma unroll
    for (int k = kTerms - 2; k >= 0; --k) s = fma(s, y, t.c[k]);
    return s * f;
}

template <class Real>
__global__ void __launch_bounds__(kNodeTile) node_reduce_kernel(const double *E_grid, int n_E, const double *line_E,
                                                                const double *line_a, const double *line_w,
                                                                const int32_t *line_dir,
                                                                const unsigned long long *line_count,
                                                                int64_t capacity, double *spec) {
    __shared__ double sE[kNodeTile], sA[kNodeTile], sW[kNodeTile];
    __shared__ int sD[kNodeTile];
    const int e = blockIdx.x * blockDim.x + threadIdx.x;
    int64_t n_lines = (int64_t)*line_count;
    if (n_lines > capacity) n_lines = capacity;
    const int64_t per = (n_lines + gridDim.y - 1) / gridDim.y;
    const int64_t j0 = per * blockIdx.y;
    const int64_t j1 = j0 + per < n_lines ? j0 + per : n_lines;
    const double E = e < n_E ? E_grid[e] : 0.0;
    const auto term = [&](int k) {
        constexpr double kRound = 6755399441055744.0;  // 1.5 2^52
        const double x = sA[k] * (E - sE[k]);
        const double f = x - __dsub_rn(__dadd_rn(x, kRound), kRound);
        double s;
        if constexpr (sizeof(Real) == 8) s = sin_pi_series(f);
        else s = (double)__sinf((float)(kPi * f));
        const double v = sW[k] * (s * s) / (x * x);
        return fabs(x) > 1.0e-20 ? v : sW[k] * (kPi * kPi);  // sinc^2(0) = 1
    };
    // Accumulate per direction seen in this chunk (directions are few).
    double acc = 0.0;
    int cur_dir = -1;
    for (int64_t t0 = j0; t0 < j1; t0 += kNodeTile) {
        const int nt = (int)((j1 - t0) < kNodeTile ? (j1 - t0) : kNodeTile);
        __syncthreads();
        for (int j = threadIdx.x; j < nt; j += blockDim.x) {
            sE[j] = line_E[t0 + j];
            sA[j] = line_a[t0 + j] / kPi;
            sW[j] = line_w[t0 + j] / (kPi * kPi);
            sD[j] = line_dir[t0 + j];
        }
        __syncthreads();
        if (e < n_E) {
            int k = 0;
            while (k < nt) {
                if (sD[k] != cur_dir) {
                    if (cur_dir >= 0 && acc != 0.0) atomicAdd(&spec[(int64_t)cur_dir * n_E + e], acc);
                    acc = 0.0;
                    cur_dir = sD[k];
                }
                if (k + 4 <= nt && sD[k + 1] == cur_dir && sD[k + 2] == cur_dir && sD[k + 3] == cur_dir) {
                    const double t0v = term(k), t1v = term(k + 1), t2v = term(k + 2), t3v = term(k + 3);
                    acc += (t0v + t1v) + (t2v + t3v);
                    k += 4;
                } else {
                    acc += term(k);
                    k += 1;
                }
            }
        }
    }
    if (e < n_E && cur_dir >= 0 && acc != 0.0) atomicAdd(&spec[(int64_t)cur_dir * n_E + e], acc);
}

template <class Real>
static size_t cxr_smem_bytes(const pb_cxr_args &a, bool tab_smem) {
    constexpr int kRowChunk = row_chunk<Real>();
    constexpr int kQueue = surv_queue<Real>();
    size_t b = sizeof(RowPre<Real>) * kRowChunk + sizeof(SegPre<Real>) * 2 * kSegTile + 16;
    b += sizeof(Real) * 3 * line_queue<Real>() + 16 +
         (sizeof(WinLine<Real>) + sizeof(uint16_t) * (kWinClasses / 2)) * kWideCap + sizeof(int) * 64 +
         sizeof(uint16_t) * kQueue + 16;
    if (tab_smem) b += sizeof(Real) * (size_t)a.tables.n_tab * (3 + a.tables.n_mu);
    b += 16;
    if (a.quadrature == PB_QUAD_BINMEAN)
        b += sizeof(double) * (size_t)a.n_E + (sizeof(Real) == 4 ? sizeof(float) * ((size_t)a.n_E + 1) : 0);
    if (a.n_layer > 0)
        b += 16 + sizeof(EscSeg<Real>) * 2 * kSegTile + sizeof(double) * 2 * kMaxEscLayers + sizeof(Real) * kMaxEscLayers;
    return b;
}



template <class Real>
static cudaError_t launch_cxr_t(const pb_cxr_args &a, cudaStream_t s, int sms, int far_pad) {
    const bool binmean = a.quadrature == PB_QUAD_BINMEAN;
    const int K_far = (binmean && a.exact_widths > 0.0 && a.far_moments && far_pad >= 0) ? 2 : 0;
    if (K_far == 0) far_pad = 0;
    if (a.n_layer < 0 || a.n_layer > kMaxEscLayers) return cudaErrorInvalidValue;
    if (a.n_layer > 0 && (!a.z_top || !a.z_bot || !a.mu_off || !a.mu_knot || !a.mu_value || !a.mu_slope))
        return cudaErrorInvalidValue;
    // FP64 tables that do not fit beside the queues and the spectrum are read from
    // global memory (without the prefilter, as tables beyond kMaxTab are).
    constexpr size_t kMaxSmem = 220 * 1024;
    bool tab_smem = a.tables.n_tab <= kMaxTab;
    size_t smem = cxr_smem_bytes<Real>(a, tab_smem);
    if (sizeof(Real) == 8 && tab_smem && smem > kMaxSmem) {
        tab_smem = false;
        smem = cxr_smem_bytes<Real>(a, false);
    }
    if (smem > kMaxSmem || (binmean && a.n_E > 65535)) return cudaErrorInvalidValue;
    // The float path reads its tables from the shared-memory staging only.
    if (sizeof(Real) == 4 && a.tables.n_tab > kMaxTab) return cudaErrorInvalidValue;
    auto kern = a.n_layer > 0 ? cxr_kernel<Real, true> : cxr_kernel<Real, false>;
    cudaError_t err = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (err != cudaSuccess) return err;
    if (K_far > 0) {
        err = cudaMemsetAsync(a.far_moments, 0,
                              sizeof(double) * (size_t)a.n_dir * (a.n_E + 2 * far_pad) * 3, s);
        if (err != cudaSuccess) return err;
    }
    if (a.line_count) {
        err = cudaMemsetAsync(a.line_count, 0, sizeof(unsigned long long), s);
        if (err != cudaSuccess) return err;
    }
    int per_sm = 0;
    err = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, kCxrThreads, smem);
    if (err != cudaSuccess) return err;
    if (per_sm < 1) per_sm = 1;
    constexpr int kRowChunk = row_chunk<Real>();
    const int64_t work = (a.n_seg + 3) / 4 * (int64_t)a.n_dir * ((a.tables.n_g + kRowChunk - 1) / kRowChunk);
    int64_t gx = (int64_t)sms * per_sm;
    if (gx > work) gx = work;
    if (gx < 1) gx = 1;
    kern<<<(unsigned)gx, kCxrThreads, smem, s>>>(a, K_far, far_pad, tab_smem);
    err = cudaGetLastError();
    if (err != cudaSuccess) return err;
    if (K_far > 0) {
        // far moments are enabled on uniform edges only
        dim3 cg((unsigned)((a.n_E + kFarBins - 1) / kFarBins), (unsigned)a.n_dir);
        far_field_conv_kernel<Real><<<cg, 32 * kFarSlices, 0, s>>>(a.edges, a.n_E, far_pad, a.far_moments, a.spec, K_far);
        err = cudaGetLastError();
        if (err != cudaSuccess) return err;
    }
    if (a.quadrature == PB_QUAD_NODE && a.line_E != nullptr && a.spec != nullptr) {
        // about eight blocks an SM over the node tiles
        const unsigned gx = (unsigned)((a.n_E + kNodeTile - 1) / kNodeTile);
        const unsigned gy = std::max(1u, (unsigned)(sms * 8) / gx);
        dim3 ng(gx, gy);
        node_reduce_kernel<Real><<<ng, kNodeTile, 0, s>>>(a.E_grid, a.n_E, a.line_E, a.line_a, a.line_w,
                                                    a.line_dir, a.line_count, a.line_capacity, a.spec);
        err = cudaGetLastError();
    }
    return err;
}

cudaError_t launch_cxr(const pb_cxr_args &a, cudaStream_t s, int sms) {
    if (a.precision == PB_MIXED) return launch_cxr_t<float>(a, s, sms, a.far_pad);
    return launch_cxr_t<double>(a, s, sms, a.far_pad);
}

// ---------------------------------------------------------------------------
// Coherent route: per-row line records from the segment list (FP64).
//
// For every (segment, reflection row) pair the chain of pair_amps gives the
// complex PXR+CBS amplitude of both polarisations; the record adds the
// segment's escape-piece ends and formation coefficients, the exact vacuum
// line centre and width with the recoil phase over the electron's age, and
// the phase terms (cxr/_batched.py:561-660, cxr/_formation.py:58-81,
// cxr/_recoil.py:118-147, cxr/_setup.py:1023-1026). Rows hold their kept
// pairs in segment order, row after row (row_off), as the reference's block
// loop lays them out and pb_coherent_reduce reads them: pass 1 flags the kept
// pairs [row][segment], pass 2 scans each row, pass 3 writes the records.
// ---------------------------------------------------------------------------
struct CohRec {
    double f[13];  // E_vac, a_vac, phase_slope, g_phase, cs_re, cs_im, cp_re, cp_im, L_esc, half_dL, apb, bma, q
};

// cxr/_formation.py:58-81
__device__ __forceinline__ void formation_coefficients(double tau_start, double tau_end, double &apb, double &bma,
                                                       double &q) {
    q = 0.25 * (tau_end - tau_start);
    if (fabs(q) < 0.5) {
        const double c0 = exp(-0.25 * (tau_start + tau_end));
        apb = 2.0 * c0 * cosh(q);
        bma = -2.0 * c0 * sinh(q);
    } else {
        const double ea = exp(-0.5 * tau_start), eb = exp(-0.5 * tau_end);
        apb = ea + eb;
        bma = eb - ea;
    }
}

__device__ bool coh_record(const pb_cxr_args &a, const double *t_start, int64_t s, int g, const TabIndex &ti,
                           CohRec *rec) {
    SegPre<double> sp;
    seg_precompute<double>(sp, a, s, a.n_hat);
    RowPre<double> rw;
    const double *nh = a.n_hat;
    for (int c = 0; c < 3; ++c) {
        rw.G[c] = a.tables.G[3 * g + c];
        rw.ES[c] = a.tables.ES[3 * g + c];
        rw.EP[c] = a.tables.EP[3 * g + c];
    }
    rw.g2 = rw.G[0] * rw.G[0] + rw.G[1] * rw.G[1] + rw.G[2] * rw.G[2];
    rw.n_dot_g = rw.G[0] * nh[0] + rw.G[1] * nh[1] + rw.G[2] * nh[2];
    rw.g_dot_es = rw.G[0] * rw.ES[0] + rw.G[1] * rw.ES[1] + rw.G[2] * rw.ES[2];
    rw.g_dot_ep = rw.G[0] * rw.EP[0] + rw.G[1] * rw.EP[1] + rw.G[2] * rw.EP[2];
    rw.wm = a.tables.WM[g];
    rw.row = a.tables.row_table[g];
    const int n_tab = a.tables.n_tab;
    const PairAmps<double> p = pair_amps<double, false>(sp, rw, a.tables.E_tab, a.tables.delta, a.tables.log_mu,
                                                        n_tab, a.tables.n_mu, a.tables, ti);
    if (!p.keep) return false;
    double apb, bma, qq;
    formation_coefficients(sp.path0 * p.mu, sp.path1 * p.mu, apb, bma, qq);
    // exact vacuum centre / width and recoil phase over the age, with the
    // vacuum denominator and n.g of the row (cxr/_recoil.py:118-147)
    const double numerator = p.v_dot_g - p.r_num;
    const double den = sp.denom_row + p.r_den;
    const double E_c = kHbarcEvAng * numerator / den;
    const double x = numerator / den * sp.inv_E;
    const double kappa = 1.0 / (1.0 - x);
    const double a_vac = kappa * den * sp.t_L / (2.0 * kHbarcEvAng);
    const double t_mid = (t_start ? t_start[s] : 0.0) + 0.5 * sp.t_L;
    const double rx = a.r_mid[3 * s], ry = a.r_mid[3 * s + 1], rz = a.r_mid[3 * s + 2];
    const double d_geom = t_mid - (rx * nh[0] + ry * nh[1] + rz * nh[2]);
    const double d_shift = kappa * (x * sp.denom_row + p.r_den) * t_mid;
    const double g_shift = kappa * (x * p.v_dot_g - p.r_num) * t_mid;
    const double amp = sqrt(kAlphaFs * p.omega / (4.0 * (kPi * kPi) * kHbarcEvAng));
    const double cs_re = amp * sp.t_L * p.A_re[0], cs_im = amp * sp.t_L * p.A_im[0];
    const double cp_re = amp * sp.t_L * p.A_re[1], cp_im = amp * sp.t_L * p.A_im[1];
    const bool good = p.keep && isfinite(amp) && amp > 0.0 && sp.t_L > 0.0 && isfinite(apb) && apb > 0.0 &&
                      isfinite(bma) && isfinite(cs_re) && isfinite(cs_im) && isfinite(cp_re) && isfinite(cp_im);
    if (rec && good) {
        // record fields (cxr/_batched.py:646-660)
        rec->f[0] = E_c;
        rec->f[1] = a_vac;
        rec->f[2] = (d_geom + d_shift) / kHbarcEvAng;
        rec->f[3] = rx * rw.G[0] + ry * rw.G[1] + rz * rw.G[2] + g_shift;
        rec->f[4] = cs_re;
        rec->f[5] = cs_im;
        rec->f[6] = cp_re;
        rec->f[7] = cp_im;
        rec->f[8] = 0.5 * (sp.path0 + sp.path1);
        rec->f[9] = 0.5 * (sp.path1 - sp.path0);
        rec->f[10] = apb;
        rec->f[11] = bma;
        rec->f[12] = qq;
    }
    return good;
}

__device__ __forceinline__ TabIndex tab_index_of(const pb_cxr_tables &t) {
    TabIndex ti{};
    ti.geometric = t.tab_log_step > 0.0;
    ti.log0 = t.tab_log0;
    ti.inv_h = ti.geometric ? 1.0 / t.tab_log_step : 0.0;
    return ti;
}

// Pass 1: kept flags, row-major [g][s].
__global__ void coh_rec_flags_kernel(const pb_cxr_args a, const double *t_start, int64_t n_seg, uint8_t *flags) {
    const TabIndex ti = tab_index_of(a.tables);
    const int n_g = a.tables.n_g;
    const int64_t n = n_seg * (int64_t)n_g;
    for (int64_t q = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; q < n; q += (int64_t)gridDim.x * blockDim.x) {
        const int64_t s = q / n_g;
        const int g = (int)(q - s * n_g);
        flags[(int64_t)g * n_seg + s] = coh_record(a, t_start, s, g, ti, nullptr) ? 1 : 0;
    }
}

// Pass 2: exclusive scan of one row's flags (one block per row) and its count.
__global__ void __launch_bounds__(1024) coh_rec_scan_kernel(int64_t n_seg, const uint8_t *flags, int32_t *pos,
                                                           int64_t *count) {
    __shared__ int64_t warp_sum[32];
    __shared__ int64_t carry;
    const int g = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint8_t *f = flags + (int64_t)g * n_seg;
    int32_t *o = pos + (int64_t)g * n_seg;
    if (tid == 0) carry = 0;
    __syncthreads();
    for (int64_t base = 0; base < n_seg; base += 1024) {
        const int64_t s = base + tid;
        const int v = s < n_seg ? f[s] : 0;
        int incl = v;
        for (int d = 1; d < 32; d <<= 1) {
            const int u = __shfl_up_sync(0xffffffffu, incl, d);
            if (lane >= d) incl += u;
        }
        if (lane == 31) warp_sum[warp] = incl;
        __syncthreads();
        if (warp == 0) {
            int64_t w = warp_sum[lane];
            int64_t wi = w;
            for (int d = 1; d < 32; d <<= 1) {
                const int64_t u = __shfl_up_sync(0xffffffffu, wi, d);
                if (lane >= d) wi += u;
            }
            warp_sum[lane] = wi - w;  // exclusive prefix of the warps
        }
        __syncthreads();
        const int64_t excl = carry + warp_sum[warp] + incl - v;
        if (s < n_seg) o[s] = (int32_t)excl;
        __syncthreads();
        if (tid == 1023) carry = excl + v;
        __syncthreads();
    }
    if (tid == 0) count[g] = carry;
}

// Row offsets from the counts: one warp, 32 rows at a time.
__global__ void coh_rec_offsets_kernel(int n_g, const int64_t *count, int64_t *row_off) {
    const int lane = threadIdx.x;
    int64_t run = 0;
    if (lane == 0) row_off[0] = 0;
    for (int g0 = 0; g0 < n_g; g0 += 32) {
        int64_t v = g0 + lane < n_g ? count[g0 + lane] : 0;
        for (int d = 1; d < 32; d <<= 1) {
            const int64_t u = __shfl_up_sync(0xffffffffu, v, d);
            if (lane >= d) v += u;
        }
        if (g0 + lane < n_g) row_off[g0 + lane + 1] = run + v;
        run += __shfl_sync(0xffffffffu, v, 31);
    }
}

// Pass 3: the records of the kept pairs at their row positions.
__global__ void coh_rec_write_kernel(const pb_coherent_records_args r, const uint8_t *flags, const int32_t *pos) {
    const pb_cxr_args &a = r.cxr;
    const TabIndex ti = tab_index_of(a.tables);
    const int n_g = a.tables.n_g;
    const int64_t n_seg = a.n_seg;
    const int64_t n = n_seg * (int64_t)n_g;
    double *const out[13] = {r.E_vac, r.a_vac, r.phase_slope, r.g_phase, r.cs_re, r.cs_im, r.cp_re,
                             r.cp_im, r.L_esc, r.half_dL, r.apb, r.bma, r.q};
    for (int64_t q = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; q < n; q += (int64_t)gridDim.x * blockDim.x) {
        const int64_t s = q / n_g;
        const int g = (int)(q - s * n_g);
        const int64_t fi = (int64_t)g * n_seg + s;
        if (!flags[fi]) continue;
        CohRec rec;
        if (!coh_record(a, r.t_start, s, g, ti, &rec)) continue;
        const int64_t slot = r.row_off[g] + pos[fi];
        if (slot >= r.capacity) {
            set_status(r.status, PB_DEV_QUEUE_OVERFLOW);
            continue;
        }
#pragma unroll
        for (int k = 0; k < 13; ++k) out[k][slot] = rec.f[k];
        if (r.elec_out) r.elec_out[slot] = a.elec_id[s];
    }
}

uint64_t coherent_records_work_bytes(int64_t n_seg, int n_g) {
    const uint64_t pairs = (uint64_t)n_seg * (uint64_t)n_g;
    const auto al = [](uint64_t b) { return (b + 255) / 256 * 256; };
    return al(pairs) + al(pairs * 4) + al((uint64_t)n_g * 8);
}

cudaError_t launch_coherent_records(const pb_coherent_records_args &r, cudaStream_t s, int sms) {
    const int64_t n_seg = r.cxr.n_seg;
    const int n_g = r.cxr.tables.n_g;
    const uint64_t pairs = (uint64_t)n_seg * (uint64_t)n_g;
    const auto al = [](uint64_t b) { return (b + 255) / 256 * 256; };
    uint8_t *flags = static_cast<uint8_t *>(r.work);
    int32_t *pos = reinterpret_cast<int32_t *>(static_cast<uint8_t *>(r.work) + al(pairs));
    int64_t *count = reinterpret_cast<int64_t *>(static_cast<uint8_t *>(r.work) + al(pairs) + al(pairs * 4));
    const int64_t blocks = std::max<int64_t>(1, std::min<int64_t>((int64_t)((pairs + 255) / 256), (int64_t)sms * 8));
    coh_rec_flags_kernel<<<(unsigned)blocks, 256, 0, s>>>(r.cxr, r.t_start, n_seg, flags);
    coh_rec_scan_kernel<<<(unsigned)n_g, 1024, 0, s>>>(n_seg, flags, pos, count);
    coh_rec_offsets_kernel<<<1, 32, 0, s>>>(n_g, count, r.row_off);
    coh_rec_write_kernel<<<(unsigned)blocks, 256, 0, s>>>(r, flags, pos);
    return cudaGetLastError();
}

// Coarse per-pair binning of a line buffer (surrogate training targets).
__global__ void bin_lines_kernel(int64_t n_lines, const double *line_E, const double *line_a, const double *line_w,
                                 const int32_t *line_dir, const int64_t *line_seg, int dir0, int n_dir_chunk,
                                 int64_t n_seg, double lo, double width, int n_bins, float *target) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n_lines;
         i += (int64_t)gridDim.x * blockDim.x) {
        const int dl = line_dir[i] - dir0;
        if (dl < 0 || dl >= n_dir_chunk) continue;
        const int64_t pair = (int64_t)dl * n_seg + line_seg[i];
        const double E_r = line_E[i], a = line_a[i];
        const float s = (float)(a / kPi);
        const float scale = (float)(line_w[i] * kPi / a / width);
        const int c = (int)floor((E_r - lo) / width);
        int K = (int)ceil(64.0 * kPi / (a * width));
        K = K < 1 ? 1 : (K > 64 ? 64 : K);
        const int b0 = max(c - K, 0), b1 = min(c + K, n_bins - 1);
        float r_lo = 0.0f;
        for (int b = b0; b <= b1; ++b) {
            const float x_lo = s * (float)(lo + b * width - E_r);
            const float x_hi = s * (float)(lo + (b + 1) * width - E_r);
            if (b == b0) r_lo = sincsq_tail_f32(x_lo);
            const float r_hi = sincsq_tail_f32(x_hi);
            const float m = r_hi - r_lo + ((x_lo < 0.0f && x_hi >= 0.0f) ? 1.0f : 0.0f);
            r_lo = r_hi;
            if (m != 0.0f) atomicAdd(&target[pair * n_bins + b], scale * m);
        }
    }
}

cudaError_t launch_bin_lines(int64_t n_lines, const double *line_E, const double *line_a, const double *line_w,
                             const int32_t *line_dir, const int64_t *line_seg, int dir0, int n_dir_chunk,
                             int64_t n_seg, double lo, double width, int n_bins, float *target, cudaStream_t st) {
    if (n_lines <= 0) return cudaSuccess;
    const int64_t blocks = std::min<int64_t>((n_lines + 255) / 256, 148 * 16);
    bin_lines_kernel<<<(unsigned)blocks, 256, 0, st>>>(n_lines, line_E, line_a, line_w, line_dir, line_seg, dir0,
                                                        n_dir_chunk, n_seg, lo, width, n_bins, target);
    return cudaGetLastError();
}

}  // namespace pb

// ---------------------------------------------------------------------------
// pb_cxr_score_noalloc: the bin-mean scorer for callers that cannot allocate
// device memory (code running inside a host-side allocator or memory-pool
// callback, an embedding runtime that owns all device memory and forbids
// cudaMalloc, or a static-memory deployment that fixes every allocation at
// load time). Its far-field workspace is this file-scope device array; every
// GPU that loads the library reserves it until the process exits.
// ---------------------------------------------------------------------------
namespace {

constexpr size_t kNoAllocFarDoubles = size_t(1) << 18;  // 2 MiB of FP64 moments
static __device__ __align__(256) double g_noalloc_far[kNoAllocFarDoubles];

// The array's device address differs per CUDA context (a module is loaded
// once per context), so the resolved address is cached per context: keyed by
// the driver's context ID, which stays unique for the life of the process --
// a context re-created after cudaDeviceReset, or one the caller made with the
// driver API, gets a new ID and so a fresh lookup. The two driver functions
// are reached through the runtime (cudaGetDriverEntryPoint), so the library
// does not link the driver library directly.
using CtxGetCurrentFn = CUresult (*)(CUcontext *);
using CtxGetIdFn = CUresult (*)(CUcontext, unsigned long long *);

struct NoAllocSlot {
    unsigned long long ctx_id;
    double *ptr;
};
constexpr int kNoAllocSlots = 64;

std::mutex g_noalloc_mu;
NoAllocSlot g_noalloc_cache[kNoAllocSlots] = {};
int g_noalloc_next = 0;
bool g_ctx_fns_tried = false;
CtxGetCurrentFn g_ctx_get_current = nullptr;
CtxGetIdFn g_ctx_get_id = nullptr;
thread_local char g_noalloc_err[256] = "";

int noalloc_fail(int code, const char *msg) {
    snprintf(g_noalloc_err, sizeof(g_noalloc_err), "%s", msg);
    pb::set_last_error(g_noalloc_err);
    return code;
}

// ID of this thread's current context, making the device's primary context
// current first if none is (cudaSetDevice initialises it). False when the
// driver functions are unavailable or the query fails: the caller then
// resolves the address without the cache.
bool current_ctx_id(int dev, unsigned long long *id) {
    if (!g_ctx_fns_tried) {
        g_ctx_fns_tried = true;
        void *f0 = nullptr, *f1 = nullptr;
        cudaDriverEntryPointQueryResult q0 = cudaDriverEntryPointSymbolNotFound, q1 = q0;
        if (cudaGetDriverEntryPoint("cuCtxGetCurrent", &f0, cudaEnableDefault, &q0) == cudaSuccess &&
            cudaGetDriverEntryPoint("cuCtxGetId", &f1, cudaEnableDefault, &q1) == cudaSuccess &&
            q0 == cudaDriverEntryPointSuccess && q1 == cudaDriverEntryPointSuccess) {
            g_ctx_get_current = reinterpret_cast<CtxGetCurrentFn>(f0);
            g_ctx_get_id = reinterpret_cast<CtxGetIdFn>(f1);
        }
    }
    if (!g_ctx_get_current || !g_ctx_get_id) return false;
    CUcontext ctx = nullptr;
    if (g_ctx_get_current(&ctx) != CUDA_SUCCESS) return false;
    if (!ctx) {
        if (cudaSetDevice(dev) != cudaSuccess || g_ctx_get_current(&ctx) != CUDA_SUCCESS || !ctx) return false;
    }
    return g_ctx_get_id(ctx, id) == CUDA_SUCCESS;
}

}  // namespace

extern "C" int pb_cxr_score_noalloc(const pb_cxr_args *args, void *stream) {
    if (!args) return noalloc_fail(PB_ERR_INVALID, "pb_cxr_score_noalloc: args is NULL");
    if (args->quadrature != PB_QUAD_BINMEAN)
        return noalloc_fail(PB_ERR_UNSUPPORTED,
                            "pb_cxr_score_noalloc: only bin-mean quadrature (node sampling needs a line buffer)");
    // The same argument checks as pb_cxr_score (the far-field workspace is
    // this file's array, so far_moments may be NULL).
    const int v = pb::validate_cxr(*args, "pb_cxr_score_noalloc", true);
    if (v != PB_OK || args->n_seg == 0) return v;
    const bool far = args->exact_widths > 0.0 && args->far_pad >= 0;
    if (far) {
        const size_t need = (size_t)args->n_dir * ((size_t)args->n_E + 2 * (size_t)args->far_pad) * 3;
        if (need > kNoAllocFarDoubles) {
            char msg[256];
            snprintf(msg, sizeof(msg),
                     "pb_cxr_score_noalloc: the far field needs %zu FP64 moments (n_dir * (n_E + 2 far_pad) * 3), "
                     "over the fixed workspace of %zu; score fewer directions per call",
                     need, kNoAllocFarDoubles);
            return noalloc_fail(PB_ERR_CAPACITY, msg);
        }
    }
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0)
        return noalloc_fail(PB_ERR_CUDA, "pb_cxr_score_noalloc: no current CUDA device");
    double *ws = nullptr;
    {
        // First call in a context: resolve the array's device address (host
        // code must not use the symbol itself as a pointer).
        std::lock_guard<std::mutex> lock(g_noalloc_mu);
        unsigned long long cid = 0;
        const bool keyed = current_ctx_id(dev, &cid);
        if (keyed) {
            for (const NoAllocSlot &e : g_noalloc_cache)
                if (e.ptr && e.ctx_id == cid) ws = e.ptr;
        }
        if (!ws) {
            void *p = nullptr;
            const cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_far);
            if (e != cudaSuccess) {
                char msg[256];
                snprintf(msg, sizeof(msg), "pb_cxr_score_noalloc: cudaGetSymbolAddress: %s", cudaGetErrorString(e));
                return noalloc_fail(PB_ERR_CUDA, msg);
            }
            ws = static_cast<double *>(p);
            if (keyed) {
                g_noalloc_cache[g_noalloc_next] = NoAllocSlot{cid, ws};
                g_noalloc_next = (g_noalloc_next + 1) % kNoAllocSlots;
            }
        }
    }
    pb_cxr_args a = *args;
    a.far_moments = far ? ws : nullptr;
    int sms = 148;
    if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) sms = 148;
    const cudaError_t e = pb::launch_cxr(a, (cudaStream_t)stream, sms);
    if (e != cudaSuccess) {
        char msg[256];
        snprintf(msg, sizeof(msg), "pb_cxr_score_noalloc: launch: %s", cudaGetErrorString(e));
        return noalloc_fail(PB_ERR_CUDA, msg);
    }
    return PB_OK;
}

// Depth-node form of the mixed single-slab Bethe-Heitler + Elwert scorer.
//
// The per-(segment, energy) form (pb_brem.cu, brem.py:829-1239) evaluates,
// for every segment s and photon energy k,
//   spec[d][k] += (c0 / k) sum_el w_el(s) J_el(T_s, k) Tbar_d(s, k),
// with w_el = n_el L Z_el^2 den_i(T_s), J_el the electron-energy part of the
// cross section (beta_i / p_i^2 ln((p_i + p_f)/(p_i - p_f)) / beta_f /
// (1 - exp(-2 pi alpha Z_el / beta_f))), and Tbar_d the segment-mean escape
// exp(-mu(k) f_d z') over the segment's depth extent [a_s, b_s] below the exit
// face (f_d = 1/|n_z,d|). Both factors that couple a segment to an energy are
// smooth in one segment variable each, so the double sum factorises:
//
//  * Electron energy. The segments whose T lies in a window [T_lo, T_hi]
//    just below the batch's highest T (T_hi / T_lo <= 1.1, T_lo >= 2.5 k_max)
//    see J_el(T, k) as a degree-5 polynomial in u = (T - T_c) / T_h, fitted at
//    six Chebyshev nodes per (energy, element) and checked at five other
//    points to 1e-7 (else the launch falls back to the per-pair form).
//  * Depth. exp(-lambda z') on cell c of a depth grid is the degree-7
//    polynomial through eight Chebyshev nodes of the cell, whose error is at
//    most (lambda h / 2)^8 e^(lambda h) / (2^7 8!) of the cell's smallest
//    value. The first five cells are h_min = 1/lambda_max wide (lambda_max =
//    max_k mu f_max, so lambda h <= 1: below 2e-9); deeper cells start at z
//    and are 0.2 z wide, where for any lambda the error against the surface
//    value, (0.1 lambda z)^8 e^(-0.8 lambda z) / (2^7 8!), stays below
//    6.5e-11. The segment mean of a polynomial is exact: mean_t t^j over the
//    segment's overlap with a cell, from the cancellation-free divided
//    difference D_{j+1}(t_a, t_b) = sum_i t_b^i t_a^(j-i).
//
// So one pass over the segments accumulates, per (element, face, cell), the
// moments S[p][j] = sum_s w_el u^p mean(t^j) (48 per cell), and one block per
// photon energy contracts them:
//   spec[d][k] += (c0 / k) sum_c sum_i exp(-mu f_d z_ci) W_ci,
//   W_ci = sum_j Lm[i][j] sum_el sum_p A_el,p(k) S_el,face(d),c[p][j],
// Lm the Lagrange basis of the cell nodes in monomials. The work per segment
// no longer depends on the number of energies, and the 16 detector tiles need
// no direction moments. Segments outside the window (and all of them when a
// check fails) go through a list to the per-pair kernels.
//
// Where the electrons slow down through many energies, one window would leave
// most of them out: the list is then ordered by quarter octaves of T (T_hi /
// T_lo <= 1.25, T_lo >= 2.5 k_max) and each has its own polynomials and
// moments, which the contraction sums; a quarter octave whose polynomials miss
// the 1e-7 goes to the per-pair kernels alone.
#include <cstdint>

#include "pb_brem_node.cuh"
#include "pb_common.cuh"

namespace pb {

namespace {

constexpr double kNodeMc2 = 510.99895;
constexpr int kNodeThreads = 256;
constexpr int kContractThreads = 256;
constexpr int kNodeWinTile = 512;  // the same where the list has windows: enough tiles for every block
constexpr int kNodeTile = 2048;  // segments a block orders by depth cell at a time (1024: 7 % slower, 4096: 3 %)

__device__ __forceinline__ bool node_radiates(const pb_brem_args &a, int64_t s) {
    return a.elec_id[s] < a.Ne && (a.seg_layer == nullptr || a.seg_layer[s] == a.emit_layer);
}

__device__ __forceinline__ int64_t node_live(const pb_brem_args &a) {
    int64_t live = a.n_seg;
    if (a.n_seg_device && (int64_t)*a.n_seg_device < live) live = (int64_t)*a.n_seg_device;
    return live;
}

// J_el(T, k) in FP64 (the per-pair FP64 form without w_el and c0 / k), in units
// of m c^2: x = T, y = T - k, gamma = 1 + x, p = sqrt(x (x + 2)), beta = p / gamma,
//   J = ln((p_i + p_f)^2 / (p_i^2 - p_f^2)) (gamma_f / p_f) / (p_i gamma_i (1 - exp(-2 pi alpha Z gamma_f / p_f))),
// the logarithm's p_i^2 - p_f^2 = k (x + y + 2) without cancellation.
__device__ double node_J(double T, double k, double Z) {
    const double Tf = T - k;
    if (!(Tf > 0.0) || !(k > 0.0)) return 0.0;
    constexpr double kInv = 1.0 / kNodeMc2;
    const double x = T * kInv, y = Tf * kInv;
    const double p_i = sqrt(x * (x + 2.0)), p_f = sqrt(y * (y + 2.0));
    const double s = p_i + p_f;
    const double bl = log(s * s / (k * kInv * (x + y + 2.0)));
    const double inv_bf = (1.0 + y) / p_f;
    return bl * inv_bf / (p_i * (1.0 + x) * (1.0 - exp(-2.0 * kPi * kAlphaFs * Z * inv_bf)));
}

// Cell of depth z (boundaries zb, n cells): the closed form of the grid, then
// a step either way against the stored boundaries.
__device__ __forceinline__ int node_cell(const double *zb, int n, double h_min, double z_g, double z) {
    int c;
    if (z < z_g) c = (int)(z / h_min);
    else c = kNodeUniform + (int)(log(z / z_g) * (1.0 / log(kNodeGrowth)));
    c = c < 0 ? 0 : (c > n - 1 ? n - 1 : c);
    while (c > 0 && z < zb[c]) --c;
    while (c < n - 1 && z >= zb[c + 1]) ++c;
    return c;
}

// Extent of the launch: the largest and smallest electron energy of the
// radiating segments and, for a list with windows, their count and their
// histogram over sixteenths of an octave. One atomic a block for each extreme: a
// warp's atomic each on the two addresses took most of this kernel (200,000
// segments, with the histogram: 8.1 -> 5.2 us).
__global__ void __launch_bounds__(kNodeThreads) brem_node_range_kernel(const pb_brem_args a, BremNodeHdr *h,
                                                                       bool count) {
    __shared__ unsigned int hist[kNodeBins];
    __shared__ unsigned long long red[2][kNodeThreads / 32];
    __shared__ unsigned int n_rad;
    const int tid = threadIdx.x;
    for (int q = tid; q < kNodeBins; q += blockDim.x) hist[q] = 0u;
    if (tid == 0) n_rad = 0u;
    __syncthreads();
    const int64_t live = node_live(a);
    unsigned long long mx = 0ULL, mnc = 0ULL;
    unsigned int rads = 0u;
    const int64_t rounds = (live + blockDim.x * (int64_t)gridDim.x - 1) / (blockDim.x * (int64_t)gridDim.x);
    for (int64_t r = 0; r < rounds; ++r) {
        const int64_t s = (r * gridDim.x + blockIdx.x) * (int64_t)blockDim.x + tid;
        const bool rad = s < live && node_radiates(a, s);
        rads += rad ? 1u : 0u;
        const double T = rad ? a.E_keV[s] : 0.0;
        const bool valid = T > 0.0 && T < 1e300;
        if (valid) {
            const unsigned long long b = (unsigned long long)__double_as_longlong(T);
            mx = b > mx ? b : mx;
            mnc = ~b > mnc ? ~b : mnc;
        }
        if (count) {
            // neighbours mostly share a bin: one add a warp then
            const int q = valid ? node_bin(T) : -1;
            int same = 0;
            __match_all_sync(0xffffffffu, q, &same);
            if (same) {
                if ((tid & 31) == 0 && q >= 0 && q < kNodeBins) atomicAdd(&hist[q], 32u);
            } else if (q >= 0 && q < kNodeBins) {
                atomicAdd(&hist[q], 1u);
            }
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const unsigned long long x = __shfl_xor_sync(0xffffffffu, mx, o);
        const unsigned long long y = __shfl_xor_sync(0xffffffffu, mnc, o);
        mx = x > mx ? x : mx;
        mnc = y > mnc ? y : mnc;
    }
    rads = __reduce_add_sync(0xffffffffu, rads);
    if ((tid & 31) == 0) {
        red[0][tid >> 5] = mx;
        red[1][tid >> 5] = mnc;
        if (rads) atomicAdd(&n_rad, rads);
    }
    __syncthreads();
    if (tid == 0) {
        for (int w = 1; w < kNodeThreads / 32; ++w) {
            mx = red[0][w] > mx ? red[0][w] : mx;
            mnc = red[1][w] > mnc ? red[1][w] : mnc;
        }
        if (mx != 0ULL) {
            atomicMax(&h->t_max_bits, mx);
            atomicMax(&h->t_minc_bits, mnc);
        }
        if (n_rad) atomicAdd(&h->n_rad, (unsigned long long)n_rad);
    }
    for (int q = tid; count && q < kNodeBins; q += blockDim.x)
        if (hist[q]) atomicAdd(&h->hist[q], hist[q]);
}

// T_m(t) of the Lagrange basis in monomials: T_{m+1} = 2 t T_m - T_{m-1}.
struct ChebMonomials {
    double c[kNodePts][kNodePts];
};
constexpr ChebMonomials cheb_monomials() {
    ChebMonomials t{};
    t.c[0][0] = 1.0;
    t.c[1][1] = 1.0;
    for (int m = 1; m + 1 < kNodePts; ++m)
        for (int k = 0; k < kNodePts; ++k) t.c[m + 1][k] = (k > 0 ? 2.0 * t.c[m][k - 1] : 0.0) - t.c[m - 1][k];
    return t;
}
__constant__ const ChebMonomials kCheb = cheb_monomials();

// The window or windows, the depth grid, its nodes and the Lagrange basis (one
// block). Directions, cell boundaries and histogram bins go one to a thread:
// a single thread's loops of divisions and powers took 23 us (now 10).
//
// Windows: the one window holds the electrons of a beam that hardly slows
// down. Where the energies spread, the segments certainly below it decide, each
// priced at n_E evaluations of the per-pair form and as much again for its
// place in the list: above kNodePairWork the quarter octaves clear of the
// spectrum's tip become one window each. 200,000 electrons of 8 keV to 10 MeV
// on 2,048 energies: 58 % of them lie in 24 windows, of which the three from 2,048,
// 4,096 and 8,192 keV (1.25 wide, the first quarter of an octave) miss the fit's
// 1e-7 by up to 2.8 times at 1 keV, so 49 % are scored in 21; per-pair form 958 ->
// 490 us (340 on the ordered list); fit, list, moments and contraction of the
// windows 145 us, against 141 us for a list of nearly every segment that the one
// window then gave up. At 300 energies a list of 40,000 takes 324 us through the
// entry point, 436 before; below the line the two are within 10 us.
constexpr double kNodePairWork = 16777216.0;

__global__ void __launch_bounds__(kNodeThreads) brem_node_setup_kernel(const pb_brem_args a, BremNodeHdr *h,
                                                                       int max_win) {
    constexpr int kWarps = kNodeThreads / 32;
    __shared__ double red[3][kWarps];
    __shared__ int n_s, go_s;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    double kmax = 0.0, mumax = 0.0, f_max = 0.0;
    bool finite = true, up = false, down = false;
    for (int e = tid; e < a.n_E; e += blockDim.x) {
        kmax = fmax(kmax, a.E_grid[e] / 1e3);
        const double m = a.mu[e];
        finite = finite && m >= 0.0 && m < 1e300;
        mumax = fmax(mumax, m);
    }
    for (int d = tid; d < a.n_dir; d += blockDim.x) {
        const double nz = a.n_hat[3 * d + 2];
        f_max = fmax(f_max, 1.0 / fmax(fabs(nz), 1.0e-12));
        if (nz < 0.0) up = true;
        else down = true;
    }
    const bool all_finite = __syncthreads_and(finite);
    const unsigned int faces = (__syncthreads_or(up) ? 1u : 0u) | (__syncthreads_or(down) ? 2u : 0u);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        kmax = fmax(kmax, __shfl_xor_sync(0xffffffffu, kmax, o));
        mumax = fmax(mumax, __shfl_xor_sync(0xffffffffu, mumax, o));
        f_max = fmax(f_max, __shfl_xor_sync(0xffffffffu, f_max, o));
    }
    if (lane == 0) {
        red[0][warp] = kmax;
        red[1][warp] = mumax;
        red[2][warp] = f_max;
    }
    if (tid == 0) n_s = kNodeMaxCells + 1;
    __syncthreads();
    for (int w = 0; w < kWarps; ++w) {
        kmax = fmax(kmax, red[0][w]);
        mumax = fmax(mumax, red[1][w]);
        f_max = fmax(f_max, red[2][w]);
    }
    const double T_hi = __longlong_as_double((long long)h->t_max_bits);
    const double T_min = __longlong_as_double((long long)~h->t_minc_bits);
    const double T_lo = fmax(T_min, fmax(T_hi / kNodeWindow, kNodeTip * kmax));
    const double T_slab = a.thickness;
    bool ok = h->t_max_bits != 0ULL && all_finite && T_slab > 0.0;
    // the depth grid: boundary n on thread n, the first at or below the slab's far face ends it
    const double lam = mumax * f_max;
    const double h_min = lam > 0.0 ? fmin(1.0 / lam, T_slab) : T_slab;
    const double z_g = kNodeUniform * h_min;
    double zb = 0.0;
    if (tid <= kNodeMaxCells) {
        zb = tid <= kNodeUniform ? tid * h_min : z_g * pow(kNodeGrowth, (double)(tid - kNodeUniform));
        if (tid > 0 && !(zb < T_slab)) atomicMin(&n_s, tid);
    }
    __syncthreads();
    const int n = n_s;
    ok = ok && n <= kNodeMaxCells;
    if (ok && tid <= n) h->zb[tid] = tid < n ? zb : T_slab;
    int n_win = 0;
    if (warp == 0) {
        // two quarter octaves a lane, upwards in energy
        unsigned int below = 0u, in_bins = 0u;
        unsigned int c[2];
        unsigned int use[2];
        for (int k = 0; k < 2; ++k) {
            const int q = lane + 32 * k;
            c[k] = 0u;
            for (int t = 4 * q; t < 4 * q + 4; ++t) {
                c[k] += h->hist[t];
                if (node_bin_lo(t + 1) <= T_lo) below += h->hist[t];
            }
            in_bins += c[k];
            use[k] = __ballot_sync(0xffffffffu, c[k] > 0u && node_bin_lo(4 * q) >= kNodeTip * kmax);
        }
        below = __reduce_add_sync(0xffffffffu, below);
        in_bins = __reduce_add_sync(0xffffffffu, in_bins);
        // (bins only count where the list has windows)
        const unsigned long long left = in_bins ? h->n_rad - in_bins + below : 0ULL;
        if (ok && max_win > 1 && (double)left * (a.n_E + 1024.0) > kNodePairWork) n_win = min(__popc(use[0]) + __popc(use[1]), max_win);
        for (int k = 0; k < 2; ++k) {
            const int q = lane + 32 * k;
            const int w = __popc(use[k] & ((1u << lane) - 1u)) + (k ? __popc(use[0]) : 0);
            const bool on = ((use[k] >> lane) & 1u) && w < n_win;
            h->win_of[q] = on ? w : -1;
            if (on) {
                const double lo = node_bin_lo(4 * q), hi = node_bin_lo(4 * q + 4);
                h->win_Tc[w] = 0.5 * (lo + hi);
                h->win_Th[w] = 0.5 * (hi - lo);
                h->win_n[w] = c[k];
            }
        }
        if (lane == 0) {
            ok = ok && (n_win > 0 || T_lo <= T_hi);
            h->n_cells = ok ? n : 0;
            h->faces = faces;
            h->n_win = n_win;
            h->T_lo = T_lo;
            h->T_hi = T_hi;
            h->Tc = 0.5 * (T_lo + T_hi);
            h->Th = 0.5 * (T_hi - T_lo);
            h->h_min = h_min;
            h->z_g = z_g;
            if (n_win == 0) {
                h->win_Tc[0] = 0.5 * (T_lo + T_hi);
                h->win_Th[0] = 0.5 * (T_hi - T_lo);
            }
            go_s = ok ? 1 : 0;
        }
    }
    __syncthreads();
    if (!go_s) return;  // h->ok stays 0 (the workspace was zeroed)
    // the cells' Chebyshev nodes
    for (int q = tid; q < n * kNodePts; q += blockDim.x) {
        const int c = q / kNodePts, i = q - c * kNodePts;
        const double mid = 0.5 * (h->zb[c] + h->zb[c + 1]), hw = 0.5 * (h->zb[c + 1] - h->zb[c]);
        h->node[q] = mid + hw * cospi((2 * i + 1) * (1.0 / (2 * kNodePts)));
    }
    // Lagrange basis of the Chebyshev nodes x_i: l_i(t) = (1/n) [1 + 2 sum_m T_m(x_i) T_m(t)]
    if (tid < kNodePts * kNodePts) {
        const int i = tid / kNodePts, j = tid - i * kNodePts;
        double v = 0.0;
        for (int m = 0; m < kNodePts; ++m)
            v += (m == 0 ? 1.0 : 2.0) / kNodePts * cospi(m * (2 * i + 1) * (1.0 / (2 * kNodePts))) * kCheb.c[m][j];
        h->Lm[tid] = v;
    }
    __syncthreads();
    if (tid == 0) h->ok = 1u;
}

// J_el over a window as a degree-5 polynomial in u, per (energy, element):
// Chebyshev coefficients from six nodes, then monomials; checked against J
// at u = -1, -1/2, 0, 1/2, 1 to 1e-7 (a miss turns the node form off, or the
// window where there are several). 16 lanes take one polynomial, one
// evaluation of J a lane (one thread for all eleven: 23 us for 2,048 energies,
// now 5).
constexpr int kFitLanes = 16;
__global__ void __launch_bounds__(128) brem_node_fit_kernel(const pb_brem_args a, BremNodeHdr *h, double *A) {
    const int w = blockIdx.y;
    if (!__syncthreads_and(h->ok != 0u && w < max(h->n_win, 1))) return;
    const int q = (int)((blockIdx.x * blockDim.x + threadIdx.x) / kFitLanes);
    const int lane = threadIdx.x % kFitLanes;
    const bool on = q < a.n_E * a.n_el;
    const int e = on ? q / a.n_el : 0, el = on ? q - e * a.n_el : 0;
    const double k = a.E_grid[e] / 1e3;
    // lanes 0..5: the nodes; 6..10: the points of the check
    const double cos_l = cospi((threadIdx.x & 31) * (1.0 / (2 * kNodeTDeg)));  // of the warp's lane: cos(l pi / 12)
    const double x_l = __shfl_sync(0xffffffffu, cos_l, 2 * lane + 1);
    const double u = lane < kNodeTDeg ? x_l : -1.0 + 0.5 * (lane - kNodeTDeg);
    const bool eval = on && lane < kNodeTDeg + 5 && k > 0.0;
    const double J = eval ? node_J(h->win_Tc[w] + h->win_Th[w] * u, k, a.Z[el]) : 0.0;
    double c = 0.0;  // lane p < 6: the coefficient of T_p
    for (int m = 0; m < kNodeTDeg; ++m)
        c += __shfl_sync(0xffffffffu, J, m, kFitLanes) *
             __shfl_sync(0xffffffffu, cos_l, lane * (2 * m + 1) % (4 * kNodeTDeg));
    c *= (lane == 0 ? 1.0 : 2.0) / kNodeTDeg;
    double cp[kNodeTDeg];
    for (int p = 0; p < kNodeTDeg; ++p) cp[p] = __shfl_sync(0xffffffffu, c, p, kFitLanes);
    // T_0..T_5 in monomials
    const double P[kNodeTDeg] = {cp[0] - cp[2] + cp[4],      cp[1] - 3.0 * cp[3] + 5.0 * cp[5],
                                 2.0 * cp[2] - 8.0 * cp[4],  4.0 * cp[3] - 20.0 * cp[5],
                                 8.0 * cp[4],                16.0 * cp[5]};
    const double pv = ((((P[5] * u + P[4]) * u + P[3]) * u + P[2]) * u + P[1]) * u + P[0];
    if (on && lane == 0) {
        double *out = A + ((int64_t)w * a.n_E * a.n_el + q) * kNodeTDeg;
#pragma unroll
        for (int p = 0; p < kNodeTDeg; ++p) out[p] = P[p];
    }
    if (eval && lane >= kNodeTDeg && !(fabs(pv - J) <= 1e-7 * fabs(J))) {
        atomicExch(&h->win_bad[w], 1u);
        if (h->n_win == 0) atomicExch(&h->ok, 0u);
    }
}

// Where the windows' segments go in the list: the left-out ones first, then
// window by window (a window whose fit missed has no part). Whole warps.
__device__ __forceinline__ void node_window_offsets(const BremNodeHdr *h, int n_win, int lane, int64_t &off,
                                                    unsigned int &n) {
    n = lane < n_win && !h->win_bad[lane] ? h->win_n[lane] : 0u;
    unsigned long long incl = n;
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned long long v = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += v;
    }
    const unsigned long long all = __shfl_sync(0xffffffffu, incl, 31);
    off = (int64_t)(h->n_rad - all + incl - n);
}

// Segment list by window, the left-out part by sixteenths of an octave (its
// chunks then span little energy, which the per-pair kernel's cubic and its
// test against the photon energy need: 490 -> 340 us for 84,000 electrons of 8 to
// 160 keV and 18,000 of windows given up, 2,048 energies to 60 keV): each block counts a tile's segments per
// place in shared memory, reserves them with one atomic a place and writes them.
constexpr int kListPer = 4;  // segments per thread and tile
constexpr int kListPlaces = kNodeBins + 1 + kNodeMaxWin;  // bins, outside of them, windows
__global__ void __launch_bounds__(kNodeThreads) brem_node_list_kernel(const pb_brem_args a, BremNodeHdr *h,
                                                                      int64_t *idx, int64_t cap) {
    static_assert(kNodeThreads == kNodeBins, "a bin a thread in the scan");
    __shared__ unsigned int cnt[kListPlaces];
    __shared__ int64_t base[kListPlaces];
    __shared__ int64_t off_s[kListPlaces];
    __shared__ int win_s[kNodeQuarters];
    __shared__ unsigned int sum_s[kNodeThreads / 32];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int n_win = h->n_win;
    if (!h->ok || n_win == 0) return;
    if (tid < kNodeQuarters) {
        const int w = h->win_of[tid];
        win_s[tid] = w >= 0 && !h->win_bad[w] ? w : -1;
    }
    __syncthreads();
    {
        const unsigned int n = win_s[tid >> 2] < 0 ? h->hist[tid] : 0u;
        unsigned int incl = n;
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned int v = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += v;
        }
        if (lane == 31) sum_s[warp] = incl;
        __syncthreads();
        for (int w = 0; w < warp; ++w) incl += sum_s[w];
        off_s[tid] = incl - n;
        // outside the bins: after them; the windows follow
        if (tid == kNodeThreads - 1) off_s[kNodeBins] = incl;
    }
    if (warp == 0) {
        int64_t off;
        unsigned int n;
        node_window_offsets(h, n_win, lane, off, n);
        off_s[kNodeBins + 1 + lane] = off;
        if (blockIdx.x == 0 && lane == 0) h->n_out = (unsigned long long)off;  // window 0 starts behind the left-out ones
    }
    const int64_t live = node_live(a);
    constexpr int kTile = kNodeThreads * kListPer;
    for (int64_t t0 = blockIdx.x * (int64_t)kTile; t0 < live; t0 += gridDim.x * (int64_t)kTile) {
        for (int q = tid; q < kListPlaces; q += blockDim.x) cnt[q] = 0u;
        __syncthreads();
        int place[kListPer];
        unsigned int rank[kListPer];
#pragma unroll
        for (int k = 0; k < kListPer; ++k) {
            const int64_t s = t0 + k * kNodeThreads + tid;
            place[k] = -1;
            rank[k] = 0u;
            if (s < live && node_radiates(a, s)) {
                const double T = a.E_keV[s];
                const int q = T > 0.0 && T < 1e300 ? node_bin(T) : -1;
                place[k] = kNodeBins;
                if (q >= 0 && q < kNodeBins) place[k] = win_s[q >> 2] >= 0 ? kNodeBins + 1 + win_s[q >> 2] : q;
                rank[k] = atomicAdd(&cnt[place[k]], 1u);
            }
        }
        __syncthreads();
        for (int q = tid; q < kListPlaces; q += blockDim.x)
            if (cnt[q])
                base[q] = off_s[q] + atomicAdd(q <= kNodeBins ? &h->fill[q] : &h->win_fill[q - kNodeBins - 1], cnt[q]);
        __syncthreads();
#pragma unroll
        for (int k = 0; k < kListPer; ++k) {
            if (place[k] < 0) continue;
            const int64_t at = base[place[k]] + rank[k];
            if (at < cap) idx[at] = t0 + k * kNodeThreads + tid;
        }
    }
}

// D += A B on the FP64 tensor cores, one m8n8k4 tile: lane l holds
// A[l / 4][l % 4], B[l % 4][l / 4] and D[l / 4][2 (l % 4) + {0, 1}].
__device__ __forceinline__ void dmma_884(double &d0, double &d1, double a, double b) {
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
                 : "+d"(d0), "+d"(d1)
                 : "d"(a), "d"(b));
}

// One pass over the segments, a warp per group of 32 consecutive segments, a
// lane per segment. Each lane tests its segment against the window (the
// others are appended to the left-out list, one atomic per warp) and forms
// its weights w_el u^p and each face's depth extent. Then the lanes walk
// their segments' cells in rounds: in each round every lane with a piece left
// forms the piece's eight depth moments mean(t^j), and the lanes whose pieces
// share a cell add their outer products w_el u^p x mean(t^j) in one FP64
// tensor-core product (the 6 x 32 weights times the 32 x 8 moments, as eight
// m8n8k4 steps over the lanes); 48 lanes' worth of sums then go to the
// block's float accumulator in shared memory, one address per lane.
// Consecutive segments come from one transport step of neighbouring
// histories, so a round's pieces mostly share a cell and a warp issues a few
// tensor-core products per round. The block's sums are folded into the FP64
// moments at the end.
constexpr int kNodeWarps = kNodeThreads / 32;

// Dynamic shared memory of the moment pass: the block's float accumulator,
// then per warp the lanes' weights and piece moments.
constexpr int kNodeRow = kNodePts + 1;  // padded row of the staged weights and moments (2-way bank conflicts)
__host__ __device__ constexpr size_t node_accum_smem(int n_el) {
    return sizeof(double) * (size_t)kNodeWarps * (n_el + 1) * 32 * kNodeRow +
           sizeof(float) * (size_t)n_el * 2 * kNodeMaxCells * kNodePJ;
}

template <int NEL>
__global__ void __launch_bounds__(kNodeThreads, 2) brem_node_accum_kernel(const pb_brem_args a, BremNodeHdr *h,
                                                                           double *S, int64_t *idx, int64_t cap) {
    constexpr int kWarps = kNodeWarps;
    extern __shared__ __align__(16) unsigned char node_smem[];
    // weights w_el u^p of each lane's piece (p < 6) and its depth moments
    double (*sW)[NEL][32][kNodeRow] = reinterpret_cast<double (*)[NEL][32][kNodeRow]>(node_smem);
    double (*sM)[32][kNodeRow] =
        reinterpret_cast<double (*)[32][kNodeRow]>(node_smem + sizeof(double) * kWarps * NEL * 32 * kNodeRow);
    float *Ss = reinterpret_cast<float *>(node_smem + sizeof(double) * kWarps * (NEL + 1) * 32 * kNodeRow);
    __shared__ double zb_s[kNodeMaxCells + 1];
    __shared__ double mid_s[kNodeMaxCells], ihw_s[kNodeMaxCells];  // cell centre and 2 / width
    __shared__ unsigned short ord_s[kNodeTile];   // the tile's window segments in cell order
    __shared__ unsigned char key_s[kNodeTile];    // start cell per segment (kNodeMaxCells: not in the window)
    __shared__ int cnt_s[kNodeMaxCells + 1];
    __shared__ int n_in_s;
    __shared__ int64_t off_s[kNodeMaxWin];   // windows: start in the list, segments, first tile
    __shared__ unsigned int win_n_s[kNodeMaxWin];
    __shared__ int win_t_s[kNodeMaxWin + 1];
    __shared__ double prm[4];
    __shared__ int go_s, nc_s, n_win_s;
    __shared__ unsigned int faces_s;
    const int tid = threadIdx.x;
    if (tid == 0) {
        go_s = h->ok ? 1 : 0;
        nc_s = h->n_cells;
        n_win_s = h->n_win;
        faces_s = h->faces;
        prm[0] = h->T_lo;
        prm[1] = h->T_hi;
        prm[2] = h->h_min;
        prm[3] = h->z_g;
    }
    __syncthreads();
    if (!go_s) return;
    const int nc = nc_s, n_win = n_win_s;
    if (n_win > 0 && tid < 32) {
        int64_t off;
        unsigned int n;
        node_window_offsets(h, n_win, tid, off, n);
        off_s[tid] = off;
        win_n_s[tid] = n;
        int incl = (int)((n + kNodeWinTile - 1) / kNodeWinTile);
        const int own = incl;
        for (int o = 1; o < 32; o <<= 1) {
            const int v = __shfl_up_sync(0xffffffffu, incl, o);
            if (tid >= o) incl += v;
        }
        win_t_s[tid] = incl - own;
        if (tid == 31) win_t_s[32] = incl;
    }
    const unsigned int faces = faces_s;
    for (int c = tid; c <= nc; c += blockDim.x) zb_s[c] = h->zb[c];
    for (int c = tid; c < nc; c += blockDim.x) {
        mid_s[c] = 0.5 * (h->zb[c] + h->zb[c + 1]);
        ihw_s[c] = 2.0 / (h->zb[c + 1] - h->zb[c]);
    }
    for (int q = tid; q < NEL * 2 * kNodeMaxCells * kNodePJ; q += blockDim.x) Ss[q] = 0.0f;
    __syncthreads();
    const double T_lo = prm[0], T_hi = prm[1], h_min = prm[2], z_g = prm[3];
    double Tc = h->win_Tc[0], inv_Th = h->win_Th[0] > 0.0 ? 1.0 / h->win_Th[0] : 0.0;
    const double T_slab = a.thickness;
    const double za = 2.0 * kPi * kAlphaFs;
    const int64_t live = node_live(a);
    const unsigned int lane = tid & 31;
    const int warp = tid >> 5;
    const int grow = (int)(lane >> 2), gcol = (int)(lane & 3);  // tile row / column group of this lane
    constexpr double kInvJ1[kNodePts] = {1.0, 1.0 / 2, 1.0 / 3, 1.0 / 4, 1.0 / 5, 1.0 / 6, 1.0 / 7, 1.0 / 8};
    // Tiles of kNodeTile consecutive segments, ordered by the depth cell of
    // their start on the first face in use (a counting sort in shared
    // memory), so that the 32 segments a warp takes share their cells and a
    // round of pieces needs one or two tensor-core products.
    const int f0 = (faces & 1u) ? 0 : 1;
    // The block's sums of window w into the FP64 moments.
    const auto fold = [&](int w, bool clear) {
        const int per = nc * kNodePJ;
        for (int q = tid; q < NEL * 2 * per; q += blockDim.x) {
            const int ef = q / per, r = q - ef * per;
            if (!((faces >> (ef & 1)) & 1u)) continue;
            const int off = ef * kNodeMaxCells * kNodePJ + r;
            const float v = Ss[off];
            if (v != 0.0f) atomicAdd(&S[(int64_t)w * NEL * 2 * kNodeMaxCells * kNodePJ + off], (double)v);
            if (clear) Ss[off] = 0.0f;
        }
    };
    // One window: the blocks stride over the tiles of the segment list. Several:
    // each takes a contiguous run of the windows' tiles, so that its sums change
    // window seldom.
    const int64_t n_tiles = n_win > 0 ? win_t_s[32] : (live + kNodeTile - 1) / kNodeTile;
    const int64_t tile_0 = n_win > 0 ? n_tiles * blockIdx.x / gridDim.x : blockIdx.x;
    const int64_t tile_1 = n_win > 0 ? n_tiles * (blockIdx.x + 1) / gridDim.x : n_tiles;
    int win = 0;
    bool any = false;
    for (int64_t tile = tile_0; tile < tile_1; tile += n_win > 0 ? 1 : gridDim.x) {
        int64_t t0 = tile * kNodeTile;       // first segment, or first entry of the list
        int64_t t_end = live;
        int rounds = kNodeTile / kNodeThreads;
        if (n_win > 0) {
            int w = win;
            while (w + 1 < n_win && tile >= win_t_s[w + 1]) ++w;
            if (w != win || !any) {
                if (any) {
                    fold(win, true);
                    __syncthreads();
                }
                win = w;
                Tc = h->win_Tc[w];
                inv_Th = 1.0 / h->win_Th[w];
            }
            t0 = off_s[w] + (tile - win_t_s[w]) * kNodeWinTile;
            t_end = off_s[w] + win_n_s[w];
            rounds = kNodeWinTile / kNodeThreads;
        }
        any = true;
        for (int q = tid; q <= kNodeMaxCells; q += blockDim.x) cnt_s[q] = 0;
        __syncthreads();
#pragma unroll 1
        for (int k = 0; k < rounds; ++k) {
            const int li = k * kNodeThreads + tid;
            int64_t s = t0 + li;
            bool in_win = s < t_end, left = false;
            if (n_win > 0) {
                if (in_win) s = idx[s];
            } else {
                const bool rad = in_win && node_radiates(a, s);
                const double T = rad ? a.E_keV[s] : 0.0;
                in_win = rad && T >= T_lo && T <= T_hi;
                left = rad && !in_win;
            }
            const unsigned int lm = __ballot_sync(0xffffffffu, left);
            if (lm) {
                const int ld = __ffs(lm) - 1;
                unsigned long long q0 = 0ULL;
                if ((int)lane == ld) q0 = atomicAdd(&h->n_out, (unsigned long long)__popc(lm));
                q0 = __shfl_sync(0xffffffffu, q0, ld);
                if (left) {
                    const unsigned long long q = q0 + (unsigned long long)__popc(lm & ((1u << lane) - 1u));
                    if (q < (unsigned long long)cap) idx[q] = s;
                    else atomicExch(&h->ok, 0u);  // list full: the per-pair form takes every segment
                }
            }
            int key = kNodeMaxCells;  // outside the window: after every cell
            if (in_win) {
                const double half = 0.5 * a.L[s];
                const double zm = a.r_mid[3 * s + 2], vz = a.v_hat[3 * s + 2];
                const double d0 = fmin(fmax(zm - half * vz, 0.0), T_slab);
                const double d1 = fmin(fmax(zm + half * vz, 0.0), T_slab);
                const double zs = f0 == 0 ? fmin(d0, d1) : T_slab - fmax(d0, d1);
                key = node_cell(zb_s, nc, h_min, z_g, zs);
            }
            key_s[li] = (unsigned char)key;
            atomicAdd(&cnt_s[key], 1);
        }
        __syncthreads();
        if (tid == 0) {
            int run = 0;
            for (int c = 0; c <= kNodeMaxCells; ++c) {
                const int v = cnt_s[c];
                cnt_s[c] = run;
                run += v;
            }
            n_in_s = cnt_s[kNodeMaxCells];
        }
        __syncthreads();
#pragma unroll 1
        for (int k = 0; k < rounds; ++k) {
            const int li = k * kNodeThreads + tid;
            const int pos = atomicAdd(&cnt_s[key_s[li]], 1);
            ord_s[pos] = (unsigned short)li;
        }
        __syncthreads();
        const int n_in = n_in_s;
        for (int g = warp; g * 32 < n_in; g += kWarps) {
            const int pos = g * 32 + (int)lane;
            const bool in_win = pos < n_in;
            int64_t s = in_win ? t0 + ord_s[pos] : 0;
            if (n_win > 0 && in_win) s = idx[s];
            const double T = in_win ? a.E_keV[s] : 0.0;
            double lo = 0.0, hi = 0.0;
            if (in_win) {
                const double u = (T - Tc) * inv_Th;
                // 1 / beta_i = (T + m c^2) / sqrt(T (T + 2 m c^2))
                const double inv_bi = (T + kNodeMc2) / sqrt(T * (T + 2.0 * kNodeMc2));
                const double Lc = a.L[s];
    #pragma unroll
                for (int el = 0; el < NEL; ++el) {
                    const double Z = a.Z[el];
                    double wp = a.n_ang3[el] * 1e24 * (Lc * 1e-8) * (Z * Z) * (1.0 - exp(-za * Z * inv_bi));
    #pragma unroll
                    for (int p = 0; p < kNodePts; ++p) {
                        sW[warp][el][lane][p] = p < kNodeTDeg ? wp : 0.0;
                        wp *= u;
                    }
                }
                const double half = 0.5 * Lc;
                const double zm = a.r_mid[3 * s + 2], vz = a.v_hat[3 * s + 2];
                const double d0 = fmin(fmax(zm - half * vz, 0.0), T_slab);
                const double d1 = fmin(fmax(zm + half * vz, 0.0), T_slab);
                lo = fmin(d0, d1);
                hi = fmax(d0, d1);
            }
    #pragma unroll
            for (int f = 0; f < 2; ++f) {
                if (!((faces >> f) & 1u)) continue;
                const double za_ = f == 0 ? lo : T_slab - hi;
                const double zb_ = f == 0 ? hi : T_slab - lo;
                int c = 0, cend = -1;
                bool point = false;
                double inv_len = 0.0;
                if (in_win) {
                    c = node_cell(zb_s, nc, h_min, z_g, za_);
                    point = !(zb_ - za_ > 1e-9 * (zb_s[c + 1] - zb_s[c]));
                    cend = point ? c : node_cell(zb_s, nc, h_min, z_g, zb_);
                    inv_len = point ? 0.0 : 1.0 / (zb_ - za_);
                }
                while (__any_sync(0xffffffffu, c <= cend)) {
                    const bool have = c <= cend;
                    double M[kNodePts];
    #pragma unroll
                    for (int j = 0; j < kNodePts; ++j) M[j] = 0.0;
                    if (have) {
                        const double mid = mid_s[c], ihw = ihw_s[c];
                        if (point) {
                            const double t = fmin(fmax((za_ - mid) * ihw, -1.0), 1.0);
                            M[0] = 1.0;
    #pragma unroll
                            for (int j = 1; j < kNodePts; ++j) M[j] = M[j - 1] * t;
                        } else {
                            const double oa = fmax(za_, zb_s[c]), ob = fmin(zb_, zb_s[c + 1]);
                            if (ob > oa) {
                                const double ta = fmin(fmax((oa - mid) * ihw, -1.0), 1.0);
                                const double tb = fmin(fmax((ob - mid) * ihw, -1.0), 1.0);
                                const double frac = (ob - oa) * inv_len;
                                // D_1 = 1, D_{n+1} = t_b D_n + t_a^n; mean of t^j = frac D_{j+1} / (j + 1)
                                double D = 1.0, tan = ta;
                                M[0] = frac;
    #pragma unroll
                                for (int j = 1; j < kNodePts; ++j) {
                                    D = fma(tb, D, tan);
                                    tan *= ta;
                                    M[j] = frac * D * kInvJ1[j];
                                }
                            }
                        }
                    }
    #pragma unroll
                    for (int j = 0; j < kNodePts; ++j) sM[warp][lane][j] = M[j];
                    __syncwarp();
                    const int key = have ? c : -1;
                    unsigned int pending = __ballot_sync(0xffffffffu, have);
                    while (pending) {
                        const int ld = __ffs(pending) - 1;
                        const int K = __shfl_sync(0xffffffffu, key, ld);
                        const unsigned int grp = __ballot_sync(0xffffffffu, have && key == K);
                        pending &= ~grp;
    #pragma unroll
                        for (int el = 0; el < NEL; ++el) {
                            double d0 = 0.0, d1 = 0.0;
    #pragma unroll
                            for (int st = 0; st < 8; ++st) {
                                const int l = 4 * st + gcol;
                                const double av = ((grp >> l) & 1u) ? sW[warp][el][l][grow] : 0.0;
                                dmma_884(d0, d1, av, sM[warp][l][grow]);
                            }
                            if (grow < kNodeTDeg) {
                                float *row = Ss + ((el * 2 + f) * kNodeMaxCells + K) * kNodePJ + grow * kNodePts + 2 * gcol;
                                if (d0 != 0.0) atomicAdd(row, (float)d0);
                                if (d1 != 0.0) atomicAdd(row + 1, (float)d1);
                            }
                        }
                    }
                    __syncwarp();
                    ++c;
                }
            }
        }
        __syncthreads();  // the next tile reuses the order
    }
    __syncthreads();
    if (any) fold(win, false);
}

// kE photon energies a block: the moments of the windows summed over
// the energy polynomial, W_ci from them, then every direction's sum over the
// cells' nodes, a warp per (direction, energy) with its lanes over the nodes of
// all cells. The moments are read once for the block's energies (windows: up
// to 0.8 MB of them), else the exponentials bound it (one window, 16 directions
// x 2,048 energies, lanes over cells before: 59 -> 34-40 us).
constexpr int kE = 4;             // photon energies a block (8: 34 -> 59 us, too few blocks)
constexpr int kContractWin = 16;  // windows whose coefficients are staged at a time

template <int NEL>
__global__ void __launch_bounds__(kContractThreads) brem_node_contract_kernel(const pb_brem_args a,
                                                                              const BremNodeHdr *h, const double *A,
                                                                              const double *S) {
    __shared__ double Zs[kE][kNodeMaxCells * kNodePts];  // then W
    __shared__ double Lm_s[kNodePts][kNodePts + 1];
    __shared__ double A_s[kContractWin][NEL * kNodeTDeg][kE];
    const int tid = threadIdx.x;
    const int e0 = blockIdx.x * kE;
    if (!h->ok) return;
    const int nc = h->n_cells;
    const int n_win = h->n_win > 0 ? h->n_win : 1;
    const unsigned int faces = h->faces;
    for (int q = tid; q < kNodePts * kNodePts; q += blockDim.x) Lm_s[q / kNodePts][q % kNodePts] = h->Lm[q];
    constexpr int kPer = (kNodeMaxCells * kNodePts + kContractThreads - 1) / kContractThreads;
    for (int f = 0; f < 2; ++f) {
        if (!((faces >> f) & 1u)) continue;
        // Z_cj = sum over windows, elements and powers of A S, a (cell, power of t) a thread
        double Z[kPer][kE];
#pragma unroll
        for (int r = 0; r < kPer; ++r)
#pragma unroll
            for (int x = 0; x < kE; ++x) Z[r][x] = 0.0;
        for (int w0 = 0; w0 < n_win; w0 += kContractWin) {
            const int nw = min(kContractWin, n_win - w0);
            __syncthreads();
            // (a window whose fit missed has no moments)
            for (int q = tid; q < nw * NEL * kNodeTDeg * kE; q += blockDim.x) {
                const int ep = q % (NEL * kNodeTDeg), r = q / (NEL * kNodeTDeg);
                const int x = r % kE, w = r / kE;
                const int e = e0 + x;
                A_s[w][ep][x] = e < a.n_E && a.E_grid[e] > 0.0 && !h->win_bad[w0 + w]
                                    ? A[((int64_t)(w0 + w) * a.n_E + e) * NEL * kNodeTDeg + ep] : 0.0;
            }
            __syncthreads();
#pragma unroll 2
            for (int w = 0; w < nw; ++w) {
#pragma unroll
                for (int el = 0; el < NEL; ++el) {
                    const double *Sw = S + (((int64_t)(w0 + w) * NEL + el) * 2 + f) * kNodeMaxCells * kNodePJ;
#pragma unroll
                    for (int r = 0; r < kPer; ++r) {
                        const int q = r * kContractThreads + tid;
                        if (q >= nc * kNodePts) break;
                        const double *row = Sw + (q / kNodePts) * kNodePJ + q % kNodePts;
#pragma unroll
                        for (int p = 0; p < kNodeTDeg; ++p) {
                            const double v = row[p * kNodePts];
#pragma unroll
                            for (int x = 0; x < kE; ++x) Z[r][x] = fma(A_s[w][el * kNodeTDeg + p][x], v, Z[r][x]);
                        }
                    }
                }
            }
        }
        __syncthreads();  // the other face's W has been read
#pragma unroll
        for (int r = 0; r < kPer; ++r) {
            const int q = r * kContractThreads + tid;
            if (q >= nc * kNodePts) break;
#pragma unroll
            for (int x = 0; x < kE; ++x) Zs[x][q] = Z[r][x];
        }
        __syncthreads();
        // W_ci = sum_j Lm[i][j] Z_cj, the cell's eight in place
#pragma unroll
        for (int r = 0; r < kPer; ++r) {
            const int q = r * kContractThreads + tid;
            const int c8 = q / kNodePts * kNodePts, i = q % kNodePts;
            if (q >= nc * kNodePts) break;
#pragma unroll
            for (int x = 0; x < kE; ++x) {
                double v = 0.0;
#pragma unroll
                for (int j = 0; j < kNodePts; ++j) v = fma(Lm_s[i][j], Zs[x][c8 + j], v);
                Z[r][x] = v;
            }
        }
        __syncthreads();
#pragma unroll
        for (int r = 0; r < kPer; ++r) {
            const int q = r * kContractThreads + tid;
            if (q >= nc * kNodePts) break;
#pragma unroll
            for (int x = 0; x < kE; ++x) Zs[x][q] = Z[r][x];
        }
        __syncthreads();
        const int warp = tid >> 5, lane = tid & 31;
        for (int t = warp; t < a.n_dir * kE; t += kContractThreads / 32) {
            const int d = t / kE, x = t - d * kE, e = e0 + x;
            const double nz = a.n_hat[3 * d + 2];
            if (e >= a.n_E || !(a.E_grid[e] > 0.0) || (nz < 0.0 ? 0 : 1) != f) continue;
            const double lam = a.mu[e] / fmax(fabs(nz), 1.0e-12);
            double acc = 0.0;
            for (int q = lane; q < nc * kNodePts; q += 32) acc = fma(exp(-lam * h->node[q]), Zs[x][q], acc);
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
            const double scale = 16.0 / 3.0 * kAlphaFs * kReCm2 / a.E_grid[e];
            if (lane == 0 && acc != 0.0) atomicAdd(&a.spec[(int64_t)d * a.n_E + e], scale * acc);
        }
    }
}

}  // namespace

cudaError_t launch_brem_node(const pb_brem_args &a, cudaStream_t s, int sms, const BremNodeHdr **hdr,
                             const int64_t **idx) {
    *hdr = nullptr;
    *idx = nullptr;
    if (a.work == nullptr || !brem_node_applies(a) || a.n_seg <= 0) return cudaSuccess;
    const BremNodeLayout l = brem_node_layout(a);
    if (a.work_bytes < (int64_t)l.total) return cudaSuccess;
    unsigned char *w = static_cast<unsigned char *>(a.work);
    BremNodeHdr *h = reinterpret_cast<BremNodeHdr *>(w + l.hdr);
    double *A = reinterpret_cast<double *>(w + l.A);
    double *S = reinterpret_cast<double *>(w + l.S);
    int64_t *ix = reinterpret_cast<int64_t *>(w + l.idx);
    cudaError_t err = cudaMemsetAsync(w, 0, l.zero_bytes, s);
    if (err != cudaSuccess) return err;
    brem_node_range_kernel<<<sms * 4, kNodeThreads, 0, s>>>(a, h, l.n_win > 1);
    brem_node_setup_kernel<<<1, kNodeThreads, 0, s>>>(a, h, l.n_win);
    constexpr int kFitPer = 128 / kFitLanes;
    const int nq = a.n_E * a.n_el;
    brem_node_fit_kernel<<<dim3((nq + kFitPer - 1) / kFitPer, l.n_win), 128, 0, s>>>(a, h, A);
    if (l.n_win > 1) brem_node_list_kernel<<<sms * 4, kNodeThreads, 0, s>>>(a, h, ix, l.cap);
    err = cudaGetLastError();
    if (err != cudaSuccess) return err;
    using Accum = void (*)(const pb_brem_args, BremNodeHdr *, double *, int64_t *, int64_t);
    using Contract = void (*)(const pb_brem_args, const BremNodeHdr *, const double *, const double *);
    const Accum acc = a.n_el == 1 ? brem_node_accum_kernel<1> : brem_node_accum_kernel<2>;
    const Contract con = a.n_el == 1 ? brem_node_contract_kernel<1> : brem_node_contract_kernel<2>;
    const int smem = (int)node_accum_smem(a.n_el);
    err = cudaFuncSetAttribute(acc, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (err != cudaSuccess) return err;
    err = cudaFuncSetAttribute(acc, cudaFuncAttributePreferredSharedMemoryCarveout, (int)cudaSharedmemCarveoutMaxShared);
    if (err != cudaSuccess) return err;
    int per_sm = 0;
    err = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, acc, kNodeThreads, smem);
    if (err != cudaSuccess) return err;
    if (per_sm < 1) per_sm = 1;
    acc<<<sms * per_sm, kNodeThreads, smem, s>>>(a, h, S, ix, l.cap);
    con<<<(a.n_E + kE - 1) / kE, kContractThreads, 0, s>>>(a, h, A, S);
    err = cudaGetLastError();
    if (err != cudaSuccess) return err;
    *hdr = h;
    *idx = ix;
    return cudaSuccess;
}

}  // namespace pb

// Depth-node form of the mixed single-slab bremsstrahlung scorer: state
// shared between its kernels (pb_brem_node.cu) and the per-(segment, energy)
// kernels that score the segments it leaves out (pb_brem.cu).
#pragma once

#include <cstdint>

#include "pb_internal.h"

namespace pb {

constexpr int kNodeMaxCells = 64;   // depth cells of the escape interpolation
constexpr int kNodePts = 8;         // Chebyshev nodes per cell (degree 7)
constexpr int kNodeTDeg = 6;        // coefficients of the electron-energy polynomial (degree 5)
constexpr int kNodePJ = kNodeTDeg * kNodePts;  // moments per (element, face, cell)
constexpr int kNodeMaxEl = 2;       // elements the shared accumulator holds
constexpr double kNodeWindow = 1.1; // T_hi / T_lo of the energy window at most
constexpr int kNodeMaxWin = 32;     // energy windows of a launch whose electrons slow down (a quarter octave each)
constexpr int kNodeBins = 256;      // sixteenths of an octave of the electron energy counted: 4 keV to 262 MeV
constexpr int kNodeQuarters = kNodeBins / 4;
constexpr int64_t kNodeWinSeg = (int64_t)1 << 22;  // longest segment list with windows (its index list: 32 MB)
constexpr double kNodeTip = 2.5;    // T_lo >= 2.5 k_max: the window stays clear of the spectrum's tip
constexpr int kNodeUniform = 5;     // cells of width h_min before the geometric growth
constexpr double kNodeGrowth = 1.2;  // deeper cells: width a fifth of their start depth

// Launch state in the caller's workspace (zeroed before each launch).
struct BremNodeHdr {
    unsigned long long t_max_bits;   // atomicMax of T over radiating segments (bits of a non-negative double)
    unsigned long long t_minc_bits;  // atomicMax of ~bits: the smallest T
    unsigned long long n_out;        // segments left to the per-(segment, energy) form
    unsigned int ok;                 // the node form scores this launch
    unsigned int faces;              // bit 0: a direction leaves through the top face, bit 1: the bottom
    int n_cells;
    int n_win;                       // windows of the launch (0: one window below the highest energy)
    double T_lo, T_hi, Tc, Th;       // electron-energy window [T_lo, T_hi], centre and half-width
    double h_min, z_g;               // uniform cell width and the depth where the growth starts
    double zb[kNodeMaxCells + 1];    // cell boundaries, depth below the exit face
    double node[kNodeMaxCells * kNodePts];
    double Lm[kNodePts * kNodePts];  // Lagrange basis of the cell nodes in monomials of t: [i][j]
    unsigned long long n_rad;        // radiating segments
    unsigned int hist[kNodeBins];    // radiating segments by sixteenth of an octave of T
    unsigned int fill[kNodeBins + 1];    // those listed so far where the bin has no window (the last: outside the bins)
    int win_of[kNodeQuarters];       // window of a quarter octave, -1: none
    double win_Tc[kNodeMaxWin], win_Th[kNodeMaxWin];  // a window's centre and half-width
    unsigned int win_n[kNodeMaxWin];     // its segments
    unsigned int win_fill[kNodeMaxWin];  // those listed so far
    unsigned int win_bad[kNodeMaxWin];   // its fit missed: the per-pair form takes its segments
};

// Sixteenth of an octave of T (> 0) counted from 4 keV: the exponent and the
// four leading bits of the fraction.
__device__ __forceinline__ int node_bin(double T) {
    return (int)((__double_as_longlong(T) >> 48) - (long long)((1023 + 2) << 4));
}
__device__ __forceinline__ double node_bin_lo(int q) {
    return __longlong_as_double((long long)(((1023 + 2) << 4) + q) << 48);
}

// Byte offsets of the workspace parts.
struct BremNodeLayout {
    size_t hdr, A, S, idx, total, zero_bytes;
    int64_t cap;  // capacity of the segment list
    int n_win;    // windows the workspace holds
};

__host__ __device__ inline BremNodeLayout brem_node_parts(const pb_brem_args &a, int64_t n_seg) {
    BremNodeLayout l;
    auto up = [](size_t x) { return (x + 255) & ~(size_t)255; };
    // With windows the list holds every segment (left out, then window by window).
    const bool win = n_seg <= kNodeWinSeg;
    l.n_win = win ? kNodeMaxWin : 1;
    l.hdr = 0;
    l.S = up(sizeof(BremNodeHdr));
    l.A = up(l.S + sizeof(double) * (size_t)l.n_win * (size_t)a.n_el * 2 * kNodeMaxCells * kNodePJ);
    l.idx = up(l.A + sizeof(double) * (size_t)l.n_win * (size_t)a.n_E * (size_t)a.n_el * kNodeTDeg);
    l.cap = win ? (n_seg > 4096 ? n_seg : 4096) : n_seg / 8 + 4096;
    l.total = l.idx + sizeof(int64_t) * (size_t)l.cap;
    l.zero_bytes = l.A;  // header and moments
    return l;
}

// A workspace sized for a list holds every shorter one: past the longest list
// with windows, whose parts alone need less, the size stays at that list's
// (38 MB for 2,048 energies and one element) until the longer list needs more.
__host__ __device__ inline BremNodeLayout brem_node_layout(const pb_brem_args &a) {
    BremNodeLayout l = brem_node_parts(a, a.n_seg);
    if (a.n_seg > kNodeWinSeg) {
        const size_t least = brem_node_parts(a, kNodeWinSeg).total;
        if (l.total < least) l.total = least;
    }
    return l;
}

// Whether the node form can take these arguments at all (the device then
// decides per launch from the segments and the directions).
__host__ __device__ inline bool brem_node_applies(const pb_brem_args &a) {
    return a.precision == PB_MIXED && a.n_layer == 0 && a.n_el >= 1 && a.n_el <= kNodeMaxEl && a.n_E >= 1;
}

// Runs the node form's kernels when the workspace is set; *hdr and *idx then
// point at the launch state and the left-out segment list the
// per-(segment, energy) kernels read, else they are null.
cudaError_t launch_brem_node(const pb_brem_args &a, cudaStream_t s, int sms, const BremNodeHdr **hdr,
                             const int64_t **idx);

}  // namespace pb

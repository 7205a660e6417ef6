// Characteristic-line yields of a segment list (sm_100a).
//
// Per segment row r and direction d, for every line j of one emitting
// element (src/pyrite/montecarlo/spectrum/characteristic.py:837-900 and the
// fused chunk kernel _characteristic_chunk_kernel.py:120-190):
//   sigma_s  = masked linear interpolation of shell s's ionisation table at
//              the row's energy (characteristic.py:760-801, numpy interp);
//   sigma_j  = sum_s sigma_s response[s][j]                (shells in order);
//   per linear escape piece p of the row (segment_escape.py:191-268):
//     tau0/1 = sum_k path_start/end[p][k] mu[k][j]         (layers in order),
//     y     += n 1e24 (L f_p 1e-8) sigma_j <exp(-tau)>(tau0, tau1);
// and line_yield[d][j] += sum over rows.
//
// Work split: a block takes one line, up to 16 directions and a share of the
// segments, one per thread in turn; sums stay in registers until the end.
// Directions of one detector (one exit face, path factors within 2 % in FP64, 1 %
// mixed) share two exponentials a piece through moments (pb_moments.cuh); others
// take two each. Only the shells that feed the line are interpolated. The first
// form kept every direction and line of a segment in one thread, each with its
// own exponentials, shell sum and warp reduction: 918 us for 200,000 segments, 7
// lines, 16 directions in a three-layer stack, 184 us now (158 with depths counted
// from the face, which light from below an absorber does not bear); bound by FP64 issue.
#include <algorithm>
#include <cstdint>
#include <type_traits>

#include "pb_common.cuh"
#include "pb_internal.h"
#include "pb_moments.cuh"

namespace pb {

constexpr int kCharThreads = 256;
constexpr int kCharMaxShell = 40;
constexpr int kCharMaxLine = 256;
constexpr int kCharMaxLayer = 8;

// numpy.interp at q on one shell table, with the scorer's in-range mask.
__device__ __forceinline__ double shell_interp(double q, const double *e, const double *v, int64_t n) {
    if (!(q >= e[0] && q <= e[n - 1])) return 0.0;
    int64_t lo = 0, hi = n - 1;  // e[lo] <= q < e[hi] (or q == e[n-1])
    if (q == e[n - 1]) return v[n - 1];
    while (hi - lo > 1) {
        const int64_t m = (lo + hi) >> 1;
        if (e[m] <= q) lo = m; else hi = m;
    }
    const double slope = (v[hi] - v[lo]) / (e[hi] - e[lo]);
    return slope * (q - e[lo]) + v[lo];
}

// Segment mean of exp(-tau) for tau linear between t0 and t1
// (segment_escape.py:291-303): exp(-min) (1 - exp(-d))/d, series below 1e-4.
template <bool kMixed>
__device__ __forceinline__ double mean_transmission_d(double t0, double t1) {
    const double lo = fmin(t0, t1);
    const double d = fabs(t1 - t0);
    if constexpr (kMixed) {
        const float df = (float)d;
        const float ratio = d > 1.0e-4 ? -expm1f(-df) / df : (1.0f - 0.5f * df) + (df * df) * (1.0f / 6.0f);
        return (double)(__expf(-(float)lo) * ratio);
    } else {
        const double ratio = d > 1.0e-4 ? -expm1(-d) / d : (1.0 - 0.5 * d) + (d * d) / 6.0;
        return exp(-lo) * ratio;
    }
}

// Extent of layer k between depth z and the exit face (segment_escape.py:33-76
// for the laterally infinite slab / layer stack, before the factor 1 / |n_z|).
__device__ __forceinline__ double extent(double z, bool up, double z_top, double z_bot) {
    return up ? fmax(fmin(z, z_bot) - z_top, 0.0) : fmax(z_bot - fmax(z, z_top), 0.0);
}

constexpr int kCharDirs = 16;  // directions a block scores

template <bool kMixed>
__global__ void __launch_bounds__(kCharThreads, 2) char_yield_kernel(const pb_char_args a) {
    using Real = typename std::conditional<kMixed, float, double>::type;
    constexpr int kOrder = kMixed ? 3 : 9;
    __shared__ double z_top[kCharMaxLayer], z_bot[kCharMaxLayer], mu[kCharMaxLayer];
    __shared__ double inv_nz[kCharDirs];
    __shared__ bool up[kCharDirs];
    __shared__ double red[kCharThreads / 32];
    int64_t n_seg = a.n_seg;
    if (a.n_seg_device && (int64_t)*a.n_seg_device < n_seg) n_seg = (int64_t)*a.n_seg_device;
    const int n_line = a.n_line, n_shell = a.n_shell;
    const int n_k = a.n_layer > 0 ? a.n_layer : 1;
    const int line = blockIdx.y % n_line, d0 = (blockIdx.y / n_line) * kCharDirs;
    const int nd = min(a.n_dir - d0, kCharDirs);
    const int tid = threadIdx.x, lane = tid & 31;
    if (tid < n_k) {
        // the single slab: one layer, paths clipped to its faces
        z_top[tid] = a.n_layer > 0 ? a.z_top[tid] : 0.0;
        z_bot[tid] = a.n_layer > 0 ? a.z_bot[tid] : a.thickness;
        mu[tid] = a.mu[(int64_t)tid * n_line + line];
    }
    if (tid < nd) {
        const double nz = a.n_hat[3 * (d0 + tid) + 2];
        inv_nz[tid] = 1.0 / fmax(fabs(nz), 1.0e-12);
        up[tid] = nz < 0.0;
    }
    __syncthreads();
    double f_c, dl;
    const bool moments = one_face(a.n_hat, d0, nd, moment_limit<Real>(), f_c, dl);
    // Moments 0 .. kOrder, or one sum per direction.
    double acc[kCharDirs];
#pragma unroll
    for (int i = 0; i < kCharDirs; ++i) acc[i] = 0.0;
    // Optical depth below the exit face that the moments count from, the whole
    // absorber's at first.
    double ref = 0.0;
    for (int k = 0; k < n_k; ++k) ref += mu[k] * (z_bot[k] - z_top[k]);
    const double above = -(double)moment_above<Real>() / f_c;
    const auto rebase = [&](double to) {
        if (acc[0] == 0.0) {  // nothing summed yet
            ref = to;
            return;
        }
        const double c = -(ref - to) * dl, sc = exp(-(ref - to) * f_c);
#pragma unroll
        for (int n = kOrder; n >= 0; --n) {
            double v = acc[n], t = 1.0;
#pragma unroll
            for (int j = n - 1; j >= 0; --j) {
                t *= c * ((double)(j + 1) / (double)(n - j));
                v = fma(t, acc[j], v);
            }
            acc[n] = sc * v;
        }
        ref = to;
    };

    for (int64_t s = (int64_t)blockIdx.x * blockDim.x + tid; s < n_seg; s += (int64_t)gridDim.x * blockDim.x) {
        if (!(a.elec_id[s] < a.Ne && (a.seg_layer == nullptr || a.seg_layer[s] == a.emit_layer))) continue;
        const double q = a.E_keV[s] * 1.0e3;
        double sj = 0.0;
        for (int sh = 0; sh < n_shell; ++sh) {
            const double resp = a.response[(int64_t)sh * n_line + line];
            if (resp == 0.0) continue;
            const int64_t o = a.shell_offset[sh];
            sj = sj + shell_interp(q, a.shell_E + o, a.shell_sigma + o, a.shell_offset[sh + 1] - o) * resp;
        }
        if (sj == 0.0) continue;
        const double L = a.L[s], vz = a.v_hat[3 * s + 2], zm = a.r_mid[3 * s + 2];
        const double r0z = zm - 0.5 * L * vz, dz = (zm + 0.5 * L * vz) - r0z;
        const double w = a.n_atoms * 1.0e24 * (L * 1.0e-8) * sj;
        // Pieces: cut fractions at the interior layer boundaries, sorted.
        double cuts[kCharMaxLayer + 1];
        int n_cut = 0;
        cuts[n_cut++] = 0.0;
        cuts[n_cut++] = 1.0;
        for (int k = 1; k < a.n_layer; ++k) {
            const double st = r0z - z_top[k], en = r0z + dz - z_top[k];
            const double den = st - en;
            const double f = st / (den == 0.0 ? 1.0 : den);
            if (!(f > 0.0 && f < 1.0)) continue;  // a cut at 1 bounds no piece
            int j = n_cut++;
            for (; j > 0 && cuts[j - 1] > f; --j) cuts[j] = cuts[j - 1];
            cuts[j] = f;
        }
        for (int c = 0; c + 1 < n_cut; ++c) {
            const double frac = cuts[c + 1] - cuts[c];
            if (!(frac > 1.0e-12)) continue;
            // Depths along the face normal at the piece's ends. Layers: sampled at
            // 1/4 and 3/4 and extrapolated (segment_escape.py:256-268).
            const double za = r0z + (cuts[c] + 0.25 * frac) * dz, zb = r0z + (cuts[c] + 0.75 * frac) * dz;
            const auto depths = [&](bool face_up, double &t0, double &t1) {
                t0 = t1 = 0.0;
                for (int k = 0; k < n_k; ++k) {
                    double p0, p1;
                    if (a.n_layer == 0) {
                        const double e0 = fmin(fmax(r0z, 0.0), z_bot[0]), e1 = fmin(fmax(r0z + dz, 0.0), z_bot[0]);
                        p0 = face_up ? e0 : z_bot[0] - e0;
                        p1 = face_up ? e1 : z_bot[0] - e1;
                    } else {
                        const double q1 = extent(za, face_up, z_top[k], z_bot[k]);
                        const double q3 = extent(zb, face_up, z_top[k], z_bot[k]);
                        p0 = fmax(1.5 * q1 - 0.5 * q3, 0.0);
                        p1 = fmax(1.5 * q3 - 0.5 * q1, 0.0);
                    }
                    t0 = t0 + p0 * mu[k];
                    t1 = t1 + p1 * mu[k];
                }
            };
            const double wp = a.n_layer == 0 ? w : w * frac;
            double t0, t1;
            if (moments) {
                depths(up[0], t0, t1);
                const double lo = fmin(t0, t1);
                if (lo - ref < above) rebase(lo);
                Real Q[kOrder + 1] = {};
                add_moments<kOrder>((Real)1, (Real)(lo - ref), (Real)fabs(t1 - t0), (Real)f_c,
                                    (Real)(f_c * 1.4426950408889634), (Real)dl, Q);
#pragma unroll
                for (int n = 0; n <= kOrder; ++n) acc[n] = fma(wp, (double)Q[n], acc[n]);
            } else {
                double u0, u1;
                depths(false, t0, t1);
                depths(true, u0, u1);
#pragma unroll
                for (int d = 0; d < kCharDirs; ++d)
                    if (d < nd)
                        acc[d] += wp * mean_transmission_d<kMixed>((up[d] ? u0 : t0) * inv_nz[d],
                                                                   (up[d] ? u1 : t1) * inv_nz[d]);
            }
        }
    }
    if (moments) {  // one reference for the block: its nearest
        double r = ref;
        for (int o = 16; o > 0; o >>= 1) r = fmin(r, __shfl_xor_sync(0xffffffffu, r, o));
        if (lane == 0) red[tid >> 5] = r;
        __syncthreads();
        for (int k = 0; k < kCharThreads / 32; ++k) r = fmin(r, red[k]);
        if (r < ref) rebase(r);
        __syncthreads();
    }
    // Block sums in thread order, one global add per direction.
    double sum[kCharDirs];
#pragma unroll
    for (int i = 0; i < kCharDirs; ++i) {
        double v = acc[i];
        for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
        __syncthreads();
        if (lane == 0) red[tid >> 5] = v;
        __syncthreads();
        v = red[0];
        for (int k = 1; k < kCharThreads / 32; ++k) v += red[k];
        sum[i] = v;
    }
    if (tid == 0) {
#pragma unroll
        for (int d = 0; d < kCharDirs; ++d) {
            if (d >= nd) break;
            double v = sum[d];
            if (moments) {
                const double f = inv_nz[d], h = dl > 0.0 ? (f - f_c) / dl : 0.0;
                v = sum[kOrder];
#pragma unroll
                for (int n = kOrder; n > 0; --n) v = fma(v, h / (double)n, sum[n - 1]);
                v *= exp(-ref * f) / f;
            }
            if (v != 0.0) atomicAdd(&a.line_yield[(int64_t)(d0 + d) * n_line + line], v);
        }
    }
}

__global__ void char_spectrum_kernel(int n_line, int n_E, const double *yield, const double *profiles,
                                     double *spec) {
    const int d = blockIdx.y;
    const int b = blockIdx.x * blockDim.x + threadIdx.x;
    if (b >= n_E) return;
    double acc = 0.0;
    for (int j = 0; j < n_line; ++j) acc += yield[(int64_t)d * n_line + j] * profiles[(int64_t)j * n_E + b];
    spec[(int64_t)d * n_E + b] += acc;
}

cudaError_t launch_char(const pb_char_args &a, cudaStream_t s, int sms) {
    if (a.n_shell > kCharMaxShell || a.n_line > kCharMaxLine || a.n_layer > kCharMaxLayer)
        return cudaErrorInvalidValue;
    const int64_t n_seg = a.n_seg;  // capacity; the kernel reads n_seg_device itself
    if (n_seg <= 0) return cudaSuccess;
    // (the limit of the interface, from a per-block yield table)
    if (sizeof(double) * (size_t)a.n_dir * a.n_line > 200 * 1024) return cudaErrorInvalidValue;
    auto kern = a.precision == PB_MIXED ? char_yield_kernel<true> : char_yield_kernel<false>;
    // About eight blocks an SM over (line, direction group), at most one segment
    // per thread.
    const int64_t rows = (int64_t)a.n_line * ((a.n_dir + kCharDirs - 1) / kCharDirs);
    int64_t gx = std::max<int64_t>(1, (int64_t)sms * 8 / rows);
    gx = std::min(gx, (n_seg + kCharThreads - 1) / kCharThreads);
    if (rows > 65535) return cudaErrorInvalidValue;
    kern<<<dim3((unsigned)gx, (unsigned)rows), kCharThreads, 0, s>>>(a);
    return cudaGetLastError();
}

cudaError_t launch_char_spectrum(int n_dir, int n_line, int n_E, const double *yield, const double *profiles,
                                 double *spec, cudaStream_t s) {
    dim3 grid((unsigned)((n_E + 127) / 128), (unsigned)n_dir);
    char_spectrum_kernel<<<grid, 128, 0, s>>>(n_line, n_E, yield, profiles, spec);
    return cudaGetLastError();
}

}  // namespace pb

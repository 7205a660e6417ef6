// Direction moments of the segment-mean escape.
//
// A piece of a segment escapes towards a direction with path factor f = 1/|n_z|
// with the mean of exp(-(a + b u) f) over u in [0, 1]: a the optical depth of the
// end nearer the exit face, b the depth difference of the ends, both along the
// face normal. g(f) = (exp(-a f) - exp(-(a + b) f)) / b, its Taylor coefficients
// about a centre f_c follow without cancellation and do not depend on the
// direction, so the directions of one detector share two exponentials.
#pragma once

#include "pb_common.cuh"

namespace pb {

// Base-2 exponential on the SFU (about 2 ulp), for the float path.
__device__ __forceinline__ float ex2_approx(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// Reciprocal on the SFU (about 1 ulp), for the float path.
__device__ __forceinline__ float rcp_approx(float x) {
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// Whether the directions d0 .. d0 + nd - 1 leave through one face with path
// factors 1 / |n_z| in f_c +- dl, dl <= limit f_min. Kernels that share a launch
// make the same test, so exactly one of them scores it.
__device__ __forceinline__ bool one_face(const double *n_hat, int d0, int nd, double limit, double &f_c, double &dl) {
    int n_up = 0;
    double f_lo = 1e300, f_hi = 0.0;
    for (int dd = 0; dd < nd; ++dd) {
        const double nz = n_hat[3 * (d0 + dd) + 2];
        n_up += nz < 0.0 ? 1 : 0;
        const double f = 1.0 / fmax(fabs(nz), 1.0e-12);
        f_lo = fmin(f_lo, f);
        f_hi = fmax(f_hi, f);
    }
    f_c = 0.5 * (f_lo + f_hi);
    dl = 0.5 * (f_hi - f_lo);
    return (n_up == nd || n_up == 0) && dl <= limit * f_lo;
}

// The directions d0 .. d0 + nd - 1 (nd <= 32) as at most kMaxGroups groups of one
// face and path factors in f_c +- dl, dl <= limit f_min, by one warp: each group
// is the first direction left and those within 0.98 limit of its path factor.
// ``of`` gets each direction's group; returns kMaxGroups + 1 where more are needed.
constexpr int kMaxGroups = 4;
struct DirGroups {
    double f_c[kMaxGroups], dl[kMaxGroups];
    int up[kMaxGroups], of[32];
    int n;
};
__device__ __forceinline__ void direction_groups(const double *n_hat, int d0, int nd, double limit, DirGroups &g) {
    const int lane = threadIdx.x & 31;
    const double nz = lane < nd ? n_hat[3 * (d0 + lane) + 2] : 0.0;
    const double f = 1.0 / fmax(fabs(nz), 1.0e-12);
    const int up = nz < 0.0 ? 1 : 0;
    unsigned left = __ballot_sync(0xffffffffu, lane < nd);
    int n = 0;
    while (left && n < kMaxGroups) {
        const int lead = __ffs(left) - 1;
        const double f0 = __shfl_sync(0xffffffffu, f, lead);
        const int up0 = __shfl_sync(0xffffffffu, up, lead);
        const bool in = ((left >> lane) & 1u) && up == up0 && fabs(f - f0) <= 0.98 * limit * fmin(f, f0);
        double lo = in ? f : f0, hi = lo;
        for (int o = 16; o > 0; o >>= 1) {
            lo = fmin(lo, __shfl_xor_sync(0xffffffffu, lo, o));
            hi = fmax(hi, __shfl_xor_sync(0xffffffffu, hi, o));
        }
        if (in) g.of[lane] = n;
        if (lane == lead) {
            g.f_c[n] = 0.5 * (lo + hi);
            g.dl[n] = 0.5 * (hi - lo);
            g.up[n] = up;
        }
        left &= ~(__ballot_sync(0xffffffffu, in) | (1u << lead));
        ++n;
    }
    if (lane == 0) g.n = left ? kMaxGroups + 1 : n;
}

// Direction moments of the segment-mean escape, for the FP64 bremsstrahlung, the
// layered absorber and the characteristic lines (the mixed single-slab kernels
// carry packed forms of the same recurrence). The truncation after order N is below
// rho^(N+1) / sqrt(2 pi (N+1)) of the term without attenuation: FP64 takes N = 5 for
// rho <= 0.002 and N = 9 for rho <= 0.02 (both below 2e-17), the mixed layered
// path N = 3 for rho <= 0.01 (2e-9). Where all light comes from below an absorber
// that would be much of what is left of it, so depths count from a reference near
// the shallowest piece (moved by rebase_moments when a piece lies more than
// kAbove / f_c above it) and each direction is attenuated to there by an
// exponential of its own. A piece kAbove / f_c above the reference is off by
// (kAbove rho)^(N+1) / (N+1)! of itself: FP64 2e-16, mixed 7e-9.
template <class Real>
constexpr double moment_limit() { return sizeof(Real) == 8 ? 0.02 : 0.01; }
template <class Real>
constexpr Real moment_above() { return sizeof(Real) == 8 ? (Real)6 : (Real)2; }

// The moments Q(0) .. Q(N) of depths from a reference ``delta`` (optical depth per
// unit path factor) nearer the exit face: the sums times exp(-delta f), a factor
// exp(-delta f_c) and a binomial convolution with the powers of -delta dl.
template <class F>
__device__ __forceinline__ void rebase_moments(int N, double delta, double f_c, double dl, F Q) {
    if (Q(0) == 0.0) return;  // nothing summed yet
    const double c = -delta * dl, s = exp(-delta * f_c);
#pragma unroll 1
    for (int n = N; n >= 0; --n) {
        double v = Q(n), t = 1.0;
#pragma unroll 1
        for (int j = n - 1; j >= 0; --j) {
            t *= c * (double)(j + 1) / (double)(n - j);
            v = fma(t, Q(j), v);
        }
        Q(n) = s * v;
    }
}

// Q_n += w P_n of one affine piece: a = optical depth of its shallower end along
// the face normal, b = the depth difference of its ends, both per unit path
// factor. Two exponentials serve every direction of the group, where each
// direction took two of its own.
template <int N>
__device__ __forceinline__ void add_moments(double w, double a, double b, double f_c, double, double dl,
                                            double (&Q)[N + 1]) {
    const double x = b * f_c;
    const double Ea = exp(-a * f_c), em = -expm1(-x);
    double P = w * Ea * f_c * (x > 1.0e-5 ? em / x : 1.0 - 0.5 * x + x * x / 6.0);
    Q[0] += P;
    if constexpr (N > 0) {
        const double ah = -dl * a, ch = -dl * (a + b);
        double R = w * dl * (Ea - Ea * em);
#pragma unroll
        for (int n = 1; n <= N; ++n) {
            P = fma(ah, P, R);
            R *= ch;
            Q[n] += P;
        }
    }
}
// In float the exponentials are the SFU's, of products with c2 = f_c log2(e) rounded
// once (the rounding of an optical depth dominates their own 2 ulp), and 1 - e^-x is a series to x = 1,
// where the difference has lost less than one bit: phi(x) = (1 - e^-x) / x =
// phi(h) (1 - h phi(h) / 2), h = x / 2, phi(h) to h^8 (truncation 3e-10).
template <int N>
__device__ __forceinline__ void add_moments(float w, float a, float b, float f_c, float c2, float dl,
                                            float (&Q)[N + 1]) {
    const float x = b * f_c;
    const float Ea = ex2_approx(-(a * c2));
    float em, phi;
    if (x > 1.0f) {
        em = 1.0f - ex2_approx(-(b * c2));
        phi = em * rcp_approx(x);
    } else {
        const float h = 0.5f * x;
        float p = fmaf(h, 1.0f / 362880.0f, -1.0f / 40320.0f);
        p = fmaf(h, p, 1.0f / 5040.0f);
        p = fmaf(h, p, -1.0f / 720.0f);
        p = fmaf(h, p, 1.0f / 120.0f);
        p = fmaf(h, p, -1.0f / 24.0f);
        p = fmaf(h, p, 1.0f / 6.0f);
        p = fmaf(h, p, -0.5f);
        p = fmaf(h, p, 1.0f);
        phi = fmaf(-0.5f * h * p, p, p);
        em = x * phi;
    }
    const float Ec = Ea - Ea * em;
    float P = w * Ea * (f_c * phi);
    Q[0] += P;
    if constexpr (N > 0) {
        const float ah = -dl * a, ch = -dl * (a + b);
        float R = w * dl * Ec;
#pragma unroll
        for (int n = 1; n <= N; ++n) {
            P = fmaf(ah, P, R);
            R *= ch;
            Q[n] += P;
        }
    }
}

// (1 / f) sum_n ((f - f_c) / dl)^n Q_n / n! from the summed moments Q(n).
template <class F>
__device__ __forceinline__ double moments_at(int N, double f, double f_c, double dl, F Q) {
    const double h = dl > 0.0 ? (f - f_c) / dl : 0.0;
    double v = Q(N);
    for (int n = N; n > 0; --n) v = fma(v, h / (double)n, Q(n - 1));
    return v / f;
}

}  // namespace pb

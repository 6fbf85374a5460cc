// Shared by the routes that use the permutational symmetries of the RDMs and
// integrals (bamat_sym.cu, koop_sym.cu): pair indices and the device-side checks
// that decide, for each state, whether its inputs have those symmetries.
#pragma once
#include "nvpt2_internal.h"

namespace nvpt {

// Elements that a symmetry makes equal may differ by this share of the largest
// |Gamma1| (RDMs) or |(ii|ii)| (integrals): above the rounding of an RDM builder
// or an integral transformation, far below anything else.
constexpr double kSymTol = 0x1p-45;

__host__ __device__ __forceinline__ int pidx(int i, int j) { return i * (i + 1) / 2 + j; }  // i >= j
__device__ __forceinline__ int pmx(int i, int j) { return i > j ? pidx(i, j) : pidx(j, i); }
__device__ __forceinline__ void unpair(int p, int &i, int &j) {  // p = pidx(i, j)
    i = (int)((sqrtf(8.0f * p + 1.0f) - 1.0f) * 0.5f);
    if (pidx(i + 1, 0) <= p) ++i;
    if (pidx(i, 0) > p) --i;
    j = p - pidx(i, 0);
}

// Scales are compared by their leading 32 bits: comparisons of doubles run on the FP64
// pipe (16 clocks a warp), and every block takes its own scale.
__device__ __forceinline__ unsigned abs_hi(double x) { return (unsigned)__double2hiint(x) & 0x7fffffffu; }

// Tolerance of the RDM checks of state s (0-based): all threads of the block.  raised:
// whether the state's flag was raised already.
__device__ __forceinline__ double rdm_tolerance(const Rdm &r, int s, const int *flag, bool &raised) {
    const bool seen = threadIdx.x == 0 && *(volatile const int *)(flag + s) != 0;
    __shared__ unsigned red[8];
    unsigned m = 0;
    for (int i = threadIdx.x; i < r.n * r.n; i += blockDim.x) m = max(m, abs_hi(r.d1[s + (ll)r.M * i]));
    m = __reduce_max_sync(0xffffffffu, m);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = m;
    raised = __syncthreads_or(seen);
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) m = max(m, red[w]);
    return kSymTol * __hiloint2double((int)m, 0);
}
__device__ __forceinline__ bool sym_differ(double x, double y, double tol) { return !(fabs(x - y) <= tol); }

// Element t < n^6 of Gamma3 (and t < n^4, n^2 of Gamma2, Gamma1) against its images.
__device__ __forceinline__ bool rdm_asymmetric(const Rdm &r, int s, ll t, double tol) {
    const int n = r.n, M = r.M;
    ll x = t;
    int q[6];
    for (int i = 0; i < 6; ++i) { q[i] = (int)(x % n); x /= n; }
    auto d3 = [&](int a, int b, int c, int d, int e, int f) {
        return r.d3[s + (ll)M * (a + n * (b + n * (c + (ll)n * (d + n * (e + (ll)n * f)))))];
    };
    // an image is compared by the larger of the two elements
    auto key6 = [n](int a, int b, int c, int d, int e, int f) {
        return a + n * (b + n * (c + n * (d + n * (e + n * f))));
    };
    const double v = r.d3[s + (ll)M * t];
    bool bad = (t > key6(q[1], q[0], q[2], q[4], q[3], q[5]) && sym_differ(v, d3(q[1], q[0], q[2], q[4], q[3], q[5]), tol)) ||
               (t > key6(q[0], q[2], q[1], q[3], q[5], q[4]) && sym_differ(v, d3(q[0], q[2], q[1], q[3], q[5], q[4]), tol)) ||
               (t >= key6(q[3], q[4], q[5], q[0], q[1], q[2]) && sym_differ(v, d3(q[3], q[4], q[5], q[0], q[1], q[2]), tol));
    if (t < (ll)n * n * n * n) {
        auto d2 = [&](int a, int b, int c, int d) { return r.d2[s + (ll)M * (a + n * (b + n * (c + (ll)n * d)))]; };
        const double w = r.d2[s + (ll)M * t];
        bad = bad || sym_differ(w, d2(q[1], q[0], q[3], q[2]), tol) || sym_differ(w, d2(q[2], q[3], q[0], q[1]), tol);
    }
    if (t < (ll)n * n) bad = bad || sym_differ(r.d1[s + (ll)M * t], r.d1[s + (ll)M * (q[1] + n * q[0])], tol);
    return bad;
}

// Element (i,j,k,l) of the integrals against its images.
__device__ __forceinline__ bool integral_asymmetric(const double *atwo, int n, int i, int j, int k, int l) {
    auto at = [&](int a, int b, int c, int d) { return atwo[a + n * (b + n * (c + (ll)n * d))]; };
    unsigned scale = 0;
    for (int q = 0; q < n; ++q) scale = max(scale, abs_hi(at(q, q, q, q)));
    const double v = at(i, j, k, l), tol = kSymTol * __hiloint2double((int)scale, 0);
    return sym_differ(v, at(j, i, k, l), tol) || sym_differ(v, at(k, l, i, j), tol);
}

}  // namespace nvpt

// The PC pencils of small order in tridiagonal form, K~ = Q T Q^T, and the labels'
// resolvents (T + sigma)^-1, one label a thread.
//
// These classes have few functions (orders of 10 to 512) and up to thousands of
// labels.  An elimination on a band of half width 32 costs 2048 FMAs a row and label,
// one on the tridiagonal form 10, and what the reduction costs is latency: the matrix
// stays in the shared memory of a few CTAs, and a column is one exchange between them.
#include <algorithm>

#include "../../include/nvpt2.h"
#include "band.cuh"
#include "grid_bar.cuh"

namespace nvpt {
namespace s2 {
namespace {

constexpr int TB = 256;
constexpr int NB = kBand;  // reflectors of a panel of Q

struct TriArgs {
    const double *A;  // n x n, both triangles
    int n;
    double *d, *e, *tau, *V;   // V: panels as in wy_apply with first = 1
    unsigned long long *msg;   // [n][2][n], all kNoMsg on entry
    int *err;                  // 0 once a wait gave up
    unsigned spin;
};

__device__ __forceinline__ long long panel_at(long long n, int p) {  // first element of panel p of V
    return ((long long)p * (n - 1) - (long long)NB * p * (p - 1) / 2) * NB;
}

// Householder tridiagonalisation.  Row i lives in CTA i mod G.  With v, w of the last
// column, one pass over a CTA's rows applies A -= v w^T + w v^T and takes the products
// A v' with the next reflector; the CTA publishes them and the next column's entries
// before that column's own update, which every CTA applies for itself.  So a column
// is one exchange (a stored word that is not kNoMsg has arrived) where the two-barrier
// form needs two and a counter each: 5 us a column at orders 100 to 220, 16 before.
__global__ void __launch_bounds__(TB, 1) k_tri_reduce(TriArgs a) {
    extern __shared__ double sm[];
    const int n = a.n, G = gridDim.x, b = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    double *x = sm, *v = x + n, *vo = v + n, *w = vo + n, *p = w + n, *As = p + n;  // As [rows][n]
    __shared__ double red[TB], s_scal, s_tau, s_half;
    for (int i = b; i < n; i += G)
        for (int k = tid; k < n; k += TB) As[(i / G) * n + k] = a.A[(long long)i * n + k];
    for (int k = tid; k < n; k += TB) {
        x[k] = a.A[k];
        vo[k] = w[k] = 0.0;
    }
    for (int i = b; i < n; i += G)  // own rows of V: zero where no reflector reaches
        for (int p = warp; p * NB + 1 <= i && p * NB + 2 < n; p += TB / 32)
            a.V[panel_at(n, p) + (long long)(i - p * NB - 1) * NB + lane] = 0.0;
    __syncthreads();
    // sum over the block, in warp 0
    auto total = [&](double s) {
        red[tid] = s;
        __syncthreads();
        double t = 0.0;
        if (warp == 0) {
#pragma unroll
            for (int q = 0; q < TB / 32; ++q) t += red[lane + 32 * q];
            for (int o = 16; o; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
        }
        return t;
    };
    for (int j = 0; j + 2 < n; ++j) {
        double s = 0.0;
        for (int i = j + 2 + tid; i < n; i += TB) s = fma(x[i], x[i], s);
        s = total(s);
        if (warp == 0) {
            const double alpha = x[j + 1];
            double tau = 0.0, beta = alpha, scal = 0.0;
            if (s != 0.0) {
                beta = -copysign(sqrt(fma(alpha, alpha, s)), alpha);
                tau = (beta - alpha) / beta;
                scal = 1.0 / (alpha - beta);
            }
            if (lane == 0) {
                s_tau = tau;
                s_scal = scal;
                if (b == 0) {
                    a.d[j] = x[j];
                    a.e[j] = beta;
                    a.tau[j] = tau;
                }
            }
        }
        __syncthreads();
        const double scal = s_scal, tau = s_tau;
        for (int i = j + 1 + tid; i < n; i += TB) v[i] = i == j + 1 ? 1.0 : scal * x[i];
        __syncthreads();
        unsigned long long *msg = a.msg + (long long)j * 2 * n;
        double *V = a.V + panel_at(n, j / NB) + j % NB;
        const int s0 = (j / NB) * NB + 1;
        for (int i = b + ((j + 1 - b + G - 1) / G) * G + warp * G; i < n; i += G * (TB / 32)) {
            double *row = As + (i / G) * n, t = 0.0;
            const double vi = vo[i], wi = w[i];
            for (int k = j + 1 + lane; k < n; k += 32) {
                const double r = fma(-wi, vo[k], fma(-vi, w[k], row[k]));
                row[k] = r;
                t = fma(r, v[k], t);
            }
            for (int o = 16; o; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
            if (lane == 0) {
                send_word(msg + i, t);
                send_word(msg + n + i, row[j + 1]);
                V[(long long)(i - s0) * NB] = v[i];
            }
        }
        unsigned long long m0[2] = {0, 0}, m1[2] = {0, 0};
        int ok = 1;
        for (unsigned spins = 0;;) {
            bool all = true;
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                const int i = j + 1 + tid + q * TB;
                if (i < n) {
                    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(m0[q]) : "l"(msg + i) : "memory");
                    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(m1[q]) : "l"(msg + n + i) : "memory");
                }
            }
#pragma unroll
            for (int q = 0; q < 2; ++q) all = all && m0[q] != kNoMsg && m1[q] != kNoMsg;
            if (all) break;
            if (++spins > a.spin || (spins % 64 == 0 && !*(volatile int *)a.err)) {
                atomicExch(a.err, 0);
                ok = 0;
                break;
            }
        }
        s = 0.0;
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            const int i = j + 1 + tid + q * TB;
            if (i < n) {
                p[i] = __longlong_as_double(m0[q]);
                x[i] = __longlong_as_double(m1[q]);
                s = fma(p[i], v[i], s);
            }
        }
        if (!__syncthreads_and(ok)) return;
        s = total(s);
        if (tid == 0) s_half = 0.5 * tau * tau * s;
        __syncthreads();
        const double half = s_half, w1 = tau * p[j + 1] - half;  // v[j + 1] = 1
        for (int i = j + 1 + tid; i < n; i += TB) {
            const double vi = v[i], wi = tau * p[i] - half * vi;
            vo[i] = vi;
            w[i] = wi;
            x[i] = x[i] - vi * w1 - wi;
        }
        __syncthreads();
    }
    if (b == 0 && tid == 0) {
        a.d[n - 1 > 1 ? n - 2 : 0] = x[n - 1 > 1 ? n - 2 : 0];
        if (n > 1) a.e[n - 2] = x[n - 1];
    }
    if (n > 1 && b == (n - 1) % G && tid == 0)
        a.d[n - 1] = As[((n - 1) / G) * n + n - 1] - (n > 2 ? 2.0 * vo[n - 1] * w[n - 1] : 0.0);
}

// T of each panel of Q (compact WY): the Gram matrix of its reflectors, then the recurrence.
__global__ void __launch_bounds__(TB) k_tri_wy(int n, const double *__restrict__ Vall, const double *__restrict__ tau,
                                               double *Tm) {
    __shared__ double vs[32][NB + 1], g[NB][NB + 1];
    const int p = blockIdx.x, tid = threadIdx.x, m = n - (p * NB + 1), r = tid >> 3, c0 = (tid & 7) * 4;
    const double *V = Vall + panel_at(n, p);
    double acc[4] = {};
    for (int i0 = 0; i0 < m; i0 += 32) {
        for (int e = tid; e < 32 * NB; e += TB) vs[e / NB][e % NB] = i0 + e / NB < m ? V[(long long)i0 * NB + e] : 0.0;
        __syncthreads();
#pragma unroll 8
        for (int i = 0; i < 32; ++i)
#pragma unroll
            for (int q = 0; q < 4; ++q) acc[q] = fma(vs[i][r], vs[i][c0 + q], acc[q]);
        __syncthreads();
    }
#pragma unroll
    for (int q = 0; q < 4; ++q) g[r][c0 + q] = acc[q];
    __syncthreads();
    if (tid >= 32) return;
    double t[NB];
#pragma unroll
    for (int c = 0; c < NB; ++c) {
        const double tc = p * NB + c + 2 < n ? tau[p * NB + c] : 0.0;
        double x = 0.0;
#pragma unroll
        for (int l = 0; l < c; ++l) x = fma(l >= tid ? t[l] : 0.0, g[l][c], x);
        t[c] = tid < c ? -tc * x : tid == c ? tc : 0.0;
        Tm[((long long)p * NB + tid) * NB + c] = t[c];
    }
}

__device__ __forceinline__ void warp_add(double v, double *dst) {
    for (int o = 16; o; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    if ((threadIdx.x & 31) == 0) atomicAdd(dst, v);
}

// A label a thread: elimination with partial pivoting down the rows, the factors of the
// group's labels side by side in memory (fac [3][n][group]), then the back substitution,
// with the sums taken on the way up.  One division a row; outputs as band_resolvent's.
__global__ void __launch_bounds__(64) k_tri_solve(const double *__restrict__ d, const double *__restrict__ e, int n,
                                                  const double *__restrict__ Y, long long ncol, long long L,
                                                  long long l0, int group, int nother, const double *__restrict__ sig,
                                                  double *__restrict__ fac, double *__restrict__ ys, double *acc,
                                                  double *__restrict__ xout) {
    __shared__ double sd[512], se[512];
    for (int i = threadIdx.x; i < n; i += 64) {
        sd[i] = d[i];
        se[i] = i + 1 < n ? e[i] : 0.0;
    }
    __syncthreads();
    const int g = blockIdx.x * 64 + threadIdx.x;
    const long long l = l0 + g;
    const bool live = g < group;
    double en = 0.0, ps = 0.0, offs[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    if (live) {
        const double s = sig[l];
        const long long plane = (long long)n * group;
        double *fi = fac + g, *fc = fi + plane, *fd = fc + plane, *fy = ys + g;
        double b = sd[0] + s, cc = se[0], y = Y[l];
#pragma unroll 8
        for (int i = 0; i < n - 1; ++i) {
            const double a1 = se[i], b1 = sd[i + 1] + s, c1 = se[i + 1], y1 = Y[(i + 1) * ncol + l];
            const bool keep = fabs(b) >= fabs(a1);
            const double inv = 1.0 / (keep ? b : a1), f = (keep ? a1 : b) * inv;
            const double u1 = keep ? cc : b1, u2 = keep ? 0.0 : c1, uy = keep ? y : y1;
            fi[(long long)i * group] = inv;
            fc[(long long)i * group] = u1;
            fd[(long long)i * group] = u2;
            fy[(long long)i * group] = uy;
            b = (keep ? b1 : cc) - f * u1;
            cc = (keep ? c1 : 0.0) - f * u2;
            y = (keep ? y1 : y) - f * uy;
        }
        double x1 = y / b, x2 = 0.0;
        auto sums = [&](int i, double x) {
            if (xout) xout[(long long)i * L + l] = x;
            en -= Y[i * ncol + l] * x;
            ps += x * x;
            for (int k = 0; k < nother && k < 8; ++k) offs[k] -= Y[i * ncol + (k + 1) * L + l] * x;
        };
        sums(n - 1, x1);
#pragma unroll 4
        for (int i = n - 2; i >= 0; --i) {
            const double x = (fy[(long long)i * group] - fc[(long long)i * group] * x1 - fd[(long long)i * group] * x2) *
                             fi[(long long)i * group];
            sums(i, x);
            x2 = x1;
            x1 = x;
        }
    }
    warp_add(en, acc);
    warp_add(ps, acc + 1);
    for (int k = 0; k < nother && k < 8; ++k) warp_add(offs[k], acc + 2 + k);
}

// rho[l nd + k] -= Y[:, dcol0 + k] . x_l
__global__ void k_tri_rho(const double *__restrict__ Y, long long ncol, long long dcol0, const double *__restrict__ X,
                          int n, long long L, int nd, double *rho) {
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= L * nd) return;
    const long long l = t % L;
    const int k = (int)(t / L);
    double v = 0.0;
    for (int i = 0; i < n; ++i) v = fma(Y[i * ncol + dcol0 + k], X[(long long)i * L + l], v);
    rho[l * nd + k] -= v;
}

}  // namespace

int tri_reduce(Ctx &c, const double *A, long long n, double *d, double *e, double *V, double *Tm) {
    if (n > kTriMost) throw Error(NVPT_EINVAL, "tridiagonal form: order too large");
    const int np = wy_panels(n, 1), ni = (int)n;
    // eight rows a CTA and more: the exchange's cost grows with the CTAs, the pass's falls
    const int G = (int)std::max<long long>(1, std::min<long long>(64, n / 8)), rows = (ni + G - 1) / G;
    const size_t smem = sizeof(double) * (size_t)(5 + rows) * n;
    if ((long long)smem > raise_dynamic_smem((const void *)k_tri_reduce))
        throw Error(NVPT_EINVAL, "tridiagonal form: order above the shared-memory limit");
    T tau = alloc(c, {n}, false), msg = alloc(c, {2 * n * n + 1}, false);  // the messages, the error word
    ck(cudaMemsetAsync(msg.p, 0xff, sizeof(double) * (2 * n * n + 1), c.st), "memset");
    int *err = (int *)(msg.p + 2 * n * n);
    TriArgs a{A, ni, d, e, tau.p, V, (unsigned long long *)msg.p, err, c.wait_limit ? c.wait_limit : kBarSpin};
    void *args[] = {&a};
    ck(cudaLaunchCooperativeKernel((const void *)k_tri_reduce, dim3(G), dim3(TB), args, smem, c.st),
       "cooperative launch");
    if (np) k_tri_wy<<<np, TB, 0, c.st>>>(ni, V, tau.p, Tm);
    g_launches.fetch_add(2, std::memory_order_relaxed);
    ck(cudaGetLastError(), "tridiagonal reduction");
    int h = 0;
    ck(cudaMemcpyAsync(&h, err, sizeof(int), cudaMemcpyDeviceToHost, c.st), "wait state");
    ck(cudaStreamSynchronize(c.st), "tridiagonal sync");
    return h ? 0 : 4;
}

void tri_resolvent(Ctx &c, const double *d, const double *e, long long n, const double *Y, long long ncol, long long L,
                   int nother, const double *sig, double *acc, int nd, long long dcol0, double *rho, double *xout) {
    const long long most = std::min<long long>(L, 8192);  // labels at a time: bounds the factors
    T fac = alloc(c, {4, n, most}, false), X;
    if (nd && !xout) {
        X = alloc(c, {n, L}, false);
        xout = X.p;
    }
    for (long long l0 = 0; l0 < L; l0 += most) {
        const int group = (int)std::min(most, L - l0);
        k_tri_solve<<<(group + 63) / 64, 64, 0, c.st>>>(d, e, (int)n, Y, ncol, L, l0, group, nother, sig, fac.p,
                                                       fac.p + 3 * n * group, acc, xout);
        g_launches.fetch_add(1, std::memory_order_relaxed);
    }
    if (nd) {
        k_tri_rho<<<(unsigned)((L * nd + 255) / 256), 256, 0, c.st>>>(Y, ncol, dcol0, xout, (int)n, L, nd, rho);
        g_launches.fetch_add(1, std::memory_order_relaxed);
    }
    ck(cudaGetLastError(), "tridiagonal resolvent");
}

}  // namespace s2
}  // namespace nvpt

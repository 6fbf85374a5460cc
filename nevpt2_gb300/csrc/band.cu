// The order-n^3 PC pencils in band form: K~ = Q B Q^T with B symmetric of half
// bandwidth 32, and the labels' resolvents (B + sigma)^-1 by banded elimination.
//
// A one-stage tridiagonalisation pays two grid-wide barriers for each of its n
// columns (16 us a column at n = 1000, 28 at 2744: latency, not FP64 work) and
// half of its flops are matrix-vector products.  Reducing to a band instead
// synchronises a few CTAs within a panel of 32 columns and does the rest as
// products with 32 columns.  Per panel P = A[r0:, j0:j0+32], r0 = j0 + 32:
//   k_band_qr      P = V-reflectors R (Householder; V, T of the compact WY form)
//   k_band_z       Z = A22 V
//   k_band_g       G = V^T Z
//   k_band_w       W = (Z - 1/2 V (T^T G)) T
//   k_band_update  A22 -= V W^T + W V^T
// which is A22 <- Q^T A22 Q.  The 4n^3/3 flops run at the FP64 rate, the panel
// costs latency only.  The resolvents need no eigenvectors and no further
// reduction: a banded LU with partial pivoting per label is 2048 n FMAs.
// CAS(14), two pencils of order 2744: energy stage 338 -> 305 ms; CAS(12), order
// 1728: 141 -> 125 ms.
#include <algorithm>
#include <cstdlib>

#include "../../include/nvpt2.h"
#include "band.cuh"
#include "grid_bar.cuh"

namespace nvpt {
namespace s2 {
namespace {

constexpr int NB = kBand;      // panel width = half bandwidth
constexpr int TB = 256;        // threads per CTA
constexpr int LP = NB + 1;     // padded row of a panel in shared memory

struct QrArgs {
    double *A;            // column-major n x n; panel columns j0 .. j0 + NB - 1, rows r0 .. n - 1
    long long n;
    int j0, m;            // m = n - r0 panel rows
    int chunk;            // rows per CTA (CTA 0 holds the pivot rows)
    double *V, *T, *G;    // V [m][NB] row-major, T [NB][NB] row-major; G [NB][NB] is zeroed for k_band_g
    double *acc;          // [3][2 NB]: column sums and pivot rows, triple-buffered; zero on entry
    Bar *bar;
    unsigned spin;
};

// Householder QR of one panel, its rows in the shared memory of a few CTAs.  A
// column costs one grid barrier: lane k of a warp holds entry k of a row, so the
// sums a^T p_k over the rows below the pivot give, for k >= c, the reflector's
// norm and the products it is applied with and, for k < c, the products with the
// earlier reflectors that T needs.
__global__ void __launch_bounds__(TB, 1) k_band_qr(QrArgs a) {
    extern __shared__ double P[];  // [chunk][LP]
    __shared__ double red[TB / 32][NB], s_d[NB], s_p[NB], Gs[NB][NB + 1], tau_s[NB];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, r0 = a.j0 + NB;
    const int i0 = blockIdx.x * a.chunk, rows = max(0, min(a.chunk, a.m - i0)), nref = min(NB, a.m);
    unsigned gen = *(volatile unsigned *)&a.bar->gen;
    if (blockIdx.x == 0)
        for (int i = tid; i < NB * NB; i += TB) a.G[i] = 0.0;
    for (int i = tid; i < rows * NB; i += TB) {
        const int row = i % rows, k = i / rows;
        P[row * LP + k] = a.A[(r0 + i0 + row) + (a.j0 + k) * a.n];
    }
    __syncthreads();
    for (int c = 0; c < nref; ++c) {
        double *acc = a.acc + (c % 3) * 2 * NB, *accz = a.acc + ((c + 2) % 3) * 2 * NB;
        double s = 0.0;
        for (int row = warp; row < rows; row += TB / 32) {
            const double p = P[row * LP + lane], x = __shfl_sync(0xffffffffu, p, c);
            if (i0 + row > c) s = fma(x, p, s);
        }
        red[warp][lane] = s;
        __syncthreads();
        if (warp == 0) {
            double t = 0.0;
            for (int w = 0; w < TB / 32; ++w) t += red[w][lane];
            atomicAdd(acc + lane, t);
            if (blockIdx.x == 0) __stcg(acc + NB + lane, P[c * LP + lane]);
        }
        if (!grid_bar(a.bar, gridDim.x, gen, a.spin)) return;
        // this buffer's sums were last read before this barrier and are next added to after the coming one
        if (blockIdx.x == 0 && tid < 2 * NB) __stcg(accz + tid, 0.0);
        if (warp == 0) {
            s_d[lane] = __ldcg(acc + lane);
            s_p[lane] = __ldcg(acc + NB + lane);
        }
        __syncthreads();
        const double alpha = s_p[c], x2 = s_d[c];
        double tau = 0.0, beta = alpha, scal = 0.0;
        if (x2 != 0.0) {
            beta = -copysign(sqrt(alpha * alpha + x2), alpha);
            tau = (beta - alpha) / beta;
            scal = 1.0 / (alpha - beta);
        }
        const double dot = s_p[lane] + scal * s_d[lane];  // v_c . p_k
        if (blockIdx.x == 0 && warp == 0) {
            Gs[lane][c] = dot;  // k < c: v_k . v_c
            if (lane == 0) tau_s[c] = tau;
        }
        const double w = lane > c ? tau * dot : 0.0;
        for (int row = warp; row < rows; row += TB / 32) {
            const int i = i0 + row;
            double p = P[row * LP + lane];
            const double v = i == c ? 1.0 : scal * __shfl_sync(0xffffffffu, p, c);
            if (i < c) continue;
            p = fma(-v, w, p);
            if (lane == c) p = i == c ? beta : v;
            P[row * LP + lane] = p;
        }
        __syncthreads();
    }
    // R into A, V with its unit diagonal
    for (int i = tid; i < rows * NB; i += TB) {
        const int k = i % NB, row = i / NB, gi = i0 + row;
        const double p = P[row * LP + k];
        a.V[(long long)gi * NB + k] = k >= nref || gi < k ? 0.0 : gi == k ? 1.0 : p;
        if (gi < NB) a.A[(r0 + gi) + (a.j0 + k) * a.n] = gi <= k ? p : 0.0;
    }
    if (blockIdx.x == 0 && warp == 0) {
        // T (upper triangular): T[c][c] = tau_c, T[:c, c] = -tau_c T[:c, :c] (V^T v_c); lane = row
        double t[NB];
#pragma unroll
        for (int c = 0; c < NB; ++c) {
            double x = 0.0;
            if (c < nref) {
#pragma unroll
                for (int l = 0; l < c; ++l) x = fma(l >= lane ? t[l] : 0.0, Gs[l][c], x);
                x = lane < c ? -tau_s[c] * x : lane == c ? tau_s[c] : 0.0;
            }
            t[c] = x;
            a.T[lane * NB + c] = x;
        }
    }
}

// Zp[split][m][NB]: the split's share of A22 V.  Tiles of 32 rows, all columns.
__global__ void __launch_bounds__(TB) k_band_z(const double *__restrict__ A, long long n, int r0, int m, int per,
                                               const double *__restrict__ V, double *__restrict__ Zp) {
    __shared__ double As[32][33], Vs[32][NB];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, i0 = blockIdx.x * 32;
    const int ka = blockIdx.y * per, kb = min(m, ka + per);
    double acc[4] = {};
    for (int k0 = ka; k0 < kb; k0 += 32) {
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const int k = k0 + warp + 8 * q, i = i0 + lane;
            As[warp + 8 * q][lane] = k < kb && i < m ? A[(r0 + i) + (r0 + k) * n] : 0.0;
            Vs[warp + 8 * q][lane] = k < kb ? V[(long long)k * NB + lane] : 0.0;
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < 32; ++k) {
            const double v = Vs[k][lane];
#pragma unroll
            for (int q = 0; q < 4; ++q) acc[q] = fma(As[k][warp * 4 + q], v, acc[q]);
        }
        __syncthreads();
    }
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const int i = i0 + warp * 4 + q;
        if (i < m) Zp[((long long)blockIdx.y * m + i) * NB + lane] = acc[q];
    }
}

constexpr int kGRows = 16;
// Z (into the first share) and G += V^T Z, 16 rows per CTA.
__global__ void __launch_bounds__(TB) k_band_g(int m, int splits, const double *__restrict__ V, double *Zp, double *G) {
    __shared__ double zs[kGRows][NB], vs[kGRows][NB];
    const int tid = threadIdx.x, i0 = blockIdx.x * kGRows;
    for (int e = tid; e < kGRows * NB; e += TB) {
        const int i = i0 + e / NB;
        double z = 0.0;
        if (i < m) {
            for (int s = 0; s < splits; ++s) z += Zp[((long long)s * m + i) * NB + e % NB];
            if (splits > 1) Zp[(long long)i * NB + e % NB] = z;
        }
        zs[e / NB][e % NB] = z;
        vs[e / NB][e % NB] = i < m ? V[(long long)i * NB + e % NB] : 0.0;
    }
    __syncthreads();
    for (int e = tid; e < NB * NB; e += TB) {
        double g = 0.0;
#pragma unroll
        for (int i = 0; i < kGRows; ++i) g = fma(vs[i][e / NB], zs[i][e % NB], g);
        atomicAdd(G + e, g);
    }
}

// W = (Z - 1/2 V N) T with N = T^T G, 16 rows per CTA.
__global__ void __launch_bounds__(TB) k_band_w(int m, const double *__restrict__ V, const double *__restrict__ Z,
                                               const double *__restrict__ Tm, const double *__restrict__ G, double *W) {
    __shared__ double ts[NB][NB], gs[NB][NB], ns[NB][NB], vs[kGRows][NB], us[kGRows][NB];
    const int tid = threadIdx.x, i0 = blockIdx.x * kGRows;
    for (int e = tid; e < NB * NB; e += TB) {
        ts[e / NB][e % NB] = Tm[e];
        gs[e / NB][e % NB] = G[e];
    }
    for (int e = tid; e < kGRows * NB; e += TB) {
        const int i = i0 + e / NB;
        vs[e / NB][e % NB] = i < m ? V[(long long)i * NB + e % NB] : 0.0;
    }
    __syncthreads();
    for (int e = tid; e < NB * NB; e += TB) {
        const int p = e / NB, q = e % NB;
        double x = 0.0;
        for (int k = 0; k <= p; ++k) x = fma(ts[k][p], gs[k][q], x);
        ns[p][q] = x;
    }
    __syncthreads();
    for (int e = tid; e < kGRows * NB; e += TB) {
        const int i = i0 + e / NB, q = e % NB;
        double x = 0.0;
#pragma unroll 8
        for (int k = 0; k < NB; ++k) x = fma(vs[e / NB][k], ns[k][q], x);
        us[e / NB][q] = (i < m ? Z[(long long)i * NB + q] : 0.0) - 0.5 * x;
    }
    __syncthreads();
    for (int e = tid; e < kGRows * NB; e += TB) {
        const int i = i0 + e / NB, q = e % NB;
        double x = 0.0;
        for (int k = 0; k <= q; ++k) x = fma(us[e / NB][k], ts[k][q], x);
        if (i < m) W[(long long)i * NB + q] = x;
    }
}

// A22 -= V W^T + W V^T, 64 x 64 tiles of the lower triangle, each also written
// to its mirror image (the matrix stays in full storage).
__global__ void __launch_bounds__(TB) k_band_update(double *__restrict__ A, long long n, int r0, int m,
                                                    const double *__restrict__ V, const double *__restrict__ W) {
    __shared__ double Ls[64][LP], Rs[64][LP];
    // tile (I >= J) of the triangle
    int I = (int)((sqrtf(8.0f * blockIdx.x + 1.0f) - 1.0f) * 0.5f);
    while ((I + 1) * (I + 2) / 2 <= (int)blockIdx.x) ++I;
    while (I * (I + 1) / 2 > (int)blockIdx.x) --I;
    const int J = blockIdx.x - I * (I + 1) / 2, i0 = I * 64, jq = J * 64, tid = threadIdx.x;
    const int tr = tid & 15, tc = tid >> 4;
    double acc[4][4] = {};
    for (int half = 0; half < 2; ++half) {
        const double *L = half ? W : V, *Rr = half ? V : W;
        for (int e = tid; e < 64 * NB; e += TB) {
            const int i = e / NB, k = e % NB;
            Ls[i][k] = i0 + i < m ? L[(long long)(i0 + i) * NB + k] : 0.0;
            Rs[i][k] = jq + i < m ? Rr[(long long)(jq + i) * NB + k] : 0.0;
        }
        __syncthreads();
#pragma unroll 8
        for (int k = 0; k < NB; ++k) {
            double l[4], r[4];
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                l[q] = Ls[tr + 16 * q][k];
                r[q] = Rs[tc + 16 * q][k];
            }
#pragma unroll
            for (int p = 0; p < 4; ++p)
#pragma unroll
                for (int q = 0; q < 4; ++q) acc[p][q] = fma(l[p], r[q], acc[p][q]);
        }
        __syncthreads();
    }
    // the new tile, through shared memory for the mirror image
    double *S = &Ls[0][0];  // [64][33] halves: 64 x 32 at a time
    for (int h = 0; h < 2; ++h) {
#pragma unroll
        for (int q = 0; q < 2; ++q)
#pragma unroll
            for (int p = 0; p < 4; ++p) {
                const int i = i0 + tr + 16 * p, jl = tc + 16 * q, j = jq + 32 * h + jl;
                double v = 0.0;
                if (i < m && j < m && i >= j) {
                    double *x = A + (r0 + i) + (r0 + j) * n;
                    v = *x - acc[p][2 * h + q];
                    *x = v;
                }
                S[(tr + 16 * p) * LP + jl] = v;
            }
        __syncthreads();
        for (int e = tid; e < 64 * 32; e += TB) {
            const int jl = e & 31, i = i0 + (e >> 5), j = jq + 32 * h + jl;
            if (i < m && j < m && i > j) A[(r0 + j) + (r0 + i) * n] = S[(e >> 5) * LP + jl];
        }
        __syncthreads();
    }
}

// AB[k][i] = B(i + k, i), k <= NB, from the reduced matrix.
__global__ void k_band_extract(const double *__restrict__ A, long long n, double *AB) {
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= n * (NB + 1)) return;
    const long long i = t % n, k = t / n;
    AB[t] = i + k < n ? A[i + k + i * n] : 0.0;
}

// One column of Y (column-major, ld n) per CTA: Y <- Q^T Y (forward) or Q Y, the
// column in shared memory, panel after panel.
__global__ void __launch_bounds__(TB) k_band_apply(long long n, int npanel, const double *__restrict__ V,
                                                   const double *__restrict__ Tm, double *Y, int forward) {
    extern __shared__ double y[];
    __shared__ double red[TB / 32][NB], t_s[NB], s_s[NB];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    double *col = Y + blockIdx.x * n;
    for (long long i = tid; i < n; i += TB) y[i] = col[i];
    __syncthreads();
    for (int q = 0; q < npanel; ++q) {
        const int p = forward ? q : npanel - 1 - q, r0 = (p + 1) * NB, m = (int)n - r0;
        // panels are packed one after another: rows n - NB (1 + p') for p' < p before this one
        const double *v = V + ((long long)p * n - (long long)NB * p * (p + 1) / 2) * NB, *T = Tm + (long long)p * NB * NB;
        double s = 0.0;
        for (int i = warp; i < m; i += TB / 32) s = fma(v[(long long)i * NB + lane], y[r0 + i], s);
        red[warp][lane] = s;
        __syncthreads();
        if (warp == 0) {
            double x = 0.0;
            for (int w = 0; w < TB / 32; ++w) x += red[w][lane];
            t_s[lane] = x;
            __syncwarp();
            x = 0.0;
            if (forward)
                for (int k = 0; k <= lane; ++k) x = fma(T[k * NB + lane], t_s[k], x);
            else
                for (int k = lane; k < NB; ++k) x = fma(T[lane * NB + k], t_s[k], x);
            s_s[lane] = x;
        }
        __syncthreads();
        for (int i = tid; i < m; i += TB) {
            const double2 *vr = reinterpret_cast<const double2 *>(v + (long long)i * NB);
            double x0 = 0.0, x1 = 0.0;
#pragma unroll
            for (int k = 0; k < NB / 2; ++k) {
                const double2 b = vr[k];
                x0 = fma(b.x, s_s[2 * k], x0);
                x1 = fma(b.y, s_s[2 * k + 1], x1);
            }
            y[r0 + i] -= x0 + x1;
        }
        __syncthreads();
    }
    for (long long i = tid; i < n; i += TB) col[i] = y[i];
}

__device__ __forceinline__ void block_add2(double v, double *dst) {
    __shared__ double red[32];
    for (int o = 16; o; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    __syncthreads();
    if (l == 0) red[w] = v;
    __syncthreads();
    if (w == 0) {
        v = l < (int)(blockDim.x >> 5) ? red[l] : 0.0;
        for (int o = 16; o; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
        if (l == 0) atomicAdd(dst, v);
    }
}

constexpr int UW = 2 * NB + 2;  // stored row of U: 1 / pivot, 2 NB entries right of it, the reduced right-hand side
constexpr int WC = 128;         // circular column window (2 NB + 2 columns in use)
// The type-0 PC sums of one label (a CTA) from (B + sig)^-1 y: elimination with
// partial pivoting over the NB + 1 rows a column reaches, kept in slots of shared
// memory (a pivot is not moved: its slot takes the next row of B), rows of U
// streamed out, then the back substitution by one warp.  Outputs as
// k_tridiag_resolvent.  Bound by the FP64 pipe of one SM (2 NB^2 FMAs a column).
__global__ void __launch_bounds__(TB) k_band_resolvent(const double *__restrict__ AB, long long n, const double *Y,
                                                       long long ncol, long long L, long long l0, int nother,
                                                       const double *sig, double *U, double *acc, int nd,
                                                       long long dcol0, double *rho, double *xout) {
    extern __shared__ double x[];  // solution, n
    __shared__ double Wn[NB + 1][WC + 1], ys[NB + 1];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const long long l = l0 + blockIdx.x;
    const double s = sig[l];
    double *Ul = U + (long long)blockIdx.x * n * UW;
    for (int e = tid; e < (NB + 1) * (WC + 1); e += TB) Wn[0][e] = 0.0;
    __syncthreads();
    // element t of row r: column r - NB + t
    auto band = [&](long long r, int t) {
        const long long c = r - NB + t;
        if (r >= n || c < 0 || c >= n) return 0.0;
        const int k = t < NB ? NB - t : t - NB;
        return AB[k * n + (c < r ? c : r)] + (k == 0 ? s : 0.0);
    };
    for (int e = tid; e < (NB + 1) * (2 * NB + 1); e += TB) {
        const int r = e / (2 * NB + 1), t = e % (2 * NB + 1), c = r - NB + t;
        if (c >= 0 && r < n) Wn[r][c & (WC - 1)] = band(r, t);
    }
    if (tid <= NB) ys[tid] = tid < n ? Y[tid * ncol + l] : 0.0;
    __syncthreads();
    int live = (int)min((long long)(NB + 1), n);  // slots 0 .. live - 1 hold rows (all slots but at the end)
    unsigned long long dead = 0;                  // slots whose row is used up and not replaced
    for (int e = live; e <= NB; ++e) dead |= 1ull << e;
    for (long long j = 0; j < n; ++j) {
        const int cj = (int)(j & (WC - 1));
        const long long rn = j + NB + 1;
        double next = 0.0, ynext = 0.0;  // the row that takes the pivot's slot
        if (tid <= 2 * NB) next = band(rn, tid);
        else if (tid == 2 * NB + 1 && rn < n) ynext = Y[rn * ncol + l];
        // the pivot: every warp finds the same one
        double best = (dead >> lane & 1) ? -1.0 : fabs(Wn[lane][cj]);
        int p = lane;
        if (lane == 0 && !(dead >> NB & 1)) {
            const double b = fabs(Wn[NB][cj]);
            if (b > best) { best = b; p = NB; }
        }
#pragma unroll
        for (int o = 16; o; o >>= 1) {
            const double b = __shfl_xor_sync(0xffffffffu, best, o);
            const int q = __shfl_xor_sync(0xffffffffu, p, o);
            if (b > best || (b == best && q < p)) { best = b; p = q; }
        }
        const double inv = 1.0 / Wn[p][cj], yp = ys[p];
        const int c0 = (cj + 1 + lane) & (WC - 1), c1 = (cj + 1 + NB + lane) & (WC - 1), cz = (cj + 1 + 2 * NB) & (WC - 1);
        const double p0 = Wn[p][c0], p1 = Wn[p][c1];
        if (warp == 7) {
            Ul[j * UW + 1 + lane] = p0;
            Ul[j * UW + 1 + NB + lane] = p1;
            if (lane == 0) Ul[j * UW] = inv;
            if (lane == 1) Ul[j * UW + 2 * NB + 1] = yp;
        }
        for (int q = warp; q <= NB; q += TB / 32) {
            if (q == p || (dead >> q & 1)) continue;
            const double f = Wn[q][cj] * inv;
            Wn[q][c0] = fma(-f, p0, Wn[q][c0]);
            Wn[q][c1] = fma(-f, p1, Wn[q][c1]);
            if (lane == 0) {
                ys[q] = fma(-f, yp, ys[q]);
                Wn[q][cz] = 0.0;  // a column that enters the window
            }
        }
        __syncthreads();
        if (rn < n) {
            if (tid <= 2 * NB) Wn[p][(int)((j + 1 + tid) & (WC - 1))] = next;
            else if (tid == 2 * NB + 1) ys[p] = ynext;
        } else {
            dead |= 1ull << p;
        }
        __syncthreads();
    }
    // back substitution: a warp, two entries of a row per lane, rows prefetched
    if (warp == 0) {
        constexpr int PF = 4;
        double u0[PF], u1[PF], dv[PF], yv[PF];
        auto load = [&](long long j, int q) {
            const double *u = Ul + max(j, 0ll) * UW;
            u0[q] = __ldcg(u + 1 + lane);
            u1[q] = __ldcg(u + 1 + NB + lane);
            dv[q] = __ldcg(u);
            yv[q] = __ldcg(u + 2 * NB + 1);
        };
#pragma unroll
        for (int q = 0; q < PF; ++q) load(n - 1 - q, q);
        for (long long jb = n - 1; jb >= 0; jb -= PF)
#pragma unroll
            for (int q = 0; q < PF; ++q) {
                const long long j = jb - q;
                if (j >= 0) {
                    const long long a = j + 1 + lane, b = a + NB;
                    double t = (a < n ? u0[q] * x[a] : 0.0) + (b < n ? u1[q] * x[b] : 0.0);
                    for (int o = 16; o; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
                    const double xj = (yv[q] - t) * dv[q];
                    if (lane == 0) x[j] = xj;
                    __syncwarp();
                }
                load(j - PF, q);
            }
    }
    __syncthreads();
    if (xout)
        for (long long i = tid; i < n; i += TB) xout[i * L + l] = x[i];
    double en = 0.0, ps = 0.0, offs[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    for (long long i = tid; i < n; i += TB) {
        const double v = x[i];
        en -= Y[i * ncol + l] * v;
        ps += v * v;
        for (int k = 0; k < nother && k < 8; ++k) offs[k] -= Y[i * ncol + (k + 1) * L + l] * v;
    }
    block_add2(en, acc + 0);
    block_add2(ps, acc + 1);
    for (int k = 0; k < nother && k < 8; ++k) block_add2(offs[k], acc + 2 + k);
    for (int k = 0; k < nd; ++k) {
        double v = 0.0;
        for (long long i = tid; i < n; i += TB) v -= Y[i * ncol + dcol0 + k] * x[i];
        block_add2(v, rho + l * nd + k);
    }
}

}  // namespace

long long band_rows(long long n) {  // rows of all panels
    const long long np = band_panels(n);
    return np * n - kBand * np * (np + 1) / 2;
}

int band_reduce(Ctx &c, double *A, long long n, double *V, double *Tm, double *AB) {
    const int np = band_panels(n);
    T W = alloc(c, {n, NB}, false), G = alloc(c, {NB, NB}, false);
    T ctl = alloc(c, {2 + 6 * NB}, true);  // Bar, column sums
    Bar *bar = (Bar *)ctl.p;
    double *acc = ctl.p + 2;
    int sms = 0, dev = 0;
    ck(cudaGetDevice(&dev), "cudaGetDevice");
    ck(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev), "attr");
    const int lim = raise_dynamic_smem((const void *)k_band_qr);
    // shares of A22 V: enough CTAs for the chip, at least 128 of K each
    const int most = (int)std::max<long long>(1, std::min<long long>(8, n / 128));
    T Zp = alloc(c, {most, n, NB}, false);
    double *v = V;
    for (int p = 0; p < np; ++p) {
        const int j0 = p * NB, r0 = j0 + NB, m = (int)n - r0;
        double *t = Tm + (long long)p * NB * NB;
        // 64 to 128 panel rows per CTA: the column's latency falls with its rows, and rises with the CTAs
        const int G0 = std::max(1, std::min(sms / 4, m / 64));
        const int chunk = std::max(NB, (m + G0 - 1) / G0), ctas = (m + chunk - 1) / chunk;
        const size_t smem = sizeof(double) * (size_t)chunk * LP;
        if ((long long)smem > lim) throw Error(1, "band: order too large for the panel's shared memory");
        if (p) ck(cudaMemsetAsync(acc, 0, sizeof(double) * 6 * NB, c.st), "memset");
        QrArgs q{A, n, j0, m, chunk, v, t, G.p, acc, bar, c.wait_limit ? c.wait_limit : kBarSpin};
        void *args[] = {&q};
        ck(cudaLaunchCooperativeKernel((const void *)k_band_qr, dim3(ctas), dim3(TB), args, smem, c.st),
           "cooperative launch");
        const int tiles = (m + 31) / 32, splits = std::max(1, std::min(most, std::min((2 * sms + tiles - 1) / tiles, m / 128)));
        const int per = ((m + splits - 1) / splits + 31) / 32 * 32, ns = (m + per - 1) / per;
        k_band_z<<<dim3(tiles, ns), TB, 0, c.st>>>(A, n, r0, m, per, v, Zp.p);
        k_band_g<<<(m + kGRows - 1) / kGRows, TB, 0, c.st>>>(m, ns, v, Zp.p, G.p);
        k_band_w<<<(m + kGRows - 1) / kGRows, TB, 0, c.st>>>(m, v, Zp.p, t, G.p, W.p);
        const int t64 = (m + 63) / 64;
        k_band_update<<<t64 * (t64 + 1) / 2, TB, 0, c.st>>>(A, n, r0, m, v, W.p);
        g_launches.fetch_add(5, std::memory_order_relaxed);
        v += (long long)m * NB;
    }
    k_band_extract<<<(unsigned)((n * (NB + 1) + 255) / 256), 256, 0, c.st>>>(A, n, AB);
    g_launches.fetch_add(1, std::memory_order_relaxed);
    ck(cudaGetLastError(), "band reduction");
    int h[3] = {0, 0, 0};
    ck(cudaMemcpyAsync(h, ctl.p, sizeof(int) * 3, cudaMemcpyDeviceToHost, c.st), "barrier state");
    ck(cudaStreamSynchronize(c.st), "band sync");
    return h[2] ? 4 : 0;
}

void band_apply(Ctx &c, long long n, const double *V, const double *Tm, double *Y, long long m, bool forward) {
    const int np = band_panels(n);
    if (np == 0 || m == 0) return;
    const size_t smem = sizeof(double) * (size_t)n;
    if ((long long)smem > raise_dynamic_smem((const void *)k_band_apply))
        throw Error(NVPT_EINVAL, "band: order above the shared-memory limit");
    k_band_apply<<<(unsigned)m, TB, smem, c.st>>>(n, np, V, Tm, Y, forward ? 1 : 0);
    g_launches.fetch_add(1, std::memory_order_relaxed);
    ck(cudaGetLastError(), "band apply");
}

void band_resolvent(Ctx &c, const double *AB, long long n, const double *Y, long long ncol, long long L, int nother,
                    const double *sig, double *acc, int nd, long long dcol0, double *rho, double *xout) {
    const size_t smem = sizeof(double) * (size_t)n;
    if ((long long)smem > raise_dynamic_smem((const void *)k_band_resolvent))
        throw Error(NVPT_EINVAL, "resolvent: pencil order above the shared-memory limit");
    const long long group = std::min<long long>(L, 304);  // labels at a time: bounds the factors
    T U = alloc(c, {group, n, UW}, false);
    for (long long l0 = 0; l0 < L; l0 += group) {
        k_band_resolvent<<<(unsigned)std::min(group, L - l0), TB, smem, c.st>>>(AB, n, Y, ncol, L, l0, nother, sig, U.p,
                                                                               acc, nd, dcol0, rho, xout);
        g_launches.fetch_add(1, std::memory_order_relaxed);
    }
    ck(cudaGetLastError(), "band resolvent");
}

}  // namespace s2
}  // namespace nvpt

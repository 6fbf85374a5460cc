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

constexpr int kQrMost = 39;  // CTAs of a panel: with the pivot row, at most 5 messages a thread

struct QrArgs {
    double *A;            // column-major n x n; panel columns j0 .. j0 + NB - 1, rows r0 .. n - 1
    long long n;
    int j0, m;            // m = n - r0 panel rows
    int chunk;            // rows per CTA (CTA 0 holds the pivot rows)
    double *V, *T, *G;    // V [m][NB] row-major, T [NB][NB] row-major; G [NB][NB] is zeroed for k_band_g
    unsigned long long *msg;  // [NB][CTAs + 1][NB], all kNoMsg on entry
    int *err;             // raised once a wait gave up
    unsigned spin;        // polls before a wait gives up
};

// Householder QR of one panel, its rows in the shared memory of a few CTAs.  Lane k
// of a warp holds entry k of a row, so the sums a^T p_k over the rows below the
// pivot give, for k >= c, the reflector's norm and the products it is applied with
// and, for k < c, the products with the earlier reflectors that T needs.
// Bound by latency: a column is one exchange of those sums between the CTAs.  Each
// CTA stores its share where every other one polls for it (a word that is not
// kNoMsg has arrived: one trip instead of the sums, fence, counter and flag of a
// grid barrier, and the order of the additions is fixed); one warp turns the sums
// into the reflector (a square root and two divisions in all eight would fill the
// FP64 pipe for 2 us) and the update of a row also takes its share of the next
// column's sums.  Order 2744: 7.3 -> 5.4 us a column.
__global__ void __launch_bounds__(TB, 1) k_band_qr(QrArgs a) {
    extern __shared__ double P[];  // [chunk][LP]
    __shared__ double red[TB / 32][NB], red2[TB / 32][NB], s_p[NB], s_w[NB], Gs[NB][NB + 1], tau_s[NB], s_beta, s_scal;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, r0 = a.j0 + NB, ctas = gridDim.x;
    const int i0 = blockIdx.x * a.chunk, rows = max(0, min(a.chunk, a.m - i0)), nref = min(NB, a.m);
    if (blockIdx.x == 0)
        for (int i = tid; i < NB * NB; i += TB) a.G[i] = 0.0;
    for (int i = tid; i < rows * NB; i += TB) {
        const int row = i % rows, k = i / rows;
        P[row * LP + k] = a.A[(r0 + i0 + row) + (a.j0 + k) * a.n];
    }
    __syncthreads();
    double s = 0.0;
    for (int row = warp; row < rows; row += TB / 32) {
        const double p = P[row * LP + lane], x = __shfl_sync(0xffffffffu, p, 0);
        if (i0 + row > 0) s = fma(x, p, s);
    }
    for (int c = 0; c < nref; ++c) {
        unsigned long long *msg = a.msg + (long long)c * (ctas + 1) * NB;
        red[warp][lane] = s;
        __syncthreads();
        if (warp == 0) {
            double t = 0.0;
#pragma unroll
            for (int w = 0; w < TB / 32; ++w) t += red[w][lane];
            send_word(msg + blockIdx.x * NB + lane, t);
        } else if (warp == 1 && blockIdx.x == 0) {
            send_word(msg + ctas * NB + lane, P[c * LP + lane]);
        }
        unsigned long long v[5];
        int ok = 1;
        for (unsigned spins = 0;;) {
            bool all = true;
#pragma unroll
            for (int q = 0; q < 5; ++q) {
                const int b = warp + q * (TB / 32);
                v[q] = 0;
                if (b <= ctas)
                    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v[q]) : "l"(msg + b * NB + lane) : "memory");
            }
#pragma unroll
            for (int q = 0; q < 5; ++q) all = all && v[q] != kNoMsg;
            if (all) break;
            if (++spins > a.spin || (spins % 64 == 0 && *(volatile int *)a.err)) {
                atomicExch(a.err, 1);
                ok = 0;
                break;
            }
        }
        double t = 0.0;
#pragma unroll
        for (int q = 0; q < 5; ++q) {
            const int b = warp + q * (TB / 32);
            if (b < ctas) t += __longlong_as_double(v[q]);
            if (b == ctas) s_p[lane] = __longlong_as_double(v[q]);
        }
        red2[warp][lane] = t;
        if (!__syncthreads_and(ok)) return;
        if (warp == 0) {
            double d = 0.0;
#pragma unroll
            for (int w = 0; w < TB / 32; ++w) d += red2[w][lane];
            const double x2 = __shfl_sync(0xffffffffu, d, c), alpha = s_p[c];
            double tau = 0.0, beta = alpha, scal = 0.0;
            if (x2 != 0.0) {
                beta = -copysign(sqrt(fma(alpha, alpha, x2)), alpha);
                tau = (beta - alpha) / beta;
                scal = 1.0 / (alpha - beta);
            }
            const double dot = fma(scal, d, s_p[lane]);  // v_c . p_k
            s_w[lane] = lane > c ? tau * dot : 0.0;
            if (lane == 0) {
                s_beta = beta;
                s_scal = scal;
                tau_s[c] = tau;
            }
            Gs[lane][c] = dot;  // k < c: v_k . v_c
        }
        __syncthreads();
        const double w = s_w[lane], scal = s_scal, beta = s_beta;
        s = 0.0;
        for (int row = warp; row < rows; row += TB / 32) {
            const int i = i0 + row;
            if (i < c) continue;
            double p = P[row * LP + lane];
            const double v = i == c ? 1.0 : scal * __shfl_sync(0xffffffffu, p, c);
            p = fma(-v, w, p);
            if (lane == c) p = i == c ? beta : v;
            P[row * LP + lane] = p;
            const double x = __shfl_sync(0xffffffffu, p, (c + 1) & 31);
            if (i > c + 1) s = fma(x, p, s);
        }
    }
    __syncthreads();
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

// W = (Z - 1/2 V N) T with N = T^T G, 16 rows per CTA; the messages are reset for the next panel.
__global__ void __launch_bounds__(TB) k_band_w(int m, const double *__restrict__ V, const double *__restrict__ Z,
                                               const double *__restrict__ Tm, const double *__restrict__ G, double *W,
                                               unsigned long long *msg, int words) {
    for (int i = blockIdx.x * TB + threadIdx.x; i < words; i += gridDim.x * TB) msg[i] = kNoMsg;
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

// A22 -= V W^T + W V^T, 32 x 32 tiles of the lower triangle, each also written to its
// mirror image (the matrix stays in full storage).  Bound by the FP64 pipe; tiles of 64
// left SMs idle in the last wave of each panel.  Order 2744, all panels: 15.4 -> 12.3 ms
// (2/3 n^3 flops, 12.1 ms at the FP64 rate).
__global__ void __launch_bounds__(TB) k_band_update(double *__restrict__ A, long long n, int r0, int m,
                                                    const double *__restrict__ V, const double *__restrict__ W) {
    __shared__ double Ls[2][32][LP], Rs[2][32][LP];
    // tile (I >= J) of the triangle
    int I = (int)((sqrtf(8.0f * blockIdx.x + 1.0f) - 1.0f) * 0.5f);
    while ((I + 1) * (I + 2) / 2 <= (int)blockIdx.x) ++I;
    while (I * (I + 1) / 2 > (int)blockIdx.x) --I;
    const int i0 = I * 32, j0 = (blockIdx.x - I * (I + 1) / 2) * 32, tid = threadIdx.x;
    const int tr = tid & 15, tc = tid >> 4;
    for (int e = tid; e < 32 * NB; e += TB) {
        const int r = e / NB, k = e % NB;
        const bool li = i0 + r < m, lj = j0 + r < m;
        const long long a = (long long)(i0 + r) * NB + k, b = (long long)(j0 + r) * NB + k;
        Ls[0][r][k] = li ? V[a] : 0.0;
        Ls[1][r][k] = li ? W[a] : 0.0;
        Rs[0][r][k] = lj ? W[b] : 0.0;
        Rs[1][r][k] = lj ? V[b] : 0.0;
    }
    // the old tile arrives meanwhile
    double old[2][2], acc[2][2] = {};
#pragma unroll
    for (int p = 0; p < 2; ++p)
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            const int i = i0 + tr + 16 * p, j = j0 + tc + 16 * q;
            old[p][q] = i < m && j < m ? A[(r0 + i) + (r0 + j) * n] : 0.0;
        }
    __syncthreads();
#pragma unroll
    for (int h = 0; h < 2; ++h)
#pragma unroll 8
        for (int k = 0; k < NB; ++k) {
            const double l0 = Ls[h][tr][k], l1 = Ls[h][tr + 16][k], r0_ = Rs[h][tc][k], r1 = Rs[h][tc + 16][k];
            acc[0][0] = fma(l0, r0_, acc[0][0]);
            acc[0][1] = fma(l0, r1, acc[0][1]);
            acc[1][0] = fma(l1, r0_, acc[1][0]);
            acc[1][1] = fma(l1, r1, acc[1][1]);
        }
    __syncthreads();
    // the new tile, through shared memory for the mirror image
#pragma unroll
    for (int p = 0; p < 2; ++p)
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            const int i = i0 + tr + 16 * p, j = j0 + tc + 16 * q;
            const double v = old[p][q] - acc[p][q];
            if (i < m && j < m && i >= j) A[(r0 + i) + (r0 + j) * n] = v;
            Ls[0][tr + 16 * p][tc + 16 * q] = v;
        }
    __syncthreads();
    for (int e = tid; e < 32 * 32; e += TB) {
        const int j = j0 + (e & 31), i = i0 + (e >> 5);
        if (i < m && j < m && i > j) A[(r0 + j) + (r0 + i) * n] = Ls[0][e >> 5][e & 31];
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
__global__ void __launch_bounds__(TB) k_wy_apply(long long n, int npanel, int first, const double *__restrict__ V,
                                                   const double *__restrict__ Tm, double *Y, int forward) {
    extern __shared__ double y[];
    __shared__ double red[TB / 32][NB], t_s[NB], s_s[NB];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    double *col = Y + blockIdx.x * n;
    for (long long i = tid; i < n; i += TB) y[i] = col[i];
    __syncthreads();
    for (int q = 0; q < npanel; ++q) {
        const int p = forward ? q : npanel - 1 - q, r0 = p * NB + first, m = (int)n - r0;
        // panels are packed one after another: n - first - NB p' rows for each p' < p before this one
        const double *v = V + (p * (n - first) - (long long)NB * p * (p - 1) / 2) * NB, *T = Tm + (long long)p * NB * NB;
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
constexpr int SL = NB + 2;      // slots: the NB + 1 rows that a column reaches and the row that comes in
// The type-0 PC sums of one label (a CTA) from (B + sig)^-1 y: elimination with
// partial pivoting over the NB + 1 rows a column reaches, kept in slots of shared
// memory (a row is not moved: its slot is refilled once it was the pivot), rows of U
// streamed out, then the back substitution by one warp.  The pivot is the largest
// by the leading 32 bits.
// Bound by the FP64 pipe of the label's SM (2 NB^2 FMAs, 66 warp instructions of 16
// clocks, a column).  Warp 0 runs one column ahead of the others (its update,
// pivot, reciprocal and multipliers, so that the chain of the search is hidden
// behind the other columns' updates and its division done once), warp 7 moves the
// rows in and out, so a column is one block barrier.  Order 2744, with the other
// classes running: 4.6 -> 1.8 us a column.
__global__ void __launch_bounds__(TB) k_band_resolvent(const double *__restrict__ AB, long long n, const double *Y,
                                                       long long ncol, long long L, long long l0, int nother,
                                                       const double *sig, double *U, double *acc, int nd,
                                                       long long dcol0, double *rho, double *xout) {
    extern __shared__ double x[];  // solution, n
    __shared__ double Wn[SL][WC + 1], ys[SL], fs[2][SL], s_inv[2];
    __shared__ int s_piv[2];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const long long l = l0 + blockIdx.x;
    const double s = sig[l];
    double *Ul = U + (long long)blockIdx.x * n * UW;
    // element t of row r: column r - NB + t
    auto band = [&](long long r, int t) {
        const long long c = r - NB + t;
        if (r >= n || c < 0 || c >= n) return 0.0;
        const int k = t < NB ? NB - t : t - NB;
        return AB[k * n + (c < r ? c : r)] + (k == 0 ? s : 0.0);
    };
    for (int e = tid; e < SL * (WC + 1); e += TB) Wn[0][e] = 0.0;
    __syncthreads();
    for (int e = tid; e < (NB + 1) * (2 * NB + 1); e += TB) {
        const int r = e / (2 * NB + 1), t = e % (2 * NB + 1), c = r - NB + t;
        if (c >= 0 && r < n) Wn[r][c & (WC - 1)] = band(r, t);
    }
    if (tid < SL) ys[tid] = tid <= NB && tid < n ? Y[tid * ncol + l] : 0.0;
    __syncthreads();
    // slots without a row: the one that is filled next (free) and, at the end, used-up ones
    int free_slot = NB + 1;
    unsigned long long none = ~0ull << min((long long)(NB + 1), n);
    double f0 = 0.0, f1 = 0.0;  // warp 0: the multipliers of slots lane and 32 + lane
    // warp 0: pivot, reciprocal and multipliers of column j from its entries v0, v1 in the slots
    auto select = [&](long long j, double v0, double v1, unsigned long long off) {
        unsigned k0 = off >> lane & 1 ? 0u : ((unsigned)__double2hiint(v0) & 0x7fffffffu) + 1u;
        unsigned k1 = lane >= SL - 32 || (off >> (32 + lane) & 1) ? 0u : ((unsigned)__double2hiint(v1) & 0x7fffffffu) + 1u;
        const unsigned top = __reduce_max_sync(0xffffffffu, max(k0, k1));
        const int from = __ffs(__ballot_sync(0xffffffffu, max(k0, k1) == top)) - 1;
        const double pv = __shfl_sync(0xffffffffu, k1 > k0 ? v1 : v0, from);
        const int slot = __shfl_sync(0xffffffffu, k1 > k0 ? 32 + lane : lane, from);
        const double inv = 1.0 / pv;
        f0 = v0 * inv;
        f1 = v1 * inv;
        const int b = (int)(j & 1);
        fs[b][lane] = f0;
        if (lane < SL - 32) fs[b][32 + lane] = f1;
        if (lane == 0) {
            s_piv[b] = slot;
            s_inv[b] = inv;
        }
    };
    if (warp == 0) select(0, Wn[lane][0], lane < SL - 32 ? Wn[32 + lane][0] : 0.0, none);
    // rows that come in, PF columns ahead: warp 7 whole rows, warp 0 their first entries
    constexpr int PF = 4;
    double a0[PF], a1[PF], a2[PF];
    auto fetch = [&](long long j, int q) {
        const long long r = j + NB + 1;
        if (warp == 7) {
            a0[q] = band(r, lane);
            a1[q] = band(r, NB + lane);
            a2[q] = lane == 0 ? band(r, 2 * NB) : lane == 1 && r < n ? Y[r * ncol + l] : 0.0;
        } else if (warp == 0) {
            a0[q] = band(r, 0);
        }
    };
#pragma unroll
    for (int q = 0; q < PF; ++q) fetch(q, q);
    __syncthreads();
    for (long long jb = 0; jb < n; jb += PF) {
#pragma unroll
        for (int q = 0; q < PF; ++q) {
            const long long j = jb + q;
            if (j >= n) break;
            const int b = (int)(j & 1), p = s_piv[b], in = free_slot, c1 = (int)((j + 1) & (WC - 1));
            const bool more = j + NB + 1 < n;
            const unsigned long long off = none | 1ull << p;  // slots not updated
            unsigned long long next = off;                    // slots without a row after this column
            if (more) next &= ~(1ull << in);
            if (warp == 0) {
                const double pc = Wn[p][c1];
                double v0 = off >> lane & 1 ? 0.0 : fma(-f0, pc, Wn[lane][c1]), v1 = 0.0;
                if (lane < SL - 32 && !(off >> (32 + lane) & 1)) v1 = fma(-f1, pc, Wn[32 + lane][c1]);
                if (more && lane == in) v0 = a0[q];
                if (more && 32 + lane == in) v1 = a0[q];
                if (j + 1 < n) select(j + 1, v0, v1, next);
            } else if (warp < 7) {
                // columns j + 2 .. j + 65; the last one enters the window
                const int ca = (int)((j + 2 + lane) & (WC - 1)), cb = (int)((j + 2 + NB + lane) & (WC - 1));
                const double pa = Wn[p][ca], pb = Wn[p][cb];
#pragma unroll
                for (int k = 0; k < 6; ++k) {
                    const int r = warp - 1 + 6 * k;
                    if (r < SL && !(off >> r & 1)) {
                        const double f = fs[b][r];
                        Wn[r][ca] = fma(-f, pa, Wn[r][ca]);
                        Wn[r][cb] = lane == 31 ? 0.0 : fma(-f, pb, Wn[r][cb]);
                    }
                }
            } else {
                const double yp = ys[p];
                double *u = Ul + j * UW;
                u[1 + lane] = Wn[p][(int)((j + 1 + lane) & (WC - 1))];
                u[1 + NB + lane] = Wn[p][(int)((j + 1 + NB + lane) & (WC - 1))];
                if (lane == 0) u[0] = s_inv[b];
                if (lane == 1) u[2 * NB + 1] = yp;
                if (!(off >> lane & 1)) ys[lane] = fma(-fs[b][lane], yp, ys[lane]);
                if (lane < SL - 32 && !(off >> (32 + lane) & 1)) ys[32 + lane] = fma(-fs[b][32 + lane], yp, ys[32 + lane]);
                if (more) {
                    Wn[in][(int)((j + 1 + lane) & (WC - 1))] = a0[q];
                    Wn[in][(int)((j + 1 + NB + lane) & (WC - 1))] = a1[q];
                    if (lane == 0) Wn[in][(int)((j + 1 + 2 * NB) & (WC - 1))] = a2[q];
                    if (lane == 1) ys[in] = a2[q];
                }
            }
            fetch(j + PF, q);
            none = next;
            free_slot = p;
            __syncthreads();
        }
    }
    // back substitution: a warp, two entries of a row per lane, rows prefetched
    if (warp == 0) {
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

int band_reduce(Ctx &c, double *A, long long n, double *V, double *Tm, double *AB) {
    const int np = wy_panels(n, NB);
    T W = alloc(c, {n, NB}, false), G = alloc(c, {NB, NB}, false);
    T msg = alloc(c, {NB, kQrMost + 1, NB}, false), ctl = alloc(c, {1}, true);
    int *err = (int *)ctl.p;
    int sms = 0, dev = 0;
    ck(cudaGetDevice(&dev), "cudaGetDevice");
    ck(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev), "attr");
    const int lim = raise_dynamic_smem((const void *)k_band_qr);
    // shares of A22 V: eight CTAs an SM, so that the last one costs little, at least 64 of K each
    // (two an SM: 15.7 ms for all panels of order 2744, eight: 12.6)
    const int most = (int)std::max<long long>(1, std::min<long long>(16, n / 64));
    T Zp = alloc(c, {most, n, NB}, false);
    double *v = V;
    for (int p = 0; p < np; ++p) {
        const int j0 = p * NB, r0 = j0 + NB, m = (int)n - r0;
        double *t = Tm + (long long)p * NB * NB;
        // 64 to 128 panel rows per CTA: the column's latency falls with its rows, and rises with the CTAs
        const int G0 = std::max(1, std::min(std::min(sms / 4, kQrMost), m / 64));
        const int chunk = std::max(NB, (m + G0 - 1) / G0), ctas = (m + chunk - 1) / chunk;
        const size_t smem = sizeof(double) * (size_t)chunk * LP;
        if ((long long)smem > lim) throw Error(1, "band: order too large for the panel's shared memory");
        if (!p) ck(cudaMemsetAsync(msg.p, 0xff, sizeof(double) * NB * (ctas + 1) * NB, c.st), "memset");
        QrArgs q{A, n, j0, m, chunk, v, t, G.p, (unsigned long long *)msg.p, err, c.wait_limit ? c.wait_limit : kBarSpin};
        void *args[] = {&q};
        ck(cudaLaunchCooperativeKernel((const void *)k_band_qr, dim3(ctas), dim3(TB), args, smem, c.st),
           "cooperative launch");
        const int tiles = (m + 31) / 32, splits = std::max(1, std::min(most, std::min((8 * sms + tiles / 2) / tiles, m / 64)));
        const int per = ((m + splits - 1) / splits + 31) / 32 * 32, ns = (m + per - 1) / per;
        k_band_z<<<dim3(tiles, ns), TB, 0, c.st>>>(A, n, r0, m, per, v, Zp.p);
        k_band_g<<<(m + kGRows - 1) / kGRows, TB, 0, c.st>>>(m, ns, v, Zp.p, G.p);
        k_band_w<<<(m + kGRows - 1) / kGRows, TB, 0, c.st>>>(m, v, Zp.p, t, G.p, W.p,
                                                           (unsigned long long *)msg.p, NB * (ctas + 1) * NB);
        k_band_update<<<tiles * (tiles + 1) / 2, TB, 0, c.st>>>(A, n, r0, m, v, W.p);
        g_launches.fetch_add(5, std::memory_order_relaxed);
        v += (long long)m * NB;
    }
    k_band_extract<<<(unsigned)((n * (NB + 1) + 255) / 256), 256, 0, c.st>>>(A, n, AB);
    g_launches.fetch_add(1, std::memory_order_relaxed);
    ck(cudaGetLastError(), "band reduction");
    int h = 0;
    ck(cudaMemcpyAsync(&h, err, sizeof(int), cudaMemcpyDeviceToHost, c.st), "wait state");
    ck(cudaStreamSynchronize(c.st), "band sync");
    return h ? 4 : 0;
}

void wy_apply(Ctx &c, long long n, int first, const double *V, const double *Tm, double *Y, long long m, bool forward) {
    const int np = wy_panels(n, first);
    if (np == 0 || m == 0) return;
    const size_t smem = sizeof(double) * (size_t)n;
    if ((long long)smem > raise_dynamic_smem((const void *)k_wy_apply))
        throw Error(NVPT_EINVAL, "reflectors: order above the shared-memory limit");
    k_wy_apply<<<(unsigned)m, TB, smem, c.st>>>(n, np, first, V, Tm, Y, forward ? 1 : 0);
    g_launches.fetch_add(1, std::memory_order_relaxed);
    ck(cudaGetLastError(), "reflectors");
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

// Reduction of the order-n^3 pencils K v = w S v to standard form through the
// inverse Cholesky factor W = L^-1 of S = L L^T: K~ = W K W^T.
//
// FP64 runs at 2 FMAs a clock and SM here, so an O(n^3) step is bound by that pipe
// wherever it is a product of tiles, and by latency wherever it is a triangular
// solve.  Everything below is therefore a 64 x 64 tile product; the only serial
// part is the factorisation of a diagonal block.  All matrices are padded to whole
// 64-blocks (identity in S, zero in K), so no tile has a ragged edge.
//   factor   for each block column k: k_spd_panel   L21 = A21 W11^T, W[k, :] = W11 R[k, :]
//                                     k_spd_step    A22 -= L21 L21^T, R[i, :] -= L21 W[k, :],
//                                                   and the next diagonal block's L11, W11
//            (R, the identity under elimination, ends as W; n^3/3 + n^3/3 flops)
//   product  k_spd_n    N = W M, K = M + M^T with M lower triangular   (n^3/3)
//   product  k_spd_k    K~ = N W^T + W N^T, the lower tiles mirrored  (2n^3/3)
// W also gives tr S^-1 = |W|^2, which bounds the smallest metric eigenvalue (no second
// factorisation of S - thr in the common case), and takes right-hand sides by products.
// Order 2744 (with the library's two factorisations, triangular solves and rank-2k
// updates before): 90 -> 36 ms.
#include <algorithm>
#include <cstring>

#include "spd.cuh"

namespace nvpt {
namespace s2 {
namespace {

constexpr int B = 64;    // block
constexpr int KS = 16;   // slab of a tile product
constexpr int LS = B + 2;
constexpr int TP = 256;

struct Slab {
    double a[KS][LS], b[KS][LS];
};

// acc += A B^T (BT: B [64][ldb], k along the rows) or A B (B [K][ldb]) for the 16 R x K
// tile A [16 R][lda]; K a multiple of KS.  Thread (ty, tx) holds rows {2ty, 2ty+1} (R = 4:
// and {32+2ty, 33+2ty}) and columns {2tx, 2tx+1, 32+2tx, 33+2tx}; the next slab's loads are
// issued before the FMAs.
template <bool BT, int R>
__device__ __forceinline__ void tile(double (&acc)[R][4], const double *A, long long lda, const double *Bm, long long ldb,
                                     int K, Slab &s) {
    const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
    const bool la = R == 4 || tid < 128;
    const double *pa = A + (la ? tid >> 2 : 0) * lda + (tid & 3) * 4;
    const double *pb = BT ? Bm + (tid >> 2) * ldb + (tid & 3) * 4 : Bm + (long long)(tid >> 4) * ldb + (tid & 15) * 4;
    double2 ra0, ra1, rb0, rb1;
    auto fetch = [&]() {
        ra0 = *reinterpret_cast<const double2 *>(pa);
        ra1 = *reinterpret_cast<const double2 *>(pa + 2);
        rb0 = *reinterpret_cast<const double2 *>(pb);
        rb1 = *reinterpret_cast<const double2 *>(pb + 2);
        pa += KS;
        pb += BT ? KS : KS * ldb;
    };
    fetch();
    for (int k0 = 0; k0 < K; k0 += KS) {
        __syncthreads();
        {
            const int r = tid >> 2, k = (tid & 3) * 4;
            if (la) {
                s.a[k][r] = ra0.x; s.a[k + 1][r] = ra0.y; s.a[k + 2][r] = ra1.x; s.a[k + 3][r] = ra1.y;
            }
            if (BT) {
                s.b[k][r] = rb0.x; s.b[k + 1][r] = rb0.y; s.b[k + 2][r] = rb1.x; s.b[k + 3][r] = rb1.y;
            } else {
                *reinterpret_cast<double2 *>(&s.b[tid >> 4][(tid & 15) * 4]) = rb0;
                *reinterpret_cast<double2 *>(&s.b[tid >> 4][(tid & 15) * 4 + 2]) = rb1;
            }
        }
        __syncthreads();
        if (k0 + KS < K) fetch();
#pragma unroll
        for (int k = 0; k < KS; ++k) {
            const double2 a0 = *reinterpret_cast<const double2 *>(&s.a[k][2 * ty]);
            const double2 a1 = R == 4 ? *reinterpret_cast<const double2 *>(&s.a[k][32 + 2 * ty]) : a0;
            const double2 b0 = *reinterpret_cast<const double2 *>(&s.b[k][2 * tx]);
            const double2 b1 = *reinterpret_cast<const double2 *>(&s.b[k][32 + 2 * tx]);
            const double a[4] = {a0.x, a0.y, a1.x, a1.y}, b[4] = {b0.x, b0.y, b1.x, b1.y};
#pragma unroll
            for (int p = 0; p < R; ++p)
#pragma unroll
                for (int q = 0; q < 4; ++q) acc[p][q] = fma(a[p], b[q], acc[p][q]);
        }
    }
}

__device__ __forceinline__ int own(int t, int p) { return (p >> 1) * 32 + 2 * t + (p & 1); }

// row r and position in it of the triangle's element x (row r has r + 1 of them)
__device__ __forceinline__ void triangle(int x, int &r, int &at) {
    r = (int)((sqrtf(8.0f * x + 1.0f) - 1.0f) * 0.5f);
    while ((r + 1) * (r + 2) / 2 <= x) ++r;
    while (r * (r + 1) / 2 > x) --r;
    at = x - r * (r + 1) / 2;
}

// W11 = L11^-1 of the 64 x 64 block D, live rows of it (identity below): in place, the
// columns already eliminated hold the inverse of the unit-lower factor, the others the
// reduced block, so that a column is one FMA for each element of the rows below,
//   M[i][j] -= m_i src[j],  m_i = M[i][c] / M[c][c],  src = (M[c][j < c], 1, M[j > c][c]).
// Warp 0 runs a column ahead (its entries, reciprocal and multipliers), so the division
// and its chain are hidden behind the other warps' rows and a column is one barrier;
// the square roots come last, all rows at once.  *bad is raised on a pivot that is not
// positive.  A whole block: 125 us (a square root, two barriers and two kinds of
// element a column) -> 63 us.
struct Diag {
    double m[B][B + 1], col[2][B], mul[2][B], d[B];
};
__device__ void factor_block(Diag &s, double *W, long long ld, int live, int *bad) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    // warp 0: column c's entries v0, v1 (rows lane, 32 + lane), their multipliers
    auto column = [&](int c, double v0, double v1) {
        const int b = c & 1;
        double d = __shfl_sync(0xffffffffu, c < 32 ? v0 : v1, c & 31);
        if (!(d > 0.0)) {
            if (lane == 0) atomicExch(bad, 1);
            d = 1.0;
        }
        const double inv = 1.0 / d;
        s.col[b][lane] = v0;
        s.col[b][32 + lane] = v1;
        s.mul[b][lane] = v0 * inv;
        s.mul[b][32 + lane] = v1 * inv;
        if (lane == 0) s.d[c] = d;
    };
    __syncthreads();
    if (warp == 0) column(0, s.m[lane][0], s.m[32 + lane][0]);
    __syncthreads();
    for (int c = 0; c < live; ++c) {
        const int b = c & 1;
        if (warp == 0) {
            if (c + 1 < live) {
                const double x = s.col[b][c + 1];
                double v0 = 0.0, v1 = 0.0;
                if (lane > c) v0 = fma(-s.mul[b][lane], x, s.m[lane][c + 1]);
                if (32 + lane > c) v1 = fma(-s.mul[b][32 + lane], x, s.m[32 + lane][c + 1]);
                column(c + 1, v0, v1);
            }
        } else {
            // warp 0 reads column c + 1 as it was: it is not written here, the next column's
            // entries are in col
            const double s0 = lane < c ? s.m[c][lane] : lane == c ? 1.0 : s.col[b][lane];
            const double s1 = 32 + lane < c ? s.m[c][32 + lane] : 32 + lane == c ? 1.0 : s.col[b][32 + lane];
            for (int i = c + warp; i < live; i += TP / 32 - 1) {
                const double f = -s.mul[b][i];
                if (lane <= i && lane != c + 1) s.m[i][lane] = fma(f, s0, lane == c ? 0.0 : s.m[i][lane]);
                if (i >= 32 && 32 + lane <= i && 32 + lane != c + 1)
                    s.m[i][32 + lane] = fma(f, s1, 32 + lane == c ? 0.0 : s.m[i][32 + lane]);
            }
        }
        __syncthreads();
    }
    if (tid < B) s.d[tid] = tid < live ? 1.0 / sqrt(s.d[tid]) : 1.0;
    __syncthreads();
    for (int e = tid; e < B * B; e += TP) {
        const int i = e / B, j = e % B;
        W[i * ld + j] = i == j ? s.d[i] : j < i && i < live ? s.m[i][j] * s.d[i] : 0.0;
    }
}

// L (lower) <- S, W <- 0, padding as in the identity; block 0: W11 of the first diagonal
// block, while the others copy.
__global__ void __launch_bounds__(TP) k_spd_load(const double *__restrict__ S, int n, long long ld, double *L, double *W,
                                                 int *bad) {
    extern __shared__ __align__(16) unsigned char smem[];
    auto at = [&](int i, int j) { return j < n && i < n ? S[(long long)j * n + i] : i == j ? 1.0 : 0.0; };
    if (blockIdx.x == 0) {
        Diag &s = *reinterpret_cast<Diag *>(smem);
        for (int e = threadIdx.x; e < B * B; e += TP) s.m[e % B][e / B] = e / B <= e % B ? at(e % B, e / B) : 0.0;
        factor_block(s, W, ld, min(B, n), bad);
        return;
    }
    const long long t = (long long)(blockIdx.x - 1) * TP + threadIdx.x;
    if (t >= ld * ld) return;
    const int j = (int)(t / ld), i = (int)(t % ld);  // i along the rows of S: its upper triangle is read in order
    if (i >= B || j >= B) W[t] = 0.0;
    if (j <= i) L[i * ld + j] = at(i, j);
}

// M (lower, half the diagonal, zeros above) of K = M + M^T.
__global__ void k_spd_half(const double *__restrict__ K, int n, long long ld, double *M) {
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= ld * ld) return;
    const int j = (int)(t / ld), i = (int)(t % ld);
    const double v = j < n && i < n && j <= i ? K[(long long)j * n + i] : 0.0;
    M[i * ld + j] = i == j ? 0.5 * v : v;
}

// 16 rows of L21 = A21 W11^T, or 16 columns of W[k, :] = W11 R[k, :], a CTA (in place).
__global__ void __launch_bounds__(TP) k_spd_panel(double *L, double *W, long long ld, int k, int nb, const int *bad) {
    __shared__ double w[B][B + 1], x[16][B + 1];
    if (*bad) return;
    const int tid = threadIdx.x, below = 4 * (nb - 1 - k);
    const double *W11 = W + (long long)k * B * ld + k * B;
    const bool rows = (int)blockIdx.x < below;
    double *P = rows ? L + ((long long)(k + 1) * B + 16 * blockIdx.x) * ld + k * B
                     : W + (long long)k * B * ld + 16 * ((int)blockIdx.x - below);
    for (int e = tid; e < B * B; e += TP) w[e / B][e % B] = W11[(e / B) * ld + e % B];
    for (int e = tid; e < 16 * B; e += TP) {
        if (rows) x[e / B][e % B] = P[(e / B) * ld + e % B];
        else x[e % 16][e / 16] = P[(e / 16) * ld + e % 16];
    }
    __syncthreads();
    // out[r][c] = sum_q x[r][q] w[c][q], the same for both
    const int r = tid >> 4, c0 = tid & 15;
    double acc[4] = {};
#pragma unroll 8
    for (int q = 0; q < B; ++q) {
        const double xv = x[r][q];
#pragma unroll
        for (int p = 0; p < 4; ++p) acc[p] = fma(xv, w[c0 + 16 * p][q], acc[p]);
    }
    __syncthreads();
#pragma unroll
    for (int p = 0; p < 4; ++p) x[r][c0 + 16 * p] = acc[p];
    __syncthreads();
    for (int e = tid; e < 16 * B; e += TP) {
        if (rows) P[(e / B) * ld + e % B] = x[e / B][e % B];
        else P[(e / 16) * ld + e % 16] = x[e % 16][e / 16];
    }
}

// Block 0: the next diagonal block, which is then factored while the other tiles run;
// then the rest of A22's lower tiles and the tiles of R below row k, a half (32 rows) a
// block, so that the last wave leaves less of the chip idle (order 2744, all steps: 15.9 ->
// 13.3 ms).
__global__ void __launch_bounds__(TP) k_spd_step(double *L, double *W, long long ld, int k, int nb, int n, int *bad) {
    extern __shared__ __align__(16) unsigned char smem[];
    if (__syncthreads_or(*(volatile int *)bad)) return;  // W is not used then
    const int t = nb - 1 - k, tri = t * (t + 1) / 2, tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
    Slab &s = *reinterpret_cast<Slab *>(smem);
    if (blockIdx.x == 0) {
        const double *P = L + (long long)(k + 1) * B * ld + k * B, *C = P + B;
        double acc[4][4] = {};
        tile<true, 4>(acc, P, ld, P, ld, B, s);
        __syncthreads();
        Diag &d = *reinterpret_cast<Diag *>(smem);
#pragma unroll
        for (int p = 0; p < 4; ++p)
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const int a = own(ty, p), b = own(tx, q);
                d.m[a][b] = b <= a ? C[a * ld + b] - acc[p][q] : 0.0;
            }
        factor_block(d, W + (long long)(k + 1) * B * ld + (k + 1) * B, ld, min(B, n - (k + 1) * B), bad);
        return;
    }
    const int x = ((int)blockIdx.x + 1) / 2, half = ((int)blockIdx.x + 1) % 2 * 32;  // tile x >= 1
    double acc[2][4] = {};
    double *C;
    int i, j;
    if (x < tri) {
        triangle(x, i, j);
        i += k + 1;
        j += k + 1;
        tile<true, 2>(acc, L + ((long long)i * B + half) * ld + k * B, ld, L + (long long)j * B * ld + k * B, ld, B, s);
        C = L + ((long long)i * B + half) * ld + j * B;
    } else {
        i = k + 1 + (x - tri) / (k + 1);
        j = (x - tri) % (k + 1);
        tile<false, 2>(acc, L + ((long long)i * B + half) * ld + k * B, ld, W + (long long)k * B * ld + j * B, ld, B, s);
        C = W + ((long long)i * B + half) * ld + j * B;
    }
#pragma unroll
    for (int p = 0; p < 2; ++p)
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            double2 *c2 = reinterpret_cast<double2 *>(C + (2 * ty + p) * ld + 32 * q + 2 * tx);
            double2 v = *c2;
            v.x -= acc[p][2 * q];
            v.y -= acc[p][2 * q + 1];
            *c2 = v;
        }
}

// out[0] += |row i of W|^2, out[2] = max(out[2], S_ii), a row a block.
__global__ void __launch_bounds__(TP) k_spd_norm(const double *__restrict__ W, const double *__restrict__ S, int n,
                                                 long long ld, double *out) {
    __shared__ double red[TP / 32];
    double v = 0.0;
    const int i = blockIdx.x;
    for (int j = threadIdx.x; j <= i; j += TP) {
        const double w = W[i * ld + j];
        v = fma(w, w, v);
    }
    for (int o = 16; o; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < TP / 32; ++w) v += red[w];
        atomicAdd(out, v);
        const double d = S[(long long)i * n + i];  // magnitudes order like their bits
        if (d > 0.0) atomicMax((unsigned long long *)(out + 2), (unsigned long long)__double_as_longlong(d));
    }
}

// N = W M: tile (i, j) is the sum over the blocks j .. i, a half (32 rows) a block, the
// longest first.
__global__ void __launch_bounds__(TP) k_spd_n(const double *__restrict__ W, const double *__restrict__ M, long long ld,
                                              int nb, int n, double *N) {
    __shared__ __align__(16) Slab s;
    int r, j;
    triangle(blockIdx.x / 2, r, j);
    const int i = j + nb - 1 - r, tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
    const long long ro = ((long long)i * B + blockIdx.x % 2 * 32) * ld + j * B;
    double acc[2][4] = {};
    tile<false, 2>(acc, W + ro, ld, M + (long long)j * B * ld + j * B, ld,
                   min((i - j + 1) * B, (n + KS - 1) / KS * KS - j * B), s);
    double *C = N + ro;
#pragma unroll
    for (int p = 0; p < 2; ++p)
#pragma unroll
        for (int q = 0; q < 2; ++q)
            *reinterpret_cast<double2 *>(C + (2 * ty + p) * ld + 32 * q + 2 * tx) = make_double2(acc[p][2 * q], acc[p][2 * q + 1]);
}

// K~ = N W^T + W N^T: tile (i, j <= i) sums over the blocks 0 .. j, a half (32 rows) a block,
// the longest first (order 2744 13.2 -> 13.0 ms; order 1000 1.33 ms, where the longest whole
// tile is 32 block products of 67 us).
__global__ void __launch_bounds__(TP) k_spd_k(const double *__restrict__ W, const double *__restrict__ N, long long ld,
                                              int nb, int n, double *out) {
    __shared__ __align__(16) Slab s;
    int r, x;
    triangle(blockIdx.x / 2, r, x);
    const int j = nb - 1 - r, i0 = (j + x) * B + blockIdx.x % 2 * 32, tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
    double acc[2][4] = {};
    const long long ro = i0 * ld, co = (long long)j * B * ld;
    const int K = min((j + 1) * B, (n + KS - 1) / KS * KS);  // M has only zeros in the padding
    tile<true, 2>(acc, N + ro, ld, W + co, ld, K, s);
    tile<true, 2>(acc, W + ro, ld, N + co, ld, K, s);
#pragma unroll
    for (int p = 0; p < 2; ++p)
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const int a = i0 + 2 * ty + p, b = j * B + own(tx, q);
            if (a < n && b <= a) {
                out[(long long)a * n + b] = acc[p][q];
                out[(long long)b * n + a] = acc[p][q];
            }
        }
}

// A step of at most this many blocks an SM is as long as its first one (update and
// factorisation of the next diagonal block), which is slowed by a block beside it on its SM:
// these steps ask for so much shared memory that none is (order 512 165 -> 127 us, order 1000
// 192 -> 146).
constexpr int kStepAlone = 3;
constexpr size_t kAloneSmem = 120 * 1024;

unsigned blocks(long long count) { return (unsigned)((count + TP - 1) / TP); }

}  // namespace

void spd_inverse_factor_async(Ctx &c, const double *S, long long n, double *W, double *stat, bool trace) {
    const long long ld = spd_ld(n);
    const int nb = (int)(ld / B);
    T L = alloc(c, {ld, ld}, false);
    int *bad = (int *)(stat + 1);
    raise_dynamic_smem((const void *)k_spd_load);
    raise_dynamic_smem((const void *)k_spd_step);
    int sms = 0, dev = 0;
    ck(cudaGetDevice(&dev), "cudaGetDevice");
    ck(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev), "attr");
    k_spd_load<<<1 + blocks(ld * ld), TP, sizeof(Diag), c.st>>>(S, (int)n, ld, L.p, W, bad);
    for (int k = 0; k < nb; ++k) {
        const int t = nb - 1 - k;
        if (t + k) k_spd_panel<<<4 * (t + k), TP, 0, c.st>>>(L.p, W, ld, k, nb, bad);
        const int grid = 2 * (t * (t + 1) / 2 + t * (k + 1)) - 1;
        if (t)
            k_spd_step<<<grid, TP, grid <= kStepAlone * sms ? kAloneSmem : sizeof(Diag), c.st>>>(L.p, W, ld, k, nb, (int)n, bad);
    }
    if (trace) k_spd_norm<<<(unsigned)n, TP, 0, c.st>>>(W, S, (int)n, ld, stat);
    g_launches.fetch_add(2 * nb - 1 + (trace ? 1 : 0), std::memory_order_relaxed);
    ck(cudaGetLastError(), "inverse factor");
}

bool spd_failed(const double *stat_on_host) {
    int failed;
    memcpy(&failed, stat_on_host + 1, sizeof(int));
    return failed != 0;
}

bool spd_inverse_factor(Ctx &c, const double *S, long long n, double *W, double &inv_trace, double &top) {
    T stat = alloc(c, {3}, true);  // |W|^2, bad pivot, largest diagonal element
    spd_inverse_factor_async(c, S, n, W, stat.p, true);
    double h[3];
    ck(cudaMemcpyAsync(h, stat.p, sizeof(h), cudaMemcpyDeviceToHost, c.st), "status copy");
    ck(cudaStreamSynchronize(c.st), "inverse factor sync");
    inv_trace = h[0];
    top = h[2];
    return !spd_failed(h);
}

void spd_congruence(Ctx &c, const double *W, const double *K, long long n, double *out) {
    const long long ld = spd_ld(n);
    const int nb = (int)(ld / B);
    T M = alloc(c, {ld, ld}, false), N = alloc(c, {ld, ld}, false);
    k_spd_half<<<blocks(ld * ld), TP, 0, c.st>>>(K, (int)n, ld, M.p);
    k_spd_n<<<nb * (nb + 1), TP, 0, c.st>>>(W, M.p, ld, nb, (int)n, N.p);
    k_spd_k<<<nb * (nb + 1), TP, 0, c.st>>>(W, N.p, ld, nb, (int)n, out);
    g_launches.fetch_add(3, std::memory_order_relaxed);
    ck(cudaGetLastError(), "congruence");
}

}  // namespace s2
}  // namespace nvpt

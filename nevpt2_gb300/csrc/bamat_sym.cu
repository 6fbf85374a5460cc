// A-matrices of the (+-1') classes (src/koopro4QD.F90:3974-4104) from one n^9
// contraction.
//
// The reference's loop needs four contractions of the four-operator products
// with the active integrals.  For RDMs with their physical symmetries
//   Gamma_k[P1 .. Pk] invariant under permutations of the pairs P = (creator,
//   annihilator) and under exchange of all creators with all annihilators,
// and integrals with (ij|kl) = (ji|kl) = (kl|ij), the Gamma4 part of each is
// the same tensor with other arguments,
//   F[A,B;c,a] = sum_{d,f,e} Gamma4[A, B, (d,f), (e,c)] (df|ea),
// F is symmetric under A <-> B, and (df| is symmetric, so n^9 flops take the
// place of 8 n^9.  What normal ordering adds is of order n^8 in Gamma3,
//   J[P1,P2;x,y]     = sum_{d,f} Gamma3[P1, P2, (d,f)] (df|xy)
//   Kx[P1,P2;x,y]    = sum_{d,e} Gamma3[P1, P2, (d,e)] (xd|ye)
//   Wca[p,(q,r),s;x,y] = sum_{f,e} Gamma3[(p,f), (q,r), (e,s)] (xf|ye)
//   Waa[p,(q,r),t;x,y] = sum_{f,e} Gamma3[(p,f), (q,r), (t,e)] (xf|ye)
// each with a two-fold symmetry in its row labels, and n^7 and below.  The
// one-electron operator g = f + K/2, K(x,y) = sum_z (xz|zy), goes into F, J and
// the two-operator J2 as
//   F += sum_d Gamma3[A, B, (d,c)] g(d,a),  J += Gamma2[P1, P2] g(x,y),
//   J2[p,q;x,y] = sum_{d,f} Gamma2[(p,q), (d,f)] (df|xy) + Gamma1[p,q] g(x,y)
// and appears nowhere else.  With A = (cp,ap), B = (bp,b), B' = (b,bp),
// P^T = (annihilator, creator):
//   amat  = F[A,B;c,a] - F[A^T,B^T;a,c] - F[A^T,(c,a);bp,b]
//         + Wca[cp,B,c;ap,a] + J[(cp,c),B;ap,a] - Waa[cp,B,a;ap,c] - Waa[bp,A,a;b,c]
//         - Waa[cp,(a,c),bp;ap,b] + Kronecker-delta terms (k_sym_out)
// and likewise atmat.  tests/test_bamat_sym.py evaluates these sums in numpy
// against the reference's loop.
//
// Which inputs take this route is decided on the device, for each state,
// without a host synchronisation: k_sym_unpack checks every symmetry that is
// used, to 2^-45 of the largest element of Gamma1 (and of the largest (ii|ii)
// for the integrals) -- the rounding of an RDM builder is below, anything else
// is not -- and raises the state's flag.  Every kernel here returns at once for
// a flagged state, and every kernel of the general route (bamat_gemm.cu)
// returns at once for the others.
#include <algorithm>

#include "bamat_sym.cuh"
#include "ozaki.cuh"
#include "sym_check.cuh"

namespace nvpt {
namespace {

constexpr int kSymXRows = 4;  // rows per warp of k_sym_x

// Packed rank (0-based) of a descending quadruple of 0-based indices.
__device__ __forceinline__ int rank4(const int v[4]) { return lindice4(v[0] + 1, v[1] + 1, v[2] + 1, v[3] + 1) - 1; }

// Sorts v descending; o[j] = original position of the j-th largest.
__device__ __forceinline__ void sort4(int v[4], int o[4]) {
    o[0] = 0; o[1] = 1; o[2] = 2; o[3] = 3;
#define NV_CE(i, j)                       \
    if (v[i] < v[j]) {                    \
        int t = v[i]; v[i] = v[j]; v[j] = t; \
        t = o[i]; o[i] = o[j]; o[j] = t;  \
    }
    NV_CE(0, 1) NV_CE(2, 3) NV_CE(0, 2) NV_CE(1, 3) NV_CE(1, 2)
#undef NV_CE
}

#define AT(i, j, k, l) atwo[(i) + (ll)n * ((j) + (ll)n * ((k) + (ll)n * (l)))]

// Integral operands, key table and the symmetry check of the integrals (n^4
// threads, once per call).
__global__ void __launch_bounds__(256) k_sym_ops(const double *atwo, const double *f, int ncore, int n, SymScratch S,
                                                 int M, int *flag) {
    const ll t = (ll)blockIdx.x * blockDim.x + threadIdx.x;
    const ll n2 = (ll)n * n, n4 = n2 * n2;
    if (t >= n4) return;
    const int l = (int)(t % n), k = (int)((t / n) % n), j = (int)((t / n2) % n), i = (int)(t / (n2 * n));
    const double v = AT(i, j, k, l);
    if (integral_asymmetric(atwo, n, i, j, k, l))
        for (int s = 0; s < M; ++s) flag[s] = 1;
    const int np = n * (n + 1) / 2;
    if (i >= j && j >= k && k >= l) {
        const int key[4] = {i, j, k, l};
        S.key[rank4(key)] = i | j << 4 | k << 8 | l << 12;
    }
    if (i >= j) S.Bf[((ll)k * np + pidx(i, j)) * n + l] = v;  // [(e, df), a] = (df|ea)
    S.I4[((ll)j * n + l) * n2 + (ll)i * n + k] = v;           // [(f, e), (x, y)] = (xf|ye)
    if (k >= l) S.IJ[((ll)j * n + i) * np + pidx(k, l)] = v;  // [(f, d), (x y)] = (df|xy)
    if (t < n2) {                                             // (x, y) = (k, l)
        double kk = 0.0;
        for (int z = 0; z < n; ++z) kk += AT(k, z, z, l);
        const double g = f[tri_index(k + 1 + ncore, l + 1 + ncore) - 1] + 0.5 * kk;
        S.g[t] = g;
        S.Bf[(ll)n * np * n + t] = g;  // the last K chunk of F
        if (k >= l) S.IJ[n2 * np + pidx(k, l)] = g;
    }
}

// H[K][l1 + n l2 + n^2 l3 + n^3 l4] = Gamma4 with creators the key K and any
// annihilators: the transpose of the packed 4-RDM, completed over the
// annihilators of higher rank than K (where the packed form keeps the
// exchanged element).  Reads are coalesced along K, writes along l1.  The
// blocks from nub on check Gamma1..3.  Bound by HBM (16 W n^4 bytes) and by the
// gathers of the completed half; n = 16: 3.0 ms.
__global__ void __launch_bounds__(256) k_sym_unpack(Rdm r, int s, const int *key, unsigned nub, double *H, int *flag) {
    const int n = r.n;
    const ll n2 = (ll)n * n, n3 = n2 * n, n4 = n2 * n2, W = r.W;
    bool raised;
    const double tol = rdm_tolerance(r, s, flag, raised);
    if (raised) return;  // the state's H is not used
    if (blockIdx.x >= nub) {
        const ll t = (ll)(blockIdx.x - nub) * blockDim.x + threadIdx.x;
        if (t < n3 * n3 && rdm_asymmetric(r, s, t, tol)) flag[s] = 1;
        return;
    }
    bool bad = false;
    auto differ = [tol](double x, double y) { return sym_differ(x, y, tol); };
    __shared__ double tile[32][33];
    const double *ro4 = r.ro4 + W * n4 * s;
    const unsigned kb = (unsigned)((W + 31) / 32);
    const ll K0 = (ll)(blockIdx.x % kb) * 32, L0 = (ll)(blockIdx.x / kb) * 32;
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
    const ll K = K0 + tx;
    const int pk = K < W ? key[K] : 0;
    const int k[4] = {pk & 15, pk >> 4 & 15, pk >> 8 & 15, pk >> 12 & 15};
    const ll pw[4] = {1, n, n2, n3};
    for (int y = ty; y < 32; y += 8) {
        const ll L = L0 + y;
        double v = 0.0;
        if (L < n4 && K < W) {
            const int l[4] = {(int)(L % n), (int)((L / n) % n), (int)((L / n2) % n), (int)(L / n3)};
            int q[4] = {l[0], l[1], l[2], l[3]}, o[4];
            sort4(q, o);
            const int rl = rank4(q);
            ll mate = 0;  // the annihilators of the exchanged element
#pragma unroll
            for (int j = 0; j < 4; ++j) mate += pw[j] * (o[j] == 0 ? k[0] : o[j] == 1 ? k[1] : o[j] == 2 ? k[2] : k[3]);
            if (rl > K) {
                v = ro4[rl + W * mate];
            } else {
                v = ro4[K + W * L];
                if (rl == K) bad = bad || differ(v, ro4[K + W * mate]);
#pragma unroll
                for (int j = 0; j < 3; ++j)  // equal creators: their annihilators may be exchanged
                    if (k[j] == k[j + 1] && l[j] < l[j + 1])
                        bad = bad || differ(v, ro4[K + W * (L + (l[j + 1] - l[j]) * (pw[j] - pw[j + 1]))]);
            }
        }
        tile[tx][y] = v;
    }
    if (bad) flag[s] = 1;
    __syncthreads();
    for (int y = ty; y < 32; y += 8)
        if (K0 + y < W && L0 + tx < n4) H[(K0 + y) * n4 + L0 + tx] = tile[y][tx];
}

// F for the creators (cp >= bp): rows ((cp,bp), ap, b, c), columns a,
//   F = sum_e sum_{d >= f} X_e[(b,c), df] (df|ea),
//   X_e[(b,c), df] = Gamma4[cp,bp,d,e; ap,b,f,c] + (d > f) Gamma4[cp,bp,f,e; ap,b,d,c]
// plus sum_d Gamma3[(cp,ap),(bp,b),(d,c)] g(d,a) as one more K chunk (e = n).
// One CTA owns (cp,bp), ap and bc values of b.  For each e it gathers X_e from
// H into shared memory -- the sort of the four creators is done once per d and
// turns the annihilators' offsets into four strides -- and multiplies: threads
// are (row group, column), RPT rows each.  Bound by the FP64 pipe (2 FMA per
// clock and SM): the gathers (two loads per n FMAs) run under the products of
// the SM's other CTAs.  n = 16: 36.3 ms for 3.9e10 flops, 1.07 TFLOP/s (the four
// products it replaced took 459 ms at 1.20); n = 11: 1.5 ms.
struct FBlock {  // what one CTA owns: (cp >= bp) = pair pr, ap, rows (b0 .. b0 + R / n, c)
    int pr, cp, bp, ap, b0, R;
};
__device__ __forceinline__ FBlock f_block(int n, int bc, int blk) {
    FBlock f;
    const int nchunk = (n + bc - 1) / bc;
    f.b0 = (blk % nchunk) * bc;
    blk /= nchunk;
    f.ap = blk % n;
    f.pr = blk / n;
    unpair(f.pr, f.cp, f.bp);
    f.R = min(bc, n - f.b0) * n;
    return f;
}
// X_e of the block into shared memory, X[row * ldx + k]: k = df for e < n, k = d
// (Gamma3) for e = n.  Starts and ends with all threads of the CTA together.
__device__ __forceinline__ void f_gather(const Rdm &r, int s, const FBlock &f, int e, const double *__restrict__ H,
                                         double *X, int ldx) {
    __shared__ ll s_base[16];
    __shared__ int s_w[16][3];
    const int n = r.n, n2 = n * n, n4 = n2 * n2, np = n * (n + 1) / 2, tid = threadIdx.x, R = f.R;
    if (e < n && tid < n) {
        int v[4] = {f.cp, f.bp, tid, e}, o[4], w[4], p = 1;
        sort4(v, o);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
#pragma unroll
            for (int i = 0; i < 4; ++i)
                if (o[j] == i) w[i] = p;
            p *= n;
        }
        s_base[tid] = (ll)rank4(v) * n4 + f.ap * w[0] + f.b0 * w[1];
        s_w[tid][0] = w[1];
        s_w[tid][1] = w[2];
        s_w[tid][2] = w[3];
    }
    __syncthreads();
    if (e == n) {  // Gamma3 with its annihilators exchanged, d the fastest index
        const double *d3 = r.d3 + s + (ll)r.M * (n * f.cp + n2 * f.bp + (ll)n4 * (f.ap + n * f.b0));
        for (int i = tid; i < R * n; i += 256) {
            const int row = i % R, d = i / R;
            X[row * ldx + d] = d3[(ll)r.M * (d + n2 * n * (row % n) + (ll)n4 * n * (row / n))];
        }
    } else {
        for (int i = tid; i < R * np; i += 256) {
            const int row = i % R, df = i / R;
            const int c = row % n, b = row / n;
            int d, g;
            unpair(df, d, g);
            double x = H[s_base[d] + b * s_w[d][0] + g * s_w[d][1] + c * s_w[d][2]];
            if (d != g) x += H[s_base[g] + b * s_w[g][0] + d * s_w[g][1] + c * s_w[g][2]];
            X[row * ldx + df] = x;
        }
    }
    __syncthreads();
}

template <int RPT>
__global__ void __launch_bounds__(256) k_sym_f(Rdm r, int s, int bc, const double *__restrict__ H,
                                               const double *__restrict__ Bf, double *__restrict__ F,
                                               const int *flag) {
    if (*flag) return;
    extern __shared__ double sm[];
    const int n = r.n, np = n * (n + 1) / 2, tid = threadIdx.x, ldx = np | 1;  // odd: no bank conflicts down a column
    const FBlock f = f_block(n, bc, blockIdx.x);
    double *X = sm, *B = sm + bc * n * ldx;
    const int groups = 256 / n, col = tid % n, grp = tid / n;
    double acc[RPT];
    int ro[RPT];
#pragma unroll
    for (int i = 0; i < RPT; ++i) {
        acc[i] = 0.0;
        ro[i] = min(grp + i * groups, f.R - 1) * ldx;
    }
    for (int e = 0; e <= n; ++e) {
        const int nk = e < n ? np : n;
        for (int i = tid; i < nk * n; i += 256) B[i] = Bf[(ll)e * np * n + i];
        f_gather(r, s, f, e, H, X, ldx);
        if (grp < groups) {
#pragma unroll 4
            for (int k = 0; k < nk; ++k) {
                const double y = B[k * n + col];
#pragma unroll
                for (int i = 0; i < RPT; ++i) acc[i] = fma(X[ro[i] + k], y, acc[i]);
            }
        }
        __syncthreads();
    }
    if (grp >= groups) return;
#pragma unroll
    for (int i = 0; i < RPT; ++i) {
        const int row = grp + i * groups;
        if (row < f.R) F[(((ll)f.pr * n + f.ap) * n * n + f.b0 * n + row) * n + col] = acc[i];
    }
}

// The operand of F as rows in memory, for the digit product: rows ((cp,bp) from
// pr0, ap, b, c), K = n (np + 1) columns (e, df) and d, with each row's largest
// magnitude.  A CTA gathers as above; its warps write whole rows (n = 14: 4.2 ms
// for 3.4 GB, bound by the gathers).
__global__ void __launch_bounds__(256) k_sym_x(Rdm r, int s, int bc, int pr0, const double *__restrict__ H,
                                               double *__restrict__ X, unsigned long long *__restrict__ rmax,
                                               const int *flag) {
    if (*flag) return;
    extern __shared__ double sm[];
    const int n = r.n, np = n * (n + 1) / 2, ldx = np | 1, K = n * (np + 1);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    FBlock f = f_block(n, bc, blockIdx.x + pr0 * n * ((n + bc - 1) / bc));
    const ll row0 = ((ll)(f.pr - pr0) * n + f.ap) * n * n + f.b0 * n;
    double mx[kSymXRows];
#pragma unroll
    for (int i = 0; i < kSymXRows; ++i) mx[i] = 0.0;
    for (int e = 0; e <= n; ++e) {
        const int nk = e < n ? np : n;
        f_gather(r, s, f, e, H, sm, ldx);
#pragma unroll
        for (int i = 0; i < kSymXRows; ++i) {
            const int row = warp + 8 * i;
            if (row >= f.R) break;
            for (int k = lane; k < nk; k += 32) {
                const double x = sm[row * ldx + k];
                mx[i] = fmax(mx[i], fabs(x));
                X[(row0 + row) * K + e * np + k] = x;
            }
        }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < kSymXRows; ++i) {
        const int row = warp + 8 * i;
        if (row >= f.R) break;
        for (int o = 16; o; o >>= 1) mx[i] = fmax(mx[i], __shfl_xor_sync(0xffffffffu, mx[i], o));
        if (lane == 0) rmax[row0 + row] = (unsigned long long)__double_as_longlong(mx[i]);
    }
}

// The n^8 contractions, blockIdx.z: 0 Wca, 1 Waa, 2 Kx, 3 J.  Rows ((p >= p'),
// q, r): Wca and Waa have p' their second creator (s or t) and (q,r) the free
// pair, Kx and J the pairs (p,q), (p',r).  The rows of Gamma3 are affine in the
// two summed indices, lo the one with stride M, so the tile loads need no
// intermediate matrix.  Bound by the FP64 pipe (n = 16: 10.5 ms for 1.23e10 flops, 1.17
// TFLOP/s).  32 x 32 tiles, 2 x 2 per thread: a tile of 64 is four times as long and leaves
// SMs idle in the last wave and columns in the last tile; 32 / 64, us: n = 4 9 / 22, n = 8
// 70 / 73, n = 9 175 / 298, n = 12 1230 / 1590, n = 14 4420 / 4990, n = 16 10540 / 10960.
constexpr int kN8 = 32, kN8K = 16;
// Kx and J keep their value under the exchange of creators and annihilators (Kx with x, y
// exchanged), so their rows are pairs of pairs: (p >= p') of index ua >= ub of (q,r), and q,
// r in either order, about half of the others' np n^2.
__host__ __device__ __forceinline__ ll n8_rows(int n, int kind) {
    const ll np = n * (n + 1) / 2;
    return kind < 2 ? np * n * n : np * (np + 1);
}
__host__ __device__ __forceinline__ ll n8_at(int n, int kind) {  // first element of a kind's results, and rows x n^2
    const ll n2 = (ll)n * n;
    return (kind < 3 ? kind * n8_rows(n, 0) : 2 * n8_rows(n, 0) + n8_rows(n, 2)) * n2;
}
__device__ __forceinline__ void n8_labels(int n, int kind, ll row, int &p, int &p2, int &q1, int &q2) {
    if (kind < 2) {
        q2 = (int)(row % n);
        q1 = (int)((row / n) % n);
        unpair((int)(row / (n * n)), p, p2);
    } else {
        int ua, ub;
        unpair((int)(row >> 1), ua, ub);
        unpair(ua, p, p2);
        unpair(ub, q1, q2);
        if (row & 1) {
            const int t = q1;
            q1 = q2;
            q2 = t;
        }
    }
}
// Offset of a row of Gamma3 (in units of M) and the stride of its slow summed index.
__device__ __forceinline__ ll n8_row(int n, int kind, ll row) {
    const ll n1 = n, n2 = n1 * n, n3 = n2 * n, n4 = n2 * n2, n5 = n4 * n;
    int p, p2, q1, q2;
    n8_labels(n, kind, row, p, p2, q1, q2);
    if (kind == 0) return n1 * p + n2 * q1 + n3 * p2 + n5 * q2;       // (e,s), (p,f), (q,r)
    if (kind == 1) return n2 * q2 + n3 * p2 + n4 * p + n5 * q1;       // (e,t), (f,p), (r,q): exchanged
    if (kind == 2) return n1 * q1 + n2 * q2 + n4 * p + n5 * p2;       // (e,d), (q,p), (r,p'): exchanged
    return n1 * p + n2 * p2 + n4 * q1 + n5 * q2;                      // (d,f), (p,q), (p',r)
}
__device__ __forceinline__ ll n8_hi(int n, int kind) {
    return kind == 0 ? (ll)n * n * n * n : kind == 1 ? (ll)n : (ll)n * n * n;
}
// Gamma2 factor of a row of J
__device__ __forceinline__ double n8_pair2(const Rdm &r, int s, ll row) {
    const int n = r.n;
    int p, p2, q1, q2;
    n8_labels(n, 3, row, p, p2, q1, q2);
    return r.d2[s + (ll)r.M * (p + n * (p2 + n * (q1 + n * q2)))];
}
__global__ void __launch_bounds__(256) k_sym_n8(Rdm r, int s, const double *__restrict__ I4,
                                                const double *__restrict__ IJ, double *out, const int *flag) {
    if (*flag) return;
    constexpr int P = kN8 / 16;  // rows and columns of a thread
    __shared__ double As[kN8K][kN8 + 1], Bs[kN8K][kN8];
    const int n = r.n, np = n * (n + 1) / 2, kind = blockIdx.z;
    const ll M = r.M, n2 = (ll)n * n, rows = n8_rows(n, kind);
    const int N = kind == 3 ? np : (int)n2;
    const int c0 = blockIdx.y * kN8;
    const ll r0 = (ll)blockIdx.x * kN8;
    if (c0 >= N || r0 >= rows) return;
    const double *Bm = kind == 3 ? IJ : I4;
    double *C = out + n8_at(n, kind);
    const ll hi = M * n8_hi(n, kind);
    const int tid = threadIdx.x, lk = tid & 15, lr = tid >> 4;
    const double *base[P];
#pragma unroll
    for (int i = 0; i < P; ++i) {
        const ll row = min(r0 + lr + 16 * i, rows - 1);
        base[i] = r.d3 + s + M * n8_row(n, kind, row);
    }
    double acc[P][P] = {};
    const int tc = (tid & 15) * P, tr = (tid >> 4) * P;
    const int K = (int)n2;
    for (int k0 = 0; k0 < K; k0 += kN8K) {
        const int k = k0 + lk;
        const ll ko = (k / n) * hi + (k % n) * M;
#pragma unroll
        for (int i = 0; i < P; ++i) As[lk][lr + 16 * i] = k < K ? base[i][ko] : 0.0;
#pragma unroll
        for (int i = 0; i < P; ++i) {
            const int kk = tid / kN8 + 256 / kN8 * i, c = tid % kN8;
            Bs[kk][c] = (k0 + kk < K && c0 + c < N) ? Bm[(ll)(k0 + kk) * N + c0 + c] : 0.0;
        }
        __syncthreads();
#pragma unroll
        for (int kk = 0; kk < kN8K; ++kk) {
            double a[P], b[P];
#pragma unroll
            for (int i = 0; i < P; ++i) {
                a[i] = As[kk][tr + i];
                b[i] = Bs[kk][tc + i];
            }
#pragma unroll
            for (int i = 0; i < P; ++i)
#pragma unroll
                for (int j = 0; j < P; ++j) acc[i][j] = fma(a[i], b[j], acc[i][j]);
        }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < P; ++i) {
        const ll row = r0 + tr + i;
        if (row >= rows) break;
        const double w = kind == 3 ? n8_pair2(r, s, row) : 0.0;  // J += Gamma2[(p,q), (p',r)] g(x,y)
#pragma unroll
        for (int j = 0; j < P; ++j) {
            const int col = c0 + tc + j;
            if (col >= N) break;
            double v = acc[i][j];
            if (kind == 3) v = fma(w, IJ[n2 * np + col], v);
            C[row * N + col] = v;
        }
    }
}

// The operands of the n^8 contractions as rows in memory, for the digit
// products: kinds 0-2 [row][n^2], J [row][n^2 + 1] with its Gamma2 factor last.
__global__ void __launch_bounds__(256) k_sym_rows(Rdm r, int s, double *__restrict__ R, const int *flag) {
    if (*flag) return;
    const int n = r.n, kind = blockIdx.y, n2 = n * n, K = kind == 3 ? n2 + 1 : n2;
    const ll t = (ll)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= n8_rows(n, kind) * K) return;
    const ll row = t / K;
    const int k = (int)(t % K);
    R[n8_at(n, kind) + t] = k == n2 ? n8_pair2(r, s, row)
                                      : r.d3[s + (ll)r.M * (n8_row(n, kind, row) + (k / n) * n8_hi(n, kind) + k % n)];
}

// Accessors of the intermediates (0-based labels).
struct SymView {
    Rdm r;
    int s, n;
    ll n2, rows;  // rows of one n^8 block
    const double *F, *N8, *G1, *G3, *Q1, *JW, *J2, *Z, *atwo, *g, *T3;

    __device__ __forceinline__ double d1(int a, int b) const { return r.d1[s + (ll)r.M * (a + n * b)]; }
    __device__ __forceinline__ double d2(int a, int b, int c, int d) const {
        return r.d2[s + (ll)r.M * (a + n * (b + n * (c + n * d)))];
    }
    __device__ __forceinline__ double ai(int i, int j, int k, int l) const {
        return atwo[i + n * (j + n * (k + n * l))];
    }
    // F[(p,q), (p2,q2); c, a]
    __device__ __forceinline__ double f4(int p, int q, int p2, int q2, int c, int a) const {
        const ll row = p >= p2 ? (ll)(pidx(p, p2) * n + q) * n + q2 : (ll)(pidx(p2, p) * n + q2) * n + q;
        return F[(row * n + c) * n + a];
    }
    __device__ __forceinline__ ll row3(int p, int p2, int q, int q2) const {
        return (ll)(pidx(p, p2) * n + q) * n + q2;
    }
    __device__ __forceinline__ double wca(int p, int q, int q2, int t, int x, int y) const {
        return p >= t ? N8[row3(p, t, q, q2) * n2 + x * n + y] : N8[row3(t, p, q2, q) * n2 + y * n + x];
    }
    __device__ __forceinline__ double waa(int p, int q, int q2, int t, int x, int y) const {
        const double *A = N8 + rows * n2;
        return p >= t ? A[row3(p, t, q, q2) * n2 + x * n + y] : A[row3(t, p, q, q2) * n2 + y * n + x];
    }
    // row of ((p,q), (p2,q2)) in Kx and J; tr: of its transpose
    __device__ __forceinline__ ll rowk(int p, int q, int p2, int q2, bool &tr) const {
        int ua = pmx(p, p2), ub = pmx(q, q2);
        tr = ua < ub;
        const bool flip = tr ? q < q2 : p < p2, less = tr ? p < p2 : q < q2;  // of the leading pair, of the other
        const int up = tr ? ub : ua, lo = tr ? ua : ub;
        return (ll)pidx(up, lo) * 2 + (flip != less ? 1 : 0);
    }
    __device__ __forceinline__ double kx(int p, int q, int p2, int q2, int x, int y) const {
        bool tr;
        const ll row = rowk(p, q, p2, q2, tr);
        return N8[n8_at(n, 2) + row * n2 + (tr ? y * n + x : x * n + y)];
    }
    __device__ __forceinline__ double jj(int p, int q, int p2, int q2, int x, int y) const {
        bool tr;
        const ll row = rowk(p, q, p2, q2, tr);
        return N8[n8_at(n, 3) + row * (n * (n + 1) / 2) + pmx(x, y)];
    }
    __device__ __forceinline__ double t3(int x1, int x2, int x3, int p, int q, int r) const {
        return T3[(((ll)(x1 * n + x2) * n + x3) * (n * (n + 1) / 2) + pmx(q, r)) * n + p];
    }
    __device__ __forceinline__ ll i4(int a, int b, int c, int d) const { return ((ll)(a * n + b) * n + c) * n + d; }
};

// T3[x1,x2,x3; (q r), p] = sum_d Gamma2[(x1,d),(x2,x3)] (pd|qr): every n^7 sum of the
// output is an element of it.  Rows (x1,x2,x3), columns (pair, p), K = n in one slab;
// 64 x 64 tiles, bound by the FP64 pipe (n^7/2 FMAs; n = 16: 243 us, n = 8: 13).
__global__ void __launch_bounds__(256) k_sym_t3(Rdm r, int s, const double *__restrict__ atwo, double *T3, const int *flag) {
    if (*flag) return;
    __shared__ double As[16][65], Bs[16][64];
    const int n = r.n, np = n * (n + 1) / 2, n3 = n * n * n, cols = np * n, tid = threadIdx.x;
    const int r0 = blockIdx.x * 64, c0 = blockIdx.y * 64;
    for (int e = tid; e < 64 * n; e += 256) {
        const int d = e % n, row = min(r0 + e / n, n3 - 1), x3 = row % n, x2 = (row / n) % n, x1 = row / (n * n);
        As[d][e / n] = r.d2[s + (ll)r.M * (d + n * (x3 + n * (x1 + n * x2)))];
    }
    for (int e = tid; e < 64 * n; e += 256) {
        const int d = e / 64, col = min(c0 + e % 64, cols - 1), p = col % n;
        int q, t;
        unpair(col / n, q, t);
        Bs[d][e % 64] = AT(p, d, q, t);
    }
    __syncthreads();
    const int tc = (tid & 15) * 4, tr = (tid >> 4) * 4;
    double acc[4][4] = {};
    for (int k = 0; k < n; ++k) {
        double a[4], b[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            a[i] = As[k][tr + i];
            b[i] = Bs[k][tc + i];
        }
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) acc[i][j] = fma(a[i], b[j], acc[i][j]);
    }
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j)
            if (r0 + tr + i < n3 && c0 + tc + j < cols) T3[(ll)(r0 + tr + i) * cols + c0 + tc + j] = acc[i][j];
}

// n^6 sums over two indices, kSmallLanes threads per n^4 element (a chain of n^2 steps and
// an idle chip at small n otherwise; n = 8: 32 -> 10 us, n = 16: 174 -> 156):
//   G1[p,q,c,a] = sum_e J[(p,q),(e,c);e,a]         G3[p,q,r,x] = sum_e J[(p,e),(q,r);x,e]
//   Q1[p,t,x,y] = sum Gamma2[(p,f),(t,e)] (xf|ye)  J2 as above
//   JW = J2 + sum Gamma2[(p,f),(e,q)] (xf|ey)      Z[p,c,q,b] = 2 J2 - sum Gamma2[(p,c),(e,f)] (qf|be)
constexpr int kSmallLanes = 4;
__global__ void __launch_bounds__(64) k_sym_small(SymView v, double *G1, double *G3, double *Q1, double *JW,
                                                  double *J2, double *Z, const int *flag) {
    if (*flag) return;
    const int n = v.n, e0 = threadIdx.x % kSmallLanes;
    const ll t = ((ll)blockIdx.x * blockDim.x + threadIdx.x) / kSmallLanes;
    const ll u = t < v.n2 * v.n2 ? t : 0;
    const int d = (int)(u % n), c = (int)((u / n) % n), b = (int)((u / v.n2) % n), a = (int)(u / (v.n2 * n));
    double g1 = 0.0, g3 = 0.0, q1 = 0.0, w2 = 0.0, j2 = e0 ? 0.0 : v.d1(a, b) * v.g[c * n + d], y2 = 0.0;
    for (int e = e0; e < n; e += kSmallLanes) {
        g1 += v.jj(a, b, e, c, e, d);
        g3 += v.jj(a, e, b, c, d, e);
#pragma unroll 4
        for (int f = 0; f < n; ++f) {
            const double x = v.ai(c, f, d, e);
            q1 = fma(v.d2(a, b, f, e), x, q1);
            w2 = fma(v.d2(a, e, f, b), x, w2);
            y2 = fma(v.d2(a, e, b, f), x, y2);
            j2 = fma(v.d2(a, e, b, f), v.ai(e, f, c, d), j2);
        }
    }
    auto sum = [](double x) {
        for (int o = kSmallLanes / 2; o; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
        return x;
    };
    g1 = sum(g1); g3 = sum(g3); q1 = sum(q1); w2 = sum(w2); j2 = sum(j2); y2 = sum(y2);
    if (e0 || t >= v.n2 * v.n2) return;
    G1[t] = g1; G3[t] = g3; Q1[t] = q1; JW[t] = j2 + w2; J2[t] = j2; Z[t] = 2.0 * j2 - y2;
}

// amat/atmat(s, ap,bp,cp,a,b,c), a thread an element, a fastest, then c, so that most
// gathers of F and the n^8 tensors (whose last indices are a, c or b) share sectors.
// Bound by the FP64 pipe (some 35 additions an element, with the Kronecker deltas more in
// most warps).  Blocks of 64 spread the small spaces over the SMs and cost the large ones
// nothing.  With the n^7 sums formed here (6 n FMAs an element) 27 / 63 / 5850 us at n =
// 4 / 8 / 16, now 8 / 33 / 1990 and k_sym_t3.
constexpr int kOutTb = 64;
__global__ void __launch_bounds__(kOutTb) k_sym_out(SymView v, double *amat, double *atmat, const int *flag) {
    if (*flag) return;
    const int n = v.n;
    const ll n5 = v.n2 * v.n2 * n;
    const ll t = (ll)blockIdx.x * kOutTb + threadIdx.x;
    if (t >= n5) return;
    ll x = t;
    const int a = (int)(x % n); x /= n;
    const int c = (int)(x % n); x /= n;
    const int b = (int)(x % n); x /= n;
    const int bp = (int)(x % n); x /= n;
    const int cp = (int)x, ap = blockIdx.y;
    const double d1 = v.d1(cp, c);
    double A = v.f4(cp, ap, bp, b, c, a) - v.f4(ap, cp, b, bp, a, c) - v.f4(ap, cp, c, a, bp, b);
    double T = v.f4(ap, cp, bp, b, a, c) - v.f4(cp, ap, b, bp, c, a) - v.f4(cp, ap, a, c, bp, b);
    A += v.wca(cp, bp, b, c, ap, a) + v.jj(cp, c, bp, b, ap, a) - v.waa(cp, bp, b, a, ap, c) -
         v.waa(bp, cp, ap, a, b, c) - v.waa(cp, a, c, bp, ap, b);
    T += v.waa(cp, b, bp, a, ap, c) + v.waa(b, cp, ap, a, bp, c) - v.waa(c, ap, cp, bp, a, b) -
         v.wca(cp, b, bp, c, ap, a) - v.wca(b, cp, ap, c, bp, a) - v.wca(cp, a, c, bp, ap, b);
    T += 2.0 * v.jj(cp, ap, a, c, b, bp) - v.jj(cp, c, b, bp, ap, a) - v.jj(cp, ap, b, c, bp, a) -
         v.jj(cp, bp, a, c, ap, b) - v.kx(cp, ap, a, c, b, bp);
    T += 2.0 * (v.t3(c, ap, cp, a, b, bp) + v.t3(cp, a, c, ap, b, bp)) - v.t3(c, ap, cp, b, bp, a) -
         v.t3(cp, a, c, bp, b, ap) - v.t3(cp, b, c, ap, bp, a) - v.t3(b, cp, c, bp, ap, a) -
         v.t3(c, bp, cp, a, ap, b) - v.t3(bp, c, cp, b, ap, a);
    T += d1 * (2.0 * v.ai(ap, a, b, bp) - v.ai(bp, a, b, ap));
    // Kronecker deltas
    auto q2 = [&]() {  // sum_e J2[cp,e;c,e]
        double q = 0.0;
        for (int e = 0; e < n; ++e) q += v.J2[v.i4(cp, e, c, e)];
        return q;
    };
    if (ap == bp) {
        A += v.G1[v.i4(cp, b, c, a)] - v.G1[v.i4(b, cp, a, c)] - v.G3[v.i4(cp, a, c, b)] - v.Q1[v.i4(cp, a, b, c)];
        if (a == b) A -= q2();
    }
    if (ap == a) {
        A -= v.G3[v.i4(cp, bp, b, c)] + v.G3[v.i4(bp, cp, c, b)] + v.Q1[v.i4(bp, cp, b, c)];
        T += v.G3[v.i4(cp, b, bp, c)] + v.Q1[v.i4(b, cp, bp, c)] - v.G1[v.i4(cp, c, bp, b)] + v.Z[v.i4(cp, c, bp, b)];
    }
    if (a == b) A -= v.G3[v.i4(bp, cp, ap, c)] + v.Q1[v.i4(cp, bp, ap, c)];
    if (ap == b) {
        T += v.G1[v.i4(bp, cp, a, c)] - v.G1[v.i4(cp, bp, c, a)] - v.JW[v.i4(cp, c, bp, a)] + v.Q1[v.i4(cp, a, bp, c)];
        if (bp == a) T += q2();
    }
    if (bp == a)
        T += v.G3[v.i4(b, cp, ap, c)] + v.Q1[v.i4(cp, b, ap, c)] - v.G1[v.i4(cp, ap, c, b)] - v.JW[v.i4(cp, c, ap, b)];
    if (b == bp) {
        T += 2.0 * (v.G1[v.i4(cp, ap, c, a)] + v.JW[v.i4(cp, c, ap, a)] - v.G3[v.i4(a, cp, ap, c)] -
                    v.Q1[v.i4(cp, a, ap, c)]);
        if (a == ap) T -= 2.0 * q2();
    }
    const ll o = v.s + (ll)v.r.M * (ap + n * (bp + n * (cp + n * (a + (ll)n * (b + n * c)))));
    amat[o] = A;
    atmat[o] = T;
}
#undef AT

// Values of b per CTA of k_sym_f and rows per thread: the split with the least
// idle row slots whose tile leaves two CTAs per SM (at most 72 KB of X).  Rows per
// thread: 2 at n = 10 and 12, 5 at n = 13, 4 at n = 14, 1 at the other sizes.
struct FShape {
    int bc = 1, rpt = 1;
};
FShape f_shape(int n) {
    const int np = n * (n + 1) / 2, groups = 256 / n;
    FShape best;
    double eff = 0.0;
    for (int bc = 1; bc <= n; ++bc) {
        const int R = bc * n, rpt = (R + groups - 1) / groups;
        if (rpt > kSymMaxRpt || (ll)R * (np | 1) * 8 > 72 * 1024) break;
        const int chunks = (n + bc - 1) / bc;
        const double e = (double)(n * n) / ((double)chunks * rpt * groups);
        if (e > eff * 1.02) {
            eff = e;
            best.bc = bc;
            best.rpt = rpt;
        }
    }
    return best;
}

using FKernel = void (*)(Rdm, int, int, const double *, const double *, double *, const int *);
FKernel f_kernel(int rpt) {
    switch (rpt) {
        case 1: return k_sym_f<1>;
        case 2: return k_sym_f<2>;
        case 4: return k_sym_f<4>;
        default: return k_sym_f<5>;
    }
}

}  // namespace

ll SymScratch::doubles(int n) {
    const ll n2 = (ll)n * n, n4 = n2 * n2, np = n * (n + 1) / 2;
    const ll W = (ll)n * (n + 1) * (n + 2) * (n + 3) / 24;
    return W * n4 + np * n4 + n8_at(n, 3) + n8_rows(n, 3) * np + 7 * n4 + 2 * np * n2 + np + 2 * n2 + W / 2 + 1;
}

SymScratch::SymScratch(int n, double *w) {
    const ll n2 = (ll)n * n, n4 = n2 * n2, np = n * (n + 1) / 2;
    const ll W = (ll)n * (n + 1) * (n + 2) * (n + 3) / 24;
    auto take = [&w](ll k) {
        double *p = w;
        w += k;
        return p;
    };
    H = take(W * n4);
    F = take(np * n4);
    N8 = take(n8_at(n, 3) + n8_rows(n, 3) * np);
    for (double **p : {&G1, &G3, &Q1, &JW, &J2, &Z}) *p = take(n4);
    Bf = take((np + 1) * n2);
    I4 = take(n4);
    IJ = take((n2 + 1) * np);
    g = take(n2);
    key = (int *)take(W / 2 + 1);
}

void launch_sym_ops(const double *atwo, const double *f, int ncore, int n, const SymScratch &S, int M, int *flag,
                    cudaStream_t st) {
    const ll n4 = (ll)n * n * n * n;
    k_sym_ops<<<(unsigned)((n4 + 255) / 256), 256, 0, st>>>(atwo, f, ncore, n, S, M, flag);
    g_launches.fetch_add(1, std::memory_order_relaxed);
}

namespace {
void sym_finish(const SymView &v, const SymScratch &S, double *amat, double *atmat, const int *fl, cudaStream_t st) {
    const ll n = v.n, n4 = n * n * n * n;
    k_sym_small<<<(unsigned)((kSmallLanes * n4 + 63) / 64), 64, 0, st>>>(v, S.G1, S.G3, S.Q1, S.JW, S.J2, S.Z, fl);
    const dim3 gt((unsigned)((n * n * n + 63) / 64), (unsigned)((n * n * (n + 1) / 2 + 63) / 64));
    k_sym_t3<<<gt, 256, 0, st>>>(v.r, v.s, v.atwo, S.H, fl);
    const dim3 go((unsigned)((n4 * n + kOutTb - 1) / kOutTb), (unsigned)n);
    k_sym_out<<<go, kOutTb, 0, st>>>(v, amat, atmat, fl);
    g_launches.fetch_add(3, std::memory_order_relaxed);
}
void sym_unpack(const Rdm &r, int s, const SymScratch &S, int *flag, cudaStream_t st) {
    const ll n = r.n, n4 = n * n * n * n;
    const ll ub = ((r.W + 31) / 32) * ((n4 + 31) / 32), cb = (n4 * n * n + 255) / 256;
    k_sym_unpack<<<(unsigned)(ub + cb), 256, 0, st>>>(r, s, S.key, (unsigned)ub, S.H, flag);
    g_launches.fetch_add(1, std::memory_order_relaxed);
}
SymView sym_view(const Rdm &r, int s, const double *atwo, const SymScratch &S) {
    const ll n2 = (ll)r.n * r.n;
    return SymView{r, s, r.n, n2, r.n * (r.n + 1) / 2 * n2, S.F, S.N8, S.G1, S.G3, S.Q1, S.JW, S.J2, S.Z, atwo, S.g, S.H};
}
}  // namespace

int launch_sym_state(const Rdm &r, int s, const double *atwo, const SymScratch &S, double *amat, double *atmat,
                     int *flag, cudaStream_t st) {
    const int n = r.n, np = n * (n + 1) / 2, *fl = flag + s;
    const ll n2 = (ll)n * n, rows = std::max(n8_rows(n, 0), n8_rows(n, 2));
    sym_unpack(r, s, S, flag, st);
    const dim3 g8((unsigned)((rows + kN8 - 1) / kN8), (unsigned)((n2 + kN8 - 1) / kN8), 4);
    k_sym_n8<<<g8, 256, 0, st>>>(r, s, S.I4, S.IJ, S.N8, fl);
    const FShape fs = f_shape(n);
    const FKernel fk = f_kernel(fs.rpt);
    const int smem = (fs.bc * n * (np | 1) + np * n) * (int)sizeof(double);
    if (smem > 48 * 1024 &&
        cudaFuncSetAttribute((const void *)fk, cudaFuncAttributeMaxDynamicSharedMemorySize, 100 * 1024) != cudaSuccess)
        return 1;
    fk<<<(unsigned)(np * n * ((n + fs.bc - 1) / fs.bc)), 256, smem, st>>>(r, s, fs.bc, S.H, S.Bf, S.F, fl);
    g_launches.fetch_add(2, std::memory_order_relaxed);
    sym_finish(sym_view(r, s, atwo, S), S, amat, atmat, fl, st);
    return cudaPeekAtLastError() == cudaSuccess ? 0 : 1;
}

int launch_sym_state_split(const Rdm &r, int s, const double *atwo, const SymScratch &S, double *rows_buf,
                           void *oz_work, int *oz_err, double *amat, double *atmat, int *flag, cudaStream_t st) {
    const int n = r.n, np = n * (n + 1) / 2, *fl = flag + s;
    const ll n2 = (ll)n * n, n3 = n2 * n, rows = std::max(n8_rows(n, 0), n8_rows(n, 2));
    const oz::Gate gate{fl, false};
    sym_unpack(r, s, S, flag, st);
    // F: the operand rows of some creator pairs at a time, then their digit product
    const int bc = std::max(1, kSymXRows * 8 / n), K = n * (np + 1), prs = sym_split_pairs(n);
    const int smem = bc * n * (np | 1) * (int)sizeof(double);
    if (smem > 48 * 1024 && cudaFuncSetAttribute((const void *)k_sym_x, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                 100 * 1024) != cudaSuccess)
        return 1;
    for (int p0 = 0; p0 < np; p0 += prs) {
        const int p = std::min(prs, np - p0);
        unsigned long long *rmax = (unsigned long long *)(rows_buf + p * n3 * K);
        k_sym_x<<<(unsigned)(p * n * ((n + bc - 1) / bc)), 256, smem, st>>>(r, s, bc, p0, S.H, rows_buf, rmax, fl);
        g_launches.fetch_add(1, std::memory_order_relaxed);
        const double *X[1] = {rows_buf}, *B[1] = {S.Bf};
        double *F[1] = {S.F + p0 * n3 * n};
        const unsigned long long *rm[1] = {rmax};
        if (oz::oz_gemm_skinny(oz::OzPlan(1, p * n3, K, n), X, B, F, n, n, oz_work, st, rm, gate, oz_err)) return 1;
    }
    // the n^8 tensors: Wca, Waa and Kx share their right-hand operand
    const dim3 gr((unsigned)((rows * (n2 + 1) + 255) / 256), 4);
    k_sym_rows<<<gr, 256, 0, st>>>(r, s, rows_buf, fl);
    g_launches.fetch_add(1, std::memory_order_relaxed);
    oz::WideGemm g;
    g.m = n8_at(n, 3) / n2; g.n = n2; g.K = (int)n2;
    g.A = rows_buf; g.a_r = n2; g.a_k = 1;
    g.B = S.I4; g.b_c = 1; g.b_k = n2;
    g.C = S.N8; g.ldc = n2;
    if (oz::oz_gemm_wide(g, oz_work, oz_err, st)) return 1;
    g.m = n8_rows(n, 3); g.n = np; g.K = (int)n2 + 1;
    g.A = rows_buf + n8_at(n, 3); g.a_r = n2 + 1;
    g.B = S.IJ; g.b_k = np;
    g.C = S.N8 + n8_at(n, 3); g.ldc = np;
    if (oz::oz_gemm_wide(g, oz_work, oz_err, st)) return 1;
    sym_finish(sym_view(r, s, atwo, S), S, amat, atmat, fl, st);
    return cudaPeekAtLastError() == cudaSuccess ? 0 : 1;
}

int sym_split_pairs(int n) { return std::max(1, std::min(n * (n + 1) / 2, 65536 / (n * n * n))); }

ll sym_split_rows_doubles(int n) {
    const ll n2 = (ll)n * n, np = n * (n + 1) / 2, xr = sym_split_pairs(n) * n2 * n;
    return std::max(xr * (n * (np + 1) + 1), n8_at(n, 3) + n8_rows(n, 3) * (n2 + 1));
}

size_t sym_split_oz_bytes(int n) {
    const ll n2 = (ll)n * n, np = n * (n + 1) / 2;
    return std::max({oz::OzPlan(1, sym_split_pairs(n) * n2 * n, n * (int)(np + 1), n).bytes(),
                     oz::oz_wide_bytes(n8_at(n, 3) / n2, n2, (int)n2), oz::oz_wide_bytes(n8_rows(n, 3), np, (int)n2 + 1)});
}

}  // namespace nvpt

// Stage-1 kernels: partial traces of the packed 4-RDM, active integrals and
// the generalised Koopmans matrices, FP64.
//
// No atomics: results are deterministic.  The reference loop nests each kernel
// restates are cited on the kernel.  The n^9 A-matrix builder has its own files
// (bamat*.cu); this file holds the n^5..n^7 work.
#include "koop_sym.cuh"
#include "nvpt2_internal.h"

#include <algorithm>

namespace nvpt {

#define ATWO(i, j, k, l) atwo[((i)-1) + (ll)n * (((j)-1) + (ll)n * (((k)-1) + (ll)n * ((l)-1)))]
#define FF(i, j) f[tri_index((i) + ncore, (j) + ncore) - 1]
#define AJ(i, j) aj[tri_index((i) + ncore, (j) + ncore) - 1]
#define O3(arr, s, a, b) arr[((s)-1) + (ll)M * (((a)-1) + (ll)n * ((b)-1))]
#define O5(arr, s, a, b, c, d) arr[((s)-1) + (ll)M * (((a)-1) + (ll)n * (((b)-1) + (ll)n * (((c)-1) + (ll)n * ((d)-1))))]

// Decode a flat 0-based index into `k` 1-based orbital indices, first fastest.
__device__ __forceinline__ void decode(ll x, int n, int k, int *out) {
    for (int i = 0; i < k; ++i) { out[i] = (int)(x % n) + 1; x /= n; }
}

// ---------------------------------------------------------------------------
// One-electron operator of each builder (src/koop_matrices.F90:191-200 and
// siblings): active upper triangle of f, mode 0: aj; 1: aj - 1/2 sum_c
// atwo(a,c,c,b); 2: aj - sum_c atwo(a,c,c,b).
__global__ void k_build_f(double *f, const double *aj, const double *atwo, int n, int ncore, int mode) {
    int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= n * n) return;
    int a = t % n + 1, b = t / n + 1;
    if (b < a) return;
    double v = AJ(a, b);
    if (mode != 0)
        for (int c = 1; c <= n; ++c) v -= (mode == 1 ? 0.5 : 1.0) * ATWO(a, c, c, b);
    FF(a, b) = v;
}

// ---------------------------------------------------------------------------
// src/koopro4QD.F90:4881-4959 bro3.
// bro3 as two passes over case-A terms.  Each term of the reference's sum,
// ro4[ord8(i,j,k,l; ii,jj,kk,l)], is read with the key taken from the group
// of larger normind (the first on ties).  Call a term "case A" for the output
// O = (i,j,k; ii,jj,kk) when that is the first group.  A term of O that is
// not case A is, entry for entry, a strict case-A term of the transposed
// output O^T = (ii,jj,kk; i,j,k): ord8 sees the same key group with the same
// partner.  So with
//   P[O] = sum of the case-A terms of O,  Q[O] = the strict (>) ones,
// daaa[O] = (P[O] + Q[O^T]) / (nele - 3).  In the first pass one CTA owns
// the column group (ii,jj,kk) and its threads the rows (i,j,k): every term's
// partner is a permutation of (ii,jj,kk,l), so a CTA reads at most 24 n
// columns of ro4, each W contiguous doubles, and the CTAs of the
// permutations of one multiset -- which read the same columns -- run side by
// side (blockIdx orders them together).  The second pass is a tiled
// transpose-add.  Summation order per element: the case-A terms in l order,
// then the others in l order (the reference adds all in l order).
constexpr int kBro3States = 8;  // states per pass of the first kernel
__global__ void __launch_bounds__(256) k_bro3_case_a(Rdm r, int s0, int ns, double *P, double *Q) {
    const int n = r.n, M = r.M;
    const ll n3 = (ll)n * n * n;
    // block = 6 multiset + permutation; a permutation equal to an earlier one has nothing to do
    int m = blockIdx.x / 6, v[3] = {0, 0, 0};
    while ((v[2] + 1) * (v[2] + 2) * (v[2] + 3) / 6 <= m) ++v[2];
    m -= v[2] * (v[2] + 1) * (v[2] + 2) / 6;
    while ((v[1] + 1) * (v[1] + 2) / 2 <= m) ++v[1];
    v[0] = m - v[1] * (v[1] + 1) / 2;  // v[0] <= v[1] <= v[2]
    const int pm = blockIdx.x % 6;
    const unsigned distinct = v[0] == v[1] ? (v[1] == v[2] ? 0x01 : 0x13) : (v[1] == v[2] ? 0x0d : 0x3f);
    if (!(distinct >> pm & 1)) return;
    const int i0 = pm >> 1, ii = v[i0] + 1, jj = v[(i0 + 1 + (pm & 1)) % 3] + 1, kk = v[(i0 + 2 - (pm & 1)) % 3] + 1;
    const int c = ii - 1 + n * (jj - 1 + n * (kk - 1));
    __shared__ int s_n2[16];  // normind(ii,jj,kk,l) per l
    if (threadIdx.x < n) s_n2[threadIdx.x] = normind4(ii, jj, kk, threadIdx.x + 1);
    __syncthreads();
    for (ll rr = threadIdx.x; rr < n3; rr += blockDim.x) {
        const int i = (int)(rr % n) + 1, j = (int)((rr / n) % n) + 1, k = (int)(rr / ((ll)n * n)) + 1;
        double p[kBro3States], q[kBro3States];
#pragma unroll
        for (int t = 0; t < kBro3States; ++t) p[t] = q[t] = 0.0;
        for (int l = 1; l <= n; ++l) {
            // ord8 with the first group as key (case A): its selection sort,
            // the same swaps on the partner; lindice of the sorted key is
            // normind of the first group
            int kq[4] = {i, j, k, l}, pq[4] = {ii, jj, kk, l};
#pragma unroll
            for (int a = 0; a < 4; ++a) {
                int imax = kq[a], jmax = a;
#pragma unroll
                for (int b = a + 1; b < 4; ++b)
                    if (kq[b] > imax) { imax = kq[b]; jmax = b; }
#pragma unroll
                for (int b = a + 1; b < 4; ++b)  // static indices: the arrays stay in registers
                    if (jmax == b) {
                        int t = kq[a]; kq[a] = kq[b]; kq[b] = t;
                        t = pq[a]; pq[a] = pq[b]; pq[b] = t;
                    }
            }
            const int n1 = lindice4(kq[0], kq[1], kq[2], kq[3]), n2 = s_n2[l - 1];
            if (n1 < n2) continue;
            const int ind = n1, q0 = pq[0], q1 = pq[1], q2 = pq[2], q3 = pq[3];
#pragma unroll
            for (int t = 0; t < kBro3States; ++t) {
                if (t >= ns) break;
                const double x = r.R4(ind, q0, q1, q2, q3, s0 + t + 1);
                p[t] += x;
                if (n1 > n2) q[t] += x;
            }
        }
        const ll o = (ll)M * (rr + n3 * c);
#pragma unroll
        for (int t = 0; t < kBro3States; ++t)
            if (t < ns) {
                P[o + s0 + t] = p[t];
                Q[o + s0 + t] = q[t];
            }
    }
}

// daaa[s, r, c] = (P[s, r, c] + Q[s, c, r]) * inv over the n^3 x n^3 matrix
// of each state (r = (i,j,k), c = (ii,jj,kk), r fastest), 32 x 32 tiles
// through shared memory so both reads and the write are coalesced.
__global__ void __launch_bounds__(256) k_bro3_combine(const double *P, const double *Q, double *daaa, ll n3, int M,
                                                      double inv) {
    __shared__ double t[32][33];
    const ll r0 = (ll)blockIdx.x * 32, c0 = (ll)blockIdx.y * 32;
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
    for (int s = 0; s < M; ++s) {
        // Q tile at (row c0.., col r0..): element Q[s, c, r] with c fastest
        for (int y = ty; y < 32; y += 8) {
            const ll c = c0 + tx, rr = r0 + y;
            t[y][tx] = (c < n3 && rr < n3) ? Q[s + (ll)M * (c + n3 * rr)] : 0.0;
        }
        __syncthreads();
        for (int y = ty; y < 32; y += 8) {
            const ll rr = r0 + tx, c = c0 + y;
            if (rr < n3 && c < n3) {
                const ll o = s + (ll)M * (rr + n3 * c);
                daaa[o] = (P[o] + t[tx][y]) * inv;
            }
        }
        __syncthreads();
    }
}

// src/koopro4QD.F90:4961-5000 bro2
__global__ void k_bro2(Rdm r, double *taa, double inv) {
    const int n = r.n, M = r.M;
    ll t = (ll)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= (ll)n * n * n * n) return;
    int x[4];
    decode(t, n, 4, x);
    for (int s = 1; s <= M; ++s) {
        double acc = 0.0;
        for (int l = 1; l <= n; ++l) acc += r.D3(s, x[0], x[1], l, x[2], x[3], l);
        taa[(s - 1) + (ll)M * t] = acc * inv;
    }
}

// src/koopro4QD.F90:5002-5049 bro1
__global__ void k_bro1(Rdm r, double *dal, double inv) {
    const int n = r.n, M = r.M;
    int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= n * n) return;
    int i = t % n + 1, j = t / n + 1;
    for (int s = 1; s <= M; ++s) {
        double acc = 0.0;
        for (int l = 1; l <= n; ++l) acc += r.D2(s, i, l, j, l);
        dal[(s - 1) + (ll)M * t] = acc * inv;
    }
}

// ---------------------------------------------------------------------------
// src/koopro4QD.F90:3900-3971 get_aj_atwo with the Cholesky integrals of
// src/ijkl_utils.F90:637-688: (ij|kl) = sum_Q L(Q,indice(i,j)) L(Q,indice(k,l)).
//
// Columns L(.,pair) are contiguous and a CTA owns one active pair, a warp a dot
// product: blocks [0, np): atwo for the pairs up to its own, written to the
// eight equal positions; [np, 2 np): aj = oneint + sum_j [2 (ab|jj) - (aj|jb)];
// the rest copy oneint to the other elements of aj.
__global__ void __launch_bounds__(256) k_aj_atwo(const double *__restrict__ oneint, const double *__restrict__ L, int Q,
                                                 int n, int ncore, ll npair, double *atwo, double *aj) {
    __shared__ double red[8];
    const int np = n * (n + 1) / 2, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    int pr = blockIdx.x;
    if (pr >= 2 * np) {
        for (ll i = (ll)(pr - 2 * np) * 256 + threadIdx.x; i < npair; i += (ll)(gridDim.x - 2 * np) * 256) {
            // row of the triangle holding i: the active block is rows and columns ncore + 1 .. ncore + n
            ll row = (ll)((sqrt(8.0 * (double)i + 1.0) - 1.0) * 0.5);
            while ((row + 1) * (row + 2) / 2 <= i) ++row;
            while (row * (row + 1) / 2 > i) --row;
            const ll c = i - row * (row + 1) / 2;
            if (!(row >= ncore && row < ncore + n && c >= ncore)) aj[i] = oneint[i];
        }
        return;
    }
    const bool one = pr >= np;
    if (one) pr -= np;
    int a = 0;
    while ((a + 1) * (a + 2) / 2 <= pr) ++a;
    const int b = pr - a * (a + 1) / 2;  // a >= b
    const ll pab = tri_index(a + 1 + ncore, b + 1 + ncore) - 1;
    const double *x = L + (ll)Q * pab;
    if (!one) {
        for (int p2 = warp; p2 <= pr; p2 += 8) {
            int c = 0;
            while ((c + 1) * (c + 2) / 2 <= p2) ++c;
            const int d = p2 - c * (c + 1) / 2;
            const double *y = L + (ll)Q * (tri_index(c + 1 + ncore, d + 1 + ncore) - 1);
            double v = 0.0;
            for (int q = lane; q < Q; q += 32) v = fma(x[q], y[q], v);
            for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
            if (lane < 8) {  // (ab|cd) at its eight places
                const int i = lane & 1 ? b : a, j = lane & 1 ? a : b, k = lane & 2 ? d : c, l = lane & 2 ? c : d;
                if (lane & 4) ATWO(k + 1, l + 1, i + 1, j + 1) = v;
                else ATWO(i + 1, j + 1, k + 1, l + 1) = v;
            }
        }
        return;
    }
    double v = 0.0;
    for (int j = warp; j < ncore; j += 8) {
        const double *jj = L + (ll)Q * (tri_index(j + 1, j + 1) - 1);
        const double *aj_ = L + (ll)Q * (tri_index(a + 1 + ncore, j + 1) - 1);
        const double *jb = L + (ll)Q * (tri_index(b + 1 + ncore, j + 1) - 1);
        for (int q = lane; q < Q; q += 32) v += 2.0 * x[q] * jj[q] - aj_[q] * jb[q];
    }
    for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if (lane == 0) red[warp] = v;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < 8; ++w) v += red[w];
        aj[pab] = oneint[pab] + v;
    }
}

// ---------------------------------------------------------------------------
// The generalised Koopmans matrices: koopE, koop2E, koopman0pE
// (src/koop_matrices.F90:165-591), bbmat, bcmat, bdmat (src/koopro4QD.F90:4231-4459).
//
// Their n^7 sums are contractions of an operand G(r1,r2,z; k1,k2,k3), a few
// accessors of one state's RDMs, with the active integrals over (k1,k2,k3):
// P[(r1,r2,z), x] = sum_k G T(k; x).  A CTA owns some pairs (r1,r2) with all z
// and x, evaluates G into shared memory 32 k at a time -- rows r1 first, which
// is the index that most of the 3-RDM loads have fastest -- and multiplies.
// What the reference adds to an output element are P's of the same pair with z
// and x exchanged, so the CTA finishes its elements itself: nothing is
// materialised, and koop_matrices_ctl is one launch.  Small spaces are bound by
// latency (CTAs of one pair, the k range split over the threads left), large
// ones by the FP64 pipe and the accessors.
enum KoopOp { IP1, IP2, EA1, EA2, A1, A2, D1, D2, B1, BT, C1, C2, C3, CT1, CT2, CT3 };

__device__ __forceinline__ double koop0p_e1(const Rdm &r, int c, int d, int ie, int bp, int ap, int a, int s) {
    double e1 = -r.eee2(c, ie, a, ap, bp, d, s) - r.eee2(a, ap, bp, d, c, ie, s);
    if (ap == a) e1 += 2.0 * (r.ee2(c, ie, bp, d, s) + r.ee2(bp, d, c, ie, s));
    if (bp == ap) e1 += r.ee2(c, ie, a, d, s) + r.ee2(a, d, c, ie, s);
    if (ap == c) {
        e1 -= r.ee2(a, ie, bp, d, s);
        if (ie == a) e1 += 2.0 * r.D1(s, bp, d);
    }
    if (bp == ie) {
        e1 += r.ee2(a, ap, c, d, s);
        if (ap == a) e1 -= 2.0 * r.D1(s, c, d);
    }
    return e1;
}
__device__ __forceinline__ double koop0p_e2(const Rdm &r, int c, int d, int ie, int bp, int ap, int b, int s) {
    double e2 = -r.eee2(c, ie, d, ap, bp, b, s) - r.eee2(d, ap, bp, b, c, ie, s);
    if (ap == d) e2 += 2.0 * (r.ee2(c, ie, bp, b, s) + r.ee2(bp, b, c, ie, s));
    if (bp == ap) e2 += r.ee2(c, ie, d, b, s) + r.ee2(d, b, c, ie, s);
    if (ap == c) {
        e2 -= r.ee2(d, ie, bp, b, s);
        if (d == ie) e2 += 2.0 * r.D1(s, bp, b);
    }
    if (bp == ie) {
        e2 += r.ee2(d, ap, c, b, s);
        if (d == ap) e2 -= 2.0 * r.D1(s, c, b);
    }
    return e2;
}

// G of one operation at 1-based labels.
template <int OP>
__device__ __forceinline__ double koop_operand(const Rdm &r, int s, int r1, int r2, int z, int k1, int k2, int k3) {
    if constexpr (OP == IP1 || OP == IP2) {  // (ap,bp,b) / (ap,bp,a); (d,ie,ief)
        const int ap = r1, bp = r2, d = k1, ie = k2, ief = k3;
        double v;
        if constexpr (OP == IP1) {
            v = r.D3(s, ap, bp, d, ief, z, ie);
            if (d == ief) v += 0.5 * r.D2(s, ap, bp, ie, z);
            if (d == z) v += 0.5 * r.D2(s, ap, bp, ief, ie);
        } else {
            v = r.D3(s, ap, bp, d, z, ief, ie);
            if (d == z) v += 0.5 * r.D2(s, ap, bp, ie, ief);
            if (d == ief) v += 0.5 * r.D2(s, ap, bp, z, ie);
        }
        return v;
    } else if constexpr (OP == EA1 || OP == EA2) {  // (ap,bp,b) / (ap,bp,a); (c,d,ie)
        const int ap = r1, bp = r2, c = k1, d = k2, ie = k3;
        double v;
        if constexpr (OP == EA1) {
            v = -r.ro3t(ap, bp, ie, d, z, c, s);
            if (c == ie) v += 2.0 * r.ro2t(ap, bp, d, z, s);
            if (d == ie) v -= 0.5 * r.ro2t(ap, bp, c, z, s);
            if (z == ie) v -= 0.5 * r.ro2t(ap, bp, d, c, s);
        } else {
            v = -r.ro3t(ap, bp, ie, z, d, c, s);
            if (c == ie) v += 2.0 * r.ro2t(ap, bp, z, d, s);
            if (z == ie) v -= 0.5 * r.ro2t(ap, bp, c, d, s);
            if (d == ie) v -= 0.5 * r.ro2t(ap, bp, z, c, s);
        }
        return v;
    } else if constexpr (OP == A1) {  // (bp,ap,b); (c,d,ie)
        return r.eee2(r1, r2, k1, k3, k2, z, s) + r.eee2(r1, r2, k2, z, k1, k3, s);
    } else if constexpr (OP == A2) {  // (bp,ap,a); (c,d,ie)
        return r.eee2(r1, r2, z, k3, k1, k2, s) + r.eee2(r1, r2, k1, k2, z, k3, s);
    } else if constexpr (OP == D1) {
        return koop0p_e2(r, k1, k2, k3, r1, r2, z, s);
    } else if constexpr (OP == D2) {
        return koop0p_e1(r, k1, k2, k3, r1, r2, z, s);
    } else if constexpr (OP == B1) {  // (cp,ap,bp); (ie,c,ief)
        return r.eee2(r1, r2, z, k1, k2, k3, s);
    } else if constexpr (OP == BT) {
        return r.eee2t(r1, r2, z, k1, k2, k3, s);
    } else if constexpr (OP == C1) {  // (ap,b,c); (d,ief,ie)
        return r.eee2(r1, r2, k1, k2, k3, z, s);
    } else if constexpr (OP == C2) {  // (ap,b,a)
        return r.eee2(r1, r2, k1, k2, z, k3, s);
    } else if constexpr (OP == C3) {  // (ap,a,c)
        return r.eee2(r1, k3, k1, k2, r2, z, s);
    } else if constexpr (OP == CT1) {
        return r.eee2tl(r1, r2, k1, k2, k3, z, s);
    } else if constexpr (OP == CT2) {
        return r.eee2tl(r1, r2, k1, k2, z, k3, s);
    } else {
        return r.eee2tl(r1, k3, k1, k2, r2, z, s);
    }
}

// Strides of the integral T(k; x) in k1, k2, k3, x.
template <int OP>
__device__ __forceinline__ void koop_strides(int n, int &s1, int &s2, int &s3, int &sx) {
    const int p1 = n, p2 = n * n, p3 = n * n * n;
    if constexpr (OP == IP1 || OP == IP2) { s1 = 1; s2 = p1; s3 = p3; sx = p2; }                 // (d,ie,x,ief)
    else if constexpr (OP == EA1 || OP == EA2 || OP == A1 || OP == D1) { s1 = 1; s2 = p2; s3 = p1; sx = p3; }  // (c,ie,d,x)
    else if constexpr (OP == A2) { s1 = p2; s2 = p3; s3 = p1; sx = 1; }                           // (x,ie,c,d)
    else if constexpr (OP == D2) { s1 = 1; s2 = p3; s3 = p1; sx = p2; }                           // (c,ie,x,d)
    else if constexpr (OP == B1 || OP == BT) { s1 = p1; s2 = p2; s3 = p3; sx = 1; }               // (x,ie,c,ief)
    else if constexpr (OP == C1 || OP == CT1) { s1 = 1; s2 = p1; s3 = p2; sx = p3; }              // (d,ief,ie,x)
    else { s1 = 1; s2 = p1; s3 = p3; sx = p2; }                                                   // (d,ief,x,ie)
}

constexpr int kKoopRpt = 4;     // most rows per thread
struct KoopTile {
    int n, pair0, npair, R;     // pairs of the CTA, rows R = npair n (row = z npair + pair)
    int kc;                     // k per shared-memory chunk
    double *A, *B, *P;          // [kc][R + 1], [kc][n], results [2][R][n]
};
// k per chunk: about 2048 operand elements, so that a small CTA does not
// synchronise more often than it computes
__host__ __device__ __forceinline__ int koop_chunk(int n, int G) { return max(32, min(256, 2048 / (G * n))); }

// P[slot][row][x] of one operation; all threads of the CTA.
template <int OP>
__device__ __forceinline__ void koop_contract(const Rdm &r, int s, const double *__restrict__ atwo, const KoopTile &t,
                                              int slot) {
    const int n = t.n, R = t.R, lda = R + 1, tid = threadIdx.x, K = n * n * n;
    int s1, s2, s3, sx;
    koop_strides<OP>(n, s1, s2, s3, sx);
    // threads: column, row group, and -- when one row per thread leaves room -- a share of the k's,
    // no more shares than k's: they are added up one after another (n = 1: 256 of them took 100 us)
    const int groups = 256 / n, rpt = (R + groups - 1) / groups;
    const int slices = rpt == 1 ? min(256 / (R * n), K) : 1, per = rpt == 1 ? R * n : 256;
    const int slice = tid / per, q = tid % per, col = q % n, grp = q / n;
    const bool live = slice < slices && grp < groups && (rpt > 1 || grp < R);
    double acc[kKoopRpt] = {};
    for (int k0 = 0; k0 < K; k0 += t.kc) {
        const int nk = min(t.kc, K - k0);
        for (int i = tid; i < nk * R; i += 256) {
            const int row = i % R, kk = i / R, k = k0 + kk;
            const int pair = t.pair0 + row % t.npair, z = row / t.npair;
            t.A[kk * lda + row] =
                koop_operand<OP>(r, s, pair % n + 1, pair / n + 1, z + 1, k % n + 1, (k / n) % n + 1, k / (n * n) + 1);
        }
        for (int i = tid; i < nk * n; i += 256) {
            const int x = i % n, k = k0 + i / n;
            t.B[i] = atwo[(k % n) * s1 + ((k / n) % n) * s2 + (k / (n * n)) * s3 + x * sx];
        }
        __syncthreads();
        if (live) {
            if (rpt == 1) {
                for (int kk = slice; kk < nk; kk += slices) acc[0] = fma(t.A[kk * lda + grp], t.B[kk * n + col], acc[0]);
            } else {
                for (int kk = 0; kk < nk; ++kk) {
                    const double b = t.B[kk * n + col];
#pragma unroll
                    for (int i = 0; i < kKoopRpt; ++i)
                        if (i < rpt) acc[i] = fma(t.A[kk * lda + min(grp + i * groups, R - 1)], b, acc[i]);
                }
            }
        }
        __syncthreads();
    }
    double *P = t.P + slot * R * n;
    if (rpt == 1) {
        for (int sl = 0; sl < slices; ++sl) {  // slices in order: a fixed sum
            if (live && slice == sl) P[grp * n + col] = sl ? P[grp * n + col] + acc[0] : acc[0];
            __syncthreads();
        }
    } else {
        if (live)
#pragma unroll
            for (int i = 0; i < kKoopRpt; ++i)
                if (i < rpt && grp + i * groups < R) P[(grp + i * groups) * n + col] = acc[i];
        __syncthreads();
    }
}

// The builder's one-electron operator on the active block (mode 0: aj, 1: aj -
// K/2, 2: aj - K with K(a,b) = sum_c (ac|cb)) in shared memory, and, by one CTA
// of the launch, in the upper triangle of f(*).
__device__ __forceinline__ void koop_operator(double *ff, const double *aj, const double *atwo, int n, int ncore,
                                              int mode, double *f) {
    for (int i = threadIdx.x; i < n * n; i += blockDim.x) {
        const int x = i % n + 1, y = i / n + 1, a = min(x, y), b = max(x, y);
        double v = AJ(a, b);
        if (mode != 0)
            for (int c = 1; c <= n; ++c) v -= (mode == 1 ? 0.5 : 1.0) * ATWO(a, c, c, b);
        ff[i] = v;
        if (f && x <= y) FF(x, y) = v;
    }
    __syncthreads();
}
#define FS(i, j) ff[((j)-1) * n + (i)-1]

__device__ __forceinline__ double block_reduce(double v, double *red) {
    for (int o = 16; o; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    __syncthreads();
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
    __syncthreads();
    double t = 0.0;
    for (int w = 0; w < 8; ++w) t += red[w];
    return t;
}

struct KoopOut {
    double *p[8];
};

// koop_matrices_ctl.  blockIdx.y: 0 2-IP, 1 2-EA and the 2-HRDM, 2 A and 3 D of
// the 0' class, 4 koopE and the 0' F (a CTA per element); blockIdx.z: state.
// out: ipko1, eako1, hrdm2, ipko2, eako2, gk0pa, gk0pd, gk0pf.
__global__ void __launch_bounds__(256) k_koop_ctl(Rdm r, const double *__restrict__ atwo, const double *__restrict__ aj,
                                                  int ncore, int G, double *f, KoopOut out, const int *flag) {
    const int part = blockIdx.y;
    if (part != 4 && flag && !flag[blockIdx.z]) return;
    extern __shared__ double sm[];
    const int n = r.n, M = r.M, s = blockIdx.z + 1, tid = threadIdx.x;
    double *ff = sm;
    KoopTile t;
    t.n = n;
    t.kc = koop_chunk(n, G);
    t.A = ff + n * n;
    t.B = t.A + t.kc * (G * n + 1);
    t.P = t.B + t.kc * n;
    koop_operator(ff, aj, atwo, n, ncore, 1, part == 4 && blockIdx.x == 0 && blockIdx.z == 0 ? f : nullptr);
    if (part == 4) {
        for (int it = blockIdx.x; it < n * n; it += gridDim.x) {
            const int x = it % n + 1, y = it / n + 1;  // koopE (ap, a); F (a, b)
            double ip = 0.0, ea = 0.0, fv = 0.0;
            for (int k = tid; k < n * n * n; k += 256) {
                const int c = k % n + 1, d = (k / n) % n + 1, ie = k / (n * n) + 1;
                ip -= ATWO(c, ie, y, d) * r.D2(s, x, c, d, ie);
                fv += ATWO(c, ie, d, x) * (r.ee2(c, ie, d, y, s) + r.ee2(d, y, c, ie, s)) -
                      ATWO(y, ie, c, d) * (r.ee2(x, ie, c, d, s) + r.ee2(c, d, x, ie, s));
                if (ie == 1) ea += (2.0 * ATWO(c, d, x, y) - ATWO(x, d, c, y)) * r.D1(s, c, d);
            }
            for (int c = tid + 1; c <= n; c += 256) {
                ip -= AJ(y, c) * r.D1(s, x, c);
                fv += 2.0 * (FS(c, x) * r.D1(s, c, y) - FS(y, c) * r.D1(s, x, c));
            }
            double *red = t.A;
            ip = block_reduce(ip, red);
            ea = block_reduce(ea, red);
            fv = block_reduce(fv, red);
            if (tid == 0) {
                O3(out.p[0], s, x, y) = 2.0 * ip;
                O3(out.p[1], s, x, y) = 2.0 * ip + 2.0 * (2.0 * AJ(x, y) + ea);
                O3(out.p[7], s, x, y) = fv;
            }
        }
        return;
    }
    t.pair0 = blockIdx.x * G;
    t.npair = min(G, n * n - t.pair0);
    t.R = t.npair * n;
    switch (part) {
    case 0: koop_contract<IP1>(r, s, atwo, t, 0); koop_contract<IP2>(r, s, atwo, t, 1); break;
    case 1: koop_contract<EA1>(r, s, atwo, t, 0); koop_contract<EA2>(r, s, atwo, t, 1); break;
    case 2: koop_contract<A1>(r, s, atwo, t, 0); koop_contract<A2>(r, s, atwo, t, 1); break;
    default: koop_contract<D1>(r, s, atwo, t, 0); koop_contract<D2>(r, s, atwo, t, 1); break;
    }
    const double *P0 = t.P, *P1 = t.P + t.R * n;  // [z npair + pair][x]
    for (int i = tid; i < t.R * n; i += 256) {
        const int g = i % t.npair, a0 = (i / t.npair) % n, b0 = i / (t.npair * n), a = a0 + 1, b = b0 + 1;
        const int p = (t.pair0 + g) % n + 1, q = (t.pair0 + g) / n + 1;
        const double x0 = P0[(b0 * t.npair + g) * n + a0], x1 = P1[(a0 * t.npair + g) * n + b0];
        double v = 0.0;
        if (part == 0) {  // (ap,bp) = (p,q)
            for (int d = 1; d <= n; ++d) v -= FS(a, d) * r.D2(s, p, q, d, b) + FS(b, d) * r.D2(s, p, q, a, d);
            O5(out.p[3], s, p, q, a, b) = v - x0 - x1;
        } else if (part == 1) {
            for (int c = 1; c <= n; ++c) v += FS(a, c) * r.ro2t(p, q, c, b, s) + FS(b, c) * r.ro2t(p, q, a, c, s);
            O5(out.p[4], s, p, q, a, b) = v + x0 + x1;
            O5(out.p[2], s, p, q, a, b) = r.ro2t(p, q, a, b, s);
        } else if (part == 2) {  // (bp,ap) = (p,q)
            for (int c = 1; c <= n; ++c) v += 2.0 * (FS(c, a) * r.ee2(p, q, c, b, s) - FS(b, c) * r.ee2(p, q, a, c, s));
            O5(out.p[5], s, p, q, a, b) = v + x0 - x1;
        } else {
            for (int c = 1; c <= n; ++c) {
                double d1 = -r.ee2(a, q, p, c, s), d2 = -r.ee2(c, q, p, b, s);
                if (a == q) d1 += 2.0 * r.D1(s, p, c);
                if (c == q) d2 += 2.0 * r.D1(s, p, b);
                if (p == q) {
                    d1 += r.D1(s, a, c);
                    d2 += r.D1(s, c, b);
                }
                v += FS(c, a) * d2 - FS(b, c) * d1;
            }
            O5(out.p[6], s, p, q, a, b) = v + 0.5 * x0 - 0.5 * x1;
        }
    }
}

// bbmat (blockIdx.y 0 B, 1 B~; rows (cp,ap,bp)) and the two passes of bcmat
// (kind 1: the first two contractions and all lower terms of C / C~, rows
// (ap,b,.); kind 2: the third, rows (ap,a,c), added to it).  B~ multiplies the
// one-electron part by aj, not by the modified f (reference quirk kept).
__global__ void __launch_bounds__(256) k_koop_bc(Rdm r, const double *__restrict__ atwo, const double *__restrict__ aj,
                                                 int ncore, int G, int kind, double *f, double *x0, double *x1,
                                                 const int *flag) {
    const bool first = blockIdx.x == 0 && blockIdx.y == 0 && blockIdx.z == 0, skip = flag && !flag[blockIdx.z];
    if (skip && !first) return;
    extern __shared__ double sm[];
    const int n = r.n, M = r.M, s = blockIdx.z + 1, part = blockIdx.y, tid = threadIdx.x;
    double *ff = sm;
    KoopTile t;
    t.n = n;
    t.kc = koop_chunk(n, G);
    t.A = ff + n * n;
    t.B = t.A + t.kc * (G * n + 1);
    t.P = t.B + t.kc * n;
    t.pair0 = blockIdx.x * G;
    t.npair = min(G, n * n - t.pair0);
    t.R = t.npair * n;
    koop_operator(ff, aj, atwo, n, ncore, kind == 0 ? 2 : 1, first && kind != 2 ? f : nullptr);
    if (skip) return;
    if (kind == 0) {
        if (part == 0) koop_contract<B1>(r, s, atwo, t, 0);
        else koop_contract<BT>(r, s, atwo, t, 0);
    } else if (kind == 1) {
        if (part == 0) { koop_contract<C1>(r, s, atwo, t, 0); koop_contract<C2>(r, s, atwo, t, 1); }
        else { koop_contract<CT1>(r, s, atwo, t, 0); koop_contract<CT2>(r, s, atwo, t, 1); }
    } else {
        if (part == 0) koop_contract<C3>(r, s, atwo, t, 0);
        else koop_contract<CT3>(r, s, atwo, t, 0);
    }
    const double *P0 = t.P, *P1 = t.P + t.R * n;
    double *out = part == 0 ? x0 : x1;
    for (int i = tid; i < t.R * n; i += 256) {
        const int g = i % t.npair, z0 = (i / t.npair) % n, w0 = i / (t.npair * n);
        const int p = (t.pair0 + g) % n + 1, q = (t.pair0 + g) / n + 1, z = z0 + 1, w = w0 + 1;
        double v = 0.0;
        if (kind == 0) {  // (cp,ap) = (p,q), bp = z, a = w
            const double x = P0[(z0 * t.npair + g) * n + w0];
            if (part == 0)
                for (int c = 1; c <= n; ++c) v -= FS(c, w) * r.ee2(p, q, z, c, s);
            else
                for (int c = 1; c <= n; ++c) v += AJ(c, w) * r.ee2tr(p, q, z, c, s);
            O5(out, s, q, z, p, w) = part == 0 ? v - x : v + x;
        } else if (kind == 1) {  // (ap,b) = (p,q), a = z, c = w
            const int ap = p, b = q, a = z, c = w;
            auto e = [&](int i1, int i2, int i3, int i4) {
                return part == 0 ? r.ee2(i1, i2, i3, i4, s) : r.ee2t(i1, i2, i3, i4, s);
            };
            const double sg = part == 0 ? -1.0 : 1.0;
            for (int d = 1; d <= n; ++d) {
                v += FS(d, a) * e(ap, b, d, c) - FS(c, d) * e(ap, b, a, d) + sg * FS(b, d) * e(ap, d, a, c);
                for (int ie = 1; ie <= n; ++ie) {
                    const double dint1 = ATWO(c, ie, d, a), dint2 = ATWO(d, ie, ie, a);
                    const double dint3 = ATWO(c, d, d, ie), dint4 = ATWO(b, d, d, ie);
                    v += e(ap, b, d, ie) * dint1 -
                         0.5 * (e(ap, b, d, c) * dint2 + e(ap, b, a, ie) * dint3 - e(ap, ie, a, c) * dint4);
                }
            }
            O5(out, s, ap, a, b, c) = v + P0[(w0 * t.npair + g) * n + z0] - P1[(z0 * t.npair + g) * n + w0];
        } else {  // (ap,a) = (p,q), c = z, b = w
            const double x = P0[(z0 * t.npair + g) * n + w0];
            O5(out, s, p, q, w, z) += part == 0 ? -x : x;
        }
    }
}

// bdmat: a CTA per (ap,a) and state; the EA part uses aj.
__global__ void __launch_bounds__(256) k_koop_d(Rdm r, const double *atwo, const double *aj, int ncore, double *f,
                                                double *dmat, double *dtmat) {
    __shared__ double ff[256], red[8];
    const int n = r.n, M = r.M, s = blockIdx.y + 1;
    koop_operator(ff, aj, atwo, n, ncore, 2, blockIdx.x == 0 && blockIdx.y == 0 ? f : nullptr);
    const int ap = blockIdx.x % n + 1, a = blockIdx.x / n + 1;
    double D = 0.0, Dt = 0.0;
    for (int k = threadIdx.x; k < n * n * n; k += 256) {
        const int ie = k % n + 1, c = (k / n) % n + 1, ief = k / (n * n) + 1;
        const double dint = ATWO(a, ie, c, ief);
        D -= r.ee2(ap, ie, c, ief, s) * dint;
        Dt += r.ee2t(ap, ie, c, ief, s) * dint;
    }
    for (int c = threadIdx.x + 1; c <= n; c += 256) {
        const double g = r.D1(s, ap, c);
        D -= FS(c, a) * g;
        Dt += AJ(c, a) * ((ap == c ? 2.0 : 0.0) - g);
    }
    D = block_reduce(D, red);
    Dt = block_reduce(Dt, red);
    if (threadIdx.x == 0) {
        O3(dmat, s, ap, a) = D;
        O3(dtmat, s, ap, a) = Dt;
    }
}
#undef FS

// ---------------------------------------------------------------------------
// Host launchers.
static inline unsigned blocks_for(ll work, int tpb) { return (unsigned)((work + tpb - 1) / tpb); }

void launch_build_f(double *f, const double *aj, const double *atwo, int n, int ncore, int mode, cudaStream_t st) {
    k_build_f<<<blocks_for((ll)n * n, 128), 128, 0, st>>>(f, aj, atwo, n, ncore, mode);
    g_launches.fetch_add(1, std::memory_order_relaxed);
}

int launch_bro3(const Rdm &r, double *daaa, int nele, cudaStream_t st) {
    const int n = r.n, M = r.M;
    const ll n3 = (ll)n * n * n, n6 = n3 * n3;
    double *P = nullptr;
    if (cudaMallocAsync((void **)&P, sizeof(double) * 2 * (size_t)(M * n6), st) != cudaSuccess) return 2;
    double *Q = P + (size_t)M * n6;
    ProfSpan span;
    span.begin("bro3", st, 0);
    for (int s0 = 0; s0 < M; s0 += kBro3States) {
        k_bro3_case_a<<<(unsigned)(n * (n + 1) * (n + 2)), 256, 0, st>>>(r, s0, std::min(kBro3States, M - s0), P, Q);
        g_launches.fetch_add(1, std::memory_order_relaxed);
    }
    dim3 g((unsigned)((n3 + 31) / 32), (unsigned)((n3 + 31) / 32));
    k_bro3_combine<<<g, 256, 0, st>>>(P, Q, daaa, n3, M, 1.0 / (double)(nele - 3));
    span.end();
    g_launches.fetch_add(1, std::memory_order_relaxed);
    cudaFreeAsync(P, st);
    return 0;
}
void launch_bro2(const Rdm &r, double *taa, int nele, cudaStream_t st) {
    ll n4 = (ll)r.n * r.n * r.n * r.n;
    k_bro2<<<blocks_for(n4, 256), 256, 0, st>>>(r, taa, 1.0 / (double)(nele - 2));
    g_launches.fetch_add(1, std::memory_order_relaxed);
}
void launch_bro1(const Rdm &r, double *dal, int nele, cudaStream_t st) {
    k_bro1<<<blocks_for((ll)r.n * r.n, 128), 128, 0, st>>>(r, dal, 1.0 / (double)(nele - 1));
    g_launches.fetch_add(1, std::memory_order_relaxed);
}

void launch_aj_atwo(const double *oneint, const double *L, int Q, int n, int ncore, int norb, double *atwo,
                    double *aj, cudaStream_t st) {
    const ll npair = (ll)norb * (norb + 1) / 2;
    const unsigned np = n * (n + 1) / 2, copy = (unsigned)std::min<ll>((npair + 255) / 256, 304);
    k_aj_atwo<<<2 * np + copy, 256, 0, st>>>(oneint, L, Q, n, ncore, npair, atwo, aj);
    g_launches.fetch_add(1, std::memory_order_relaxed);
}

// Pairs per CTA: few idle rows, and enough CTAs for the chip.
static int koop_pairs(int n, int parts) {
    const int groups = 256 / n;
    int best = 1;
    double top = 0.0;
    for (int G = 1; G * n <= kKoopRpt * groups && G <= 6; ++G) {
        const int rpt = (G * n + groups - 1) / groups;
        const double fill = rpt == 1 ? 1.0 : (double)(G * n) / (rpt * groups);
        const double ctas = (double)((n * n + G - 1) / G) * parts;
        // a CTA evaluates each operand once for n products: more rows only fill the threads
        const double score = fill * std::min(1.0, ctas / 304.0) * (rpt == 1 && G > 1 ? 0.99 : 1.0);
        if (score > top) {
            top = score;
            best = G;
        }
    }
    return best;
}
static size_t koop_smem(int n, int G) {
    const int kc = koop_chunk(n, G);
    return sizeof(double) * (size_t)(n * n + kc * (G * n + 1) + kc * n + 2 * G * n * n);
}

// The one-contraction route (koop_sym.cu) with the direct kernels behind its
// flags, from kKoopSymMin active orbitals on; below, the direct kernels alone
// have fewer launches (all builders of one state, sums / direct, us: n = 4 143 / 111,
// n = 5 151 / 144, n = 6 163 / 202, n = 8 210 / 465).  Without room for the route's
// scratch: the direct kernels.
constexpr int kKoopSymMin = 6;
namespace {
struct SymFlags {
    int *p = nullptr;
    cudaStream_t st;
    SymFlags(const Rdm &r, const double *atwo, const double *aj, int ncore, int kind, double *const out[5],
             cudaStream_t s)
        : st(s) {
        if (r.n < kKoopSymMin || cudaMallocAsync((void **)&p, sizeof(int) * r.M, st) != cudaSuccess) {
            p = nullptr;
            return;
        }
        cudaMemsetAsync(p, 0, sizeof(int) * r.M, st);
        if (launch_koop_sym(r, atwo, aj, ncore, kind, out, p, st)) {
            cudaFreeAsync(p, st);
            p = nullptr;
        }
    }
    ~SymFlags() {
        if (p) cudaFreeAsync(p, st);
    }
};
}  // namespace

void launch_koop_ctl(const Rdm &r, const double *atwo, const double *aj, int ncore, double *f, double *const out[8],
                     cudaStream_t st) {
    const int n = r.n, G = koop_pairs(n, 4 * r.M);
    double *const so[5] = {out[3], out[4], out[5], out[6], out[2]};
    const SymFlags flag(r, atwo, aj, ncore, 0, so, st);
    KoopOut o;
    for (int i = 0; i < 8; ++i) o.p[i] = out[i];
    k_koop_ctl<<<dim3((n * n + G - 1) / G, 5, r.M), 256, koop_smem(n, G), st>>>(r, atwo, aj, ncore, G, f, o, flag.p);
    g_launches.fetch_add(1, std::memory_order_relaxed);
}
void launch_bbmat(const Rdm &r, const double *atwo, const double *aj, int ncore, double *f, double *b, double *bt,
                  cudaStream_t st) {
    const int n = r.n, G = koop_pairs(n, 2 * r.M);
    double *const so[5] = {b, bt};
    const SymFlags flag(r, atwo, aj, ncore, 1, so, st);
    k_koop_bc<<<dim3((n * n + G - 1) / G, 2, r.M), 256, koop_smem(n, G), st>>>(r, atwo, aj, ncore, G, 0, f, b, bt,
                                                                              flag.p);
    g_launches.fetch_add(1, std::memory_order_relaxed);
}
void launch_bcmat(const Rdm &r, const double *atwo, const double *aj, int ncore, double *f, double *c, double *ct,
                  cudaStream_t st) {
    const int n = r.n, G = koop_pairs(n, 2 * r.M);
    double *const so[5] = {c, ct};
    const SymFlags flag(r, atwo, aj, ncore, 2, so, st);
    for (int kind = 1; kind <= 2; ++kind)
        k_koop_bc<<<dim3((n * n + G - 1) / G, 2, r.M), 256, koop_smem(n, G), st>>>(r, atwo, aj, ncore, G, kind, f, c, ct,
                                                                                  flag.p);
    g_launches.fetch_add(2, std::memory_order_relaxed);
}
void launch_bdmat(const Rdm &r, const double *atwo, const double *aj, int ncore, double *f, double *d, double *dt,
                  cudaStream_t st) {
    k_koop_d<<<dim3(r.n * r.n, r.M), 256, 0, st>>>(r, atwo, aj, ncore, f, d, dt);
    g_launches.fetch_add(1, std::memory_order_relaxed);
}

}  // namespace nvpt

// The Koopmans matrices of koop_matrices_ctl, bbmat and bcmat
// (src/koop_matrices.F90:16-591, src/koopro4QD.F90:4231-4397) from one n^7
// contraction.
//
// The reference's builders sum sixteen different contractions of the 3-RDM with
// the active integrals.  For RDMs and integrals with their physical symmetries
// (see bamat_sym.cu) they are one tensor with other arguments,
//   F3[p,q;c,a] = sum_{d,f,e} Gamma3[(p,q),(d,f),(e,c)] (df|ea) + sum_d Gamma2[(p,q),(d,c)] h(d,a),
// h = aj the core-dressed one-electron operator and (df| symmetric, plus sums of
// Gamma2 and Gamma1 of order n^6:
//   J2[p,q;x,y] = sum Gamma2[(p,q),(d,f)] (df|xy) + Gamma1[p,q] h(x,y)
//   W2[p,s;x,y] = sum Gamma2[(p,f),(e,s)] (xf|ye)   Q1[p,t;x,y] = sum Gamma2[(p,f),(t,e)] (xf|ye)
//   X2[p,q;x,y] = sum Gamma2[(p,q),(d,e)] (xd|ye)   T1[p;x,y,z] = sum_f Gamma1[p,f] (xy|zf)
//   Q2[p,c] = sum_e J2[p,e;c,e]                      G1[c,a] = sum_e J2[e,c;e,a]
//   Y[c,a] = G1[c,a] - 2 sum Gamma1[d,f] (df|ca) + sum Gamma1[d,f] (cd|fa) - 2 h(c,a)
// 2-EA is 2-IP with the hole RDMs for Gamma3 and Gamma2; written out in Gamma they
// give the same sums again (f3r, q1r below).  k_ks_out holds the resulting
// formulas; tests/test_koop_sym.py evaluates them in numpy against the reference's
// loops.
//
// As in bamat_sym.cu a state whose inputs lack a symmetry is flagged on the
// device, every kernel here skips it and the direct kernels (koop_kernels.cu)
// take it; they skip the others.
#include <algorithm>

#include "koop_sym.cuh"
#include "sym_check.cuh"

namespace nvpt {
namespace {

#define AT(i, j, k, l) atwo[(i) + (ll)n * ((j) + (ll)n * ((k) + (ll)n * (l)))]

struct KsScratch {
    // per call: F3's right-hand operand [(df, e) | d][a]; per state: F3, J2, W2, Q1,
    // X2, T1 (n^4 each) and Y without its G1
    double *B, *st;
    ll per;
    int n;
    __device__ __forceinline__ double *arr(int s, int k) const {
        return st + s * per + (ll)k * n * n * n * n;
    }
};
enum { kF3, kJ2, kW2, kQ1, kX2, kT1, kY };

// Checks and operands; the threads of a state (blockIdx.y) loop over its n^6 elements.
__global__ void __launch_bounds__(256) k_ks_prep(Rdm r, const double *__restrict__ atwo,
                                                 const double *__restrict__ aj, int ncore, KsScratch S, int ns,
                                                 int *flag) {
    const int n = r.n, s = blockIdx.y, np = n * (n + 1) / 2;
    const ll n2 = (ll)n * n, n4 = n2 * n2, n6 = n4 * n2;
    bool raised;
    const double tol = rdm_tolerance(r, s, flag, raised);
    const ll t0 = (ll)blockIdx.x * blockDim.x + threadIdx.x, step = (ll)gridDim.x * blockDim.x;
    bool bad = false;
    if (!raised)
        for (ll t = t0; t < n6; t += step) bad = rdm_asymmetric(r, s, t, tol) || bad;
    if (bad) flag[s] = 1;
    if (blockIdx.y) return;
    for (ll t = t0; t < n4; t += step) {
        const int l = (int)(t % n), k = (int)((t / n) % n), j = (int)((t / n2) % n), i = (int)(t / (n2 * n));
        if (integral_asymmetric(atwo, n, i, j, k, l))
            for (int q = 0; q < ns; ++q) flag[q] = 1;
        if (i >= j) S.B[((ll)pidx(i, j) * n + k) * n + l] = AT(i, j, k, l);
        if (t < n2) S.B[(ll)np * n2 + t] = aj[tri_index(k + 1 + ncore, l + 1 + ncore) - 1];  // (d, a) = (k, l)
    }
}

// blockIdx.x < nf: F3 of a tile of R rows (p,q,c), all columns a: K = n np + n, the
// rows of Gamma3 affine in (d, f, e) with e the fastest index, two loads per K for
// the symmetric pair (d,f).  The other blocks: the n^6 sums, one or four threads per element
// (n = 8, the whole kernel: 31 -> 16 us with four).
// blockIdx.y: the state.
constexpr int kKsRpt = 4;
template <int kSumLanes>
__global__ void __launch_bounds__(256) k_ks_sums(Rdm r, const double *__restrict__ atwo, KsScratch S, int nf,
                                                 int R, int kc, const int *flag) {
    extern __shared__ double sm[];
    const int n = r.n, s = blockIdx.y, tid = threadIdx.x;
    if (flag[s]) return;
    const ll M = r.M, n1 = n, n2 = n1 * n, n3 = n2 * n, n4 = n3 * n, n5 = n4 * n;
    const int np = n * (n + 1) / 2;
    if (blockIdx.x >= nf) {
        // kSumLanes threads an element, e over them
        const ll t = ((ll)(blockIdx.x - nf) * 256 + tid) / kSumLanes;
        const int e0 = tid % kSumLanes;
        const bool in = t < n4;
        const ll u = in ? t : 0;
        const int d = (int)(u % n), c = (int)((u / n) % n), b = (int)((u / n2) % n), a = (int)(u / n3);
        auto d2 = [&](int i, int j, int k, int l) { return r.d2[s + M * (i + n * (j + n * (k + n * l)))]; };
        auto d1 = [&](int i, int j) { return r.d1[s + M * (i + n * j)]; };
        const double h = S.B[(ll)np * n2 + c * n + d];
        double j2 = e0 ? 0.0 : d1(a, b) * h, w2 = 0.0, q1 = 0.0, x2 = 0.0, t1 = 0.0;
        for (int e = e0; e < n; e += kSumLanes) {
            t1 = fma(d1(a, e), AT(b, c, d, e), t1);
#pragma unroll 4
            for (int f = 0; f < n; ++f) {
                const double x = AT(c, f, d, e);
                j2 = fma(d2(a, e, b, f), AT(e, f, c, d), j2);
                w2 = fma(d2(a, e, f, b), x, w2);
                q1 = fma(d2(a, b, f, e), x, q1);
                x2 = fma(d2(a, f, b, e), x, x2);
            }
        }
        auto sum = [](double v) {
            for (int o = kSumLanes / 2; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
            return v;
        };
        j2 = sum(j2); w2 = sum(w2); q1 = sum(q1); x2 = sum(x2); t1 = sum(t1);
        if (in && e0 == 0) {
            S.arr(s, kJ2)[t] = j2;
            S.arr(s, kW2)[t] = w2;
            S.arr(s, kQ1)[t] = q1;
            S.arr(s, kX2)[t] = x2;
            S.arr(s, kT1)[t] = t1;
        }
        if (__any_sync(0xffffffffu, t < n2)) {  // a = b = 0
            double y = e0 ? 0.0 : -2.0 * h;
            for (int e = e0; e < n; e += kSumLanes)
                for (int f = 0; f < n; ++f) y += d1(e, f) * (AT(c, f, d, e) - 2.0 * AT(e, f, c, d));
            y = sum(y);
            if (t < n2 && e0 == 0) S.arr(s, kY)[t] = y;
        }
        return;
    }
    const int lda = R | 1, K = n * np + n, row0 = blockIdx.x * R, rows = min(R, (int)n3 - row0);
    double *A = sm, *B = sm + kc * lda;
    const int groups = 256 / n, rpt = (R + groups - 1) / groups;
    const int slices = rpt == 1 ? 256 / (R * n) : 1, per = rpt == 1 ? R * n : 256;
    const int slice = tid / per, q = tid % per, col = q % n, grp = q / n;
    const bool live = slice < slices && grp < groups && (rpt > 1 || grp < R);
    double acc[kKsRpt] = {};
    for (int k0 = 0; k0 < K; k0 += kc) {
        const int nk = min(kc, K - k0);
        for (int i = tid; i < nk * R; i += 256) {
            const int kk = i % nk, row = i / nk, k = k0 + kk, rw = row0 + min(row, rows - 1);
            const int c = rw % n, qq = (rw / n) % n, p = rw / (n * n);
            double v;
            if (k < n * np) {  // Gamma3[(e,c),(d,f),(p,q)]
                const int e = k % n;
                int d, f;
                unpair(k / n, d, f);
                const double *x = r.d3 + s + M * (e + n2 * p + n3 * c + n5 * qq);
                v = x[M * (n1 * d + n4 * f)];
                if (d != f) v += x[M * (n1 * f + n4 * d)];
            } else {
                v = r.d2[s + M * (p + n * (k - n * np + n * (qq + n * c)))];
            }
            A[kk * lda + row] = v;
        }
        for (int i = tid; i < nk * n; i += 256) B[i] = S.B[(ll)k0 * n + i];
        __syncthreads();
        if (live) {
            if (rpt == 1) {
                for (int kk = slice; kk < nk; kk += slices) acc[0] = fma(A[kk * lda + grp], B[kk * n + col], acc[0]);
            } else {
#pragma unroll 4
                for (int kk = 0; kk < nk; ++kk) {
                    const double b = B[kk * n + col];
#pragma unroll
                    for (int i = 0; i < kKsRpt; ++i)
                        if (i < rpt) acc[i] = fma(A[kk * lda + min(grp + i * groups, R - 1)], b, acc[i]);
                }
            }
        }
        __syncthreads();
    }
    double *F = S.arr(s, kF3) + (ll)row0 * n;
    if (slices > 1) {  // slices in order: a fixed sum
        for (int sl = 0; sl < slices; ++sl) {
            if (live && slice == sl) A[grp * n + col] = sl ? A[grp * n + col] + acc[0] : acc[0];
            __syncthreads();
        }
        if (live && slice == 0 && grp < rows) F[grp * n + col] = A[grp * n + col];
    } else if (live) {
#pragma unroll
        for (int i = 0; i < kKsRpt; ++i)
            if (i < rpt && grp + i * groups < rows) F[(grp + i * groups) * n + col] = acc[i];
    }
}

// The matrices, a thread per (s, i, j, k, l), i fastest.  kind 0: ipko2, eako2, gk0pa,
// gk0pd, hrdm2; 1: bmat, btmat; 2: cmat, ctmat.
struct KsOut {
    double *p[5];
};
__global__ void __launch_bounds__(256) k_ks_out(Rdm r, const double *__restrict__ atwo, KsScratch S, int kind,
                                                KsOut out, const int *flag) {
    const int n = r.n, s = blockIdx.y;
    if (flag[s]) return;
    const ll n2 = (ll)n * n, n4 = n2 * n2, M = r.M;
    const ll t = (ll)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= n4) return;
    const int i = (int)(t % n), j = (int)((t / n) % n), k = (int)((t / n2) % n), l = (int)(t / (n2 * n));
    auto at = [&](int which, int a, int b, int c, int d) { return S.arr(s, which)[((ll)(a * n + b) * n + c) * n + d]; };
    auto q2 = [&](int p, int c) {
        double v = 0.0;
        for (int e = 0; e < n; ++e) v += at(kJ2, p, e, c, e);
        return v;
    };
    auto g1 = [&](int c, int a) {
        double v = 0.0;
        for (int e = 0; e < n; ++e) v += at(kJ2, e, c, e, a);
        return v;
    };
    const ll o = s + M * t;
    if (kind == 0) {
        const int p = i, q = j, a = k, b = l;  // 2-IP, 2-EA: (ap,bp,a,b); 0': (bp,ap,a,b)
        out.p[0][o] = -at(kF3, b, q, p, a) - at(kF3, a, p, q, b) - at(kQ1, p, q, a, b);
        auto y = [&](int u, int v) { return S.arr(s, kY)[u * n + v] + g1(u, v); };
        auto f3r = [&](int p, int q, int c, int a) {  // F3 of the holes
            double v = 2.0 * (at(kJ2, p, q, c, a) + at(kT1, c, q, p, a) + at(kT1, p, c, a, q) + at(kT1, q, c, a, p) +
                              AT(c, p, q, a)) - 4.0 * AT(q, p, c, a) - at(kF3, p, q, c, a) - at(kJ2, p, c, q, a) -
                       at(kW2, p, c, q, a) - at(kX2, p, q, a, c) - at(kQ1, q, c, p, a) - at(kT1, p, q, a, c) -
                       at(kT1, q, c, p, a) - at(kT1, c, q, a, p);
            if (p == q) v += 2.0 * y(c, a);
            if (c == p) v -= y(q, a);
            return v;
        };
        const double q1r = at(kQ1, p, q, a, b) + at(kT1, q, b, p, a) + at(kT1, p, a, q, b) + 4.0 * AT(a, p, b, q) -
                           2.0 * (at(kT1, q, a, p, b) + at(kT1, p, b, q, a) + AT(a, q, b, p));
        out.p[1][o] = -f3r(b, q, p, a) - f3r(a, p, q, b) - q1r;
        double A = at(kF3, p, q, b, a) - at(kF3, q, p, a, b) + at(kJ2, p, b, q, a) + at(kW2, p, b, q, a) -
                   at(kQ1, p, a, q, b);
        double D = at(kF3, q, a, p, b) - at(kF3, p, b, q, a) + 2.0 * at(kJ2, p, b, q, a) - at(kX2, p, b, a, q) +
                   at(kQ1, a, p, q, b);
        if (q == a) {
            const double x = q2(p, b);
            A -= x;
            D -= 2.0 * x;
        }
        out.p[2][o] = 2.0 * A;
        out.p[3][o] = D;
        out.p[4][o] = r.ro2t(p + 1, q + 1, a + 1, b + 1, s + 1);
    } else if (kind == 1) {
        const int p = i, q = j, c = k, a = l;  // (ap,bp,cp,a)
        double B = at(kF3, p, c, q, a) + at(kQ1, c, q, p, a);
        if (p == q) B += q2(c, a);
        out.p[0][o] = -B;
        out.p[1][o] = 2.0 * (at(kJ2, c, p, a, q) + at(kT1, c, a, q, p)) - at(kT1, c, a, p, q) - at(kF3, c, p, q, a) -
                      at(kX2, c, p, a, q) - at(kW2, c, q, p, a) - at(kJ2, c, q, p, a);
    } else {
        const int q = i, a = j, b = k, c = l;  // (ap,a,b,c)
        double C = at(kF3, q, b, c, a) - at(kF3, b, q, a, c) - at(kF3, c, a, q, b) - at(kQ1, q, a, b, c);
        double T = at(kF3, q, b, a, c) - at(kF3, b, q, c, a) - at(kF3, a, c, q, b) - at(kJ2, b, c, q, a) -
                   at(kW2, b, c, q, a) + at(kQ1, b, a, q, c) - at(kX2, a, c, b, q) - at(kQ1, c, q, a, b) +
                   2.0 * (at(kJ2, a, c, b, q) + at(kT1, c, b, q, a)) - at(kT1, c, q, a, b);
        if (a == b) C -= q2(q, c);
        if (q == a) T += q2(b, c) - g1(c, b);
        if (b == q) T += 2.0 * (g1(c, a) - q2(a, c));
        out.p[0][o] = C;
        out.p[1][o] = T;
    }
}
#undef AT

}  // namespace

// Four threads an element of the n^6 sums up to this many elements, one above: four fill
// the chip, and read Gamma2 across its stride.  The kernel with four / one thread, us:
// n = 8 16 / 31, n = 11 51 / 79, n = 13 140 / 150, n = 13 with two states 305 / 238.
constexpr ll kSumLanesMost = 32768;

int launch_koop_sym(const Rdm &r, const double *atwo, const double *aj, int ncore, int kind, double *const out[5],
                    int *flag, cudaStream_t st) {
    const int n = r.n, np = n * (n + 1) / 2;
    const ll n2 = (ll)n * n, n3 = n2 * n, n4 = n2 * n2, n6 = n4 * n2;
    KsScratch S;
    S.n = n;
    S.per = 6 * n4 + n2;
    const ll bsz = np * n2 + n2;
    double *w = nullptr;
    if (cudaMallocAsync((void **)&w, sizeof(double) * (size_t)(bsz + r.M * S.per), st) != cudaSuccess) return 2;
    S.B = w;
    S.st = w + bsz;
    KsOut o{};
    for (int i = 0; i < 5; ++i) o.p[i] = out[i];
    const int ns = r.M;
    k_ks_prep<<<dim3((unsigned)std::min<ll>((n6 + 255) / 256, std::max(1, 2432 / ns)), ns), 256, 0, st>>>(
        r, atwo, aj, ncore, S, ns, flag);
    // rows per tile: enough tiles for the chip, at most kKsRpt rows per thread
    const int most = std::min<int>(32, kKsRpt * (256 / n));
    const int R = (int)std::max<ll>(std::min<ll>(most, n3 * ns / 304), std::min(4, most));
    const int kc = std::max(32, std::min(256, 2048 / R)), nf = (int)((n3 + R - 1) / R);
    const size_t smem = sizeof(double) * (size_t)std::max(kc * (R | 1) + kc * n, R * n);
    const int lanes = n4 * ns <= kSumLanesMost ? 4 : 1;
    const dim3 g((unsigned)(nf + (lanes * n4 + 255) / 256), ns);
    if (lanes == 4) k_ks_sums<4><<<g, 256, smem, st>>>(r, atwo, S, nf, R, kc, flag);
    else k_ks_sums<1><<<g, 256, smem, st>>>(r, atwo, S, nf, R, kc, flag);
    k_ks_out<<<dim3((unsigned)((n4 + 255) / 256), ns), 256, 0, st>>>(r, atwo, S, kind, o, flag);
    g_launches.fetch_add(3, std::memory_order_relaxed);
    cudaFreeAsync(w, st);
    return 0;
}

}  // namespace nvpt

// Implementation of the device tensor toolkit (see s2_tensor.cuh).
#include "s2_tensor.cuh"

#include <algorithm>
#include <cmath>

#include "band.cuh"
#include "ozaki.cuh"
#include "spd.cuh"

namespace nvpt {
namespace s2 {

namespace {
constexpr int TPB = 256;
inline unsigned nblk(long long n) { return (unsigned)((n + TPB - 1) / TPB); }

struct PermArgs {
    int nd;
    long long shape[6];
    long long stride[6];  // input stride of each output axis
    long long off;
};

__global__ void k_permute(const double *__restrict__ in, double *__restrict__ out, PermArgs a, long long total,
                          double alpha, int acc) {
    long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= total) return;
    long long x = t, src = a.off;
    for (int k = a.nd - 1; k >= 0; --k) {
        long long i = x % a.shape[k];
        x /= a.shape[k];
        src += i * a.stride[k];
    }
    double v = alpha * in[src];
    out[t] = acc ? out[t] + v : v;
}

__global__ void k_fill(double *p, long long n, double v) {
    long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t < n) p[t] = v;
}

__global__ void k_axpby(long long n, double a, const double *x, double b, const double *y, double *o) {
    long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t < n) o[t] = a * x[t] + b * (y ? y[t] : 0.0);
}

__global__ void k_symm_upper(const double *A, long long n, double *o) {
    long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= n * n) return;
    long long r = t / n, c = t % n;
    o[t] = r <= c ? A[r * n + c] : A[c * n + r];
}

// qdnevpt-local accessors, C-ordered tensors (index arithmetic only).
__global__ void k_ee2L(const double *taa, const double *dal, int n, double *o) {
    long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    long long n2 = (long long)n * n;
    if (t >= n2 * n2) return;
    int d = t % n, c = (t / n) % n, b = (t / n2) % n, a = (int)(t / (n2 * n));
    // ee2(a,b,c,d) = taa(b,d,a,c) + [b==c] dal(d,a)
    double v = taa[((long long)(b * n + d) * n + a) * n + c];
    if (b == c) v += dal[d * n + a];
    o[t] = v;
}

__global__ void k_eee2L(const double *daaa, const double *taa, const double *dal, int n, double *o) {
    long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    long long n2 = (long long)n * n, n3 = n2 * n;
    if (t >= n3 * n3) return;
    long long x = t;
    int f = x % n; x /= n;
    int e = x % n; x /= n;
    int d = x % n; x /= n;
    int c = x % n; x /= n;
    int b = x % n; x /= n;
    int a = (int)x;
    auto D2 = [&](int i, int j, int k, int l) { return taa[((long long)(i * n + j) * n + k) * n + l]; };
    // eee2(a,b,c,d,e,f) = daaa(b,d,f,a,c,e) + [e==d] taa(b,f,a,c) + [e==b] taa(f,d,a,c)
    //                     + [b==c] taa(d,f,a,e) + [b==c][e==d] dal(f,a)
    double v = daaa[((((((long long)b * n + d) * n + f) * n + a) * n + c) * n) + e];
    if (e == d) v += D2(b, f, a, c);
    if (e == b) v += D2(f, d, a, c);
    if (b == c) v += D2(d, f, a, e);
    if (b == c && e == d) v += dal[f * n + a];
    o[t] = v;
}

__global__ void k_eee2tL(const double *E3, const double *E2, int n, double *o) {
    long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    long long n2 = (long long)n * n, n3 = n2 * n;
    if (t >= n3 * n3) return;
    long long x = t;
    int f = x % n; x /= n;
    int e = x % n; x /= n;
    int d = x % n; x /= n;
    int c = x % n; x /= n;
    int b = x % n; x /= n;
    int a = (int)x;
    // eee2t(a,b,c,d,e,f) = -eee2(a,b,d,c,e,f) + [c==d] 2 ee2(a,b,e,f)
    double v = -E3[(((((long long)a * n + b) * n + d) * n + c) * n + e) * n + f];
    if (c == d) v += 2.0 * E2[((long long)(a * n + b) * n + e) * n + f];
    o[t] = v;
}

__global__ void k_ee2trL(const double *E2, const double *dal, int n, double *o) {
    long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    long long n2 = (long long)n * n;
    if (t >= n2 * n2) return;
    int d = t % n, c = (t / n) % n, b = (t / n2) % n, a = (int)(t / (n2 * n));
    // ee2tr(a,b,c,d) = -ee2(a,b,d,c) + [c==d] 2 dal(b,a)
    double v = -E2[((long long)(a * n + b) * n + d) * n + c];
    if (c == d) v += 2.0 * dal[b * n + a];
    o[t] = v;
}

__global__ void k_ee2tlL(const double *E2, const double *dal, int n, double *o) {
    long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    long long n2 = (long long)n * n;
    if (t >= n2 * n2) return;
    int d = t % n, c = (t / n) % n, b = (t / n2) % n, a = (int)(t / (n2 * n));
    // ee2tl(a,b,c,d) = -ee2(b,a,c,d) + [a==b] 2 dal(d,c)
    double v = -E2[((long long)(b * n + a) * n + c) * n + d];
    if (a == b) v += 2.0 * dal[d * n + c];
    o[t] = v;
}

__global__ void k_ro2toff(const double *d2, const double *d1, int n, double *o) {
    long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    long long n2 = (long long)n * n;
    if (t >= n2 * n2) return;
    int b = t % n, a = (t / n) % n, bp = (t / n2) % n, ap = (int)(t / (n2 * n));
    double v = d2[t];
    if (ap == a) v -= 2.0 * d1[bp * n + b];
    if (bp == b) v -= 2.0 * d1[ap * n + a];
    if (ap == b) v += d1[bp * n + a];
    if (bp == a) v += d1[ap * n + b];
    o[t] = v;
}

__global__ void k_add_diag_pairs(double *T4, int n, int pos1, int pos2, const double *M2, int transM, double alpha) {
    // For a 4-index tensor T[i0,i1,i2,i3]: where i_pos1 == i_pos2, add
    // alpha * M[other indices in order] (transposed if transM).
    long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    long long n2 = (long long)n * n;
    if (t >= n2 * n2) return;
    int idx[4] = {(int)(t / (n2 * n)), (int)((t / n2) % n), (int)((t / n) % n), (int)(t % n)};
    if (idx[pos1] != idx[pos2]) return;
    int o[2], k = 0;
    for (int q = 0; q < 4; ++q)
        if (q != pos1 && q != pos2) o[k++] = idx[q];
    T4[t] += alpha * (transM ? M2[o[1] * n + o[0]] : M2[o[0] * n + o[1]]);
}
}  // namespace

T alloc_v(Ctx &c, const std::vector<long long> &shape, bool zero) {
    T t;
    t.st = c.st;
    t.nd = (int)shape.size();
    for (int i = 0; i < t.nd; ++i) t.sh[i] = shape[i];
    long long n = t.size();
    const size_t bytes = sizeof(double) * (size_t)(n > 0 ? n : 1);
    if (c.arena && bytes <= Arena::kMost) {
        t.p = (double *)c.arena->take(bytes, c.st, t.cls);
        t.arena = c.arena;
    } else {
        ck(cudaMallocAsync((void **)&t.p, bytes, c.st), "cudaMallocAsync");
    }
    if (zero) ck(cudaMemsetAsync(t.p, 0, sizeof(double) * (size_t)(n > 0 ? n : 1), c.st), "memset");
    return t;
}

T alloc(Ctx &c, std::initializer_list<long long> shape, bool zero) {
    return alloc_v(c, std::vector<long long>(shape), zero);
}

void gather(Ctx &c, const double *in, long long off, const std::vector<long long> &shape,
            const std::vector<long long> &stride, double *out, double alpha, bool accumulate) {
    PermArgs a;
    a.nd = (int)shape.size();
    a.off = off;
    long long total = 1;
    for (int k = 0; k < a.nd; ++k) {
        a.shape[k] = shape[k];
        a.stride[k] = stride[k];
        total *= shape[k];
    }
    if (total == 0) return;
    k_permute<<<nblk(total), TPB, 0, c.st>>>(in, out, a, total, alpha, accumulate ? 1 : 0);
    g_launches.fetch_add(1, std::memory_order_relaxed);
    ck(cudaGetLastError(), "permute launch");
}

void permute(Ctx &c, const double *in, const std::vector<long long> &in_shape, const std::vector<int> &axes,
             double *out, double alpha, bool accumulate) {
    int nd = (int)in_shape.size();
    std::vector<long long> istr(nd);
    long long s = 1;
    for (int k = nd - 1; k >= 0; --k) {
        istr[k] = s;
        s *= in_shape[k];
    }
    std::vector<long long> shape(nd), stride(nd);
    for (int k = 0; k < nd; ++k) {
        shape[k] = in_shape[axes[k]];
        stride[k] = istr[axes[k]];
    }
    gather(c, in, 0, shape, stride, out, alpha, accumulate);
}

T permuted(Ctx &c, const T &in, const std::vector<int> &axes, double alpha) {
    std::vector<long long> ish(in.sh.begin(), in.sh.begin() + in.nd), osh(in.nd);
    for (int k = 0; k < in.nd; ++k) osh[k] = ish[axes[k]];
    T out = alloc_v(c, osh, false);
    permute(c, in.p, ish, axes, out.p, alpha, false);
    return out;
}

namespace {
// Products big enough to pay for the digit splits; alpha = +-2^e.  A product
// with few rows runs transposed (its columns fill the 128-row tiles).
bool split_product(const Ctx &c, long long m, long long n, long long k, double alpha) {
    if (!c.split || k < 64 || k > oz::kWideMaxK) return false;
    if (!((m >= 64 && n >= 16) || (m >= 16 && n >= 128))) return false;
    if ((double)m * (double)n * (double)k < 6.7e7) return false;
    int e = 0;
    return std::frexp(std::fabs(alpha), &e) == 0.5;
}
void split_gemm(Ctx &c, const oz::WideGemm &g) {
    void *w = nullptr;
    ck(cudaMallocAsync(&w, oz::oz_wide_bytes(g.m, g.n, g.K), c.st), "cudaMallocAsync");
    const int rc = oz::oz_gemm_wide(g, w, c.oz_err, c.st);
    cudaFreeAsync(w, c.st);
    if (rc) throw Error(2, "split-precision product failed to launch");
}
}  // namespace

void gemm(Ctx &c, bool ta, bool tb, long long m, long long n, long long k, double alpha, const double *A, long long lda,
          const double *B, long long ldb, double beta, double *C, long long ldc) {
    if (m == 0 || n == 0) return;
    if (split_product(c, m, n, k, alpha)) {
        oz::WideGemm g;
        g.K = (int)k;
        g.alpha = alpha; g.beta = beta; g.C = C; g.ldc = ldc;
        if (m >= 64) {
            g.m = m; g.n = n;
            g.A = A; g.a_r = ta ? 1 : lda; g.a_k = ta ? lda : 1;
            g.B = B; g.b_c = tb ? ldb : 1; g.b_k = tb ? 1 : ldb;
        } else {  // C^T = op(B)^T op(A)^T: rows of the product are the columns of C
            g.m = n; g.n = m;
            g.A = B; g.a_r = tb ? ldb : 1; g.a_k = tb ? 1 : ldb;
            g.B = A; g.b_c = ta ? 1 : lda; g.b_k = ta ? lda : 1;
            g.c_trans = true;
        }
        split_gemm(c, g);
        return;
    }
    // Row-major C = op(A) op(B)  <=>  column-major C^T = op(B)^T op(A)^T.
    ck(cublasDgemm(c.blas, tb ? CUBLAS_OP_T : CUBLAS_OP_N, ta ? CUBLAS_OP_T : CUBLAS_OP_N, (int)n, (int)m, (int)k,
                   &alpha, B, (int)ldb, A, (int)lda, &beta, C, (int)ldc),
       "cublasDgemm");
}

void gemm_batched(Ctx &c, bool ta, bool tb, long long m, long long n, long long k, double alpha, const double *A,
                  long long lda, long long sA, const double *B, long long ldb, long long sB, double beta, double *C,
                  long long ldc, long long sC, long long batch) {
    if (m == 0 || n == 0 || batch == 0) return;
    ck(cublasDgemmStridedBatched(c.blas, tb ? CUBLAS_OP_T : CUBLAS_OP_N, ta ? CUBLAS_OP_T : CUBLAS_OP_N, (int)n,
                                 (int)m, (int)k, &alpha, B, (int)ldb, sB, A, (int)lda, sA, &beta, C, (int)ldc, sC,
                                 (int)batch),
       "cublasDgemmStridedBatched");
}

void symmetrize_upper(Ctx &c, const double *A, long long n, double *out) {
    k_symm_upper<<<nblk(n * n), TPB, 0, c.st>>>(A, n, out);
    g_launches.fetch_add(1, std::memory_order_relaxed);
}

namespace {
// cuSOLVER workspace of `count` doubles + info word, stream-ordered.
struct SolverWork {
    Ctx &c;
    T buf, inf;
    double *w = nullptr;
    int *info = nullptr;
    SolverWork(Ctx &cc, int count) : c(cc), buf(alloc(cc, {std::max(count, 1)}, false)), inf(alloc(cc, {1}, false)) {
        w = buf.p;
        info = (int *)inf.p;
    }
    int status() {
        int h = -1;
        ck(cudaMemcpyAsync(&h, info, sizeof(int), cudaMemcpyDeviceToHost, c.st), "info copy");
        ck(cudaStreamSynchronize(c.st), "solver sync");
        return h;
    }
};
}  // namespace

void eigh_upper(Ctx &c, const double *A, long long n, double *w, double *V) {
    if (n == 0) return;
    // Symmetric copy, so that the triangle cuSOLVER reads is the reference's upper one.
    symmetrize_upper(c, A, n, V);
    int lwork = 0;
    ck(cusolverDnDsyevd_bufferSize(c.sol, CUSOLVER_EIG_MODE_VECTOR, CUBLAS_FILL_MODE_UPPER, (int)n, V, (int)n, w,
                                   &lwork),
       "syevd_bufferSize");
    SolverWork sw(c, lwork);
    ck(cusolverDnDsyevd(c.sol, CUSOLVER_EIG_MODE_VECTOR, CUBLAS_FILL_MODE_UPPER, (int)n, V, (int)n, w, sw.w, lwork,
                        sw.info),
       "syevd");
    const int hinfo = sw.status();
    if (hinfo != 0) throw Error(2, "syevd failed, info=" + std::to_string(hinfo));
    // The symmetric input makes row-/column-major identical; cuSOLVER stores
    // eigenvector k as column k (column-major) = row k of the row-major array.
}

__global__ void k_add_diag(double *A, long long n, double v) {
    long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) A[i * n + i] += v;
}

__global__ void k_mirror_lower(double *o, long long m) {
    long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= m * m) return;
    long long r = t / m, col = t % m;
    if (r < col) o[t] = o[col * m + r];
}

void gram(Ctx &c, const double *X, long long Q, long long m, double *out) {
    if (m == 0) return;
    if (split_product(c, m, m, Q, 1.0)) {
        // the tiles meeting the lower triangle of out = X^T X, then mirrored
        oz::WideGemm g;
        g.m = m; g.n = m; g.K = (int)Q;
        g.A = X; g.a_r = 1; g.a_k = m;
        g.B = X; g.b_c = 1; g.b_k = m;
        g.C = out; g.ldc = m; g.lower = true;
        split_gemm(c, g);
        k_mirror_lower<<<nblk(m * m), TPB, 0, c.st>>>(out, m);
        g_launches.fetch_add(1, std::memory_order_relaxed);
        return;
    }
    const double one = 1.0, zero = 0.0;
    // column-major view: X is m x Q (ld m); C = X X^T fills the column-major
    // upper triangle = the row-major lower triangle of out
    ck(cublasDsyrk(c.blas, CUBLAS_FILL_MODE_UPPER, CUBLAS_OP_N, (int)m, (int)Q, &one, X, (int)m, &zero, out, (int)m),
       "cublasDsyrk");
    k_mirror_lower<<<nblk(m * m), TPB, 0, c.st>>>(out, m);
    g_launches.fetch_add(1, std::memory_order_relaxed);
}

int raise_dynamic_smem(const void *kernel) {
    int dev = 0, optin = 0;
    ck(cudaGetDevice(&dev), "cudaGetDevice");
    // once per device and kernel: three driver calls otherwise, in front of most launches
    static std::mutex mu;
    static std::map<std::pair<int, const void *>, int> known;
    std::lock_guard<std::mutex> g(mu);
    const auto it = known.find({dev, kernel});
    if (it != known.end()) return it->second;
    cudaFuncAttributes fa{};
    ck(cudaFuncGetAttributes(&fa, kernel), "cudaFuncGetAttributes");
    ck(cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev), "attr");
    const int lim = optin - (int)fa.sharedSizeBytes;
    ck(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, lim), "smem attr");
    known[{dev, kernel}] = lim;
    return lim;
}

bool metric_above(Ctx &c, const double *A, long long n, double thr) {
    if (n == 0) return true;
    T M = alloc(c, {n, n}, false);
    symmetrize_upper(c, A, n, M.p);
    k_add_diag<<<nblk(n), TPB, 0, c.st>>>(M.p, n, -thr);
    g_launches.fetch_add(1, std::memory_order_relaxed);
    int lwork = 0;
    ck(cusolverDnDpotrf_bufferSize(c.sol, CUBLAS_FILL_MODE_UPPER, (int)n, M.p, (int)n, &lwork), "potrf_bufferSize");
    SolverWork sw(c, lwork);
    ck(cusolverDnDpotrf(c.sol, CUBLAS_FILL_MODE_UPPER, (int)n, M.p, (int)n, sw.w, lwork, sw.info), "potrf");
    return sw.status() == 0;
}

namespace {
// A += rel * (largest diagonal element) on the diagonal; that element into *top.
__global__ void k_shift_diag(double *A, long long n, double rel, double *top) {
    __shared__ double red[TPB];
    double m = 0.0;
    for (long long i = threadIdx.x; i < n; i += TPB) m = fmax(m, A[i * n + i]);
    red[threadIdx.x] = m;
    __syncthreads();
    for (int t = 0; t < TPB; ++t) m = fmax(m, red[t]);
    for (long long i = threadIdx.x; i < n; i += TPB) A[i * n + i] += rel * m;
    if (threadIdx.x == 0) *top = m;
}

// *out += |X[r] . Y[r]|, a row a block.
__global__ void k_dot_abs(const double *X, const double *Y, long long n, double *out) {
    __shared__ double red[TPB];
    double v = 0.0;
    for (long long i = threadIdx.x; i < n; i += TPB) v = fma(X[blockIdx.x * n + i], Y[blockIdx.x * n + i], v);
    red[threadIdx.x] = v;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int t = 1; t < TPB; ++t) v += red[t];
        atomicAdd(out, fabs(v));
    }
}

// Deterministic start vectors of the inverse iteration, in [-0.5, 0.5): the outputs of
// Steele, Lea and Flood's SplitMix64 generator (OOPSLA 2014) at the element's index.
__global__ void k_start_block(double *X, long long count) {
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= count) return;
    unsigned long long z = (unsigned long long)(t + 1) * 0x9E3779B97F4A7C15ull;
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    X[t] = (double)((z ^ (z >> 31)) >> 11) * 0x1p-53 - 0.5;
}

// The null vectors of the positive semidefinite S (full storage), if its
// eigenvalues below thr are all null: N [k, n] orthonormal rows.  With delta = 1e-11 of
// the largest diagonal element, delta tr (S + delta)^-1 counts them (a kept eigenvalue
// w adds delta / w); two steps of inverse iteration on S + delta from k random vectors
// gain a factor w / delta each, and the block is orthonormalised through the inverse
// factor of its Gram matrix, twice.  Null means that the Rayleigh quotients of the block
// add up to at most 1e-12 of that element; a threshold below this line may keep such an
// eigenvalue, and its pencil is not deflated.  False if the metric is not of this
// kind.  All products and one factorisation of order n: the QR factorisations of a
// wider block that this replaces took 5 ms at order 216, latency for the most part.
bool metric_null(Ctx &c, const double *S, long long n, double thr, T &N, long long &k) {
    Ctx f = c;
    f.split = false;
    k = 0;
    const long long ld = spd_ld(n);
    T L = alloc(c, {n, n}, false), W = alloc(c, {ld, ld}, false), top = alloc(c, {1}, true);
    ck(cudaMemcpyAsync(L.p, S, sizeof(double) * n * n, cudaMemcpyDeviceToDevice, c.st), "copy");
    k_shift_diag<<<1, TPB, 0, c.st>>>(L.p, n, 1e-11, top.p);
    g_launches.fetch_add(1, std::memory_order_relaxed);
    double tr = 0.0, st[2], big = 0.0, shifted = 0.0;
    ck(cudaMemcpyAsync(&big, top.p, sizeof(double), cudaMemcpyDeviceToHost, c.st), "diagonal");
    if (!spd_inverse_factor(c, L.p, n, W.p, tr, shifted) || !(big > 0.0)) return false;  // synchronises
    const double null = 1e-12 * big;
    if (!(thr >= null)) return false;
    const double count = tr * 1e-11 * big;
    if (!(count < (double)n)) return false;
    k = std::llround(count);
    if (k < 1 || 2 * k > n || std::fabs(count - (double)k) > 0.1) return false;
    T X = alloc(c, {k, n}, false), Y = alloc(c, {k, n}, false), G = alloc(c, {k, k}, false);
    const long long lk = spd_ld(k);
    T R = alloc(c, {lk, lk}, false), stat = alloc(c, {2}, true);
    k_start_block<<<nblk(k * n), TPB, 0, c.st>>>(X.p, k * n);
    g_launches.fetch_add(1, std::memory_order_relaxed);
    for (int it = 0; it < 2; ++it) {
        gemm(f, false, true, k, n, n, 1.0, X.p, n, W.p, ld, 0.0, Y.p, n);
        gemm(f, false, false, k, n, n, 1.0, Y.p, n, W.p, ld, 0.0, X.p, n);
    }
    for (int it = 0; it < 2; ++it) {
        gemm(f, false, true, k, k, n, 1.0, X.p, n, X.p, n, 0.0, G.p, k);
        spd_inverse_factor_async(c, G.p, k, R.p, stat.p, false);
        gemm(f, false, false, k, n, k, 1.0, R.p, lk, X.p, n, 0.0, Y.p, n);
        std::swap(X, Y);
    }
    // the Rayleigh quotients, none negative but for rounding: their sum bounds each
    gemm(f, false, false, k, n, n, 1.0, X.p, n, S, n, 0.0, Y.p, n);
    ck(cudaMemsetAsync(top.p, 0, sizeof(double), c.st), "memset");
    k_dot_abs<<<(unsigned)k, TPB, 0, c.st>>>(X.p, Y.p, n, top.p);
    g_launches.fetch_add(1, std::memory_order_relaxed);
    double w = 0.0;
    ck(cudaMemcpyAsync(&w, top.p, sizeof(double), cudaMemcpyDeviceToHost, c.st), "quotients");
    ck(cudaMemcpyAsync(st, stat.p, sizeof(st), cudaMemcpyDeviceToHost, c.st), "status");
    ck(cudaStreamSynchronize(c.st), "sync");
    if (spd_failed(st) || !(w <= null)) return false;
    N = std::move(X);
    return true;
}
}  // namespace

bool pencil_tridiag(Ctx &c, const double *K, const double *S, long long n, double thr, PencilTridiag &P) {
    P.n = n;
    P.k = 0;
    if (n == 0) return true;
    const long long ld = spd_ld(n);
    P.W = alloc(c, {ld, ld}, false);
    ProfSpan sp;
    // Every eigenvalue above thr, by the smallest one's bounds 1 / tr S^-1 and n / tr S^-1
    // where they decide (the factor 2 is for the rounding of tr), else by S - thr.  null:
    // whether some may be null, which none is while 1 / tr S^-1 is above that line.
    bool null = false;
    auto factor = [&](const double *M) {
        double tr = 0.0, top = 0.0;
        sp.begin("pencil_potrf", c.st, 0);
        const bool ok = spd_inverse_factor(c, M, n, P.W.p, tr, top);
        sp.end();
        null = !ok || !(2e-12 * top * tr < 1.0);
        if (!ok || tr * thr > 2.0 * n) return false;
        return (thr >= 0.0 && tr * thr <= 0.999) || metric_above(c, M, n, thr);
    };
    T S2, K2;
    const double *Kp = K;
    if (!factor(S)) {
        if (!null) return false;
        S2 = alloc(c, {n, n}, false);
        symmetrize_upper(c, S, n, S2.p);
        if (!metric_null(c, S2.p, n, thr, P.N, P.k)) return false;
        const long long k = P.k;
        // S + N^T N, then every eigenvalue has to be above the threshold
        gemm(c, true, false, n, n, k, 1.0, P.N.p, n, P.N.p, n, 1.0, S2.p, n);
        if (!factor(S2.p)) return false;
        // P K P + N^T N = K - N^T G - G^T N + N^T (1 + G N^T) N with G = N K
        K2 = alloc(c, {n, n}, false);
        symmetrize_upper(c, K, n, K2.p);
        T G = alloc(c, {k, n}, false), M = alloc(c, {k, k}, false), Q = alloc(c, {k, n}, false);
        gemm(c, false, false, k, n, n, 1.0, P.N.p, n, K2.p, n, 0.0, G.p, n);
        gemm(c, false, true, k, k, n, 1.0, G.p, n, P.N.p, n, 0.0, M.p, k);
        k_add_diag<<<nblk(k), TPB, 0, c.st>>>(M.p, k, 1.0);
        g_launches.fetch_add(1, std::memory_order_relaxed);
        gemm(c, false, false, k, n, k, 0.5, M.p, k, P.N.p, n, 0.0, Q.p, n);
        axpby(c, k * n, 1.0, Q.p, -1.0, G.p, Q.p);  // Q = (1 + G N^T) N / 2 - G
        gemm(c, true, false, n, n, k, 1.0, P.N.p, n, Q.p, n, 1.0, K2.p, n);
        gemm(c, true, false, n, n, k, 1.0, Q.p, n, P.N.p, n, 1.0, K2.p, n);
        Kp = K2.p;
    }
    S2.release();
    T A = alloc(c, {n, n}, false);
    sp.begin("pencil_reduce", c.st, 0);
    spd_congruence(c, P.W.p, Kp, n, A.p);
    sp.end();
    K2.release();
    sp.begin("pencil_sytrd", c.st, 0);
    const bool tri = n <= kTriMost;
    const int first = tri ? 1 : kBand;
    P.V = alloc(c, {wy_rows(n, first), kBand}, false);
    P.Tm = alloc(c, {wy_panels(n, first), kBand, kBand}, false);
    int rc;
    if (tri) {
        P.d = alloc(c, {n}, false);
        P.e = alloc(c, {n}, false);
        rc = tri_reduce(c, A.p, n, P.d.p, P.e.p, P.V.p, P.Tm.p);
    } else {
        P.AB = alloc(c, {kBand + 1, n}, false);
        rc = band_reduce(c, A.p, n, P.V.p, P.Tm.p, P.AB.p);
    }
    sp.end();
    if (rc != 0) throw Error(4, "pencil reduction: a device wait timed out");
    return true;
}

void pencil_rhs(Ctx &c, const PencilTridiag &P, double *Y, long long m) {
    if (P.n == 0 || m == 0) return;
    ProfSpan sp;
    sp.begin("pencil_rhs", c.st, 0);
    Ctx f = c;
    f.split = false;
    T Z = alloc(c, {m, P.n}, false);
    ck(cudaMemcpyAsync(Z.p, Y, sizeof(double) * m * P.n, cudaMemcpyDeviceToDevice, c.st), "copy");
    if (P.k) {  // rows without their components along the null vectors
        T a = alloc(c, {m, P.k}, false);
        gemm(c, false, true, m, P.k, P.n, 1.0, Y, P.n, P.N.p, P.n, 0.0, a.p, P.k);
        gemm(c, false, false, m, P.n, P.k, -1.0, a.p, P.k, P.N.p, P.n, 1.0, Z.p, P.n);
    }
    gemm(f, false, true, m, P.n, P.n, 1.0, Z.p, P.n, P.W.p, spd_ld(P.n), 0.0, Y, P.n);
    wy_apply(c, P.n, P.n <= kTriMost ? 1 : kBand, P.V.p, P.Tm.p, Y, m, true);
    sp.end();
}

void pencil_back(Ctx &c, const PencilTridiag &P, double *X, long long m) {
    if (P.n == 0 || m == 0) return;
    ProfSpan sp;
    sp.begin("pencil_rhs", c.st, 0);
    Ctx f = c;
    f.split = false;
    wy_apply(c, P.n, P.n <= kTriMost ? 1 : kBand, P.V.p, P.Tm.p, X, m, false);
    T Z = alloc(c, {m, P.n}, false);
    ck(cudaMemcpyAsync(Z.p, X, sizeof(double) * m * P.n, cudaMemcpyDeviceToDevice, c.st), "copy");
    gemm(f, false, false, m, P.n, P.n, 1.0, Z.p, P.n, P.W.p, spd_ld(P.n), 0.0, X, P.n);
    sp.end();
}

void build_ee2L(Ctx &c, const double *taa, const double *dal, int n, double *out) {
    long long N = (long long)n * n * n * n;
    k_ee2L<<<nblk(N), TPB, 0, c.st>>>(taa, dal, n, out);
    g_launches.fetch_add(1, std::memory_order_relaxed);
}
void build_eee2L(Ctx &c, const double *daaa, const double *taa, const double *dal, int n, double *out) {
    long long N = (long long)n * n * n * n * n * n;
    k_eee2L<<<nblk(N), TPB, 0, c.st>>>(daaa, taa, dal, n, out);
    g_launches.fetch_add(1, std::memory_order_relaxed);
}
void build_eee2tL(Ctx &c, const double *E3, const double *E2, int n, double *out) {
    long long N = (long long)n * n * n * n * n * n;
    k_eee2tL<<<nblk(N), TPB, 0, c.st>>>(E3, E2, n, out);
    g_launches.fetch_add(1, std::memory_order_relaxed);
}
void build_ee2trL(Ctx &c, const double *E2, const double *dal, int n, double *out) {
    long long N = (long long)n * n * n * n;
    k_ee2trL<<<nblk(N), TPB, 0, c.st>>>(E2, dal, n, out);
    g_launches.fetch_add(1, std::memory_order_relaxed);
}
void build_ee2tlL(Ctx &c, const double *E2, const double *dal, int n, double *out) {
    long long N = (long long)n * n * n * n;
    k_ee2tlL<<<nblk(N), TPB, 0, c.st>>>(E2, dal, n, out);
    g_launches.fetch_add(1, std::memory_order_relaxed);
}
void build_ro2toff(Ctx &c, const double *taa, const double *dal, int n, double *out) {
    long long N = (long long)n * n * n * n;
    k_ro2toff<<<nblk(N), TPB, 0, c.st>>>(taa, dal, n, out);
    g_launches.fetch_add(1, std::memory_order_relaxed);
}
void axpby(Ctx &c, long long count, double a, const double *x, double b, const double *y, double *out) {
    k_axpby<<<nblk(count), TPB, 0, c.st>>>(count, a, x, b, y, out);
    g_launches.fetch_add(1, std::memory_order_relaxed);
}
void fill(Ctx &c, double *p, long long count, double v) {
    k_fill<<<nblk(count), TPB, 0, c.st>>>(p, count, v);
    g_launches.fetch_add(1, std::memory_order_relaxed);
}
void add_diag_pairs(Ctx &c, double *T4, int n, int pos1, int pos2, const double *M2, bool transposeM, double alpha) {
    long long N = (long long)n * n * n * n;
    k_add_diag_pairs<<<nblk(N), TPB, 0, c.st>>>(T4, n, pos1, pos2, M2, transposeM ? 1 : 0, alpha);
    g_launches.fetch_add(1, std::memory_order_relaxed);
}

}  // namespace s2
}  // namespace nvpt

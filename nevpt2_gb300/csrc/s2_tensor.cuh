// Device tensor toolkit for the NEVPT2 energy stage.
//
// Tensors are dense, C-ordered (last index fastest) FP64 arrays with up to 6
// axes.  The stage-2 algebra is expressed with a few primitives: an axis
// permutation (materialised), the accessor builders of the reference's
// qdnevpt-local normal-ordered products (src/qdnevpt.F:6448-6519), dense
// GEMMs (cuBLAS FP64, or split-precision digit products on the tensor cores
// in split mode), symmetric eigendecompositions (cuSOLVER syevd) and, for
// the order-n^3 pencils, the reduction to standard form (spd.cu) and to a band
// (band.cu).  All work of one context is enqueued on
// its stream; allocations are stream-ordered.
#pragma once
#include <cublas_v2.h>
#include <cuda_runtime.h>
#include <cusolverDn.h>

#include <array>
#include <map>
#include <mutex>
#include <stdexcept>
#include <string>
#include <vector>

#include "nvpt2_internal.h"

namespace nvpt {
namespace s2 {

struct Error : std::runtime_error {
    int code;
    Error(int c, const std::string &m) : std::runtime_error(m), code(c) {}
};

inline void ck(cudaError_t e, const char *what) {
    if (e != cudaSuccess) throw Error(e == cudaErrorMemoryAllocation ? 3 : 2, std::string(what) + ": " + cudaGetErrorString(e));
}
inline void ck(cublasStatus_t e, const char *what) {
    if (e != CUBLAS_STATUS_SUCCESS) throw Error(2, std::string(what) + ": cuBLAS status " + std::to_string((int)e));
}
inline void ck(cusolverStatus_t e, const char *what) {
    if (e != CUSOLVER_STATUS_SUCCESS) throw Error(2, std::string(what) + ": cuSOLVER status " + std::to_string((int)e));
}

// Small device blocks of one call (at most kMost bytes), carved from slabs and kept in
// per-stream free lists: a block given back on a stream is only taken again on that
// stream, so its reuse is ordered like that of a stream-ordered free.  The concurrent
// tasks of a call made thousands of driver allocations, each behind the driver's lock;
// these are a few hundred nanoseconds of host time.  Slabs go back when the call ends.
class Arena {
  public:
    static constexpr size_t kMost = 1u << 20, kSlab = 4u << 20;
    // home: where the slabs are freed, once every other stream's work has been waited for
    explicit Arena(cudaStream_t home) : home_(home) {}
    Arena(const Arena &) = delete;
    Arena &operator=(const Arena &) = delete;
    ~Arena() {
        cudaStreamSynchronize(home_);
        for (void *p : slabs_) cudaFreeAsync(p, home_);
    }
    // classes of 256 bytes * {4, 5, 6, 7} / 4 * 2^k; cls receives the block's
    void *take(size_t bytes, cudaStream_t st, int &cls) {
        size_t size = 256;
        cls = 0;
        while (size < bytes) {
            ++cls;
            size = (size_t)(64 * (4 + cls % 4)) << (cls / 4);
        }
        size = (size + 255) / 256 * 256;
        std::lock_guard<std::mutex> g(mu_);
        Lane &l = lanes_[st];
        if ((size_t)cls >= l.free.size()) l.free.resize(cls + 1);
        if (!l.free[cls].empty()) {
            void *p = l.free[cls].back();
            l.free[cls].pop_back();
            return p;
        }
        if (l.left < size) {
            void *p = nullptr;
            ck(cudaMallocAsync(&p, kSlab, st), "cudaMallocAsync");
            slabs_.push_back(p);
            l.cur = (char *)p;
            l.left = kSlab;
        }
        void *p = l.cur;
        l.cur += size;
        l.left -= size;
        return p;
    }
    void give(void *p, int cls, cudaStream_t st) {
        std::lock_guard<std::mutex> g(mu_);
        Lane &l = lanes_[st];
        if ((size_t)cls >= l.free.size()) l.free.resize(cls + 1);
        l.free[cls].push_back(p);
    }

  private:
    struct Lane {
        char *cur = nullptr;
        size_t left = 0;
        std::vector<std::vector<void *>> free;
    };
    cudaStream_t home_;
    std::mutex mu_;
    std::map<cudaStream_t, Lane> lanes_;
    std::vector<void *> slabs_;
};

// Owning device tensor (stream-ordered allocation, or a block of an arena), or a
// non-owning view of one (T::view) that never frees.
struct T {
    double *p = nullptr;
    int nd = 0;
    std::array<long long, 6> sh{{1, 1, 1, 1, 1, 1}};
    cudaStream_t st = nullptr;
    bool own = true;
    Arena *arena = nullptr;  // whose block of class cls this is
    int cls = 0;
    T() = default;
    T(const T &) = delete;
    T &operator=(const T &) = delete;
    T(T &&o) noexcept { *this = std::move(o); }
    T &operator=(T &&o) noexcept {
        release();
        p = o.p; nd = o.nd; sh = o.sh; st = o.st; own = o.own; arena = o.arena; cls = o.cls;
        o.p = nullptr;
        return *this;
    }
    ~T() { release(); }
    static T view(const T &o) {
        T v;
        v.p = o.p; v.nd = o.nd; v.sh = o.sh; v.st = o.st; v.own = false;
        return v;
    }
    void release() {
        if (p && own) {
            if (arena) arena->give(p, cls, st);
            else cudaFreeAsync(p, st);
        }
        p = nullptr;
    }
    long long size() const {
        long long s = 1;
        for (int i = 0; i < nd; ++i) s *= sh[i];
        return s;
    }
    long long dim(int i) const { return sh[i]; }
};

struct Ctx {
    cudaStream_t st;
    cublasHandle_t blas;
    cusolverDnHandle_t sol;
    // Split precision: large GEMMs (and Gram matrices) run as Ozaki digit
    // products on the tensor cores; a pipeline timeout sets *oz_err.
    bool split = false;
    int *oz_err = nullptr;
    // Polls a device-side wait (grid barrier) makes before it gives up and
    // the call reports NVPT_ETIMEDOUT; 0 = the built-in limit.
    unsigned wait_limit = 0;
    Arena *arena = nullptr;  // small allocations of the call, if any
};

T alloc(Ctx &c, std::initializer_list<long long> shape, bool zero = true);
T alloc_v(Ctx &c, const std::vector<long long> &shape, bool zero = true);
// Non-owning 1-D view helpers are plain pointers.

// out = alpha * permute(in, axes) (+ out if accumulate).  `in` has shape
// in_shape (C order); axes as numpy.transpose.
void permute(Ctx &c, const double *in, const std::vector<long long> &in_shape, const std::vector<int> &axes,
             double *out, double alpha = 1.0, bool accumulate = false);
T permuted(Ctx &c, const T &in, const std::vector<int> &axes, double alpha = 1.0);

// Gather of a strided sub-block: out[i0..] = in[off + sum i_k * stride_k],
// out C-ordered with shape `shape`.
void gather(Ctx &c, const double *in, long long off, const std::vector<long long> &shape,
            const std::vector<long long> &stride, double *out, double alpha = 1.0, bool accumulate = false);

// Row-major GEMM: C[m,n] = alpha op(A)[m,k] op(B)[k,n] + beta C.
void gemm(Ctx &c, bool ta, bool tb, long long m, long long n, long long k, double alpha, const double *A, long long lda,
          const double *B, long long ldb, double beta, double *C, long long ldc);
void gemm_batched(Ctx &c, bool ta, bool tb, long long m, long long n, long long k, double alpha, const double *A,
                  long long lda, long long sA, const double *B, long long ldb, long long sB, double beta, double *C,
                  long long ldc, long long sC, long long batch);

// Symmetric eigendecomposition of the matrix whose upper triangle (row <=
// col) is held in A (n x n, row-major), as dsyev('V','U') of the reference
// sees it.  w ascending; V[k][i] = component i of eigenvector k.
void eigh_upper(Ctx &c, const double *A, long long n, double *w, double *V);
// out[m,m] (row-major) = X^T X for X [Q, m] row-major: the symmetric rank-Q
// update (cublasDsyrk, half the flops of a GEMM) mirrored to a full matrix.
void gram(Ctx &c, const double *X, long long Q, long long m, double *out);
// True if every eigenvalue of the symmetric matrix (upper triangle of A) is
// above thr: a Cholesky factorisation of A - thr I succeeds.
bool metric_above(Ctx &c, const double *A, long long n, double thr);
// Raise kernel's dynamic shared-memory limit to the most the current device
// allows next to its static shared memory, and return that limit.  The value
// is the same for every caller, so host threads launching the kernel with
// different sizes concurrently cannot undercut one another's launches.
int raise_dynamic_smem(const void *kernel);
// Symmetric copy: out = triu(A) + triu(A,1)^T.
void symmetrize_upper(Ctx &c, const double *A, long long n, double *out);

// The pencil K v = w S v in band form, without its eigenvectors: S = L L^T (its
// symmetric view), W = L^-1, W K W^T = Q B Q^T (K's symmetric view; Householder).
// W and Q stay in the struct, which then maps right-hand sides into B's basis.
// A metric with exact null vectors (those of a spin eigenfunction) and every other
// eigenvalue above the threshold is deflated: with N its null vectors (rows, k of
// them) and P = 1 - N^T N the pencil is P K P + N^T N, S + N^T N, whose null part is
// a block of its own, and right-hand sides are projected by P.
struct PencilTridiag {
    T W;           // inverse Cholesky factor of the metric (spd.cuh)
    T V, Tm;       // W K W^T = Q B Q^T (band.cuh)
    T AB;          // B as a band, orders above kTriMost
    T d, e;        // B tridiagonal, the others
    T N;           // null vectors of the metric [k, n]
    long long n = 0, k = 0;
};
// False, with nothing kept, unless every eigenvalue of S is above thr or null; the null
// ones are at most half of them, their Rayleigh quotients add up to at most 1e-12 of the
// largest diagonal element, and thr is not below that.
bool pencil_tridiag(Ctx &c, const double *K, const double *S, long long n, double thr, PencilTridiag &P);
// Householder tridiagonalisation of the symmetric A (column-major, both triangles
// valid) in the output form of dsytrd('L'): d[n], e[n-1], tau[n-1], reflectors below
// the subdiagonal of A (tridiag.cu).  0, or 4 if a grid barrier timed out.
int sytrd_lower(Ctx &c, double *A, long long n, double *d, double *e, double *tau);
// Y <- Q^T W Y for Y column-major [n, m] (= row-major [m, n]): each row
// z of the row-major view becomes y with z^T (K + s S)^-1 z = y^T (B + s)^-1 y.
void pencil_rhs(Ctx &c, const PencilTridiag &P, double *Y, long long m);
// The inverse map of m vectors of the band's basis (columns of a
// column-major [n, m] X, in place): X <- W^T Q X.
void pencil_back(Ctx &c, const PencilTridiag &P, double *X, long long m);

// Accessor builders (C-ordered n-index tensors of one state or pair).
void build_ee2L(Ctx &c, const double *taa, const double *dal, int n, double *out);
void build_eee2L(Ctx &c, const double *daaa, const double *taa, const double *dal, int n, double *out);
void build_eee2tL(Ctx &c, const double *E3, const double *E2, int n, double *out);
void build_ee2trL(Ctx &c, const double *E2, const double *dal, int n, double *out);
void build_ee2tlL(Ctx &c, const double *E2, const double *dal, int n, double *out);
void build_ro2toff(Ctx &c, const double *taa, const double *dal, int n, double *out);

// Elementwise helpers.
void axpby(Ctx &c, long long count, double a, const double *x, double b, const double *y, double *out);
void fill(Ctx &c, double *p, long long count, double v);
void add_diag_pairs(Ctx &c, double *T4, int n, int pos1, int pos2, const double *M2, bool transposeM, double alpha);

}  // namespace s2
}  // namespace nvpt

// Band and tridiagonal forms of a symmetric matrix and resolvents in them (band.cu,
// tri.cu).
#pragma once
#include "s2_tensor.cuh"

namespace nvpt {
namespace s2 {

constexpr int kBand = 32;               // half bandwidth, and reflectors of a panel of Q
// Largest order of the tridiagonal form.  Its elimination costs O(1) a row and label where
// the band's costs 2 kBand^2, its reduction needs the matrix in shared memory.  A class
// alone, tridiagonal / band: order 128 with 1800 labels (CAS(8), 0') 8.1 / 8.9 ms, 343 and
// 512 with 12 labels (CAS(7), CAS(8), +1') 11.2 / 12.1 and 14.5 / 14.9 ms, of which 6 ms
// are not the pencil's; above 512 the products with 32 columns win over the row passes.
constexpr long long kTriMost = 512;

// Q is kept as compact WY panels of kBand reflectors; panel p acts on the rows from
// p kBand + first on (first: kBand for the band, 1 for the tridiagonal form).  V: the
// panels one after another, [rows][kBand] each; Tm [panels][kBand][kBand].
inline int wy_panels(long long n, int first) { return n - 1 > first ? (int)((n - 2 - first) / kBand) + 1 : 0; }
inline long long wy_rows(long long n, int first) {
    const long long np = wy_panels(n, first);
    return np * (n - first) - kBand * np * (np - 1) / 2;
}
// Y <- Q^T Y (forward) or Q Y for m columns (column-major, ld n).
void wy_apply(Ctx &c, long long n, int first, const double *V, const double *Tm, double *Y, long long m, bool forward);

// A (column-major n x n, both triangles valid) = Q B Q^T: AB[k][i] = B(i + k, i)
// for k <= kBand ([kBand + 1][n]); A is overwritten.  0, or 4 if a device wait timed out.
int band_reduce(Ctx &c, double *A, long long n, double *V, double *Tm, double *AB);
// A = Q T Q^T, T tridiagonal: d[n], e[n - 1]; n <= kTriMost.  0, or 4.
int tri_reduce(Ctx &c, const double *A, long long n, double *d, double *e, double *V, double *Tm);

// For each label l < L with x_l = (B + sig_l)^-1 y_l (y_l = column l of Y, row-major
// [n][ncol]): acc[0] -= y_l . x_l, acc[1] += x_l . x_l, acc[2 + k] -= y_{k+1,l} . x_l
// for k < nother (column (k + 1) L + l), rho[l nd + k] -= Y[:, dcol0 + k] . x_l, and
// x_l into column l of xout [n][L] when given.
void band_resolvent(Ctx &c, const double *AB, long long n, const double *Y, long long ncol, long long L, int nother,
                    const double *sig, double *acc, int nd, long long dcol0, double *rho, double *xout);
void tri_resolvent(Ctx &c, const double *d, const double *e, long long n, const double *Y, long long ncol, long long L,
                   int nother, const double *sig, double *acc, int nd, long long dcol0, double *rho, double *xout);

}  // namespace s2
}  // namespace nvpt

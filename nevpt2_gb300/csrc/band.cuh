// Band form of a symmetric matrix and resolvents in it (band.cu).
#pragma once
#include "s2_tensor.cuh"

namespace nvpt {
namespace s2 {

constexpr int kBand = 32;  // half bandwidth
// Panels of the reduction of order n, and the rows of their reflectors in all.
inline int band_panels(long long n) { return n > kBand + 1 ? (int)((n - 2) / kBand) : 0; }
long long band_rows(long long n);

// A (column-major n x n, both triangles valid) <- Q B Q^T: AB[k][i] = B(i + k, i)
// for k <= kBand ([kBand + 1][n]); Q as compact WY panels: V [band_rows(n)][kBand]
// (panel p: rows (p + 1) kBand .. n - 1), Tm [panels][kBand][kBand].  A is
// overwritten.  0, or 4 if a grid barrier timed out.
int band_reduce(Ctx &c, double *A, long long n, double *V, double *Tm, double *AB);
// Y <- Q^T Y (forward) or Q Y for m columns (column-major, ld n).
void band_apply(Ctx &c, long long n, const double *V, const double *Tm, double *Y, long long m, bool forward);
// For each label l < L with x_l = (B + sig_l)^-1 y_l (y_l = column l of Y, row-major
// [n][ncol]): acc[0] -= y_l . x_l, acc[1] += x_l . x_l, acc[2 + k] -= y_{k+1,l} . x_l
// for k < nother (column (k + 1) L + l), rho[l nd + k] -= Y[:, dcol0 + k] . x_l, and
// x_l into column l of xout [n][L] when given.
void band_resolvent(Ctx &c, const double *AB, long long n, const double *Y, long long ncol, long long L, int nother,
                    const double *sig, double *acc, int nd, long long dcol0, double *rho, double *xout);

}  // namespace s2
}  // namespace nvpt

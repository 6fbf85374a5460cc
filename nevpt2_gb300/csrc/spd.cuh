// Inverse Cholesky factors and congruences with them (spd.cu).
#pragma once
#include "s2_tensor.cuh"

namespace nvpt {
namespace s2 {

// Row length of the padded matrices: whole 64-blocks.
inline long long spd_ld(long long n) { return (n + 63) / 64 * 64; }

// W = L^-1 (row-major, lower, [spd_ld][spd_ld], identity in the padding) of the
// symmetric S = L L^T given by its upper triangle (row <= col, row-major n x n).
// False if a pivot was not positive.  inv_trace = tr S^-1 = |W|_F^2, top = the largest
// diagonal element of S.
bool spd_inverse_factor(Ctx &c, const double *S, long long n, double *W, double &inv_trace, double &top);
// Without the read-back: with trace stat[0] += tr S^-1 and stat[2] = top, spd_failed(stat) once
// a pivot was not positive (stat, two words or with trace three, on the device, zero before; a
// raised one makes later factorisations void).
void spd_inverse_factor_async(Ctx &c, const double *S, long long n, double *W, double *stat, bool trace);
bool spd_failed(const double *stat_on_host);
// out (n x n, both triangles) = W K W^T, K given by its upper triangle.
void spd_congruence(Ctx &c, const double *W, const double *K, long long n, double *out);

}  // namespace s2
}  // namespace nvpt

// The A-matrices from one n^9 contraction (bamat_sym.cu): scratch layout and
// launchers.
#pragma once
#include <cstddef>

#include "nvpt2_internal.h"

namespace nvpt {

constexpr int kSymMaxRpt = 5;  // rows per thread of the n^9 product

// Views into one scratch block of doubles(n) doubles, reused for every state.
struct SymScratch {
    double *H, *F, *N8;                       // unpacked 4-RDM [W][n^4], then T3; F; the four n^8 tensors
    double *G1, *G3, *Q1, *JW, *J2, *Z;       // n^4 sums
    double *Bf, *I4, *IJ, *g;                 // integral operands, f + K/2
    int *key;                                 // packed key quadruples [W]
    SymScratch(int n, double *w);
    static ll doubles(int n);
};

// Integral operands and the check of the integrals' symmetry: sets flag[0..M)
// (zeroed by the caller) where it fails.
void launch_sym_ops(const double *atwo, const double *f, int ncore, int n, const SymScratch &S, int M, int *flag,
                    cudaStream_t st);
// One state: the check of its RDMs (flag[s]) and, unless flagged, its
// A-matrices.  0, or 1 on a launch failure.
int launch_sym_state(const Rdm &r, int s, const double *atwo, const SymScratch &S, double *amat, double *atmat,
                     int *flag, cudaStream_t st);

// The same with the n^9 and n^8 contractions as digit products on the tensor
// cores: rows_buf holds sym_split_rows_doubles(n) doubles (operand rows, of
// sym_split_pairs(n) creator pairs at a time for F), oz_work
// sym_split_oz_bytes(n) bytes; a wait that timed out sets *oz_err.
int launch_sym_state_split(const Rdm &r, int s, const double *atwo, const SymScratch &S, double *rows_buf,
                           void *oz_work, int *oz_err, double *amat, double *atmat, int *flag, cudaStream_t st);
int sym_split_pairs(int n);
ll sym_split_rows_doubles(int n);
size_t sym_split_oz_bytes(int n);

}  // namespace nvpt

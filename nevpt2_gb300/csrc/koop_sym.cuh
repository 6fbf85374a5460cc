// The Koopmans matrices from one n^7 contraction (koop_sym.cu).
#pragma once
#include "nvpt2_internal.h"

namespace nvpt {

// Matrices of every state whose inputs have their physical symmetries; sets
// flag[s] (flag[0..M) zeroed by the caller) for the others.  kind 0: out = ipko2,
// eako2, gk0pa, gk0pd, hrdm2; 1: bmat, btmat; 2: cmat, ctmat.  0, or 2 on a failed
// allocation (nothing launched).
int launch_koop_sym(const Rdm &r, const double *atwo, const double *aj, int ncore, int kind, double *const out[5],
                    int *flag, cudaStream_t st);

}  // namespace nvpt

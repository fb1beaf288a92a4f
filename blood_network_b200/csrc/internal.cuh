// Internal (non-exported) interfaces shared by the library's translation units.
#pragma once
#include "common.cuh"

namespace bn {

// ---- csr_ops.cu
void transpose(const CSR& A, CSR& T, cudaStream_t s, bool with_val);
void add_scaled(const CSR& A, const CSR& B, double scale, CSR& C, cudaStream_t s);
void symmetrize(const CSR& A, CSR& out, cudaStream_t s);
int validate(const int* ia, const int* ja, int n, int m, int nnz, cudaStream_t s);

// ---- strength.cu
// S = strong part of A (reference rs_strength); returns max row length of A
// (floored at 1) in *max_lam.
void strength(const CSR& A, double theta, CSR& S, int* max_lam, cudaStream_t s);

// ---- coarsen.cu
enum Coarsening : int { COARSEN_RS = 0, COARSEN_PMIS = 1, COARSEN_HMIS = 2 };
// cf[i] = +1 (C) / -1 (F); returns the number of C points.
// rand() draws after srand(12345) on the device, kept for the levels of one
// hierarchy.  host_ok: sequences of up to host_max may come from the C library
// itself (which moves its state).
struct RandDraws {
  DBuf<int> d;
  int host_max = 32768;
  const int* first(int n, bool host_ok, cudaStream_t s);
};
int coarsen(const CSR& S, int method, int max_lam, int* cf, cudaStream_t s, RandDraws& draws);
// The C library's rand() state as the reference's PMIS of n points leaves it
// (rs_classical.c:246-371: srand(12345), n draws).
void pmis_rand_state(int n);

// ---- interp.cu
// distinct: no row of A or S holds a column twice (true of a solver's matrices);
// otherwise that is looked for.
void interpolation(const CSR& A, const CSR& S, const int* cf, int n_coarse, CSR& P,
                   cudaStream_t s, bool distinct = true);
void interpolation_pattern(const CSR& S, const int* cf, int n_coarse, CSR& P, cudaStream_t s);
void interpolation_values(const CSR& A, const CSR& S, const int* cf, CSR& P, cudaStream_t s,
                          bool distinct = true);

// ---- rap.cu
void rap(const CSR& R, const CSR& A, const CSR& P, CSR& Ac, cudaStream_t s);

}  // namespace bn

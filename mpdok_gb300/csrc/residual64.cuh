// FP64 residuals of several columns on the tensor cores (residual64.cu).
#pragma once
#include "common.cuh"

namespace mpdok {

// Groups of K columns; group g starts at column g K.
constexpr int MAX_GROUPS = 16;
struct ColGroups {
  int n;
  int id[MAX_GROUPS];
};

// Whether R = B - A X of nc columns should take residual64 (else the FP64 GEMV):
// a tile of up to 32 columns costs 2.0e-12 n^2 s, the FP64 pipe 1.6e-12 n^2 s per
// column, and below n = 2048 the extra launches and the ramp-up of one CTA per
// SM weigh as much as the product.
bool residual64_pays(long long n, int nc);
size_t residual64_work_bytes(long long n, int K, int ng);  // of up to ng groups; 0 where it does not pay
// The row exponents and column weights of A (kept in the workspace until A changes).
int residual64_prepare(const double* A, long long lda, long long n, void* work, cudaStream_t s);
// R = B - A X for the listed groups; *err = 5 when a bounded wait ran out.  lossy[c]
// (device) is set to 1 where the FP64 product of column c is the more accurate
// one, else to 0; the rule reads A and the column only.
int residual64(const double* A, long long lda, long long n, const double* X, long long ldx, int K,
               const ColGroups& groups, const double* B, long long ldb, double* R, long long ldr, void* work,
               int* lossy, int* err, cudaStream_t s);

}  // namespace mpdok

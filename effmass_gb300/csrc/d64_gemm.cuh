// d64_gemm.cuh — interface of the FP64-accurate tensor-core GEMMs (d64_gemm.cu).
#pragma once

#include "kernels.cuh"

// Power-of-two exponents of a complex128 matrix A [M][K] that the digit split
// divides out: ek[k] the largest biased exponent of column k, fm[m] the (biased)
// exponent of row m after the columns are scaled to below one.  Without ek the columns
// are not scaled.
struct D64Scale {
    int* ek = nullptr;  // [K]
    int* fm = nullptr;  // [M]
};

cudaError_t d64_scales(int M, int K, const double2* A, size_t lda, D64Scale s, cudaStream_t st);

// Projection: part[z][m][n] = sum over K range z of conj(A[m][k]) B[n][k],
// z < d64_proj_splits (every split holds part of K).  ws: d64_proj_ws bytes.
int d64_proj_splits(int M, int N, int K);
size_t d64_proj_ws(int M, int N, int K);
cudaError_t d64_proj(int M, int N, int K, const double2* A, size_t lda, D64Scale s, const double2* B, size_t ldb,
                     double2* part, unsigned char* ws, int* err, cudaStream_t st);

// W[m][n] = scale[m % period] sum_z part[z][m][n] (scale null: 1)
cudaError_t d64_reduce(int M, int N, int nz, const double2* part, const double* scale, int period, double2* W,
                       cudaStream_t st);

// Expansion: out[n][k] += sum_m W[m][n] A[m][k].  ws: d64_expand_ws bytes.
size_t d64_expand_ws(int M, int N, int K);
cudaError_t d64_expand(int M, int N, int K, const double2* W, size_t ldw, const double2* A, size_t lda, D64Scale s,
                       double2* out, size_t ldo, unsigned char* ws, int* err, cudaStream_t st);

// Expansions of dH/dk: with A the 4 P rows (p, d_x p, d_y p, d_z p) and W [4 P][N],
// for every out[a] not null
//   out[a][n][k] += sum_p W[(a + 1) P + p][n] A[p][k] + W[p][n] A[(a + 1) P + p][k]
size_t d64_expand_grad_ws(int P, int N, int K, int nd);
cudaError_t d64_expand_grad(int P, int N, int K, const double2* W, size_t ldw, const double2* A, size_t lda, D64Scale s,
                            double2* const out[3], size_t ldo, unsigned char* ws, int* err, cudaStream_t st);

// Test hook: poll limit of the MMA issuer's wait (polls < 0: the default).
cudaError_t d64_set_issue_wait_limit(long polls);

// d64_gemm.cuh — interface of the FP64-accurate tensor-core GEMMs (d64_gemm.cu).
#pragma once

#include "kernels.cuh"

// Groups of the P rows of a block of A: rows that share a radial function (device
// arrays).  A matrix of 4 P rows (values and three derivatives) has 4 ng groups,
// group set * ng + g in block `set`.  ng = 0: no groups.
struct D64Rows {
    int P = 0, ng = 0;
    const int* order = nullptr;  // [P] rows group by group
    const int* off = nullptr;    // [ng + 1] first of each group in order
    const int* gid = nullptr;    // [P] group of a row
};

// Power-of-two exponents of a complex128 matrix A [M][K] that the digit split
// divides out: ek[k] the largest biased exponent of column k (high 16 bits) and a
// group that has it (low 16), fm[m] the (biased) exponent of row m after the columns
// are scaled to below one; eg[g][k] and fg[g] the same per group of rows; with 4 P rows
// ed[a][k] like ek over the values and derivative a alone (ng + group: a derivative).
// Without groups the columns are not scaled (ek = null).
struct D64Scale {
    int *ek = nullptr, *fm = nullptr, *eg = nullptr, *fg = nullptr, *ed = nullptr;
    D64Rows rows;
};
// ints behind one another: ek [K], fm [M], eg [groups][K], fg [groups], ed [3][K]
size_t d64_scale_ints(int M, int K, const D64Rows& rows);
D64Scale d64_scale_at(int* at, int M, int K, const D64Rows& rows);

cudaError_t d64_scales(int M, int K, const double2* A, size_t lda, D64Scale s, cudaStream_t st);

// Projection: part[z][m][n] = sum over K range z of conj(A[m][k]) B[n][k],
// z < d64_proj_splits (every split holds part of K).  ws: d64_proj_ws bytes.
int d64_proj_splits(int M, int N, int K);
size_t d64_proj_ws(int M, int N, int K, const D64Rows& rows);
cudaError_t d64_proj(int M, int N, int K, const double2* A, size_t lda, D64Scale s, const double2* B, size_t ldb,
                     double2* part, unsigned char* ws, int* err, cudaStream_t st);

// W[m][n] = scale[m % period] sum_z part[z][m][n] (scale null: 1) after d64_proj on the
// same operands and ws; sums that the digits do not hold well enough are formed
// in FP64.  The sums without scale are left in part[0] with keep.  Without groups the
// guard needs the largest elements of A's rows (ca) and of B's (cb).
cudaError_t d64_reduce(int M, int N, int K, int nz, double2* part, const double* scale, int period, double2* W,
                       const double2* A, size_t lda, D64Scale s, const double2* B, size_t ldb, unsigned char* ws,
                       bool keep, cudaStream_t st, const int2* ca = nullptr, const int2* cb = nullptr);

// out[row][i] = (k, biased exponent + 1) of the largest element of row x[row][.] in
// the i-th of D64_TOPS segments of K
constexpr int D64_TOPS = 32;
cudaError_t d64_tops(int rows, int K, const double2* x, size_t ld, int2* out, cudaStream_t st);

// Expansion: out[n][k] += sum_m W[m][n] A[m][k].  ws: d64_expand_ws bytes.
size_t d64_expand_ws(int M, int N, int K, const D64Rows& rows);
cudaError_t d64_expand(int M, int N, int K, const double2* W, size_t ldw, const double2* A, size_t lda, D64Scale s,
                       double2* out, size_t ldo, unsigned char* ws, int* err, cudaStream_t st);

// Expansions of dH/dk: with A the 4 P rows (p, d_x p, d_y p, d_z p) and W [4 P][N],
// for every out[a] not null
//   out[a][n][k] += sum_p W[(a + 1) P + p][n] A[p][k] + W[p][n] A[(a + 1) P + p][k]
size_t d64_expand_grad_ws(int P, int N, int K, int nd, const D64Rows& rows);
cudaError_t d64_expand_grad(int P, int N, int K, const double2* W, size_t ldw, const double2* A, size_t lda, D64Scale s,
                            double2* const out[3], size_t ldo, unsigned char* ws, int* err, cudaStream_t st);

// Test hook: poll limit of the MMA issuer's wait (polls < 0: the default).
cudaError_t d64_set_issue_wait_limit(long polls);

// selftest.cu — device check of the integer-pipe FP64 <-> FP32 conversions
// (d2f_bits, f2d_bits in common.cuh) against the hardware conversions.
#include <cuda_runtime.h>

#include "hpsi_gb300.h"
#include "common.cuh"
#include "d64_gemm.cuh"
#include "tc_gemm.cuh"

namespace {

__global__ void convert_kernel(const double* __restrict__ x, long n, float* f_bits, float* f_hw, double* d_bits,
                               double* d_hw)
{
    const long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const double v = x[i];
    const float h = __double2float_rn(v);
    f_bits[i] = d2f_bits(v);
    f_hw[i] = h;
    d_bits[i] = f2d_bits(h);
    d_hw[i] = (double)h;
}

__global__ void sum_kernel(const float* __restrict__ x, long rows, double* sum, double* wide)
{
    const long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= rows) return;
    float a[16];
    for (int k = 0; k < 16; ++k) {
        a[k] = x[16 * i + k];
        wide[16 * i + k] = widen(a[k]);
    }
    sum[i] = sum_floats(a);
}

}  // namespace

// sums of 16 floats each (x [rows][16]) as the band-pair reduction takes them, and
// every float widened as the FP32 GEMMs widen theirs
extern "C" int hpsi_selftest_sums(const float* x, long rows, double* sum, double* wide)
{
    if (rows < 0 || (rows > 0 && (!x || !sum || !wide))) return HPSI_ERR_BAD_ARG;
    if (rows == 0) return HPSI_OK;
    const size_t n = (size_t)rows * 16;
    unsigned char* m = nullptr;
    if (cudaMalloc(&m, n * 12 + rows * 8) != cudaSuccess) return HPSI_ERR_OOM;
    double *dw = reinterpret_cast<double*>(m), *ds = dw + n;
    float* dx = reinterpret_cast<float*>(ds + rows);
    cudaError_t e = cudaMemcpy(dx, x, n * sizeof(float), cudaMemcpyHostToDevice);
    if (!e) sum_kernel<<<(unsigned)((rows + 127) / 128), 128>>>(dx, rows, ds, dw);
    if (!e) e = cudaGetLastError();
    if (!e) e = cudaMemcpy(sum, ds, rows * sizeof(double), cudaMemcpyDeviceToHost);
    if (!e) e = cudaMemcpy(wide, dw, n * sizeof(double), cudaMemcpyDeviceToHost);
    cudaFree(m);
    return e ? HPSI_ERR_CUDA : HPSI_OK;
}

extern "C" int hpsi_selftest_convert(const double* x, long n, float* f_bits, float* f_hw, double* d_bits,
                                     double* d_hw)
{
    if (n < 0 || (n > 0 && (!x || !f_bits || !f_hw || !d_bits || !d_hw))) return HPSI_ERR_BAD_ARG;
    if (n == 0) return HPSI_OK;
    const size_t nd = (size_t)n * sizeof(double), nf = (size_t)n * sizeof(float);
    char* m = nullptr;
    if (cudaMalloc(&m, 3 * nd + 2 * nf) != cudaSuccess) return HPSI_ERR_OOM;
    double* dx = reinterpret_cast<double*>(m);
    double* db = dx + n;
    double* dh = db + n;
    float* fb = reinterpret_cast<float*>(dh + n);
    float* fh = fb + n;
    cudaError_t e = cudaMemcpy(dx, x, nd, cudaMemcpyHostToDevice);
    if (!e) {
        convert_kernel<<<ceil_div(n, 256), 256>>>(dx, n, fb, fh, db, dh);
        e = cudaGetLastError();
    }
    if (!e) e = cudaMemcpy(f_bits, fb, nf, cudaMemcpyDeviceToHost);
    if (!e) e = cudaMemcpy(f_hw, fh, nf, cudaMemcpyDeviceToHost);
    if (!e) e = cudaMemcpy(d_bits, db, nd, cudaMemcpyDeviceToHost);
    if (!e) e = cudaMemcpy(d_hw, dh, nd, cudaMemcpyDeviceToHost);
    cudaFree(m);
    return e ? HPSI_ERR_CUDA : HPSI_OK;
}

// Test hook of the bounded pipeline waits: lowers the poll limit of the
// tensor-core GEMMs' MMA issuer (0: it gives up at once) so that a test can
// watch a wait run out and the error reach the caller as HPSI_ERR_TIMEOUT.
extern "C" int hpsi_selftest_wait_limit(long polls)
{
    return tc_set_issue_wait_limit(polls) == cudaSuccess && d64_set_issue_wait_limit(polls) == cudaSuccess
               ? HPSI_OK : HPSI_ERR_CUDA;
}

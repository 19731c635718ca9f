// gemm.cu — register-tiled SIMT complex GEMMs for the nonlocal term: the FP32
// path, and FP64 where the digit-sliced GEMMs (d64_gemm.cu) have no workspace.
//
// The reference applies each projector separately with two passes over the
// G-sphere per (atom, l, m, i) (src/H_psi/hamiltonian_callable.cpp:259-297):
//   inner = sum_G conj(p(G)) psi(G);   hpsi(G) += lambda * inner * p(G).
// For a block of nb bands these are two complex GEMMs over the projector
// matrix Pr[P][npw]:
//   projection  W[P][nb]   = conj(Pr) psi^T       (K = npw, split over K)
//   expansion   hpsi[nb][G] += (lambda W)^T Pr     (K = P)
// Tiles: up to 64 x 64 outputs per 256-thread block, 16-deep K slices staged in
// shared memory; each thread owns up to a 4 x 4 block of outputs at stride 16 so
// that shared-memory reads of a warp are bank-conflict free.  What bounds them on
// the smaller cells is the latency of a block's loads and too few blocks, so the
// next slice is fetched while one is multiplied, and tiles shrink while blocks do
// not fill the SMs.  FP32, us before -> now: H|psi> of 2 atoms, 32 bands 41 -> 35..37;
// 8 atoms, 48 bands 85 -> 58 (projection 26 -> 13, expansion 26 -> 13); 16 atoms,
// 37 bands 197 -> 156; 64 atoms, 16 bands 878 -> 646; gradient, 8 atoms, 48 bands
// 194 -> 109.  All sums keep their order: the results are the same bits.
#include <type_traits>
#include "kernels.cuh"

template <typename Acc, typename T>
HPSI_D Acc load_as(const T& v);
template <> HPSI_D double2 load_as<double2, double2>(const double2& v) { return v; }
template <> HPSI_D float2 load_as<float2, double2>(const double2& v) { return to_c64(v); }
template <> HPSI_D float2 load_as<float2, float2>(const float2& v) { return v; }
template <> HPSI_D double2 load_as<double2, float2>(const float2& v) { return to_c128(v); }

// r + i s += conj(a) b.  In FP32 the roundings are written out, so that a result
// does not depend on the tile that computes it: the product of the imaginary
// parts is the one rounded by itself, with YFIRST that of the real parts.
template <bool YFIRST>
HPSI_D void mac_conj(double& r, double& s, double2 a, double2 b)
{
    r += a.x * b.x + a.y * b.y;
    s += a.x * b.y - a.y * b.x;
}
template <bool YFIRST>
HPSI_D void mac_conj(float& r, float& s, float2 a, float2 b)
{
    r = __fadd_rn(r, YFIRST ? __fmaf_rn(a.y, b.y, __fmul_rn(a.x, b.x)) : __fmaf_rn(a.x, b.x, __fmul_rn(a.y, b.y)));
    s = __fadd_rn(s, __fmaf_rn(a.x, b.y, -__fmul_rn(a.y, b.x)));
}

constexpr int GB_K = 16;  // K slice staged per iteration

// Projection tile: (16 TM) x (16 TN) outputs per 256-thread block, each thread
// TM x TN at stride 16 (conflict-free shared-memory reads).  The launcher picks
// the tile from M and N so that small problems (a few bands, few projectors)
// do not spend the block on padding.
template <typename TA, typename TB, typename Acc, int TM, int TN, bool YFIRST>
__global__ void __launch_bounds__(256) proj_gemm_kernel(int M, int N, int K, const TA* __restrict__ A, size_t lda,
                                                        const TB* __restrict__ B, size_t ldb, Acc* __restrict__ part,
                                                        int kchunk)
{
    using R = typename Real<Acc>::type;
    constexpr int BM = 16 * TM, BN = 16 * TN;
    __shared__ Acc As[GB_K][BM + 1];
    __shared__ Acc Bs[GB_K][BN + 1];
    const int m0 = blockIdx.x * BM, n0 = blockIdx.y * BN, s = blockIdx.z;
    const int kbeg = s * kchunk;
    const int kend = min(K, kbeg + kchunk);
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
    R accr[TM][TN], acci[TM][TN];
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) accr[i][j] = acci[i][j] = 0;

    // The next slice's elements travel in registers while a slice is multiplied:
    // a block of a short split is bound by the latency of its loads.
    const int kk0 = threadIdx.x % GB_K, r0 = threadIdx.x / GB_K;
    Acc av[TM], bv[TN];
    auto fetch = [&](int k0) {
        const int gk = k0 + kk0;
#pragma unroll
        for (int i = 0; i < TM; ++i) {
            const int r = m0 + r0 + 16 * i;
            av[i] = (r < M && gk < kend) ? load_as<Acc>(A[(size_t)r * lda + gk]) : cmake<Acc>(0, 0);
        }
#pragma unroll
        for (int j = 0; j < TN; ++j) {
            const int r = n0 + r0 + 16 * j;
            bv[j] = (r < N && gk < kend) ? load_as<Acc>(B[(size_t)r * ldb + gk]) : cmake<Acc>(0, 0);
        }
    };
    if (kbeg < kend) fetch(kbeg);
    for (int k0 = kbeg; k0 < kend; k0 += GB_K) {
#pragma unroll
        for (int i = 0; i < TM; ++i) As[kk0][r0 + 16 * i] = av[i];
#pragma unroll
        for (int j = 0; j < TN; ++j) Bs[kk0][r0 + 16 * j] = bv[j];
        __syncthreads();
        if (k0 + GB_K < kend) fetch(k0 + GB_K);
#pragma unroll
        for (int kk = 0; kk < GB_K; ++kk) {
            Acc a[TM], b[TN];
#pragma unroll
            for (int i = 0; i < TM; ++i) a[i] = As[kk][ty + 16 * i];
#pragma unroll
            for (int j = 0; j < TN; ++j) b[j] = Bs[kk][tx + 16 * j];
#pragma unroll
            for (int i = 0; i < TM; ++i)
#pragma unroll
                for (int j = 0; j < TN; ++j) {
                    mac_conj<YFIRST>(accr[i][j], acci[i][j], a[i], b[j]);
                }
        }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < TM; ++i) {
        const int m = m0 + ty + 16 * i;
        if (m >= M) continue;
#pragma unroll
        for (int j = 0; j < TN; ++j) {
            const int n = n0 + tx + 16 * j;
            if (n < N) part[((size_t)s * M + m) * N + n] = cmake<Acc>(accr[i][j], acci[i][j]);
        }
    }
}

static inline int tile_mult(int extent) { return extent <= 16 ? 1 : (extent <= 32 ? 2 : 4); }

template <typename TA, typename TB, typename Acc, int TM, int TN, bool YFIRST = false>
static void proj_launch(dim3 g, int M, int N, int K, const TA* A, size_t lda, const TB* B, size_t ldb, Acc* part,
                        int kchunk, cudaStream_t st)
{
    proj_gemm_kernel<TA, TB, Acc, TM, TN, YFIRST><<<g, 256, 0, st>>>(M, N, K, A, lda, B, ldb, part, kchunk);
}

template <typename TA, typename TB, typename Acc>
cudaError_t launch_proj_gemm(int M, int N, int K, const TA* A, size_t lda, const TB* B, size_t ldb, Acc* part,
                             int nsplit, cudaStream_t st)
{
    if (M == 0 || N == 0) return cudaSuccess;
    int kchunk = ceil_div(K, nsplit);
    kchunk = ceil_div(kchunk, GB_K) * GB_K;
    int tm = tile_mult(M), tn = tile_mult(N);
    const bool one_tile = tm == 1 && tn == 1;
    // smaller tiles while the blocks do not fill the SMs (P = 64, K = 3000, 48 bands: 26 -> 17 us);
    // the splits stay, and with them the order of the sums
    const auto blocks = [&] { return ceil_div(M, 16 * tm) * ceil_div(N, 16 * tn) * nsplit; };
    while (tn > 1 && blocks() < 152) tn /= 2;
    while (tm > 1 && blocks() < 152) tm /= 2;
    dim3 g(ceil_div(M, 16 * tm), ceil_div(N, 16 * tn), nsplit);
    // nsplit partial slabs are written even when K is split finer than needed (empty chunks write zeros)
    if (one_tile) proj_launch<TA, TB, Acc, 1, 1, true>(g, M, N, K, A, lda, B, ldb, part, kchunk, st);
    else if (tm == 1 && tn == 1) proj_launch<TA, TB, Acc, 1, 1>(g, M, N, K, A, lda, B, ldb, part, kchunk, st);
    else if (tm == 1 && tn == 2) proj_launch<TA, TB, Acc, 1, 2>(g, M, N, K, A, lda, B, ldb, part, kchunk, st);
    else if (tm == 2 && tn == 1) proj_launch<TA, TB, Acc, 2, 1>(g, M, N, K, A, lda, B, ldb, part, kchunk, st);
    else if (tm == 2 && tn == 2) proj_launch<TA, TB, Acc, 2, 2>(g, M, N, K, A, lda, B, ldb, part, kchunk, st);
    else if (tm == 1) proj_launch<TA, TB, Acc, 1, 4>(g, M, N, K, A, lda, B, ldb, part, kchunk, st);
    else if (tn == 1) proj_launch<TA, TB, Acc, 4, 1>(g, M, N, K, A, lda, B, ldb, part, kchunk, st);
    else if (tm == 2) proj_launch<TA, TB, Acc, 2, 4>(g, M, N, K, A, lda, B, ldb, part, kchunk, st);
    else if (tn == 2) proj_launch<TA, TB, Acc, 4, 2>(g, M, N, K, A, lda, B, ldb, part, kchunk, st);
    else proj_launch<TA, TB, Acc, 4, 4>(g, M, N, K, A, lda, B, ldb, part, kchunk, st);
    return cudaGetLastError();
}

// Split count for a projection of an M x N result over K: enough blocks for
// every SM (two per SM), at least 64 of K per split.
int proj_gemm_splits(int M, int N, int K)
{
    const int blocks = ceil_div(M, 16 * tile_mult(M)) * ceil_div(N, 16 * tile_mult(N));
    const int want = ceil_div(2 * 152, blocks);
    const int maxs = K / 64 > 1 ? K / 64 : 1;
    return want < 1 ? 1 : (want < maxs ? want : maxs);
}

template <typename Acc, typename CW>
__global__ void reduce_splits_kernel(int M, int N, int nsplit, const Acc* __restrict__ part,
                                     const double* __restrict__ scale, int period, CW* __restrict__ W, size_t ldw)
{
    const size_t idx = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= (size_t)M * N) return;
    const int m = (int)(idx / N), n = (int)(idx % N);
    if constexpr (std::is_same<Acc, float2>::value && std::is_same<CW, float2>::value) {
        Sum2f re, im;  // complex64: compensated FP32, no FP64 pipe
        for (int s = 0; s < nsplit; ++s) {
            const float2 v = part[(size_t)s * M * N + idx];
            re.add(v.x);
            im.add(v.y);
        }
        const float f = scale ? d2f_bits(scale[m % period]) : 1.f;
        W[(size_t)m * ldw + n] = make_float2(f * re.value(), f * im.value());
        return;
    }
    double sr = 0.0, si = 0.0;
    for (int s = 0; s < nsplit; ++s) {
        double2 v = as_c128(part[(size_t)s * M * N + idx]);
        sr += v.x;
        si += v.y;
    }
    const double f = scale ? scale[m % period] : 1.0;
    W[(size_t)m * ldw + n] = from_c128<CW>(make_double2(f * sr, f * si));
}

template <typename Acc, typename CW>
cudaError_t launch_reduce_splits(int M, int N, int nsplit, const Acc* part, const double* scale, int scale_period,
                                 CW* W, size_t ldw, cudaStream_t st)
{
    size_t tot = (size_t)M * N;
    if (tot == 0) return cudaSuccess;
    reduce_splits_kernel<Acc, CW><<<ceil_div((long)tot, 256), 256, 0, st>>>(M, N, nsplit, part, scale,
                                                                           scale_period > 0 ? scale_period : M, W, ldw);
    return cudaGetLastError();
}

template <typename C, int TM, int TN>
__global__ void __launch_bounds__(256) expand_gemm_kernel(int M, int N, int K, const C* __restrict__ W, size_t ldw,
                                                          const C* __restrict__ A, size_t lda,
                                                          double2* __restrict__ out, size_t ldo)
{
    // out[n][k] += sum_m W[m][n] * A[m][k]; block tile: (16 TM) n x (16 TN) k, slices of 16 m
    using R = typename Real<C>::type;
    constexpr int BN = 16 * TM, BK = 16 * TN;
    __shared__ C Ws[GB_K][BN + 1];
    __shared__ C As[GB_K][BK + 1];
    const int k0 = blockIdx.x * BK, n0 = blockIdx.y * BN;
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
    R accr[TM][TN], acci[TM][TN];
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) accr[i][j] = acci[i][j] = 0;
    // small tiles fetch their outputs beside the first slice
    constexpr bool EARLY = TM * TN <= 8;
    double2 o[TM][TN];
    auto fetch_out = [&]() {
#pragma unroll
        for (int i = 0; i < TM; ++i)
#pragma unroll
            for (int j = 0; j < TN; ++j) {
                const int n = n0 + ty + 16 * i, k = k0 + tx + 16 * j;
                o[i][j] = (n < N && k < K) ? out[(size_t)n * ldo + k] : make_double2(0.0, 0.0);
            }
    };
    // the next slice travels in registers while a slice is multiplied
    C wv[TM], av[TN];
    auto fetch = [&](int m0) {
#pragma unroll
        for (int i = 0; i < TM; ++i) {
            const int e = threadIdx.x + 256 * i, gm = m0 + e / BN, c = n0 + e % BN;
            wv[i] = (gm < M && c < N) ? W[(size_t)gm * ldw + c] : cmake<C>(0, 0);
        }
#pragma unroll
        for (int j = 0; j < TN; ++j) {
            const int e = threadIdx.x + 256 * j, gm = m0 + e / BK, c = k0 + e % BK;
            av[j] = (gm < M && c < K) ? A[(size_t)gm * lda + c] : cmake<C>(0, 0);
        }
    };
    if (M > 0) fetch(0);
    if (EARLY) fetch_out();
    for (int m0 = 0; m0 < M; m0 += GB_K) {
#pragma unroll
        for (int i = 0; i < TM; ++i) Ws[(threadIdx.x + 256 * i) / BN][(threadIdx.x + 256 * i) % BN] = wv[i];
#pragma unroll
        for (int j = 0; j < TN; ++j) As[(threadIdx.x + 256 * j) / BK][(threadIdx.x + 256 * j) % BK] = av[j];
        __syncthreads();
        if (m0 + GB_K < M) fetch(m0 + GB_K);
#pragma unroll
        for (int mm = 0; mm < GB_K; ++mm) {
            C w[TM], a[TN];
#pragma unroll
            for (int i = 0; i < TM; ++i) w[i] = Ws[mm][ty + 16 * i];
#pragma unroll
            for (int j = 0; j < TN; ++j) a[j] = As[mm][tx + 16 * j];
#pragma unroll
            for (int i = 0; i < TM; ++i)
#pragma unroll
                for (int j = 0; j < TN; ++j) {
                    accr[i][j] += w[i].x * a[j].x - w[i].y * a[j].y;
                    acci[i][j] += w[i].x * a[j].y + w[i].y * a[j].x;
                }
        }
        __syncthreads();
    }
    // all loads of the read-modify-write first, so that they overlap
    if (!EARLY) fetch_out();
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) {
            const int n = n0 + ty + 16 * i, k = k0 + tx + 16 * j;
            if (n < N && k < K) {
                o[i][j].x += widen(accr[i][j]);
                o[i][j].y += widen(acci[i][j]);
                out[(size_t)n * ldo + k] = o[i][j];
            }
        }
}

template <typename C>
cudaError_t launch_expand_gemm(int M, int N, int K, const C* W, size_t ldw, const C* A, size_t lda, double2* out,
                               size_t ldo, cudaStream_t st)
{
    if (N == 0 || K == 0 || M == 0) return cudaSuccess;
    // few bands: a narrow band tile; four G-columns per thread, or one where that
    // would leave SMs without a block (P = 64, K = 3000, 48 bands: 26 -> 12 us)
    const bool small = ceil_div(K, 64) * ceil_div(N, 64) < 152;
    auto go = [&](auto kernel, int bn, int bk) {
        kernel<<<dim3(ceil_div(K, bk), ceil_div(N, bn)), 256, 0, st>>>(M, N, K, W, ldw, A, lda, out, ldo);
    };
    if (N <= 16) small ? go(expand_gemm_kernel<C, 1, 1>, 16, 16) : go(expand_gemm_kernel<C, 1, 4>, 16, 64);
    else if (N <= 32 || small) small ? go(expand_gemm_kernel<C, 2, 1>, 32, 16) : go(expand_gemm_kernel<C, 2, 4>, 32, 64);
    else go(expand_gemm_kernel<C, 4, 4>, 64, 64);
    return cudaGetLastError();
}

template <typename C>
__global__ void convert_kernel(size_t n, const double2* __restrict__ in, C* __restrict__ out)
{
    size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) out[i] = from_c128<C>(in[i]);
}

template <typename C>
cudaError_t launch_convert(size_t n, const double2* in, C* out, cudaStream_t st)
{
    if (n == 0) return cudaSuccess;
    convert_kernel<C><<<ceil_div((long)n, 256), 256, 0, st>>>(n, in, out);
    return cudaGetLastError();
}

// instantiations
template cudaError_t launch_proj_gemm<double2, double2, double2>(int, int, int, const double2*, size_t, const double2*,
                                                                 size_t, double2*, int, cudaStream_t);
template cudaError_t launch_proj_gemm<float2, float2, float2>(int, int, int, const float2*, size_t, const float2*,
                                                              size_t, float2*, int, cudaStream_t);
template cudaError_t launch_proj_gemm<float2, double2, float2>(int, int, int, const float2*, size_t, const double2*,
                                                               size_t, float2*, int, cudaStream_t);
template cudaError_t launch_proj_gemm<double2, double2, float2>(int, int, int, const double2*, size_t, const double2*,
                                                                size_t, float2*, int, cudaStream_t);
template cudaError_t launch_reduce_splits<double2, double2>(int, int, int, const double2*, const double*, int,
                                                            double2*, size_t, cudaStream_t);
template cudaError_t launch_reduce_splits<float2, float2>(int, int, int, const float2*, const double*, int, float2*,
                                                          size_t, cudaStream_t);
template cudaError_t launch_reduce_splits<float2, double2>(int, int, int, const float2*, const double*, int, double2*,
                                                           size_t, cudaStream_t);
template cudaError_t launch_reduce_splits<double2, float2>(int, int, int, const double2*, const double*, int, float2*,
                                                           size_t, cudaStream_t);
template cudaError_t launch_expand_gemm<double2>(int, int, int, const double2*, size_t, const double2*, size_t,
                                                 double2*, size_t, cudaStream_t);
template cudaError_t launch_expand_gemm<float2>(int, int, int, const float2*, size_t, const float2*, size_t, double2*,
                                                size_t, cudaStream_t);
template cudaError_t launch_convert<float2>(size_t, const double2*, float2*, cudaStream_t);

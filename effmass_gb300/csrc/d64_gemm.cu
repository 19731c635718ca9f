// d64_gemm.cu — complex128 GEMMs of the nonlocal term on the FP16 tensor cores.
//
// GB300 runs FP64 at 1/64 of the FP32 rate (0.6 T multiply-adds/s on the whole
// part), so the FP64 projector sums were 94% of an FP64 H|psi> on the 64-atom
// cell.  Here each operand is written as a sum of S = 8 slices of base-256
// digits and the products of the slices run as exact integer arithmetic on the
// tensor cores (the splitting scheme of Ozaki, Ogita, Oishi and Rump,
// "Error-free transformations of matrix multiplication", Numer. Algorithms 59,
// 2012):
//   x 2^-(scales) = sum_i d_i 2^(-6 - 8 i),  i < 8, |d_i| <= 128 (FP16-exact),
// a fixed-point number of 62 bits.  A slice product is at most 2^14, so FP32
// accumulation of up to 1024 of them is exact; slice pairs (i, j) of one
// diagonal d = i + j share an accumulator (at most 8 pairs), which is read out
// every 128 of K.  Diagonals 0..7 are kept (36 of 64 pairs); the largest of the
// dropped ones is 2^-62 of the product of the scales.  The read-outs are added as
// 64-bit integers and rounded to FP64 once per output.
//
// Scales: the columns of A (one per K index) are divided by a power of two to
// at most one and B multiplied by it, then every row of A and of B is divided by
// its own power of two.  So the digits of an element are relative to the largest
// scaled element of its row, of A and of B: projectors decay as
// exp(-q^2 rc^2/4) over the G-sphere, bands grow or decay independently of that.
// Where both rows are large at the same K, that is relative to the largest term of
// the sum.
//
// Guard: where they are large at different K (a wide projector, and a band where
// only the narrow ones have not decayed), the digits lose the bits between.  The
// largest term of a group of rows with one radial function is known from exponents
// alone, eg[g][k] of the group's columns and those of the band, so the loss is too:
// sums that lose more than LOSS_MAX bits are formed in FP64 instead (projection: in
// d64_reduce; expansion: at the store).  Silicon-like cells with two projectors per l
// lose 0 to 4 bits, 5 or 6 in one of a hundred sums; two radii, 0.8 and 1.8, and a
// band beyond q = 5 lose 13.  Error of the projections of such cells against 80-bit sums,
// relative to the 2-norm of a sum's terms, by bits lost (seven slices / eight / FP64
// sums in chains of 192): 2 bits 9e-16 / 9e-17 / 6e-16, 4 bits 6e-15 / 4e-16 / 6e-16,
// 6 bits 6e-15 / 4e-16 / 3e-16.  The pair matrix of the velocities has no groups: its
// rows are bands, which say nothing about one another, so their columns are not
// scaled, and the largest term of an entry is taken among the largest elements of
// both rows in 32 segments of K.  That is 0 to 3 bits too small (8- and 64-atom cells),
// so entries may seem to lose two bits more.
//
// What bounds it: the tensor pipe on large cells (64-atom cell, 128 bands: 80% of
// the measured bf16 rate in the GEMMs).  The eight slices of a B tile lie one
// after the other in shared memory and the eight diagonals in TMEM, so one MMA
// of up to N = 256 multiplies slice i of A with all its slices of B into their
// diagonals: 8 MMAs per 16 of K instead of 36, which the issuing thread could not
// feed (70 clocks each).  Tiles of 16 bands (32 rows of B) leave TMEM room for two
// sets of accumulators, so that one is read out under the next chunk's MMAs;
// against tiles of 32 bands with one set, H|psi> us (seven slices, no guard): 8-atom
// cell, 48 bands 187 -> 173; 16 atoms, 37 bands 266 -> 234; 64 atoms, 128 bands
// 5542 -> 5404; gradient, 8 atoms 129 -> 101.  The eighth slice and the guard: 64 atoms
// 5420 -> 5720, 8 atoms 182 -> 187, gradient 103 -> 117.  What is left beside
// the MMAs is writing the slices of A: 0.7 ms of the 64-atom call, at the rate
// of the memory.  Tiles of A fetched by half or by a quarter do not change the
// GEMMs' time, so A is not multicast.  Measured and not kept: integers by FP32
// magic adds in place of F2I, 32 of K per stage (SWIZZLE_64B).
//
// Layout: K-major tiles of (rows x 16) FP16 digits, slice after slice: an A tile
// is 8 x 4 KB and a B tile 8 x NT x 32 bytes of contiguous memory, already in
// the SWIZZLE_32B order of the MMA descriptors, so that a pipeline stage is two
// bulk copies.
#include <algorithm>
#include <cuda_fp16.h>

#include "d64_gemm.cuh"
#include "tcgen05.cuh"

namespace {

constexpr int S = 8;                      // slices per operand
constexpr int ND = 8;                     // diagonals kept: i + j < ND
constexpr int TM = 128;                   // A rows per tile
constexpr int BT = 16;                    // bands per tile
constexpr int NT = 2 * BT;                // B rows per tile: two sets of ND accumulators fill TMEM
constexpr int KB = 16;                    // real K per pipeline stage (one MMA deep)
constexpr int CHUNK = 8;                  // stages per read-out of the accumulators (128 of K)
constexpr int FIX = 62;                   // bits of the fixed-point form
constexpr int A_STAGE = S * TM * KB * 2;  // 32 KB
constexpr int B_STAGE = S * NT * KB * 2;  // 8 KB
constexpr int STAGE = A_STAGE + B_STAGE;
constexpr int STAGES = 220 * 1024 / STAGE;  // that fit shared memory beside the barriers
constexpr int DRAIN_WARPS = 16;
constexpr int THREADS = 64 + 32 * DRAIN_WARPS;
constexpr uint32_t TMEM_ALL = 512;
constexpr size_t A_CAP = 1536ull << 20;    // bytes of A slices resident at once
constexpr int N_CAP = 256;                // bands per pass
constexpr int LOSS_MAX = 6;               // bits that a sum may lose to the scales
constexpr int LOSS_PAIR = 8;              // the same where the largest term is known from below (0 to 3 bits short)
constexpr int G_CHUNK = 8;                // groups per guard block of a projection
constexpr int G_BANDS = 16;               // its bands
constexpr int G_SEGS = 32;                // K segments of a projection's guard at most

// Row and band exponents are stored with a bias, so that 0 means "no nonzero element".
constexpr int F_BIAS = 8192;
constexpr int F_BAD = 1 << 20;            // an infinity or NaN in the row

__device__ uint32_t g_issue_wait_limit = WAIT_LIMIT;

__device__ __forceinline__ int clean(int f) { return (f == 0 || f >= F_BAD) ? 0 : f - F_BIAS; }

__device__ __forceinline__ int exp_of(double x) { return (__double2hiint(x) >> 20) & 0x7ff; }

// biased exponent of the larger part, -1 for zero
__device__ __forceinline__ int exp_of(double2 v)
{
    if (v.x == 0.0 && v.y == 0.0) return -1;
    return max(exp_of(v.x), exp_of(v.y));
}

constexpr unsigned long long DIGIT_BIAS = 0x8080808080808080ull;

// rint(x 2^sh) + DIGIT_BIAS for |x 2^sh| < 2^62: byte i of the sum, minus
// 128, is the base-256 digit of weight 2^(8 i); the top digit is at most 64.
__device__ __forceinline__ unsigned long long fixed_digits(double x, int sh)
{
    const uint32_t hi = (uint32_t)__double2hiint(x), lo = (uint32_t)__double2loint(x);
    const int e = (hi >> 20) & 0x7ff;
    const unsigned long long m =
        ((unsigned long long)((hi & 0xfffffu) | (e ? 0x100000u : 0u)) << 32 | lo) << 10;  // 63 bits
    // value = m 2^(e' - 1085 + sh), e' the exponent of a normal number: shift right by r > 0, rounding
    const int r = 1085 - sh - (e ? e : 1);
    const unsigned long long t = m >> min(max(r - 1, 0), 63);
    unsigned long long y = (t + 1) >> 1;
    if (hi >> 31) y = 0ull - y;
    return y + DIGIT_BIAS;
}

// slice i (0 the most significant) of two fixed-point values as an FP16 pair
template <int I>
__device__ __forceinline__ uint32_t slice_pair(unsigned long long u0, unsigned long long u1)
{
    constexpr int b = S - 1 - I, c = b & 3;  // byte
    const uint32_t w0 = b < 4 ? (uint32_t)u0 : (uint32_t)(u0 >> 32), w1 = b < 4 ? (uint32_t)u1 : (uint32_t)(u1 >> 32);
    uint32_t t = __byte_perm(w0, w1, c | (c << 4) | ((4 + c) << 8) | ((4 + c) << 12)) & 0x00ff00ffu;
    t |= 0x64006400u;  // FP16 1024 + digit + 128, exact
    const __half2 h = __hsub2(*reinterpret_cast<const __half2*>(&t), __floats2half2_rn(1152.f, 1152.f));
    return *reinterpret_cast<const uint32_t*>(&h);
}

// byte offset of 16-byte chunk c of row r within a slice (SWIZZLE_32B)
__device__ __forceinline__ int slice_off(int r, int c) { return 32 * r + 16 * (c ^ ((r >> 2) & 1)); }

// SMEM descriptor of a K-major tile in the SWIZZLE_32B layout: 8-row x 32-byte
// atoms stacked every 256 bytes
__device__ __forceinline__ uint64_t sdesc_sw32(uint32_t saddr)
{
    return (uint64_t)((saddr & 0x3FFFFu) >> 4) | (uint64_t)1 << 16 | (uint64_t)(256 >> 4) << 32 | (uint64_t)1 << 46 |
           (uint64_t)6 << 61;
}

template <int I>
__device__ __forceinline__ void store_slices(unsigned char* at, size_t stride, const unsigned long long (&u)[8])
{
    uint4 v;
    v.x = slice_pair<I>(u[0], u[1]);
    v.y = slice_pair<I>(u[2], u[3]);
    v.z = slice_pair<I>(u[4], u[5]);
    v.w = slice_pair<I>(u[6], u[7]);
    *reinterpret_cast<uint4*>(at + I * stride) = v;
    if constexpr (I + 1 < S) store_slices<I + 1>(at, stride, u);
}

// ---- scales -----------------------------------------------------------------
__device__ __forceinline__ int ceil_div_d(int a, int b) { return (a + b - 1) / b; }

// exponents of the columns of A: eg over a group of rows (blockIdx.y), ek over all
__global__ void col_exp_kernel(D64Rows rows, int K, const double2* __restrict__ A, size_t lda, int* eg, int* ek)
{
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= K) return;
    const int g = blockIdx.y, set = g / rows.ng, r = g - set * rows.ng, i1 = rows.off[r + 1];
    int e = 0;
#pragma unroll 4
    for (int i = rows.off[r] + blockIdx.z; i < i1; i += gridDim.z) {
        const double2 v = A[((size_t)set * rows.P + rows.order[i]) * lda + k];
        const int x = exp_of(v.x), y = exp_of(v.y);
        if (x != 0x7ff) e = max(e, x);
        if (y != 0x7ff) e = max(e, y);
    }
    if (e == 0) return;
    atomicMax(eg + (size_t)g * K + k, e);
    atomicMax(ek + k, e << 16 | g);
}

// ed: per column the largest of the values and of one derivative
__global__ void dir_exp_kernel(int ng, int K, const int* __restrict__ eg, int* ed)
{
    const int k = blockIdx.x * blockDim.x + threadIdx.x, a = blockIdx.y;
    if (k >= K) return;
    int e = 0;
    for (int g = 0; g < ng; ++g) {
        e = max(e, eg[(size_t)g * K + k] << 16 | g);
        e = max(e, eg[(size_t)((a + 1) * ng + g) * K + k] << 16 | (ng + g));
    }
    ed[(size_t)a * K + k] = e;
}

__global__ void row_exp_kernel(int K, const double2* __restrict__ A, size_t lda, const int* __restrict__ ek, int kper,
                               int* fm, D64Rows rows, int* fg)
{
    const int m = blockIdx.x, k0 = blockIdx.y * kper, k1 = min(K, k0 + kper);
    int f = 0;
    for (int k = k0 + threadIdx.x; k < k1; k += blockDim.x) {
        const int e = exp_of(A[(size_t)m * lda + k]);
        if (e >= 0) f = max(f, e == 0x7ff ? F_BAD : e - (ek ? ek[k] >> 16 : 1022) + F_BIAS);
    }
    f = __reduce_max_sync(0xffffffffu, f);
    if ((threadIdx.x & 31) == 0 && f) {
        atomicMax(fm + m, f);
        if (fg && f < F_BAD) atomicMax(fg + m / rows.P * rows.ng + rows.gid[m % rows.P], f);
    }
}

// ---- slices -----------------------------------------------------------------
// K index k of a GEMM -> row of A and row of W.  The expansion of dH/dk_a joins two
// blocks of rows into one K: k < split: p rows against <d_a p|psi>, then d_a p
// rows against <p|psi>.
struct KMap {
    int split, a1, w0, w1;
    __device__ __forceinline__ int a(int k) const { return k < split ? k : k + a1; }
    __device__ __forceinline__ int w(int k) const { return k < split ? k + w0 : k + w1; }
};

// Operands of nd GEMMs (the directions of an expansion; 1 for a projection)
struct SplitArgs {
    const double2 *A, *B;
    size_t lda, ldb;
    const int *ek, *fm;     // exponents of A's columns and rows
    const int *eg, *fg;     // and per group
    D64Rows rows;
    int sets;               // blocks of A's rows that take part
    int g_blocks;           // guard blocks per GEMM
    int* gt;                // projection: largest terms [segments][groups + 1][ngt], the last over all rows
    int ngt, kpt, b_bands;  // bands of the projection; K per thread of a segment; bands padded to tiles
    int* wg;                // expansion: [nd][sets ng][bands padded] exponents of W by group, + 1
    int R, row0;            // rows of the GEMM's A operand; first of this chunk
    int nb, K, KT;          // bands, complex K, stages
    int a_x, a_blocks;      // A blocks per row of blocks, per GEMM
    int b_seg, b_blocks;    // B blocks per band, per GEMM
    unsigned char *a, *b;   // slices, nd times a_bytes / b_bytes
    size_t a_bytes, b_bytes;
    int* fb;                // [nd][bands padded to tiles]
    KMap map[3];
};

// biased exponent that column k of A is divided by
__device__ __forceinline__ int col_exp(const int* ek, int k) { return ek ? ek[k] >> 16 : 1022; }

// One stage holds 8 complex K values.  TRANS = false: the projection (A row r is
// A[r][.], scales fm and ek; B row b is B[b][.]); TRANS = true: the expansion (A row
// r is column r of A, scales ek and fm; band b is column b of W).

// 64 rows x 16 K values of A.  A quad of lanes holds one row: 256-byte row reads (or
// 128-byte column runs), and each slice store of a warp fills two runs of 256 bytes.
template <bool TRANS>
__device__ __forceinline__ void split_a(const SplitArgs& s, int g, int block)
{
    const int bx = block % s.a_x, by = block / s.a_x;
    const int rl = by * 64 + (threadIdx.x >> 2), r = s.row0 + rl;
    const int kt = bx * 2 + ((threadIdx.x >> 1) & 1), c = threadIdx.x & 1;
    if (kt >= s.KT) return;
    const int k0 = kt * 8 + c * 4;
    const KMap map = s.map[g];
    unsigned long long u[8];
    double2 v[4];
    int sk[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int k = k0 + i;
        v[i] = make_double2(0.0, 0.0);
        sk[i] = 0;
        if (r < s.R && k < s.K) {
            const int ka = TRANS ? map.a(k) : k;
            v[i] = TRANS ? s.A[(size_t)ka * s.lda + r] : s.A[(size_t)r * s.lda + ka];
            sk[i] = TRANS ? -clean(s.fm[ka]) : 1022 - col_exp(s.ek, ka);
        }
    }
    const int sr = FIX + (r < s.R ? (TRANS ? 1022 - col_exp(s.ek, r) : -clean(s.fm[r])) : 0);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        u[2 * i] = fixed_digits(v[i].x, sr + sk[i]);
        u[2 * i + 1] = fixed_digits(v[i].y, sr + sk[i]);
    }
    unsigned char* tile = s.a + g * s.a_bytes + ((size_t)(rl >> 7) * s.KT + kt) * A_STAGE;
    store_slices<0>(tile + slice_off(rl & 127, c), TM * KB * 2, u);
}

template <bool TRANS>
__device__ __forceinline__ int band_exp(const SplitArgs& s, const KMap& map, int b, int k)
{
    const double2 v = TRANS ? s.B[(size_t)map.w(k) * s.ldb + b] : s.B[(size_t)b * s.ldb + k];
    const int e = exp_of(v);
    return e < 0 ? 0 : e == 0x7ff ? F_BAD : e - 1022 + (TRANS ? clean(s.fm[map.a(k)]) : col_exp(s.ek, k) - 1022) + F_BIAS;
}

// Exponents fb of the bands of long K, over blocks of B_SEG values
constexpr int B_SEG = 4096;
template <bool TRANS>
__global__ void __launch_bounds__(256) band_exp_kernel(SplitArgs s, int bands)
{
    const int b = blockIdx.y, g = blockIdx.z, k1 = min(s.K, (int)(blockIdx.x + 1) * B_SEG);
    if (b >= s.nb) return;
    int f = 0;
#pragma unroll 4
    for (int k = blockIdx.x * B_SEG + threadIdx.x; k < k1; k += 256) f = max(f, band_exp<TRANS>(s, s.map[g], b, k));
    f = __reduce_max_sync(0xffffffffu, f);
    if ((threadIdx.x & 31) == 0 && f) atomicMax(s.fb + g * bands + b, f);
}

// B rows of one band (or B_SEG of its K values): band b of tile t = b / BT sits in
// rows j = b % BT (real part of the result) and BT + j (imaginary part).  The
// projection's rows are (b_r, b_i) and (b_i, -b_r), for conj(A) B; the expansion's
// (W_r, -W_i) and (W_i, W_r).  Short K: the block takes the band's exponent
// first.  Bands past nb are zero.
template <bool TRANS>
__device__ __forceinline__ void split_b(const SplitArgs& s, int g, int block)
{
    __shared__ int red[8];
    const int bands = s.b_blocks / s.b_seg, b = block % bands, seg = block / bands, t = b / BT, j = b % BT;
    const KMap map = s.map[g];
    int f = 0;
    if (s.b_seg == 1) {
        if (b < s.nb) {
#pragma unroll 4
            for (int k = threadIdx.x; k < s.K; k += 256) f = max(f, band_exp<TRANS>(s, map, b, k));
        }
        f = __reduce_max_sync(0xffffffffu, f);
        if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = f;
        __syncthreads();
#pragma unroll
        for (int i = 0; i < 8; ++i) f = max(f, red[i]);
        if (threadIdx.x == 0) s.fb[g * bands + b] = f;
    } else if (b < s.nb) {
        f = s.fb[g * bands + b];
    }
    f = clean(f);
    const size_t slice = (size_t)2 * BT * KB * 2;
    unsigned char* out = s.b + g * s.b_bytes + (size_t)t * s.KT * S * slice;
    const int per = s.b_seg == 1 ? 2 * s.KT : B_SEG / 4, q1 = min(2 * s.KT, (seg + 1) * per);
#pragma unroll 2
    for (int q = seg * per + threadIdx.x; q < q1; q += 256) {
        const int kt = q >> 1, c = q & 1;
        unsigned long long re[8], im[8];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int k = kt * 8 + c * 4 + i;
            double2 v = make_double2(0.0, 0.0);
            int sh = 0;
            if (b < s.nb && k < s.K) {
                v = TRANS ? s.B[(size_t)map.w(k) * s.ldb + b] : s.B[(size_t)b * s.ldb + k];
                sh = FIX - f + (TRANS ? clean(s.fm[map.a(k)]) : col_exp(s.ek, k) - 1022);
            }
            const unsigned long long x = fixed_digits(v.x, sh), y = fixed_digits(v.y, sh);
            re[2 * i] = x;
            re[2 * i + 1] = TRANS ? 2 * DIGIT_BIAS - y : y;  // 2 bias - u: the digits of the negated value
            im[2 * i] = y;
            im[2 * i + 1] = TRANS ? x : 2 * DIGIT_BIAS - x;
        }
        unsigned char* tile = out + (size_t)kt * S * slice;
        store_slices<0>(tile + slice_off(j, c), slice, re);
        store_slices<0>(tile + slice_off(BT + j, c), slice, im);
    }
}

// Guard of a projection, for one K segment, G_BANDS bands and G_CHUNK groups of rows:
// the terms of group g's sums are below 2^t, t = max_k eg[g][k] + e(B[b][k]); the same
// with ek for all rows.  Stored + 1, so that 0 means no term.
__device__ __forceinline__ void guard_proj(const SplitArgs& s, int block)
{
    __shared__ int red[8][G_BANDS][G_CHUNK + 1];
    const int groups = s.sets * s.rows.ng, gc = ceil_div_d(groups, G_CHUNK), bc = ceil_div_d(s.nb, G_BANDS);
    const int g0 = block % gc * G_CHUNK, b0 = block / gc % bc * G_BANDS, seg = block / (gc * bc);
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    int x[G_CHUNK + 1];
    for (int j = 0; j < s.kpt; ++j) {
        const int k = (seg * s.kpt + j) * 256 + threadIdx.x;
        if (k < s.K) x[G_CHUNK] = col_exp(s.ek, k) + 1;
#pragma unroll
        for (int g = 0; g < G_CHUNK; ++g) {
            const int e = k < s.K && g0 + g < groups ? s.eg[(size_t)(g0 + g) * s.K + k] : 0;
            x[g] = e > 0 ? e + 1 : -4096;
        }
#pragma unroll 4
        for (int b = 0; b < G_BANDS; ++b) {
            int e = -1;
            if (k < s.K && b0 + b < s.nb) e = exp_of(s.B[(size_t)(b0 + b) * s.ldb + k]);
            if (e == 0x7ff) e = -1;
#pragma unroll
            for (int g = 0; g <= G_CHUNK; ++g) {
                const int t = __reduce_max_sync(0xffffffffu, e < 0 ? 0 : max(0, e + x[g]));
                if (lane == g) red[w][b][g] = j ? max(red[w][b][g], t) : t;
            }
        }
    }
    __syncthreads();
    for (int i = threadIdx.x; i < G_BANDS * (G_CHUNK + 1); i += 256) {
        const int g = i / G_BANDS, b = i - g * G_BANDS;
        if (b0 + b >= s.nb) continue;
        int t = 0;
#pragma unroll
        for (int y = 0; y < 8; ++y) t = max(t, red[y][b][g]);
        const int row = g == G_CHUNK ? groups : g0 + g;
        if (g == G_CHUNK ? g0 == 0 : row < groups) s.gt[((size_t)seg * (groups + 1) + row) * s.ngt + b0 + b] = t;
    }
}

// Guard of an expansion: the exponents of W over one group of rows, for 32 bands
__device__ __forceinline__ void guard_expand(const SplitArgs& s, int g, int block)
{
    __shared__ int red[8][32];
    const int ng = s.rows.ng, q = block % (s.sets * ng), set = q / ng, r = q - set * ng;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, b = block / (s.sets * ng) * 32 + lane;
    const KMap map = s.map[g];
    int x = 0;
    if (b < s.nb) {
#pragma unroll 4
        for (int i = s.rows.off[r] + w; i < s.rows.off[r + 1]; i += 8) {
            const int e = exp_of(s.B[(size_t)map.w(set * s.rows.P + s.rows.order[i]) * s.ldb + b]);
            if (e != 0x7ff) x = max(x, e + 1);
        }
    }
    red[w][lane] = x;
    __syncthreads();
    if (w) return;
#pragma unroll
    for (int y = 1; y < 8; ++y) x = max(x, red[y][lane]);
    const int bands = s.b_bands;
    if (b < bands) s.wg[((size_t)g * s.sets * ng + q) * bands + b] = x;
}

// both operands of a GEMM in one launch, B's blocks first (they take longest)
template <bool TRANS>
__global__ void __launch_bounds__(256) split_kernel(SplitArgs s)
{
    const int block = blockIdx.x, g = blockIdx.y;
    if (block < s.b_blocks) {
        split_b<TRANS>(s, g, block);
    } else if (block < s.b_blocks + s.g_blocks) {
        if (TRANS) guard_expand(s, g, block - s.b_blocks);
        else guard_proj(s, block - s.b_blocks);
    } else {
        split_a<TRANS>(s, g, block - s.b_blocks - s.g_blocks);
    }
}

// ---- GEMM -------------------------------------------------------------------
struct D64Smem {
    uint64_t full[STAGES], empty[STAGES];
    uint64_t dfull[2], dempty[2];  // accumulator set: a chunk's products final; read out
    uint64_t done;
    uint32_t tmem_base;
    uint32_t abort_flag;
};

struct D64Out {
    double2* part;   // projection: [z][M][ldn], first band of the pass
    int ldn;
    double2* out[3]; // expansion: [N][ldo] of each GEMM, +=
    size_t ldo;
    size_t a_bytes, b_bytes;  // operands of one GEMM
    int bands;       // column exponents of one GEMM
    const int* er;   // row exponents (fm, or ek)
    const int* fb;   // column exponents
    int M, N, row0;  // result rows and bands; first row of this launch's A chunk
    // guard of an expansion
    const int *eg, *ed, *wg;  // exponents of A (by group, by direction) and of W by group
    int ng, sets, K, dir[3];  // sets of ng groups (set 1: block dir of A's rows); row stride of eg
    int rows_P;               // rows of a set
    const double2 *A, *W;
    size_t lda, ldw;
    KMap map[3];
};

// one output of an expansion in FP64
__device__ __noinline__ double2 expand_exact(const double2* A, size_t lda, int row, const double2* W, size_t ldw, int n,
                                             int K, KMap map)
{
    double re = 0.0, im = 0.0;
    for (int k = 0; k < K; ++k) {
        const double2 a = A[(size_t)map.a(k) * lda + row], w = W[(size_t)map.w(k) * ldw + n];
        re = fma(a.x, w.x, fma(-a.y, w.y, re));
        im = fma(a.x, w.y, fma(a.y, w.x, im));
    }
    return make_double2(re, im);
}

// bits of the bands n0 .. n0 + 3 whose output at row loses more than LOSS_MAX bits to the
// scales of GEMM g; f: the bands' exponents (biased), e: that of the row's column of A
__device__ __noinline__ unsigned expand_loses(const D64Out& o, int g, int row, int n0, int4 f, int e)
{
    const int* wg = o.wg + (size_t)g * o.sets * o.ng * o.bands + n0;
    int4 t = make_int4(0, 0, 0, 0);
    for (int s = 0; s < o.sets; ++s) {
        const int* eg = o.eg + (size_t)(s ? o.dir[g] : 0) * o.ng * o.K + row;
#pragma unroll 4
        for (int r = 0; r < o.ng; ++r) {
            const int4 x = *reinterpret_cast<const int4*>(wg + (size_t)(s * o.ng + r) * o.bands);
            const int a = eg[(size_t)r * o.K];
            if (a > 0) {
                if (x.x > 0) t.x = max(t.x, a + x.x);
                if (x.y > 0) t.y = max(t.y, a + x.y);
                if (x.z > 0) t.z = max(t.z, a + x.z);
                if (x.w > 0) t.w = max(t.w, a + x.w);
            }
        }
    }
    auto loses = [&](int f, int t) { return f != 0 && f < F_BAD && t > 0 && e + f - F_BIAS - (t - 1023) > LOSS_MAX; };
    return loses(f.x, t.x) | loses(f.y, t.y) << 1 | loses(f.z, t.z) << 2 | loses(f.w, t.w) << 3;
}

__device__ __forceinline__ void tmem_ld4(uint32_t addr, uint32_t (&r)[4])
{
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0, %1, %2, %3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(addr));
}

// (h 2^32 + l) 2^e rounded once to FP64, on the integer pipe
__device__ __forceinline__ double round_sum(long long h, long long l, int e)
{
    const __int128 v = ((__int128)h << 32) + l;
    if (v == 0) return 0.0;
    const bool neg = v < 0;
    const unsigned __int128 a = neg ? (unsigned __int128)-v : (unsigned __int128)v;
    const unsigned long long ah = (unsigned long long)(a >> 64), al = (unsigned long long)a;
    const int lz = ah ? __clzll((long long)ah) : 64 + __clzll((long long)al);
    const unsigned __int128 n = a << lz;
    const unsigned long long top = (unsigned long long)(n >> 64), rest = (unsigned long long)n;
    unsigned long long m = top >> 11;
    const unsigned long long dropped = top & 0x7ffu;
    if (dropped > 0x400u || (dropped == 0x400u && (rest != 0 || (m & 1)))) ++m;
    const int be = 127 - lz + e + 1023;  // biased exponent
    const unsigned long long sign = neg ? 1ull << 63 : 0ull;
    if (be >= 1 && be < 2046) return __longlong_as_double((long long)(sign + ((unsigned long long)(be - 1) << 52) + m));
    const double x = __longlong_as_double((long long)(sign + (1022ull << 52) + m));  // [1, 2]
    return scalbn(x, be - 1023);
}

template <bool EXPAND>
__global__ void __launch_bounds__(THREADS, 1)
    d64_gemm_kernel(const unsigned char* __restrict__ A, const unsigned char* __restrict__ B, D64Out o, int KT,
                    int chunks_per_split, int* err)
{
    constexpr int NBUF = TMEM_ALL / (ND * NT), BPW = BT / 4;  // accumulator sets, bands per warp
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    const uint32_t raw = smem_u32(smem_raw);
    unsigned char* tiles = smem_raw + (((raw + 1023u) & ~1023u) - raw);
    D64Smem* sh = reinterpret_cast<D64Smem*>(tiles + STAGES * STAGE);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    // blockIdx.z: the K split of a projection, the GEMM of an expansion
    const int z = EXPAND ? 0 : blockIdx.z, gemm = EXPAND ? blockIdx.z : 0;
    const int kt0 = z * chunks_per_split * CHUNK, kt1 = min(KT, kt0 + chunks_per_split * CHUNK);
    const int nk = kt1 - kt0, nchunk = (nk + CHUNK - 1) / CHUNK;

    if (threadIdx.x == 0) {
        for (int s = 0; s < STAGES; ++s) {
            mbar_init(&sh->full[s], 1);
            mbar_init(&sh->empty[s], 1);
        }
        for (int a = 0; a < 2; ++a) {
            mbar_init(&sh->dfull[a], 1);
            mbar_init(&sh->dempty[a], DRAIN_WARPS);
        }
        mbar_init(&sh->done, 1);
        sh->abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&sh->tmem_base)),
                     "r"(TMEM_ALL));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = sh->tmem_base;
    volatile uint32_t* abort = &sh->abort_flag;

    if (warp == 0 && lane == 0) {
        // ---- bulk copies: one A tile and one B tile per stage
        const unsigned char* a = A + gemm * o.a_bytes + ((size_t)blockIdx.y * KT + kt0) * A_STAGE;
        const unsigned char* b = B + gemm * o.b_bytes + ((size_t)blockIdx.x * KT + kt0) * B_STAGE;
        int issued = 0;
        for (int it = 0; it < nk; ++it) {
            const int s = it % STAGES;
            if (!mbar_wait_abort(&sh->empty[s], ((it / STAGES) & 1) ^ 1, &sh->abort_flag)) {
                if (!*abort) { atomicExch(err, 11); *abort = 1; }
                break;
            }
            if (*abort) break;
            unsigned char* st = tiles + s * STAGE;
            mbar_arrive_expect_tx(&sh->full[s], STAGE);
            bulk_load(st, a + (size_t)it * A_STAGE, A_STAGE, &sh->full[s]);
            bulk_load(st + A_STAGE, b + (size_t)it * B_STAGE, B_STAGE, &sh->full[s]);
            issued = it + 1;
        }
        // drain: copies in flight must land before the CTA exits (bounded)
        for (int it = max(0, issued - STAGES); it < issued; ++it) mbar_wait(&sh->full[it % STAGES], (it / STAGES) & 1);
    } else if (warp == 1 && lane == 0) {
        // ---- MMA issuer
        const uint32_t lim = g_issue_wait_limit;
        bool stop = false;
        for (int c = 0; c < nchunk && !stop; ++c) {
            const int buf = c % NBUF;
            if (!mbar_wait_abort(&sh->dempty[buf], ((c / NBUF) & 1) ^ 1, &sh->abort_flag)) {
                if (!*abort) { atomicExch(err, 12); *abort = 1; }
                break;
            }
            tc_fence_after();
            const uint32_t acc = tmem + buf * (ND * NT);
            const int i1 = min(nk, (c + 1) * CHUNK);
            for (int it = c * CHUNK; it < i1; ++it) {
                const int s = it % STAGES;
                if (!mbar_wait_n(&sh->full[s], (it / STAGES) & 1, lim)) {
                    atomicExch(err, 13);
                    *abort = 1;
                    stop = true;
                    break;
                }
                tc_fence_after();
                const uint32_t st = smem_u32(tiles + s * STAGE);
                const uint64_t ad = sdesc_sw32(st), bd = sdesc_sw32(st + A_STAGE);
                const bool first = it == c * CHUNK;
                // Slice i of A against slices 0 .. ND - 1 - i of B in one MMA: their rows
                // follow each other in shared memory, and their diagonals i + j in TMEM.
                // The first products (i = 0: all diagonals) overwrite what the last
                // read-out left.
#pragma unroll
                for (int i = 0; i < S; ++i)
                    tc_mma(acc + i * NT, ad + ((i * TM * KB * 2) >> 4), bd, idesc_f16(TM, (ND - i) * NT, 0),
                           first && i == 0 ? 0u : 1u);
                tc_commit(&sh->empty[s]);
            }
            if (!stop) tc_commit(&sh->dfull[buf]);
        }
        // every MMA issued has completed before the accumulators are freed (bounded)
        tc_commit(&sh->done);
        mbar_wait(&sh->done, 0);
    } else if (warp >= 2) {
        // ---- read-out: warp w holds TMEM lanes 32 (w % 4) .. +31 (rows) and
        // bands sub BPW .. +BPW-1 of the tile, real and imaginary columns
        const int q = warp & 3, sub = (warp - 2) >> 2;
        const int row = o.row0 + blockIdx.y * TM + q * 32 + lane;
        // Bands whose output loses more than LOSS_MAX bits: candidates are those where the
        // group of A's rows that has the column's largest element has a small W.  (Done
        // here, under the first copies.)
        unsigned slow = 0;
        if (EXPAND && row < o.M) {
            const int e = o.er[row], b = (o.sets > 1 ? o.ed[(size_t)(o.dir[gemm] - 1) * o.K + row] : e);
            const int n0 = blockIdx.x * BT + sub * BPW;
            const int4 x = *reinterpret_cast<const int4*>(
                o.wg + ((size_t)gemm * o.sets * o.ng + (b & 0xffff)) * o.bands + n0);
            const int4 f = *reinterpret_cast<const int4*>(o.fb + (size_t)gemm * o.bands + n0);
            auto loses = [&](int f, int x) {
                return f != 0 && f < F_BAD && (x == 0 || (e >> 16) - (b >> 16) + f - F_BIAS - (x - 1023) > LOSS_MAX);
            };
            slow = loses(f.x, x.x) | loses(f.y, x.y) << 1 | loses(f.z, x.z) << 2 | loses(f.w, x.w) << 3;
            if (slow) slow &= expand_loses(o, gemm, row, n0, f, e >> 16);
        }
        long long h[2 * BPW], l[2 * BPW];
#pragma unroll
        for (int i = 0; i < 2 * BPW; ++i) h[i] = l[i] = 0;
        bool go = true;
        for (int c = 0; c < nchunk; ++c) {
            const int buf = c % NBUF;
            const bool ok = mbar_wait_abort(&sh->dfull[buf], (c / NBUF) & 1, &sh->abort_flag);
            if (!ok && !*abort) { atomicExch(err, 14); *abort = 1; }
            // warp-uniform: tcgen05.ld is a .sync.aligned warp instruction
            go = __all_sync(0xffffffffu, ok && !*abort);
            if (!go) break;
            tc_fence_after();
            const uint32_t base = tmem + ((uint32_t)(q * 32) << 16) + buf * (ND * NT) + sub * BPW;
#pragma unroll
            for (int p = 0; p < 2 * BPW; p += BPW) {
                const uint32_t at = base + (p < BPW ? p : BT + p - BPW);
                uint32_t v[ND][BPW];
#pragma unroll
                for (int d = 0; d < ND; ++d) tmem_ld4(at + d * NT, v[d]);
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                if (p + BPW >= 2 * BPW) {
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&sh->dempty[buf]);
                }
#pragma unroll
                for (int i = 0; i < BPW; ++i) {
                    // exact integers: |diagonal d| <= 128 (d + 1) 2^14, pairs with a top digit half of
                    // that, so all are below 2^24 and the sums of two adjacent high ones within 32 bits
                    int D[ND];
#pragma unroll
                    for (int d = 0; d < ND; ++d) D[d] = __float2int_rn(__uint_as_float(v[d][i]));
                    const int t01 = D[0] * 256 + D[1], t23 = D[2] * 256 + D[3];
                    h[p + i] += (long long)t01 * 65536 + t23;
                    l[p + i] += ((long long)D[4] * 16777216 + (long long)D[5] * 65536) + ((long long)D[6] * 256 + D[7]);
                }
            }
        }
        double2* out = gemm == 0 ? o.out[0] : gemm == 1 ? o.out[1] : o.out[2];
        if (go && row < o.M) {
            // h counts diagonal 3, l diagonal 7: weights 2^-36 and 2^-68
            const int fr = o.er[row];
            const bool bad = !EXPAND && fr >= F_BAD;
            const int er = (EXPAND ? (fr >> 16) - 1022 : clean(fr)) - 68;
#pragma unroll
            for (int i = 0; i < BPW; ++i) {
                const int n = blockIdx.x * BT + sub * BPW + i;
                if (n < o.N) {
                    const int f = o.fb[gemm * o.bands + n], e = er + clean(f);
                    double2 v = make_double2(round_sum(h[i], l[i], e), round_sum(h[BPW + i], l[BPW + i], e));
                    if (bad || f >= F_BAD) v.x = v.y = __longlong_as_double(0x7ff8000000000000ll);
                    if (EXPAND) {
                        if (slow >> i & 1)
                            v = expand_exact(o.A, o.lda, row, o.W, o.ldw, n, o.sets * o.rows_P, o.map[gemm]);
                        double2* at = out + (size_t)n * o.ldo + row;
                        double2 x = *at;
                        x.x += v.x;
                        x.y += v.y;
                        *at = x;
                    } else {
                        o.part[((size_t)blockIdx.z * o.M + row) * o.ldn + n] = v;
                    }
                }
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(TMEM_ALL));
    }
}

template <bool EXPAND>
cudaError_t launch_gemm(dim3 grid, const unsigned char* A, const unsigned char* B, const D64Out& o, int KT, int cps,
                        int* err, cudaStream_t st)
{
    constexpr size_t smem = (size_t)STAGES * STAGE + 1024 + sizeof(D64Smem);
    const cudaError_t e =
        cudaFuncSetAttribute(d64_gemm_kernel<EXPAND>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e) return e;
    d64_gemm_kernel<EXPAND><<<grid, THREADS, smem, st>>>(A, B, o, KT, cps, err);
    return cudaGetLastError();
}

int sms()
{
    static const int n = [] {
        int dev = 0, v = 152;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev);
        return v;
    }();
    return n;
}

// Shape of one GEMM: R result rows (A operand), N bands, K complex terms.
struct Plan {
    int tiles_n;            // band tiles
    int n_pass;             // bands per pass
    int KT;                 // stages over K
    int mt, mt_chunk;       // row tiles, row tiles per A chunk
    int cps, nz;            // chunks per split, splits
    size_t a_bytes, b_bytes, fb_bytes;
    int ng;                 // GEMMs run together
    int kpt, segs;          // guard of a projection: K per thread, segments
    size_t guard_bytes;     // gt of a projection; wg of an expansion
};

// groups: of the rows that take part (both sets of a gradient's expansion)
Plan plan(int R, int N, int K, bool split_k, int ng, int groups)
{
    Plan p;
    p.n_pass = std::min(N, N_CAP);
    p.tiles_n = ceil_div(p.n_pass, BT);
    p.KT = ceil_div(2l * K, KB);
    p.mt = ceil_div(R, TM);
    const int cap = (int)std::max<size_t>(1, std::min<size_t>(p.mt, A_CAP / ((size_t)p.KT * A_STAGE)));
    p.mt_chunk = ceil_div(p.mt, ceil_div(p.mt, cap));  // chunks of equal size
    const int nch = ceil_div(p.KT, CHUNK);
    p.cps = nch;
    if (split_k) {
        // split K over the SMs: the split count that minimises waves x (chunks + the
        // epilogue and set-up of a CTA, about two chunks)
        const long tiles_mn = (long)p.mt_chunk * p.tiles_n;
        double best = 1e300;
        for (int nz = 1; nz <= std::min(nch, 256); ++nz) {
            const int cps = ceil_div(nch, nz), z = ceil_div(nch, cps);
            const double t = (double)ceil_div(tiles_mn * z, sms()) * (cps + 2.0) + 0.02 * z;
            if (t < best) { best = t; p.cps = cps; }
        }
    }
    p.nz = ceil_div(nch, p.cps);
    p.a_bytes = (size_t)p.mt_chunk * p.KT * A_STAGE;
    p.b_bytes = (size_t)p.tiles_n * p.KT * B_STAGE;
    p.fb_bytes = ((size_t)p.tiles_n * BT * sizeof(int) + 255) / 256 * 256;
    p.ng = ng;
    p.kpt = ceil_div(K, 256 * G_SEGS);
    p.segs = ceil_div(K, 256 * p.kpt);
    p.guard_bytes = split_k ? (groups ? (size_t)p.segs * (groups + 1) * N * sizeof(int) : 0) : (size_t)ng * groups * p.tiles_n * BT * sizeof(int);
    p.guard_bytes = (p.guard_bytes + 255) / 256 * 256;
    return p;
}

size_t plan_bytes(const Plan& p) { return p.ng * (p.a_bytes + p.b_bytes + p.fb_bytes) + p.guard_bytes; }
int* plan_guard(const Plan& p, unsigned char* ws)
{
    return reinterpret_cast<int*>(ws + p.ng * (p.a_bytes + p.b_bytes + p.fb_bytes));
}

// The GEMMs of an expansion run together when their A slices fit the cap.
Plan expand_plan(int M, int N, int K, int ng, int groups)
{
    const Plan p = plan(K, N, M, false, ng, groups);
    return ng > 1 && ng * p.a_bytes > A_CAP ? plan(K, N, M, false, 1, groups) : p;
}

Plan proj_plan(int M, int N, int K, const D64Rows& rows)
{
    return plan(M, N, K, true, 1, rows.ng ? M / rows.P * rows.ng : 0);
}

// rows of A in chunks against all bands, the bands in passes of N_CAP
template <bool EXPAND>
cudaError_t run(const Plan& p, int R, int N, int K, const double2* A, size_t lda, D64Scale sc, const double2* B,
                size_t ldb, double2* part, const KMap* maps, const int* dirs, double2* const* out, size_t ldo,
                unsigned char* ws, int* err, cudaStream_t st)
{
    SplitArgs s{};
    s.A = A; s.lda = lda; s.ldb = ldb; s.ek = sc.ek; s.fm = sc.fm; s.eg = sc.eg; s.fg = sc.fg; s.rows = sc.rows;
    const int groups = sc.rows.ng;
    s.sets = groups ? (EXPAND ? K : R) / sc.rows.P : 0;
    s.ngt = N;
    s.kpt = p.kpt;
    s.R = R; s.K = K; s.KT = p.KT;
    s.a = ws; s.b = ws + p.ng * p.a_bytes;
    s.a_bytes = p.a_bytes; s.b_bytes = p.b_bytes;
    s.fb = reinterpret_cast<int*>(s.b + p.ng * p.b_bytes);
    const int bands = p.tiles_n * BT;
    s.b_bands = bands;
    s.wg = plan_guard(p, ws);
    s.b_seg = K > 2 * B_SEG ? ceil_div(p.KT, B_SEG / 8) : 1;
    s.a_x = ceil_div(p.KT, 2);
    for (int g = 0; g < p.ng; ++g) s.map[g] = maps[g];
    for (int n0 = 0; n0 < N; n0 += p.n_pass) {
        s.nb = std::min(p.n_pass, N - n0);
        s.B = EXPAND ? B + n0 : B + (size_t)n0 * ldb;
        if (s.b_seg > 1) {
            const cudaError_t e = cudaMemsetAsync(s.fb, 0, (size_t)p.ng * bands * sizeof(int), st);
            if (e) return e;
            band_exp_kernel<EXPAND><<<dim3(ceil_div(K, B_SEG), s.nb, p.ng), 256, 0, st>>>(s, bands);
        }
        for (int m = 0; m < p.mt; m += p.mt_chunk) {
            const int mt = std::min(p.mt_chunk, p.mt - m);
            s.row0 = m * TM;
            s.b_blocks = m == 0 ? bands * s.b_seg : 0;
            s.gt = plan_guard(p, ws) + n0;
            s.g_blocks = m > 0 || !groups ? 0 : EXPAND ? s.sets * groups * ceil_div(s.nb, 32)
                         : p.segs * ceil_div(s.nb, G_BANDS) * ceil_div(s.sets * groups, G_CHUNK);
            s.a_blocks = n0 == 0 || p.mt > p.mt_chunk ? s.a_x * 2 * mt : 0;
            if (s.a_blocks + s.b_blocks)
                split_kernel<EXPAND><<<dim3(s.a_blocks + s.b_blocks + s.g_blocks, p.ng), 256, 0, st>>>(s);
            D64Out o{};
            o.part = EXPAND ? nullptr : part + n0;
            o.ldn = N;
            for (int g = 0; g < p.ng; ++g) o.out[g] = EXPAND ? out[g] + (size_t)n0 * ldo : nullptr;
            o.ldo = ldo;
            o.a_bytes = p.a_bytes; o.b_bytes = p.b_bytes; o.bands = bands;
            o.er = EXPAND ? sc.ek : sc.fm;
            o.fb = s.fb;
            o.M = R; o.N = s.nb; o.row0 = s.row0;
            if (EXPAND) {
                o.eg = sc.eg; o.ed = sc.ed; o.wg = s.wg; o.ng = groups; o.sets = s.sets; o.K = R; o.rows_P = sc.rows.P;
                o.A = A; o.lda = lda; o.W = s.B; o.ldw = ldb;
                for (int g = 0; g < p.ng; ++g) { o.map[g] = maps[g]; o.dir[g] = dirs[g]; }
            }
            const cudaError_t e = launch_gemm<EXPAND>(dim3(p.tiles_n, mt, EXPAND ? p.ng : p.nz), s.a, s.b, o, p.KT,
                                                      p.cps, err, st);
            if (e) return e;
        }
    }
    return cudaGetLastError();
}

// Sums of a projection that the digits do not hold (guard), and their operands
struct Guard {
    const int* gt;     // largest terms [segs][groups + 1][N], null: no guard
    const int* fg;
    int segs, groups;
    const int2 *ca, *cb;  // largest elements by segment of A's and B's rows (d64_tops), null: none
    D64Rows rows;
    const double2 *A, *B;
    size_t lda, ldb;
    int K;
};

// W[m][n] = scale[m % period] sum_z part[z][m][n]: 32 outputs per block, the splits
// in SL slices that are added in order; flagged sums by the whole block in FP64
template <int SL>
__global__ void __launch_bounds__(32 * SL) d64_reduce_kernel(int N, size_t total, int nz, double2* __restrict__ part,
                                                             const double* __restrict__ scale, int period,
                                                             double2* __restrict__ W, Guard gd, bool keep)
{
    __shared__ double2 sum[SL][32];
    __shared__ int2 tf[SL][32];
    __shared__ unsigned todo;
    const size_t i = (size_t)blockIdx.x * 32 + threadIdx.x;
    const int per = ceil_div_d(nz, SL), z1 = min(nz, (int)(threadIdx.y + 1) * per);
    double re = 0.0, im = 0.0;
    int t = 0, f = 0, fg = 0;  // largest term; the scales: f over the columns or of A's row, fg of the other
    __shared__ int fb[SL][32];
    if (gd.gt && i < total) {
        const int m = (int)(i / N), n = (int)(i - (size_t)m * N), set = m / gd.rows.P;
        const int g = set * gd.rows.ng + gd.rows.gid[m - set * gd.rows.P];
        fg = clean(gd.fg[g]);
#pragma unroll 4
        for (int q = threadIdx.y; q < gd.segs; q += SL) {
            const int* at = gd.gt + (size_t)q * (gd.groups + 1) * N + n;
            t = max(t, at[(size_t)g * N]);
            f = max(f, at[(size_t)gd.groups * N]);
        }
    }
    if (gd.ca && i < total) {
        // at least one of the rows' largest elements by segment is near the largest term
        const int m = (int)(i / N), n = (int)(i - (size_t)m * N);
#pragma unroll 4
        for (int q = threadIdx.y; q < D64_TOPS; q += SL) {
            const int2 a = gd.ca[(size_t)m * D64_TOPS + q], b = gd.cb[(size_t)n * D64_TOPS + q];
            f = max(f, a.y);
            fg = max(fg, b.y);
            if (a.y > 0) {
                const int e = exp_of(gd.B[(size_t)n * gd.ldb + a.x]);
                if (e >= 0 && e != 0x7ff) t = max(t, a.y + e + 1);
            }
            if (b.y > 0) {
                const int e = exp_of(gd.A[(size_t)m * gd.lda + b.x]);
                if (e >= 0 && e != 0x7ff) t = max(t, b.y + e + 1);
            }
        }
    }
    if (i < total) {
#pragma unroll 4
        for (int z = threadIdx.y * per; z < z1; ++z) {
            const double2 v = part[(size_t)z * total + i];
            re += v.x;
            im += v.y;
        }
    }
    sum[threadIdx.y][threadIdx.x] = make_double2(re, im);
    tf[threadIdx.y][threadIdx.x] = make_int2(t, f);
    fb[threadIdx.y][threadIdx.x] = fg;
    __syncthreads();
    if (threadIdx.y == 0) {
#pragma unroll
        for (int y = 1; y < SL; ++y) {
            re += sum[y][threadIdx.x].x;
            im += sum[y][threadIdx.x].y;
            t = max(t, tf[y][threadIdx.x].x);
            f = max(f, tf[y][threadIdx.x].y);
            if (gd.ca) fg = max(fg, fb[y][threadIdx.x]);
        }
        // t = 0: no term among those known; with groups no term at all
        const unsigned b = __ballot_sync(0xffffffffu, gd.ca ? f > 0 && fg > 0 && fg + f - t > LOSS_PAIR
                                                            : t > 0 && fg + f - t > LOSS_MAX);
        if (threadIdx.x == 0) todo = b;
    }
    const bool guarded = gd.gt || gd.ca;
    if (guarded) __syncthreads();
    for (unsigned left = guarded ? todo : 0u; left; left &= left - 1) {
        const int j = __ffs((int)left) - 1;
        const size_t at = (size_t)blockIdx.x * 32 + j;
        const int m = (int)(at / N), n = (int)(at - (size_t)m * N);
        const double2 *a = gd.A + (size_t)m * gd.lda, *b = gd.B + (size_t)n * gd.ldb;
        double x = 0.0, y = 0.0;
#pragma unroll 4
        for (int k = threadIdx.y * 32 + threadIdx.x; k < gd.K; k += 32 * SL) {
            const double2 u = a[k], v = b[k];
            x = fma(u.x, v.x, fma(u.y, v.y, x));
            y = fma(u.x, v.y, fma(-u.y, v.x, y));
        }
        for (int o = 16; o > 0; o >>= 1) {
            x += __shfl_xor_sync(0xffffffffu, x, o);
            y += __shfl_xor_sync(0xffffffffu, y, o);
        }
        __syncthreads();
        if (threadIdx.x == 0) sum[threadIdx.y][0] = make_double2(x, y);
        __syncthreads();
        if (threadIdx.y == 0 && threadIdx.x == j) {
            re = im = 0.0;
#pragma unroll
            for (int q = 0; q < SL; ++q) {
                re += sum[q][0].x;
                im += sum[q][0].y;
            }
        }
    }
    if (threadIdx.y == 0 && i < total) {
        const double f = scale ? scale[(int)(i / N) % period] : 1.0;
        W[i] = make_double2(f * re, f * im);
        if (keep) part[i] = make_double2(re, im);
    }
}

// one block per row, four segments per warp
__global__ void __launch_bounds__(256) tops_kernel(int K, const double2* __restrict__ x, size_t ld, int2* out)
{
    const double2* row = x + (size_t)blockIdx.x * ld;
    const int lane = threadIdx.x & 31, len = ceil_div_d(K, D64_TOPS);
    for (int q = threadIdx.x >> 5; q < D64_TOPS; q += 8) {
        const int k1 = min(K, (q + 1) * len);
        int e = 0, at = 0;
#pragma unroll 4
        for (int k = q * len + lane; k < k1; k += 32) {
            const int y = exp_of(row[k]) + 1;
            if (y > e && y != 0x800) {
                e = y;
                at = k;
            }
        }
        const int top = __reduce_max_sync(0xffffffffu, e);
        at = __reduce_max_sync(0xffffffffu, e == top ? at : 0);
        if (lane == 0) out[(size_t)blockIdx.x * D64_TOPS + q] = make_int2(at, top);
    }
}

}  // namespace

cudaError_t d64_tops(int rows, int K, const double2* x, size_t ld, int2* out, cudaStream_t st)
{
    if (rows == 0) return cudaSuccess;
    tops_kernel<<<rows, 256, 0, st>>>(K, x, ld, out);
    return cudaGetLastError();
}

size_t d64_scale_ints(int M, int K, const D64Rows& rows)
{
    const size_t groups = rows.ng ? (size_t)(M / rows.P) * rows.ng : 0;
    return (size_t)(groups ? K : 0) + M + groups * K + groups + (groups && M > rows.P ? 3 * (size_t)K : 0);
}

D64Scale d64_scale_at(int* at, int M, int K, const D64Rows& rows)
{
    D64Scale s;
    s.rows = rows;
    if (!rows.ng) {
        s.fm = at;
        return s;
    }
    s.ek = at;
    s.fm = s.ek + K;
    s.eg = s.fm + M;
    const int groups = M / rows.P * rows.ng;
    s.fg = s.eg + (size_t)groups * K;
    if (M > rows.P) s.ed = s.fg + groups;
    return s;
}

cudaError_t d64_scales(int M, int K, const double2* A, size_t lda, D64Scale s, cudaStream_t st)
{
    if (M == 0 || K == 0) return cudaSuccess;
    cudaError_t e;
    if ((e = cudaMemsetAsync(s.ek ? s.ek : s.fm, 0, d64_scale_ints(M, K, s.rows) * sizeof(int), st))) return e;
    if (s.ek) {
        const int groups = M / s.rows.P * s.rows.ng, gx = ceil_div(K, 128);
        const int gz = std::max(1, std::min(ceil_div(M, groups), ceil_div(16 * sms(), gx * groups)));
        col_exp_kernel<<<dim3(gx, groups, gz), 128, 0, st>>>(s.rows, K, A, lda, s.eg, s.ek);
        if (s.ed) dir_exp_kernel<<<dim3(gx, 3), 128, 0, st>>>(s.rows.ng, K, s.eg, s.ed);
    }
    const int kper = 8192;
    // rows in x: a gradient of many projectors has more of them than y can hold
    row_exp_kernel<<<dim3(M, ceil_div(K, kper)), 256, 0, st>>>(K, A, lda, s.ek, kper, s.fm, s.rows, s.fg);
    return cudaGetLastError();
}

int d64_proj_splits(int M, int N, int K) { return plan(M, N, K, true, 1, 0).nz; }

size_t d64_proj_ws(int M, int N, int K, const D64Rows& rows) { return plan_bytes(proj_plan(M, N, K, rows)); }

size_t d64_expand_ws(int M, int N, int K, const D64Rows& rows) { return plan_bytes(expand_plan(M, N, K, 1, rows.ng)); }

size_t d64_expand_grad_ws(int P, int N, int K, int nd, const D64Rows& rows)
{
    return plan_bytes(expand_plan(2 * P, N, K, nd, 2 * rows.ng));
}

cudaError_t d64_proj(int M, int N, int K, const double2* A, size_t lda, D64Scale s, const double2* B, size_t ldb,
                     double2* part, unsigned char* ws, int* err, cudaStream_t st)
{
    if (M == 0 || N == 0 || K == 0) return cudaSuccess;
    const KMap map{K, 0, 0, 0};
    return run<false>(proj_plan(M, N, K, s.rows), M, N, K, A, lda, s, B, ldb, part, &map, nullptr, nullptr, 0, ws, err,
                      st);
}

cudaError_t d64_reduce(int M, int N, int K, int nz, double2* part, const double* scale, int period, double2* W,
                       const double2* A, size_t lda, D64Scale s, const double2* B, size_t ldb, unsigned char* ws,
                       bool keep, cudaStream_t st, const int2* ca, const int2* cb)
{
    const size_t total = (size_t)M * N;
    if (total == 0) return cudaSuccess;
    const Plan p = proj_plan(M, N, K, s.rows);
    const Guard g{s.rows.ng ? plan_guard(p, ws) : nullptr, s.fg, p.segs, s.rows.ng ? M / s.rows.P * s.rows.ng : 0,
                  ca, cb, s.rows, A, B, lda, ldb, K};
    const int blocks = ceil_div((long)total, 32);
    // eight slices also where sums of many terms may have to be formed
    if (nz >= 16 || (ca && K > 2048))
        d64_reduce_kernel<8><<<blocks, dim3(32, 8), 0, st>>>(N, total, nz, part, scale, period, W, g, keep);
    else d64_reduce_kernel<1><<<blocks, dim3(32, 1), 0, st>>>(N, total, nz, part, scale, period, W, g, keep);
    return cudaGetLastError();
}

cudaError_t d64_expand(int M, int N, int K, const double2* W, size_t ldw, const double2* A, size_t lda, D64Scale s,
                       double2* out, size_t ldo, unsigned char* ws, int* err, cudaStream_t st)
{
    if (M == 0 || N == 0 || K == 0) return cudaSuccess;
    const KMap map{M, 0, 0, 0};
    const int dir = 0;
    return run<true>(expand_plan(M, N, K, 1, s.rows.ng), K, N, M, A, lda, s, W, ldw, nullptr, &map, &dir, &out, ldo, ws,
                     err, st);
}

cudaError_t d64_expand_grad(int P, int N, int K, const double2* W, size_t ldw, const double2* A, size_t lda, D64Scale s,
                            double2* const out[3], size_t ldo, unsigned char* ws, int* err, cudaStream_t st)
{
    if (P == 0 || N == 0 || K == 0) return cudaSuccess;
    KMap map[3];
    double2* to[3];
    int nd = 0, dir[3];
    for (int a = 0; a < 3; ++a)
        if (out[a]) {
            dir[nd] = a + 1;
            map[nd] = KMap{P, a * P, (a + 1) * P, -P};
            to[nd++] = out[a];
        }
    if (nd == 0) return cudaSuccess;
    const Plan p = expand_plan(2 * P, N, K, nd, 2 * s.rows.ng);
    for (int g = 0; g < nd; g += p.ng) {
        const cudaError_t e =
            run<true>(p, K, N, 2 * P, A, lda, s, W, ldw, nullptr, map + g, dir + g, to + g, ldo, ws, err, st);
        if (e) return e;
    }
    return cudaSuccess;
}

cudaError_t d64_set_issue_wait_limit(long polls)
{
    const uint32_t v = polls < 0 ? WAIT_LIMIT : (uint32_t)std::min<long>(polls, (long)WAIT_LIMIT);
    return cudaMemcpyToSymbol(g_issue_wait_limit, &v, sizeof(v));
}

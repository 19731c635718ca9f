// local64.cu — the FP64 form of the local term (local.cu): the same three passes
// over T[band][plane][j][k] (complex128), with the line transforms in 64-bit
// fixed point (fft_q64.cuh).
//
//   g2r64      (plane, band): scatter psi, z-rows in use, y-columns, T
//   xpass64    (j, k-tile, bands): x G->r, times V, x r->G, in place in T
//   r2g64      (plane, band): y-columns, z-rows in use, gather into hpsi
//   xdensity64 (j, k-tile), all bands: x G->r, rho += occ |psi(r)|^2
//
// Every line has its own unit 2^u: before each axis the lines' largest
// magnitudes are taken in shared memory (an atomicMax per element at most, 1-2%
// of a transform's work), and elements are shifted into the unit of their new
// line as the first stage reads them.  V is a Q62 fraction of its tile's maximum.
// A line that holds an infinity or NaN comes out as NaN.
#include <algorithm>
#include <type_traits>

#include "fft_q64.cuh"
#include "kernels.cuh"

namespace {

using q64::Lines;
using q64::RowLines;

// Plane kernels: 640 threads, one block per SM, for planes that fill its shared
// memory; 192 threads, three blocks per SM, up to 48 x 48.
struct BigPlane { static constexpr int threads = 640, blocks = 1; };
struct SmallPlane { static constexpr int threads = 192, blocks = 3; };
constexpr int X_THREADS = 288;
// Kernels by grid: radices to 9 and axes to LONG; axes beyond it; an axis with a
// factor of 7, 11 or 13.  (The sums of long lines cost the plain kernels registers: 64
// atoms, 128 bands 5.48 -> 5.94 ms in one kernel for all.)
enum Kind { PLAIN, LONG_AXIS, WIDE_RADIX };

// rows of a plane that hold sphere points (PlaneRows of local.cu)
struct Rows {
    int jr, n, count, gap;
    HPSI_D Rows(int jr_, int n_) : jr(jr_), n(n_)
    {
        const bool all = 2 * jr_ + 1 >= n_;
        if (all) jr = n_;
        count = all ? n_ : 2 * jr_ + 1;
        gap = n_ - count;
    }
    HPSI_D int row(int L) const { return L + (L > jr ? gap : 0); }
    HPSI_D bool holds(int j) const { return j <= jr || j >= n - jr; }
};

// per band: the item's pointers in a batched launch
struct Band {
    int b, npw, nxs;
    const int *plane_off, *ent_ig, *ent_jk, *plane_jr;
    const double* kinetic;
    const double2* psi;
    double2* hpsi;
    size_t t0;  // first element of the band's planes in T
    HPSI_D Band(const LocalArgs& a, int band, const double2* psi_, double2* hpsi_, const double* kin_, size_t plane)
        : b(band), npw(a.npw), nxs(a.nxs), plane_off(a.plane_off), ent_ig(a.ent_ig), ent_jk(a.ent_jk),
          plane_jr(a.plane_jr), kinetic(kin_), psi(psi_), hpsi(hpsi_), t0(0)
    {
        if (a.items) {
            const LocalItem I = a.items[a.band_item[b]];
            b -= I.band0;
            npw = I.npw; nxs = I.nxs;
            plane_off = I.plane_off; ent_ig = I.ent_ig; ent_jk = I.ent_jk; plane_jr = I.plane_jr;
            kinetic = I.kinetic; psi = I.psi; hpsi = I.hpsi;
            t0 = I.t_off;
        }
        t0 += (size_t)b * nxs * plane;
        psi += (size_t)b * npw;
        if (hpsi) hpsi += (size_t)b * npw;
    }
};

// double-valued lines read into a line's unit
struct LoadRows {  // rows in use of the scatter buffer
    const double2* b;
    const int* unit;
    int ls;
    Rows r;
    HPSI_D longlong2 operator()(int L, int e) const
    {
        const int j = r.row(L);
        return q64::from_double(b[j * ls + e], unit[j]);
    }
};

// columns (unit cu) from rows (unit ru; rows not in use are zero)
struct ColsFromRows {
    const longlong2* b;
    const int *ru, *cu;
    int ls;
    Rows r;
    HPSI_D longlong2 operator()(int L, int e) const
    {
        return r.holds(e) ? q64::shift(b[e * ls + L], ru[e] - cu[L]) : make_longlong2(0, 0);
    }
};

struct LoadCols {
    const double2* b;
    const int* unit;
    int ls;
    HPSI_D longlong2 operator()(int L, int e) const { return q64::from_double(b[e * ls + L], unit[L]); }
};

// rows in use (unit ru) from columns (unit cu)
struct RowsFromCols {
    const longlong2* b;
    const int *ru, *cu;
    int ls;
    Rows r;
    HPSI_D longlong2 operator()(int L, int e) const
    {
        const int j = r.row(L);
        return q64::shift(b[j * ls + e], cu[e] - ru[j]);
    }
};

// shared memory of the plane kernels: two planes with odd row stride, the rows'
// and columns' exponents and units, and the twiddles where they still fit (the
// largest planes read them from global memory)
size_t plane_bytes(const LocalArgs& a, bool tw)
{
    return sizeof(double2) * 2 * (size_t)a.n2 * (a.n3 + 1) + 2 * sizeof(int) * (a.n2 + a.n3) +
           (tw ? sizeof(int4) * (a.n2 + a.n3) : 0);
}
constexpr size_t SMEM_MAX = 227 * 1024;

struct PlaneSmem {
    longlong2 *b0, *b1;
    int *re, *ru, *ce, *cu;  // exponents and units of rows and columns
    const int4 *twy, *twz;
    HPSI_D PlaneSmem(unsigned char* raw, int n2, int n3, bool tw_smem, const int4* twy_g, const int4* twz_g)
    {
        const int n23p = n2 * (n3 + 1);
        b0 = reinterpret_cast<longlong2*>(raw);
        b1 = b0 + n23p;
        int4* t = reinterpret_cast<int4*>(b1 + n23p);
        re = reinterpret_cast<int*>(t + (tw_smem ? n2 + n3 : 0));
        ru = re + n2;
        ce = ru + n2;
        cu = ce + n3;
        twy = tw_smem ? t : twy_g;
        twz = tw_smem ? t + n2 : twz_g;
        if (tw_smem) {
            for (int i = threadIdx.x; i < n2; i += blockDim.x) t[i] = twy_g[i];
            for (int i = threadIdx.x; i < n3; i += blockDim.x) t[n2 + i] = twz_g[i];
        }
        for (int i = threadIdx.x; i < n2; i += blockDim.x) re[i] = q64::EXP_NONE;
        for (int i = threadIdx.x; i < n3; i += blockDim.x) ce[i] = q64::EXP_NONE;
    }
};

// Units of `lines` lines of n points from their exponents (callers synchronise before
// and after).  Long lines need the sums of their magnitudes: mag(L, i) of element i < m.
template <int R, typename M>
HPSI_D void take_units(int lines, int n, const int* e, int* u, int m, const M& mag)
{
    if (R != PLAIN && n > q64::LONG) {
        unsigned* sum = reinterpret_cast<unsigned*>(u);
        for (int i = threadIdx.x; i < lines; i += blockDim.x) sum[i] = 0u;
        __syncthreads();
        for (int t = threadIdx.x; t < lines * m; t += blockDim.x) atomicAdd(sum + t % lines, mag(t % lines, t / lines));
        __syncthreads();
        for (int i = threadIdx.x; i < lines; i += blockDim.x) u[i] = q64::unit_of(e[i], q64::headroom(n, sum[i]));
    } else {
        const int fb = q64::headroom(n);
        for (int i = threadIdx.x; i < lines; i += blockDim.x) u[i] = q64::unit_of(e[i], fb);
    }
}

template <typename SZ, int R>
__global__ void __launch_bounds__(SZ::threads, R == WIDE_RADIX ? 1 : SZ::blocks)
    g2r64(LocalArgs a, const double2* __restrict__ psi_, double2* __restrict__ T, const int4* __restrict__ twy_g,
          const int4* __restrict__ twz_g, int tw_smem)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int n2 = a.n2, n3 = a.n3, n3p = n3 + 1, n23 = n2 * n3, p = blockIdx.x;
    const Band B(a, blockIdx.y, psi_, nullptr, nullptr, n23);
    if (p >= B.nxs) return;  // uniform per block, before any barrier
    const PlaneSmem s(smem_raw, n2, n3, tw_smem, twy_g, twz_g);
    const Rows rows(B.plane_jr ? B.plane_jr[p] : n2, n2);
    double2* grid = reinterpret_cast<double2*>(s.b0);
    for (int t = threadIdx.x; t < n2 * n3p; t += blockDim.x) grid[t] = make_double2(0.0, 0.0);
    __syncthreads();
    const int e1 = B.plane_off[p + 1];
    for (int e = B.plane_off[p] + threadIdx.x; e < e1; e += blockDim.x) {
        const int ig = B.ent_ig[e];
        if (ig < 0) continue;  // a later G shares its grid point: the last write wins
        const int jk = B.ent_jk[e], j = jk / n3, k = jk - j * n3;
        const double2 v = B.psi[ig];
        grid[j * n3p + k] = v;
        atomicMax(s.re + j, q64::exp_of(v));
    }
    __syncthreads();
    take_units<R>(n2, n3, s.re, s.ru, n3, [&](int j, int k) { return q64::magnitude(grid[j * n3p + k], s.re[j]); });
    __syncthreads();
    // z: rows in use, b0 -> b1 (-> b0 ...)
    const bool zb = q64::transform<R == WIDE_RADIX, +1>(LoadRows{grid, s.ru, n3p, rows}, RowLines{s.b1, n3p, rows.jr, rows.gap},
                                             RowLines{s.b0, n3p, rows.jr, rows.gap}, a.Lz, rows.count, s.twz);
    longlong2 *z = zb ? s.b0 : s.b1, *o = zb ? s.b1 : s.b0;
    // columns' exponents: thread = (column, slice of rows)
    const int slices = max(1, (int)blockDim.x / n3);
    for (int t = threadIdx.x; t < slices * n3; t += blockDim.x) {
        const int sl = t / n3, k = t - sl * n3;
        int e = q64::EXP_NONE;
        for (int L = sl; L < rows.count; L += slices) {
            const int j = rows.row(L);
            if (s.re[j] == q64::EXP_NONE) continue;
            e = max(e, s.re[j] >= q64::EXP_BAD ? q64::EXP_BAD : s.ru[j] + q64::bits_of(z[j * n3p + k]));
        }
        atomicMax(s.ce + k, e);
    }
    __syncthreads();
    take_units<R>(n3, n2, s.ce, s.cu, rows.count, [&](int k, int L) {
        const int j = rows.row(L);
        return s.re[j] == q64::EXP_NONE ? 0u : q64::magnitude(z[j * n3p + k], s.ru[j], s.ce[k]);
    });
    __syncthreads();
    const bool yb = q64::transform<R == WIDE_RADIX, +1>(ColsFromRows{z, s.ru, s.cu, n3p, rows}, Lines{o, 1, n3p},
                                             Lines{z, 1, n3p}, a.Ly, n3, s.twy);
    const longlong2* y = yb ? z : o;
    double2* Tp = T + B.t0 + (size_t)p * n23;
    const q64::Div d3(n3);
    for (int t = threadIdx.x; t < n23; t += blockDim.x) {
        const int j = d3(t), k = t - j * n3;
        Tp[t] = q64::to_double(y[j * n3p + k], s.cu[k], s.ce[k] >= q64::EXP_BAD);
    }
}

template <typename SZ, int R>
__global__ void __launch_bounds__(SZ::threads, R == WIDE_RADIX ? 1 : SZ::blocks)
    r2g64(LocalArgs a, const double2* __restrict__ T, const double2* __restrict__ psi_, double2* __restrict__ hpsi_,
          const double* __restrict__ kinetic_, const int4* __restrict__ twy_g, const int4* __restrict__ twz_g,
          int tw_smem)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int n2 = a.n2, n3 = a.n3, n3p = n3 + 1, n23 = n2 * n3, p = blockIdx.x;
    const Band B(a, blockIdx.y, psi_, hpsi_, kinetic_, n23);
    if (p >= B.nxs) return;
    const PlaneSmem s(smem_raw, n2, n3, tw_smem, twy_g, twz_g);
    const Rows rows(B.plane_jr ? B.plane_jr[p] : n2, n2);
    __syncthreads();
    const double2* Tp = T + B.t0 + (size_t)p * n23;
    double2* grid = reinterpret_cast<double2*>(s.b0);
    const int slices = max(1, (int)blockDim.x / n3);
    for (int t = threadIdx.x; t < slices * n3; t += blockDim.x) {
        const int sl = t / n3, k = t - sl * n3;
        int e = q64::EXP_NONE;
#pragma unroll 4
        for (int j = sl; j < n2; j += slices) {
            const double2 v = Tp[j * n3 + k];
            grid[j * n3p + k] = v;
            e = max(e, q64::exp_of(v));
        }
        atomicMax(s.ce + k, e);
    }
    __syncthreads();
    take_units<R>(n3, n2, s.ce, s.cu, n2, [&](int k, int j) { return q64::magnitude(grid[j * n3p + k], s.ce[k]); });
    __syncthreads();
    const bool yb = q64::transform<R == WIDE_RADIX, -1>(LoadCols{grid, s.cu, n3p}, Lines{s.b1, 1, n3p}, Lines{s.b0, 1, n3p}, a.Ly,
                                             n3, s.twy);
    longlong2 *y = yb ? s.b0 : s.b1, *o = yb ? s.b1 : s.b0;
    // rows' exponents: one warp per row in use
    for (int L = threadIdx.x >> 5; L < rows.count; L += blockDim.x >> 5) {
        const int j = rows.row(L);
        int e = q64::EXP_NONE;
        for (int k = threadIdx.x & 31; k < n3; k += 32)
            if (s.ce[k] != q64::EXP_NONE)
                e = max(e, s.ce[k] >= q64::EXP_BAD ? q64::EXP_BAD : s.cu[k] + q64::bits_of(y[j * n3p + k]));
        e = __reduce_max_sync(0xffffffffu, e);
        if ((threadIdx.x & 31) == 0) s.re[j] = e;
    }
    __syncthreads();
    take_units<R>(n2, n3, s.re, s.ru, n3, [&](int j, int k) {
        return !rows.holds(j) || s.ce[k] == q64::EXP_NONE ? 0u : q64::magnitude(y[j * n3p + k], s.cu[k], s.re[j]);
    });
    __syncthreads();
    const bool zb = q64::transform<R == WIDE_RADIX, -1>(RowsFromCols{y, s.ru, s.cu, n3p, rows}, RowLines{o, n3p, rows.jr, rows.gap},
                                             RowLines{y, n3p, rows.jr, rows.gap}, a.Lz, rows.count, s.twz);
    const longlong2* z = zb ? y : o;
    const int e1 = B.plane_off[p + 1];
    for (int e = B.plane_off[p] + threadIdx.x; e < e1; e += blockDim.x) {
        const int ig = B.ent_ig[e] & 0x7fffffff, jk = B.ent_jk[e], j = jk / n3, k = jk - j * n3;
        const double2 g = q64::to_double(z[j * n3p + k], s.ru[j], s.re[j] >= q64::EXP_BAD);
        const double2 c = B.psi[ig];
        const double kin = B.kinetic[ig];
        double2 h = B.hpsi[ig];
        h.x += kin * c.x + g.x * a.inv_n;
        h.y += kin * c.y + g.y * a.inv_n;
        B.hpsi[ig] = h;
    }
}

// ---- x passes ---------------------------------------------------------------
// Block: the NL = KT BB x-lines of (j, k0..k0+KT) for BB bands, element x of line
// L = bb KT + kk at [x NL + L].
struct XSmem {
    longlong2 *b0, *b1;
    int4* tw;
    int2* vq;         // V tile in Q62 words (l, h) [x KT + kk]
    int *xpl, *e, *u;  // plane of x (-1: none); lines' exponents and units
    unsigned* mag;    // OR of the magnitudes' high words of V psi
    int* ev;          // exponent of the V tile
    double* tail;     // energy and density sums
};

HPSI_D XSmem x_smem(unsigned char* raw, int n1, int KT, int NL, bool v)
{
    XSmem s;
    s.b0 = reinterpret_cast<longlong2*>(raw);
    s.b1 = s.b0 + n1 * NL;
    s.tw = reinterpret_cast<int4*>(s.b1 + n1 * NL);
    s.vq = reinterpret_cast<int2*>(s.tw + n1);
    s.tail = reinterpret_cast<double*>(s.vq + (v ? n1 * KT : 0));
    return s;
}
// the int arrays follow the tail of `tail` doubles
HPSI_D void x_smem_ints(XSmem& s, int tail, int n1, int NL)
{
    s.xpl = reinterpret_cast<int*>(s.tail + tail);
    s.e = s.xpl + n1;
    s.u = s.e + NL;
    s.mag = reinterpret_cast<unsigned*>(s.u + NL);
    s.ev = reinterpret_cast<int*>(s.mag + NL);
}

HPSI_D int parts_per_line(int NL) { return max(1, X_THREADS / NL); }

size_t x_bytes(const LocalArgs& a, bool v, size_t tail)
{
    const size_t NL = (size_t)a.kt * a.bb;
    return sizeof(longlong2) * 2 * (size_t)a.n1 * NL + sizeof(int4) * a.n1 + (v ? sizeof(int2) * (size_t)a.n1 * a.kt : 0) +
           sizeof(double) * tail + sizeof(int) * (a.n1 + 3 * NL + 1);
}
size_t energy_tail(const LocalArgs& a)
{
    const size_t NL = (size_t)a.kt * a.bb, tpl = X_THREADS / NL > 1 ? X_THREADS / NL : 1;
    return 2 * NL + 2 * NL * tpl;
}
size_t xpass_bytes(const LocalArgs& a) { return x_bytes(a, true, a.epart ? energy_tail(a) : 0); }
size_t xdensity_bytes(const LocalArgs& a) { return x_bytes(a, false, (size_t)a.n1 * a.kt); }

// x-lines from the planes of T held in b1, zero between them
struct XLoad {
    const double2* b;
    const int *xpl, *unit;
    int NL;
    HPSI_D longlong2 operator()(int L, int x) const
    {
        return xpl[x] < 0 ? make_longlong2(0, 0) : q64::from_double(b[x * NL + L], unit[L]);
    }
};

struct XShift {
    const longlong2* b;
    const int* sh;
    int NL;
    HPSI_D longlong2 operator()(int L, int x) const { return q64::shift(b[x * NL + L], sh[L]); }
};

// The block's lines of T into b1, with their exponents; ends with a barrier.
// NL lines, `on` lines of them per band group: line (bb, kk) exists for kk < kt, bb < nbb.
HPSI_D void x_load(const XSmem& s, const double2* __restrict__ T, const int* __restrict__ plane_x, int nxs, size_t plane,
                   size_t base, int KT, int NL, int kt, int nbb, int bb0)
{
    double2* b = reinterpret_cast<double2*>(s.b1);
    const q64::Div dnl(NL), dkt(KT);
    const int total = nxs * NL;
#pragma unroll 4
    for (int t = threadIdx.x; t < total; t += blockDim.x) {
        const int pl = dnl(t), L = t - pl * NL, bb = dkt(L), kk = L - bb * KT;
        double2 v = make_double2(0.0, 0.0);
        if (kk < kt && bb < nbb) v = T[((size_t)(bb0 + bb) * nxs + pl) * plane + base + kk];
        b[plane_x[pl] * NL + L] = v;
        atomicMax(s.e + L, q64::exp_of(v));
    }
    __syncthreads();
}

template <int R, bool ENERGY>
__global__ void __launch_bounds__(X_THREADS, R == WIDE_RADIX ? 1 : 3)
    xpass64(LocalArgs a, int nb, double2* __restrict__ T, const double* __restrict__ vloc, const int4* __restrict__ tw_g)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int n1 = a.n1, n2 = a.n2, n3 = a.n3, KT = a.kt, BB = a.bb, NL = KT * BB;
    const int TPL = parts_per_line(NL);
    XSmem s = x_smem(smem_raw, n1, KT, NL, true);
    x_smem_ints(s, ENERGY ? 2 * NL + 2 * NL * TPL : 0, n1, NL);
    const int j = blockIdx.y, k0 = blockIdx.x * KT, kt = min(KT, n3 - k0);
    int bb0 = blockIdx.z * BB, nxs = a.nxs;
    const int* plane_x = a.plane_x;
    if (a.items) {  // batched: (item, first band) of this band block
        const int2 xb = a.xblk[blockIdx.z];
        const LocalItem I = a.items[xb.x];
        bb0 = xb.y;
        nb = I.nb;
        nxs = I.nxs;
        plane_x = I.plane_x;
        T += I.t_off;
    }
    const int nbb = min(BB, nb - bb0);
    const size_t plane = (size_t)n2 * n3, base = (size_t)j * n3 + k0;
    const q64::Div dkt(KT), dnl(NL);
    for (int t = threadIdx.x; t < n1; t += blockDim.x) { s.tw[t] = tw_g[t]; s.xpl[t] = -1; }
    for (int t = threadIdx.x; t < NL; t += blockDim.x) { s.e[t] = q64::EXP_NONE; s.mag[t] = 0u; }
    if (threadIdx.x == 0) *s.ev = q64::EXP_NONE;
    __syncthreads();
    int ve = q64::EXP_NONE;
    for (int t = threadIdx.x; t < n1 * KT; t += blockDim.x) {
        const int x = dkt(t), kk = t - x * KT;
        const double v = kk < kt ? vloc[(size_t)x * plane + base + kk] : 0.0;
        s.vq[t] = make_int2(__double2loint(v), __double2hiint(v));
        ve = max(ve, q64::exp_of(make_double2(v, 0.0)));
    }
    ve = __reduce_max_sync(0xffffffffu, ve);
    if ((threadIdx.x & 31) == 0) atomicMax(s.ev, ve);
    for (int t = threadIdx.x; t < nxs; t += blockDim.x) s.xpl[plane_x[t]] = t;
    x_load(s, T, plane_x, nxs, plane, base, KT, NL, kt, nbb, bb0);
    const bool vbad = *s.ev >= q64::EXP_BAD;
    const int vu = (*s.ev == q64::EXP_NONE || vbad) ? 0 : *s.ev;  // |V| < 2^vu
    const auto x_mag = [&](int L, int x) {
        return s.xpl[x] < 0 ? 0u : q64::magnitude(reinterpret_cast<const double2*>(s.b1)[x * NL + L], s.e[L]);
    };
    take_units<R>(NL, n1, s.e, s.u, n1, x_mag);
    for (int t = threadIdx.x; t < n1 * KT; t += blockDim.x) {
        const int2 w = s.vq[t];
        // Q62 of V 2^-vu; 2^62 - 1 at most, so that the high word stays below 2^30
        const long long q = min(q64::from_double(__hiloint2double(w.y, w.x), vu - 62), (1ll << 62) - 1);
        int h, l;
        q64::words(q, h, l);
        s.vq[t] = make_int2(l, h);
    }
    __syncthreads();
    const bool gb = q64::transform<R == WIDE_RADIX, +1>(XLoad{reinterpret_cast<const double2*>(s.b1), s.xpl, s.u, NL},
                                             Lines{s.b0, 1, NL}, Lines{s.b1, 1, NL}, a.Lx, NL, s.tw);
    longlong2 *f = gb ? s.b1 : s.b0, *o = gb ? s.b0 : s.b1;
    if constexpr (ENERGY) {
        // FP64 sums of V|psi(r)|^2 and |psi(r)|^2: TPL strided slices of x per
        // line, combined in a fixed order
        double *lsum = s.tail, *psum = s.tail + 2 * NL;
        for (int t = threadIdx.x; t < NL * TPL; t += blockDim.x) {
            const int part = dnl(t), L = t - part * NL, kk = L - dkt(L) * KT;
            double s1 = 0.0, s0 = 0.0;
            for (int x = part; x < n1; x += TPL) {
                const double2 v = q64::to_double(f[x * NL + L], s.u[L], s.e[L] >= q64::EXP_BAD);
                const double w = kk < kt ? vloc[(size_t)x * plane + base + kk] : 0.0;
                const double m = v.x * v.x + v.y * v.y;
                s0 += m;
                s1 += w * m;
            }
            psum[2 * t] = s1;
            psum[2 * t + 1] = s0;
        }
        __syncthreads();
        for (int L = threadIdx.x; L < NL; L += blockDim.x) {
            double s1 = 0.0, s0 = 0.0;
            for (int part = 0; part < TPL; ++part) {
                s1 += psum[2 * (part * NL + L)];
                s0 += psum[2 * (part * NL + L) + 1];
            }
            lsum[2 * L] = s1;
            lsum[2 * L + 1] = s0;
        }
        __syncthreads();
        const int nslots = gridDim.x * gridDim.y, slot = blockIdx.y * gridDim.x + blockIdx.x;
        for (int bb = threadIdx.x; bb < nbb; bb += blockDim.x) {
            double s1 = 0.0, s0 = 0.0;
            for (int kk = 0; kk < kt; ++kk) {
                s1 += lsum[2 * (bb * KT + kk)];
                s0 += lsum[2 * (bb * KT + kk) + 1];
            }
            double* e = a.epart + ((size_t)(a.e_band0 + bb0 + bb) * nslots + slot) * 2;
            e[0] = s1;
            e[1] = s0;
        }
    }
    // psi(r) V, and the lines' magnitudes
    {
        int cur = -1;
        unsigned m = 0u;
        for (int t = threadIdx.x; t < n1 * NL; t += blockDim.x) {
            const int x = dnl(t), L = t - x * NL, kk = L - dkt(L) * KT;
            if (L != cur) {
                if (cur >= 0) atomicOr(s.mag + cur, m);
                cur = L;
                m = 0u;
            }
            const longlong2 v = f[t];
            const int2 w = s.vq[x * KT + kk];
            const longlong2 q = make_longlong2(q64::mul(v.x, w.x, w.y), q64::mul(v.y, w.x, w.y));
            const int p = (int)(q.x >> 32), r = (int)(q.y >> 32);
            m |= (unsigned)(p ^ (p >> 31)) | (unsigned)(r ^ (r >> 31));
            f[t] = q;
        }
        if (cur >= 0) atomicOr(s.mag + cur, m);
    }
    __syncthreads();
    for (int L = threadIdx.x; L < NL; L += blockDim.x) {
        // |V psi| < 2^bits units 2^(u + vu): to the line's bits
        const int bits = 64 - __clz(s.mag[L]);
        int fb = q64::headroom(n1);
        if (R != PLAIN && n1 > q64::LONG) {
            unsigned sum = 0u;
            for (int x = 0; x < n1; ++x) sum += q64::magnitude(f[x * NL + L], 0, bits);
            fb = q64::headroom(n1, sum);
        }
        const int sh = fb - bits;
        s.mag[L] = (unsigned)sh;
        s.u[L] += vu - sh;
    }
    __syncthreads();
    const bool rb = q64::transform<R == WIDE_RADIX, -1>(XShift{f, reinterpret_cast<const int*>(s.mag), NL}, Lines{o, 1, NL},
                                             Lines{f, 1, NL}, a.Lx, NL, s.tw);
    const longlong2* r = rb ? f : o;
    const int total = nxs * NL;
    for (int t = threadIdx.x; t < total; t += blockDim.x) {
        const int pl = dnl(t), L = t - pl * NL, bb = dkt(L), kk = L - bb * KT;
        if (kk < kt && bb < nbb)
            T[((size_t)(bb0 + bb) * nxs + pl) * plane + base + kk] =
                q64::to_double(r[plane_x[pl] * NL + L], s.u[L], vbad || s.e[L] >= q64::EXP_BAD);
    }
}

template <int R>
__global__ void __launch_bounds__(X_THREADS, R == WIDE_RADIX ? 1 : 3)
    xdensity64(LocalArgs a, int nb, const double2* __restrict__ T, const double* __restrict__ occ,
               double* __restrict__ rho, const int4* __restrict__ tw_g)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int n1 = a.n1, n2 = a.n2, n3 = a.n3, KT = a.kt, BB = a.bb, NL = KT * BB;
    XSmem s = x_smem(smem_raw, n1, KT, NL, false);
    x_smem_ints(s, n1 * KT, n1, NL);
    double* acc = s.tail;
    const int j = blockIdx.y, k0 = blockIdx.x * KT, kt = min(KT, n3 - k0);
    const size_t plane = (size_t)n2 * n3, base = (size_t)j * n3 + k0;
    const q64::Div dkt(KT);
    for (int t = threadIdx.x; t < n1; t += blockDim.x) { s.tw[t] = tw_g[t]; s.xpl[t] = -1; }
    for (int t = threadIdx.x; t < n1 * KT; t += blockDim.x) acc[t] = 0.0;
    __syncthreads();
    for (int t = threadIdx.x; t < a.nxs; t += blockDim.x) s.xpl[a.plane_x[t]] = t;
    for (int bb0 = 0; bb0 < nb; bb0 += BB) {
        const int nbb = min(BB, nb - bb0);
        for (int t = threadIdx.x; t < NL; t += blockDim.x) s.e[t] = q64::EXP_NONE;
        __syncthreads();
        x_load(s, T, a.plane_x, a.nxs, plane, base, KT, NL, kt, nbb, bb0);
        take_units<R>(NL, n1, s.e, s.u, n1, [&](int L, int x) {
            return s.xpl[x] < 0 ? 0u : q64::magnitude(reinterpret_cast<const double2*>(s.b1)[x * NL + L], s.e[L]);
        });
        __syncthreads();
        const bool gb = q64::transform<R == WIDE_RADIX, +1>(XLoad{reinterpret_cast<const double2*>(s.b1), s.xpl, s.u, NL},
                                                 Lines{s.b0, 1, NL}, Lines{s.b1, 1, NL}, a.Lx, NL, s.tw);
        const longlong2* f = gb ? s.b1 : s.b0;
        for (int t = threadIdx.x; t < n1 * KT; t += blockDim.x) {
            const int x = dkt(t), kk = t - x * KT;
            double r = acc[t];
            for (int bb = 0; bb < nbb; ++bb) {
                const int L = bb * KT + kk;
                const double2 v = q64::to_double(f[x * NL + L], s.u[L], s.e[L] >= q64::EXP_BAD);
                r += occ[bb0 + bb] * (v.x * v.x + v.y * v.y);
            }
            acc[t] = r;
        }
        __syncthreads();
    }
    for (int t = threadIdx.x; t < n1 * KT; t += blockDim.x) {
        const int x = dkt(t), kk = t - x * KT;
        if (kk < kt) rho[(size_t)x * plane + base + kk] += acc[t];
    }
}

// ---- launches ---------------------------------------------------------------
bool wide(const LocalArgs& a) { return fft_needs_wide(a.Lx) || fft_needs_wide(a.Ly) || fft_needs_wide(a.Lz); }

template <typename K>
cudaError_t smem_limit(K kernel, size_t bytes)
{
    return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
}

// f(plane size, kind) with the kernel variant of the grid
template <typename F>
cudaError_t with_variant(const LocalArgs& a, F&& f)
{
    const bool small = plane_bytes(a, true) * SmallPlane::blocks <= SMEM_MAX;
    if (wide(a)) return f(BigPlane{}, std::integral_constant<int, WIDE_RADIX>{});
    if (std::max({a.n1, a.n2, a.n3}) > q64::LONG) {
        using R = std::integral_constant<int, LONG_AXIS>;
        return small ? f(SmallPlane{}, R{}) : f(BigPlane{}, R{});
    }
    using R = std::integral_constant<int, PLAIN>;
    return small ? f(SmallPlane{}, R{}) : f(BigPlane{}, R{});
}

template <typename SZ, int R>
cudaError_t run_local(const LocalArgs& a, int nb, const double2* psi, double2* hpsi, const double* kinetic, double2* T,
                      const double* vloc, const int4* twx, const int4* twy, const int4* twz, dim3 gp, dim3 gx,
                      cudaStream_t st, Prof* prof)
{
    const int tw = plane_bytes(a, true) <= SMEM_MAX;
    const size_t sp = plane_bytes(a, tw), sx = xpass_bytes(a);
    auto g2r = g2r64<SZ, R>;
    auto r2g = r2g64<SZ, R>;
    auto xp = a.epart ? xpass64<R, true> : xpass64<R, false>;
    cudaError_t e;
    if ((e = smem_limit(g2r, sp)) || (e = smem_limit(r2g, sp)) || (e = smem_limit(xp, sx))) return e;
    for (int i = 0; i < 2; ++i)
        if (a.psi_in[i] && (e = cudaStreamWaitEvent(st, a.psi_in[i], 0))) return e;
    int h = prof ? prof->open(PH_G2R, st) : -1;
    g2r<<<gp, SZ::threads, sp, st>>>(a, psi, T, twy, twz, tw);
    if (prof) prof->close(h, st);
    if (a.after_g2r && (e = cudaEventRecord(a.after_g2r, st))) return e;
    h = prof ? prof->open(PH_XPASS, st) : -1;
    xp<<<gx, X_THREADS, sx, st>>>(a, nb, T, vloc, twx);
    if (prof) prof->close(h, st);
    h = prof ? prof->open(PH_R2G, st) : -1;
    r2g<<<gp, SZ::threads, sp, st>>>(a, T, psi, hpsi, kinetic, twy, twz, tw);
    if (prof) prof->close(h, st);
    return cudaGetLastError();
}

}  // namespace

size_t local64_xpass_smem(const LocalArgs& a) { return xpass_bytes(a); }

// 32 lines per block: 8 z-values (128-byte runs of T) by 4 bands, halved until
// two blocks share an SM
void local64_xpass_shape(LocalArgs* a)
{
    a->kt = std::min(8, a->n3);
    a->bb = 4;
    while (a->bb > 1 && 2 * sizeof(longlong2) * (size_t)a->n1 * a->kt * a->bb > 100 * 1024) a->bb /= 2;
    while (a->kt > 1 && 2 * sizeof(longlong2) * (size_t)a->n1 * a->kt * a->bb > 100 * 1024) a->kt /= 2;
}

template <>
cudaError_t launch_local<double2, double>(const LocalArgs& a0, int nb, const double2* psi, double2* hpsi,
                                          const double* kinetic, double2* T, const double* vloc, const int4* twx,
                                          const int4* twy, const int4* twz, cudaStream_t st, Prof* prof)
{
    if (a0.nxs == 0 || nb == 0) return cudaSuccess;
    LocalArgs a = a0;
    while (a.bb > 1 && a.bb / 2 >= nb) a.bb /= 2;  // no lines for bands that are not there
    const dim3 gp(a.nxs, nb), gx(ceil_div(a.n3, a.kt), a.n2, ceil_div(nb, a.bb));
    return with_variant(a, [&](auto sz, auto w) {
        return run_local<decltype(sz), decltype(w)::value>(a, nb, psi, hpsi, kinetic, T, vloc, twx, twy, twz, gp, gx,
                                                           st, prof);
    });
}

template <>
cudaError_t launch_local_batch<double2, double>(const LocalArgs& a, int nbands, int max_nxs, int nxblk, double2* T,
                                                const double* vloc, const int4* twx, const int4* twy, const int4* twz,
                                                cudaStream_t st)
{
    if (!a.items || a.epart) return cudaErrorInvalidValue;
    if (max_nxs == 0 || nbands == 0 || nxblk == 0) return cudaSuccess;
    const dim3 gp(max_nxs, nbands), gx(ceil_div(a.n3, a.kt), a.n2, nxblk);
    return with_variant(a, [&](auto sz, auto w) {
        return run_local<decltype(sz), decltype(w)::value>(a, 0, nullptr, nullptr, nullptr, T, vloc, twx, twy, twz, gp,
                                                           gx, st, nullptr);
    });
}

template <typename SZ, int R>
static cudaError_t run_density(const LocalArgs& a, int nb, const double2* psi, const double* occ, double* rho, double2* T,
                               const int4* twx, const int4* twy, const int4* twz, cudaStream_t st)
{
    const int tw = plane_bytes(a, true) <= SMEM_MAX;
    const size_t sp = plane_bytes(a, tw), sx = xdensity_bytes(a);
    auto g2r = g2r64<SZ, R>;
    cudaError_t e;
    if ((e = smem_limit(g2r, sp)) || (e = smem_limit(xdensity64<R>, sx))) return e;
    g2r<<<dim3(a.nxs, nb), SZ::threads, sp, st>>>(a, psi, T, twy, twz, tw);
    xdensity64<R><<<dim3(ceil_div(a.n3, a.kt), a.n2), X_THREADS, sx, st>>>(a, nb, T, occ, rho, twx);
    return cudaGetLastError();
}

template <>
cudaError_t launch_density<double2>(const LocalArgs& a, int nb, const double2* psi, const double* occ, double* rho,
                                    double2* T, const int4* twx, const int4* twy, const int4* twz, cudaStream_t st,
                                    double*)
{
    if (a.items || a.epart) return cudaErrorInvalidValue;
    if (a.nxs == 0 || nb == 0) return cudaSuccess;
    return with_variant(a, [&](auto sz, auto w) {
        return run_density<decltype(sz), decltype(w)::value>(a, nb, psi, occ, rho, T, twx, twy, twz, st);
    });
}

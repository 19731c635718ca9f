// fft_q64.cuh — line transforms of the FP64 local term in 64-bit fixed point.
//
// GB300 executes FP64 at 1/64 of the FP32 rate, so a complex128 butterfly is
// bound by the FP64 pipe (a 72-point line: 1530 FP64 instructions, 715 clocks of
// an SM).  Here the lines are 64-bit integers in a unit 2^u of their own, and a
// butterfly is integer adds and 32 x 32 -> 64 bit multiply-adds, which run at
// 32 to 64 lanes per clock.  A line enters with its largest component at 2^FB, where
// FB leaves room for the growth of a transform of n points (every component of
// every partial sum stays below n sqrt(2) 2^FB < 2^62).  Rounding errors are then
// absolute, about three units per output, where the largest input is 2^55 units
// for n = 72: against long double transforms the 3-D round trip of the 8-atom
// cell is 6e-17 off in the 2-norm, the complex128 one 5e-16.  A bound by n wastes bits
// that lines of more than LONG points cannot spare (a few large elements of 500: 3e-15
// off, where complex128 is 5e-16), so these take their unit from the sum of their
// elements' magnitudes, which bounds every partial sum too.
//
// Twiddles are Q62 constants, each as two signed words (l, h): value
// (h 2^32 + l) 2^-62.  A product drops the l x l term (below one unit).
#pragma once

#include <climits>
#include <cmath>

#include "fft.cuh"

template <> struct Real<longlong2> { using type = long long; };

// exp(2 pi i j / n) as Q62 words (cos l, cos h, sin l, sin h): value (h 2^32 + l) 2^-62.
// Evaluated in the first octant in long double (at least 64 bits).
inline int4 q62_twiddle(int j, int n)
{
    const long double pi = 3.14159265358979323846264338327950288L;
    long long r = 8ll * j;  // eighths of a turn, in units of 1/n
    const int oct = (int)(r / n);
    r -= (long long)oct * n;
    const long double t = pi / 4 * (long double)((oct & 1) ? n - r : r) / (long double)n;
    long double c = std::cos(t), s = std::sin(t), x = 0, y = 0;
    switch (oct) {
        case 0: x = c; y = s; break;
        case 1: x = s; y = c; break;
        case 2: x = -s; y = c; break;
        case 3: x = -c; y = s; break;
        case 4: x = -c; y = -s; break;
        case 5: x = -s; y = -c; break;
        case 6: x = s; y = -c; break;
        default: x = c; y = -s; break;
    }
    auto words = [](long double v, int& l, int& h) {
        const long long q = std::llrint(std::ldexp(v, 62));
        l = (int)(uint32_t)q;
        if (l == INT_MIN) ++l;  // -l is formed for the conjugate
        h = (int)((q - l) >> 32);
    };
    int4 w;
    words(x, w.x, w.y);
    words(y, w.z, w.w);
    return w;
}

namespace q64 {

constexpr int EXP_NONE = -100000;  // exponent of a line without a nonzero element
constexpr int EXP_BAD = 100000;    // exponent of a line with an infinity or NaN

// bits of a line's largest input component: n sqrt(2) 2^FB < 2^62
HPSI_D int headroom(int n) { return 62 - (32 - __clz((int)(1.41422f * (float)n))); }

// e with |v.x|, |v.y| < 2^e (EXP_NONE for zero, EXP_BAD for an infinity or NaN)
HPSI_D int exp_of(double2 v)
{
    const int e = max((__double2hiint(v.x) >> 20) & 0x7ff, (__double2hiint(v.y) >> 20) & 0x7ff);
    if (e == 0x7ff) return EXP_BAD;
    return (v.x == 0.0 && v.y == 0.0) ? EXP_NONE : e - 1022;
}

// e with |v.x|, |v.y| < 2^e, at least 32
HPSI_D int bits_of(longlong2 v)
{
    const int a = (int)(v.x >> 32), b = (int)(v.y >> 32);
    const unsigned o = (unsigned)(a ^ (a >> 31)) | (unsigned)(b ^ (b >> 31));
    return 64 - __clz(o);
}

// Lines of more points take their unit from the sum of their magnitudes.  Below, the
// bound by n leaves 54 bits or more to the largest element: round trips of axes of 90
// to 120 points are 1.8e-16 to 3.5e-16 off, complex128 ones 3.1e-16 to 4.9e-16.  With it
// axes of 128 to 180 points were up to 5.3e-16 off (2.9e-16 to 4.6e-16).
constexpr int LONG = 120;

// |re| + |im| in units of 2^(e - 20) (e: the line's exponent), rounded up.  Integers, so
// that a sum does not depend on its order.
HPSI_D unsigned magnitude(double2 v, int e)
{
    if (e <= EXP_NONE || e >= EXP_BAD / 2) return 0u;
    return 1u + (unsigned)(scalbn(fabs(v.x), 20 - e) + scalbn(fabs(v.y), 20 - e));
}
// the same of v 2^u, v an integer of the transforms
HPSI_D unsigned magnitude(longlong2 v, int u, int e)
{
    if (e <= EXP_NONE || e >= EXP_BAD / 2) return 0u;
    const int a = (int)(v.x >> 32), b = (int)(v.y >> 32);
    const long long t = (long long)(a ^ (a >> 31)) + (b ^ (b >> 31)) + 2;  // the magnitude is below t 2^(32 + u)
    const int s = 52 + u - e;
    return s >= 0 ? (unsigned)(t << min(s, 31)) : 1u + (unsigned)(t >> min(-s, 63));
}

// bits of the largest element where the magnitudes add up to sum (in units of 2^(e - 20))
HPSI_D int headroom(int n, unsigned sum)
{
    return sum ? max(headroom(n), min(60, 62 - (12 - __clz((int)sum)))) : headroom(n);
}

// unit of a line whose components are below 2^e, for fb bits
HPSI_D int unit_of(int e, int fb) { return (e == EXP_NONE || e >= EXP_BAD / 2) ? 0 : e - fb; }

// rint(x 2^-u), |result| < 2^62
HPSI_D long long from_double(double x, int u)
{
    const uint32_t hi = (uint32_t)__double2hiint(x), lo = (uint32_t)__double2loint(x);
    const int e = (hi >> 20) & 0x7ff;
    const unsigned long long m = ((unsigned long long)((hi & 0xfffffu) | (e ? 0x100000u : 0u)) << 32 | lo) << 10;
    const int r = 1085 + u - (e ? e : 1);  // x = m 2^(e - 1085): shift right by r >= 1, rounding
    const unsigned long long t = m >> min(max(r - 1, 0), 63);
    const long long y = (long long)((t + 1) >> 1);
    return (int)hi < 0 ? -y : y;
}

HPSI_D longlong2 from_double(double2 v, int u) { return make_longlong2(from_double(v.x, u), from_double(v.y, u)); }

// v 2^u rounded to FP64 (half to even), on the integer pipe
HPSI_D double to_double(long long v, int u)
{
    if (v == 0) return 0.0;
    const unsigned long long a = v < 0 ? 0ull - (unsigned long long)v : (unsigned long long)v;
    const int lz = __clzll((long long)a);
    const unsigned long long n = a << lz;
    unsigned long long m = n >> 11;
    const uint32_t dropped = (uint32_t)n & 0x7ffu;
    m += (dropped + ((uint32_t)m & 1u) + 0x3ffu) >> 11;
    const int be = 63 - lz + u + 1023;
    const unsigned long long sign = (unsigned long long)v & (1ull << 63);
    if (be >= 1 && be < 2046) return __longlong_as_double((long long)(sign + ((unsigned long long)(be - 1) << 52) + m));
    return scalbn(__longlong_as_double((long long)(sign + (1022ull << 52) + m)), be - 1023);
}

HPSI_D double2 to_double(longlong2 v, int u, bool bad)
{
    const double nan = __longlong_as_double(0x7ff8000000000000ll);
    return bad ? make_double2(nan, nan) : make_double2(to_double(v.x, u), to_double(v.y, u));
}

// v 2^s, rounding when s < 0
HPSI_D long long shift(long long v, int s)
{
    if (s >= 0) return v << min(s, 63);
    const long long t = v >> min(-s - 1, 63);
    return (t + 1) >> 1;
}

HPSI_D longlong2 shift(longlong2 v, int s) { return make_longlong2(shift(v.x, s), shift(v.y, s)); }

// x = h 2^32 + l, both signed words
HPSI_D void words(long long x, int& h, int& l)
{
    l = (int)x;
    h = (int)(x >> 32) + (int)((uint32_t)l >> 31);
}

// (t 2^32 + m) 2^-30
HPSI_D long long combine(long long t, long long m)
{
    t += m >> 32;
    const uint32_t tl = (uint32_t)t, th = (uint32_t)((unsigned long long)t >> 32);
    const uint32_t hi = __funnelshift_l(tl, th, 2), lo = __funnelshift_l((uint32_t)m, tl, 2);
    return (long long)((unsigned long long)hi << 32 | lo);
}

// x c, c = (cl, ch) in Q62
HPSI_D long long mul(long long x, int cl, int ch)
{
    int h, l;
    words(x, h, l);
    return combine((long long)h * ch, (long long)h * cl + (long long)l * ch + (1ll << 29));
}

// x c + y d
HPSI_D long long dot(long long x, int cl, int ch, long long y, int dl, int dh)
{
    int xh, xl, yh, yl;
    words(x, xh, xl);
    words(y, yh, yl);
    return combine((long long)xh * ch + (long long)yh * dh,
                   (long long)xh * cl + (long long)xl * ch + (long long)yh * dl + (long long)yl * dh + (1ll << 29));
}

// a (re + i im), constants given as (l, h) words
HPSI_D longlong2 cmul(longlong2 a, int rl, int rh, int il, int ih)
{
    int xh, xl, yh, yl;
    words(a.x, xh, xl);
    words(a.y, yh, yl);
    const long long r = 1ll << 29;
    return make_longlong2(
        combine((long long)xh * rh + (long long)yh * -ih,
                (long long)xh * rl + (long long)xl * rh + (long long)yh * -il + (long long)yl * -ih + r),
        combine((long long)xh * ih + (long long)yh * rh,
                (long long)xh * il + (long long)xl * ih + (long long)yh * rl + (long long)yl * rh + r));
}

// a W, W from the table (cos l, cos h, sin l, sin h) of exp(+2 pi i j / n), conjugated for SIGN < 0
template <int SIGN>
HPSI_D longlong2 cmul(longlong2 a, int4 w)
{
    return cmul(a, w.x, w.y, SIGN > 0 ? w.z : -w.z, SIGN > 0 ? w.w : -w.w);
}

template <int SIGN>
HPSI_D void dft3(longlong2& a, longlong2& b, longlong2& c)
{
    const longlong2 s = cadd(b, c), d = csub(b, c);
    const longlong2 m = make_longlong2(a.x - (s.x >> 1), a.y - (s.y >> 1));
    a = cadd(a, s);
    // sin(2 pi / 3)
    const long long tx = mul(d.y, -1332128537, 929887697), ty = mul(d.x, -1332128537, 929887697);
    const longlong2 t = SIGN > 0 ? make_longlong2(-tx, ty) : make_longlong2(tx, -ty);
    b = cadd(m, t);
    c = csub(m, t);
}

template <int SIGN>
HPSI_D void dft4(longlong2& a, longlong2& b, longlong2& c, longlong2& d)
{
    const longlong2 a0 = cadd(a, c), a1 = csub(a, c), b0 = cadd(b, d), b1 = cmul_i(csub(b, d), SIGN);
    a = cadd(a0, b0);
    c = csub(a0, b0);
    b = cadd(a1, b1);
    d = csub(a1, b1);
}

// p-point DFT of v[0..P): v[q] <- sum_r v[r] W_P^{r q}
template <int P, int SIGN>
HPSI_D void dft(longlong2 (&v)[P], const int4* tw, int n)
{
    if constexpr (P == 2) {
        const longlong2 a = v[0];
        v[0] = cadd(a, v[1]);
        v[1] = csub(a, v[1]);
    } else if constexpr (P == 3) {
        dft3<SIGN>(v[0], v[1], v[2]);
    } else if constexpr (P == 4) {
        dft4<SIGN>(v[0], v[1], v[2], v[3]);
    } else if constexpr (P == 5) {
        // cos and sin of 2 pi / 5 and 4 pi / 5
        constexpr int c1l = 803819395, c1h = 331804471, s1l = -2002125123, s1h = 1021189159;
        constexpr int c2l = -803819395, c2h = -868675383, s2l = -357254181, s2h = 631129609;
        const longlong2 p = cadd(v[1], v[4]), q = cadd(v[2], v[3]), r = csub(v[1], v[4]), t = csub(v[2], v[3]);
        const longlong2 m1 = make_longlong2(v[0].x + dot(p.x, c1l, c1h, q.x, c2l, c2h),
                                            v[0].y + dot(p.y, c1l, c1h, q.y, c2l, c2h));
        const longlong2 m2 = make_longlong2(v[0].x + dot(p.x, c2l, c2h, q.x, c1l, c1h),
                                            v[0].y + dot(p.y, c2l, c2h, q.y, c1l, c1h));
        longlong2 n1 = make_longlong2(dot(r.x, s1l, s1h, t.x, s2l, s2h), dot(r.y, s1l, s1h, t.y, s2l, s2h));
        longlong2 n2 = make_longlong2(dot(r.x, s2l, s2h, t.x, -s1l, -s1h), dot(r.y, s2l, s2h, t.y, -s1l, -s1h));
        n1 = cmul_i(n1, SIGN);
        n2 = cmul_i(n2, SIGN);
        v[0] = cadd(v[0], cadd(p, q));
        v[1] = cadd(m1, n1);
        v[4] = csub(m1, n1);
        v[2] = cadd(m2, n2);
        v[3] = csub(m2, n2);
    } else if constexpr (P == 8) {
        // 2 x 4: 4-point DFTs of the even and odd elements, W_8^k on the odd ones
        dft4<SIGN>(v[0], v[2], v[4], v[6]);
        dft4<SIGN>(v[1], v[3], v[5], v[7]);
        constexpr int rl = -25716447, rh = 759250125;  // sqrt(1/2)
        const longlong2 a = v[3], b = v[7];
        // (r + i SIGN r) a, i SIGN v[5], (-r + i SIGN r) b
        const longlong2 o1 = SIGN > 0 ? make_longlong2(mul(a.x - a.y, rl, rh), mul(a.x + a.y, rl, rh))
                                      : make_longlong2(mul(a.x + a.y, rl, rh), mul(a.y - a.x, rl, rh));
        const longlong2 o2 = cmul_i(v[5], SIGN);
        const longlong2 o3 = SIGN > 0 ? make_longlong2(mul(-b.x - b.y, rl, rh), mul(b.x - b.y, rl, rh))
                                      : make_longlong2(mul(b.y - b.x, rl, rh), mul(-b.x - b.y, rl, rh));
        const longlong2 e0 = v[0], e1 = v[2], e2 = v[4], e3 = v[6], o0 = v[1];
        v[0] = cadd(e0, o0);
        v[4] = csub(e0, o0);
        v[1] = cadd(e1, o1);
        v[5] = csub(e1, o1);
        v[2] = cadd(e2, o2);
        v[6] = csub(e2, o2);
        v[3] = cadd(e3, o3);
        v[7] = csub(e3, o3);
    } else if constexpr (P == 9) {
        // 3 x 3: v[3 a + b]: 3-point DFTs over a, W_9^{b k}, 3-point DFTs over b; output k + 3 l
        dft3<SIGN>(v[0], v[3], v[6]);
        dft3<SIGN>(v[1], v[4], v[7]);
        dft3<SIGN>(v[2], v[5], v[8]);
        // W_9, W_9^2, W_9^4
        constexpr int g = SIGN;
        v[4] = cmul(v[4], -1633652124, 822533958, g * 2016164183, g * 690187940);
        v[7] = cmul(v[7], 96060625, 186453311, g * 37236404, g * 1057429273);
        v[5] = cmul(v[5], 96060625, 186453311, g * 37236404, g * 1057429273);
        v[8] = cmul(v[8], 1537591498, -1008987269, g * -1978927779, g * 367241333);
        dft3<SIGN>(v[0], v[1], v[2]);
        dft3<SIGN>(v[3], v[4], v[5]);
        dft3<SIGN>(v[6], v[7], v[8]);
        const longlong2 x1 = v[1], x2 = v[2], x5 = v[5];
        v[1] = v[3];
        v[2] = v[6];
        v[3] = x1;
        v[5] = v[7];
        v[6] = x2;
        v[7] = x5;
    } else {
        // odd prime: sums and differences of the elements r and P - r against
        // cos and sin of 2 pi q r / P from the table
        constexpr int H = (P - 1) / 2;
        const int step = n / P;
        longlong2 s[H], d[H];
#pragma unroll
        for (int r = 1; r <= H; ++r) {
            s[r - 1] = cadd(v[r], v[P - r]);
            d[r - 1] = csub(v[r], v[P - r]);
        }
        const longlong2 x0 = v[0];
#pragma unroll
        for (int r = 0; r < H; ++r) v[0] = cadd(v[0], s[r]);
#pragma unroll
        for (int q = 1; q <= H; ++q) {
            longlong2 c = x0, t = make_longlong2(0, 0);
#pragma unroll
            for (int r = 1; r <= H; ++r) {
                const int4 w = tw[((q * r) % P) * step];
                c = cadd(c, make_longlong2(mul(s[r - 1].x, w.x, w.y), mul(s[r - 1].y, w.x, w.y)));
                t = cadd(t, make_longlong2(mul(d[r - 1].x, w.z, w.w), mul(d[r - 1].y, w.z, w.w)));
            }
            t = cmul_i(t, SIGN);
            v[q] = cadd(c, t);
            v[P - q] = csub(c, t);
        }
    }
}

// t / d by one multiply, exact for t < 2^22
struct Div {
    int d;
    float inv;
    HPSI_D explicit Div(int d_) : d(d_), inv(1.0f / (float)d_) {}
    HPSI_D int operator()(int t) const { return (int)(((float)t + 0.5f) * inv); }
};

// lines in shared memory: element e of line L at b[L ls + e es]
struct Lines {
    longlong2* b;
    int ls, es;
    HPSI_D longlong2 operator()(int L, int e) const { return b[L * ls + e * es]; }
    HPSI_D void operator()(int L, int e, longlong2 v) const { b[L * ls + e * es] = v; }
};

// the plane's rows in use (PlaneRows): line L is row L or, past jr, L + gap
struct RowLines {
    longlong2* b;
    int ls, jr, gap;
    HPSI_D int row(int L) const { return L + (L > jr ? gap : 0); }
    HPSI_D longlong2 operator()(int L, int e) const { return b[row(L) * ls + e]; }
    HPSI_D void operator()(int L, int e, longlong2 v) const { b[row(L) * ls + e] = v; }
};

// one Stockham stage (fft.cuh), consecutive threads on consecutive lines
template <int P, int SIGN, typename LD, typename ST>
HPSI_D void stage(const LD& ld, const ST& st, int n, int Ns, const Div& nl, const int4* tw)
{
    const int nbf = n / P, total = nl.d * nbf, tstep = n / (Ns * P);
    const Div dns(Ns);
    for (int t = threadIdx.x; t < total; t += blockDim.x) {
        const int i = nl(t), L = t - i * nl.d, hi = dns(i), k = i - hi * Ns, tj = k * tstep;
        longlong2 v[P];
#pragma unroll
        for (int q = 0; q < P; ++q) v[q] = ld(L, i + q * nbf);
        if (k > 0) {
#pragma unroll
            for (int q = 1; q < P; ++q) v[q] = cmul<SIGN>(v[q], tw[q * tj]);
        }
        dft<P, SIGN>(v, tw, n);
        const int base = hi * Ns * P + k;
#pragma unroll
        for (int q = 0; q < P; ++q) st(L, base + q * Ns, v[q]);
    }
}

template <bool WIDE, int SIGN, typename LD, typename ST>
HPSI_D void stage_of(int p, const LD& ld, const ST& st, int n, int Ns, const Div& nl, const int4* tw)
{
    switch (p) {
        case 8: stage<8, SIGN>(ld, st, n, Ns, nl, tw); break;
        case 9: stage<9, SIGN>(ld, st, n, Ns, nl, tw); break;
        case 4: stage<4, SIGN>(ld, st, n, Ns, nl, tw); break;
        case 2: stage<2, SIGN>(ld, st, n, Ns, nl, tw); break;
        case 3: stage<3, SIGN>(ld, st, n, Ns, nl, tw); break;
        case 5: stage<5, SIGN>(ld, st, n, Ns, nl, tw); break;
        default:
            if constexpr (WIDE) {
                switch (p) {
                    case 7: stage<7, SIGN>(ld, st, n, Ns, nl, tw); break;
                    case 11: stage<11, SIGN>(ld, st, n, Ns, nl, tw); break;
                    case 13: stage<13, SIGN>(ld, st, n, Ns, nl, tw); break;
                    default: break;
                }
            }
            break;
    }
}

// Transform of nl lines: the first stage reads through ld and writes A, the
// others go back and forth between A and B.  ld must not read A (it may read B).
// Ends with a barrier; true if the result is in B.
template <bool WIDE, int SIGN, typename LD, typename ST>
HPSI_D bool transform(const LD& ld, const ST& A, const ST& B, const FftLen& L, int lines, const int4* tw)
{
    const Div nl(lines);
    if (L.nst == 0) {
        for (int t = threadIdx.x; t < lines; t += blockDim.x) A(t, 0, ld(t, 0));
        __syncthreads();
        return false;
    }
    stage_of<WIDE, SIGN>(L.rad[0], ld, A, L.n, 1, nl, tw);
    __syncthreads();
    for (int s = 1; s < L.nst; ++s) {
        stage_of<WIDE, SIGN>(L.rad[s], s & 1 ? A : B, s & 1 ? B : A, L.n, (int)L.ns[s].d, nl, tw);
        __syncthreads();
    }
    return (L.nst - 1) & 1;
}

}  // namespace q64

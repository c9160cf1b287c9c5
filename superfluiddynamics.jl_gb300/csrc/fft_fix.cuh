// fft_fix.cuh -- FP64 fields transformed in 64-bit fixed point.
//
// GB300 runs FP64 at 1.7 operations per clock and SM, 32-bit integer additions at
// 119 and 32x32 -> 64-bit multiply-adds at ~24 (measured).  A transform in
// FP64 arithmetic is bound by that pipe alone (72 operations per cell and
// pass of 256-cell lines: 2.5 ms at 256^3, against 0.08 ms of memory traffic),
// so the passes of FP64 fields hold the values of a line as 64-bit integers
// on a common quantum: a complex addition is four 32-bit additions, a product
// by a constant of 63 bits twelve multiply-adds.
//
// Accuracy and range.  The quantum of a line comes from its 2-norm: with
// ||x|| <= 2^E a value is an integer multiple of 2^(E - 60), rounded to nearest
// on entry.  A sum of m of the line's values is at most sqrt(m) ||x||, a
// transform of n cells multiplies the norm by sqrt(n), the phase (modulus at
// most 1) does not raise it, and each product by a table constant (2^62 times
// its value, used as a 2^64 one) divides by 4.  So for n <= 256 = 16 x 16 every
// stage holds at most 4 ||x|| = 2^62 in modulus: sqrt(16) after stage A,
// sqrt(256) / 4 after stage B, sqrt(16 256) / 16 after its backward part,
// 256 / 64 at the end; shorter lines stay below.  The quantum of each stage
// grows like the values do, so every rounding on the way is about 2^-57 of the
// line's rms (n = 256; smaller for shorter lines) whatever its shape, and the
// result is rounded once to FP64 (2^-53 of itself): closer to the exact pass
// than FP64 arithmetic, whose every operation rounds at 2^-53
// (tests/test_gpu_fixed_point.py holds it to that).
//
// A line that holds NaN or infinity (or a component of 2^1017 and above,
// whose square is infinite anyway) comes out as NaN throughout, as a sum over
// it would.
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

namespace gpss {

// a complex value in fixed point
struct __align__(16) fxc {
    long long x, y;
};

__device__ __forceinline__ long long fx_madw(int a, int b, long long c)
{
    long long d;
    asm("mad.wide.s32 %0, %1, %2, %3;" : "=l"(d) : "r"(a), "r"(b), "l"(c));
    return d;
}
// a = h 2^32 + l with both halves signed, so that signed multiply-adds serve
// every partial product
__device__ __forceinline__ void fx_split(long long a, int &h, int &l)
{
    l = (int)a;
    h = (int)(a >> 32) + (int)((unsigned)l >> 31);
}
// A product's partial sums: S in units of 2^64 / 2^64, X in units of 2^32 / 2^64
// of the result.  X starts at one half (rounding) plus 2^63, which keeps it
// unsigned so that its upper half adds without a sign extension; S starts at
// minus that offset.  The low-by-low product (below the rounding) is left out;
// with signed halves its mean is zero.
constexpr long long FX_S0 = -(1LL << 31);
constexpr long long FX_X0 = (long long)((1ULL << 63) + (1ULL << 31));
__device__ __forceinline__ long long fx_fold(long long S, long long X)
{
    return S + (long long)((unsigned long long)X >> 32);
}
// a (rh 2^32 + rl) 2^-64
__device__ __forceinline__ long long fx_rmul(long long a, int rh, int rl)
{
    int h, l;
    fx_split(a, h, l);
    return fx_fold(fx_madw(h, rh, FX_S0), fx_madw(l, rh, fx_madw(h, rl, FX_X0)));
}

// A table constant: 2^62 times a complex number of modulus at most 1, the
// halves of each component signed (c = h 2^32 + l).
// a * c / 4
__device__ __forceinline__ fxc fx_cmul(fxc a, int4 c)
{
    int xh, xl, yh, yl;
    fx_split(a.x, xh, xl);
    fx_split(a.y, yh, yl);
    const int rl = c.x, rh = c.y, pl = c.z, ph = c.w, ml = -c.z, mh = -c.w;
    fxc o;
    o.x = fx_fold(fx_madw(xh, rh, fx_madw(yh, mh, FX_S0)),
                  fx_madw(xl, rh, fx_madw(yl, mh, fx_madw(xh, rl, fx_madw(yh, ml, FX_X0)))));
    o.y = fx_fold(fx_madw(yh, rh, fx_madw(xh, ph, FX_S0)),
                  fx_madw(yl, rh, fx_madw(xl, ph, fx_madw(yh, rl, fx_madw(xh, pl, FX_X0)))));
    return o;
}
// a / 4, rounded: what a product by the constant 1 gives
__device__ __forceinline__ fxc fx_quarter(fxc a)
{
    return fxc{(a.x + 2) >> 2, (a.y + 2) >> 2};
}

// ---- multipliers: real factors of a spectrum that differ by orders of magnitude
//
// A multiplier pass (the Laplacian's (2 pi k / L)^2, an imaginary-time factor
// above 1) does not keep the line's norm, and its largest factor belongs to
// modes that hardly carry weight: on the quantum that this factor asks for, the
// low modes would be held in 2 log2(n / 2) bits less.  So each table entry has a
// 62-bit significand and its own exponent {low half, high half, exponent less the
// table's, 0}, and a line takes a new quantum from the 2-norm of its products
// (gen_pass_kernel and pass_kernel: one more reduction per line; 64^3 explicit
// Runge-Kutta, 8 steps, 2102 -> 2141 us; backward Euler, a step, 64^3 211 -> 215,
// 256^3 7120 -> 7560 us).

// a times the significand / 4
__device__ __forceinline__ fxc fx_mult(fxc a, int4 m) { return fxc{fx_rmul(a.x, m.y, m.x), fx_rmul(a.y, m.y, m.x)}; }
// the square of |a 2^e| 2^-20, e at most 0
__device__ __forceinline__ float fx_mult_norm2(fxc a, int e)
{
    const float f = __int_as_float((127 + max(e - 20, -126)) << 23);
    const float x = (float)a.x * f, y = (float)a.y * f;
    return fmaf(x, x, y * y);
}
// the exponent by which a line whose products have the sum of squares s (as
// above) is shifted down so that its 2-norm takes `bits` bits; below 2^-100 the
// products are rounding of zeros
__device__ __forceinline__ int fx_mult_shift(float s, int bits)
{
    const int es = (__float_as_int(fmaxf(s, 7.8886e-31f)) >> 23) - 127;  // s < 2^(es + 1)
    return ((es + 2) >> 1) + 20 - bits;
}
// v 2^s, rounded
__device__ __forceinline__ long long fx_scale2(long long v, int s)
{
    const int r = min(max(-s, 0), 62);
    return ((v << min(max(s, 0), 63)) + ((1LL << r) >> 1)) >> r;
}
__device__ __forceinline__ fxc fx_scale2(fxc a, int s) { return fxc{fx_scale2(a.x, s), fx_scale2(a.y, s)}; }

// the DFT-16's own constants as 2^64 times a number below 1/2, signed halves
constexpr long long FX_TAN16 = 0x32ebebc0aa62b00fLL;   // tan(pi/16)
constexpr long long FX_SIN8 = 0x61f78a9abaa58b47LL;    // sin(pi/8)
constexpr long long FX_1MH = 0x4afb0ccc06219b7cLL;     // 1 - sqrt(1/2)
__host__ __device__ constexpr int fx_lo(long long c) { return (int)(unsigned)(c & 0xffffffffLL); }
__host__ __device__ constexpr int fx_hi(long long c) { return (int)((c - (long long)fx_lo(c)) >> 32); }

// rotation by D pi/8 (D = +-1) in three shears (Buneman's lifting form of a
// plane rotation): 9 multiply-adds instead of 12
template <int D> __device__ __forceinline__ fxc fx_rot8(fxc a)
{
    constexpr int th = -D * fx_hi(FX_TAN16), tl = -D * fx_lo(FX_TAN16);
    constexpr int sh = D * fx_hi(FX_SIN8), sl = D * fx_lo(FX_SIN8);
    a.x += fx_rmul(a.y, th, tl);
    a.y += fx_rmul(a.x, sh, sl);
    a.x += fx_rmul(a.y, th, tl);
    return a;
}
// a sqrt(1/2)
__device__ __forceinline__ long long fx_half_sqrt(long long a)
{
    return a + fx_rmul(a, -fx_hi(FX_1MH), -fx_lo(FX_1MH));
}

// a * exp(DIR 2 pi i M / 16)
template <int M, int DIR> __device__ __forceinline__ fxc fx_mul_w16(fxc a)
{
    constexpr int m = (((DIR * M) % 16) + 16) % 16;  // exp(2 pi i m / 16)
    if constexpr (m == 0) return a;
    else if constexpr (m == 4) return fxc{-a.y, a.x};
    else if constexpr (m == 8) return fxc{-a.x, -a.y};
    else if constexpr (m == 12) return fxc{a.y, -a.x};
    else if constexpr (m % 2 == 0) {
        // (sc + i ss) / sqrt 2
        constexpr int sc = (m == 2 || m == 14) ? 1 : -1, ss = (m == 2 || m == 6) ? 1 : -1;
        const long long u = ss > 0 ? a.x - a.y : a.x + a.y;  // sc x - ss y, up to sc when sc ss > 0 ...
        const long long v = ss > 0 ? a.x + a.y : a.y - a.x;
        // (x + i y)(sc + i ss) = (sc x - ss y) + i (ss x + sc y)
        if constexpr (sc > 0) return fxc{fx_half_sqrt(u), fx_half_sqrt(v)};
        else if constexpr (ss > 0) return fxc{-fx_half_sqrt(v), fx_half_sqrt(u)};   // m = 6: -(x + y), x - y
        else return fxc{fx_half_sqrt(a.y - a.x), -fx_half_sqrt(a.x + a.y)};          // m = 10
    } else if constexpr (m == 1) return fx_rot8<1>(a);
    else if constexpr (m == 15) return fx_rot8<-1>(a);
    else if constexpr (m == 3) { const fxc b = fx_rot8<-1>(a); return fxc{-b.y, b.x}; }
    else if constexpr (m == 5) { const fxc b = fx_rot8<1>(a); return fxc{-b.y, b.x}; }
    else if constexpr (m == 7) { const fxc b = fx_rot8<-1>(a); return fxc{-b.x, -b.y}; }
    else if constexpr (m == 9) { const fxc b = fx_rot8<1>(a); return fxc{-b.x, -b.y}; }
    else if constexpr (m == 11) { const fxc b = fx_rot8<-1>(a); return fxc{b.y, -b.x}; }
    else { const fxc b = fx_rot8<1>(a); return fxc{b.y, -b.x}; }  // m = 13
}

// log2 of a line length
template <int N> struct FxLog { static constexpr int V = 1 + FxLog<N / 2>::V; };
template <> struct FxLog<1> { static constexpr int V = 0; };

// The largest upper word of the magnitudes of n values' components.  Upper
// words of non-negative doubles order like floats, and a float maximum takes
// the absolute value for free; NaN-propagating, so that words that look like a
// float NaN (2^1017 and above) win.
template <int N> __device__ __forceinline__ int fx_max_word(const double2 *v)
{
    float m = 0.f;
#pragma unroll
    for (int j = 0; j < N; j++) {
        const float a = fabsf(__int_as_float(__double2hiint(v[j].x)));
        const float b = fabsf(__int_as_float(__double2hiint(v[j].y)));
        asm("max.NaN.f32 %0, %0, %1;" : "+f"(m) : "f"(a));
        asm("max.NaN.f32 %0, %0, %1;" : "+f"(m) : "f"(b));
    }
    return __float_as_int(m);
}
// the biased exponent that sums of squares are taken relative to
__device__ __forceinline__ int fx_ref(int word) { return max(word >> 20, 64); }
// sum of the squares of n values over 2^(2 (ref - 1023)), ref at least the
// exponent of each: an upper word becomes the float of the same significand by
// a shift and an offset (components below 2^-100 of the reference count as that)
template <int N> __device__ __forceinline__ float fx_norm2(const double2 *v, int ref)
{
    const float low = __int_as_float(max(ref - 100, 0) << 20);
    const int off = 0x3f800000 - (int)((unsigned)ref << 23);
    float s = 0.f;
#pragma unroll
    for (int j = 0; j < N; j++) {
        const float a = __int_as_float((int)((unsigned)__float_as_int(fmaxf(
            fabsf(__int_as_float(__double2hiint(v[j].x))), low)) << 3) + off);
        const float b = __int_as_float((int)((unsigned)__float_as_int(fmaxf(
            fabsf(__int_as_float(__double2hiint(v[j].y))), low)) << 3) + off);
        s = fmaf(a, a, fmaf(b, b, s));
    }
    return s;
}
// log2 of the quantum of a line: its 2-norm is sqrt(s) 2^(ref - 1023), at most
// 2^(q + 60) (s, of truncated significands, is short of the true sum by less
// than 2^-18 of it, and sqrt(1 + 2^-18) is within the bounds' own slack)
__device__ __forceinline__ int fx_quantum(int ref, float s)
{
    const int es = (__float_as_int(s) >> 23) - 127;  // s < 2^(es + 1)
    return max(ref - 1023 + ((es + 2) >> 1) - 60, -1020);
}

// x on the quantum 2^q, rounded to nearest: s0 = 1084 + q.  The significand, left-justified below the sign bit, is
// shifted to half the quantum, given its sign, and rounded up by one half.
__device__ __forceinline__ long long fx_from(double x, int s0)
{
    const int hi = __double2hiint(x);
    const unsigned lo = (unsigned)__double2loint(x);
    const int s = min(s0 - ((hi >> 20) & 0x7ff), 63);  // 0 and denormals: to 0
    const unsigned mh = (__funnelshift_l(lo, (unsigned)hi, 10) & 0x3fffffffu) | 0x40000000u;
    const unsigned long long m = ((unsigned long long)mh << 32) | (unsigned long long)(lo << 10);
    const long long sg = (long long)(hi >> 31);
    return ((((long long)(m >> s)) ^ sg) - sg + 1) >> 1;
}

// v 2^q in FP64 by integer operations, |q| <= 900, rounded to nearest (halves away
// from zero)
__device__ __forceinline__ double fx_double(long long v, int q)
{
    const int sg = (int)(v >> 63);
    const unsigned long long m = (unsigned long long)((v ^ (long long)sg) - (long long)sg);
    const unsigned mh = (unsigned)(m >> 32), ml = (unsigned)m;
    const bool small = mh == 0;
    const int z = __clz((int)(small ? ml : mh));
    const unsigned nh = small ? ml << (z & 31) : __funnelshift_l(ml, mh, z);
    const unsigned nl = small ? 0u : ml << z;
    // the top bit, at 63, becomes the significand's implicit one
    const unsigned lo = __funnelshift_r(nl, nh, 11), r = lo + ((nl >> 10) & 1u);
    const unsigned e = (unsigned)((1023 + 62 + q - z - (small ? 32 : 0)) << 20) | ((unsigned)sg & 0x80000000u);
    const unsigned hi = (nh >> 11) + e + (r < lo ? 1u : 0u);
    return m == 0 ? 0.0 : __hiloint2double((int)hi, (int)r);
}
// ---- the nonlinear flow of real time on fixed-point values ----
//
// psi <- exp(-i theta) psi with theta = (V + beta |psi|^2) dt in turns, as a
// 64-bit fraction whose overflow is the reduction modulo one turn: |psi|^2
// from the integers, times beta dt / 2 pi (63 bits and an exponent), plus V dt
// / 2 pi, the exact product of V and dt / 2 pi (fx_vturn).  The nearest 128th
// of a turn comes from a table of exp(2 pi i k / 128), the rest (at most
// pi / 128) from the Taylor series, to 2^-58; one complex product joins the
// two and one applies the result.  About 48 multiply-adds, 4 more with a
// potential, where FP64 needs some 70 operations at a 14th of their rate (the
// epilogue of the 256^3 z pass 0.20 ms, 0.22 with a potential, where FP64 took
// 0.6 more).
constexpr int FX_NL_TAB = 128;
// The line-independent part of a call: beta dt / (2 pi) = (gh 2^32 + gl) 2^ge,
// dt / (2 pi) = d 2^de.
struct FxNlArgs {
    int gh, gl, ge, de;
    long long d;
    const int4 *tab;         // exp(2 pi i k / 128), k < 128, as table constants
    const long long *tab2;   // 2^(k / 128) 2^61, k < 128 (imaginary time)
};
// series of cos and sin of (pi / 128) u, |u| <= 1, in z = u^2: Taylor
// coefficients times 4 per power of z (a product by z comes out as z / 4)
// and 2^64; the last two of the sine 2^60
constexpr long long FX_C2 = 0x4ef4f326f91779LL, FX_C4 = 0x40f07c206d7LL;
constexpr int FX_C6 = 0x155d3c7e;
constexpr long long FX_S1 = 0x6487ed5110b4612LL, FX_S3 = 0xa55de7312df3LL;
constexpr int FX_S5 = 0x519af19e, FX_S7 = 0x132d3;

// exp(2 pi i th / 2^64), 2^62 times its components
__device__ __forceinline__ fxc fx_expi(long long th, const int4 *tab)
{
    const unsigned k = (unsigned)((unsigned long long)(th + (1LL << 56)) >> 57);
    const long long u = (long long)((unsigned long long)th << 6) - ((long long)((unsigned long long)k << 63));
    // u = 2^62 times the remainder over a 256th of a turn: th - k 2^57, times 64
    int uh, ul;
    fx_split(u, uh, ul);
    const long long z = (fx_madw(uh, uh, 0) << 2) + (fx_madw(ul, uh, 1LL << 28) >> 29);  // 2^62 u^2
    const int zh = (int)(z >> 32);
    const long long c4 = FX_C4 - (long long)__mulhi(zh, FX_C6);
    int ch, cl;
    fx_split(c4, ch, cl);
    const long long c2 = FX_C2 - fx_rmul(z, ch, cl);
    fx_split(c2, ch, cl);
    const long long co = (1LL << 62) - (fx_rmul(z, ch, cl) >> 2);
    const int s5 = FX_S5 - __mulhi(zh, FX_S7);
    const long long s3 = FX_S3 - ((long long)__mulhi(zh, s5) << 4);
    fx_split(s3, ch, cl);
    const long long s1 = FX_S1 - fx_rmul(z, ch, cl);
    fx_split(s1, ch, cl);
    const long long si = fx_rmul(u, ch, cl);
    // exp(i theta) in units of 2^-62
    fxc f = fx_cmul(fxc{co, si}, tab[k & (FX_NL_TAB - 1)]);
    f.x <<= 2;
    f.y <<= 2;
    return f;
}

// exp(-2 pi i th / 2^64) c / 4, c of modulus at most 2^62
__device__ __forceinline__ fxc fx_rotate(fxc c, long long th, const int4 *tab)
{
    int xh, xl, yh, yl;
    fx_split(c.x, xh, xl);
    fx_split(c.y, yh, yl);
    const fxc f = fx_expi(th, tab);
    // c conj(f) / 4 (run-time constants are negated whole, not by halves: a
    // low half of -2^31 has no negative)
    int fh, fl, gh, gl, nh, nl;
    fx_split(f.x, fh, fl);
    fx_split(f.y, gh, gl);
    fx_split(-f.y, nh, nl);
    fxc o;
    o.x = fx_fold(fx_madw(xh, fh, fx_madw(yh, gh, FX_S0)),
                  fx_madw(xl, fh, fx_madw(yl, gh, fx_madw(xh, fl, fx_madw(yh, gl, FX_X0)))));
    o.y = fx_fold(fx_madw(yh, fh, fx_madw(xh, nh, FX_S0)),
                  fx_madw(yl, fh, fx_madw(xl, nh, fx_madw(yh, fl, fx_madw(xh, nl, FX_X0)))));
    return o;
}

// One cell: c of modulus at most 2^62; theta = |c|^2 2^-62 (gh 2^32 + gl) 2^-64
// shifted left by lsh and right by rsh, plus vt.  Returns exp(-i theta) c / 4.
__device__ __forceinline__ fxc fx_nl_real(fxc c, long long vt, int gh, int gl, int lsh, int rsh, const int4 *tab)
{
    int xh, xl, yh, yl;
    fx_split(c.x, xh, xl);
    fx_split(c.y, yh, yl);
    // the squares of the low halves, left out, are 2/3 of a unit on average
    constexpr long long kX = (1LL << 28) + (2LL << 29) / 3;
    const long long S = fx_madw(xh, xh, fx_madw(yh, yh, 0));
    const long long X = fx_madw(xl, xh, fx_madw(yl, yh, kX));
    const long long rho = (S << 2) + (X >> 29);
    return fx_rotate(c, ((fx_rmul(rho, gh, gl) << lsh) >> rsh) + vt, tab);
}

// theta / (2 pi) of rho = |psi|^2 >= 0 in FP64 (without the potential's part), 2^64
// to a turn: the significand of rho times beta dt / (2 pi), at the place of the
// exponents
__device__ __forceinline__ long long fx_theta(double rho, int gh, int gl, int ge)
{
    const int hi = __double2hiint(rho);
    const unsigned lo = (unsigned)__double2loint(rho);
    const int e = (hi >> 20) & 0x7ff;
    const unsigned mh = (__funnelshift_l(lo, (unsigned)hi, 10) & 0x3fffffffu) | 0x40000000u;
    const long long m = (long long)(((unsigned long long)mh << 32) | (unsigned long long)(lo << 10));
    const int sh = e ? e + ge - 957 : -63;  // 0 and denormals: 0
    return (fx_rmul(m, gh, gl) << min(max(sh, 0), 63)) >> min(max(-sh, 0), 63);
}

// 64-bit shifts whose amounts beyond 63 (negative ones, as unsigned, among them)
// give 0
__device__ __forceinline__ unsigned long long fx_shr(unsigned long long v, int s)
{
    asm("shr.b64 %0, %0, %1;" : "+l"(v) : "r"(s));
    return v;
}
__device__ __forceinline__ unsigned long long fx_shl(unsigned long long v, int s)
{
    asm("shl.b64 %0, %0, %1;" : "+l"(v) : "r"(s));
    return v;
}
__device__ __forceinline__ unsigned long long fx_madw_u(unsigned a, unsigned b, unsigned long long c)
{
    unsigned long long r;
    asm("mad.wide.u32 %0, %1, %2, %3;" : "=l"(r) : "r"(a), "r"(b), "l"(c));
    return r;
}
// V d 2^de in 2^64ths of a turn (modulo one): the 53-bit significand of V times
// |d| of at most 62 bits, exact, at the place of the exponents (denormals count
// as 0).  *top keeps the largest exponent seen: 0x7ff for NaN and infinity, whose
// angle means nothing.  A table of the products instead (one per time step, 8 bytes
// per cell each) took memory that a field may not leave and was filled on the
// first step after each change of V or dt.  Last pass with the flow, table -> here:
// 64^2 4.5 -> 4.8 us, 128^2 5.5 -> 5.5, 256^2 6.0 -> 6.5, 128^3 63 -> 67, 256^3 496
// -> 510, 240^3 765 -> 820; a new V, one step and the mass at 128^3 500 -> 404 us.
__device__ __forceinline__ long long fx_vturn(double V, long long d, int de, int *top)
{
    const int hi = __double2hiint(V);
    const unsigned lo = (unsigned)__double2loint(V);
    const int e = (hi >> 20) & 0x7ff;
    *top = max(*top, e);
    const unsigned mh = (__funnelshift_l(lo, (unsigned)hi, 10) & 0x3fffffffu) | 0x40000000u, ml = lo << 10;
    const unsigned long long md = (unsigned long long)(d < 0 ? -d : d);
    const unsigned dh = (unsigned)(md >> 32), dl = (unsigned)md;
    const unsigned long long p0 = fx_madw_u(ml, dl, 0);
    const unsigned long long p1 = fx_madw_u(mh, dl, fx_madw_u(ml, dh, p0 >> 32));
    const unsigned long long p2 = fx_madw_u(mh, dh, p1 >> 32);  // the product over 2^64
    const int sh = e ? e + de - 957 : -64;
    unsigned long long t = fx_shr(p2, -sh);
    // an eighth of a turn and above: the product's lower half as well (a branch of
    // the warp, which the compiler does not turn into selections)
    if (__any_sync(__activemask(), sh > 0) && sh > 0) {
        const unsigned long long pl = (p1 << 32) | (unsigned)p0;
        t = fx_shl(p2, sh) | fx_shr(pl, 64 - sh) | fx_shl(pl, sh - 64);
    }
    const long long sg = (long long)((hi >> 31) ^ (int)(d >> 63));
    return ((long long)t ^ sg) - sg;
}

// ---- 2^-x for FP64 x on the integer pipes (the flow of imaginary time) ----
//
// -x as a 52-bit fraction below an 11-bit integer; the nearest 128th from a
// table, the rest r (at most 1/256) from the series of 2^r to 2^-60, the integer
// as the exponent: an FP64 value off by its last rounding and the 2^-53 of x's,
// and 0 below 2^-1022 (a pass has no quantum for subnormal values).
// 17 multiply-adds, where FP64 exp is some 20 operations at a 14th of their
// rate (128^3 imaginary-time x pass 151 -> 92 us).
constexpr long long FX_E1 = 0x2c5c85fdf473de7LL, FX_E2 = 0x3d7f7bff058b2LL, FX_E3 = 0x38d611ae094LL, FX_E4 = 0x276556df7LL;
constexpr int FX_E5 = 0x15d87fe, FX_E6 = 0xa185;
__device__ __forceinline__ double fx_exp2neg(double x, const long long *tab2)
{
    const int hi = __double2hiint(x);
    const unsigned lo = (unsigned)__double2loint(x);
    const int ex = (hi >> 20) & 0x7ff;
    const unsigned mh = (__funnelshift_l(lo, (unsigned)hi, 10) & 0x3fffffffu) | 0x40000000u;
    const unsigned long long m = ((unsigned long long)mh << 32) | (unsigned long long)(lo << 10);
    // round(-x 2^52): |x| below 2^10 (beyond: 0, infinity or NaN, below)
    const long long sg = ~(long long)(hi >> 31);
    const long long E = ((((long long)(m >> (min(max(1032 - ex, 0), 63)))) ^ sg) - sg + 1) >> 1;
    const int k7 = (int)((E + (1LL << 44)) >> 45);  // nearest 128th
    const long long u = (E - ((long long)k7 << 45)) << 18;  // 2^62 times the remainder over 1/256
    const int uh = (int)(u >> 32);
    const long long t4 = FX_E4 + (long long)__mulhi(uh, FX_E5 + __mulhi(uh, FX_E6));
    int ch, cl;
    fx_split(t4, ch, cl);
    const long long t3 = FX_E3 + fx_rmul(u, ch, cl);
    fx_split(t3, ch, cl);
    const long long t2 = FX_E2 + fx_rmul(u, ch, cl);
    fx_split(t2, ch, cl);
    const long long t1 = FX_E1 + fx_rmul(u, ch, cl);
    fx_split(t1, ch, cl);
    const long long p = fx_rmul(u, ch, cl);  // 2^64 (2^r - 1)
    fx_split(p, ch, cl);
    const long long T = tab2[k7 & 127];
    const unsigned long long v = (unsigned long long)(T + fx_rmul(T, ch, cl));  // top bit 60 or 61
    const int z = 2 + (int)((v >> 61) ^ 1u);  // leading zeros
    const int e = 1024 - z + (k7 >> 7);  // the biased exponent less one: the top bit, below, adds it
    const unsigned long long n = v << z;
    const unsigned long long bits = ((unsigned long long)(unsigned)e << 52) + (n >> 11) + ((n >> 10) & 1u);
    double r = e < 0 ? 0.0 : __longlong_as_double((long long)bits);
    if (ex > 1032) r = hi < 0 ? __longlong_as_double(0x7ff0000000000000LL) : 0.0;
    return x != x ? x : r;
}

// Leaving fixed point: an integer v times 2^q as the FP64 nearest to it, in two
// ways.  fp: the halves of v are placed in the significands of 2^84 2^q and 2^52
// 2^q, so two FP64 additions (the first exact) give the value.  integer: the
// magnitude, normalised by its leading zeros and rounded at bit 11, under the
// exponent.  Additions alone keep the narrow FP64 pipe busy for half of a 256^3
// pass and are the longest part of one warp's work on a small field; integers
// alone are some 40 instructions per cell.  All additions / half / a quarter /
// none, us per pass: 256^3 x 306 / 292 / 306 / 325, 128^3 43.5 / 38.6 / 39.1 /
// 40.0, 64^3 8.4 / 7.2 / 6.8 / 6.7: half of them for lines of 256, else a quarter.
// q outside the range that the exponents leave is applied as a second factor.
struct FxOut {
    int qc;
    double k, f;
    bool scaled, bad;
    __device__ __forceinline__ FxOut(int q, bool bad_, double scale, bool with_scale) : bad(bad_)
    {
        qc = min(max(q, -900), 900);
        const int d = min(max(q - qc, -1000), 1000);
        k = __hiloint2double(0x45300000 + qc * (1 << 20), (int)0x80100000);
        scaled = with_scale || d != 0;
        f = __hiloint2double((1023 + d) << 20, 0) * scale;
    }
    __device__ __forceinline__ double fp(long long v) const
    {
        const double h = __hiloint2double(0x45300000 + qc * (1 << 20), (int)((unsigned)(v >> 32) ^ 0x80000000u));
        const double l = __hiloint2double(0x43300000 + qc * (1 << 20), (int)v);
        return (h - k) + l;
    }
    // with_fp: the real part by additions
    __device__ __forceinline__ double2 operator()(fxc c, bool with_fp) const
    {
        double2 o = make_double2(with_fp ? fp(c.x) : fx_double(c.x, qc), fx_double(c.y, qc));
        if (bad) o.x = o.y = __longlong_as_double(0x7ff8000000000000LL);
        if (scaled) {
            o.x *= f;
            o.y *= f;
        }
        return o;
    }
};

}  // namespace gpss

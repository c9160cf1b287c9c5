// gpss_internal.h -- declarations shared by the translation units of libgpss.
#pragma once
#include <cuda_runtime.h>
#include <algorithm>
#include <climits>
#include <cmath>
#include <cstdint>
#include <cstring>
#include <string>
#include <vector>
#include "pass_kernel.cuh"
#include "pass_generic.cuh"
#include "pass_generic32.cuh"

namespace gpss {

// ---- host-side tables shared by the context, the batch and the no-alloc path

// (cos, sin) of 2 pi k / n in long double, reduced to the first octant so
// that the symmetric values are exact.
inline void unit_root(int64_t k, int64_t n, long double *cs, long double *sn)
{
    const long double half_pi = 1.570796326794896619231321691639751442L;
    k %= n;
    if (k < 0) k += n;
    const int64_t q = (4 * k) / n, r4 = 4 * k - q * n;
    long double cc, ss;
    if (2 * r4 <= n) {
        const long double a = half_pi * (long double)r4 / (long double)n;
        cc = cosl(a); ss = sinl(a);
    } else {
        const long double a = half_pi * (long double)(n - r4) / (long double)n;
        cc = sinl(a); ss = cosl(a);
    }
    switch (q) {
    case 0: *cs = cc; *sn = ss; break;
    case 1: *cs = -ss; *sn = cc; break;
    case 2: *cs = -cc; *sn = -ss; break;
    default: *cs = ss; *sn = -cc; break;
    }
}

// The twiddles w_n^{r k1} = exp(-2 pi i r k1 / n) of a line of n cells in the
// pass kernel's two orders: row 0 at m = k1*N2 + r (stage A), row 1 at
// m = r*N1 + k1 (stage B), N1 of the passes of a precision (split_n1), N2 = n / N1;
// FP64: then row 2, w_n^k in natural order (the radix-4 stages of small fields).
inline void twiddle_rows(int64_t n, int precision_bytes, std::vector<long double> &re, std::vector<long double> &im)
{
    const int64_t N1 = split_n1(n, precision_bytes), N2 = n / N1;
    const int64_t rows = precision_bytes == 8 ? 3 : 2;
    re.assign((size_t)(rows * n), 0.0L);
    im.assign((size_t)(rows * n), 0.0L);
    std::vector<long double> cs((size_t)n), sn((size_t)n);
    for (int64_t k = 0; k < n; k++) unit_root(k, n, &cs[(size_t)k], &sn[(size_t)k]);
    auto put = [&](int64_t i, int64_t k) {
        re[(size_t)i] = cs[(size_t)k];
        im[(size_t)i] = -sn[(size_t)k];
    };
    for (int64_t k1 = 0; k1 < N1; k1++)
        for (int64_t r = 0; r < N2; r++) {
            put(k1 * N2 + r, r * k1);
            put(n + r * N1 + k1, r * k1);
        }
    if (rows == 3)
        for (int64_t k = 0; k < n; k++) put(2 * n + k, k);
}

// Complex values in rows of n (long double) as double-word pairs of the field
// precision: per row hi[n] then lo[n], hi + lo = value.
template <typename T>
std::vector<vec2<T>> dw_split(const std::vector<long double> &re, const std::vector<long double> &im, int64_t n)
{
    const int64_t rows = (int64_t)re.size() / n;
    std::vector<vec2<T>> out((size_t)(2 * n * rows));
    for (int64_t r = 0; r < rows; r++)
        for (int64_t k = 0; k < n; k++) {
            const size_t i = (size_t)(r * n + k);
            const T hr = (T)re[i], hi = (T)im[i];
            vec2<T> h, l;
            h.x = hr;
            h.y = hi;
            l.x = (T)(re[i] - (long double)hr);
            l.y = (T)(im[i] - (long double)hi);
            out[(size_t)(r * 2 * n + k)] = h;
            out[(size_t)(r * 2 * n + n + k)] = l;
        }
    return out;
}

// One component of a fixed-point table constant (fft_fix.cuh): 2^62 v for
// |v| <= 1 as halves h 2^32 + l, both signed.  l = -2^31 has no negative, so
// it moves by one unit of 2^-62.
inline void fx_halves(long double v, int &l, int &h)
{
    int64_t c = (int64_t)llroundl(v * 4611686018427387904.0L);
    if ((uint32_t)c == 0x80000000u) c += c < 0 ? -1 : 1;
    l = (int)(uint32_t)c;
    h = (int)((c - (int64_t)l) >> 32);
}
inline int4 fx_const(long double re, long double im)
{
    int4 c;
    fx_halves(re, c.x, c.y);
    fx_halves(im, c.z, c.w);
    return c;
}
// Constants of modulus at most 1 in fixed point.
inline std::vector<int4> fx_table(const std::vector<long double> &re, const std::vector<long double> &im)
{
    std::vector<int4> t(re.size());
    for (size_t i = 0; i < t.size(); i++) t[i] = fx_const(re[i], im[i]);
    return t;
}
// A fixed-point table of phases or decaying factors: a leading entry with the exponent e,
// then the values divided by 2^e, the smallest power of two at or above their
// largest modulus.  A non-finite value makes every result of a pass with the
// table NaN or infinite in FP64; here its exponent overflows the pass's result.
inline std::vector<int4> fx_phase_table(const std::vector<long double> &re, const std::vector<long double> &im)
{
    long double m = 0.0L;
    bool finite = true;
    for (size_t i = 0; i < re.size(); i++) {
        const long double a = hypotl(re[i], im[i]);
        finite = finite && std::isfinite((double)a);
        if (a > m) m = a;
    }
    int e = 0;
    if (finite && m > 0.0L) {
        const long double f = frexpl(m, &e);  // m = f 2^e, f in [1/2, 1)
        // unit moduli are 1 up to the rounding of the long double values
        if (f <= 0.5L * (1.0L + 1e-17L)) e--;
    }
    std::vector<int4> t(re.size() + 1);
    t[0] = make_int4(finite ? e : 1 << 20, 0, 0, 0);
    for (size_t i = 0; i < re.size(); i++)
        t[i + 1] = finite ? fx_const(ldexpl(re[i], -e), ldexpl(im[i], -e)) : fx_const(1.0L, 0.0L);
    return t;
}

// A multiplier table (fft_fix.cuh): a leading entry with the exponent e of the
// largest value, then per value a 62-bit significand as halves and its exponent
// less e.  Non-finite values as above.
inline std::vector<int4> fx_mult_table(const std::vector<long double> &v)
{
    std::vector<int4> t(v.size() + 1, make_int4(0, 1 << 30, 0, 0));
    int top = INT_MIN;
    for (size_t i = 0; i < v.size(); i++) {
        if (!std::isfinite((double)v[i])) {
            std::fill(t.begin(), t.end(), make_int4(0, 1 << 30, 0, 0));
            t[0] = make_int4(1 << 20, 0, 0, 0);
            return t;
        }
        int e = 0;
        fx_halves(frexpl(v[i], &e), t[i + 1].x, t[i + 1].y);
        t[i + 1].z = e;
        if (v[i] != 0.0L) top = std::max(top, e);
    }
    t[0] = make_int4(top == INT_MIN ? 0 : top, 0, 0, 0);
    for (size_t i = 0; i < v.size(); i++) t[i + 1].z = v[i] != 0.0L ? t[i + 1].z - t[0].x : 0;
    return t;
}

// exp(i theta) scale as a table constant, theta in FP64 (exact), |scale| <= 1 as
// 2^62 scale: theta in turns from 1/(2 pi) to 128 bits, the nearest 128th of a
// turn from a table, the rest (at most pi/128) from the Taylor series in 68-bit
// fixed point; within 2^-63 of the exact value like the long double functions
// it stands for, which on Arm are software (a rotating frame's tables have a row
// per node: 64 x 48 x 56 first pass 6.8 -> 1.4 ms).  Large arguments (2^40 and
// above) take the long double functions.
inline int4 fx_phase_const(double theta, int64_t scale62)
{
    static const std::vector<int64_t> root = [] {  // exp(2 pi i k / 128) 2^68 as high part (2^62) and 6 bits
        std::vector<int64_t> r;
        for (int k = 0; k < 128; k++) {
            long double v[2];
            unit_root(k, 128, &v[0], &v[1]);
            for (long double x : v) {
                const int64_t hi = (int64_t)floorl(ldexpl(x, 62));
                r.push_back(hi);
                r.push_back((int64_t)llroundl(ldexpl(x - ldexpl((long double)hi, -62), 68)));
            }
        }
        return r;
    }();
    using i128 = __int128;
    using u128 = unsigned __int128;
    auto mul = [](int64_t a, int64_t b, int shift) { return (int64_t)(((i128)a * b) >> shift); };
    i128 re, im;  // 2^68
    int e;
    const double f = std::frexp(std::fabs(theta), &e);
    if (!(f >= 0.5) && theta == 0.0) {
        re = (i128)1 << 68;
        im = 0;
    } else if (e > 40) {
        re = (i128)llroundl(ldexpl(cosl((long double)theta), 62)) << 6;
        im = (i128)llroundl(ldexpl(sinl((long double)theta), 62)) << 6;
    } else {
        const uint64_t m = (uint64_t)std::ldexp(f, 53);  // |theta| = m 2^(e - 53)
        const u128 p0 = (u128)m * 0x7f09d5f47d4d3770ULL, p1 = (u128)m * 0x28be60db9391054aULL + (p0 >> 64);
        // |theta| / (2 pi) 2^128 = (p1 2^64 + low word of p0) 2^(e - 53), modulo 2^128
        const uint64_t w[3] = {(uint64_t)p0, (uint64_t)p1, (uint64_t)(p1 >> 64)};
        const int s = 53 - e;  // 13 and above: a right shift of the 192-bit product
        auto word = [&](int i) { return i < 3 ? w[i] : (uint64_t)0; };
        const int q = s / 64, b = s % 64;
        const uint64_t l = b ? (word(q) >> b) | (word(q + 1) << (64 - b)) : word(q);
        const uint64_t h = b ? (word(q + 1) >> b) | (word(q + 2) << (64 - b)) : word(q + 1);
        u128 turns = ((u128)h << 64) | l;
        if (theta < 0) turns = 0 - turns;
        const int k = (int)((uint64_t)((turns + ((u128)1 << 120)) >> 121) & 127);
        const int64_t u = (int64_t)((i128)(turns - ((u128)k << 121)) >> 58);  // 2^70 turns
        const int64_t X = mul(u, 0x6487ed5110b4611aLL, 62);                               // radians, 2^68
        const int64_t Z = mul(X, X, 68);
        const int64_t one = 1LL << 62;
        int64_t t = one / 5040 - mul(Z, one / 362880, 68);
        t = one / 120 - mul(Z, t, 68);
        t = one / 6 - mul(Z, t, 68);
        const int64_t S = X - mul(X, mul(Z, t, 62), 68);  // sin
        t = one / 720 - mul(Z, one / 40320, 68);
        t = one / 24 - mul(Z, t, 68);
        t = one / 2 - mul(Z, t, 68);
        const int64_t D = mul(Z, t, 62);                  // 1 - cos
        const int64_t *r = &root[(size_t)(4 * k)];
        const int64_t c = r[0], n = r[2];
        re = ((i128)c << 6) + r[1] - (((i128)c * D + (i128)n * S) >> 62);
        im = ((i128)n << 6) + r[3] - (((i128)n * D - (i128)c * S) >> 62);
    }
    auto put = [&](i128 v, int &l, int &h) {  // 2^68 v scale, rounded to 2^62
        const i128 x = scale62 == (1LL << 62) ? v : (v >> 4) * scale62 >> 58;
        int64_t o = (int64_t)((x + 32) >> 6);
        if ((uint32_t)o == 0x80000000u) o += o < 0 ? -1 : 1;
        l = (int)(uint32_t)o;
        h = (int)((o - (int64_t)l) >> 32);
    };
    int4 o;
    put(re, o.x, o.y);
    put(im, o.z, o.w);
    return o;
}

// x / (2 pi) as m 2^e with m of 62 bits and a sign (0: m = 0)
inline void fx_turns(long double x, int64_t &m, int &e)
{
    const long double two_pi = 6.283185307179586476925286766559005768L;
    m = 0;
    e = 0;
    if (x == 0.0L) return;
    const long double f = frexpl(x / two_pi, &e);
    m = (int64_t)llroundl(ldexpl(f, 62));
    e -= 62;
}

// The FP64 generic pass's tables: its roots w_n^k = exp(-2 pi i k / n), k < n, then the spectrum's order: mode
// at each position, position of each mode
inline std::vector<unsigned char> gen_roots_table(const GenPlan &p)
{
    const int n = p.n;
    std::vector<long double> re((size_t)n), im((size_t)n);
    std::vector<int> order((size_t)(2 * n));
    for (int k = 0; k < n; k++) {
        long double cs, sn;
        unit_root(k, n, &cs, &sn);
        re[(size_t)k] = cs;
        im[(size_t)k] = -sn;
        order[(size_t)k] = gen_mode_at(p, k);
        order[(size_t)(n + order[(size_t)k])] = k;
    }
    std::vector<unsigned char> out((size_t)n * 16 + order.size() * sizeof(int));
    std::memcpy(out.data(), fx_table(re, im).data(), (size_t)n * 16);
    std::memcpy(out.data() + (size_t)n * 16, order.data(), order.size() * sizeof(int));
    return out;
}

// pass launchers (pass_f32.cu / pass_f64.cu)
cudaError_t launch_pass_f32(int mode, bool xl, int n, const PassArgs<float> &a, int blocks,
                            cudaStream_t s);
cudaError_t launch_pass_f64(int mode, bool xl, int n, const PassArgs<double> &a, int blocks,
                            cudaStream_t s);
// lines of a CTA in the passes of a field of `total` cells
int pass_lines_per_cta_f32(int n, bool xl, int64_t total);
int pass_lines_per_cta_f64(int n, bool xl, int64_t total);
// pipelined fused pass (FP32; n in {64, 128, 256}; tiles of 4096/n lines)
cudaError_t launch_pipe_f32(bool xl, int n, const PassArgs<float> &a, int ntiles, cudaStream_t s);

// the generic-length pass (pass_gen.cu)
cudaError_t launch_gen_f32(int mode, const PassArgs<float> &a, const Gen32Plan &p, cudaStream_t s);
cudaError_t launch_gen_f64(int mode, const PassArgs<double> &a, const GenPlan &p, cudaStream_t s);

template <typename T> struct PassLauncher;
template <> struct PassLauncher<float> {
    static cudaError_t launch(int mode, bool xl, int n, const PassArgs<float> &a, int blocks,
                              cudaStream_t s) { return launch_pass_f32(mode, xl, n, a, blocks, s); }
    static int lines(int n, bool xl, int64_t total) { return pass_lines_per_cta_f32(n, xl, total); }
    static cudaError_t pipe(bool xl, int n, const PassArgs<float> &a, int ntiles, cudaStream_t s)
    {
        return launch_pipe_f32(xl, n, a, ntiles, s);
    }
    static cudaError_t gen(int mode, const PassArgs<float> &a, const GenPlan &, const Gen32Plan &p, cudaStream_t s)
    {
        return launch_gen_f32(mode, a, p, s);
    }
};
template <> struct PassLauncher<double> {
    static cudaError_t launch(int mode, bool xl, int n, const PassArgs<double> &a, int blocks,
                              cudaStream_t s) { return launch_pass_f64(mode, xl, n, a, blocks, s); }
    static int lines(int n, bool xl, int64_t total) { return pass_lines_per_cta_f64(n, xl, total); }
    static cudaError_t pipe(bool, int, const PassArgs<double> &, int, cudaStream_t) { return cudaErrorInvalidValue; }
    static cudaError_t gen(int mode, const PassArgs<double> &a, const GenPlan &p, const Gen32Plan &, cudaStream_t s)
    {
        return launch_gen_f64(mode, a, p, s);
    }
};

// Is a line of n cells taken by the register kernel (a power of two up to
// 256)?  Otherwise the generic pass runs it.
inline bool reg_line(int64_t n) { return n >= 2 && n <= 256 && (n & (n - 1)) == 0; }

// pointwise kernels (pointwise.cu)
cudaError_t launch_f64_to_f32(const double *in, float *out, int64_t count, cudaStream_t s);
cudaError_t launch_f32_to_f64(const float *in, double *out, int64_t count, cudaStream_t s);
template <typename T>
cudaError_t launch_mul_phase(vec2<T> *data, const vec2<T> *phase, int64_t prow, int axis,
                             const int64_t *n, int64_t total, cudaStream_t s);
template <typename T>
cudaError_t launch_nl(vec2<T> *psi, const T *V, double beta, double dt, int imag, int64_t total,
                      cudaStream_t s);
template <typename T>
cudaError_t launch_scale(vec2<T> *psi, const double *scale, int64_t total, cudaStream_t s);
// implicit schemes (implicit.cu); the scheme numbers are the GPSS_IMPLICIT_* of gpss.h
enum {
    IM_SCHEME_BE = 0, IM_SCHEME_BE_NOPRE = 1, IM_SCHEME_CN = 2, IM_SCHEME_CN_QN = 3, IM_SCHEME_CN_T = 4,
    IM_SCHEME_CN_QN_T = 5
};
template <typename T>
cudaError_t im_prep_be(const vec2<T> *phi, const T *V, double beta, double dt, int scheme, vec2<T> *M, T *Anl,
                       vec2<T> *b, int64_t total, cudaStream_t s);
template <typename T>
cudaError_t im_prep_cn(const vec2<T> *phi, const vec2<T> *phi1, const T *V, double beta, double dt, int scheme,
                       vec2<T> *psim, T *Anl, vec2<T> *Anl2, vec2<T> *M, int64_t total, cudaStream_t s);
template <typename T>
cudaError_t im_rhs_cn(const vec2<T> *phi, const vec2<T> *phi1, const vec2<T> *psim, const vec2<T> *lap, const T *V,
                      double beta, double dt, int tsch, vec2<T> *b, int64_t total, cudaStream_t s);
template <typename T>
cudaError_t im_axmy(vec2<T> *out, const vec2<T> *x, double alpha, const vec2<T> *y, int64_t total, cudaStream_t s);

// The scalars of one BiCGStab solve (krylov.jl:1-67), kept on the device so
// that iterations run without a host round trip: the dot products are
// finished on the device, one thread forms alpha, omega, beta and the
// stopping test from them in FP64 (the same operations, in the same order, as
// the reference), and the vector updates read them from here.  Once `done`
// is set (converged, out of iterations, or a non-finite residual) every later
// update of the same solve is a no-op, so the host may issue iterations in
// chunks and read this back once per chunk.
struct KrylovDev {
    double normb, rr2, alpha, omega, beta;
    int done, niter, nonfinite, it;
};
// what the dot products of a kernel are for (see implicit.cu)
enum { KRY_NONE = 0, KRY_INIT = 1, KRY_ALPHA = 2, KRY_OMEGA = 3, KRY_CHECK = 4 };
constexpr int KRY_MAX_CTAS = 152 * 8;  // of a kernel with dot products
struct KryScratch {
    double *partials;        // [2 * KRY_MAX_CTAS]
    double *dots;            // the last two sums
    unsigned int *counter;   // 0 between launches
    KrylovDev *K;
};
template <typename T>
cudaError_t im_op(const vec2<T> *x, const vec2<T> *lap, int scheme, double dt, const vec2<T> *M, const T *Anl,
                  const vec2<T> *Anl2, const vec2<T> *b, int precond, vec2<T> *out, int64_t total, const vec2<T> *r,
                  const vec2<T> *r2, const KryScratch &k, int what, cudaStream_t s);
template <typename T>
cudaError_t im_norm2(const vec2<T> *a, int64_t total, const KryScratch &k, int what, cudaStream_t s);
// s = r - alpha Ap;  phi = (phi + alpha p) + omega s, r = s - omega As;  p = r + beta (p - omega Ap)
template <typename T>
cudaError_t im_axmy_k(vec2<T> *out, const vec2<T> *x, const vec2<T> *y, const KrylovDev *K, int64_t total,
                      cudaStream_t s);
template <typename T>
cudaError_t im_update_k(vec2<T> *phi, const vec2<T> *p, const vec2<T> *sv, const vec2<T> *As, vec2<T> *r,
                        const vec2<T> *r2, const KryScratch &k, double tol, int nkrylov, int64_t total,
                        cudaStream_t s);
template <typename T>
cudaError_t im_pdir_k(vec2<T> *p, const vec2<T> *r, const vec2<T> *Ap, const KrylovDev *K, int64_t total,
                      cudaStream_t s);
template <typename T>
cudaError_t im_mfield(vec2<T> *out, const vec2<T> *M, const vec2<T> *x, int64_t total, cudaStream_t s);

// explicit Runge-Kutta helpers (pointwise.cu)
template <typename T>
cudaError_t launch_nl_term(const vec2<T> *q, const T *V, double beta, vec2<T> *t, int64_t total, cudaStream_t s);
template <typename T>
cudaError_t launch_rk_combine(const vec2<T> *k, const vec2<T> *t, const vec2<T> *psi0, vec2<T> *acc, vec2<T> *out,
                              int acc_mode, double acc_w, double cf, int from_acc, int64_t total, cudaStream_t s);

// discrete adjoint (adjoint.cu)
// z[0..1] = dV * sum conj(a) b; partials needs 2 * 152 * 8 doubles
template <typename T>
cudaError_t launch_overlap(const vec2<T> *a, const vec2<T> *b, int64_t total, double *partials, double dV,
                           double *z, cudaStream_t s);
template <typename T>
cudaError_t launch_seed(vec2<T> *g, const vec2<T> *target, const double *z, double dV, int64_t total,
                        cudaStream_t s);
template <typename T>
cudaError_t launch_nl_adjoint(vec2<T> *g, const vec2<T> *psi_in, const T *V, double *dLdV, double beta, double dt,
                              int64_t total, cudaStream_t s);
}  // namespace gpss

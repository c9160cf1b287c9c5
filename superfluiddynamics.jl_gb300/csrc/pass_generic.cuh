// pass_generic.cuh -- the directional pass of FP64 fields for line lengths that
// the register kernel (pass_kernel.cuh, powers of two up to 256) does not take:
// any n up to GEN_MAX_N whose prime factors are at most 31 (FP32 fields:
// pass_generic32.cuh).  The reference plans every
// length with FFTW (plan_fft, src/Discretization/Plans.jl:846-847); its own
// tests run grids such as 48^3, 48x36 and 64x48x56.
//
// A CTA of 128 threads holds a tile of W lines in shared memory and transforms
// it in place: decimation in frequency forward,
//     stage s of radix R with blocks of L = R M cells: for j < M
//     v[q] = x[p + q M], p = block L + j;  DFT_R(v);  x[p + q M] = v[q] w_L^{j q}
// and its mirror (decimation in time) backward.  A butterfly writes the slots
// it has read, so a stage needs one barrier and one buffer; the spectrum comes
// out in digit-reversed order, which the phase table follows, and the last
// forward and first backward stage (M = 1) are one trip through registers
// with the phase between them.  Forward and backward share their code: the
// backward transform is the forward one of the values with real and imaginary
// part exchanged.
//
// Every thread works on one line of the tile throughout (a group of
// 128 / W threads per line), so its addresses need no division but the one by
// M (a multiplication by a host-made reciprocal).  Radices 2..16 (2 3 4 5 7 8 16
// and, by the prime factor algorithm, 6 10 12 14 15) are straight-line code,
// primes 11..31 a loop.  Lines are transformed in 64-bit fixed point
// (fft_fix.cuh).  64 x 48 x 56 with rotation, 10 steps, 4650 -> 1000 us against
// a Stockham form of this pass with run-time divisions, table look-ups in
// global memory and FP64 arithmetic.
//
// Modes and features are those of pass_kernel<MODE_FUSED/FWD/INV/DIAG> that the
// split steps, energies, explicit RK and implicit schemes use, the merged
// imaginary-time step's prologue and inner product among them.  The adjoint,
// stacked planes, the pipelined and the compensated passes take power-of-two
// lines only.
#pragma once
#include <cmath>
#include "pass_kernel.cuh"

namespace gpss {

constexpr int GEN_MAX_N = 1024;
constexpr int GEN_MAX_STAGES = 10;
constexpr int GEN_THREADS = 128;
constexpr int GEN_SMEM_MAX = 112 * 1024;  // 1024-cell FP64 columns: 64 KB of tile, 32 KB of tables

struct GenPlan {
    int n;
    int lw;                       // log2 of the lines per tile
    int nst;                      // stages
    int radix[GEN_MAX_STAGES];
    int m[GEN_MAX_STAGES];        // M of each stage: cells between a butterfly's values
    unsigned magic[GEN_MAX_STAGES];  // ceil(2^32 / M): b / M = umulhi(b, magic) for M > 1
    // fixed point (FP64): every product by a table constant divides by 4; left
    // shifts that the next stage has room for, after the products of the
    // forward stages, the phase, and the backward stages (a pass that starts
    // with the spectrum has its own); and the resulting exponents
    int kf[GEN_MAX_STAGES], kp, kb[GEN_MAX_STAGES], ki[GEN_MAX_STAGES];
    int bits_f, bits_i;           // the line's 2-norm takes this many bits
    int bits_p;                   // and may take this many after the phase
    int ef, et, ei;               // exponent of the spectrum, the result, the inverse alone
    int lines() const { return 1 << lw; }
};

inline bool gen_radix_is_loop(int r) { return r > 16 || r == 11 || r == 13; }

// The stages of n with radices up to `cap` (and prime ones above it): as few as
// possible, then with the smallest largest radix, larger radices first; false
// if n has a prime factor above 31 or is too long.
inline bool gen_plan_radices(int n, GenPlan &p, int cap = 16)
{
    p.n = n;
    p.nst = 0;
    if (n < 2 || n > GEN_MAX_N) return false;
    static const int kRadix[] = {2, 3, 4, 5, 6, 7, 8, 10, 11, 12, 13, 14, 15, 16, 17, 19, 23, 29, 31};
    int best[GEN_MAX_STAGES] = {0}, cur[GEN_MAX_STAGES] = {0}, nbest = GEN_MAX_STAGES + 1;
    // depth-first over non-increasing radices
    auto dfs = [&](auto &self, int m, int depth, int top) -> void {
        if (m == 1) {
            if (depth < nbest || (depth == nbest && cur[0] < best[0])) {
                nbest = depth;
                for (int i = 0; i < depth; i++) best[i] = cur[i];
            }
            return;
        }
        if (depth >= GEN_MAX_STAGES || depth + 1 > nbest) return;
        for (int i = (int)(sizeof(kRadix) / sizeof(kRadix[0])) - 1; i >= 0; i--) {
            const int r = kRadix[i];
            const bool prime = r == 2 || r == 3 || r == 5 || r == 7 || r == 11 || r == 13 || r > 16;
            if (r > top || m % r || (r > cap && !prime)) continue;
            cur[depth] = r;
            self(self, m / r, depth + 1, r);
        }
    };
    dfs(dfs, n, 0, n);
    if (nbest > GEN_MAX_STAGES) return false;
    p.nst = nbest;
    int L = n;
    for (int s = 0; s < p.nst; s++) {
        p.radix[s] = best[s];
        L /= best[s];
        p.m[s] = L;
        p.magic[s] = L > 1 ? (unsigned)(((1ULL << 32) + (unsigned)L - 1) / (unsigned)L) : 0u;
    }
    // fixed point: moduli stay at or below 2^62 on entry to a product and
    // inside a butterfly (whose sums of R values gain sqrt(R) in the 2-norm
    // bound; a loop radix multiplies every value and so divides by 4 as well)
    auto gain = [](int r) { return 0.5 * std::log2((double)r) - (gen_radix_is_loop(r) ? 2.0 : 0.0); };
    auto room = [&](int r, double b) {
        const double g = gain(r) > 0.0 ? gain(r) : 0.0;
        const int k = (int)std::floor(62.0 - g - b + 1e-9);
        return k > 0 ? k : 0;
    };
    const int S = p.nst;
    auto run = [&](bool fwd, int *kb, int &bits, int &espec, int &eres) {
        const int first = fwd ? p.radix[0] : p.radix[S - 1];
        bits = room(first, 0.0);
        double b = bits;
        int e = 0;
        auto step = [&](int r) {
            b += gain(r);
            if (gen_radix_is_loop(r)) e += 2;
        };
        auto product = [&](int next) {
            b -= 2.0;
            const int k = room(next, b);
            b += k;
            e += 2 - k;
            return k;
        };
        if (fwd) {
            for (int s = 0; s < S; s++) {
                step(p.radix[s]);
                if (s < S - 1) p.kf[s] = product(p.radix[s + 1]);
            }
            espec = e;
            p.kp = product(p.radix[S - 1]);
            p.bits_p = (int)std::floor(b + 1e-9);
        }
        step(p.radix[S - 1]);
        for (int s = S - 2; s >= 0; s--) {
            kb[s] = product(p.radix[s]);
            step(p.radix[s]);
        }
        eres = e;
    };
    int unused = 0;
    run(true, p.kb, p.bits_f, p.ef, p.et);
    run(false, p.ki, p.bits_i, unused, p.ei);
    return true;
}

// The spectrum's order: mode k of the natural order at each position of a line.
inline int gen_mode_at(const GenPlan &p, int pos)
{
    int k = 0, scale = 1;
    for (int s = 0; s < p.nst; s++) {
        k += scale * ((pos / p.m[s]) % p.radix[s]);
        scale *= p.radix[s];
    }
    return k;
}

// Lines per tile (a power of two): the thread group of a line has 128 / W
// threads, and a stage of radix R gives each ceil(n / R / group) butterflies, so
// a group that does not divide the butterflies leaves lanes idle (240 = 16 x 15
// with 32 threads per line: half of them; 240^3 x pass 966 us, with 16: 700).
// A tile's time goes with the cells of its busiest thread (a stage's barrier
// and addresses count as two, or one where an SM has more than four tiles), c, times the tiles an SM works through -- four at
// a time, which take 1.9 times as long as one alone (measured on fields of one to
// four tiles per SM) -- and the W that makes that product smallest is taken, at
// least 4 adjacent columns for strided lines (32 or 64 contiguous bytes) and
// at most 44 KB of tile (four per SM, with their tables).  The product itself
// goes to *time.  (152 SMs: those of a GB300, whose measurements these are.)
inline int gen_tile_log(int n, const int *radix, int nst, int64_t nlines, bool xl, int most, double *time = nullptr)
{
    const int low = xl ? 0 : 2;
    int best = low;
    double least = 0.0;
    for (int lw = low; lw <= most; lw++) {
        if (lw > low && ((size_t)n << lw) * 16 > 44 * 1024) break;
        const int group = 128 >> lw;
        const double tiles = (double)((nlines + (1 << lw) - 1) >> lw), t = std::ceil(tiles / 152.0);
        double c = 0.0;
        for (int s = 0; s < nst; s++)
            c += (double)((n / radix[s] + group - 1) / group) * radix[s] + (t <= 4.0 ? 2.0 : 1.0);
        const double cost = c * (t <= 4.0 ? 0.7 + 0.3 * t : 1.9 * t / 4.0);
        if (lw == low || cost < least) {
            least = cost;
            best = lw;
        }
    }
    if (time) *time = least;
    return best;
}

// The plan of an FP64 axis of a field: the fewest stages; or, where that leaves
// at most four tiles per SM, of the largest radices 16, 10, 8, 6, 5 and 4 the one
// whose tiles take the least time by the rule above.  A line of a small field
// has more threads than butterflies of a large radix (100 = 10 x 10: 10 of 128
// threads work), so its stages are smaller and more (100 x 100 12.4 / 14.8 -> 10.1
// / 12.4 us); on a full chip an extra stage's products and exchanges cost more
// than idle lanes (240^3 with 8 x 6 x 5 908 us, with 16 x 15 700).
inline bool gen_plan_field(int n, int64_t nlines, bool xl, GenPlan &p)
{
    double least = 0.0;
    bool found = false;
    for (int cap : {16, 10, 8, 6, 5, 4}) {
        GenPlan q;
        if (!gen_plan_radices(n, q, cap)) continue;
        double time;
        q.lw = gen_tile_log(n, q.radix, q.nst, nlines, xl, 6, &time);
        if (!found || time < least) {
            least = time;
            p = q;
            found = true;
        }
        if (((nlines + p.lines() - 1) >> p.lw) > 4 * 152) break;
    }
    return found;
}

// ---- small transforms of fixed-point values ----

// a real constant of the odd butterflies, 2^64 f with c = f, or c = +-(1 - f)
// where |c| >= 1/2
struct GenConst {
    long long f;
    int kind;  // 0: c = f;  +-1: c = +-(1 - f)
};
template <int R, int M> struct GenCos;  // cos(2 pi M / R)
template <int R, int M> struct GenSin;
#define GPSS_GEN_CONST(NAME, R, M, F, KIND)                                     \
    template <> struct NAME<R, M> {                                             \
        static constexpr GenConst v = {F, KIND};                                \
    };
GPSS_GEN_CONST(GenSin, 3, 1, 0x224c28bd3d9aac62LL, 1)
GPSS_GEN_CONST(GenCos, 5, 1, 0x4f1bbcdcbfa53e0bLL, 0)
GPSS_GEN_CONST(GenSin, 5, 1, 0x0c878f65dd58050dLL, 1)
GPSS_GEN_CONST(GenCos, 5, 2, 0x30e44323405ac1f5LL, -1)
GPSS_GEN_CONST(GenSin, 5, 2, 0x6986e7dc552d1092LL, 1)
GPSS_GEN_CONST(GenCos, 7, 1, 0x6062f8eba091749aLL, 1)
GPSS_GEN_CONST(GenSin, 7, 1, 0x37d9e457d10da7a2LL, 1)
GPSS_GEN_CONST(GenCos, 7, 2, -0x38f721c6048b04d3LL, 0)
GPSS_GEN_CONST(GenSin, 7, 2, 0x066b1fd538b4b8e3LL, 1)
GPSS_GEN_CONST(GenCos, 7, 3, 0x195a1ab1a51c796dLL, -1)
GPSS_GEN_CONST(GenSin, 7, 3, 0x6f130135c6af0401LL, 0)
#undef GPSS_GEN_CONST

// a times the constant C::v
template <typename C> __device__ __forceinline__ long long gen_real(long long a)
{
    const long long t = fx_rmul(a, fx_hi(C::v.f), fx_lo(C::v.f));
    if constexpr (C::v.kind == 0) return t;
    else if constexpr (C::v.kind > 0) return a - t;
    else return t - a;
}
template <typename C> __device__ __forceinline__ fxc gen_scale(fxc a) { return fxc{gen_real<C>(a.x), gen_real<C>(a.y)}; }

// forward DFT of an odd prime R (3, 5, 7): X_k, X_{R-k} = A_k -+ i B_k with
// A_k = x0 + sum_m cos(2 pi k m / R) (x_m + x_{R-m}), B_k the same with sin and
// the differences
template <int R, int K, int M>
__device__ __forceinline__ void gen_odd_terms(const fxc *s, const fxc *d, fxc &A, fxc &B)
{
    constexpr int H = (R - 1) / 2, j = (K * M) % R;
    constexpr int f = j <= H ? j : R - j;
    const fxc sn = gen_scale<GenSin<R, f>>(d[M - 1]);
    if constexpr (R == 3) {
        A = csub(A, fxc{(s[0].x + 1) >> 1, (s[0].y + 1) >> 1});  // cos(2 pi / 3) = -1/2
    } else {
        A = cadd(A, gen_scale<GenCos<R, f>>(s[M - 1]));
    }
    if constexpr (M == 1) B = j <= H ? sn : fxc{-sn.x, -sn.y};
    else B = j <= H ? cadd(B, sn) : csub(B, sn);
    if constexpr (M < H) gen_odd_terms<R, K, M + 1>(s, d, A, B);
}
template <int R, int K>
__device__ __forceinline__ void gen_odd_out(fxc *v, const fxc &x0, const fxc *s, const fxc *d)
{
    fxc A = x0, B;
    gen_odd_terms<R, K, 1>(s, d, A, B);
    v[K] = fxc{A.x + B.y, A.y - B.x};
    v[R - K] = fxc{A.x - B.y, A.y + B.x};
    if constexpr (K < (R - 1) / 2) gen_odd_out<R, K + 1>(v, x0, s, d);
}
template <int R> __device__ __forceinline__ void gen_dft(fxc *v);
// Good-Thomas: R = R1 R2 with coprime factors, no twiddles
template <int R1, int R2> __device__ __forceinline__ void gen_dft_pfa(fxc *v)
{
    constexpr int R = R1 * R2;
    fxc t[R];
#pragma unroll
    for (int n2 = 0; n2 < R2; n2++) {
        fxc u[R1];
#pragma unroll
        for (int n1 = 0; n1 < R1; n1++) u[n1] = v[(n1 * R2 + n2 * R1) % R];
        gen_dft<R1>(u);
#pragma unroll
        for (int k1 = 0; k1 < R1; k1++) t[k1 * R2 + n2] = u[k1];
    }
#pragma unroll
    for (int k1 = 0; k1 < R1; k1++) {
        gen_dft<R2>(t + k1 * R2);
#pragma unroll
        for (int k2 = 0; k2 < R2; k2++) {
            // the k with k = k1 mod R1 and k = k2 mod R2
            int k = k1;
            while (k % R2 != k2) k += R1;
            v[k] = t[k1 * R2 + k2];
        }
    }
}
template <int R> __device__ __forceinline__ void gen_dft(fxc *v)
{
    if constexpr (R == 2 || R == 4 || R == 8 || R == 16) dft<R, -1>(v);
    else if constexpr (R == 6) gen_dft_pfa<2, 3>(v);
    else if constexpr (R == 10) gen_dft_pfa<2, 5>(v);
    else if constexpr (R == 12) gen_dft_pfa<4, 3>(v);
    else if constexpr (R == 14) gen_dft_pfa<2, 7>(v);
    else if constexpr (R == 15) gen_dft_pfa<3, 5>(v);
    else {
        constexpr int H = (R - 1) / 2;
        fxc s[H], d[H];
        const fxc x0 = v[0];
#pragma unroll
        for (int m = 1; m <= H; m++) {
            s[m - 1] = cadd(v[m], v[R - m]);
            d[m - 1] = csub(v[m], v[R - m]);
            v[0] = cadd(v[0], s[m - 1]);
        }
        gen_odd_out<R, 1>(v, x0, s, d);
    }
}

__device__ __forceinline__ fxc gen_shift(fxc a, int k) { return fxc{a.x << k, a.y << k}; }

// a fixed-point value on the quantum 2^q in FP64, out of line (energy sums)
static __device__ __noinline__ double2 gen_value(fxc u, int q, bool bad) { return FxOut(q, bad, 1.0, false)(u, false); }

enum { GEN_FWD = 0, GEN_MID = 1, GEN_BWD = 2 };

// One thread's share of a stage on its line.  `at(pos)` is the slot of a
// position, `mid(u, p)` the spectral work on R values at positions p..p + R - 1.
template <int R, typename AT, typename MID>
__device__ __forceinline__ void gen_stage(const GenPlan &p, int s, int kind, int i0, int step, bool fwd, bool bwd,
                                          const int4 *roots, const int *shifts, fxc *data, AT at, MID mid)
{
    const int M = p.m[s], nb = p.n / R;
    const int tws = nb / M;  // n / L
    for (int b = i0; b < nb; b += step) {
        const int g = M > 1 ? (int)__umulhi((unsigned)b, p.magic[s]) : b, j = b - g * M;
        const int p0 = g * R * M + j;
        fxc v[R];
#pragma unroll
        for (int q = 0; q < R; q++) v[q] = data[at(p0 + q * M)];
        const int t = j * tws;
        if (kind == GEN_BWD) {
            const int k = shifts[s];
            v[0] = gen_shift(fx_quarter(v[0]), k);
#pragma unroll
            for (int q = 1; q < R; q++) v[q] = gen_shift(fx_cmul(v[q], roots[q * t]), k);
        }
        // one copy of the butterfly: forward then (MID) backward
#pragma unroll 1
        for (int d = kind == GEN_MID && !fwd ? 1 : 0; d < (kind == GEN_MID && bwd ? 2 : 1); d++) {
            gen_dft<R>(v);
            if (kind == GEN_MID && d == 0) mid(v, p0);
        }
        if (kind == GEN_FWD) {
            const int k = shifts[s];
            v[0] = gen_shift(fx_quarter(v[0]), k);
#pragma unroll
            for (int q = 1; q < R; q++) v[q] = gen_shift(fx_cmul(v[q], roots[q * t]), k);
        }
#pragma unroll
        for (int q = 0; q < R; q++) data[at(p0 + q * M)] = v[q];
    }
}

// the same for a prime radix from 11 to 31: direct sums of products (rare
// lengths)
template <typename AT, typename MID1>
__device__ __noinline__ void gen_stage_loop(const GenPlan &p, int s, int kind, int i0, int step, bool fwd, bool bwd,
                                            const int4 *roots, const int *shifts, fxc *data, AT at, MID1 mid1)
{
    const int R = p.radix[s], M = p.m[s], nb = p.n / R, tws = nb / M;
    for (int b = i0; b < nb; b += step) {
        const int g = M > 1 ? (int)__umulhi((unsigned)b, p.magic[s]) : b, j = b - g * M;
        const int p0 = g * R * M + j;
        fxc v[31];
#pragma unroll 1
        for (int q = 0; q < R; q++) {
            v[q] = data[at(p0 + q * M)];
            if (kind == GEN_BWD) v[q] = gen_shift(q ? fx_cmul(v[q], roots[q * j * tws]) : fx_quarter(v[q]), shifts[s]);
        }
#pragma unroll 1
        for (int d = kind == GEN_MID && !fwd ? 1 : 0; d < (kind == GEN_MID && bwd ? 2 : 1); d++) {
#pragma unroll 1
            for (int k = 0; k < R; k++) {
                fxc acc = fx_quarter(v[0]);
#pragma unroll 1
                for (int q = 1; q < R; q++) acc = cadd(acc, fx_cmul(v[q], roots[((q * k) % R) * (p.n / R)]));
                data[at(p0 + k * M)] = acc;
            }
#pragma unroll 1
            for (int k = 0; k < R; k++) {
                v[k] = data[at(p0 + k * M)];
                if (kind == GEN_MID && d == 0) mid1(v[k], p0 + k);
                if (kind == GEN_FWD)
                    v[k] = gen_shift(k ? fx_cmul(v[k], roots[k * j * tws]) : fx_quarter(v[k]), shifts[s]);
                data[at(p0 + k * M)] = v[k];
            }
        }
    }
}

// MULT: the phase is a multiplier table (fft_fix.cuh)
template <int MODE, bool MULT = false>
__global__ void __launch_bounds__(GEN_THREADS, 4)
gen_pass_kernel(const PassArgs<double> a, const __grid_constant__ GenPlan p)
{
    using T = double;
    using V = double2;
    constexpr bool kFwd = MODE != MODE_INV, kBwd = MODE == MODE_FUSED || MODE == MODE_INV;
    const int n = p.n, lw = p.lw, Wn = 1 << lw;
    const bool xl = a.stride == 1;
    // shared memory: roots [n], phase [n] (one row for all lines), the tile
    extern __shared__ __align__(128) unsigned char smem_raw[];
    int4 *roots = reinterpret_cast<int4 *>(smem_raw);
    int4 *sph = roots + n;
    const bool rowph = MODE == MODE_FUSED && a.prow != 0;
    const bool mask = MODE == MODE_FUSED && a.mask_lim != nullptr;
    fxc *data = reinterpret_cast<fxc *>(sph + (MODE == MODE_FUSED && !rowph && !mask ? n : 0));
    static_assert(!MULT || MODE == MODE_FUSED, "multipliers: fused passes");
    __shared__ int sword[64], smword[64];    // (m: of the multiplied spectrum)
    __shared__ unsigned ssum[64], smsum[64];
    const int tid = threadIdx.x;
    // a thread's line, its first position and its stride over the positions
    const int lstep = 7 - lw, step = 1 << lstep;
    const int w = xl ? tid >> lstep : tid & (Wn - 1), i0 = xl ? tid & (step - 1) : tid >> lw;
    // slots: x lines one after the other with a pad per 16 cells (stages of
    // radix 16 and 8 would otherwise meet in one bank), columns interleaved
    const int LS = n + (n >> 4) + 1;
    const int off = xl ? w * LS : w;
    auto at = [=](int pos) { return xl ? off + pos + (pos >> 4) : (pos << lw) + off; };
    auto tile_sync = [=] {
        if (xl && lstep <= 5) __syncwarp();  // a line's threads are lanes of one warp
        else __syncthreads();
    };

    const int4 *groots = reinterpret_cast<const int4 *>(a.tw);
    const int *mode_at = reinterpret_cast<const int *>(groots + n), *pos_of = mode_at + n;
    // a phase table starts with its exponent
    const int4 *gphase = reinterpret_cast<const int4 *>(a.phase) + 1;
    for (int i = tid; i < n; i += GEN_THREADS) {
        roots[i] = groots[i];
        if (MODE == MODE_FUSED && !rowph && !mask) sph[i] = gphase[i];
    }
    const int fxpe = MODE == MODE_FUSED && !mask ? gphase[-1].x : 0;
    (void)fxpe;
    const int red = a.red;
    const T kmult = a.kmult;

    asm volatile("griddepcontrol.wait;" ::: "memory");
    const bool scaled = a.scale != nullptr;
    const T scale = scaled ? load_scale<T>(a.scale) : (T)1;
    const bool fxnl = MODE == MODE_FUSED && a.nl_mode == NL_REAL;
    T acc_mass = 0, acc_pot = 0, acc_int = 0, acc_kin = 0, acc_rot = 0;
    double tot[RQ_COUNT] = {0.0, 0.0, 0.0, 0.0, 0.0};

    const int ntiles = (a.nlines + Wn - 1) >> lw;
    for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
        const int g = (tile << lw) + w;
        const bool valid = g < a.nlines;
        const int gg = valid ? g : 0;
        const uint32_t base = (uint32_t)((gg % a.m0) * a.s0 + (gg / a.m0) * a.s1);
        const uint32_t st = xl ? 1u : (uint32_t)a.stride;
        const int row = gg % a.rowmod;
        // ---- load the line (zeros past the last one)
        __syncthreads();  // the tables; the previous tile's epilogue
        if (i0 == 0) {
            sword[w] = 0;
            ssum[w] = 0u;
            if (MULT) {
                smword[w] = 0;
                smsum[w] = 0u;
            }
        }
        float top = 0.f;  // the largest upper word
#pragma unroll 4
        for (int i = i0; i < n; i += step) {
            const uint32_t e = base + (uint32_t)i * st;
            V x = valid ? a.in[e] : mk<V>((T)0, (T)0);
            if constexpr (MODE == MODE_FUSED) {
                if (a.nl_pre) {  // chi = N(scale * psi) of the merged imaginary-time step
                    x = NLImag64(a.nl_beta, a.nl_dt, scale, a.nl_fx.tab2)(x, a.V && valid ? a.V[e] : (T)0);
                    if (a.nl_pre_out && valid) a.nl_pre_out[e] = x;
                } else if (scaled) {
                    x = cscale(x, scale);
                }
            }
            if constexpr (MODE == MODE_DIAG) {
                if ((red & (RED_POINT | RED_MASS)) && valid) {
                    const T rho = x.x * x.x + x.y * x.y;
                    acc_mass += rho;
                    if (red & RED_POINT) {
                        acc_int += rho * rho;
                        if (a.V) acc_pot += a.V[e] * rho;
                    }
                }
            }
            const int slot = at(MODE == MODE_INV ? pos_of[i] : i);
            reinterpret_cast<double2 *>(data)[slot] = x;
            const float hx = fabsf(__int_as_float(__double2hiint(x.x)));
            const float hy = fabsf(__int_as_float(__double2hiint(x.y)));
            asm("max.NaN.f32 %0, %0, %1;" : "+f"(top) : "f"(hx));
            asm("max.NaN.f32 %0, %0, %1;" : "+f"(top) : "f"(hy));
        }
        if (MODE == MODE_DIAG && !(red & RED_KIN)) {  // no spectrum wanted
            tot[RQ_MASS] += (double)acc_mass;
            tot[RQ_POT] += (double)acc_pot;
            tot[RQ_INT] += (double)acc_int;
            acc_mass = acc_pot = acc_int = (T)0;
            continue;
        }
        // ---- the line's quantum from its 2-norm (sums of squares in whole units
        // of 2^-16, so that their order does not matter)
        tile_sync();
        atomicMax(&sword[w], __float_as_int(top));
        tile_sync();
        const int word = sword[w], ref = fx_ref(word);
        const bool bad = word >= 0x7ff00000;
        float n2 = 0.f;
        for (int i = i0; i < n; i += step) {
            const double2 x = reinterpret_cast<const double2 *>(data)[at(MODE == MODE_INV ? pos_of[i] : i)];
            n2 += fx_norm2<1>(&x, ref);
        }
        atomicAdd(&ssum[w], bad ? 0u : (unsigned)(n2 * 65536.f) + 1u);
        tile_sync();
        const int q = max(fx_quantum(ref, (float)ssum[w] * (1.f / 65536.f)) + 60 - (kFwd ? p.bits_f : p.bits_i), -1020);
        for (int i = i0; i < n; i += step) {
            const int slot = at(MODE == MODE_INV ? pos_of[i] : i);
            const double2 x = reinterpret_cast<const double2 *>(data)[slot];
            const fxc c = fxc{fx_from(x.x, 1084 + q), fx_from(x.y, 1084 + q)};
            data[slot] = MODE == MODE_INV ? fxc{c.y, c.x} : c;  // exchanged from here on
        }
        // ---- spectral work on one value at position pos: sums, mask or phase,
        // exchange
        const int lim = mask ? a.mask_lim[gg] : 0;
        const int4 *ph = rowph ? gphase + (int64_t)row * a.prow : sph;
        (void)lim;
        (void)ph;
        float s2 = 0.f;  // MULT: this thread's sum of squares
        int qm = 0;      // and the exponent that the products' quantum adds
        (void)s2;
        auto spectral = [&](fxc &u, int pos) {
            if constexpr (MODE == MODE_FUSED || MODE == MODE_DIAG) {
                if (red & RED_KIN) {
                    const int k = mode_at[pos], kk = k < (n + 1) / 2 ? k : k - n;
                    const T xi = (T)kk * kmult;
                    const V X = gen_value(u, q + p.ef, bad);
                    const T m2 = X.x * X.x + X.y * X.y;
                    acc_kin += xi * xi * m2 * (T)(1.0 / n);
                    if (a.coord) acc_rot += xi * m2 * (T)(1.0 / n) * (T)a.coord[row];
                }
            }
            if constexpr (MULT) {
                const int4 t = ph[pos];
                u = fx_mult(u, t);
                s2 += fx_mult_norm2(u, t.z);
            } else if constexpr (MODE == MODE_FUSED) {
                if (mask) {
                    const int k = mode_at[pos], kk = k < (n + 1) / 2 ? k : n - k;
                    u = kk <= lim ? gen_shift(fx_quarter(u), p.kp) : fxc{0, 0};
                } else {
                    u = gen_shift(fx_cmul(u, ph[pos]), p.kp);
                }
                u = fxc{u.y, u.x};
            }
        };
        // ---- the stages
        const int S = p.nst;
        const int *kb = kFwd ? p.kb : p.ki;
        // (MULT: the middle stage is two, with the products' quantum between them)
        const int mid2 = MULT ? S : S - 1;
#pragma unroll 1
        for (int it = kFwd ? 0 : S - 1; it < (kBwd ? mid2 + S : S); it++) {
            const int s = it < S ? it : mid2 + S - 1 - it;
            const int kind = it < S - 1 ? GEN_FWD : it <= mid2 ? GEN_MID : GEN_BWD;
            const int *sh = kind == GEN_FWD ? p.kf : kb;
            const bool fwd = kFwd && (!MULT || it < S), bwd = kBwd && (!MULT || it >= S);
            tile_sync();
            auto run = [&](auto radix) {
                constexpr int R = decltype(radix)::value;
                gen_stage<R>(p, s, kind, i0, step, fwd, bwd, roots, sh, data, at, [&](fxc *u, int p0) {
#pragma unroll
                    for (int i = 0; i < R; i++) spectral(u[i], p0 + i);
                });
            };
            switch (p.radix[s]) {
            case 2: run(std::integral_constant<int, 2>{}); break;
            case 3: run(std::integral_constant<int, 3>{}); break;
            case 4: run(std::integral_constant<int, 4>{}); break;
            case 5: run(std::integral_constant<int, 5>{}); break;
            case 6: run(std::integral_constant<int, 6>{}); break;
            case 7: run(std::integral_constant<int, 7>{}); break;
            case 8: run(std::integral_constant<int, 8>{}); break;
            case 10: run(std::integral_constant<int, 10>{}); break;
            case 12: run(std::integral_constant<int, 12>{}); break;
            case 14: run(std::integral_constant<int, 14>{}); break;
            case 15: run(std::integral_constant<int, 15>{}); break;
            case 16: run(std::integral_constant<int, 16>{}); break;
            default:
                gen_stage_loop(p, s, kind, i0, step, fwd, bwd, roots, sh, data, at, spectral);
                break;
            }
            if constexpr (MULT) {
                if (it == S - 1) {
                    // the sum over the line's threads in whole units of 2^-16 of
                    // their largest sum's exponent
                    tile_sync();
                    atomicMax(&smword[w], __float_as_int(s2));
                    tile_sync();
                    const int e = min(smword[w] >> 23, 250);
                    atomicAdd(&smsum[w], (unsigned)(s2 * __int_as_float((254 - e) << 23) * 65536.f) + 1u);
                    tile_sync();
                    qm = fx_mult_shift((float)smsum[w] * __int_as_float(max(e - 16, 1) << 23), p.bits_p);
                    for (int i = i0; i < n; i += step) {
                        const int slot = at(i);
                        const fxc u = fx_scale2(data[slot], ph[i].z - qm);
                        data[slot] = fxc{u.y, u.x};
                    }
                    qm += p.kp;
                }
            }
        }
        tile_sync();
        // ---- results: positions in natural order, or the spectrum
        if constexpr (MODE == MODE_FWD) {
            for (int k = i0; k < n; k += step) {
                const V X = FxOut(q + p.ef, bad, 1.0, false)(data[at(pos_of[k])], true);
                if (valid) a.out[base + (uint32_t)k * st] = X;
            }
        }
        if constexpr (MODE == MODE_FUSED || MODE == MODE_INV) {
            int qv = q + (MODE == MODE_FUSED ? p.et + fxpe + qm : p.ei), lsh = 0, rsh = 0;
            if (fxnl) {
                const int sh = 190 + 2 * qv + a.nl_fx.ge;
                lsh = min(max(sh, 0), 63);
                rsh = min(max(-sh, 0), 63);
                qv += 2;
            }
            (void)lsh;
            (void)rsh;
            // 1/n: in the phase table, else here
            const bool byn = MODE == MODE_INV || mask;
            const FxOut oc(qv, bad, byn ? (double)a.inv_n : 1.0, byn);
            for (int i = i0; i < n; i += step) {
                const uint32_t e = base + (uint32_t)i * st;
                fxc u = data[at(i)];
                u = fxc{u.y, u.x};
                int vtop = 0;
                if constexpr (MODE == MODE_FUSED) {
                    if (fxnl) {
                        const long long vt = a.V && valid ? fx_vturn(a.V[e], a.nl_fx.d, a.nl_fx.de, &vtop) : 0;
                        u = fx_nl_real(u, vt, a.nl_fx.gh, a.nl_fx.gl, lsh, rsh, a.nl_fx.tab);
                    }
                }
                V v = oc(u, true);
                if (vtop == 0x7ff) v.x = v.y = __longlong_as_double(0x7ff8000000000000LL);
                if (!valid) continue;
                if constexpr (MODE == MODE_FUSED) {
                    if (a.nl_mode != NL_NONE && !fxnl) {
                        v = NLImag64(a.nl_beta, a.nl_dt, 1.0, a.nl_fx.tab2)(v, a.V ? a.V[e] : (T)0);  // imaginary time
                    }
                    if (red & RED_POINT) {
                        const T rho = v.x * v.x + v.y * v.y;
                        acc_mass += rho;
                        acc_int += rho * rho;
                        if (a.V) acc_pot += a.V[e] * rho;
                    } else if (red & RED_MASS) {
                        if (a.dot_with) {
                            const V d = a.dot_with[e];
                            acc_mass += d.x * v.x + d.y * v.y;
                        } else {
                            acc_mass += v.x * v.x + v.y * v.y;
                        }
                    }
                    if (a.acc) v = cadd(a.acc[e], v);
                }
                a.out[e] = v;
            }
        }
        if (red) {
            tot[RQ_MASS] += (double)acc_mass;
            tot[RQ_POT] += (double)acc_pot;
            tot[RQ_INT] += (double)acc_int;
            tot[RQ_KIN] += (double)acc_kin;
            tot[RQ_ROT] += (double)acc_rot;
            acc_mass = acc_pot = acc_int = acc_kin = acc_rot = (T)0;
        }
    }
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    if constexpr (MODE == MODE_FUSED || MODE == MODE_DIAG) {
        if (red) {
            unsigned qmask = 0;
            if (red & (RED_POINT | RED_MASS)) qmask |= 1u << RQ_MASS;
            if (red & RED_POINT) qmask |= (1u << RQ_POT) | (1u << RQ_INT);
            if (red & RED_KIN) qmask |= (1u << RQ_KIN) | (1u << RQ_ROT);
            block_sums_store<GEN_THREADS>(tot, qmask, a.partials);
            finish_reduction<T, GEN_THREADS>(a, qmask);
        }
    }
}

}  // namespace gpss

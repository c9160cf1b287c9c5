// pass_generic32.cuh -- the directional pass of FP32 fields for line lengths that
// the register kernel does not take (see pass_generic.cuh for which).
//
// Two kernels with the same arithmetic, a Stockham autosort transform with
// double-word roots: stage s of radix R with Ns = the product of the earlier
// radices maps
//     v[q] = src[j + q n/R] * w_{Ns R}^{(j mod Ns) q},  DFT_R(v),
//     dst[(j / Ns) Ns R + (j mod Ns) + q Ns] = v[q]
// for j < n/R, which ends in natural order without a reordering pass.  Radices
// 2, 4, 8, 16 use the register DFTs of fft_core.cuh, 3 a closed form, 5 and 7
// direct sums, other primes a loop.
//
//   gen32_pass_kernel   every pass without energy sums: one group of threads per
//                       line, so that no address needs a division by a run-time
//                       number, roots and phase in shared memory, the field
//                       read by the first stage and the phase applied by the
//                       first backward one; small tiles where a pass has few
//                       lines (480 x 360 step 108 -> 44 us).  Its mass sum adds
//                       the same cells in the same order as the tile kernel's
//                       (the sums of an FP32 pass are FP32 within a tile, and
//                       the mass lock carries their rounding into the field).
//   gen32_tile_kernel   the read-only energy passes, passes with energy sums,
//                       and mass sums over tiles that are not 16 columns: a tile
//                       of W lines shared by 256 threads, element by element.
#pragma once
#include "pass_kernel.cuh"
#include "pass_generic.cuh"

namespace gpss {

constexpr int GEN32_TILE_THREADS = 256;
constexpr int GEN32_MAX_STAGES = 12;

struct Gen32Plan {
    int n;
    int W;                          // lines per tile of the tile kernel
    int lw;                         // log2 of the lines per tile of the pass kernel
    int nst;                        // stages
    int radix[GEN32_MAX_STAGES];    // radices in stage order
    unsigned magic[GEN32_MAX_STAGES];  // ceil(2^32 / Ns): j / Ns = umulhi(j, magic) for Ns > 1
};

// Stage radices of n: largest power-of-two radices first, then the odd primes
// in increasing order (n as accepted by gen_plan_radices).
inline void gen32_plan(int n, Gen32Plan &p)
{
    p.n = n;
    p.nst = 0;
    int m = n, Ns = 1;
    for (int r : {16, 8, 4, 2, 3, 5, 7, 11, 13, 17, 19, 23, 29, 31}) {
        while (m % r == 0 && p.nst < GEN32_MAX_STAGES) {
            p.magic[p.nst] = Ns > 1 ? (unsigned)(((1ULL << 32) + (unsigned)Ns - 1) / (unsigned)Ns) : 0u;
            p.radix[p.nst++] = r;
            m /= r;
            Ns *= r;
        }
    }
    // tile kernel: as many lines as fit about 96 KB (two buffers), at most 16
    int W = (int)((96u * 1024u) / (16u * (unsigned)n));
    p.W = W > 16 ? 16 : W < 1 ? 1 : W;
}

// w_n^(m) as a double-word constant from the table (hi[n], lo[n]); DIR = +1
// conjugates (exp(+2 pi i m / n))
template <int DIR, typename V>
__device__ __forceinline__ void gen32_root(const V *roots, int n, int m, V &hi, V &lo)
{
    hi = roots[m];
    lo = roots[n + m];
    if (DIR > 0) {
        hi.y = -hi.y;
        lo.y = -lo.y;
    }
}

// radix-3 butterfly: X1,2 = x0 - s/2 +- DIR i (sqrt3/2) d, s = x1 + x2,
// d = x1 - x2; sqrt3/2 = sin(2 pi / 3) is the double-word table entry of
// w_n^(n/3) (its imaginary part is -sin)
template <int DIR, typename V> __device__ __forceinline__ void gen32_dft3(V *v, const V *roots, int n)
{
    using T = decltype(V::x);
    const T h = -roots[n / 3].y, l = -roots[n + n / 3].y;
    const V s = cadd(v[1], v[2]), d = csub(v[1], v[2]);
    const V x0 = v[0];
    v[0] = cadd(x0, s);
    const V m = mk<V>(fma((T)-0.5, s.x, x0.x), fma((T)-0.5, s.y, x0.y));
    // t = DIR i (sqrt3/2) d
    const V e = mk<V>(rmul2(d.x, h, l), rmul2(d.y, h, l));
    const V t = DIR < 0 ? mk<V>(e.y, -e.x) : mk<V>(-e.y, e.x);
    v[1] = cadd(m, t);
    v[2] = csub(m, t);
}

// direct DFT of odd prime size R (5, 7) with the table's roots w_R^{jk} = w_n^{jk n/R}
template <int R, int DIR, typename V>
__device__ __forceinline__ void gen32_dft_direct(V *v, const V *roots, int n)
{
    V out[R];
    const int step = n / R;
#pragma unroll
    for (int k = 0; k < R; k++) {
        V acc = v[0];
#pragma unroll
        for (int j = 1; j < R; j++) {
            V hi, lo;
            gen32_root<DIR>(roots, n, ((j * k) % R) * step, hi, lo);
            acc = cadd(acc, cmul2(v[j], hi, lo));
        }
        out[k] = acc;
    }
#pragma unroll
    for (int k = 0; k < R; k++) v[k] = out[k];
}

template <int R, int DIR, typename V> __device__ __forceinline__ void gen32_butterfly(V *v, const V *roots, int n)
{
    if constexpr (R == 2 || R == 4 || R == 8 || R == 16) dft<R, DIR>(v);
    else if constexpr (R == 3) gen32_dft3<DIR>(v, roots, n);
    else gen32_dft_direct<R, DIR>(v, roots, n);
}

// ---- the tile kernel ----

// one Stockham stage of radix R over the W lines of the tile (src -> dst)
template <int R, int DIR, typename V>
__device__ __forceinline__ void gen32_tile_stage(const V *src, V *dst, int W, int n, int Ns, const V *roots)
{
    const int L = n / R;
    const int items = W * L;
    for (int t = threadIdx.x; t < items; t += GEN32_TILE_THREADS) {
        const int w = t % W, j = t / W;
        const int k = j % Ns;
        V v[R];
#pragma unroll
        for (int q = 0; q < R; q++) v[q] = src[(j + q * L) * W + w];
        if (Ns > 1) {
            const int scale = n / (Ns * R);
#pragma unroll
            for (int q = 1; q < R; q++) {
                V hi, lo;
                gen32_root<DIR>(roots, n, (k * q * scale) % n, hi, lo);
                v[q] = cmul2(v[q], hi, lo);
            }
        }
        gen32_butterfly<R, DIR>(v, roots, n);
        const int base = (j / Ns) * Ns * R + k;
#pragma unroll
        for (int q = 0; q < R; q++) dst[(base + q * Ns) * W + w] = v[q];
    }
}

// one stage of a prime radix R in (7, 31] (rare lengths): the same mapping
// with a run-time radix, not unrolled
template <int DIR, typename V>
__device__ __noinline__ void gen32_tile_stage_prime(const V *src, V *dst, int W, int n, int Ns, int R, const V *roots)
{
    const int L = n / R;
    const int items = W * L;
    const int step = n / R;
    for (int t = threadIdx.x; t < items; t += GEN32_TILE_THREADS) {
        const int w = t % W, j = t / W;
        const int k = j % Ns;
        V v[31];
#pragma unroll 1
        for (int q = 0; q < R; q++) {
            v[q] = src[(j + q * L) * W + w];
            if (Ns > 1 && q > 0) {
                V hi, lo;
                gen32_root<DIR>(roots, n, (k * q * (n / (Ns * R))) % n, hi, lo);
                v[q] = cmul2(v[q], hi, lo);
            }
        }
        const int base = (j / Ns) * Ns * R + k;
#pragma unroll 1
        for (int kk = 0; kk < R; kk++) {
            V acc = v[0];
#pragma unroll 1
            for (int q = 1; q < R; q++) {
                V hi, lo;
                gen32_root<DIR>(roots, n, ((q * kk) % R) * step, hi, lo);
                acc = cadd(acc, cmul2(v[q], hi, lo));
            }
            dst[(base + kk * Ns) * W + w] = acc;
        }
    }
}

// the whole transform; returns the buffer holding the result
template <int DIR, typename V>
__device__ V *gen32_tile_fft(V *b0, V *b1, const Gen32Plan &p, const V *roots)
{
    V *src = b0, *dst = b1;
    int Ns = 1;
    for (int s = 0; s < p.nst; s++) {
        const int R = p.radix[s];
        switch (R) {
        case 2: gen32_tile_stage<2, DIR>(src, dst, p.W, p.n, Ns, roots); break;
        case 3: gen32_tile_stage<3, DIR>(src, dst, p.W, p.n, Ns, roots); break;
        case 4: gen32_tile_stage<4, DIR>(src, dst, p.W, p.n, Ns, roots); break;
        case 5: gen32_tile_stage<5, DIR>(src, dst, p.W, p.n, Ns, roots); break;
        case 7: gen32_tile_stage<7, DIR>(src, dst, p.W, p.n, Ns, roots); break;
        case 8: gen32_tile_stage<8, DIR>(src, dst, p.W, p.n, Ns, roots); break;
        case 16: gen32_tile_stage<16, DIR>(src, dst, p.W, p.n, Ns, roots); break;
        default: gen32_tile_stage_prime<DIR>(src, dst, p.W, p.n, Ns, R, roots); break;
        }
        __syncthreads();
        Ns *= R;
        V *t = src;
        src = dst;
        dst = t;
    }
    return src;
}

template <int MODE>
__global__ void __launch_bounds__(GEN32_TILE_THREADS)
gen32_tile_kernel(const PassArgs<float> a, const Gen32Plan p)
{
    using T = float;
    using V = float2;
    static_assert(MODE == MODE_FUSED || MODE == MODE_DIAG, "passes with sums");
    const int n = p.n, W = p.W;
    extern __shared__ __align__(128) unsigned char smem_raw[];
    V *buf0 = reinterpret_cast<V *>(smem_raw);
    V *buf1 = buf0 + (size_t)W * n;
    const V *roots = a.tw;  // hi[n], lo[n]
    const int red = a.red;
    const T kmult = a.kmult;

    asm volatile("griddepcontrol.wait;" ::: "memory");
    const bool scaled = a.scale != nullptr;
    const T scale = scaled ? load_scale<T>(a.scale) : (T)1;
    T acc_mass = 0, acc_pot = 0, acc_int = 0, acc_kin = 0, acc_rot = 0;
    double tot[RQ_COUNT] = {0.0, 0.0, 0.0, 0.0, 0.0};

    const int ntiles = (a.nlines + W - 1) / W;
    const int cells = W * n;
    auto gbase = [&](int g) -> int64_t { return (int64_t)(g % a.m0) * a.s0 + (int64_t)(g / a.m0) * a.s1; };
    for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
        // ---- load the tile: element (w, pos) at pos * W + w
        for (int t = threadIdx.x; t < cells; t += GEN32_TILE_THREADS) {
            int w, pos;
            if (a.stride == 1) { w = t / n; pos = t % n; }  // x lines: walk along the line
            else { w = t % W; pos = t / W; }                 // y/z: adjacent columns
            const int g = tile * W + w;
            V x = mk<V>((T)0, (T)0);
            if (g < a.nlines) {
                const int64_t e = gbase(g) + (int64_t)pos * a.stride;
                x = a.in[e];
                if constexpr (MODE == MODE_DIAG) {
                    if (red & (RED_POINT | RED_MASS)) {
                        const T rho = x.x * x.x + x.y * x.y;
                        acc_mass += rho;
                        if (red & RED_POINT) {
                            acc_int += rho * rho;
                            if (a.V) acc_pot += a.V[e] * rho;
                        }
                    }
                }
            }
            buf0[pos * W + w] = x;
        }
        if (MODE == MODE_DIAG && !(red & RED_KIN)) {  // no spectrum wanted
            tot[RQ_MASS] += (double)acc_mass;
            tot[RQ_POT] += (double)acc_pot;
            tot[RQ_INT] += (double)acc_int;
            acc_mass = acc_pot = acc_int = (T)0;
            continue;
        }
        __syncthreads();
        V *spec = gen32_tile_fft<-1>(buf0, buf1, p, roots);  // X[k] at k * W + w
        // ---- spectral work: sums, phase / mask, scale
        if constexpr (MODE == MODE_FUSED || MODE == MODE_DIAG) {
            for (int t = threadIdx.x; t < cells; t += GEN32_TILE_THREADS) {
                const int w = t % W, k = t / W, g = tile * W + w;
                if (g >= a.nlines) continue;
                const int row = g % a.rowmod;
                V X = spec[k * W + w];
                if (red & RED_KIN) {
                    const int kk = k < (n + 1) / 2 ? k : k - n;
                    const T xi = (T)kk * kmult;
                    const T m2 = X.x * X.x + X.y * X.y;
                    acc_kin += xi * xi * m2 * (T)(1.0 / n);
                    if (a.coord) acc_rot += xi * m2 * (T)(1.0 / n) * (T)a.coord[row];
                }
                if constexpr (MODE == MODE_FUSED) {
                    if (a.mask_lim) {
                        const int kk = k < (n + 1) / 2 ? k : n - k;
                        X = kk <= a.mask_lim[g] ? cscale(X, a.inv_n) : mk<V>((T)0, (T)0);
                    } else {
                        const V *ph = a.phase + (a.prow ? (int64_t)row * a.prow : 0);
                        X = cmul2(X, ph[k], ph[n + k]);
                        if (scaled) X = cscale(X, scale);
                    }
                    spec[k * W + w] = X;
                }
            }
            __syncthreads();
        }
        if constexpr (MODE == MODE_FUSED) {
            V *other = spec == buf0 ? buf1 : buf0;
            V *res = gen32_tile_fft<+1>(spec, other, p, roots);
            // ---- epilogue: positions in natural order
            for (int t = threadIdx.x; t < cells; t += GEN32_TILE_THREADS) {
                int w, pos;
                if (a.stride == 1) { w = t / n; pos = t % n; }
                else { w = t % W; pos = t / W; }
                const int g = tile * W + w;
                if (g >= a.nlines) continue;
                const int64_t e = gbase(g) + (int64_t)pos * a.stride;
                V v = res[pos * W + w];
                if (a.nl_mode != NL_NONE) {
                    const NLConst<T> nlc = nl_const<T>(a.nl_split, a.nl_beta, a.nl_dt);
                    const T vv = a.V ? a.V[e] : (T)0;
                    v = a.nl_mode == NL_IMAG ? nl_apply(v, vv, nlc, true) : nl_apply_real_cell(v, vv, nlc);
                }
                if (red & RED_POINT) {
                    const T rho = v.x * v.x + v.y * v.y;
                    acc_mass += rho;
                    acc_int += rho * rho;
                    if (a.V) acc_pot += a.V[e] * rho;
                } else if (red & RED_MASS) {
                    acc_mass += v.x * v.x + v.y * v.y;
                }
                if (a.acc) v = cadd(a.acc[e], v);
                a.out[e] = v;
            }
            __syncthreads();  // the next tile's load reuses the buffers
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
    {
        if (red) {
            unsigned qmask = 0;
            if (red & (RED_POINT | RED_MASS)) qmask |= 1u << RQ_MASS;
            if (red & RED_POINT) qmask |= (1u << RQ_POT) | (1u << RQ_INT);
            if (red & RED_KIN) qmask |= (1u << RQ_KIN) | (1u << RQ_ROT);
            block_sums_store<GEN32_TILE_THREADS>(tot, qmask, a.partials);
            finish_reduction<T, GEN32_TILE_THREADS>(a, qmask);
        }
    }
}


// ---- the pass kernel ----

// One thread's share of a stage on its line: `src(pos)` reads, `dst(pos)` is the
// slot to write.
template <int R, int DIR, typename SRC, typename DST>
__device__ __forceinline__ void gen32_stage(int n, int Ns, unsigned magic, int i0, int step, const float4 *roots,
                                            SRC src, DST dst)
{
    const int L = n / R;
    const int scale = n / (Ns * R);
    for (int j = i0; j < L; j += step) {
        const int g = Ns > 1 ? (int)__umulhi((unsigned)j, magic) : j, k = j - g * Ns;
        float2 v[R];
#pragma unroll
        for (int q = 0; q < R; q++) v[q] = src(j + q * L);
        if (Ns > 1) {
            const int t = k * scale;
#pragma unroll
            for (int q = 1; q < R; q++) {
                const float4 c = roots[q * t];
                v[q] = cmul2(v[q], make_float2(c.x, DIR > 0 ? -c.y : c.y), make_float2(c.z, DIR > 0 ? -c.w : c.w));
            }
        }
        if constexpr (R == 2 || R == 4 || R == 8 || R == 16) {
            dft<R, DIR>(v);
        } else {
            // the butterflies take their roots as rows of high and low parts
            float2 rr[2 * R];
#pragma unroll
            for (int m = 0; m < R; m++) {
                const float4 c = roots[m * (n / R)];
                rr[m] = make_float2(c.x, c.y);
                rr[R + m] = make_float2(c.z, c.w);
            }
            gen32_butterfly<R, DIR>(v, rr, R);
        }
#pragma unroll
        for (int q = 0; q < R; q++) *dst(g * Ns * R + k + q * Ns) = v[q];
    }
}

// a stage of a prime radix from 11 to 31
template <int DIR, typename SRC, typename DST>
__device__ __forceinline__ void gen32_stage_prime(int n, int Ns, unsigned magic, int R, int i0, int step,
                                                  const float4 *roots, SRC src, DST dst)
{
    const int L = n / R;
    auto root = [&](int m, float2 &hi, float2 &lo) {
        const float4 c = roots[m];
        hi = make_float2(c.x, DIR > 0 ? -c.y : c.y);
        lo = make_float2(c.z, DIR > 0 ? -c.w : c.w);
    };
    for (int j = i0; j < L; j += step) {
        const int g = Ns > 1 ? (int)__umulhi((unsigned)j, magic) : j, k = j - g * Ns;
        float2 v[31], hi, lo;
#pragma unroll 1
        for (int q = 0; q < R; q++) {
            v[q] = src(j + q * L);
            if (Ns > 1 && q > 0) {
                root(k * q * (n / (Ns * R)), hi, lo);
                v[q] = cmul2(v[q], hi, lo);
            }
        }
#pragma unroll 1
        for (int kk = 0; kk < R; kk++) {
            float2 acc = v[0];
#pragma unroll 1
            for (int q = 1; q < R; q++) {
                root(((q * kk) % R) * L, hi, lo);
                acc = cadd(acc, cmul2(v[q], hi, lo));
            }
            *dst(g * Ns * R + k + kk * Ns) = acc;
        }
    }
}

template <int DIR, typename SRC, typename DST>
__device__ __forceinline__ void gen32_stage_any(const Gen32Plan &p, int s, int Ns, int i0, int step,
                                                const float4 *roots, SRC src, DST dst)
{
    const int n = p.n;
    const unsigned mg = p.magic[s];
    switch (p.radix[s]) {
    case 2: gen32_stage<2, DIR>(n, Ns, mg, i0, step, roots, src, dst); break;
    case 3: gen32_stage<3, DIR>(n, Ns, mg, i0, step, roots, src, dst); break;
    case 4: gen32_stage<4, DIR>(n, Ns, mg, i0, step, roots, src, dst); break;
    case 5: gen32_stage<5, DIR>(n, Ns, mg, i0, step, roots, src, dst); break;
    case 7: gen32_stage<7, DIR>(n, Ns, mg, i0, step, roots, src, dst); break;
    case 8: gen32_stage<8, DIR>(n, Ns, mg, i0, step, roots, src, dst); break;
    case 16: gen32_stage<16, DIR>(n, Ns, mg, i0, step, roots, src, dst); break;
    default: gen32_stage_prime<DIR>(n, Ns, mg, p.radix[s], i0, step, roots, src, dst); break;
    }
}

template <int MODE>
__global__ void __launch_bounds__(GEN_THREADS, 5)
gen32_pass_kernel(const PassArgs<float> a, const __grid_constant__ Gen32Plan p)
{
    static_assert(MODE != MODE_DIAG, "energy passes: gen32_tile_kernel");
    const int n = p.n, lw = p.lw, Wn = 1 << lw;
    const bool xl = a.stride == 1;
    // shared memory: roots [n], phase [n] (one row for all lines), two tiles
    extern __shared__ __align__(128) unsigned char smem_raw[];
    float4 *roots = reinterpret_cast<float4 *>(smem_raw);
    float4 *sph = roots + n;
    const bool rowph = MODE == MODE_FUSED && a.prow != 0, mask = MODE == MODE_FUSED && a.mask_lim != nullptr;
    const int tid = threadIdx.x;
    // a thread's line, its first position and its stride over the positions
    const int lstep = 7 - lw, step = 1 << lstep;
    const int w = xl ? tid >> lstep : tid & (Wn - 1), i0 = xl ? tid & (step - 1) : tid >> lw;
    // slots: x lines one after the other with a pad per 16 cells, columns interleaved
    const int LS = n + (n >> 4) + 1, tile_slots = xl ? LS << lw : n << lw;
    const int off = xl ? w * LS : w;
    float2 *buf0 = reinterpret_cast<float2 *>(sph + (MODE == MODE_FUSED && !rowph && !mask ? n : 0));
    float2 *buf1 = buf0 + tile_slots;
    auto at = [=](int pos) { return xl ? off + pos + (pos >> 4) : (pos << lw) + off; };
    auto tile_sync = [=] {
        if (xl && lstep <= 5) __syncwarp();  // a line's threads are lanes of one warp
        else __syncthreads();
    };
    for (int i = tid; i < n; i += GEN_THREADS) {
        roots[i] = make_float4(a.tw[i].x, a.tw[i].y, a.tw[n + i].x, a.tw[n + i].y);
        if (MODE == MODE_FUSED && !rowph && !mask)
            sph[i] = make_float4(a.phase[i].x, a.phase[i].y, a.phase[n + i].x, a.phase[n + i].y);
    }
    const int red = a.red;

    asm volatile("griddepcontrol.wait;" ::: "memory");
    const bool scaled = a.scale != nullptr;
    const float scale = scaled ? load_scale<float>(a.scale) : 1.f;
    double tot[RQ_COUNT] = {0.0, 0.0, 0.0, 0.0, 0.0};

    const int ntiles = (a.nlines + Wn - 1) >> lw;
    for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
        const int g = (tile << lw) + w;
        const bool valid = g < a.nlines;
        const int gg = valid ? g : 0;
        const uint32_t base = (uint32_t)((gg % a.m0) * a.s0 + (gg / a.m0) * a.s1);
        const uint32_t st = xl ? 1u : (uint32_t)a.stride;
        const float2 *prow = rowph ? a.phase + (int64_t)(gg % a.rowmod) * a.prow : nullptr;
        const int lim = mask ? a.mask_lim[gg] : 0;
        const int S = p.nst;
        __syncthreads();  // the tables; the previous tile's epilogue
        float2 *src = buf1, *dst = buf0;
        auto flip = [&] {
            float2 *t = src;
            src = dst;
            dst = t;
        };
        auto put = [&](int pos) { return dst + at(pos); };
        // the field (lines past the last one read line 0, whose values go nowhere)
        auto field = [&](int pos) { return a.in[base + (uint32_t)pos * st]; };
        if constexpr (MODE != MODE_INV) {
            int Ns = 1;
#pragma unroll 1
            for (int s = 0; s < S; s++) {
                gen32_stage_any<-1>(p, s, Ns, i0, step, roots,
                                    [&](int pos) { return s == 0 ? field(pos) : src[at(pos)]; }, put);
                tile_sync();
                flip();
                Ns *= p.radix[s];
            }
        }
        if constexpr (MODE == MODE_FWD) {
            for (int k = i0; k < n; k += step)
                if (valid) a.out[base + (uint32_t)k * st] = src[at(k)];
        }
        if constexpr (MODE == MODE_FUSED || MODE == MODE_INV) {
            // the spectrum with its phase (or mask) and the deferred factor
            auto spectrum = [&](int k) {
                float2 X = src[at(k)];
                if (mask) {
                    const int kk = k < (n + 1) / 2 ? k : n - k;
                    return kk <= lim ? cscale(X, a.inv_n) : make_float2(0.f, 0.f);
                }
                if (rowph) {
                    X = cmul2(X, prow[k], prow[n + k]);
                } else {
                    const float4 c = sph[k];
                    X = cmul2(X, make_float2(c.x, c.y), make_float2(c.z, c.w));
                }
                return scaled ? cscale(X, scale) : X;
            };
            int Ns = 1;
#pragma unroll 1
            for (int s = 0; s < S; s++) {
                gen32_stage_any<+1>(p, s, Ns, i0, step, roots,
                                    [&](int pos) {
                                        if (s > 0) return src[at(pos)];
                                        if constexpr (MODE == MODE_INV) return field(pos);
                                        else return spectrum(pos);
                                    },
                                    put);
                tile_sync();
                flip();
                Ns *= p.radix[s];
            }
            const NLConst<float> nlc = nl_const<float>(a.nl_split, a.nl_beta, a.nl_dt);
            for (int i = i0; i < n; i += step) {
                const uint32_t e = base + (uint32_t)i * st;
                float2 v = src[at(i)];
                if constexpr (MODE == MODE_INV) {
                    v = cscale(v, a.inv_n);
                } else {
                    if (a.nl_mode != NL_NONE) {
                        const float vv = a.V && valid ? a.V[e] : 0.f;
                        v = a.nl_mode == NL_IMAG ? nl_apply(v, vv, nlc, true) : nl_apply_real_cell(v, vv, nlc);
                    }
                    if (red & RED_MASS) dst[at(i)].x = v.x * v.x + v.y * v.y;
                    if (a.acc && valid) v = cadd(a.acc[e], v);
                }
                if (valid) a.out[e] = v;
            }
            if (MODE == MODE_FUSED && (red & RED_MASS)) {
                // columns: sixteen sums each, over every sixteenth cell
                __syncthreads();
                if (valid && i0 < 16) {
                    float acc = 0.f;
                    for (int i = i0; i < n; i += 16) acc += dst[at(i)].x;
                    tot[RQ_MASS] += (double)acc;
                }
            }
        }
    }
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    if constexpr (MODE == MODE_FUSED) {
        if (red) {
            block_sums_store<GEN_THREADS>(tot, 1u << RQ_MASS, a.partials);
            finish_reduction<float, GEN_THREADS>(a, 1u << RQ_MASS);
        }
    }
}

// Which kernel: the pass kernel's mass sum adds what a tile of 16 columns does.
inline bool gen32_fast(int mode, const PassArgs<float> &a, const Gen32Plan &p)
{
    if (mode == MODE_DIAG) return false;
    return a.red == 0 || (a.red == RED_MASS && a.stride != 1 && p.W == 16 && p.lw <= 3);
}

}  // namespace gpss

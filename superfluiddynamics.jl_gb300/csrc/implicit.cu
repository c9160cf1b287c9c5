// implicit.cu -- pointwise kernels of the implicit imaginary-/real-time
// schemes (src/NumModels/GrossPitaevskii/backward-euler.jl, crank-nicolson.jl)
// and of their BiCGStab solver (src/NumModels/krylov.jl:1-67).  lapRot comes
// from the fused directional passes (the host chains them); everything else of
// a Krylov iteration is here.
#include <algorithm>
#include "gpss_internal.h"
#include "pdl.cuh"

namespace gpss {

static int im_grid(int64_t count)
{
    int64_t b = (count + 255) / 256;
    const int64_t cap = 152 * 8;
    if (b > cap) b = cap;
    if (b < 1) b = 1;
    return (int)b;
}

#define GRID_LOOP(e, total) \
    for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < (total); e += (int64_t)gridDim.x * blockDim.x)

// ---- setup of a time step / Newton iteration

// BackwardEuler:          M = 1 / (1/dt + V + beta|phi|^2),  b = M phi / dt
// BackwardEulerNoPrecond: Anl = V + beta|phi|^2,             b = phi / dt
template <typename T>
__global__ void k_im_prep_be(const vec2<T> *__restrict__ phi, const T *__restrict__ V, double beta, double idt,
                             double dt, int scheme, vec2<T> *__restrict__ M, T *__restrict__ Anl,
                             vec2<T> *__restrict__ b, int64_t total)
{
    pdl_enter();
    GRID_LOOP(e, total) {
        const vec2<T> p = phi[e];
        const T vv = V ? V[e] : (T)0;
        const T a2 = p.x * p.x + p.y * p.y;
        if (scheme == IM_SCHEME_BE) {
            const T m = (T)1.0 / ((T)idt + vv + (T)beta * a2);
            M[e] = mk<vec2<T>>(m, (T)0);
            b[e] = mk<vec2<T>>(m * p.x / (T)dt, m * p.y / (T)dt);
        } else {
            Anl[e] = vv + (T)beta * a2;
            b[e] = mk<vec2<T>>(p.x / (T)dt, p.y / (T)dt);
        }
    }
}

// Crank-Nicolson schemes, one Newton iteration: psi = (phi1 + phi)/2,
// Anl = V + (2 or 3) beta|psi|^2, Anl2 = beta psi^2,
// M = 1 / (1/dt + d) (stationary) or 1 / (i/dt - d) (T schemes), d = (V + 3 beta|psi|^2)/2
template <typename T>
__global__ void k_im_prep_cn(const vec2<T> *__restrict__ phi, const vec2<T> *__restrict__ phi1,
                             const T *__restrict__ V, double beta, double idt, int scheme,
                             vec2<T> *__restrict__ psim, T *__restrict__ Anl, vec2<T> *__restrict__ Anl2,
                             vec2<T> *__restrict__ M, int64_t total)
{
    pdl_enter();
    const bool newton = scheme == IM_SCHEME_CN || scheme == IM_SCHEME_CN_T;
    const bool tsch = scheme == IM_SCHEME_CN_T || scheme == IM_SCHEME_CN_QN_T;
    const T bt = (T)beta;
    GRID_LOOP(e, total) {
        const vec2<T> a = phi1[e], p = phi[e];
        const vec2<T> q = mk<vec2<T>>((T)0.5 * (a.x + p.x), (T)0.5 * (a.y + p.y));
        psim[e] = q;
        const T vv = V ? V[e] : (T)0;
        const T a2 = q.x * q.x + q.y * q.y;
        Anl[e] = vv + (newton ? (T)2 : (T)3) * bt * a2;
        const T qr = bt * q.x, qi = bt * q.y;
        Anl2[e] = mk<vec2<T>>(qr * q.x - qi * q.y, qr * q.y + qi * q.x);
        const T d = (vv + (T)3 * bt * a2) * (T)0.5;
        if (!tsch) {
            M[e] = mk<vec2<T>>((T)1.0 / ((T)idt + d), (T)0);
        } else {
            const T zr = -d, zi = (T)idt, den = zr * zr + zi * zi;
            M[e] = mk<vec2<T>>(zr / den, -zi / den);
        }
    }
}

// b = (1/dt)(phi1 - phi) + f psi - lap     (stationary)
//   = (i/dt)(phi1 - phi) - f psi + lap     (T schemes),   f = V + beta|psi|^2, lap = lapRot(psi)
template <typename T>
__global__ void k_im_rhs_cn(const vec2<T> *__restrict__ phi, const vec2<T> *__restrict__ phi1,
                            const vec2<T> *__restrict__ psim, const vec2<T> *__restrict__ lap,
                            const T *__restrict__ V, double beta, double idt, int tsch, vec2<T> *__restrict__ b,
                            int64_t total)
{
    pdl_enter();
    GRID_LOOP(e, total) {
        const vec2<T> q = psim[e], L = lap[e], a = phi1[e], p = phi[e];
        const T f = (V ? V[e] : (T)0) + (T)beta * (q.x * q.x + q.y * q.y);
        const T dr = a.x - p.x, di = a.y - p.y, id = (T)idt;
        if (!tsch)
            b[e] = mk<vec2<T>>((id * dr + f * q.x) - L.x, (id * di + f * q.y) - L.y);
        else
            b[e] = mk<vec2<T>>((-(id * di) - f * q.x) + L.x, (id * dr - f * q.y) + L.y);
    }
}

// ---- dot products finished in the kernel that has the vectors at hand
//
// A BiCGStab iteration needs three pairs of dot products.  They are summed
// where one of their vectors is formed (the operator's result, the residual):
// FP64 per thread, per CTA by shuffles, and by the last CTA to arrive over the
// per-CTA partials in a fixed order; one thread of it then forms the
// iteration's scalars (KrylovDev).  With kernels of their own for the products,
// their finish and the scalars an iteration was 19 launches, now 11 (64^3
// backward Euler, 4 steps, 1696 -> 1590 us).
struct DotArgs {
    int what;                // KRY_*
    double *partials;        // [2][gridDim.x]
    unsigned int *counter;   // 0 between launches
    double *out;             // the two sums (nullable)
    KrylovDev *K;
    double tol;              // KRY_CHECK
    int nkrylov;
};

// the scalars of one solve from two dot products (krylov.jl:1-67, one thread)
__device__ void kry_scalars(const DotArgs &d, double d0, double d1)
{
    KrylovDev *K = d.K;
    if (d.what == KRY_INIT) {  // normb = sqrt(b.b) (or |M b|), a fresh solve
        K->normb = sqrt(d0);
        K->rr2 = K->alpha = K->omega = K->beta = 0.0;
        K->done = K->niter = K->nonfinite = K->it = 0;
        return;
    }
    if (d.what == KRY_NONE || K->done) return;
    if (d.what == KRY_ALPHA) {  // iteration it: rr2 = r.r2, alpha = rr2 / (Ap.r2)
        K->it += 1;
        K->rr2 = d0;
        K->alpha = d0 / d1;
    } else if (d.what == KRY_OMEGA) {  // omega = (As.s) / (As.As)
        K->omega = d0 / d1;
    } else {
        // the stopping test on |r| / normb, then niter = it and beta =
        // (r.r2) / rr2 * alpha / omega; the last allowed iteration ends the solve
        if (!isfinite(d0)) {
            K->nonfinite = 1;
            K->done = 1;
        } else if (sqrt(d0) / K->normb < d.tol) {
            K->done = 1;
        } else {
            K->niter = K->it;
            K->beta = d1 / K->rr2 * K->alpha / K->omega;
            if (K->it >= d.nkrylov) K->done = 1;
        }
    }
}

// sums of x1 and x2 over the grid (CTAs of 256 threads), then the scalars
__device__ __forceinline__ void dot_finish(double x1, double x2, const DotArgs &d)
{
    __shared__ double s1[8], s2[8];
    __shared__ bool last;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    auto cta = [&](double &a, double &b) {  // thread 0 gets the CTA's sums
        for (int o = 16; o > 0; o >>= 1) {
            a += __shfl_xor_sync(0xffffffffu, a, o);
            b += __shfl_xor_sync(0xffffffffu, b, o);
        }
        if (lane == 0) {
            s1[wid] = a;
            s2[wid] = b;
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            a = s1[0];
            b = s2[0];
            for (int i = 1; i < 8; i++) {
                a += s1[i];
                b += s2[i];
            }
        }
    };
    cta(x1, x2);
    if (threadIdx.x == 0) {
        d.partials[blockIdx.x] = x1;
        d.partials[gridDim.x + blockIdx.x] = x2;
        __threadfence();  // the partials before the arrival
        last = atomicAdd(d.counter, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    double a = 0.0, b = 0.0;
    for (unsigned i = threadIdx.x; i < gridDim.x; i += blockDim.x) {
        a += __ldcg(d.partials + i);
        b += __ldcg(d.partials + gridDim.x + i);
    }
    cta(a, b);
    if (threadIdx.x == 0) {
        if (d.out) {
            d.out[0] = a;
            d.out[1] = b;
        }
        kry_scalars(d, a, b);
        *d.counter = 0u;
    }
}

// Re(a conj b) in FP64
template <typename T> __device__ __forceinline__ double re_dot(vec2<T> a, vec2<T> b)
{
    return (double)a.x * (double)b.x + (double)a.y * (double)b.y;
}

// out = prodA(x) given lap = lapRot(x) (backward-euler.jl:87-90, 179-189;
// crank-nicolson.jl:112-114, 234-236, 356-359, 478-481); bsub: out = b - prodA(x);
// precond: out = M * out.  Dots: KRY_ALPHA r.r2 and out.r2; KRY_OMEGA out.x and out.out
template <typename T>
__global__ void k_im_op(const vec2<T> *__restrict__ x, const vec2<T> *__restrict__ lap, int scheme, double idt,
                        const vec2<T> *__restrict__ M, const T *__restrict__ Anl, const vec2<T> *__restrict__ Anl2,
                        const vec2<T> *__restrict__ b, int precond, vec2<T> *__restrict__ out, int64_t total,
                        const vec2<T> *__restrict__ r, const vec2<T> *__restrict__ r2, const DotArgs d)
{
    pdl_enter();
    const T id = (T)idt, h = (T)0.5;
    double x1 = 0.0, x2 = 0.0;
    GRID_LOOP(e, total) {
        const vec2<T> v = x[e], L = lap[e];
        T ox, oy;
        switch (scheme) {
        case IM_SCHEME_BE: {
            const T m = M[e].x;
            ox = v.x - m * L.x; oy = v.y - m * L.y;
            break;
        }
        case IM_SCHEME_BE_NOPRE: {
            const T a = id + Anl[e];
            ox = a * v.x - L.x; oy = a * v.y - L.y;
            break;
        }
        case IM_SCHEME_CN: {
            const T a = id + Anl[e];
            const vec2<T> q = Anl2[e];
            const T hx = h * q.x, hy = h * q.y;
            ox = (a * v.x + (hx * v.x + hy * v.y)) - h * L.x;
            oy = (a * v.y + (hy * v.x - hx * v.y)) - h * L.y;
            break;
        }
        case IM_SCHEME_CN_QN: {
            const T a = id + Anl[e] * h;
            ox = a * v.x - h * L.x; oy = a * v.y - h * L.y;
            break;
        }
        case IM_SCHEME_CN_T: {
            const T ar = -h * Anl[e];
            const vec2<T> q = Anl2[e];
            const T hx = h * q.x, hy = h * q.y;
            ox = ((ar * v.x - id * v.y) - (hx * v.x + hy * v.y)) + h * L.x;
            oy = ((ar * v.y + id * v.x) - (hy * v.x - hx * v.y)) + h * L.y;
            break;
        }
        default: {  // IM_SCHEME_CN_QN_T
            const T ar = -(Anl[e] * h);
            ox = (ar * v.x - id * v.y) + h * L.x;
            oy = (ar * v.y + id * v.x) + h * L.y;
            break;
        }
        }
        if (b) {
            const vec2<T> bb = b[e];
            ox = bb.x - ox; oy = bb.y - oy;
        }
        if (precond) {
            const vec2<T> m = M[e];
            const T tx = m.x * ox - m.y * oy, ty = m.x * oy + m.y * ox;
            ox = tx; oy = ty;
        }
        const vec2<T> o = mk<vec2<T>>(ox, oy);
        out[e] = o;
        if (d.what == KRY_ALPHA) {
            const vec2<T> w = r2[e];
            x1 += re_dot<T>(r[e], w);
            x2 += re_dot<T>(o, w);
        } else if (d.what == KRY_OMEGA) {
            x1 += re_dot<T>(o, v);
            x2 += re_dot<T>(o, o);
        }
    }
    if (d.what != KRY_NONE) dot_finish(x1, x2, d);
}

// ---- BiCGStab vector operations (krylov.jl)

// a.a, its sum to d.out or into the scalars
template <typename T>
__global__ void k_im_norm2(const vec2<T> *__restrict__ a, int64_t total, const DotArgs d)
{
    pdl_enter();
    double x = 0.0;
    GRID_LOOP(e, total) { x += re_dot<T>(a[e], a[e]); }
    dot_finish(x, 0.0, d);
}

// out = x - alpha y
template <typename T>
__global__ void k_im_axmy(vec2<T> *__restrict__ out, const vec2<T> *__restrict__ x, double alpha,
                          const vec2<T> *__restrict__ y, int64_t total)
{
    pdl_enter();
    const T a = (T)alpha;
    GRID_LOOP(e, total) {
        const vec2<T> u = x[e], w = y[e];
        out[e] = mk<vec2<T>>(u.x - a * w.x, u.y - a * w.y);
    }
}

// s = r - alpha Ap (alpha from the device)
template <typename T>
__global__ void k_im_axmy_k(vec2<T> *__restrict__ out, const vec2<T> *__restrict__ x, const vec2<T> *__restrict__ y,
                            const KrylovDev *__restrict__ K, int64_t total)
{
    pdl_enter();
    if (K->done) return;
    const T a = (T)K->alpha;
    GRID_LOOP(e, total) {
        const vec2<T> u = x[e], w = y[e];
        out[e] = mk<vec2<T>>(u.x - a * w.x, u.y - a * w.y);
    }
}

// phi = (phi + alpha p) + omega s;  r = s - omega As;  KRY_CHECK on r.r and r.r2
template <typename T>
__global__ void k_im_update_k(vec2<T> *__restrict__ phi, const vec2<T> *__restrict__ p,
                              const vec2<T> *__restrict__ s, const vec2<T> *__restrict__ As, vec2<T> *__restrict__ r,
                              const vec2<T> *__restrict__ r2, const KrylovDev *K, int64_t total, const DotArgs d)
{
    pdl_enter();
    if (K->done) return;  // (the last CTA, which may set it, arrives after every CTA has read it)
    const T a = (T)K->alpha, w = (T)K->omega;
    double x1 = 0.0, x2 = 0.0;
    GRID_LOOP(e, total) {
        const vec2<T> f = phi[e], pp = p[e], ss = s[e], aa = As[e];
        phi[e] = mk<vec2<T>>((f.x + a * pp.x) + w * ss.x, (f.y + a * pp.y) + w * ss.y);
        const vec2<T> rr = mk<vec2<T>>(ss.x - w * aa.x, ss.y - w * aa.y);
        r[e] = rr;
        x1 += re_dot<T>(rr, rr);
        x2 += re_dot<T>(rr, r2[e]);
    }
    dot_finish(x1, x2, d);
}

// p = r + beta (p - omega Ap)
template <typename T>
__global__ void k_im_pdir_k(vec2<T> *__restrict__ p, const vec2<T> *__restrict__ r, const vec2<T> *__restrict__ Ap,
                            const KrylovDev *__restrict__ K, int64_t total)
{
    pdl_enter();
    if (K->done) return;
    const T bt = (T)K->beta, w = (T)K->omega;
    GRID_LOOP(e, total) {
        const vec2<T> pp = p[e], rr = r[e], aa = Ap[e];
        const T qx = pp.x - w * aa.x, qy = pp.y - w * aa.y;
        p[e] = mk<vec2<T>>(rr.x + bt * qx, rr.y + bt * qy);
    }
}

// out = M x (the preconditioner applied to a vector)
template <typename T>
__global__ void k_im_mfield(vec2<T> *__restrict__ out, const vec2<T> *__restrict__ M, const vec2<T> *__restrict__ x,
                            int64_t total)
{
    pdl_enter();
    GRID_LOOP(e, total) {
        const vec2<T> m = M[e], v = x[e];
        out[e] = mk<vec2<T>>(m.x * v.x - m.y * v.y, m.x * v.y + m.y * v.x);
    }
}

// ---- host launchers

// Kernels that end in dot_finish: four cells per thread, at most eight CTAs per
// SM as in the sweeps without sums.  (Two per SM keep too few loads in flight:
// backward Euler 256^3, us per step, FP64 8100 -> 7526, FP32 3330 -> 2643; 128^3 980 ->
// 938 and 491 -> 412; smaller fields have fewer CTAs than either.)
static int dot_grid(int64_t total) { return (int)std::min<int64_t>((total + 1023) / 1024, KRY_MAX_CTAS); }
static DotArgs dot_args(const KryScratch &k, int what)
{
    DotArgs d;
    d.what = what;
    d.partials = k.partials;
    d.counter = k.counter;
    d.out = k.dots;
    d.K = k.K;
    d.tol = 0.0;
    d.nkrylov = 0;
    return d;
}

template <typename T>
cudaError_t im_mfield(vec2<T> *out, const vec2<T> *M, const vec2<T> *x, int64_t total, cudaStream_t s)
{
    launch_pdl(k_im_mfield<T>, dim3(im_grid(total)), dim3(256), 0, s, out, M, x, total);
    return cudaGetLastError();
}

template <typename T>
cudaError_t im_prep_be(const vec2<T> *phi, const T *V, double beta, double dt, int scheme, vec2<T> *M, T *Anl,
                       vec2<T> *b, int64_t total, cudaStream_t s)
{
    launch_pdl(k_im_prep_be<T>, dim3(im_grid(total)), dim3(256), 0, s,
               phi, V, beta, 1.0 / dt, dt, scheme, M, Anl, b, total);
    return cudaGetLastError();
}

template <typename T>
cudaError_t im_prep_cn(const vec2<T> *phi, const vec2<T> *phi1, const T *V, double beta, double dt, int scheme,
                       vec2<T> *psim, T *Anl, vec2<T> *Anl2, vec2<T> *M, int64_t total, cudaStream_t s)
{
    launch_pdl(k_im_prep_cn<T>, dim3(im_grid(total)), dim3(256), 0, s,
               phi, phi1, V, beta, 1.0 / dt, scheme, psim, Anl, Anl2, M, total);
    return cudaGetLastError();
}

template <typename T>
cudaError_t im_rhs_cn(const vec2<T> *phi, const vec2<T> *phi1, const vec2<T> *psim, const vec2<T> *lap, const T *V,
                      double beta, double dt, int tsch, vec2<T> *b, int64_t total, cudaStream_t s)
{
    launch_pdl(k_im_rhs_cn<T>, dim3(im_grid(total)), dim3(256), 0, s,
               phi, phi1, psim, lap, V, beta, 1.0 / dt, tsch, b, total);
    return cudaGetLastError();
}

template <typename T>
cudaError_t im_op(const vec2<T> *x, const vec2<T> *lap, int scheme, double dt, const vec2<T> *M, const T *Anl,
                  const vec2<T> *Anl2, const vec2<T> *b, int precond, vec2<T> *out, int64_t total, const vec2<T> *r,
                  const vec2<T> *r2, const KryScratch &k, int what, cudaStream_t s)
{
    launch_pdl(k_im_op<T>, dim3(what == KRY_NONE ? im_grid(total) : dot_grid(total)), dim3(256), 0, s,
               x, lap, scheme, 1.0 / dt, M, Anl, Anl2, b, precond, out, total, r, r2, dot_args(k, what));
    return cudaGetLastError();
}

template <typename T>
cudaError_t im_norm2(const vec2<T> *a, int64_t total, const KryScratch &k, int what, cudaStream_t s)
{
    launch_pdl(k_im_norm2<T>, dim3(dot_grid(total)), dim3(256), 0, s, a, total, dot_args(k, what));
    return cudaGetLastError();
}

template <typename T>
cudaError_t im_axmy(vec2<T> *out, const vec2<T> *x, double alpha, const vec2<T> *y, int64_t total, cudaStream_t s)
{
    launch_pdl(k_im_axmy<T>, dim3(im_grid(total)), dim3(256), 0, s, out, x, alpha, y, total);
    return cudaGetLastError();
}

template <typename T>
cudaError_t im_axmy_k(vec2<T> *out, const vec2<T> *x, const vec2<T> *y, const KrylovDev *K, int64_t total,
                      cudaStream_t s)
{
    launch_pdl(k_im_axmy_k<T>, dim3(im_grid(total)), dim3(256), 0, s, out, x, y, K, total);
    return cudaGetLastError();
}

template <typename T>
cudaError_t im_update_k(vec2<T> *phi, const vec2<T> *p, const vec2<T> *sv, const vec2<T> *As, vec2<T> *r,
                        const vec2<T> *r2, const KryScratch &k, double tol, int nkrylov, int64_t total,
                        cudaStream_t s)
{
    DotArgs d = dot_args(k, KRY_CHECK);
    d.tol = tol;
    d.nkrylov = nkrylov;
    launch_pdl(k_im_update_k<T>, dim3(dot_grid(total)), dim3(256), 0, s, phi, p, sv, As, r, r2,
               (const KrylovDev *)k.K, total, d);
    return cudaGetLastError();
}

template <typename T>
cudaError_t im_pdir_k(vec2<T> *p, const vec2<T> *r, const vec2<T> *Ap, const KrylovDev *K, int64_t total,
                      cudaStream_t s)
{
    launch_pdl(k_im_pdir_k<T>, dim3(im_grid(total)), dim3(256), 0, s, p, r, Ap, K, total);
    return cudaGetLastError();
}

#define GPSS_IM_INST(T)                                                                                             \
    template cudaError_t im_prep_be<T>(const vec2<T> *, const T *, double, double, int, vec2<T> *, T *, vec2<T> *,  \
                                       int64_t, cudaStream_t);                                                      \
    template cudaError_t im_prep_cn<T>(const vec2<T> *, const vec2<T> *, const T *, double, double, int, vec2<T> *, \
                                       T *, vec2<T> *, vec2<T> *, int64_t, cudaStream_t);                           \
    template cudaError_t im_rhs_cn<T>(const vec2<T> *, const vec2<T> *, const vec2<T> *, const vec2<T> *,           \
                                      const T *, double, double, int, vec2<T> *, int64_t, cudaStream_t);            \
    template cudaError_t im_op<T>(const vec2<T> *, const vec2<T> *, int, double, const vec2<T> *, const T *,        \
                                  const vec2<T> *, const vec2<T> *, int, vec2<T> *, int64_t, const vec2<T> *,       \
                                  const vec2<T> *, const KryScratch &, int, cudaStream_t);                          \
    template cudaError_t im_norm2<T>(const vec2<T> *, int64_t, const KryScratch &, int, cudaStream_t);              \
    template cudaError_t im_axmy<T>(vec2<T> *, const vec2<T> *, double, const vec2<T> *, int64_t, cudaStream_t);    \
    template cudaError_t im_axmy_k<T>(vec2<T> *, const vec2<T> *, const vec2<T> *, const KrylovDev *, int64_t,      \
                                      cudaStream_t);                                                                \
    template cudaError_t im_update_k<T>(vec2<T> *, const vec2<T> *, const vec2<T> *, const vec2<T> *, vec2<T> *,    \
                                        const vec2<T> *, const KryScratch &, double, int, int64_t, cudaStream_t);   \
    template cudaError_t im_pdir_k<T>(vec2<T> *, const vec2<T> *, const vec2<T> *, const KrylovDev *, int64_t,      \
                                      cudaStream_t);                                                                \
    template cudaError_t im_mfield<T>(vec2<T> *, const vec2<T> *, const vec2<T> *, int64_t, cudaStream_t);
GPSS_IM_INST(float)
GPSS_IM_INST(double)

}  // namespace gpss

// Instantiations and launch of the generic-length directional passes
// (pass_generic.cuh, FP64; pass_generic32.cuh, FP32).
#include "gpss_internal.h"
#include "pass_generic.cuh"
#include "pass_generic32.cuh"

namespace gpss {

namespace {

// One wave of CTAs at most, with programmatic stream serialization.  The
// shared-memory limit is the kernel's, not the launch's, so it is always set to
// the largest any launch needs (a smaller one, set by another thread between
// this and the launch, would refuse it).
template <typename T, typename P>
cudaError_t gen_launch_kernel(void (*k)(const PassArgs<T>, const P), int threads, size_t smem, int tiles,
                              const PassArgs<T> &a, const P &p, cudaStream_t s)
{
    if (smem > (size_t)GEN_SMEM_MAX) return cudaErrorInvalidConfiguration;
    int dev = 0, nb = 0, nsm = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if ((e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, GEN_SMEM_MAX)) != cudaSuccess)
        return e;
    if ((e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, k, threads, smem)) != cudaSuccess) return e;
    if ((e = cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess) return e;
    if (nb < 1) return cudaErrorInvalidConfiguration;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(tiles < nb * nsm ? tiles : nb * nsm);
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, k, a, p);
}

// cells of a tile of x lines (padded) or columns
size_t gen_slots(int n, int W, bool xl) { return (size_t)W * (size_t)(xl ? n + (n >> 4) + 1 : n); }

template <int MODE, bool MULT = false> cudaError_t gen_launch_f64(const PassArgs<double> &a, const GenPlan &p, cudaStream_t s)
{
    const int W = p.lines();
    const bool phase = MODE == MODE_FUSED && a.prow == 0 && !a.mask_lim;
    const size_t smem = 16 * ((size_t)(phase ? 2 * p.n : p.n) + gen_slots(p.n, W, a.stride == 1));
    return gen_launch_kernel(gen_pass_kernel<MODE, MULT>, GEN_THREADS, smem, (a.nlines + W - 1) / W, a, p, s);
}

template <int MODE> cudaError_t gen_launch_f32(const PassArgs<float> &a, const Gen32Plan &p, cudaStream_t s)
{
    if constexpr (MODE != MODE_DIAG) {
        if (gen32_fast(MODE, a, p)) {
            const int W = 1 << p.lw;
            const bool phase = MODE == MODE_FUSED && a.prow == 0 && !a.mask_lim;
            const size_t smem = 16 * (size_t)(phase ? 2 * p.n : p.n) + 16 * gen_slots(p.n, W, a.stride == 1);
            return gen_launch_kernel(gen32_pass_kernel<MODE>, GEN_THREADS, smem, (a.nlines + W - 1) / W, a, p, s);
        }
    }
    if constexpr (MODE == MODE_FUSED || MODE == MODE_DIAG) {
        const size_t smem = 16 * (size_t)p.W * (size_t)p.n;
        return gen_launch_kernel(gen32_tile_kernel<MODE>, GEN32_TILE_THREADS, smem, (a.nlines + p.W - 1) / p.W, a, p,
                                 s);
    }
    return cudaErrorInvalidValue;
}

}  // namespace

cudaError_t launch_gen_f32(int mode, const PassArgs<float> &a, const Gen32Plan &p, cudaStream_t s)
{
    // none of the merged imaginary-time, adjoint, stacked plane or compensated features
    if (a.nl_pre || a.dot_with || a.pre_out || a.adj_pre || a.plane_nl || a.plane_scale || a.comp)
        return cudaErrorInvalidValue;
    switch (mode) {
    case MODE_FUSED:
        if (!a.phase && !a.mask_lim) return cudaErrorInvalidValue;
        return gen_launch_f32<MODE_FUSED>(a, p, s);
    case MODE_FWD: return gen_launch_f32<MODE_FWD>(a, p, s);
    case MODE_INV: return gen_launch_f32<MODE_INV>(a, p, s);
    case MODE_DIAG: return gen_launch_f32<MODE_DIAG>(a, p, s);
    default: return cudaErrorInvalidValue;
    }
}
cudaError_t launch_gen_f64(int mode, const PassArgs<double> &a, const GenPlan &p, cudaStream_t s)
{
    // none of the adjoint, stacked plane or compensated features
    if (a.pre_out || a.adj_pre || a.plane_nl || a.plane_scale || a.comp) return cudaErrorInvalidValue;
    if ((a.nl_mode != NL_NONE || a.nl_pre) && !a.nl_fx.tab2) return cudaErrorInvalidValue;
    switch (mode) {
    case MODE_FUSED:
        if (!a.phase && !a.mask_lim) return cudaErrorInvalidValue;
        if (a.mult && (a.mask_lim || a.nl_pre)) return cudaErrorInvalidValue;
        if (a.mult) return gen_launch_f64<MODE_FUSED, true>(a, p, s);
        return gen_launch_f64<MODE_FUSED>(a, p, s);
    case MODE_FWD: return gen_launch_f64<MODE_FWD>(a, p, s);
    case MODE_INV: return gen_launch_f64<MODE_INV>(a, p, s);
    case MODE_DIAG: return gen_launch_f64<MODE_DIAG>(a, p, s);
    default: return cudaErrorInvalidValue;
    }
}

}  // namespace gpss

// sfg_tile2d.cuh -- single-grid fused stage kernels for 2-D grids: one launch
// per stage, one block per tile (bodies in sfg_tile.cuh).  The tile shapes are
// instantiated in three translation units (sfg_tile2d.cu, sfg_tile2d_small.cu,
// sfg_tile2d_large.cu).
#pragma once

#include "sfg_tile.cuh"

namespace sfg {

template <int SCHEME, int FLUX, int TX, int TY>
__global__ void __launch_bounds__(TILE_THREADS, 2) tile2d_kernel(GridView g, StageView sv) {
    extern __shared__ __align__(16) double smem[];
    if (sv.require_active && !sv.clock->active) return;
    const int ntx = (g.hi[0] - g.lo[0] + TX - 1) / TX;
    const int x0 = g.lo[0] + (blockIdx.x % ntx) * TX, y0 = g.lo[1] + (blockIdx.x / ntx) * TY;
    unsigned flags = 0, cut = 0, cores = 0;
    double sr = cfl_seen(g, sv);
    tile2d_body<SCHEME, FLUX, TX, TY>(g, sv, x0, y0, smem, flags, cut, cores, sr);
    flush_status(sv, flags, cores, cut);
    if (sv.mode & MODE_CFL) flush_cfl_block(g, sv.clock, sr);
    if (sv.mode & MODE_STEP) step_tail(sv);
}

template <int SCHEME, int FLUX, int TX, int TY>
__global__ void __launch_bounds__(TILE_THREADS, 4) tile2d_f32_kernel(GridView g, StageView sv) {
    extern __shared__ __align__(16) float smemf[];
    if (sv.require_active && !sv.clock->active) return;
    const int ntx = (g.hi[0] - g.lo[0] + TX - 1) / TX;
    const int x0 = g.lo[0] + (blockIdx.x % ntx) * TX, y0 = g.lo[1] + (blockIdx.x / ntx) * TY;
    unsigned flags = 0, cut = 0, cores = 0;
    double sr = cfl_seen(g, sv);
    tile2d_f32_body<SCHEME, FLUX, TX, TY>(g, sv, x0, y0, smemf, flags, cut, cores, sr);
    flush_status(sv, flags, cores, cut);
    if (sv.mode & MODE_CFL) flush_cfl_block(g, sv.clock, sr);
    if (sv.mode & MODE_STEP) step_tail(sv);
}

template <int SCHEME, int FLUX, typename T, int TX, int TY>
static cudaError_t launch_tile(const GridView& g, const StageView& sv, cudaStream_t st) {
    using S = TileShape<SCHEME, TX, TY>;
    constexpr size_t smem = sizeof(T) * S::ELEMS;
    static std::atomic<unsigned long long> configured{0};
    unsigned long long bit = 0;
    const int ntx = (g.hi[0] - g.lo[0] + TX - 1) / TX;
    const int nty = (g.hi[1] - g.lo[1] + TY - 1) / TY;
    auto kern = sizeof(T) == sizeof(float) ? tile2d_f32_kernel<SCHEME, FLUX, TX, TY> : tile2d_kernel<SCHEME, FLUX, TX, TY>;
    if (attributes_pending(configured, bit)) {
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return e;
        configured.fetch_or(bit, std::memory_order_release);
    }
    kern<<<ntx * nty, TILE_THREADS, smem, st>>>(g, sv);
    return cudaGetLastError();
}

template <int FLUX, typename T, int TX, int TY>
static cudaError_t launch_tile_s(int scheme, const GridView& g, const StageView& sv, cudaStream_t st) {
    switch (scheme) {
    case WENO5: return launch_tile<WENO5, FLUX, T, TX, TY>(g, sv, st);
    case TENO5: return launch_tile<TENO5, FLUX, T, TX, TY>(g, sv, st);
    case WENO3: return launch_tile<WENO3, FLUX, T, TX, TY>(g, sv, st);
    case WENO7: return launch_tile<WENO7, FLUX, T, TX, TY>(g, sv, st);
    }
    return cudaErrorInvalidValue;
}

// Rusanov and Roe in both precisions; Steger-Warming, Lax-Friedrichs and
// Lax-Wendroff faces in FP64 (the FP32 deviation form is Rusanov / Roe).
template <typename T, int TX, int TY>
static cudaError_t launch_tile_t(int scheme, int flux, const GridView& g, const StageView& sv, cudaStream_t st) {
    if (flux == RUSANOV) return launch_tile_s<RUSANOV, T, TX, TY>(scheme, g, sv, st);
    if (flux == ROE) return launch_tile_s<ROE, T, TX, TY>(scheme, g, sv, st);
    if constexpr (sizeof(T) == sizeof(double)) {
        if (flux == STEGER) return launch_tile_s<STEGER, T, TX, TY>(scheme, g, sv, st);
        if (flux == LAXF) return launch_tile_s<LAXF, T, TX, TY>(scheme, g, sv, st);
        if (flux == LAXW) return launch_tile_s<LAXW, T, TX, TY>(scheme, g, sv, st);
    }
    return cudaErrorInvalidValue;
}

template <int TX, int TY>
static cudaError_t launch_tile_p(int prec64, int scheme, int flux, const GridView& g, const StageView& sv,
                                 cudaStream_t st) {
    return prec64 ? launch_tile_t<double, TX, TY>(scheme, flux, g, sv, st)
                  : launch_tile_t<float, TX, TY>(scheme, flux, g, sv, st);
}

}  // namespace sfg

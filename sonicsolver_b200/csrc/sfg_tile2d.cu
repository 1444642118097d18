// sfg_tile2d.cu -- the 2-D tile launcher with its middle tiles (32 x 15,
// 22 x 22), and the 1-D tiles.
#include "sfg_tile2d.cuh"

namespace sfg {

cudaError_t launch_tile2d_small(int rounds, int scheme, int flux, int prec64, const GridView& g, const StageView& sv,
                                cudaStream_t st);
cudaError_t launch_tile2d_large(int scheme, int flux, int prec64, const GridView& g, const StageView& sv,
                                cudaStream_t st);

// 1-D grids: one block per T1-node tile (the body the batched kernels use, so a
// 1-D grid gives the same bits alone and in a batch): 511 nodes, two rounds of
// faces, or 255 and one round while the blocks then still fit the GPU at once
// (a stage then lasts as long as one block's rounds).
template <int SCHEME, int FLUX, typename T, int T1>
__global__ void __launch_bounds__(TILE_THREADS) tile1d_kernel(GridView g, StageView sv) {
    extern __shared__ __align__(16) unsigned char smem1[];
    if (sv.require_active && !sv.clock->active) return;
    unsigned flags = 0, cut = 0, cores = 0;
    double sr = cfl_seen(g, sv);
    tile1d_body<SCHEME, FLUX, T, T1>(g, sv, g.lo[0] + blockIdx.x * T1, reinterpret_cast<T*>(smem1), flags, cut,
                                     cores, sr);
    flush_status(sv, flags, cores, cut);
    if (sv.mode & MODE_CFL) flush_cfl_block(g, sv.clock, sr);
    if (sv.mode & MODE_STEP) step_tail(sv);
}

template <int SCHEME, int FLUX, typename T, int T1>
static cudaError_t launch_tile1_n(const GridView& g, const StageView& sv, cudaStream_t st) {
    constexpr size_t smem = sizeof(T) * Tile1Shape<SCHEME, T1>::ELEMS;
    static std::atomic<unsigned long long> configured{0};
    unsigned long long bit = 0;
    auto kern = tile1d_kernel<SCHEME, FLUX, T, T1>;
    if (attributes_pending(configured, bit)) {
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return e;
        configured.fetch_or(bit, std::memory_order_release);
    }
    kern<<<(g.hi[0] - g.lo[0] + T1 - 1) / T1, TILE_THREADS, smem, st>>>(g, sv);
    return cudaGetLastError();
}

template <int SCHEME, int FLUX, typename T>
static cudaError_t launch_tile1(const GridView& g, const StageView& sv, cudaStream_t st) {
    if ((g.hi[0] - g.lo[0] + TILE1D_SHORT - 1) / TILE1D_SHORT <= 2 * 148)
        return launch_tile1_n<SCHEME, FLUX, T, TILE1D_SHORT>(g, sv, st);
    return launch_tile1_n<SCHEME, FLUX, T, TILE1D>(g, sv, st);
}

template <int FLUX, typename T>
static cudaError_t launch_tile1_s(int scheme, const GridView& g, const StageView& sv, cudaStream_t st) {
    switch (scheme) {
    case WENO5: return launch_tile1<WENO5, FLUX, T>(g, sv, st);
    case TENO5: return launch_tile1<TENO5, FLUX, T>(g, sv, st);
    case WENO3: return launch_tile1<WENO3, FLUX, T>(g, sv, st);
    case WENO7: return launch_tile1<WENO7, FLUX, T>(g, sv, st);
    }
    return cudaErrorInvalidValue;
}

template <typename T>
static cudaError_t launch_tile1_t(int scheme, int flux, const GridView& g, const StageView& sv, cudaStream_t st) {
    if (flux == RUSANOV) return launch_tile1_s<RUSANOV, T>(scheme, g, sv, st);
    if (flux == ROE) return launch_tile1_s<ROE, T>(scheme, g, sv, st);
    if constexpr (sizeof(T) == sizeof(double)) {
        if (flux == STEGER) return launch_tile1_s<STEGER, T>(scheme, g, sv, st);
        if (flux == LAXF) return launch_tile1_s<LAXF, T>(scheme, g, sv, st);
        if (flux == LAXW) return launch_tile1_s<LAXW, T>(scheme, g, sv, st);
    }
    return cudaErrorInvalidValue;
}

cudaError_t launch_tile1d(int scheme, int flux, int prec64, const GridView& g, const StageView& sv, cudaStream_t st) {
    return prec64 ? launch_tile1_t<double>(scheme, flux, g, sv, st) : launch_tile1_t<float>(scheme, flux, g, sv, st);
}

// variant 1: 32 x 15 tile, variant 2: 22 x 22 tile (256 threads each, four
// rounds of faces); every shape gives the same bits.  A grid too small to
// fill the GPU with them takes 32 x 7 (two rounds) or 16 x 7 (one round):
// the smallest whose blocks are all resident at once (2 per SM in FP64, 4 in
// FP32), because then a stage lasts as long as one block, and a block as long
// as its rounds.  Measured, us per SSPRK3 step of three launches, 32 x 15 /
// 32 x 7 / 16 x 7: FP64 WENO5 64^2 43 / 31 / 26, 192 x 160 48 / 34 / 30,
// 257 x 193 48 / 42 / 44, 320^2 62 / 64 / 72, 512^2 107 / 114 / 145; FP32
// 64^2 36 / 28 / 24, 257 x 193 42 / 35 / 34, 320^2 48 / 44 / 44, 400^2 59 /
// 56 / 59, 512^2 69 / 71 / 87 (more blocks repeat more halo and edge faces).
// A grid of many rounds of blocks takes 32 x 23 (six rounds of faces): less halo
// and fewer edge faces, once its coarser last round of blocks no longer counts.
// 32 x 15 / 32 x 23: FP64 TENO5 700^2 182 / 184, 768^2 215 / 213, 1024^2 371 /
// 358, 2048^2 1357 / 1287; FP32 WENO5 1024^2 202 / 201, 1600^2 454 / 443, 2048^2
// 721 / 696; FP32 TENO5 1024^2 228 / 234, 2048^2 818 / 813.
cudaError_t launch_tile2d(int variant, int scheme, int flux, int prec64, const GridView& g, const StageView& sv,
                          cudaStream_t st) {
    if (variant < 1 || variant > 2) return cudaErrorInvalidValue;
    const int nx = g.hi[0] - g.lo[0], ny = g.hi[1] - g.lo[1];
    const long long resident = 148LL * (prec64 ? 2 : 4);
    auto blocks = [&](int tx, int ty) { return (long long)((nx + tx - 1) / tx) * ((ny + ty - 1) / ty); };
    if (blocks(16, 7) <= resident) return launch_tile2d_small(1, scheme, flux, prec64, g, sv, st);
    if (blocks(32, 7) <= resident) return launch_tile2d_small(2, scheme, flux, prec64, g, sv, st);
    if (variant == 2) return launch_tile_p<22, 22>(prec64, scheme, flux, g, sv, st);
    if (blocks(32, 15) >= (prec64 ? 4 : 8) * resident) return launch_tile2d_large(scheme, flux, prec64, g, sv, st);
    return launch_tile_p<32, 15>(prec64, scheme, flux, g, sv, st);
}

}  // namespace sfg

// sfg_tile2d_large.cu -- 32 x 23 tiles for large 2-D grids (rule and figures at
// launch_tile2d): 33 x 23 x faces padded to 768, 32 x 24 y faces: six rounds of
// 256; 105 KB of shared memory in FP64 (WENO7 111 KB), two blocks per SM.
#include "sfg_tile2d.cuh"

namespace sfg {

cudaError_t launch_tile2d_large(int scheme, int flux, int prec64, const GridView& g, const StageView& sv,
                                cudaStream_t st) {
    return launch_tile_p<32, 23>(prec64, scheme, flux, g, sv, st);
}

}  // namespace sfg

// sfg_tile2d_small.cu -- 2-D tiles of one and two rounds of faces for grids
// that the full-size tiles leave most SMs without (rule and figures at
// launch_tile2d).
#include "sfg_tile2d.cuh"

namespace sfg {

// rounds 1: 16 x 7 (17 x 7 x faces padded to 128, 16 x 8 y faces: 256),
// rounds 2: 32 x 7 (33 x 7 padded to 256, 32 x 8: 512).
cudaError_t launch_tile2d_small(int rounds, int scheme, int flux, int prec64, const GridView& g, const StageView& sv,
                                cudaStream_t st) {
    if (rounds == 1) return launch_tile_p<16, 7>(prec64, scheme, flux, g, sv, st);
    return launch_tile_p<32, 7>(prec64, scheme, flux, g, sv, st);
}

}  // namespace sfg

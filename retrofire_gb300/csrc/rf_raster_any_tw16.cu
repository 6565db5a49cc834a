// rf_raster_any_tw16.cu — tile rasteriser kernels for 16-pixel-wide tiles, any
// context.
#include "rf_raster.cuh"

namespace rfk {
cudaError_t launch_raster_any_tw16(int kind, RF_RASTER_PARAMS) {
    return launch_raster_for_width<16, false>(kind, RF_RASTER_ARGS);
}
}  // namespace rfk

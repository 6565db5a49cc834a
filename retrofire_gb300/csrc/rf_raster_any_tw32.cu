// rf_raster_any_tw32.cu — tile rasteriser kernels for 32-pixel-wide tiles, any
// context.
#include "rf_raster.cuh"

namespace rfk {
cudaError_t launch_raster_any_tw32(int kind, RF_RASTER_PARAMS) {
    return launch_raster_for_width<32, false>(kind, RF_RASTER_ARGS);
}
}  // namespace rfk

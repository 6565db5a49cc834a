// rf_raster_tw8.cu — tile rasteriser kernels for 8-pixel-wide tiles, default
// context on depth targets.
#include "rf_raster.cuh"

namespace rfk {
cudaError_t launch_raster_tw8(int kind, RF_RASTER_PARAMS) {
    return launch_raster_for_width<8, true>(kind, RF_RASTER_ARGS);
}
}  // namespace rfk

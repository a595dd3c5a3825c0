// Fused correlation kernel, 24x24 windows: the (windows per CTA, threads per CTA)
// variants the autotuner chooses from, and the batch-launch variants.
#include "xcorr_kernel.cuh"

namespace piv {
PIV_SHAPE(24, 24, 8, 96)
PIV_SHAPE(24, 24, 4, 96)
PIV_SHAPE(24, 24, 8, 192)
PIV_SHAPE(24, 24, 2, 64)
PIV_SHAPE_BATCH(24, 24, 8, 96)
PIV_SHAPE_BATCH(24, 24, 4, 96)
}

// Fused correlation kernel, 48x24 windows: the (windows per CTA, threads per CTA)
// variants the autotuner chooses from, and the batch-launch variants.
#include "xcorr_kernel.cuh"

namespace piv {
PIV_SHAPE(48, 24, 4, 96)
PIV_SHAPE(48, 24, 2, 64)
PIV_SHAPE(48, 24, 2, 96)
PIV_SHAPE(48, 24, 8, 192)
PIV_SHAPE_BATCH(48, 24, 4, 96)
PIV_SHAPE_BATCH(48, 24, 2, 64)
}

// Fused correlation kernel, 12x12 windows: the (windows per CTA, threads per CTA)
// variants the autotuner chooses from, and the batch-launch variants.
#include "xcorr_kernel.cuh"

namespace piv {
PIV_SHAPE(12, 12, 16, 96)
PIV_SHAPE(12, 12, 8, 96)
PIV_SHAPE(12, 12, 16, 192)
PIV_SHAPE_BATCH(12, 12, 16, 96)
PIV_SHAPE_BATCH(12, 12, 8, 96)
}

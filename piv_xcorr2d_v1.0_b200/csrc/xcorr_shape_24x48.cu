// Fused correlation kernel, 24x48 windows: the (windows per CTA, threads per CTA)
// variants the autotuner chooses from, and the batch-launch variants.
#include "xcorr_kernel.cuh"

namespace piv {
PIV_SHAPE(24, 48, 4, 96)
PIV_SHAPE(24, 48, 2, 64)
PIV_SHAPE(24, 48, 4, 128)
PIV_SHAPE(24, 48, 8, 192)
PIV_SHAPE_BATCH(24, 48, 4, 96)
PIV_SHAPE_BATCH(24, 48, 2, 64)
}

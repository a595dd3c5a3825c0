// Fused correlation kernel, 64x32 windows: the (windows per CTA, threads per CTA)
// variants the autotuner chooses from, and the batch-launch variants.
#include "xcorr_kernel.cuh"

namespace piv {
PIV_SHAPE(64, 32, 4, 128)
PIV_SHAPE(64, 32, 2, 64)
PIV_SHAPE(64, 32, 2, 128)
PIV_SHAPE_BATCH(64, 32, 4, 128)
PIV_SHAPE_BATCH(64, 32, 2, 64)
}

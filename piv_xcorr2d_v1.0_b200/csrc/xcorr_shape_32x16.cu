// Fused correlation kernel, 32x16 windows: the (windows per CTA, threads per CTA)
// variants the autotuner chooses from, and the batch-launch variants.
#include "xcorr_kernel.cuh"

namespace piv {
PIV_SHAPE(32, 16, 8, 128)
PIV_SHAPE(32, 16, 4, 64)
PIV_SHAPE(32, 16, 8, 256)
PIV_SHAPE_BATCH(32, 16, 8, 128)
PIV_SHAPE_BATCH(32, 16, 4, 64)
}

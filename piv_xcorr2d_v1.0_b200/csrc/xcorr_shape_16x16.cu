// Fused correlation kernel, 16x16 windows: the (windows per CTA, threads per CTA)
// variants the autotuner chooses from, and the batch-launch variants.
#include "xcorr_kernel.cuh"

namespace piv {
PIV_SHAPE(16, 16, 16, 128)
PIV_SHAPE(16, 16, 8, 128)
PIV_SHAPE(16, 16, 16, 256)
PIV_SHAPE(16, 16, 4, 64)
PIV_SHAPE_BATCH(16, 16, 16, 128)
PIV_SHAPE_BATCH(16, 16, 8, 128)
}

// Fused correlation kernel, 32x64 windows: the (windows per CTA, threads per CTA)
// variants the autotuner chooses from, and the batch-launch variants.
#include "xcorr_kernel.cuh"

namespace piv {
PIV_SHAPE(32, 64, 4, 128)
PIV_SHAPE(32, 64, 2, 64)
PIV_SHAPE(32, 64, 2, 128)
PIV_SHAPE_BATCH(32, 64, 4, 128)
PIV_SHAPE_BATCH(32, 64, 2, 64)
}

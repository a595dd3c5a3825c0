// Fused correlation kernel, 8x8 windows: the (windows per CTA, threads per CTA)
// variants the autotuner chooses from, and the batch-launch variants.
#include "xcorr_kernel.cuh"

namespace piv {
PIV_SHAPE(8, 8, 32, 128)
PIV_SHAPE(8, 8, 16, 128)
PIV_SHAPE(8, 8, 32, 256)
PIV_SHAPE_BATCH(8, 8, 32, 128)
PIV_SHAPE_BATCH(8, 8, 16, 128)
}

// Fused correlation kernel, 32x32 windows: the (windows per CTA, threads per CTA)
// variants the autotuner chooses from, and the batch-launch variants.
#include "xcorr_kernel.cuh"

namespace piv {
#if PIV_BATCH
template cudaError_t launch_pair_batch<4, PIV_K>(const XcorrBatch &, bool, cudaStream_t);
#else
template cudaError_t launch_pair<4, PIV_K>(const XcorrArgs &, bool, cudaStream_t);
template cudaError_t launch_shape_block<32, 32, 128, PIV_K>(const XcorrArgs &, bool, cudaStream_t);
#endif
PIV_SHAPE(32, 32, 4, 128)
PIV_SHAPE(32, 32, 2, 64)
PIV_SHAPE(32, 32, 8, 256)
PIV_SHAPE(32, 32, 4, 64)
PIV_SHAPE_BATCH(32, 32, 4, 128)
}

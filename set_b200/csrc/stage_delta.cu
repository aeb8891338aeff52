// stage_delta.cu -- the stage and batch kernels of the delta (FP64 states, FP32 differences) form.
#include "stage.cuh"

namespace sb {
template cudaError_t launch_stage_form<2>(const StageArgs&, int, int, int, cudaStream_t);
template cudaError_t launch_batch_form<2>(const BatchArgs&, int, int, int, cudaStream_t);
template cudaError_t prepare_batch_form<2>();
}  // namespace sb

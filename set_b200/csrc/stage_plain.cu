// stage_plain.cu -- the stage and batch kernels of the plain FP64 form.
#include "stage.cuh"

namespace sb {
template cudaError_t launch_stage_form<0>(const StageArgs&, int, int, int, cudaStream_t);
template cudaError_t launch_batch_form<0>(const BatchArgs&, int, int, int, cudaStream_t);
template cudaError_t prepare_batch_form<0>();
}  // namespace sb

// stage_mixed.cu -- the stage and batch kernels of the mixed (FP32 Riemann arithmetic) form.
#include "stage.cuh"

namespace sb {
template cudaError_t launch_stage_form<1>(const StageArgs&, int, int, int, cudaStream_t);
template cudaError_t launch_batch_form<1>(const BatchArgs&, int, int, int, cudaStream_t);
template cudaError_t prepare_batch_form<1>();
}  // namespace sb

// stage.cu -- launch entry points of the stage and batch kernels (stage.cuh), by form.
#include "setb_internal.cuh"

namespace sb {

cudaError_t launch_stage(const StageArgs& a, int precision, int n_state, int order, int kind, cudaStream_t s) {
    if (precision == 1) return launch_stage_form<1>(a, n_state, order, kind, s);
    if (precision == 2) return launch_stage_form<2>(a, n_state, order, kind, s);
    return launch_stage_form<0>(a, n_state, order, kind, s);
}

cudaError_t launch_batch_stage(const BatchArgs& b, int precision, int n_state, int kind, int grid, cudaStream_t s) {
    if (precision == 1) return launch_batch_form<1>(b, n_state, kind, grid, s);
    if (precision == 2) return launch_batch_form<2>(b, n_state, kind, grid, s);
    return launch_batch_form<0>(b, n_state, kind, grid, s);
}

cudaError_t prepare_batch_kernels(int precision) {
    if (precision == 1) return prepare_batch_form<1>();
    if (precision == 2) return prepare_batch_form<2>();
    return prepare_batch_form<0>();
}

int batch_ctas_per_sm(int precision) { return tile_shape(precision, kBatchShape).ctas_per_sm; }

}  // namespace sb

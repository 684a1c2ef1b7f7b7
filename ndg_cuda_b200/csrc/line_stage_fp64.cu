// The line kernel (line_stage.cuh), default form, and the rule of its use.
#include "line_launch.cuh"

namespace ndg {
namespace dev {

int line_default_tile(int N) { return line_default_elements(N); }

bool line_kernel_runs(int N, bool fp32, int64_t elements) {
    return line_order(N, fp32) && (line_every_size(N) || elements >= kLineMinElements);
}

int line_candidates_fp64(int N, int* out, int max) { return line_candidates<double>(N, out, max); }

cudaError_t prepare_line_fp64(int N, bool seam, int elements) {
    return seam ? prepare_line_seam_fp64(N, elements) : line_prepare<double, false>(N, elements);
}

cudaError_t launch_line_fp64(int N, bool seam, int elements, const StageArgs& a, cudaStream_t stream) {
    return seam ? launch_line_seam_fp64(N, elements, a, stream) : line_launch<double, false>(N, elements, a, stream);
}

cudaError_t launch_line_traces_fp64(int N, const TraceArgs& a, cudaStream_t stream) { return line_traces<double>(N, a, stream); }

}  // namespace dev
}  // namespace ndg

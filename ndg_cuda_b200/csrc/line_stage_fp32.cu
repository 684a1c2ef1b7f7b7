// The line kernel (line_stage.cuh), FP32 form.
#include "line_launch.cuh"

namespace ndg {
namespace dev {

int line_candidates_fp32(int N, int* out, int max) { return line_candidates<float>(N, out, max); }

cudaError_t prepare_line_fp32(int N, bool seam, int elements) {
    return seam ? prepare_line_seam_fp32(N, elements) : line_prepare<float, false>(N, elements);
}

cudaError_t launch_line_fp32(int N, bool seam, int elements, const StageArgs& a, cudaStream_t stream) {
    return seam ? launch_line_seam_fp32(N, elements, a, stream) : line_launch<float, false>(N, elements, a, stream);
}

cudaError_t launch_line_traces_fp32(int N, const TraceArgs& a, cudaStream_t stream) { return line_traces<float>(N, a, stream); }

}  // namespace dev
}  // namespace ndg

// The line kernel, FP32 form, on meshes with a seam whose normals are not opposite.
#include "line_launch.cuh"

namespace ndg {
namespace dev {

cudaError_t prepare_line_seam_fp32(int N, int elements) { return line_prepare<float, true>(N, elements); }

cudaError_t launch_line_seam_fp32(int N, int elements, const StageArgs& a, cudaStream_t stream) { return line_launch<float, true>(N, elements, a, stream); }

}  // namespace dev
}  // namespace ndg

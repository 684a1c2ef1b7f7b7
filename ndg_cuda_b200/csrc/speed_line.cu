// Instantiations and launchers of the line kernel's variable-speed stage
// (line_stage.cuh with SpeedStageArgs), orders 1 to 12, default tiles.
#include "line_stage.cuh"

namespace ndg {
namespace dev {

namespace {

template <int N, typename R>
constexpr bool usable() {
    return line_order(N, sizeof(R) == 4);
}

template <int N, typename R>
cudaError_t prepare(bool seam) {
    if constexpr (usable<N, R>()) {
        constexpr int E = line_default_elements(N);
        return cudaFuncSetAttribute(seam ? line_stage_kernel<N, R, E, SpeedStageArgs, true> : line_stage_kernel<N, R, E, SpeedStageArgs, false>,
                                    cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(LineTile<N, R, E>::kBytes));
    } else {
        return cudaErrorInvalidValue;
    }
}

template <int N, typename R>
cudaError_t launch(bool seam, const SpeedStageArgs& a, cudaStream_t stream) {
    if constexpr (usable<N, R>()) {
        constexpr int E = line_default_elements(N);
        using T = LineTile<N, R, E>;
        return launch_dependent(seam ? line_stage_kernel<N, R, E, SpeedStageArgs, true> : line_stage_kernel<N, R, E, SpeedStageArgs, false>,
                                dim3(static_cast<unsigned>((a.n_elements + E - 1) / E)), T::kThreads, T::kBytes, stream, a, make_line_coeffs<N, R>());
    } else {
        return cudaErrorInvalidValue;
    }
}

}  // namespace

#define NDG_SPEED_LINE_DISPATCH(FN, ...)                                                \
    switch (N) {                                                                        \
        case 1: return fp32 ? FN<1, float>(__VA_ARGS__) : FN<1, double>(__VA_ARGS__);   \
        case 2: return fp32 ? FN<2, float>(__VA_ARGS__) : FN<2, double>(__VA_ARGS__);   \
        case 3: return fp32 ? FN<3, float>(__VA_ARGS__) : FN<3, double>(__VA_ARGS__);   \
        case 4: return fp32 ? FN<4, float>(__VA_ARGS__) : FN<4, double>(__VA_ARGS__);   \
        case 5: return fp32 ? FN<5, float>(__VA_ARGS__) : FN<5, double>(__VA_ARGS__);   \
        case 6: return fp32 ? FN<6, float>(__VA_ARGS__) : FN<6, double>(__VA_ARGS__);   \
        case 7: return fp32 ? FN<7, float>(__VA_ARGS__) : FN<7, double>(__VA_ARGS__);   \
        case 8: return fp32 ? FN<8, float>(__VA_ARGS__) : FN<8, double>(__VA_ARGS__);   \
        case 9: return fp32 ? FN<9, float>(__VA_ARGS__) : FN<9, double>(__VA_ARGS__);   \
        case 10: return fp32 ? FN<10, float>(__VA_ARGS__) : FN<10, double>(__VA_ARGS__); \
        case 11: return fp32 ? FN<11, float>(__VA_ARGS__) : FN<11, double>(__VA_ARGS__); \
        case 12: return fp32 ? FN<12, float>(__VA_ARGS__) : FN<12, double>(__VA_ARGS__); \
        default: return cudaErrorInvalidValue;                                          \
    }

cudaError_t prepare_speed_line(int N, bool fp32, bool seam) { NDG_SPEED_LINE_DISPATCH(prepare, seam) }

cudaError_t launch_speed_line(int N, bool fp32, bool seam, const SpeedStageArgs& a, cudaStream_t stream) {
    NDG_SPEED_LINE_DISPATCH(launch, seam, a, stream)
}

}  // namespace dev
}  // namespace ndg

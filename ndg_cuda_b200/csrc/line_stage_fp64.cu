// Instantiations and launchers of the line kernel (line_stage.cuh), default form:
// tiles of 2, 4, 8 and 16 elements for the orders it runs (line_order).
#include "line_stage.cuh"

#include <algorithm>

namespace ndg {
namespace dev {

namespace {

using R = double;
constexpr bool kF32 = false;

template <int N, int E>
constexpr bool usable() {
    if constexpr (line_order(N, kF32)) return LineTile<N, R, E>::feasible;
    return false;
}

template <int N, int E>
cudaError_t prepare() {
    if constexpr (usable<N, E>())
        return cudaFuncSetAttribute(line_stage_kernel<N, R, E, StageArgs>, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(LineTile<N, R, E>::kBytes));
    else
        return cudaErrorInvalidValue;
}

template <int N, int E>
cudaError_t launch(const StageArgs& a, cudaStream_t stream) {
    if constexpr (usable<N, E>()) {
        using T = LineTile<N, R, E>;
        const dim3 grid(static_cast<unsigned>((a.n_elements + E - 1) / E), static_cast<unsigned>(a.n_instances));
        return launch_dependent(line_stage_kernel<N, R, E, StageArgs>, grid, T::kThreads, T::kBytes, stream, a, make_line_coeffs<N, R>());
    } else {
        return cudaErrorInvalidValue;
    }
}

template <int N>
cudaError_t traces(const TraceArgs& a, cudaStream_t stream) {
    if constexpr (line_order(N, kF32)) {
        const int64_t total = static_cast<int64_t>(a.n_instances) * a.n_elements * 4 * (N + 1);
        const int blocks = static_cast<int>(std::min<int64_t>((total + 255) / 256, 148 * 32));
        line_trace_kernel<N, R><<<blocks, 256, 0, stream>>>(a, make_line_coeffs<N, R>());
        return cudaGetLastError();
    } else {
        return cudaErrorInvalidValue;
    }
}

template <int N>
int candidates(int* out, int max) {
    const bool ok[] = {usable<N, 2>(), usable<N, 4>(), usable<N, 8>(), usable<N, 16>()};
    int count = 0;
    for (int i = 0; i < 4; ++i)
        if (ok[i] && count < max) out[count++] = 2 << i;
    return count;
}

#define NDG_LINE_TILES(FN, N_, ...)                 \
    switch (elements) {                              \
        case 2: return FN<N_, 2>(__VA_ARGS__);       \
        case 4: return FN<N_, 4>(__VA_ARGS__);       \
        case 8: return FN<N_, 8>(__VA_ARGS__);       \
        case 16: return FN<N_, 16>(__VA_ARGS__);     \
        default: return cudaErrorInvalidValue;       \
    }
#define NDG_LINE_ORDERS(CALL) \
    switch (N) {               \
        case 1: CALL(1);       \
        case 2: CALL(2);       \
        case 3: CALL(3);       \
        case 4: CALL(4);       \
        case 5: CALL(5);       \
        case 6: CALL(6);       \
        case 7: CALL(7);       \
        case 8: CALL(8);       \
        case 9: CALL(9);       \
        case 10: CALL(10);     \
        case 11: CALL(11);     \
        case 12: CALL(12);     \
        case 13: CALL(13);     \
        case 14: CALL(14);     \
        default: break;        \
    }

}  // namespace

int line_default_tile(int N) { return line_default_elements(N); }

bool line_kernel_runs(int N, bool fp32, int64_t elements) {
    return line_order(N, fp32) && (line_every_size(N) || elements >= kLineMinElements);
}

int line_candidates_fp64(int N, int* out, int max) {
#define NDG_CALL(n) return candidates<n>(out, max)
    NDG_LINE_ORDERS(NDG_CALL)
#undef NDG_CALL
    return 0;
}

cudaError_t prepare_line_fp64(int N, int elements) {
    if (elements == 0) elements = line_default_elements(N);
#define NDG_CALL(n) NDG_LINE_TILES(prepare, n)
    NDG_LINE_ORDERS(NDG_CALL)
#undef NDG_CALL
    return cudaErrorInvalidValue;
}

cudaError_t launch_line_fp64(int N, int elements, const StageArgs& a, cudaStream_t stream) {
    if (elements == 0) elements = line_default_elements(N);
#define NDG_CALL(n) NDG_LINE_TILES(launch, n, a, stream)
    NDG_LINE_ORDERS(NDG_CALL)
#undef NDG_CALL
    return cudaErrorInvalidValue;
}

cudaError_t launch_line_traces_fp64(int N, const TraceArgs& a, cudaStream_t stream) {
#define NDG_CALL(n) return traces<n>(a, stream)
    NDG_LINE_ORDERS(NDG_CALL)
#undef NDG_CALL
    return cudaErrorInvalidValue;
}

}  // namespace dev
}  // namespace ndg

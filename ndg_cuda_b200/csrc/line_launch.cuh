// Launchers of the line kernel (line_stage.cuh) over orders and tiles, for one
// form R and mesh kind Seam; instantiated by line_stage_fp64.cu and _fp32.cu
// (Seam false) and line_seam_fp64.cu and _fp32.cu (Seam true).
#pragma once

#include "line_stage.cuh"

namespace ndg {
namespace dev {

template <typename R, int N, int E>
constexpr bool line_usable() {
    if constexpr (line_order(N, sizeof(R) == 4)) return LineTile<N, R, E>::feasible;
    return false;
}

template <typename R, bool Seam, int N, int E>
cudaError_t line_prepare_tile() {
    if constexpr (line_usable<R, N, E>())
        return cudaFuncSetAttribute(line_stage_kernel<N, R, E, StageArgs, Seam>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    static_cast<int>(LineTile<N, R, E>::kBytes));
    else
        return cudaErrorInvalidValue;
}

template <typename R, bool Seam, int N, int E>
cudaError_t line_launch_tile(const StageArgs& a, cudaStream_t stream) {
    if constexpr (line_usable<R, N, E>()) {
        using T = LineTile<N, R, E>;
        const dim3 grid(static_cast<unsigned>((a.n_elements + E - 1) / E), static_cast<unsigned>(a.n_instances));
        return launch_dependent(line_stage_kernel<N, R, E, StageArgs, Seam>, grid, T::kThreads, T::kBytes, stream, a, make_line_coeffs<N, R>());
    } else {
        return cudaErrorInvalidValue;
    }
}

template <typename R, int N>
int line_tiles(int* out, int max) {
    const bool ok[] = {line_usable<R, N, 2>(), line_usable<R, N, 4>(), line_usable<R, N, 8>(), line_usable<R, N, 16>()};
    int count = 0;
    for (int i = 0; i < 4; ++i)
        if (ok[i] && count < max) out[count++] = 2 << i;
    return count;
}

#define NDG_LINE_TILES(FN, R_, SEAM_, N_, ...)             \
    switch (elements) {                                     \
        case 2: return FN<R_, SEAM_, N_, 2>(__VA_ARGS__);   \
        case 4: return FN<R_, SEAM_, N_, 4>(__VA_ARGS__);   \
        case 8: return FN<R_, SEAM_, N_, 8>(__VA_ARGS__);   \
        case 16: return FN<R_, SEAM_, N_, 16>(__VA_ARGS__); \
        default: return cudaErrorInvalidValue;              \
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

template <typename R, bool Seam>
cudaError_t line_prepare(int N, int elements) {
    if (elements == 0) elements = line_default_elements(N);
#define NDG_CALL(n) NDG_LINE_TILES(line_prepare_tile, R, Seam, n)
    NDG_LINE_ORDERS(NDG_CALL)
#undef NDG_CALL
    return cudaErrorInvalidValue;
}

template <typename R, bool Seam>
cudaError_t line_launch(int N, int elements, const StageArgs& a, cudaStream_t stream) {
    if (elements == 0) elements = line_default_elements(N);
#define NDG_CALL(n) NDG_LINE_TILES(line_launch_tile, R, Seam, n, a, stream)
    NDG_LINE_ORDERS(NDG_CALL)
#undef NDG_CALL
    return cudaErrorInvalidValue;
}

template <typename R>
int line_candidates(int N, int* out, int max) {
#define NDG_CALL(n) return line_tiles<R, n>(out, max)
    NDG_LINE_ORDERS(NDG_CALL)
#undef NDG_CALL
    return 0;
}

template <typename R, int N>
cudaError_t line_traces_order(const TraceArgs& a, cudaStream_t stream) {
    if constexpr (line_order(N, sizeof(R) == 4)) {
        const int64_t total = static_cast<int64_t>(a.n_instances) * a.n_elements * 4 * (N + 1);
        const int64_t blocks = (total + 255) / 256, most = 148 * 32;
        line_trace_kernel<N, R><<<static_cast<unsigned>(blocks < most ? blocks : most), 256, 0, stream>>>(a, make_line_coeffs<N, R>());
        return cudaGetLastError();
    } else {
        return cudaErrorInvalidValue;
    }
}

template <typename R>
cudaError_t line_traces(int N, const TraceArgs& a, cudaStream_t stream) {
#define NDG_CALL(n) return line_traces_order<R, n>(a, stream)
    NDG_LINE_ORDERS(NDG_CALL)
#undef NDG_CALL
    return cudaErrorInvalidValue;
}

}  // namespace dev
}  // namespace ndg

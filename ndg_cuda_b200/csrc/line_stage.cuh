// The uniform-order stage with one thread per (line, element), for all three
// fields: one low-storage RK3 stage per launch, as stage_kernel
// (stage_templates.cuh), for the default and the FP32 form.
//
// What it changes against one thread per (field, line, element):
//  - A line thread holds the lines of p, u and v, so their traces, the face
//    flux and the flux lines stay in its registers, and every coefficient of
//    the contraction serves three fields. A stage takes two passes over
//    shared memory: columns (xi: k <- a k + G_xi), then rows (eta: k <- k +
//    G_eta, q <- q + g dt k), then the column traces of the new q. N = 8,
//    256 x 256, FP64: 39.1 M warp instructions instead of 94.7 M and 13.8 M
//    shared wavefronts instead of 25.5 M per launch.
//  - The face flux reads the far side only through its outgoing
//    characteristic w = p - (u, v) . n (n this side's outward normal), so sides
//    exchange that one value per node instead of p, u and v: a third of the
//    trace traffic and of the scattered stores. The sender takes its own normal
//    for the opposite of n, or on a seam where it is not n itself (kSeamNormal).
//    Far slots are [instance][element][side][node].
//  - q and k arrive in shared memory together, ahead of the passes. With 16
//    elements a tile and N + 1 odd the tile needs no padding (below): one bulk
//    copy per field in, one out, issued by one thread.
//
// Bank conflicts: threads are ordered (line, element) with the element
// fastest. A wavefront of 8-byte values covers 16 threads, which with 16
// elements are one line of 16 elements: conflict-free in both sweeps at any
// odd element stride. (N + 1)^2 is odd for even N; otherwise one value of
// padding per element is needed, which rules the bulk copies out. Tiles of
// fewer elements take bank::search's strides.
//
// Measured, us per launch by events (second and third stages, the best tile of
// each kernel; FP64 / FP32 form), in parentheses the three-threads-a-line
// kernel:
//   N = 2, 256^2:  18.9 /  16.8 (45.3 / 45.4)     N = 8,  256^2: 101.4 / 102.0 (151.1 / 130.2)
//   N = 4, 256^2:  36.3 /  33.9 (63.9 / 57.3)     N = 9,  192^2:  96.5 / 106.7 (117.1 /  97.6)
//   N = 5, 256^2:  59.7 /  59.9 (93.2 / 84.3)     N = 10, 192^2:  93.6 /  95.6 (131.5 / 115.0)
//   N = 6, 256^2:  65.1 /  63.6 (104.9 / 92.4)    N = 11, 192^2: 129.8 / 156.7 (156.1 / 133.5)
//   N = 7, 256^2:  94.6 / 108.7 (123.3 / 98.6)    N = 12, 160^2: 116.2 / 126.2 (124.6 / 106.8)
// In a run the launches overlap: N = 8 94.0 / 97.6 us a stage, N = 7 89.6, N = 5
// 52.3 / 52.7, N = 2 14.1 / 12.0. N = 8 moves 502 MB a launch (part of its traces
// stays in L2), 77 us at the 6541 GB/s copy rate; what is left is latency: 3 tiles
// (15 warps) an SM, held there by shared memory (q and k) and registers alike.
// Figures below that compare variants of the kernel are theirs, from before the
// launches overlapped.
#pragma once

#include "adjoint.cuh"
#include "ndg_internal.hpp"
#include "stage_common.cuh"
#include "stage_kernels.cuh"

#include <cuda_runtime.h>

#include <climits>
#include <cstdint>
#include <type_traits>

namespace ndg {
namespace dev {

// Where the line kernel runs (line_order) and its default elements a tile.
// FP64 up to N = 14: from N = 15 a line's registers (3 (N + 1) values and
// the accumulators) and the tile leave 6 warps an SM and it loses (N = 15
// even, N = 16 167.8 against 139.8 us). FP32 form: q and k stay FP64 in
// shared memory, so it pays only where the tile is contiguous or small: N <= 6,
// N = 8 and N = 10. At N = 7 (256^2) and 9 (192^2) a run takes 95.9 against 92.7
// and 101.4 against 93.1 us a stage, at N = 11 and 12 142 against 127 and 129
// against 99.
constexpr bool line_order(int N, bool fp32) { return fp32 ? (N <= 6 || N == 8 || N == 10) : N <= 14; }
// On a mesh whose tiles all run at once a stage takes one thread's chain of
// passes, a third as long with three threads a line. Up to N = 4 the line
// kernel is ahead or within 4% at every size (64 elements: N = 1 3.1 / 4.3, N = 3
// 3.3 / 3.3, N = 4 3.6 / 3.7, FP32 N = 4 3.9 / 4.2 us per stage of a run, line /
// three threads a line); above, from kLineMinElements elements (times the
// instances). us per stage of a run at 1,024, 1,600 and 2,304 elements: FP64 N =
// 5 4.6 / 4.4, 4.7 / 5.1 and 5.0 / 5.5, N = 6 4.7 / 4.9, 4.9 / 5.5 and 5.3 / 6.0,
// N = 8 6.1 / 5.3, 6.2 / 6.2 and 6.8 / 7.4, N = 10 7.4 / 7.0, 7.4 / 8.5 and 8.0 /
// 10.2, N = 14 10.6 / 9.1, 12.0 / 11.7 and 12.5 / 15.9; FP32 N = 6 5.1 / 5.1, 5.3
// / 5.5 and 5.9 / 5.9, N = 10 7.9 / 6.8, 7.9 / 7.6 and 8.3 / 9.0. Two orders cross
// later than the rule, at about 4,096: FP64 N = 7 (5.7 / 4.9, 6.5 / 5.5 and 7.1 /
// 6.3; 4,096 8.8 / 8.7) and FP32 N = 8 (6.5 / 5.4, 6.6 / 6.0 and 7.7 / 6.8; 4,096
// 9.8 / 9.1).
constexpr bool line_every_size(int N) { return N <= 4; }
constexpr int64_t kLineMinElements = 1536;
// 16 elements up to N = 10 (8 as fast at N = 9, 4% faster at N = 7 with a launch
// on its own, 94.6 us against 98.6; slower elsewhere: N = 8 130.4 against 101.4;
// 32 slower: 145). Above, a tile of 16 is alone on its SM: 8 for even N (N =
// 12: 116.2 us, 4: 130.1, 16: 125.4), 4 for odd (N = 11: 129.8, 8: 152.3, 16: 177.8).
constexpr int line_default_elements(int N) { return N <= 10 ? 16 : (N % 2 ? 4 : 8); }

// From this order the line contraction is even-odd (dhat_even_odd): N = 8,
// 106 multiply-adds and additions a line instead of 162 with the lift. Below,
// the plain product: the launch is bound by memory either way, and the halves
// of small Dhat tables lie further from the given tables than a plain
// product's rounding (16 x 16, N = 4, 200 steps: relative L2 error against 64-
// bit tables 4.7e-15 even-odd, 2.6e-15 plain).
constexpr int kLineEvenOddMinOrder = 7;

// Coefficients of order N: nodes, Lagrange end values and the contraction's:
// the even-odd halves of Dhat and of the lift weights l(+-1)/w (hs + ha at +1
// and hs - ha at -1: the nodes are symmetric, so l(-1)[i] = l(+1)[N - i]), or
// Dhat and the lift weights themselves.
template <int N, typename R>
struct LineCoeffs {
    static constexpr int n = N + 1, H = n / 2, HO = n - n / 2;
    static constexpr bool kEvenOdd = N >= kLineEvenOddMinOrder;
    R ea[kEvenOdd ? H * HO : 1], so[kEvenOdd ? HO * H : 1];
    R hs[kEvenOdd ? HO : 1], ha[kEvenOdd ? HO : 1];
    R dhat[kEvenOdd ? 1 : n * n], lpw[kEvenOdd ? 1 : n], lmw[kEvenOdd ? 1 : n];
    R xn[n], lm[n], lp[n], iw[n];
    // The order in which line_contract hands out the nodes of a line.
    __device__ static constexpr int out_node(int i) { return kEvenOdd ? ((i & 1) ? N - (i >> 1) : (i >> 1)) : i; }
};

template <int N, typename R>
LineCoeffs<N, R> make_line_coeffs() {
    constexpr int n = N + 1;
    double dh[n * n], xn[n], lm[n], lp[n], w[n], iw[n];
    host_coefficients(N, dh, xn, lm, lp, w, iw);
    LineCoeffs<N, R> c{};
    for (int i = 0; i < n; ++i) {
        c.xn[i] = static_cast<R>(xn[i]);
        c.lm[i] = static_cast<R>(lm[i]);
        c.lp[i] = static_cast<R>(lp[i]);
        c.iw[i] = static_cast<R>(iw[i]);
    }
    if constexpr (LineCoeffs<N, R>::kEvenOdd) {
        even_odd_halves(n, dh, c.ea, c.so);
        for (int i = 0; i < c.HO; ++i) {
            c.hs[i] = static_cast<R>(0.5 * (lp[i] + lm[i]) * iw[i]);
            c.ha[i] = static_cast<R>(0.5 * (lp[i] - lm[i]) * iw[i]);
        }
    } else {
        for (int i = 0; i < n * n; ++i) c.dhat[i] = static_cast<R>(dh[i]);
        for (int i = 0; i < n; ++i) {
            c.lpw[i] = static_cast<R>(lp[i] * iw[i]);
            c.lmw[i] = static_cast<R>(lm[i] * iw[i]);
        }
    }
    return c;
}

template <int N, typename R, int E>
struct LineTile {
    static constexpr int n = N + 1, NN = n * n;
    static constexpr int kThreads = (n * E + 31) / 32 * 32;
    static constexpr int kWarps = kThreads / 32;
    static constexpr bank::Strides L = bank::search(N, E < 16 ? E : 2, 16);
    static constexpr int P = E >= 16 ? n : L.P;
    static constexpr int ES = E >= 16 ? NN | 1 : L.ES;
    static constexpr bool kBulk = E >= 16 && ES == NN;  // the tile is one contiguous range per field
    __device__ static __forceinline__ int node(int nd) {
        if constexpr (P == n) {
            return nd;
        } else {
            const int i = nd / n;
            return i * P + (nd - i * n);
        }
    }
    // Offset within a field of value i = el NN + nd of the tile's elements.
    __device__ static __forceinline__ int place(int i) {
        const int el = i / NN;
        if constexpr (P == n) return i + el * (ES - NN);
        else return el * ES + node(i - el * NN);
    }
    static constexpr int QS = E * ES;
    static constexpr int SE = (4 * n) | 1;
    static constexpr int kQ = 0, kK = 3 * QS, kDoubles = 6 * QS;  // [3][QS] q, [3][QS] k (an even count: the barrier stays 16-byte aligned)
    static constexpr int kFar = 0, kSide = (E * SE + 1) / 2 * 2, kRs = (kSide + 5 * 4 * E + 3) / 4 * 4;
    static constexpr size_t kBytes = sizeof(double) * kDoubles + 16 + sizeof(R) * kRs + sizeof(int) * 4 * E;
    // Tiles per SM: what shared memory holds, less 24 KB of L1 where the tile
    // arrives by cp.async through it (N = 7: 94.6 us with 3 tiles, 100.9 with
    // 4 and no L1 left), within a register budget a line of the order needs
    // without spills (N <= 4: 96, N = 4 34.8 us against 38.9 at 128).
    static constexpr int kRegs = N <= 4 ? 96 : 128;
    static constexpr int kFit = static_cast<int>((232448 - (kBulk ? 0 : 24 * 1024)) / (kBytes + 1024));
    static constexpr int kByRegs = 65536 / (kThreads * kRegs);
    static constexpr int kMinBlocks = kFit < 1 || kByRegs < 1 ? 1 : (kFit < kByRegs ? kFit : kByRegs);
    static constexpr bool feasible = kThreads <= 512 && kBytes <= 226 * 1024;
};

// 1 / x by Newton's iteration r <- r + r (1 - x r) from the hardware's
// approximation (relative error 2^-20, squared by each step: below 2^-79 before
// the last rounding, so it is the rounded reciprocal but for arguments whose
// reciprocal lies that close to a rounding boundary, as that of (2 - 2^-52) 2^k,
// which comes out one unit off; tests/cpp/line_rcp.cu). No special cases: the
// line kernels run on meshes whose Jacobians and reciprocals are normal numbers
// (jacobians_regular). __drcp_rn in its place takes 1 to 8% longer a launch (N =
// 6, 256 x 256 58.0 -> 60.9 us, N = 8 93.7 -> 96.8).
__device__ __forceinline__ double line_rcp(double x) {
    double r;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(x));
    r = fma(r, fma(-x, r, 1.0), r);
    r = fma(r, fma(-x, r, 1.0), r);
    return r;
}
__device__ __forceinline__ float line_rcp(float x) { return __frcp_rn(x); }

// ((1 - t) d0 + (1 + t) d1) / 4 as a + b t.
template <typename R>
struct MLine {
    R a, b;
    __device__ __forceinline__ MLine(R d0, R d1) : a(R(0.25) * (d0 + d1)), b(R(0.25) * (d1 - d0)) {}
    __device__ __forceinline__ R operator()(R t) const { return fma(t, b, a); }
};

// A side's entry in a tile's table of neighbours: the neighbour's side (element
// 4 + side, below 2^31 - 16), or ~kind on a boundary. Seam (meshes that have a
// seam whose two normals are not opposite, kSeamNormal): with the sign bit set
// on those sides. Their far normal is read where it is used, by instantiations
// of their own: in one kernel for all meshes a launch took 1 to 2% longer (N = 8,
// 40 x 40 6.1 -> 6.8 us), and with every side's in the tile 1 to 7% (N = 8, 256 x
// 256 93.8 -> 94.9 us, N = 12, 160 x 160 108 -> 115).
template <bool Seam>
__device__ __forceinline__ int side_entry(int2 lk) {
    const int kind = (lk.y >> 2) & 7;
    if (kind != kInterior) return ~kind;
    const int far = lk.x * 4 + (lk.y & 3);
    return Seam && (lk.y & kSeamNormal) ? far | INT_MIN : far;
}
template <bool Seam>
__device__ __forceinline__ bool side_interior(int entry) {
    return Seam ? static_cast<unsigned>(entry) < 0xfffffff0u : entry >= 0;
}
template <bool Seam>
__device__ __forceinline__ int64_t side_far(int entry) {
    return Seam ? entry & INT_MAX : entry;
}
// Minus the outward normal of the neighbour's side.
__device__ __forceinline__ double2 far_inward(int64_t far, const double2* normal, const int2* link) {
    const double2 nv = normal[far];
    return ((link[far].y >> 5) & 1) ? nv : double2{-nv.x, -nv.y};
}

// The outgoing characteristic p + (u, v) . n, with fixed rounding: the stage
// and the trace kernel must agree on it bit for bit.
template <typename R>
__device__ __forceinline__ R characteristic(R p, R u, R v, R nx, R ny) {
    return p + fma(v, ny, u * nx);
}

__device__ __forceinline__ void bulk_store(void* dst, const void* src, uint32_t bytes) {
    asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(dst), "r"(smem_addr(src)), "r"(bytes) : "memory");
}

// Dhat times the three fields' lines with the lift of the end fluxes fp (at
// +1) and fm (at -1): out(f, i, y) takes y = (Dhat x_f)_i + fp_f l(+1)_i / w_i
// + fm_f l(-1)_i / w_i, the nodes in the order of out_node. Every coefficient
// serves the three fields. The lift comes last: the larger term would
// otherwise round every partial sum of the product (FP32 form).
template <int N, typename R, typename Out>
__device__ __forceinline__ void line_contract(const LineCoeffs<N, R>& cf, const R (&x)[3][N + 1], const R (&fp)[3], const R (&fm)[3], Out&& out) {
    constexpr int n = N + 1, H = n / 2, HO = n - H;
    // FP32 form: l(+-1) and 1/w as factors of their own. The traces weigh the
    // nodes by the same l, so the rounded operator keeps its summation by
    // parts; with rounded products l/w it drifts (periodic 48 x 48, N = 5, 200
    // steps: 1.8e-7 relative L2 instead of 1.3e-7).
    constexpr bool kSplitLift = sizeof(R) == 4;
    const auto lifted = [&](int f, int i, R y) { return fma(fma(fm[f], cf.lm[i], fp[f] * cf.lp[i]), cf.iw[i], y); };
    if constexpr (LineCoeffs<N, R>::kEvenOdd) {
        constexpr int C = HO < 5 ? HO : 5;
        R e[3][HO], o[3][H], s[3], d[3];
#pragma unroll
        for (int f = 0; f < 3; ++f) {
#pragma unroll
            for (int j = 0; j < H; ++j) {
                e[f][j] = x[f][j] + x[f][n - 1 - j];
                o[f][j] = x[f][j] - x[f][n - 1 - j];
            }
            if constexpr (HO > H) e[f][H] = x[f][H];
            s[f] = fp[f] + fm[f];
            d[f] = fp[f] - fm[f];
        }
#pragma unroll
        for (int i0 = 0; i0 < HO; i0 += C) {
            R A[3][C], S[3][C];
#pragma unroll
            for (int c = 0; c < C; ++c)
#pragma unroll
                for (int f = 0; f < 3; ++f) {
                    if (i0 + c < H) A[f][c] = cf.ea[(i0 + c) * HO] * e[f][0];
                    if (i0 + c < HO) S[f][c] = cf.so[(i0 + c) * H] * o[f][0];
                }
#pragma unroll
            for (int j = 1; j < HO; ++j)
#pragma unroll
                for (int c = 0; c < C; ++c)
#pragma unroll
                    for (int f = 0; f < 3; ++f) {
                        if (i0 + c < H) A[f][c] = fma(cf.ea[(i0 + c) * HO + j], e[f][j], A[f][c]);
                        if (i0 + c < HO && j < H) S[f][c] = fma(cf.so[(i0 + c) * H + j], o[f][j], S[f][c]);
                    }
#pragma unroll
            for (int c = 0; c < C; ++c)
#pragma unroll
                for (int f = 0; f < 3; ++f) {
                    const int i = i0 + c;
                    if constexpr (kSplitLift) {
                        if (i < H) {
                            out(f, i, lifted(f, i, S[f][c] + A[f][c]));
                            out(f, n - 1 - i, lifted(f, n - 1 - i, S[f][c] - A[f][c]));
                        } else if (i < HO) {
                            out(f, i, lifted(f, i, S[f][c]));
                        }
                    } else {
                        if (i < H) A[f][c] = fma(cf.ha[i], d[f], A[f][c]);
                        if (i < HO) S[f][c] = fma(cf.hs[i], s[f], S[f][c]);
                        if (i < H) {
                            out(f, i, S[f][c] + A[f][c]);
                            out(f, n - 1 - i, S[f][c] - A[f][c]);
                        } else if (i < HO) {
                            out(f, i, S[f][c]);
                        }
                    }
                }
        }
    } else {
        R A[3][n];
#pragma unroll
        for (int j = 0; j < n; ++j)
#pragma unroll
            for (int i = 0; i < n; ++i)
#pragma unroll
                for (int f = 0; f < 3; ++f) A[f][i] = j == 0 ? cf.dhat[i * n] * x[f][0] : fma(cf.dhat[i * n + j], x[f][j], A[f][i]);
#pragma unroll
        for (int i = 0; i < n; ++i)
#pragma unroll
            for (int f = 0; f < 3; ++f) out(f, i, kSplitLift ? lifted(f, i, A[f][i]) : fma(fm[f], cf.lmw[i], fma(fp[f], cf.lpw[i], A[f][i])));
    }
}

// The same product without a lift.
template <int N, typename R, typename Out>
__device__ __forceinline__ void line_product(const LineCoeffs<N, R>& cf, const R (&x)[3][N + 1], Out&& out) {
    constexpr int n = N + 1, H = n / 2, HO = n - H;
    if constexpr (LineCoeffs<N, R>::kEvenOdd) {
        constexpr int C = HO < 5 ? HO : 5;
        R e[3][HO], o[3][H];
#pragma unroll
        for (int f = 0; f < 3; ++f) {
#pragma unroll
            for (int j = 0; j < H; ++j) {
                e[f][j] = x[f][j] + x[f][n - 1 - j];
                o[f][j] = x[f][j] - x[f][n - 1 - j];
            }
            if constexpr (HO > H) e[f][H] = x[f][H];
        }
#pragma unroll
        for (int i0 = 0; i0 < HO; i0 += C) {
            R A[3][C], S[3][C];
#pragma unroll
            for (int j = 0; j < HO; ++j)
#pragma unroll
                for (int c = 0; c < C; ++c)
#pragma unroll
                    for (int f = 0; f < 3; ++f) {
                        if (i0 + c < H) A[f][c] = j == 0 ? cf.ea[(i0 + c) * HO] * e[f][0] : fma(cf.ea[(i0 + c) * HO + j], e[f][j], A[f][c]);
                        if (i0 + c < HO && j < H) S[f][c] = j == 0 ? cf.so[(i0 + c) * H] * o[f][0] : fma(cf.so[(i0 + c) * H + j], o[f][j], S[f][c]);
                    }
#pragma unroll
            for (int c = 0; c < C; ++c) {
                const int i = i0 + c;
#pragma unroll
                for (int f = 0; f < 3; ++f)
                    if (i < HO) out(f, i, i < H ? S[f][c] + A[f][c] : S[f][c]);
#pragma unroll
                for (int f = 0; f < 3; ++f)
                    if (i < H) out(f, n - 1 - i, S[f][c] - A[f][c]);
            }
        }
    } else {
        R A[3][n];
#pragma unroll
        for (int j = 0; j < n; ++j)
#pragma unroll
            for (int i = 0; i < n; ++i)
#pragma unroll
                for (int f = 0; f < 3; ++f) A[f][i] = j == 0 ? cf.dhat[i * n] * x[f][0] : fma(cf.dhat[i * n + j], x[f][j], A[f][i]);
#pragma unroll
        for (int i = 0; i < n; ++i)
#pragma unroll
            for (int f = 0; f < 3; ++f) out(f, i, A[f][i]);
    }
}

// Args: StageArgs, or SpeedStageArgs for the variable-speed stage of the
// adjoint module (adjoint.cuh: the volume term times the element's speed, the
// face flux times the face's, optional copies of the stage input and of the
// receivers' pressure; one instance, no inflow sides).
template <int N, typename R, int E, typename Args, bool Seam>
__global__ void __launch_bounds__(LineTile<N, R, E>::kThreads, LineTile<N, R, E>::kMinBlocks) line_stage_kernel(Args a, const __grid_constant__ LineCoeffs<N, R> cf) {
    using T = LineTile<N, R, E>;
    constexpr int n = T::n, NN = T::NN, P = T::P, ES = T::ES, QS = T::QS, SE = T::SE;
    constexpr bool F64 = std::is_same_v<R, double>, kSpeed = std::is_same_v<Args, SpeedStageArgs>;
    extern __shared__ __align__(128) double smem[];
    double* qs = smem + T::kQ;
    double* ks = smem + T::kK;
    uint64_t* bar = reinterpret_cast<uint64_t*>(smem + T::kDoubles);
    R* rs = reinterpret_cast<R*>(bar + 2);
    R* far_s = rs + T::kFar;    // [element][SE] far characteristics
    R* side = rs + T::kSide;    // [nx, ny, edge metric, dx, dy][side][element]
    int* to_s = reinterpret_cast<int*>(rs + T::kRs);  // [side][element] side_entry
    const int tid = threadIdx.x;
    const int64_t K = a.n_elements, Kp = a.field_stride;
    const int64_t e0 = static_cast<int64_t>(blockIdx.x) * E;
    const int ne = static_cast<int>((K - e0) < E ? (K - e0) : E);
    const int64_t inst = blockIdx.y;
    double* q = a.q + inst * 3 * Kp * NN;
    double* k = a.k + inst * 3 * Kp * NN;
    const R* tr_in;
    R* tr_out;
    if constexpr (F64) {
        tr_in = a.trace_in;
        tr_out = a.trace_out;
    } else {
        tr_in = a.trace_in_f;
        tr_out = a.trace_out_f;
    }
    tr_in += inst * Kp * 4 * n;
    tr_out += inst * Kp * 4 * n;
    const int m = tid / E, e = tid % E;
    const bool active = m < n && e < ne;
    const int64_t ge = e0 + e;

    if constexpr (T::kBulk) {
        if (tid == 0) {
            mbar_init(bar, 1);
            mbar_fence_init();
        }
    }
    // Side data of the mesh plan, thread (element, side) with the side fastest.
    // The first of a thread's are read ahead of the wait for the launch before
    // and kept in registers until the tile's copies are on their way.
    struct SidePlanEntry {
        int2 lk;
        double2 nv, c0, c1;
        double speed;  // of the face (kSpeed)
    };
    const auto read_side = [&](int i) {
        const int64_t o = 4 * e0 + i;
        SidePlanEntry p{a.link[o], a.normal[o], reinterpret_cast<const double2*>(a.corners)[o],
                        reinterpret_cast<const double2*>(a.corners)[(o & ~int64_t{3}) + ((i + 1) & 3)], 1.0};
        if constexpr (kSpeed) {
            p.speed = a.c[o >> 2];
            if (((p.lk.y >> 2) & 7) == kInterior) p.speed = 0.5 * (p.speed + a.c[p.lk.x]);
        }
        return p;
    };
    const auto put_side = [&](int i, const SidePlanEntry& p) {
        const bool role = (p.lk.y >> 5) & 1;
        const R dx = R(p.c1.x - p.c0.x), dy = R(p.c1.y - p.c0.y);
        const int o = (i & 3) * E + (i >> 2);
        side[o] = R(role ? -p.nv.x : p.nv.x);
        side[4 * E + o] = R(role ? -p.nv.y : p.nv.y);
        side[8 * E + o] = R(0.5) * sqrt(dx * dx + dy * dy);
        if constexpr (kSpeed) side[8 * E + o] *= R(p.speed);
        side[12 * E + o] = dx;
        side[16 * E + o] = dy;
        to_s[o] = side_entry<Seam>(p.lk);
    };
    SidePlanEntry first_side{};
    if (tid < 4 * ne) first_side = read_side(tid);
    pdl_wait();
    if constexpr (!kSpeed)
        if (a.step_next && blockIdx.x == 0 && blockIdx.y == 0 && tid == 0) advance_step(a.step, a.step_next);
    if constexpr (T::kBulk) {
        if (tid == 0) {
            const uint32_t bytes = static_cast<uint32_t>(((ne + 1) & ~1) * NN * sizeof(double));
            mbar_expect_tx(bar, (a.first ? 3 : 6) * bytes);
            for (int f = 0; f < 3; ++f) bulk_load(qs + f * QS, q + (f * Kp + e0) * NN, bytes, bar);
            if (!a.first)
                for (int f = 0; f < 3; ++f) bulk_load(ks + f * QS, k + (f * Kp + e0) * NN, bytes, bar);
        }
    } else {
#pragma unroll
        for (int f = 0; f < 3; ++f) {
            const double* qf = q + (f * Kp + e0) * NN;
            const double* kf = k + (f * Kp + e0) * NN;
#pragma unroll 4
            for (int i = tid; i < ne * NN; i += T::kThreads) {
                const int d = f * QS + T::place(i);
                cp_async8(qs + d, qf + i);
                if (!a.first) cp_async8(ks + d, kf + i);
            }
        }
    }
    // Far characteristics: 4 n contiguous values per element.
    for (int i = tid; i < ne * 4 * n; i += T::kThreads) {
        const int el = i / (4 * n), o = i - el * 4 * n;
        if constexpr (F64)
            cp_async8(far_s + el * SE + o, tr_in + (e0 + el) * 4 * n + o);
        else
            cp_async4(far_s + el * SE + o, tr_in + (e0 + el) * 4 * n + o);
    }
    if (tid < 4 * ne) put_side(tid, first_side);
    for (int i = tid + T::kThreads; i < 4 * ne; i += T::kThreads) put_side(i, read_side(i));
    cp_async_wait_all();
    __syncthreads();
    if constexpr (T::kBulk) {
        if (!mbar_wait(bar, a.error, kWaitLimitNs)) return;
    }
    const R* xn = cf.xn;
    const R* lm = cf.lm;
    const R* lp = cf.lp;
    R ce = 1;  // element speed
    if constexpr (kSpeed) ce = active ? R(a.c[ge]) : R(1);
    const auto scaled = [&](R v) {
        if constexpr (kSpeed) return ce * v;
        return v;
    };
    if constexpr (kSpeed) {
        // The stage input, for the adjoint's gradient: out of the tile before
        // the rows overwrite it.
        if (a.q_save) {
            if constexpr (T::kBulk) {
                if (tid == 0) {
                    const uint32_t bytes = static_cast<uint32_t>(((ne + 1) & ~1) * NN * sizeof(double));
                    for (int f = 0; f < 3; ++f) bulk_store(a.q_save + (f * Kp + e0) * NN, qs + f * QS, bytes);
                    asm volatile("cp.async.bulk.commit_group;" ::: "memory");
                }
            } else {
#pragma unroll
                for (int f = 0; f < 3; ++f)
#pragma unroll 4
                    for (int i = tid; i < ne * NN; i += T::kThreads) a.q_save[(f * Kp + e0) * NN + i] = qs[f * QS + T::place(i)];
            }
        }
    }
    const R* dxs = side + 12 * E + e;
    const R* dys = side + 16 * E + e;

    // Upwind flux (Solver2D_t.cpp:48-63) of side s at its node idx, seen from
    // this element (outward normal, times the edge metric): with w = p + u.n of
    // the own trace and wR = p - u.n of the far one, (w - wR) / 2 and
    // n (w + wR) / 2. Ghost states as in stage_kernel.
    const auto side_flux = [&](int s, int idx, R op, R ou, R ov, R (&F)[3]) {
        // Keeps the loads of the contraction from being hoisted over the flux:
        // N = 8 FP64 128 registers instead of 166 (3 tiles an SM instead of 2).
        asm volatile("" ::: "memory");
        const R nx = side[s * E + e], ny = side[4 * E + s * E + e], sf = side[8 * E + s * E + e];
        const int to = to_s[s * E + e];
        R wR = far_s[e * SE + s * n + idx];
        if (!side_interior<Seam>(to)) {
            const int kind = ~to;
            R fp = R(0), fu = R(0), fv = R(0);
            if (kind == kMirror || kind == kCopy) {
                const R g = R(a.gscale[4 * ge + s]);
                fp = op * g;
                fu = ou * g;
                fv = ov * g;
                if (kind == kMirror) {
                    const R l0 = -(fu * nx + fv * ny), l1 = fv * nx - fu * ny;
                    fu = nx * l0 - ny * l1;
                    fv = ny * l0 + nx * l1;
                }
            } else if constexpr (!kSpeed) {
                if (kind == kAnalytic) {
                    const double4 gq = a.inflow[4 * ge + s];
                    const double r = (static_cast<double>(xn[N - idx]) + 1.0) * 0.5;
                    double pd, ud, vd;
                    plane_wave(gq.z * r + gq.x * (1.0 - r), gq.w * r + gq.y * (1.0 - r), a.step[0] + a.rk_b * a.step[1], pd, ud, vd);
                    fp = R(pd);
                    fu = R(ud);
                    fv = R(vd);
                }
            }
            wR = characteristic(fp, fu, fv, -nx, -ny);
        }
        const R wL = characteristic(op, ou, ov, nx, ny);
        const R h = R(0.5) * sf, sum = (wL + wR) * h;
        F[0] = (wL - wR) * h;
        F[1] = nx * sum;
        F[2] = ny * sum;
    };
    // New outgoing characteristic of side s at own node idx into the
    // neighbour's far slot.
    const auto send = [&](int s, int idx, R p, R u, R v) {
        const int to = to_s[s * E + e];
        if (!side_interior<Seam>(to)) return;
        R nx = side[s * E + e], ny = side[4 * E + s * E + e];
        if constexpr (Seam) {
            if (to < 0) {
                const double2 fn = far_inward(side_far<Seam>(to), a.normal, a.link);
                nx = R(fn.x);
                ny = R(fn.y);
            }
        }
        tr_out[side_far<Seam>(to) * n + (N - idx)] = characteristic(p, u, v, nx, ny);
    };

    if (active) {
        // xi direction, column j = m: right and left traces and fluxes, the
        // contravariant flux lines eta_y X - eta_x Y with (X, Y) = (u, v),
        // (p, 0), (0, p) (Solver2D_t.cpp:31-37, 72-80), their contraction and
        // lift (:82-101), k <- a k - (...) / J.
        const double* Q = qs + e * ES + m;
        double* Kc = ks + e * ES + m;
        R x[3][n];
        R tr[3] = {0, 0, 0}, tl[3] = {0, 0, 0};
#pragma unroll
        for (int f = 0; f < 3; ++f)
#pragma unroll
            for (int i = 0; i < n; ++i) {
                const R v = R(Q[f * QS + i * P]);
                tr[f] = fma(lp[i], v, tr[f]);
                tl[f] = fma(lm[i], v, tl[f]);
                x[f][i] = v;
            }
        R Fr[3], Fl[3];
        side_flux(1, m, tr[0], tr[1], tr[2], Fr);
        side_flux(3, N - m, tl[0], tl[1], tl[2], Fl);
        const MLine<R> x_eta(-dxs[3 * E], dxs[E]), y_eta(-dys[3 * E], dys[E]);
        const R xx = MLine<R>(dxs[0], -dxs[2 * E])(xn[m]), yx = MLine<R>(dys[0], -dys[2 * E])(xn[m]);
        const R Ja = xx * y_eta.a - x_eta.a * yx, Jb = xx * y_eta.b - x_eta.b * yx;  // J(xi) = Ja + Jb xi on this line
        const auto upd = [&](int f, int i, R y) {
            const R iJ = line_rcp(fma(xn[i], Jb, Ja));
            const R G = -y * iJ;
            double* kp = Kc + f * QS + i * P;
            *kp = a.first ? static_cast<double>(G) : fma(a.rk_a, *kp, static_cast<double>(G));
        };
#pragma unroll
        for (int i = 0; i < n; ++i) {
            const R xe = scaled(x_eta(xn[i])), ye = scaled(y_eta(xn[i]));
            const R p = x[0][i];
            x[0][i] = ye * x[1][i] - xe * x[2][i];
            x[1][i] = ye * p;
            x[2][i] = -xe * p;
        }
        line_contract<N, R>(cf, x, Fr, Fl, upd);
    }
    if constexpr (kSpeed && T::kBulk) {
        if (tid == 0) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
    }
    __syncthreads();
    if (active) {
        // eta direction, row i = m: top and bottom, flux lines -xi_y X + xi_x Y
        // (:103-113), and the RK update (:138-172); top and bottom
        // characteristics of the new q.
        double* Q = qs + e * ES + m * P;
        double* Kr = ks + e * ES + m * P;
        double gdt;
        if constexpr (kSpeed)
            gdt = a.gdt;
        else
            gdt = a.rk_g * a.step[1];
        R x[3][n];
        R tt[3] = {0, 0, 0}, tb[3] = {0, 0, 0};
#pragma unroll
        for (int f = 0; f < 3; ++f)
#pragma unroll
            for (int j = 0; j < n; ++j) {
                const R v = R(Q[f * QS + j]);
                tt[f] = fma(lp[j], v, tt[f]);
                tb[f] = fma(lm[j], v, tb[f]);
                x[f][j] = v;
            }
        R Ft[3], Fb[3];
        side_flux(2, N - m, tt[0], tt[1], tt[2], Ft);
        side_flux(0, m, tb[0], tb[1], tb[2], Fb);
        const MLine<R> x_xi(dxs[0], -dxs[2 * E]), y_xi(dys[0], -dys[2 * E]);
        const R xe = MLine<R>(-dxs[3 * E], dxs[E])(xn[m]), ye = MLine<R>(-dys[3 * E], dys[E])(xn[m]);
        const R Ja = x_xi.a * ye - xe * y_xi.a, Jb = x_xi.b * ye - xe * y_xi.b;
#pragma unroll
        for (int f = 0; f < 3; ++f) tt[f] = tb[f] = 0;
        const auto upd = [&](int f, int j, R y) {
            const R iJ = line_rcp(fma(xn[j], Jb, Ja));
            const R G = -y * iJ;
            const double kn = Kr[f * QS + j] + static_cast<double>(G);
            const double qn = fma(gdt, kn, Q[f * QS + j]);
            Kr[f * QS + j] = kn;
            Q[f * QS + j] = qn;
            tt[f] = fma(lp[j], R(qn), tt[f]);
            tb[f] = fma(lm[j], R(qn), tb[f]);
        };
#pragma unroll
        for (int j = 0; j < n; ++j) {
            const R xx = scaled(x_xi(xn[j])), yx = scaled(y_xi(xn[j]));
            const R p = x[0][j];
            x[0][j] = xx * x[2][j] - yx * x[1][j];
            x[1][j] = -yx * p;
            x[2][j] = xx * p;
        }
        line_contract<N, R>(cf, x, Ft, Fb, upd);
        send(2, N - m, tt[0], tt[1], tt[2]);
        send(0, m, tb[0], tb[1], tb[2]);
    }
    if constexpr (T::kBulk) asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    __syncthreads();
    pdl_launch_dependents();
    if constexpr (T::kBulk) {
        if (tid == 0) {
            const uint32_t bytes = static_cast<uint32_t>(((ne + 1) & ~1) * NN * sizeof(double));
            for (int f = 0; f < 3; ++f) {
                bulk_store(q + (f * Kp + e0) * NN, qs + f * QS, bytes);
                bulk_store(k + (f * Kp + e0) * NN, ks + f * QS, bytes);
            }
            asm volatile("cp.async.bulk.commit_group;" ::: "memory");
        }
    } else {
#pragma unroll
        for (int f = 0; f < 3; ++f) {
            double* qf = q + (f * Kp + e0) * NN;
            double* kf = k + (f * Kp + e0) * NN;
#pragma unroll 4
            for (int i = tid; i < ne * NN; i += T::kThreads) {
                const int d = f * QS + T::place(i);
                qf[i] = qs[d];
                kf[i] = ks[d];
            }
        }
    }
    if (active) {
        // Right and left characteristics of the new q.
        const double* Q = qs + e * ES + m;
        R tr[3] = {0, 0, 0}, tl[3] = {0, 0, 0};
#pragma unroll
        for (int f = 0; f < 3; ++f)
#pragma unroll
            for (int i = 0; i < n; ++i) {
                const R v = R(Q[f * QS + i * P]);
                tr[f] = fma(lp[i], v, tr[f]);
                tl[f] = fma(lm[i], v, tl[f]);
            }
        send(1, m, tr[0], tr[1], tr[2]);
        send(3, N - m, tl[0], tl[1], tl[2]);
    }
    if constexpr (kSpeed) {
        // Receivers' pressure of the new q, one warp, in a fixed order.
        if (a.samples && tid < 32) {
            for (int r = 0; r < a.rec.n; ++r) {
                const int64_t el = a.rec.elem[r] - e0;
                if (el < 0 || el >= ne) continue;
                const double v = receiver_value<n, P>(a.rec.w + static_cast<int64_t>(r) * NN, qs + el * ES, tid);
                if (tid == 0) a.samples[r] = v;
            }
        }
    }
    if constexpr (T::kBulk) {
        if (tid == 0) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
    }
}

// Outgoing characteristics of q into the neighbours' far slots (start of a
// run, or after the host changed q).
template <int N, typename R>
__global__ void __launch_bounds__(256) line_trace_kernel(TraceArgs a, const __grid_constant__ LineCoeffs<N, R> cf) {
    constexpr int n = N + 1, NN = n * n;
    const int64_t K = a.n_elements, Kp = a.field_stride;
    const int64_t total = static_cast<int64_t>(a.n_instances) * K * 4 * n;
    R* out;
    if constexpr (std::is_same_v<R, double>)
        out = a.trace_out;
    else
        out = a.trace_out_f;
    for (int64_t idx = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; idx < total; idx += static_cast<int64_t>(gridDim.x) * blockDim.x) {
        const int m = static_cast<int>(idx % n);
        const int s = static_cast<int>((idx / n) % 4);
        const int64_t e = (idx / (4 * n)) % K, inst = idx / (4 * n * K);
        const int2 lk = a.link[4 * e + s];
        if (((lk.y >> 2) & 7) != kInterior) continue;
        const int64_t far = 4 * static_cast<int64_t>(lk.x) + (lk.y & 3);
        double2 nv = a.normal[4 * e + s];
        if ((lk.y >> 5) & 1) nv = double2{-nv.x, -nv.y};
        if (lk.y & kSeamNormal) nv = far_inward(far, a.normal, a.link);
        const int line = (s < 2) ? m : N - m;
        const int base = (s == 0 || s == 2) ? line * n : line, stride = (s == 0 || s == 2) ? 1 : n;
        R t[3] = {0, 0, 0};
#pragma unroll
        for (int f = 0; f < 3; ++f) {
            const double* qe = a.q + ((inst * 3 + f) * Kp + e) * NN + base;
            for (int i = 0; i < n; ++i) {
                // the stage kernel's order: along rows (bottom, top) as line_contract hands the
                // nodes out, along columns node by node
                const int j = (s == 0 || s == 2) ? LineCoeffs<N, R>::out_node(i) : i;
                t[f] = fma((s == 0 || s == 3) ? cf.lm[j] : cf.lp[j], R(qe[j * stride]), t[f]);
            }
        }
        out[(inst * Kp * 4 + far) * n + (N - m)] = characteristic(t[0], t[1], t[2], R(nv.x), R(nv.y));
    }
}

}  // namespace dev
}  // namespace ndg

// The adjoint stage with one thread per (line, element), for all three fields
// (the layout and conventions of line_stage.cuh; what it computes is
// adjoint_stage_kernel's, adjoint_kernels.cu).
//
// Columns first: mu = lk + gdt lq (kept in lk's tile), nu = -mu / J, the lift
// transposes and the transposed flux of sides 1 and 3, the transposed
// contraction, lq += column part. Then rows: sides 2 and 0 and the row part,
// the misfit, lk = a mu, and nu' = -(lk + gdt_next lq) / J of the next stage
// (in the stage input's tile), whose lift transposes give the far side's
// adjoint on sides 2 and 0; a last column pass gives it on sides 1 and 3.
//
// With b = (n . psi_uv - psi_p) / 2 and a = (n . psi_uv + psi_p) / 2 of a
// side's flux adjoint psi (n outward), the transposed upwind flux is a (1, n)
// on the own trace and b (1, -n) on the far one, so sides exchange the scalar
// b: a third of the trace traffic of three components, as in the forward. The
// receiving element applies the sender's normal: the opposite of its own, or on
// a seam (kSeamNormal) the neighbour side's.
//
// Measured, backward of 60 steps with checkpoints every 20 (its recomputation
// included), ms, in parentheses three threads a line with the same launches. At
// 96 x 96, FP64: N = 1 1.18 (3.07), 2 1.39 (3.67), 3 1.80 (3.60), 4 1.97 (4.85), 5
// 2.91 (6.51), 6 3.54 (7.88), 7 5.09 (8.10), 8 5.89 (11.7), 9 10.1 (14.3), 10 10.7
// (18.9), 11 16.1 (22.8), 12 19.8 (26.8); FP32 form: N = 1 1.20 (2.29), 2 1.34
// (2.79), 3 1.96 (2.82), 4 2.13 (3.58), 5 3.03 (5.42), 6 3.90 (6.68), 8 6.14
// (9.62), 10 12.2 (16.1). By the size rule of the forward (kLineMinElements): at
// 1,600 elements FP64 N = 5 1.41 (1.97), 8 1.93 (2.77), 12 3.41 (6.14), FP32 N = 8
// 2.18 (2.74); at 100 elements N = 1 1.15 (1.37), 4 1.09 (1.58). The forward of
// the same steps is ahead too but for N = 9 and FP32 N = 10 below 2,304 elements
// (1.79 against 1.70, 1.71 against 1.57). Nine field tiles an element bound the
// tiles per SM (N = 7: 2, 7.5 warps); latency is what is left.
#include "adjoint.cuh"
#include "line_stage.cuh"

namespace ndg {
namespace dev {

namespace {

// Coefficients of the transposed contraction: Dhat transposed in the place of
// Dhat (it is centro-antisymmetric too), the lift weights l(+-1)/w.
template <int N, typename R>
struct AdjLineCoeffs {
    LineCoeffs<N, R> t;
    R lpw[N + 1], lmw[N + 1];
};

template <int N, typename R>
AdjLineCoeffs<N, R> make_adj_line_coeffs() {
    constexpr int n = N + 1;
    double dh[n * n], dt[n * n], xn[n], lm[n], lp[n], w[n], iw[n];
    host_coefficients(N, dh, xn, lm, lp, w, iw);
    for (int i = 0; i < n; ++i)
        for (int j = 0; j < n; ++j) dt[i * n + j] = dh[j * n + i];
    AdjLineCoeffs<N, R> c{};
    c.t = make_line_coeffs<N, R>();
    if constexpr (LineCoeffs<N, R>::kEvenOdd)
        even_odd_halves(n, dt, c.t.ea, c.t.so);
    else
        for (int i = 0; i < n * n; ++i) c.t.dhat[i] = static_cast<R>(dt[i]);
    for (int i = 0; i < n; ++i) {
        c.lpw[i] = static_cast<R>(lp[i] * iw[i]);
        c.lmw[i] = static_cast<R>(lm[i] * iw[i]);
    }
    return c;
}

template <int N, typename R, int E>
struct AdjLineTile {
    using L = LineTile<N, R, E>;
    static constexpr int n = N + 1, QS = L::QS;
    static constexpr int kThreads = L::kThreads;
    static constexpr int kRes = 9 * QS + (9 * QS) % 2, kMask = kRes + kMaxReceivers, kVol = kMask + (E + 1) / 2 * 2;
    static constexpr int kDoubles = kVol + (n * E + 1) / 2 * 2;  // lq, lk (mu), qs (nu'); residuals; receiver masks; volume sums
    static constexpr int kFar = 0, kSide = (E * L::SE + 1) / 2 * 2, kSum = kSide + 7 * 4 * E, kRs = (kSum + 4 * n * E + 3) / 4 * 4;
    static constexpr size_t kBytes = sizeof(double) * kDoubles + 16 + sizeof(R) * kRs + sizeof(int) * 4 * E;
    static constexpr int kFit = static_cast<int>((232448 - (L::kBulk ? 0 : 24 * 1024)) / (kBytes + 1024));
    static constexpr int kByRegs = 65536 / (kThreads * 128);
    static constexpr int kMinBlocks = kFit < 1 || kByRegs < 1 ? 1 : (kFit < kByRegs ? kFit : kByRegs);
    static constexpr bool feasible = kBytes <= 226 * 1024;
};

template <int N, typename R, int E, bool Seam>
__global__ void __launch_bounds__(AdjLineTile<N, R, E>::kThreads, AdjLineTile<N, R, E>::kMinBlocks)
    adjoint_line_kernel(AdjointStageArgs a, const __grid_constant__ AdjLineCoeffs<N, R> cf) {
    using A = AdjLineTile<N, R, E>;
    using T = LineTile<N, R, E>;
    constexpr int n = T::n, NN = T::NN, P = T::P, ES = T::ES, QS = T::QS, SE = T::SE;
    constexpr bool F64 = std::is_same_v<R, double>;
    extern __shared__ __align__(128) double smem[];
    double* ls = smem;
    double* ks = smem + 3 * QS;  // lk, then mu, then the new lk
    double* qs = smem + 6 * QS;  // the stage input, then nu'
    double* res = smem + A::kRes;
    unsigned long long* rmask = reinterpret_cast<unsigned long long*>(smem + A::kMask);
    uint64_t* bar = reinterpret_cast<uint64_t*>(smem + A::kDoubles);
    R* rs = reinterpret_cast<R*>(bar + 2);
    R* far_s = rs + A::kFar;
    R* side = rs + A::kSide;  // [nx, ny, edge metric, face speed, dx, dy, ghost scale][side][element]
    R* sum_s = rs + A::kSum;         // [side][line][element] of the speed derivative
    double* vol_s = smem + A::kVol;  // [line][element], its volume part
    int* to_s = reinterpret_cast<int*>(rs + A::kRs);
    const int tid = threadIdx.x;
    const int64_t K = a.n_elements, Kp = a.field_stride;
    const int64_t e0 = static_cast<int64_t>(blockIdx.x) * E;
    const int ne = static_cast<int>((K - e0) < E ? (K - e0) : E);
    const R* atr_in;
    R* atr_out;
    if constexpr (F64) {
        atr_in = a.atr_in;
        atr_out = a.atr_out;
    } else {
        atr_in = a.atr_in_f;
        atr_out = a.atr_out_f;
    }
    const int m = tid / E, e = tid % E;
    const bool active = m < n && e < ne;
    const int64_t ge = e0 + e;

    // Prologue: the plan ahead of the wait, then the tiles.
    if constexpr (T::kBulk) {
        if (tid == 0) {
            mbar_init(bar, 1);
            mbar_fence_init();
        }
    }
    for (int i = tid; i < 4 * ne; i += A::kThreads) {
        const int64_t o4 = 4 * e0 + i;
        const int2 lk = a.link[o4];
        const double2 nv = a.normal[o4], c0 = reinterpret_cast<const double2*>(a.corners)[o4],
                      c1 = reinterpret_cast<const double2*>(a.corners)[(o4 & ~int64_t{3}) + ((i + 1) & 3)];
        const bool role = (lk.y >> 5) & 1;
        const int kind = (lk.y >> 2) & 7;
        const R dx = R(c1.x - c0.x), dy = R(c1.y - c0.y);
        double speed = a.c[o4 >> 2];
        if (kind == kInterior) speed = 0.5 * (speed + a.c[lk.x]);
        const int o = (i & 3) * E + (i >> 2);
        side[o] = R(role ? -nv.x : nv.x);
        side[4 * E + o] = R(role ? -nv.y : nv.y);
        side[8 * E + o] = R(0.5) * sqrt(dx * dx + dy * dy);
        side[12 * E + o] = R(speed);
        side[16 * E + o] = dx;
        side[20 * E + o] = dy;
        side[24 * E + o] = (kind == kMirror || kind == kCopy) ? R(a.gscale[o4]) : R(0);
        to_s[o] = side_entry<Seam>(lk);
    }
    for (int i = tid; i < E; i += A::kThreads) rmask[i] = 0ull;
    const R ce = active ? R(a.c[ge]) : R(1);
    pdl_wait();
    if constexpr (T::kBulk) {
        if (tid == 0) {
            const uint32_t bytes = static_cast<uint32_t>(((ne + 1) & ~1) * NN * sizeof(double));
            mbar_expect_tx(bar, 9 * bytes);
            for (int f = 0; f < 3; ++f) {
                bulk_load(ls + f * QS, a.lq + (f * Kp + e0) * NN, bytes, bar);
                bulk_load(ks + f * QS, a.lk + (f * Kp + e0) * NN, bytes, bar);
                bulk_load(qs + f * QS, a.qs + (f * Kp + e0) * NN, bytes, bar);
            }
        }
    } else {
#pragma unroll
        for (int f = 0; f < 3; ++f) {
            const int64_t g = (f * Kp + e0) * NN;
#pragma unroll 4
            for (int i = tid; i < ne * NN; i += A::kThreads) {
                const int d = f * QS + T::place(i);
                cp_async8(ls + d, a.lq + g + i);
                cp_async8(ks + d, a.lk + g + i);
                cp_async8(qs + d, a.qs + g + i);
            }
        }
    }
    for (int i = tid; i < ne * 4 * n; i += A::kThreads) {
        const int el = i / (4 * n), o = i - el * 4 * n;
        if constexpr (F64)
            cp_async8(far_s + el * SE + o, atr_in + (e0 + el) * 4 * n + o);
        else
            cp_async4(far_s + el * SE + o, atr_in + (e0 + el) * 4 * n + o);
    }
    cp_async_wait_all();
    __syncthreads();
    if constexpr (T::kBulk) {
        if (!mbar_wait(bar, a.error, kWaitLimitNs)) return;
    }
    // Weighted misfit residuals of the tile's receivers (used by the rows,
    // after the next barrier).
    if (a.inject && tid < 32) {
        for (int r = 0; r < a.rec.n; ++r) {
            const int64_t el = a.rec.elem[r] - e0;
            if (el < 0 || el >= ne) continue;
            const double v = receiver_value<n, P>(a.rec.w + static_cast<int64_t>(r) * NN, qs + el * ES, tid);
            if (tid == 0) {
                res[r] = a.wdt * (v - a.target[r]);
                rmask[el] |= 1ull << r;
            }
        }
    }
    const R* xn = cf.t.xn;
    const R* lm = cf.t.lm;
    const R* lp = cf.t.lp;
    const R* dxs = side + 16 * E + e;
    const R* dys = side + 20 * E + e;

    // Half sums of side s's flux adjoint psi = l (edge metric) (face speed):
    // pp / 2 and (n . puv) / 2.
    const auto halves = [&](int s, const R (&l)[3], R& hp, R& hn) {
        const R sc = R(0.5) * (side[8 * E + s * E + e] * side[12 * E + s * E + e]);
        hp = sc * l[0];
        hn = sc * (side[s * E + e] * l[1] + side[4 * E + s * E + e] * l[2]);
    };
    // Transposed flux of side s at its node idx: t = adjoint of the own trace;
    // returns own trace . t / face speed.
    const auto side_adjoint = [&](int s, int idx, const R (&l)[3], const R (&own)[3], R (&t)[3]) {
        asm volatile("" ::: "memory");  // as in the forward: no loads hoisted over the flux
        const R nx = side[s * E + e], ny = side[4 * E + s * E + e];
        R hp, hn;
        halves(s, l, hp, hn);
        const R av = hn + hp, b = hn - hp;
        R tp = av, tn = av;
        const int to = to_s[s * E + e];
        if (side_interior<Seam>(to)) {
            const R f = far_s[e * SE + s * n + idx];
            tp += f;
            tn += f;
        } else {
            const R g = side[24 * E + s * E + e];  // 0 for a zero ghost
            tp = fma(g, b, tp);
            tn = ~to == kMirror ? fma(g, b, tn) : fma(-g, b, tn);
        }
        t[0] = tp;
        t[1] = tn * nx;
        t[2] = tn * ny;
        if constexpr (Seam) {
            if (to < 0 && side_interior<Seam>(to)) {
                const double2 fn = far_inward(side_far<Seam>(to), a.normal, a.link);
                const R f = far_s[e * SE + s * n + idx];
                t[1] = fma(f, R(fn.x), av * nx);
                t[2] = fma(f, R(fn.y), av * ny);
            }
        }
        return (own[0] * t[0] + own[1] * t[1] + own[2] * t[2]) / side[12 * E + s * E + e];
    };
    const auto publish = [&](int s, int idx, const R (&l)[3]) {
        const int to = to_s[s * E + e];
        if (!side_interior<Seam>(to)) return;
        R hp, hn;
        halves(s, l, hp, hn);
        atr_out[side_far<Seam>(to) * n + (N - idx)] = hn - hp;
    };
    // Volume part of the speed derivative on this thread's column and row: in
    // the FP32 form one FP32 sum per field, joined in FP64. One sum over the
    // three fields is further from FP64 (N = 8, 40 x 40: 2.48e-7 relative RMS
    // against 2.03e-7; three threads a line 1.95e-7); backward of 60 steps at
    // 96 x 96 6.11 -> 6.14 ms (N = 5 2.97 -> 3.03).
    R vdot[F64 ? 1 : 3] = {};
    const auto volume = [&](int f, R q, R d) {
        R& v = vdot[F64 ? 0 : f];
        v = fma(q, d, v);
    };

    if (active) {
        double* Lc = ls + e * ES + m;
        double* Kc = ks + e * ES + m;
        const double* Q = qs + e * ES + m;
        const MLine<R> x_eta(-dxs[3 * E], dxs[E]), y_eta(-dys[3 * E], dys[E]);
        const R xx = MLine<R>(dxs[0], -dxs[2 * E])(xn[m]), yx = MLine<R>(dys[0], -dys[2 * E])(xn[m]);
        const R Ja = xx * y_eta.a - x_eta.a * yx, Jb = xx * y_eta.b - x_eta.b * yx;
        R x[3][n], l1[3] = {0, 0, 0}, l3[3] = {0, 0, 0}, r[3] = {0, 0, 0}, l[3] = {0, 0, 0};
#pragma unroll
        for (int i = 0; i < n; ++i) {
            const R iJ = line_rcp(fma(xn[i], Jb, Ja));
#pragma unroll
            for (int f = 0; f < 3; ++f) {
                const int o = f * QS + i * P;
                const double mu = fma(a.gdt, Lc[o], Kc[o]);
                Kc[o] = mu;
                x[f][i] = -R(mu) * iJ;
                l1[f] = fma(x[f][i], cf.lpw[i], l1[f]);
                l3[f] = fma(x[f][i], cf.lmw[i], l3[f]);
                const R v = R(Q[o]);
                r[f] = fma(lp[i], v, r[f]);
                l[f] = fma(lm[i], v, l[f]);
            }
        }
        R t1[3], t3[3];
        sum_s[(1 * n + m) * E + e] = side_adjoint(1, m, l1, r, t1);
        sum_s[(3 * n + (N - m)) * E + e] = side_adjoint(3, N - m, l3, l, t3);
        R y[3];
        line_product<N, R>(cf.t, x, [&](int f, int i, R v) {
            y[f] = v;
            if (f < 2) return;
            const R xe = x_eta(xn[i]), ye = y_eta(xn[i]);
            const R dp = ye * y[1] - xe * y[2], du = ye * y[0], dv = -xe * y[0];
            const int o = i * P;
            volume(2, R(Q[2 * QS + o]), dv);
            volume(1, R(Q[QS + o]), du);
            volume(0, R(Q[o]), dp);
            Lc[o] += static_cast<double>(ce * dp) + static_cast<double>(fma(lp[i], t1[0], lm[i] * t3[0]));
            Lc[QS + o] += static_cast<double>(ce * du) + static_cast<double>(fma(lp[i], t1[1], lm[i] * t3[1]));
            Lc[2 * QS + o] += static_cast<double>(ce * dv) + static_cast<double>(fma(lp[i], t1[2], lm[i] * t3[2]));
        });
    }
    __syncthreads();
    if (active) {
        double* Lr = ls + e * ES + m * P;
        double* Kr = ks + e * ES + m * P;
        double* Q = qs + e * ES + m * P;
        const MLine<R> x_xi(dxs[0], -dxs[2 * E]), y_xi(dys[0], -dys[2 * E]);
        const R xe = MLine<R>(-dxs[3 * E], dxs[E])(xn[m]), ye = MLine<R>(-dys[3 * E], dys[E])(xn[m]);
        const R Ja = x_xi.a * ye - xe * y_xi.a, Jb = x_xi.b * ye - xe * y_xi.b;
        R x[3][n], l2[3] = {0, 0, 0}, l0[3] = {0, 0, 0}, tp[3] = {0, 0, 0}, bt[3] = {0, 0, 0};
#pragma unroll
        for (int j = 0; j < n; ++j) {
            const R iJ = line_rcp(fma(xn[j], Jb, Ja));
#pragma unroll
            for (int f = 0; f < 3; ++f) {
                x[f][j] = -R(Kr[f * QS + j]) * iJ;
                l2[f] = fma(x[f][j], cf.lpw[j], l2[f]);
                l0[f] = fma(x[f][j], cf.lmw[j], l0[f]);
                const R v = R(Q[f * QS + j]);
                tp[f] = fma(lp[j], v, tp[f]);
                bt[f] = fma(lm[j], v, bt[f]);
            }
        }
        R t2[3], t0[3];
        sum_s[(2 * n + (N - m)) * E + e] = side_adjoint(2, N - m, l2, tp, t2);
        sum_s[m * E + e] = side_adjoint(0, m, l0, bt, t0);
#pragma unroll
        for (int f = 0; f < 3; ++f) l2[f] = l0[f] = 0;
        const unsigned long long mask0 = rmask[e];
        R y[3];
        line_product<N, R>(cf.t, x, [&](int f, int j, R v) {
            y[f] = v;
            if (f < 2) return;
            const R xx = x_xi(xn[j]), yx = y_xi(xn[j]);
            const R d[3] = {xx * y[2] - yx * y[1], -yx * y[0], xx * y[0]};
            const R iJ = line_rcp(fma(xn[j], Jb, Ja));
#pragma unroll
            for (int g = 0; g < 3; ++g) {
                const int o = g * QS + j;
                volume(g, R(Q[o]), d[g]);
                double lq = Lr[o] + (static_cast<double>(ce * d[g]) + static_cast<double>(fma(lp[j], t2[g], lm[j] * t0[g])));
                if (g == 0) {
                    unsigned long long mask = mask0;
                    while (mask) {
                        const int rc = __ffsll(static_cast<long long>(mask)) - 1;
                        mask &= mask - 1;
                        lq = fma(res[rc], a.rec.w[static_cast<int64_t>(rc) * NN + m * n + j], lq);
                    }
                }
                const double lk = a.rk_a * Kr[o];
                Lr[o] = lq;
                Kr[o] = lk;
                const R nu = -R(fma(a.gdt_next, lq, lk)) * iJ;
                Q[o] = static_cast<double>(nu);
                l2[g] = fma(nu, cf.lpw[j], l2[g]);
                l0[g] = fma(nu, cf.lmw[j], l0[g]);
            }
        });
        if constexpr (F64)
            vol_s[m * E + e] = vdot[0];
        else
            vol_s[m * E + e] = (static_cast<double>(vdot[0]) + static_cast<double>(vdot[1])) + static_cast<double>(vdot[2]);
        publish(2, N - m, l2);
        publish(0, m, l0);
    }
    if constexpr (T::kBulk) asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    __syncthreads();
    pdl_launch_dependents();
    if constexpr (T::kBulk) {
        if (tid == 0) {
            const uint32_t bytes = static_cast<uint32_t>(((ne + 1) & ~1) * NN * sizeof(double));
            for (int f = 0; f < 3; ++f) {
                bulk_store(a.lq + (f * Kp + e0) * NN, ls + f * QS, bytes);
                bulk_store(a.lk + (f * Kp + e0) * NN, ks + f * QS, bytes);
            }
            asm volatile("cp.async.bulk.commit_group;" ::: "memory");
        }
    } else {
#pragma unroll
        for (int f = 0; f < 3; ++f) {
            const int64_t g = (f * Kp + e0) * NN;
#pragma unroll 4
            for (int i = tid; i < ne * NN; i += A::kThreads) {
                const int d = f * QS + T::place(i);
                a.lq[g + i] = ls[d];
                a.lk[g + i] = ks[d];
            }
        }
    }
    if (active) {
        const double* Q = qs + e * ES + m;
        R l1[3] = {0, 0, 0}, l3[3] = {0, 0, 0};
#pragma unroll
        for (int f = 0; f < 3; ++f)
#pragma unroll
            for (int i = 0; i < n; ++i) {
                const R v = R(Q[f * QS + i * P]);
                l1[f] = fma(v, cf.lpw[i], l1[f]);
                l3[f] = fma(v, cf.lmw[i], l3[f]);
            }
        publish(1, m, l1);
        publish(3, N - m, l3);
    }
    // Speed derivative: the element's five sums, in FP64.
    for (int i = tid; i < 5 * E; i += A::kThreads) {
        const int w = i / E, el = i % E;
        if (el < ne) {
            double s = 0.0;
            for (int j = 0; j < n; ++j) s += w == 0 ? vol_s[j * E + el] : static_cast<double>(sum_s[((w - 1) * n + j) * E + el]);
            a.acc[(e0 + el) * 5 + w] += s;
        }
    }
    if constexpr (T::kBulk) {
        if (tid == 0) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
    }
}

// Elements a tile, by the measure above (96 x 96, ms, with 16 / 8 / 4): FP64 N =
// 1 1.26 / 1.25 / 1.55, 2 1.45 / 1.54 / 1.65, 3 1.84 / 1.90 / 2.05, 4 2.01 / 2.44
// / 2.59, 5 2.89 / 3.47 / 3.66, 6 3.53 / 4.34 / 4.24, 7 5.09 / 5.46 / 5.51, 8 5.87
// / 7.33 / 8.78, 9 10.71 / 10.13 / 10.16, 10 10.78 / 12.09 / 12.16, 11 (8 / 4)
// 16.23 / 16.18, 12 19.50 / 19.84; FP32 N = 5 2.94 / 3.14 / 3.83, 8 6.10 / 7.38 /
// 8.03, 10 12.21 / 12.94 / 12.85.
template <int N>
constexpr int elements() {
    return N <= 8 || N == 10 ? 16 : (N <= 10 ? 8 : 4);
}

template <int N, typename R>
cudaError_t prepare(bool seam) {
    if constexpr (line_order(N, sizeof(R) == 4)) {
        constexpr int E = elements<N>();
        static_assert(AdjLineTile<N, R, E>::feasible);
        return cudaFuncSetAttribute(seam ? adjoint_line_kernel<N, R, E, true> : adjoint_line_kernel<N, R, E, false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    static_cast<int>(AdjLineTile<N, R, E>::kBytes));
    } else {
        return cudaErrorInvalidValue;
    }
}

template <int N, typename R>
cudaError_t launch(bool seam, const AdjointStageArgs& a, cudaStream_t stream) {
    if constexpr (line_order(N, sizeof(R) == 4)) {
        constexpr int E = elements<N>();
        using A = AdjLineTile<N, R, E>;
        return launch_dependent(seam ? adjoint_line_kernel<N, R, E, true> : adjoint_line_kernel<N, R, E, false>, dim3(static_cast<unsigned>((a.n_elements + E - 1) / E)), A::kThreads, A::kBytes, stream, a,
                                make_adj_line_coeffs<N, R>());
    } else {
        return cudaErrorInvalidValue;
    }
}

}  // namespace

#define NDG_ADJOINT_LINE_DISPATCH(FN, ...)                                              \
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

cudaError_t prepare_adjoint_line(int N, bool fp32, bool seam) { NDG_ADJOINT_LINE_DISPATCH(prepare, seam) }

cudaError_t launch_adjoint_line(int N, bool fp32, bool seam, const AdjointStageArgs& a, cudaStream_t stream) {
    NDG_ADJOINT_LINE_DISPATCH(launch, seam, a, stream)
}

}  // namespace dev
}  // namespace ndg

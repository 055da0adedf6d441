// ft_adjoint.cu -- ft_adj_lmul and ft_adj_rmul for widths 2..8 (the general
// kernel and the definition of both sums are in ft_ops.cu).
//
// A coefficient of degree m sums one term per op word of each split degree p:
// thousands of terms in the lowest degrees, one in the top.  Warps take tasks
// from a counter, most terms first, with no barrier of the CTA between degrees:
//  * degrees of fewer than 32 coefficients: right, a warp per coefficient, its
//    lanes on consecutive op and argument words (where there are 64 terms for
//    them); left, a warp per degree, lanes (u, j) on consecutive argument words,
//    u W^m + j; summed by shuffles in a fixed order;
//  * the others: a lane per coefficient, the splits p = 0 and 1 with the op's
//    coefficients in registers.  Left, lanes read consecutive argument words.
//    Right, lane j reads the block j W^p + v: where W^p is a power of two that
//    would put lanes in the same banks, each lane starts at its own v.
// The width is a compile-time constant and the term loops are unrolled, which
// is what FP32 gains from: the general kernel spends ten instructions a
// multiply-add and two CTA barriers a degree.  Bound by instruction issue in FP32
// (0.76 instructions a clock and scheduler at W5 D5), by the pipe in FP64.
// FP32 sums are formed in short blocks: shorter chains of dependent additions
// (left W5 D5 78 -> 68 us) and a smaller rounding error.
// Left / right, general kernel -> this: FP32 W5 D5 batch 4096 112 -> 68 / 119 ->
// 75 us, W8 D4 111 -> 68 / 117 -> 81, W2 D12 batch 2048 183 -> 111 / 211 -> 152;
// FP64 W5 D5 221 -> 204 / 233 -> 211, W2 D8 99 -> 47 / 137 -> 73, W2 D12 547 -> 430 /
// 591 -> 503.
#include <algorithm>
#include <type_traits>

#include "bulk_stage.cuh"
#include "common.cuh"
#include "ft_column.cuh"
#include "launch_util.cuh"
#include "ops.hpp"

namespace rpp_gb {
namespace {

using namespace ftcol;

// Tasks of the output degrees, made on the host: degree m's are [start[m],
// start[m+1]), each of run[m] coefficients (0: a warp's coefficient, or degree).
struct AdjointTasks {
    uint32_t start[kMaxDepth + 2];
    uint32_t run[kMaxDepth + 1];
};

AdjointTasks adjoint_tasks(const Geometry& g, bool left, bool fp64, int olo, int ohi, int plo, int phi, int alo, int ahi) {
    AdjointTasks k{};
    uint32_t at = 0;
    for (int m = 0; m <= g.depth; ++m) {
        k.start[m] = at;
        if (m < olo || m > ohi) continue;
        const uint32_t wm = g.pw[m];
        const int top = std::min(phi, ahi - m), low = std::max(plo, alo - m);
        const uint32_t terms = low > top ? 1u : g.db[top + 1] - g.db[low];
        // (a warp's sum takes five additions more, dear in FP64)
        if (wm < 32u && (left ? terms * wm : terms) >= (!left && wm >= 8u ? 256u : 64u)) {
            at += left ? 1u : wm;
            continue;
        }
        // about 16 terms a lane
        k.run[m] = 32u * (terms >= 16u ? 1u : terms >= 8u ? 2u : terms >= 4u ? 4u : 8u);
        at += (wm + k.run[m] - 1) / k.run[m];
    }
    k.start[g.depth + 1] = at;
    return k;
}

// acc + sum over i < n, in steps of `step` from `first`, of x[i] y[i ys].  FP32 sums
// blocks of eight first: a chain of hundreds of additions would double the
// rounding error of the general kernel's shorter ones.
template <typename T>
__device__ __forceinline__ T dot(const T* x, const T* y, uint32_t first, uint32_t n, uint32_t step, uint32_t ys, T acc) {
    if constexpr (sizeof(T) == 8) {
#pragma unroll 4
        for (uint32_t i = first; i < n; i += step) acc = fma(x[i], y[i * ys], acc);
    } else {
        uint32_t i = first;
        for (; i + 7u * step < n; i += 8u * step) {
            T part = x[i] * y[i * ys];
#pragma unroll
            for (uint32_t r = 1; r < 8; ++r) part = fma(x[i + r * step], y[(i + r * step) * ys], part);
            acc += part;
        }
        for (; i < n; i += step) acc = fma(x[i], y[i * ys], acc);
    }
    return acc;
}

template <typename T, int W, bool Left>
__global__ void __launch_bounds__(256) k_column_adjoint(Geometry G, TArg<T> out, TArg<T> op, TArg<T> arg,
                                                        int64_t batch, int64_t arg_group, int staged,
                                                        AdjointTasks tasks) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    uint64_t* bar = reinterpret_cast<uint64_t*>(smem_raw);
    T* sm = reinterpret_cast<T*>(smem_raw + kBulkHeader);
    __shared__ uint32_t s_next;
    const uint32_t pd = staged_elems<T>(G.dim);
    uint32_t phase = 0;
    if (staged) bulk_stage_init(bar);
    const int D = G.depth;
    const int ohi = imin(out.hi, D), phi = imin(op.hi, D), ahi = imin(arg.hi, D);
    const uint32_t lane = threadIdx.x & 31u;
    for (int64_t b = blockIdx.x; b < batch; b += gridDim.x) {
        const T* P = op.at(b);
        const T* A = arg.at(arg_group == 1 ? b : b / arg_group);
        T* o = out.at(b);
        if (threadIdx.x == 0) s_next = 0;
        if (staged) {
            BulkStage<T> st(bar, phase);
            P = st.add(sm, P, op.lo, phi, G);
            if (staged == 1) A = st.add(sm + pd, A, arg.lo, ahi, G);
            if (!st.commit(G.fault)) return;
        } else {
            __syncthreads();
        }
        for (;;) {
            uint32_t t = 0;
            if (lane == 0) t = atomicAdd(&s_next, 1u);
            t = __shfl_sync(0xffffffffu, t, 0);
            if (t >= tasks.start[D + 1]) break;
            int m = out.lo;
            while (t >= tasks.start[m + 1]) ++m;
            t -= tasks.start[m];
            const uint32_t run = tasks.run[m];
            const uint32_t wm = G.pw[m];
            const int pmin = imax(op.lo, arg.lo - m), pmax = imin(phi, ahi - m);
            T* om = o + G.db[m];
            if (run == 0u) {
                T acc = T(0);
                if constexpr (Left) {
                    const uint32_t us = 32u / wm, u0 = lane / wm, j = lane - u0 * wm;
                    if (u0 < us)
                        for (int p = pmin; p <= pmax; ++p) {
                            const T* Pp = P + G.db[p];
                            const T* Ap = A + G.db[m + p] + j;
                            acc = dot(Pp, Ap, u0, G.pw[p], us, wm, acc);
                        }
                    for (uint32_t off = wm; off < 32u; off *= 2u) {
                        const T x = __shfl_down_sync(0xffffffffu, acc, off);
                        if (lane + off < 32u) acc += x;
                    }
                    if (lane < wm) om[lane] = acc;
                } else {
                    uint32_t v = lane;  // carried from degree to degree
                    for (int p = pmin; p <= pmax; ++p) {
                        const T* Pp = P + G.db[p];
                        const uint32_t wp = G.pw[p];
                        const T* Ap = A + G.db[m + p] + t * wp;
#pragma unroll 4
                        for (; v < wp; v += 32u) acc = fma(Pp[v], Ap[v], acc);
                        v -= wp;
                    }
#pragma unroll
                    for (uint32_t off = 16u; off > 0u; off /= 2u) acc += __shfl_down_sync(0xffffffffu, acc, off);
                    if (lane == 0) om[t] = acc;
                }
                continue;
            }
            const uint32_t last = (t + 1u) * run, end = last < wm ? last : wm;
            const bool has0 = pmin <= 0 && pmax >= 0, has1 = pmin <= 1 && pmax >= 1;
            const T p0 = has0 ? P[0] : T(0);
            T p1[W];
#pragma unroll
            for (int a = 0; a < W; ++a) p1[a] = has1 ? P[1 + a] : T(0);
            const T* A0 = A + G.db[m];
            const T* A1 = A + G.db[m] + wm;  // degree m + 1
            for (uint32_t j = t * run + lane; j < end; j += 32u) {
                T acc = T(0);
                if (has0) acc = p0 * A0[j];
                if (has1) {
                    T v[W];
#pragma unroll
                    for (int a = 0; a < W; ++a) v[a] = Left ? A1[a * wm + j] : A1[j * W + a];
#pragma unroll
                    for (int a = 0; a < W; ++a) acc = fma(p1[a], v[a], acc);
                }
                for (int p = imax(pmin, 2); p <= pmax; ++p) {
                    const T* Pp = P + G.db[p];
                    const uint32_t wp = G.pw[p];
                    if constexpr (Left) {
                        const T* Ap = A + G.db[m + p] + j;
                        for (uint32_t u = 0; u < wp; u += W, Pp += W, Ap += W * wm) {
                            T part = sizeof(T) == 4 ? T(0) : acc;  // (FP32: blocks first, as in dot())
#pragma unroll
                            for (int a = 0; a < W; ++a) part = fma(Pp[a], Ap[a * wm], part);
                            acc = sizeof(T) == 4 ? acc + part : part;
                        }
                    } else {
                        const T* Ap = A + G.db[m + p] + j * wp;
                        if constexpr ((W & (W - 1)) == 0) {
                            constexpr uint32_t lanes = 128u / sizeof(T);  // of one pass over the banks
                            uint32_t v = (wp <= lanes ? j * wp / lanes : j) & (wp - 1u);
                            constexpr uint32_t block = W < 4 ? 4u : W;  // divides wp = W^p, p >= 2
                            for (uint32_t i = 0; i < wp; i += block) {
                                T part = sizeof(T) == 4 ? T(0) : acc;
#pragma unroll
                                for (uint32_t a = 0; a < block; ++a) {
                                    part = fma(Pp[v], Ap[v], part);
                                    v = (v + 1u) & (wp - 1u);
                                }
                                acc = sizeof(T) == 4 ? acc + part : part;
                            }
                        } else {
                            for (uint32_t v = 0; v < wp; v += W) {
                                T part = sizeof(T) == 4 ? T(0) : acc;
#pragma unroll
                                for (int a = 0; a < W; ++a) part = fma(Pp[v + a], Ap[v + a], part);
                                acc = sizeof(T) == 4 ? acc + part : part;
                            }
                        }
                    }
                }
                om[j] = acc;
            }
        }
        bulk_stage_reuse();
    }
}

}  // namespace

bool column_adjoint_width(int width) { return column_width(width); }

// `staged` as the general launcher chooses it: 0 nothing, 1 both operands, 2 the op.
template <typename T>
cudaError_t launch_column_adjoint(const Geometry& g, const DeviceInfo& dev, cudaStream_t s, bool left, TArg<T> out,
                                  TArg<T> op, TArg<T> arg, int64_t batch, int64_t arg_group, int staged) {
    const size_t one = static_cast<size_t>(staged_elems<T>(g.dim)) * sizeof(T);
    const size_t smem = kBulkHeader + (staged == 1 ? 2 : staged == 2 ? 1 : 0) * one;
    const AdjointTasks tasks = adjoint_tasks(g, left, std::is_same<T, double>::value, out.lo, out.hi, op.lo, std::min(op.hi, g.depth), arg.lo,
                                             std::min(arg.hi, g.depth));
    const int threads = g.dim < 256 ? 64 : g.dim < 2048 ? 128 : 256;
    return with_width(g.width, [&](auto w) {
        constexpr int W = decltype(w)::value;
        if (left)
            return run_column<&k_column_adjoint<T, W, true>>(dev, s, threads, smem, batch, g, out, op, arg, batch,
                                                             arg_group, staged, tasks);
        return run_column<&k_column_adjoint<T, W, false>>(dev, s, threads, smem, batch, g, out, op, arg, batch,
                                                          arg_group, staged, tasks);
    });
}

template cudaError_t launch_column_adjoint<float>(const Geometry&, const DeviceInfo&, cudaStream_t, bool, TArg<float>,
                                                  TArg<float>, TArg<float>, int64_t, int64_t, int);
template cudaError_t launch_column_adjoint<double>(const Geometry&, const DeviceInfo&, cudaStream_t, bool,
                                                   TArg<double>, TArg<double>, TArg<double>, int64_t, int64_t, int);

}  // namespace rpp_gb

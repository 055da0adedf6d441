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
// FP32 sums are formed in short blocks, these in groups and those in chains; FP64
// sums of 12 terms or more have two to eight chains where the general kernel has as
// many threads for a coefficient.  Neither rounds more than its 256 threads a tensor
// do (rms error over both, uniform inputs: FP32 0.6 to 1.06, FP64 0.7 to 1.2 in a
// degree and 1.0 in most; one chain a lane had up to 2.8 times that, W6 D5 degree 0).
// Left / right, general kernel -> this: FP32 W5 D5 batch 4096 111 -> 65 / 117 ->
// 67 us, W8 D4 110 -> 65 / 117 -> 71, W3 D6 (3000) 51 -> 22 / 52 -> 23, W2 D12 (2048)
// 183 -> 109 / 211 -> 137; FP64 W5 D5 221 -> 209 / 233 -> 224, W2 D8 99 -> 48 / 136 ->
// 75, W2 D12 545 -> 426 / 588 -> 518 (with one chain a lane 203 / 211, 47 / 73 and
// 429 / 497).
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

AdjointTasks adjoint_tasks(const Geometry& g, bool left, int olo, int ohi, int plo, int phi, int alo, int ahi) {
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

// A lane's share of a warp's sum.  One chain of the 122 terms that a lane has in
// degree 0 at W5 D5 has twice the general kernel's rounding error (256 threads of 15
// terms), these have the same.  FP32: two chains of blocks of eight terms and two of
// what is left over.  FP64, whose additions are dear: eight chains (`wide`: where a
// lane has 16 terms or more), or one.
template <typename T>
struct LaneSum {
    T block0 = T(0), block1 = T(0), rest0 = T(0), rest1 = T(0);
    __device__ __forceinline__ T total(bool) const { return (block0 + block1) + (rest0 + rest1); }
};
template <>
struct LaneSum<double> {
    double r[8] = {};
    __device__ __forceinline__ double total(bool wide) const {
        return wide ? ((r[0] + r[1]) + (r[2] + r[3])) + ((r[4] + r[5]) + (r[6] + r[7])) : r[0];
    }
};

template <typename T>
__device__ __forceinline__ T eight(const T* x, const T* y, uint32_t i, uint32_t step, uint32_t ys) {
    T part = x[i] * y[i * ys];
#pragma unroll
    for (uint32_t r = 1; r < 8; ++r) part = fma(x[i + r * step], y[(i + r * step) * ys], part);
    return part;
}

// Adds x[i] y[i ys], i = first, first + step, ... below n; returns the i after them.
template <typename T>
__device__ __forceinline__ uint32_t dot(const T* x, const T* y, uint32_t first, uint32_t n, uint32_t step, uint32_t ys,
                                        LaneSum<T>& sum, bool wide) {
    uint32_t i = first;
    if constexpr (sizeof(T) == 8) {
#pragma unroll 1
        for (; wide && i + 7u * step < n; i += 8u * step)
#pragma unroll
            for (uint32_t q = 0; q < 8; ++q) sum.r[q] = fma(x[i + q * step], y[(i + q * step) * ys], sum.r[q]);
#pragma unroll 4
        for (; i < n; i += step) sum.r[0] = fma(x[i], y[i * ys], sum.r[0]);
    } else {
#pragma unroll 1
        for (; i + 15u * step < n; i += 16u * step) {
            sum.block0 += eight(x, y, i, step, ys);
            sum.block1 += eight(x, y, i + 8u * step, step, ys);
        }
        if (i + 7u * step < n) {
            sum.block0 += eight(x, y, i, step, ys);
            i += 8u * step;
        }
#pragma unroll 1
        for (; i + step < n; i += 2u * step) {
            sum.rest0 = fma(x[i], y[i * ys], sum.rest0);
            sum.rest1 = fma(x[i + step], y[(i + step) * ys], sum.rest1);
        }
        if (i < n) {
            sum.rest0 = fma(x[i], y[i * ys], sum.rest0);
            i += step;
        }
    }
    return i;
}

// FP32: acc + the terms of split degree p >= 2 (wp = W^p of them) of one coefficient,
// in blocks of `size` (the multiply-adds that block(part) makes), W blocks to a group,
// and the groups in a chain: 5 + 5 + 5 additions one after another for the 125 terms
// of p = 3 at W5.  Two: the blocks of a group in two chains (wide right sums, whose
// few coefficients had 32 threads each in the general kernel).  Whole: whole groups
// unrolled (narrow right sums; W3 D6 29.7 -> 26.4 us, but left 22.0 -> 23.1).
template <int W, bool Two, bool Whole, typename Block>
__device__ __forceinline__ float grouped(uint32_t wp, float acc, Block&& block) {
    constexpr uint32_t size = W == 2 ? 4u : W, most = W == 2 ? 4u : W;  // (W = 2: two where p = 3, one where 2)
    const uint32_t blocks = wp / size < most ? wp / size : most;
    float sum = 0.0f;
#pragma unroll 1
    for (uint32_t i = 0; i < wp; i += blocks * size) {
        float group = 0.0f;
        if constexpr (Two) {
            float other = 0.0f;
            uint32_t k = 0;
#pragma unroll 1
            for (; k + 1 < blocks; k += 2) {
                group += block(0.0f);
                other += block(0.0f);
            }
            if (k < blocks) group += block(0.0f);
            group += other;
        } else {
            if constexpr (Whole) {
                if (blocks == most) {
#pragma unroll
                    for (uint32_t k = 0; k < most; ++k) group += block(0.0f);
                    sum += group;
                    continue;
                }
            }
#pragma unroll(W == 5 ? 1 : 2)
            for (uint32_t k = 0; k < blocks; ++k) group += block(0.0f);
        }
        sum += group;
    }
    return acc + sum;
}

// FP64: the terms of split degrees plo..phi (plo >= 2) of coefficient j of degree m in
// `chains` chains (2, 4 or 8), the blocks of W terms taken in turn.
template <typename T, int W, bool Left>
__device__ __forceinline__ T spread_sum(const Geometry& G, const T* P, const T* A, int m, uint32_t j, int plo, int phi,
                                        uint32_t wm, uint32_t chains) {
    constexpr uint32_t size = W == 2 ? 4u : W;  // divides W^p, p >= 2
    constexpr bool rotate = !Left && (W & (W - 1)) == 0;
    constexpr uint32_t lanes = 128u / sizeof(T);  // of one pass over the banks
    T r[8] = {};
    for (int p = plo; p <= phi; ++p) {
        const uint32_t wp = G.pw[p];
        const T* Pp = P + G.db[p];
        const T* Ap = A + G.db[m + p] + (Left ? j : j * wp);
        uint32_t v = rotate ? (wp <= lanes ? j * wp / lanes : j) & (wp - 1u) : 0u;
        auto block = [&](auto&& put) {
#pragma unroll
            for (uint32_t a = 0; a < size; ++a) {
                put(a, Pp[v], Ap[Left ? v * wm : v]);
                v = rotate ? (v + 1u) & (wp - 1u) : v + 1u;
            }
        };
        const uint32_t blocks = wp / size;
        if (chains == 2u) {
            for (uint32_t k = 0; k < blocks; ++k) block([&](uint32_t a, T x, T y) { r[a & 1u] = fma(x, y, r[a & 1u]); });
        } else if (chains == 4u) {
            for (uint32_t k = 0; k < blocks; ++k) block([&](uint32_t a, T x, T y) { r[a & 3u] = fma(x, y, r[a & 3u]); });
        } else {
            uint32_t k = 0;
            for (; k + 1u < blocks; k += 2u) {
                block([&](uint32_t a, T x, T y) { r[a & 3u] = fma(x, y, r[a & 3u]); });
                block([&](uint32_t a, T x, T y) { r[4u + (a & 3u)] = fma(x, y, r[4u + (a & 3u)]); });
            }
            if (k < blocks) block([&](uint32_t a, T x, T y) { r[a & 3u] = fma(x, y, r[a & 3u]); });
        }
    }
    if (chains == 2u) return r[0] + r[1];
    if (chains == 4u) return (r[0] + r[1]) + (r[2] + r[3]);
    return ((r[0] + r[1]) + (r[2] + r[3])) + ((r[4] + r[5]) + (r[6] + r[7]));
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
    bulk_stage_init(bar);
    const int D = G.depth;
    const int ohi = imin(out.hi, D), phi = imin(op.hi, D), ahi = imin(arg.hi, D);
    const uint32_t lane = threadIdx.x & 31u;
    for (int64_t b = blockIdx.x; b < batch; b += gridDim.x) {
        const T* P = op.at(b);
        const T* A = arg.at(arg_group == 1 ? b : b / arg_group);
        T* o = out.at(b);
        if (threadIdx.x == 0) s_next = 0;
        BulkStage<T> st(bar, phase);
        P = st.add(sm, P, op.lo, phi, G);
        if (staged == 1) A = st.add(sm + pd, A, arg.lo, ahi, G);
        if (!st.commit(G.fault)) return;
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
                LaneSum<T> sum;
                const bool wide = sizeof(T) == 8 && pmin <= pmax &&
                                  G.db[pmax + 1] - G.db[pmin] >= 16u * (Left ? 32u / wm : 32u);
                if constexpr (Left) {
                    const uint32_t us = 32u / wm, u0 = lane / wm, j = lane - u0 * wm;
                    if (u0 < us)
                        for (int p = pmin; p <= pmax; ++p) {
                            const T* Pp = P + G.db[p];
                            const T* Ap = A + G.db[m + p] + j;
                            dot(Pp, Ap, u0, G.pw[p], us, wm, sum, wide);
                        }
                    T acc = sum.total(wide);
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
                        v = dot(Pp, Ap, v, wp, 32u, 1u, sum, wide) - wp;
                    }
                    T acc = sum.total(wide);
#pragma unroll
                    for (uint32_t off = 16u; off > 0u; off /= 2u) acc += __shfl_down_sync(0xffffffffu, acc, off);
                    if (lane == 0) om[t] = acc;
                }
                continue;
            }
            const uint32_t last = (t + 1u) * run, end = last < wm ? last : wm;
            // FP64: where the general kernel has several threads for a coefficient of many
            // terms, its sum has several chains here
            const uint32_t terms = pmin <= pmax ? G.db[pmax + 1] - G.db[pmin] : 0u;
            const bool spread = sizeof(T) == 8 && wm < 200u && terms >= 12u;
            const uint32_t chains = wm >= 100u || terms < 24u ? 2u : terms < 64u ? 4u : 8u;
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
                    if (W >= 5 && (sizeof(T) == 4 || spread)) {  // two shorter chains
                        T odd = T(0);
#pragma unroll
                        for (int a = 0; a < W; ++a) (a & 1 ? odd : acc) = fma(p1[a], v[a], a & 1 ? odd : acc);
                        acc += odd;
                    } else {
#pragma unroll
                        for (int a = 0; a < W; ++a) acc = fma(p1[a], v[a], acc);
                    }
                }
                if constexpr (sizeof(T) == 8) {
                    if (spread) {
                        om[j] = acc + spread_sum<T, W, Left>(G, P, A, m, j, imax(pmin, 2), pmax, wm, chains);
                        continue;
                    }
                }
                for (int p = imax(pmin, 2); p <= pmax; ++p) {
                    const T* Pp = P + G.db[p];
                    const uint32_t wp = G.pw[p];
                    const T* Ap = Left ? A + G.db[m + p] + j : A + G.db[m + p] + j * wp;
                    constexpr bool two = sizeof(T) == 4 && W >= 7;
                    if constexpr (Left) {
                        auto block = [&](T part) {
                            constexpr int size = sizeof(T) == 4 && W == 2 ? 4 : W;
#pragma unroll
                            for (int a = 0; a < size; ++a) part = fma(Pp[a], Ap[a * wm], part);
                            Pp += size, Ap += size * wm;
                            return part;
                        };
                        if constexpr (sizeof(T) == 4)
                            acc = grouped<W, false, false>(wp, acc, block);
                        else
                            for (uint32_t u = 0; u < wp; u += W) acc = block(acc);
                    } else if constexpr ((W & (W - 1)) == 0) {
                        constexpr uint32_t lanes = 128u / sizeof(T);  // of one pass over the banks
                        uint32_t v = (wp <= lanes ? j * wp / lanes : j) & (wp - 1u);
                        constexpr uint32_t size = W < 4 ? 4u : W;  // divides wp = W^p, p >= 2
                        auto block = [&](T part) {
                            T odd = T(0);
#pragma unroll
                            for (uint32_t a = 0; a < size; ++a) {
                                T& chain = two && (a & 1u) ? odd : part;
                                chain = fma(Pp[v], Ap[v], chain);
                                v = (v + 1u) & (wp - 1u);
                            }
                            return two ? part + odd : part;
                        };
                        if constexpr (sizeof(T) == 4)
                            acc = grouped<W, two, W <= 4>(wp, acc, block);
                        else
                            for (uint32_t i = 0; i < wp; i += size) acc = block(acc);
                    } else {
                        uint32_t v = 0;
                        auto block = [&](T part) {
                            T odd = T(0);
#pragma unroll
                            for (int a = 0; a < W; ++a) {
                                T& chain = two && (a & 1) ? odd : part;
                                chain = fma(Pp[v + a], Ap[v + a], chain);
                            }
                            v += W;
                            return two ? part + odd : part;
                        };
                        if constexpr (sizeof(T) == 4)
                            acc = grouped<W, two, W <= 4>(wp, acc, block);
                        else
                            while (v < wp) acc = block(acc);
                    }
                }
                om[j] = acc;
            }
        }
        bulk_stage_reuse();
    }
}

}  // namespace

// Where it is the faster kernel (the op staged).  Tensors of fewer than 64
// coefficients are a few warp tasks here, one warp each in the general kernel, which
// many of them fill the SMs with better (W2 D5 batch 4096: FP64 left 13.7 us, 33.9
// here; FP32 right 8.7, 14.4; batch 320 FP64 left 0.94 of its time); not for the
// right adjoint of the smallest FP64 tensors (W4 D3 batch 8192: 24 us, 28 here) and
// of W4 from depth 5 on (D6, 732: 84, 101); nor for FP64 left W6 D5, whose argument
// is not staged, where few tensors leave its longest tasks to the end (320: 1.24
// times the general kernel's).
template <typename T>
bool column_adjoint_pays(const Geometry& g, const DeviceInfo& dev, bool left, int staged, int64_t batch) {
    if (!column_width(g.width)) return false;
    const int64_t sms = dev.sm_count;
    const bool wide_flat = g.width >= 6 && g.depth == 2;
    if (std::is_same<T, double>::value) {
        if (!left) return g.dim >= 128 && !(g.width == 4 && g.depth >= 5);
        if (g.dim < 64 && (batch * g.dim >= 184 * sms || g.width == 7 && g.depth == 2)) return false;
        return !(staged == 2 && g.width == 6 && batch < 4 * sms);
    }
    if (g.dim >= 64) return true;
    if (left) return wide_flat || batch < 13 * sms;
    return batch < (g.dim >= 30 ? 8 : 13) * sms;
}
template bool column_adjoint_pays<float>(const Geometry&, const DeviceInfo&, bool, int, int64_t);
template bool column_adjoint_pays<double>(const Geometry&, const DeviceInfo&, bool, int, int64_t);

// `staged` as the general launcher chooses it: 1 both operands, 2 the op.
template <typename T>
cudaError_t launch_column_adjoint(const Geometry& g, const DeviceInfo& dev, cudaStream_t s, bool left, TArg<T> out,
                                  TArg<T> op, TArg<T> arg, int64_t batch, int64_t arg_group, int staged) {
    const size_t one = static_cast<size_t>(staged_elems<T>(g.dim)) * sizeof(T);
    const size_t smem = kBulkHeader + (staged == 1 ? 2 : 1) * one;
    const AdjointTasks tasks = adjoint_tasks(g, left, out.lo, out.hi, op.lo, std::min(op.hi, g.depth), arg.lo,
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

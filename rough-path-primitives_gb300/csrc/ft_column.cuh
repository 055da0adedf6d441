// ft_column.cuh -- truncated products for compile-time widths, a column of
// coefficients per thread.
//
// A coefficient of a product is out[n][w] = sum_k L[n-k][prefix] R[k][suffix].
// One coefficient per thread costs an index split, two shared-memory loads
// and their addressing per multiply-add (about twelve instructions), which
// bounds it in FP32.  Here a thread owns the NC = W^SC coefficients of level n
// that share all but their first SC letters (word c s, c running over the
// first letters): for a split k inside s they share the right factor and the
// index split, so NC + 1 loads serve NC multiply-adds.  Lanes hold consecutive
// s, so the right factor's loads and the result's stores are consecutive, the
// left factor's are shared by the lanes of a prefix, and nothing conflicts for
// any width.  The splits run in increasing k, as in ft_device.cuh's split_sum:
// the same multiply-adds in the same order, so the results are the same bits.
#pragma once

#include <type_traits>

#include "common.cuh"
#include "ft_device.cuh"
#include "launch_util.cuh"

namespace rpp_gb {
namespace ftcol {

using ftdev::Opnd;

constexpr uint32_t ipow(uint32_t w, int n) {
    uint32_t r = 1;
    for (int i = 0; i < n; ++i) r *= w;
    return r;
}

// First letters of a column, and the coefficients they make (4 to 9).
template <int W>
struct Column {
    static constexpr int SC = W == 2 ? 3 : W == 3 ? 2 : 1;
    static constexpr uint32_t NC = ipow(W, SC);
};

// Widths with an instantiation.
constexpr bool column_width(int w) { return w >= 2 && w <= 8; }

// Tasks of level n: a column per suffix of the levels of at least SC letters,
// a single coefficient per word of the others.
template <int W>
__host__ __device__ __forceinline__ uint32_t level_tasks(const Geometry& G, int n) {
    return n >= Column<W>::SC ? G.pw[n - Column<W>::SC] : G.pw[n];
}
template <int W>
__host__ __device__ __forceinline__ uint32_t tensor_tasks(const Geometry& G, int lo, int hi) {
    uint32_t t = 0;
    for (int n = lo; n <= hi; ++n) t += level_tasks<W>(G, n);
    return t;
}

// Task i of the levels [lo, hi] of `per` tensors, top level first: the level,
// the tensor and the task's place in its level.
template <int W>
__device__ __forceinline__ void locate_task(const Geometry& G, uint32_t i, uint32_t per, int hi, int& n,
                                            uint32_t& tensor, uint32_t& place) {
    n = hi;
    uint32_t tasks = level_tasks<W>(G, n);
    while (i >= tasks * per) {
        i -= tasks * per;
        --n;
        tasks = level_tasks<W>(G, n);
    }
    tensor = per == 1 ? 0u : i / tasks;
    place = per == 1 ? i : i % tasks;
}

// One column: acc[c] += the splits k in [kmin, kmax] of L (x) R at the words
// c s of level n (n >= SC).
template <typename T, int W>
__device__ __forceinline__ void column_sum(const Geometry& G, const T* __restrict__ L, const T* __restrict__ R, int n,
                                           uint32_t s, int kmin, int kmax, T (&acc)[Column<W>::NC]) {
    constexpr int SC = Column<W>::SC;
    constexpr uint32_t NC = Column<W>::NC;
    // splits inside the suffix: q = s / W^k, r = s % W^k
    uint32_t q = s, r = 0, p = 1;
    const int kend = imin(kmax, n - SC);
    for (int k = 0; k <= kend; ++k) {
        if (k >= kmin) {
            const T* Lp = L + G.db[n - k] + q;
            const T rv = R[G.db[k] + r];
            const uint32_t ls = G.pw[n - k - SC];
            T lv[NC];
#pragma unroll
            for (uint32_t c = 0; c < NC; ++c) lv[c] = Lp[c * ls];
#pragma unroll
            for (uint32_t c = 0; c < NC; ++c) acc[c] = fma(lv[c], rv, acc[c]);
        }
        const uint32_t qq = q / W;
        r += (q - qq * W) * p;
        p *= W;
        q = qq;
    }
    // splits inside the first letters: the last j of them go right
    const uint32_t ws = G.pw[n - SC];
#pragma unroll
    for (int j = 1; j <= SC; ++j) {
        const int k = n - SC + j;
        if (k < kmin || k > kmax) continue;
        const uint32_t w = ipow(W, j);
        const T* Lp = L + G.db[SC - j];
        const T* Rp = R + G.db[k] + s;
#pragma unroll
        for (uint32_t c = 0; c < NC; ++c) acc[c] = fma(Lp[c / w], Rp[(c % w) * ws], acc[c]);
    }
}

// The coefficients of one task of L (x) R at level n, given to store(index in
// the level, value).
template <typename T, int W, typename Store>
__device__ __forceinline__ void task_product(const Geometry& G, const Opnd<T>& L, const Opnd<T>& R, int n,
                                             uint32_t place, Store&& store) {
    constexpr uint32_t NC = Column<W>::NC;
    if (n >= Column<W>::SC) {
        const int kmin = imax(imax(R.lo, 0), n - L.hi);
        const int kmax = imin(imin(R.hi, n), n - L.lo);
        T acc[NC];
#pragma unroll
        for (uint32_t c = 0; c < NC; ++c) acc[c] = T(0);
        column_sum<T, W>(G, L.p, R.p, n, place, kmin, kmax, acc);
        const uint32_t ws = G.pw[n - Column<W>::SC];
#pragma unroll
        for (uint32_t c = 0; c < NC; ++c) store(c * ws + place, acc[c]);
    } else {
        store(place, ftdev::split_sum<false>(G, L, R, n, place));
    }
}

// One launch over `groups` CTAs' worth of work, as many at once as fit.
template <auto kernel, typename... Args>
inline cudaError_t run_column(const DeviceInfo& dev, cudaStream_t s, int threads, size_t smem, int64_t groups,
                      Args... args) {
    cudaError_t err = allow_large_smem<kernel>(dev);
    if (err != cudaSuccess) return err;
    dim3 grid;
    if ((err = batch_grid(kernel, dev, threads, smem, groups, grid)) != cudaSuccess) return err;
    kernel<<<grid, threads, smem, s>>>(args...);
    return cudaGetLastError();
}

// f(std::integral_constant<int, W>) for a width with an instantiation.
template <typename F>
inline cudaError_t with_width(int w, F&& f) {
    switch (w) {
        case 2: return f(std::integral_constant<int, 2>{});
        case 3: return f(std::integral_constant<int, 3>{});
        case 4: return f(std::integral_constant<int, 4>{});
        case 5: return f(std::integral_constant<int, 5>{});
        case 6: return f(std::integral_constant<int, 6>{});
        case 7: return f(std::integral_constant<int, 7>{});
        case 8: return f(std::integral_constant<int, 8>{});
        default: return cudaErrorInvalidConfiguration;
    }
}

}  // namespace ftcol
}  // namespace rpp_gb

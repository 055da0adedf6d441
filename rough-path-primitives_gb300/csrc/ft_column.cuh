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

#include <algorithm>
#include <type_traits>

#include "bulk_stage.cuh"
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

// First letters of a column, and the coefficients they make.  FP32 (3 to 9) is
// bound by loads and index arithmetic, which long columns save; FP64 by its
// pipe, whose lanes short columns fill better (W3 D6: 81 columns of 9 on the
// top level, or 243 of 3).
template <typename T, int W>
struct Column {
    static constexpr int SC = sizeof(T) == 8 ? (W == 2 ? 2 : 1) : (W == 2 ? 3 : W == 3 ? 2 : 1);
    static constexpr uint32_t NC = ipow(W, SC);
};

// Widths with an instantiation.
constexpr bool column_width(int w) { return w >= 2 && w <= 8; }

// Tasks of level n: a column per suffix of the levels of at least SC letters,
// a single coefficient per word of the others.
template <typename T, int W>
__host__ __device__ __forceinline__ uint32_t level_tasks(const Geometry& G, int n) {
    return n >= Column<T, W>::SC ? G.pw[n - Column<T, W>::SC] : G.pw[n];
}
template <typename T, int W>
__host__ __device__ __forceinline__ uint32_t tensor_tasks(const Geometry& G, int lo, int hi) {
    uint32_t t = 0;
    for (int n = lo; n <= hi; ++n) t += level_tasks<T, W>(G, n);
    return t;
}

// Task i of the levels [lo, hi] of `per` tensors, top level first: the level,
// the tensor and the task's place in its level.
template <typename T, int W>
__device__ __forceinline__ void locate_task(const Geometry& G, uint32_t i, uint32_t per, int hi, int& n,
                                            uint32_t& tensor, uint32_t& place) {
    n = hi;
    uint32_t tasks = level_tasks<T, W>(G, n);
    while (i >= tasks * per) {
        i -= tasks * per;
        --n;
        tasks = level_tasks<T, W>(G, n);
    }
    tensor = per == 1 ? 0u : i / tasks;
    place = per == 1 ? i : i % tasks;
}

// One column: acc[c] += the splits k in [kmin, kmax] of L (x) R at the words
// c s of level n (n >= SC).
template <typename T, int W>
__device__ __forceinline__ void column_sum(const Geometry& G, const T* __restrict__ L, const T* __restrict__ R, int n,
                                           uint32_t s, int kmin, int kmax, T (&acc)[Column<T, W>::NC]) {
    constexpr int SC = Column<T, W>::SC;
    constexpr uint32_t NC = Column<T, W>::NC;
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
    constexpr uint32_t NC = Column<T, W>::NC;
    if (n >= Column<T, W>::SC) {
        const int kmin = imax(imax(R.lo, 0), n - L.hi);
        const int kmax = imin(imin(R.hi, n), n - L.lo);
        T acc[NC];
#pragma unroll
        for (uint32_t c = 0; c < NC; ++c) acc[c] = T(0);
        column_sum<T, W>(G, L.p, R.p, n, place, kmin, kmax, acc);
        const uint32_t ws = G.pw[n - Column<T, W>::SC];
#pragma unroll
        for (uint32_t c = 0; c < NC; ++c) store(c * ws + place, acc[c]);
    } else {
        store(place, ftdev::split_sum<false>(G, L, R, n, place));
    }
}

// exp or log of X (levels X.lo >= 1 .. X.hi, in shared memory) to degree H by
// Horner's rule.  Round d = H .. 1 multiplies the running tensor by X; what the
// later rounds read of it, and so what a round forms, are its levels up to
// H - d + 1 only -- 22 k multiply-adds at W5 D5 in all, where rounds over whole
// tensors take 57 k.  The running tensor alternates between two buffers of the
// levels below H, one barrier a round; the last round's coefficients go to
// store(n, index in the level, value), n = 1 .. H.  exp runs ft_device.cuh's
// rescaled recursion (up to its depth limit) and divides by H! before the last
// round, in what that round reads: the levels below H, not all of them.
// Returns the result's level 0.  Ends with a barrier.
template <typename T, int W, bool Log, typename Store>
__device__ __forceinline__ T horner(const Geometry& G, int H, const Opnd<T>& X, T* cur, T* next, Store&& store) {
    const auto& rc = ftdev::recip<T>();
    const bool scaled = !Log && H <= ftdev::kScaledHornerMaxDepth;
    T c = T(1);  // level 0 of the running tensor
    if (Log) c = H > 0 ? (H % 2 == 0 ? -rc.inv[H] : rc.inv[H]) : T(0);
    if (threadIdx.x == 0) cur[0] = c;
    __syncthreads();
    for (int d = H; d > 0; --d) {
        const int t = H - d + 1;
        const uint32_t tasks = tensor_tasks<T, W>(G, 1, t);
        const Opnd<T> L{cur, 0, t - 1}, R{X.p, X.lo, imin(X.hi, t)};
        if (Log) c = d > 1 ? ((d - 1) % 2 == 0 ? -rc.inv[d - 1] : rc.inv[d - 1]) : T(0);
        else if (scaled) c *= rc.num[d];
        for (uint32_t i = threadIdx.x; i < tasks; i += blockDim.x) {
            int n;
            uint32_t tensor, place;
            locate_task<T, W>(G, i, 1, t, n, tensor, place);
            task_product<T, W>(G, L, R, n, place, [&](uint32_t at, T v) {
                if (d == 1) {
                    store(n, at, v);
                    return;
                }
                if constexpr (!Log) {
                    // (wider tensors of that depth are not held in shared memory)
                    if (W == 2 && !scaled) v *= rc.inv[d];
                    if (scaled && d == 2) v *= rc.inv_fact[H];
                }
                next[G.db[n] + at] = v;
            });
        }
        if (threadIdx.x == 0 && d > 1) next[0] = scaled && d == 2 ? c * rc.inv_fact[H] : c;
        __syncthreads();
        T* swap = cur;
        cur = next;
        next = swap;
    }
    return scaled ? c * rc.inv_fact[H] : c;  // (log: 0)
}

// log with the whole result in X's buffer `x` (levels 0 .. H).
// `buf`: both running buffers, `half` elements each.  Level H replaces X's,
// which only its coefficients' own threads read; the levels below go to the
// buffer that the last round does not read, and from there to x.  Ends with a
// barrier.
template <typename T, int W>
__device__ __forceinline__ void log_in_place(const Geometry& G, int H, T* x, int xlo, int xhi, T* buf,
                                             uint32_t half) {
    // the last round reads the buffer of its parity and may fill the other
    T* low = (H & 1) ? buf + half : buf;
    const T unit = horner<T, W, true>(G, H, Opnd<T>{x, xlo, xhi}, buf, buf + half, [&](int n, uint32_t at, T v) {
        (n == H ? x : low)[G.db[n] + at] = v;
    });
    const uint32_t below = G.db[H];
    for (uint32_t i = threadIdx.x; i < below; i += blockDim.x) x[i] = i == 0 ? unit : low[i];
    if (H == 0 && threadIdx.x == 0) x[0] = unit;
    __syncthreads();
}

// o's degrees [olo, ohi] = M (x) exp(X), M (levels mlo >= olo .. mhi) and X (xlo >= 1
// .. xhi) staged, by Horner's rule on the multiplier: p_d = M + p_{d+1} (x) X / d, d =
// ohi - mlo .. 1.  X has no degree 0, so round d forms the levels up to ohi - d + 1
// only, the ones that later rounds read, as exp's rounds do: 22 k multiply-adds at W5
// D5, where exp and one product take 41 k and carry the rounding of exp's coefficients
// into the result.  The last and largest round divides by 1, so exp's rescaling, which
// would round M itself, saves nothing here.  The running tensor alternates between two
// buffers of the levels below ohi, one barrier a round.
template <typename T, int W>
__device__ __forceinline__ void horner_multiplied(const Geometry& G, T* o, int olo, int ohi, const T* m, int mlo,
                                                  int mhi, const Opnd<T>& X, T* cur, T* next) {
    const auto& rc = ftdev::recip<T>();
    const bool empty = mlo > mhi || mlo > ohi;
    const uint32_t below = G.db[empty ? ohi + 1 : mlo];
    for (uint32_t i = G.db[olo] + threadIdx.x; i < below; i += blockDim.x) o[i] = T(0);
    if (empty) return;
    const int H = ohi - mlo;
    T* start = H > 0 ? cur : o;  // (no exponent reaches the multiplier's only level)
    for (uint32_t i = G.db[mlo] + threadIdx.x; i < G.db[mlo + 1]; i += blockDim.x) start[i] = m[i];
    __syncthreads();
    for (int d = H; d > 0; --d) {
        const int t = ohi - d + 1;
        const uint32_t tasks = tensor_tasks<T, W>(G, mlo, t);
        const Opnd<T> L{cur, mlo, t - 1}, R{X.p, X.lo, imin(X.hi, t - mlo)};
        const T inv = rc.inv[d];
        T* to = d > 1 ? next : o;
        for (uint32_t i = threadIdx.x; i < tasks; i += blockDim.x) {
            int n;
            uint32_t tensor, place;
            locate_task<T, W>(G, i, 1, t, n, tensor, place);
            const T* mn = n <= mhi ? m + G.db[n] : nullptr;
            T* row = to + G.db[n];
            task_product<T, W>(G, L, R, n, place, [&](uint32_t at, T v) {
                if (d > 1) row[at] = mn ? fma(v, inv, mn[at]) : v * inv;
                else row[at] = mn ? v + mn[at] : v;
            });
        }
        __syncthreads();
        T* swap = cur;
        cur = next;
        next = swap;
    }
}

constexpr int kHornerThreads = 512;
// CTAs of kHornerThreads whose registers fit an SM: the rounds' barriers want
// many warps more than registers (42 a thread, W5 D5 FP64 log 189 us; 96 a
// thread, 248 us), except where the columns then spill.
template <typename T, int W>
constexpr int kHornerBlocks = sizeof(T) == 8 && W >= 6 ? 2 : 3;
constexpr size_t kHornerSmemLimit = 200 * 1024;

// A thread per task of a tensor (one warp for the smallest, whose rounds then
// wait for nobody), at most 256 while two CTAs fit an SM.
template <typename T, int W>
inline int horner_threads(const Geometry& g, size_t smem) {
    const uint32_t tasks = (tensor_tasks<T, W>(g, 0, g.depth) + 31) / 32 * 32;
    return static_cast<int>(std::min<uint32_t>(tasks, smem > 110 * 1024 ? kHornerThreads : 256u));
}

inline bool horner_fits(const Geometry& g, const DeviceInfo& dev, size_t smem) {
    return column_width(g.width) && g.depth >= 1 &&
           smem <= std::min(kHornerSmemLimit, static_cast<size_t>(dev.max_smem_optin));
}

// Where columns are the faster way.  A thread of them does the work of W to W^2
// threads of the general kernels one after another, so few tensors, an SM each or
// less, take longer on columns until a tensor alone has threads' worth of them
// (`alone` coefficients) or the batch does (`filled` coefficients an SM, of tensors
// of at least `least`; `many` tensors an SM of any size).  Each field at W = 2, at
// W = 3 and 4, and at W >= 5, where the columns are W coefficients long.  The lines
// are where the two kernels' times cross, at W 2..8, every depth to 6 000
// coefficients and batches of 1 to 4 096 on 152 SMs; on their far side the columns
// were up to 2.5 times slower (left adjoint FP64 W2 D5, 4 096: 13.7 -> 33.9 us), near them
// either kernel is within 5 %.
struct Worth {
    uint32_t alone[3], filled[3], least;
    uint32_t many[3] = {~0u, ~0u, ~0u};
};
constexpr uint32_t kNever = ~0u;
inline bool worth(const Worth& w, const Geometry& g, const DeviceInfo& dev, int64_t batch) {
    const int c = g.width == 2 ? 0 : g.width <= 4 ? 1 : 2;
    if (g.dim >= w.alone[c] || batch >= static_cast<int64_t>(w.many[c]) * dev.sm_count) return true;
    return g.dim >= w.least && batch * g.dim >= static_cast<int64_t>(w.filled[c]) * dev.sm_count;
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

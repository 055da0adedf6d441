// lie_column.cu -- the log-signature epilogue and the Lie-increment step
// (lie_fused.cu) for widths 2..8, on columns of coefficients (ft_column.cuh).
#include <algorithm>
#include <type_traits>

#include "bulk_stage.cuh"
#include "common.cuh"
#include "ft_column.cuh"
#include "launch_util.cuh"
#include "ops.hpp"
#include "sell.cuh"

namespace rpp_gb {
namespace {

using namespace ftcol;

// out = alpha * T2L * log(x) (lie_fused.cu's k_log_to_lie, the log's view from
// degree 0).  Batch 4096, before -> now: FP32 W5 D5 147 -> 83 us, W8 D4 139 -> 74;
// FP64 W2 D8 131 -> 103, W3 D6 (3 000) 98 -> 94, W5 D5 291 -> 285.
template <typename T, int W>
__global__ void __launch_bounds__(kHornerThreads, (kHornerBlocks<T, W>)) k_column_log_to_lie(Geometry G, CsrDevice m, TArg<T> x, int hi,
                                                                      T* out, int64_t out_stride, int64_t out_size,
                                                                      int64_t batch, T alpha) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    uint64_t* bar = reinterpret_cast<uint64_t*>(smem_raw);
    const uint32_t half = staged_elems<T>(G.db[G.depth]);
    T* buf = reinterpret_cast<T*>(smem_raw + kBulkHeader);
    T* s_x = buf + 2 * half;
    uint32_t phase = 0;
    bulk_stage_init(bar);
    const int xlo = imax(1, x.lo), xhi = imin(x.hi, hi);
    for (int64_t b = blockIdx.x; b < batch; b += gridDim.x) {
        BulkStage<T> st(bar, phase);
        T* X = st.add(s_x, x.at(b), xlo, xhi, G);
        if (!st.commit(G.fault)) return;
        log_in_place<T, W>(G, hi, X, xlo, xhi, buf, half);
        sell_rows<true, true>(m, X, out + b * out_stride, out_size, alpha);  // t2l: long rows
        bulk_stage_reuse();
    }
}

// X = alpha * L2T * lambda on degrees [lo, hi], out = exp(X) or M (x) exp(X)
// (lie_fused.cu's k_lie_exp).  With a multiplier, W5 D5 batch 4096: FP64 777 -> 395
// us, FP32 419 -> 150; W3 D6 (3 000) FP64 226 -> 112; rounding error against 128 bits
// 0.6 to 0.8 of the general kernel's.  FP64 W5 D5: that pipe 71 % busy, 7.5 of 20 stalled
// cycles an instruction on shared memory, 3.5 at barriers, three CTAs an SM.
template <typename T, int W>
__global__ void __launch_bounds__(kHornerThreads, (kHornerBlocks<T, W>)) k_column_lie_exp(Geometry G, CsrDevice mat, const T* lie,
                                                                   int64_t lie_stride, int lo, int hi, TArg<T> out,
                                                                   TArg<T> m, int64_t batch, T alpha, uint32_t room) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    uint64_t* bar = reinterpret_cast<uint64_t*>(smem_raw);
    const uint32_t pd = staged_elems<T>(G.dim), half = staged_elems<T>(G.db[G.depth]);
    T* buf = reinterpret_cast<T*>(smem_raw + kBulkHeader);  // the Lie vector, until X is formed
    T* X = buf + room;
    T* s_m = X + pd;
    uint32_t phase = 0;
    bulk_stage_init(bar);
    const int ohi = imin(out.hi, G.depth);
    const bool fm = m.p != nullptr;
    const int mlo = imax(m.lo, out.lo), mhi = imin(m.hi, ohi);
    const int H = fm ? imax(0, ohi - mlo) : ohi;
    const int xlo = imax(1, lo), xhi = imin(hi, H);
    const uint32_t view = G.db[hi + 1] - G.db[lo];
    for (int64_t b = blockIdx.x; b < batch; b += gridDim.x) {
        BulkStage<T> st(bar, phase);
        const T* l = st.add_span(buf, lie + b * lie_stride, 0, static_cast<uint32_t>(mat.cols_dim));
        const T* M = fm ? st.add(s_m, m.at(b), mlo, mhi, G) : nullptr;
        for (uint32_t i = threadIdx.x; i < G.dim; i += blockDim.x) X[i] = T(0);
        if (!st.commit(G.fault)) return;
        sell_rows<true, false>(mat, l, X + G.db[lo], static_cast<int64_t>(view), alpha);  // l2t: short rows
        __syncthreads();
        T* o = out.at(b);
        if (fm) {
            horner_multiplied<T, W>(G, o, out.lo, ohi, M, mlo, mhi, Opnd<T>{X, xlo, xhi}, buf, buf + half);
        } else {
            const T unit = horner<T, W, false>(G, H, Opnd<T>{X, xlo, xhi}, buf, buf + half,
                                               [&](int n, uint32_t at, T v) { o[G.db[n] + at] = v; });
            if (threadIdx.x == 0) o[0] = unit;
        }
        bulk_stage_reuse();
    }
}

// `room`: the running buffers, which hold the Lie vector before.
template <typename T>
uint32_t lie_room(const Geometry& g, int64_t vector) {
    return std::max(2 * staged_elems<T>(g.db[g.depth]), staged_elems<T>(static_cast<uint32_t>(vector)));
}
template <typename T>
size_t lie_smem(const Geometry& g, bool multiplier, uint32_t room) {
    return kBulkHeader + (room + (multiplier ? 2 : 1) * static_cast<size_t>(staged_elems<T>(g.dim))) * sizeof(T);
}

}  // namespace

template <typename T>
bool column_log_to_lie_fits(const Geometry& g, const DeviceInfo& dev, int lo, int64_t batch) {
    constexpr Worth k32{{64, 125, 700}, {658, 526, 1118}, 41}, k64{{500, 125, 2000}, {kNever, 1316, 1974}, 0};
    constexpr bool fp64 = std::is_same<T, double>::value;
    // (FP64 at W8, and deep tensors of W6 and W7, where t2l's rows are most of the
    // time: W6 D4 batch 4096 1.23 times the general kernel's, W7 D4 1.12)
    if (fp64 && (g.width == 8 || (g.width >= 6 && g.dim > 500))) return false;
    return lo == 0 && worth(fp64 ? k64 : k32, g, dev, batch) && horner_fits(g, dev, lie_smem<T>(g, false, lie_room<T>(g, 0)));
}

template <typename T>
cudaError_t launch_column_log_to_lie(const Geometry& g, const DeviceInfo& dev, cudaStream_t s, const CsrDevice& m,
                                     TArg<T> x, int hi, T* out, int64_t out_stride, int64_t out_size, int64_t batch,
                                     double alpha) {
    const size_t smem = lie_smem<T>(g, false, lie_room<T>(g, 0));
    const T al = static_cast<T>(alpha);
    return with_width(g.width, [&](auto w) {
        constexpr int W = decltype(w)::value;
        return run_column<&k_column_log_to_lie<T, W>>(dev, s, horner_threads<T, W>(g, smem), smem, batch, g, m, x, hi, out,
                                                      out_stride, out_size, batch, al);
    });
}

template <typename T>
bool column_lie_exp_fits(const Geometry& g, const DeviceInfo& dev, const CsrDevice& m, const TArg<T>& out,
                         bool multiplier, int lo, int hi, int64_t batch) {
    constexpr bool fp64 = std::is_same<T, double>::value;
    constexpr Worth kExp32{{150, 500, 700}, {526, 855, 1316}, 41}, kExp64{{150, 150, 700}, {0, 0, 1974}, 0};
    constexpr Worth kFmexp32{{40, 500, 700}, {263, 1053, 1053}, 0}, kFmexp64{{100, 100, 700}, {0, 0, 1600}, 0};
    if (!worth(multiplier ? (fp64 ? kFmexp64 : kFmexp32) : (fp64 ? kExp64 : kExp32), g, dev, batch)) return false;
    // (an exponent without degree one: see column_horner_fits)
    if (multiplier && (lo > 1 || hi < 1)) return false;
    // (the smallest FP64 tensors, one warp each, gain nothing: W4 D3 37 us, 35 with the general kernel)
    if (fp64 && g.dim < 128) return false;
    return out.lo <= out.hi && (multiplier || out.lo == 0) && m.cols_dim <= static_cast<int64_t>(g.dim) &&
           horner_fits(g, dev, lie_smem<T>(g, multiplier, lie_room<T>(g, m.cols_dim)));
}

template <typename T>
cudaError_t launch_column_lie_exp(const Geometry& g, const DeviceInfo& dev, cudaStream_t s, const CsrDevice& m,
                                  const T* lie, int64_t lie_stride, int lo, int hi, TArg<T> out, TArg<T> mult,
                                  int64_t batch, double alpha) {
    const uint32_t room = lie_room<T>(g, m.cols_dim);
    const size_t smem = lie_smem<T>(g, mult.p != nullptr, room);
    const T al = static_cast<T>(alpha);
    return with_width(g.width, [&](auto w) {
        constexpr int W = decltype(w)::value;
        return run_column<&k_column_lie_exp<T, W>>(dev, s, horner_threads<T, W>(g, smem), smem, batch, g, m, lie,
                                                   lie_stride, lo, hi, out, mult, batch, al, room);
    });
}

#define RPP_GB_INSTANTIATE_LIE_COLUMN(T)                                                                              \
    template bool column_log_to_lie_fits<T>(const Geometry&, const DeviceInfo&, int, int64_t);                               \
    template cudaError_t launch_column_log_to_lie<T>(const Geometry&, const DeviceInfo&, cudaStream_t,              \
                                                     const CsrDevice&, TArg<T>, int, T*, int64_t, int64_t, int64_t, \
                                                     double);                                                       \
    template bool column_lie_exp_fits<T>(const Geometry&, const DeviceInfo&, const CsrDevice&, const TArg<T>&, bool,  \
                                         int, int, int64_t);                                                                   \
    template cudaError_t launch_column_lie_exp<T>(const Geometry&, const DeviceInfo&, cudaStream_t, const CsrDevice&, \
                                                  const T*, int64_t, int, int, TArg<T>, TArg<T>, int64_t, double);

RPP_GB_INSTANTIATE_LIE_COLUMN(float)
RPP_GB_INSTANTIATE_LIE_COLUMN(double)

}  // namespace rpp_gb

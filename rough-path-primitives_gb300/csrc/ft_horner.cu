// ft_horner.cu -- ft_exp, ft_log and ft_fmexp for widths 2..8: Horner's rule on
// columns of coefficients (ft_column.cuh), each round only on the levels that
// later rounds read; fmexp is Horner's rule on the multiplier.
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

// ft_exp, ft_log (out from degree 0) and ft_fmexp.  FP64 is bound by its pipe,
// FP32 by the rounds' latency.  Batch 4096, general kernel -> this: exp W5 D5
// FP64 511 -> 200 us, FP32 311 -> 64; log FP64 212 -> 191, FP32 127 -> 69; fmexp
// FP64 717 -> 273, FP32 354 -> 75 (405 and 107 as exp and one product, whose rounding
// error is also 1.3 to 1.8 times as large); W2 D12 (2 048) exp FP64 3247 -> 983, FP32
// 1243 -> 176, fmexp 3607 -> 1021 and 1473 -> 239.
template <typename T, int W>
__global__ void __launch_bounds__(kHornerThreads, (kHornerBlocks<T, W>)) k_column_horner(Geometry G, IntermediateKind kind, TArg<T> out,
                                                                  TArg<T> x, TArg<T> m, int64_t batch) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    uint64_t* bar = reinterpret_cast<uint64_t*>(smem_raw);
    const uint32_t pd = staged_elems<T>(G.dim), half = staged_elems<T>(G.db[G.depth]);
    T* buf = reinterpret_cast<T*>(smem_raw + kBulkHeader);
    T* s_x = buf + 2 * half;
    T* s_m = s_x + pd;
    uint32_t phase = 0;
    bulk_stage_init(bar);
    const int ohi = imin(out.hi, G.depth);
    // the multiplier's levels below the output's take no part
    const int mlo = imax(m.lo, out.lo), mhi = imin(m.hi, ohi);
    const bool fm = kind == IntermediateKind::FMExp;
    const int H = fm ? imax(0, ohi - mlo) : ohi;
    const int xlo = imax(1, x.lo), xhi = imin(x.hi, H);
    for (int64_t b = blockIdx.x; b < batch; b += gridDim.x) {
        BulkStage<T> st(bar, phase);
        T* X = st.add(s_x, x.at(b), xlo, xhi, G);
        const T* M = fm ? st.add(s_m, m.at(b), mlo, mhi, G) : nullptr;
        if (!st.commit(G.fault)) return;
        T* o = out.at(b);
        if (fm) {
            horner_multiplied<T, W>(G, o, out.lo, ohi, M, mlo, mhi, Opnd<T>{X, xlo, xhi}, buf, buf + half);
        } else if (kind == IntermediateKind::Exp) {
            const T unit = horner<T, W, false>(G, H, Opnd<T>{X, xlo, xhi}, buf, buf + half,
                                               [&](int n, uint32_t at, T v) { o[G.db[n] + at] = v; });
            if (threadIdx.x == 0) o[0] = unit;
        } else {
            const T unit = horner<T, W, true>(G, H, Opnd<T>{X, xlo, xhi}, buf, buf + half,
                                              [&](int n, uint32_t at, T v) { o[G.db[n] + at] = v; });
            if (threadIdx.x == 0) o[0] = unit;
        }
        bulk_stage_reuse();
    }
}

template <typename T>
size_t horner_smem(const Geometry& g, bool multiplier) {
    return kBulkHeader + (2 * static_cast<size_t>(staged_elems<T>(g.db[g.depth])) +
                          (multiplier ? 2 : 1) * static_cast<size_t>(staged_elems<T>(g.dim))) * sizeof(T);
}

}  // namespace

template <typename T>
bool column_horner_fits(const Geometry& g, const DeviceInfo& dev, IntermediateKind kind, const TArg<T>& out,
                        const TArg<T>& x, int64_t batch) {
    constexpr bool fp64 = std::is_same<T, double>::value;
    // (depth 1 is one round: columns of exp and fmexp save the others' barriers)
    constexpr Worth kExp32{{1, 64, 80}, {0, 855, 855}, 0}, kExp64{{100, 64, 700}, {kNever, kNever, 329}, 80};
    constexpr Worth kLog32{{150, 125, 80}, {658, 658, 329}, 41}, kLog64{{300, 100, 2000}, {6000, 658, 526}, 80};
    constexpr Worth kFmexp32{{1, 64, 80}, {0, 395, 329}, 32}, kFmexp64{{64, 100, 700}, {kNever, 395, 329}, 80};
    if (!(g.depth == 1 && kind != IntermediateKind::Log) &&
        !worth(kind == IntermediateKind::Exp ? (fp64 ? kExp64 : kExp32)
               : kind == IntermediateKind::Log ? (fp64 ? kLog64 : kLog32)
                                               : (fp64 ? kFmexp64 : kFmexp32),
               g, dev, batch))
        return false;
    const bool fm = kind == IntermediateKind::FMExp;
    // (an exponent without degree one leaves degrees of the running tensor that have
    // no terms: the general kernel skips them, a product with their zeros would turn
    // the exponent's infinities into NaN)
    if (fm && (x.lo > 1 || x.hi < 1)) return false;
    return out.lo <= out.hi && (fm || out.lo == 0) && horner_fits(g, dev, horner_smem<T>(g, fm));
}

template <typename T>
cudaError_t launch_column_horner(const Geometry& g, const DeviceInfo& dev, cudaStream_t s, IntermediateKind kind,
                                 TArg<T> out, TArg<T> x, TArg<T> m, int64_t batch) {
    const size_t smem = horner_smem<T>(g, kind == IntermediateKind::FMExp);
    return with_width(g.width, [&](auto w) {
        constexpr int W = decltype(w)::value;
        return run_column<&k_column_horner<T, W>>(dev, s, horner_threads<T, W>(g, smem), smem, batch, g, kind, out, x, m,
                                                  batch);
    });
}

#define RPP_GB_INSTANTIATE_HORNER(T)                                                                                \
    template bool column_horner_fits<T>(const Geometry&, const DeviceInfo&, IntermediateKind, const TArg<T>&,       \
                                        const TArg<T>&, int64_t);                                               \
    template cudaError_t launch_column_horner<T>(const Geometry&, const DeviceInfo&, cudaStream_t, IntermediateKind, \
                                                 TArg<T>, TArg<T>, TArg<T>, int64_t);

RPP_GB_INSTANTIATE_HORNER(float)
RPP_GB_INSTANTIATE_HORNER(double)

}  // namespace rpp_gb

// ft_column.cu -- products of staged tensors, a column of coefficients per
// thread (ft_column.cuh), for widths 2..8.
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

constexpr size_t kColumnSmemLimit = 200 * 1024;
constexpr int kColumnThreads = 512;

// Whole tensors one after another: a group of rows is one span of memory.
template <typename T>
__device__ __forceinline__ bool packed(const TArg<T>& t, int hi, const Geometry& G) {
    return t.stride == static_cast<int64_t>(G.dim) && t.lo == 0 && hi == G.depth;
}

// Stages rows b0 .. b0 + held - 1 of an operand in `buf` (pd elements a row);
// staged_row gives where row i's coefficient 0 then lies (BulkStage keeps a
// row's alignment modulo 16 bytes in its buffer).
template <typename T>
__device__ __forceinline__ const T* stage_rows(BulkStage<T>& st, T* buf, uint32_t pd, const TArg<T>& t, int hi,
                                               int64_t b0, uint32_t held, const Geometry& G) {
    if (packed(t, hi, G)) return st.add_span(buf, t.at(b0), 0, held * G.dim);
    for (uint32_t i = 0; i < held; ++i) st.add(buf + i * pd, t.at(b0 + i), t.lo, hi, G);
    return nullptr;
}
template <typename T>
__device__ __forceinline__ const T* staged_row(const T* first, const T* buf, uint32_t pd, const TArg<T>& t, int64_t b0,
                                               uint32_t i, const Geometry& G) {
    if (first) return first + i * G.dim;
    return buf + i * pd + (reinterpret_cast<uintptr_t>(t.at(b0 + i)) & 15u) / sizeof(T);
}

// out = alpha*add + beta * L (x) R for `per` tensors of the batch at a time,
// both factors staged in shared memory (so the result may replace either);
// the added term is read, and the result written, once, lanes consecutive.
// FP64 is bound by its pipe, FP32 by HBM and, where W is small, shared-memory
// loads.  ft_mul in a CUDA graph, the general kernel -> this one: FP32 W5 D5
// batch 4096 114 -> 52 us (3.7 TB/s), W8 D4 115 -> 47, W2 D12 batch 2048
// 234 -> 69; FP64 W5 D5 246 -> 219 us (67 % of the FP64 peak), W2 D12 544 ->
// 426, W4 D4 batch 1024 8.3 -> 7.3.  A tile of W x W coefficients a thread
// (first and last letters) saves more loads but strides its lanes W apart:
// FP32 W5 D5 43 us, but W8 D4 100, and FP64 W8 D4 368 against 231 here.
template <typename T, int W, bool Scale>
__global__ void __launch_bounds__(kColumnThreads) k_column_product(Geometry G, TArg<T> out, TArg<T> add, TArg<T> lhs,
                                                                   TArg<T> rhs, int64_t batch, T alpha, T beta,
                                                                   uint32_t per) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    uint64_t* bar = reinterpret_cast<uint64_t*>(smem_raw);
    T* sm = reinterpret_cast<T*>(smem_raw + kBulkHeader);
    const int D = G.depth, ohi = imin(out.hi, D);
    const uint32_t pd = staged_elems<T>(G.dim);
    const uint32_t tasks = tensor_tasks<T, W>(G, out.lo, ohi);
    const int lhi = imin(lhs.hi, D), rhi = imin(rhs.hi, D);
    uint32_t phase = 0;
    bulk_stage_init(bar);
    for (int64_t b0 = static_cast<int64_t>(blockIdx.x) * per; b0 < batch; b0 += static_cast<int64_t>(gridDim.x) * per) {
        const uint32_t held = static_cast<uint32_t>(batch - b0 < per ? batch - b0 : per);
        BulkStage<T> st(bar, phase);
        const T* l0 = stage_rows(st, sm, pd, lhs, lhi, b0, held, G);
        const T* r0 = stage_rows(st, sm + per * pd, pd, rhs, rhi, b0, held, G);
        if (!st.commit(G.fault)) return;
        for (uint32_t t = threadIdx.x; t < tasks * held; t += blockDim.x) {
            int n;
            uint32_t i, place;
            locate_task<T, W>(G, t, held, ohi, n, i, place);
            const T* l = staged_row(l0, sm, pd, lhs, b0, i, G);
            const T* r = staged_row(r0, sm + per * pd, pd, rhs, b0, i, G);
            T* o = out.at(b0 + i) + G.db[n];
            const T* ad = add.p != nullptr && add.lo <= n && n <= add.hi ? add.at(b0 + i) + G.db[n] : nullptr;
            task_product<T, W>(G, Opnd<T>{l, lhs.lo, lhi}, Opnd<T>{r, rhs.lo, rhi}, n, place, [&](uint32_t at, T v) {
                if constexpr (Scale) v *= beta;
                if (ad) v = fma(alpha, ad[at], v);
                o[at] = v;
            });
        }
        bulk_stage_reuse();
    }
}

// Tensors per CTA and threads of a launch: enough tensors that their tasks
// make 128 threads, as long as the batch still gives every SM two CTAs;
// threads for the tasks, at most 256 while two CTAs fit an SM.
inline void column_shape(uint32_t tasks, size_t slot_bytes, size_t limit, int64_t batch, int sms, uint32_t& per,
                         int& threads) {
    per = 1;
    while (per < 16 && per * tasks < 128 && (per + 1) * slot_bytes <= limit &&
           batch >= 2 * sms * static_cast<int64_t>(per + 1))
        ++per;
    const uint32_t all = per * tasks;
    const uint32_t most = per * slot_bytes > limit / 2 ? kColumnThreads : 256u;
    const uint32_t rounds = (all + most - 1) / most;
    threads = std::max(64, static_cast<int>(((all + rounds - 1) / rounds + 31) / 32 * 32));
}

template <typename T>
size_t column_slot_bytes(const Geometry& g) {
    return 2 * static_cast<size_t>(staged_elems<T>(g.dim)) * sizeof(T);
}

}  // namespace

template <typename T>
bool column_product_fits(const Geometry& g, const DeviceInfo& dev, bool added, int64_t batch) {
    // (the general kernel loads the added term before its sum, which few tensors wait for)
    constexpr Worth kMul32{{60, 125, 300}, {263, 263, 460}, 0, {8, 8, 8}};
    constexpr Worth kFma32{{150, 500, 700}, {395, 395, 855}, 0, {13, 13, 13}};
    constexpr Worth kMul64{{100, 100, 2000}, {263, 263, 1974}, 0, {8, 8, 16}};
    if (!worth(std::is_same<T, double>::value ? kMul64 : added ? kFma32 : kMul32, g, dev, batch)) return false;
    // FP64: where three tensors do not fit shared memory the general kernel
    // runs unstaged, with several CTAs per SM against one here, and is as fast
    // (W6 D5, batch 2048: 283 us against 299); FP32 gains at every size.
    const size_t held = column_slot_bytes<T>(g) * (std::is_same<T, double>::value ? 3 : 2) / 2;
    return column_width(g.width) &&
           kBulkHeader + held <= std::min(kColumnSmemLimit, static_cast<size_t>(dev.max_smem_optin));
}

template <typename T>
cudaError_t launch_column_product(const Geometry& g, const DeviceInfo& dev, cudaStream_t s, TArg<T> out, TArg<T> add,
                                TArg<T> lhs, TArg<T> rhs, int64_t batch, double alpha, double beta) {
    if (batch <= 0 || out.lo > out.hi) return cudaSuccess;
    return with_width(g.width, [&](auto w) {
        constexpr int W = decltype(w)::value;
        uint32_t per;
        int threads;
        const size_t slot = column_slot_bytes<T>(g);
        const size_t limit = std::min(kColumnSmemLimit, static_cast<size_t>(dev.max_smem_optin)) - kBulkHeader;
        column_shape(tensor_tasks<T, W>(g, out.lo, out.hi), slot, limit, batch, dev.sm_count, per, threads);
        const size_t smem = kBulkHeader + per * slot;
        const int64_t groups = (batch + per - 1) / per;
        const T al = static_cast<T>(alpha), be = static_cast<T>(beta);
        if (be == T(1))
            return run_column<&k_column_product<T, W, false>>(dev, s, threads, smem, groups, g, out, add, lhs, rhs,
                                                           batch, al, be, per);
        return run_column<&k_column_product<T, W, true>>(dev, s, threads, smem, groups, g, out, add, lhs, rhs, batch,
                                                      al, be, per);
    });
}

#define RPP_GB_INSTANTIATE_COLUMN(T)                                                                                 \
    template bool column_product_fits<T>(const Geometry&, const DeviceInfo&, bool, int64_t);                                       \
    template cudaError_t launch_column_product<T>(const Geometry&, const DeviceInfo&, cudaStream_t, TArg<T>, TArg<T>, \
                                                TArg<T>, TArg<T>, int64_t, double, double);

RPP_GB_INSTANTIATE_COLUMN(float)
RPP_GB_INSTANTIATE_COLUMN(double)

}  // namespace rpp_gb

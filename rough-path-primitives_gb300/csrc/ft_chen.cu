// ft_chen.cu -- exp / fmexp for an exponent of degree one: the update of
// running signatures by one increment each.
#include <algorithm>

#include "bulk_stage.cuh"
#include "common.cuh"
#include "ft_column.cuh"
#include "launch_util.cuh"
#include "ops.hpp"

namespace rpp_gb {
namespace {

using namespace ftcol;

constexpr size_t kChenSmemLimit = 200 * 1024;
// The multiplier is staged while two CTAs fit an SM.
constexpr size_t kChenStageLimit = 100 * 1024;

// Chain storage of one stage of a Chen step: the chains n = j+1..H of level j
// in turn.
__host__ __device__ inline uint32_t chen_chain_elems(const Geometry& G, int H) {
    uint32_t most = 0;
    for (int j = 0; j < H; ++j) {
        const uint32_t s = static_cast<uint32_t>(H - j) * G.pw[j];
        if (s > most) most = s;
    }
    return most;
}

// out = M (x) exp(x), or exp(x), for an exponent of degree one (the update of
// a running signature by one increment): the Horner chains
//     T^n_j = M_j + T^n_{j-1} (x) x / (n-j+1),   out_n = T^n_n,
// with all chains of level j formed together, about 1.25 multiply-adds per
// coefficient where the general Horner rounds multiply whole tensors D times
// over.  One pass over memory: M is staged by one bulk copy (read as it goes
// where that would leave one CTA an SM), the chains of two stages are kept in
// shared memory and the result is written from the stage that forms it.  Large
// tensors are bound by HBM, small ones by the stages' latency.  ft_fmexp with
// increments, the general rounds -> this: FP32 W5 D5 batch 4096 221 -> 32 us (3.9
// TB/s), W3 D6 batch 3000 89 -> 9; FP64 W5 D5 455 -> 53 us (4.9 TB/s), W2 D12
// batch 2048 1463 -> 117, W6 D6 batch 256 1130 -> 145.
// Chains start at the output's lowest degree (levels of M below it take no
// part) and degrees that M lacks count as zero, as in those rounds.
template <typename T, int W>
__global__ void __launch_bounds__(512) k_chen_step(Geometry G, TArg<T> out, TArg<T> mult, TArg<T> x, int64_t batch,
                                                   int unit, int staged) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    uint64_t* bar = reinterpret_cast<uint64_t*>(smem_raw);
    T* sm = reinterpret_cast<T*>(smem_raw + kBulkHeader);
    const int H = imin(out.hi, G.depth), lo = out.lo;
    const uint32_t chains = chen_chain_elems(G, H);
    T* xs = sm + 2 * chains;  // xs[(m-1) W + a] = x_a / m
    T* s_m = xs + staged_elems<T>(static_cast<uint32_t>(H * W) + 2 * chains) - 2 * chains;
    const int mlo = imax(mult.lo, lo), mhi = imin(mult.hi, H);
    uint32_t phase = 0;
    if (staged) bulk_stage_init(bar);
    for (int64_t b = blockIdx.x; b < batch; b += gridDim.x) {
        const T* M = mult.p ? mult.at(b) : nullptr;
        T* o = out.at(b);
        for (uint32_t t = threadIdx.x; t < static_cast<uint32_t>(H * W); t += blockDim.x)
            xs[t] = x.at(b)[1 + t % W] * ftdev::recip<T>().inv[1 + t / W];
        if (staged) {
            BulkStage<T> st(bar, phase);
            M = st.add(s_m, M, mlo, mhi, G);
            if (!st.commit(G.fault)) return;
        } else {
            __syncthreads();
        }
        for (int j = lo; j <= H; ++j) {
            const uint32_t wj = G.pw[j], base = G.db[j], wp = j > 0 ? G.pw[j - 1] : 0u;
            const T* prev = sm + ((j + 1) & 1) * chains;  // stage j-1: chains n = j..H
            T* next = sm + (j & 1) * chains;
            const bool has = M && j >= mlo && j <= mhi;
            const T none = unit && j == 0 ? T(1) : T(0);
            if (j == lo) {  // the chains begin
                for (uint32_t i = threadIdx.x; i < wj; i += blockDim.x) {
                    const T mv = has ? M[base + i] : none;
                    o[base + i] = mv;
                    for (int n = j + 1; n <= H; ++n) next[static_cast<uint32_t>(n - j - 1) * wj + i] = mv;
                }
            } else if (j < H) {
                for (uint32_t i = threadIdx.x; i < wj; i += blockDim.x) {
                    const T mv = has ? M[base + i] : T(0);
                    const uint32_t q = i / W, a = i - q * W;
                    o[base + i] = fma(prev[q], xs[a], mv);
                    for (int n = j + 1; n <= H; ++n)
                        next[static_cast<uint32_t>(n - j - 1) * wj + i] =
                            fma(prev[static_cast<uint32_t>(n - j) * wp + q], xs[static_cast<uint32_t>(n - j) * W + a], mv);
                }
            } else {
#pragma unroll 4
                for (uint32_t i = threadIdx.x; i < wj; i += blockDim.x) {
                    const T mv = has ? M[base + i] : T(0);
                    const uint32_t q = i / W, a = i - q * W;
                    o[base + i] = fma(prev[q], xs[a], mv);
                }
            }
            __syncthreads();
        }
        if (staged) bulk_stage_reuse();
    }
}

// The chains and scaled letters, and (staged) the multiplier.
template <typename T>
size_t chen_smem(const Geometry& g, int H, bool staged) {
    const size_t own = staged_elems<T>(2 * chen_chain_elems(g, H) + static_cast<uint32_t>(H * g.width));
    return kBulkHeader + (own + (staged ? staged_elems<T>(g.db[H + 1]) : 0)) * sizeof(T);
}

}  // namespace

template <typename T>
bool chen_step_fits(const Geometry& g, const DeviceInfo& dev, const TArg<T>& out, const TArg<T>& x) {
    return column_width(g.width) && out.lo <= out.hi && out.hi >= 1 && std::max(1, x.lo) == 1 &&
           std::min(x.hi, g.depth) == 1 &&
           chen_smem<T>(g, out.hi, false) <= std::min(kChenSmemLimit, static_cast<size_t>(dev.max_smem_optin));
}

template <typename T>
cudaError_t launch_chen_step(const Geometry& g, const DeviceInfo& dev, cudaStream_t s, TArg<T> out, TArg<T> mult,
                             TArg<T> x, int64_t batch, bool unit) {
    return with_width(g.width, [&](auto w) {
        constexpr int W = decltype(w)::value;
        const bool staged = mult.p != nullptr && chen_smem<T>(g, out.hi, true) <= kChenStageLimit;
        const size_t smem = chen_smem<T>(g, out.hi, staged);
        // 14 (FP64) or 28 coefficients of the widest level a thread: what bounds small
        // tensors is the stages' latency, which more and smaller CTAs an SM hide
        // (W3 D6 batch 3000 FP32: 256 threads 17 us, 128 threads 12, 32 threads 9)
        const uint32_t each = sizeof(T) == 8 ? 14 : 28;
        const int threads = std::max(32, std::min(smem > 64 * 1024 ? 512 : 256,
                                                  static_cast<int>((g.pw[out.hi] / each + 31) / 32 * 32)));
        return run_column<&k_chen_step<T, W>>(dev, s, threads, smem, batch, g, out, mult, x, batch, unit ? 1 : 0,
                                              staged ? 1 : 0);
    });
}

#define RPP_GB_INSTANTIATE_CHEN(T)                                                                          \
    template bool chen_step_fits<T>(const Geometry&, const DeviceInfo&, const TArg<T>&, const TArg<T>&);    \
    template cudaError_t launch_chen_step<T>(const Geometry&, const DeviceInfo&, cudaStream_t, TArg<T>,     \
                                             TArg<T>, TArg<T>, int64_t, bool);

RPP_GB_INSTANTIATE_CHEN(float)
RPP_GB_INSTANTIATE_CHEN(double)

}  // namespace rpp_gb

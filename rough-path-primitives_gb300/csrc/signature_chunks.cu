// signature_chunks.cu -- signatures of few long paths, cut in time.
//
// A path is a serial chain of Chen steps, and one CTA runs it: a call with
// fewer paths than the GPU holds CTAs leaves SMs idle for the length of the
// chain (4 paths of 1 000 increments at W3 D5 FP64, forward and reverse: 10 us
// a step, four SMs).  By Chen's identity the signature of a path is the product
// of its pieces' signatures, so the pieces run at once and their products are
// joined in log2(pieces) rounds.  With p_c the product up to and with piece c
// and q_c the product of the pieces after it, the loss <seed, S> is
// <seed, p_c (x) q_c>, so the cotangent of p_c is the right adjoint multiply of
// the seed by q_c, and every piece's reverse pass runs from (p_c, that
// cotangent) by itself.
#include <algorithm>
#include <mutex>
#include <type_traits>

#include "bulk_stage.cuh"
#include "common.cuh"
#include "ft_column.cuh"
#include "launch_util.cuh"
#include "ops.hpp"

namespace rpp_gb {
namespace {

using namespace ftcol;

constexpr int kJoinThreads = 256;
constexpr size_t kJoinSmemLimit = 200 * 1024;

// out = L (x) R, whole tensors; `out` may be L or R.  WT = 0: any width, or
// operands too large for shared memory (read in place, top level first).
template <typename T, int WT>
__device__ void join(const Geometry& G, T* out, T* also, const T* L, const T* R, uint64_t* bar, uint32_t& phase,
                     T* sm) {
    const int D = G.depth;
    if constexpr (WT > 0) {
        const uint32_t pd = staged_elems<T>(G.dim);
        BulkStage<T> st(bar, phase);
        const T* l = st.add(sm, L, 0, D, G);
        const T* r = st.add(sm + pd, R, 0, D, G);
        if (!st.commit(G.fault)) return;
        const uint32_t tasks = tensor_tasks<T, WT>(G, 0, D);
        for (uint32_t t = threadIdx.x; t < tasks; t += blockDim.x) {
            int n;
            uint32_t i, place;
            locate_task<T, WT>(G, t, 1, D, n, i, place);
            task_product<T, WT>(G, Opnd<T>{l, 0, D}, Opnd<T>{r, 0, D}, n, place, [&](uint32_t at, T v) {
                out[G.db[n] + at] = v;
                if (also) also[G.db[n] + at] = v;
            });
        }
    } else {
        const Opnd<T> none{nullptr, 1, 0};
        ftdev::product_levels<T, false>(G, out, 0, D, none, T(0), Opnd<T>{L, 0, D}, Opnd<T>{R, 0, D}, T(1), true);
        if (also)
            for (uint32_t i = threadIdx.x; i < G.dim; i += blockDim.x) also[i] = out[i];
    }
}

// offsets[path chunks + c] = the first increment of piece c of the path.
__global__ void __launch_bounds__(256) k_chunk_offsets(int64_t* offsets, int64_t paths, int64_t length,
                                                       int64_t chunks, int64_t piece) {
    const int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x;
    if (i > paths * chunks) return;
    const int64_t path = i / chunks;
    offsets[i] = path * length + (i - path * chunks) * piece;
}

// Round `r` of the reduction: piece c (a multiple of 2^{r+1}) takes its product
// with piece c + 2^r; the last round's goes to the signature row.
template <typename T, int WT>
__global__ void __launch_bounds__(kJoinThreads) k_chunk_reduce(Geometry G, T* pieces, int64_t pitch, int64_t chunks,
                                                               int64_t pairs, int r, T* sig, int64_t sig_stride) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    uint64_t* bar = reinterpret_cast<uint64_t*>(smem_raw);
    uint32_t phase = 0;
    if (WT > 0) bulk_stage_init(bar);
    const int64_t path = blockIdx.x / pairs, c = (blockIdx.x - path * pairs) << (r + 1);
    T* l = pieces + (path * chunks + c) * pitch;
    const T* rr = l + (static_cast<int64_t>(1) << r) * pitch;
    const bool last = (static_cast<int64_t>(2) << r) >= chunks;
    join<T, WT>(G, last ? sig + path * sig_stride : l, nullptr, l, rr, bar, phase,
                reinterpret_cast<T*>(smem_raw + kBulkHeader));
}

// Round `r` of both scans (Sklansky's: a piece whose index has bit r set takes
// the product with the last piece of the block before its own, which the round
// does not write).  Round 0 reads the pieces' signatures and fills p and q.
// blockIdx.y = 0: p, 1: q, whose indices count from the end.
template <typename T, int WT>
__global__ void __launch_bounds__(kJoinThreads) k_chunk_scan(Geometry G, const T* pieces, T* p, T* q, int64_t pitch,
                                                             int64_t chunks, int r, T* sig, int64_t sig_stride) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    uint64_t* bar = reinterpret_cast<uint64_t*>(smem_raw);
    uint32_t phase = 0;
    const int64_t path = blockIdx.x / chunks, c = blockIdx.x - path * chunks;
    const bool suffix = blockIdx.y != 0;
    const int64_t i = suffix ? chunks - 1 - c : c;  // index in the direction of the scan
    const bool joins = (i >> r) & 1;
    if (r > 0 && !joins) return;
    T* own = (suffix ? q : p) + (path * chunks + c) * pitch;
    // what round 0 starts from: piece c, or for the suffix the piece after it
    // (nothing after the last piece: the unit)
    auto source = [&](int64_t at) -> const T* {
        if (r > 0) return (suffix ? q : p) + (path * chunks + at) * pitch;
        const int64_t piece = suffix ? at + 1 : at;
        return piece < chunks ? pieces + (path * chunks + piece) * pitch : nullptr;
    };
    const T* mine = source(c);
    const int64_t j = ((i >> r) << r) - 1;  // the partner, in scan direction
    const T* other = joins ? source(suffix ? chunks - 1 - j : j) : nullptr;
    T* also = !suffix && sig && c == chunks - 1 && (static_cast<int64_t>(2) << r) >= chunks ? sig + path * sig_stride
                                                                                             : nullptr;
    if (!other) {  // nothing to multiply with: a copy (or the unit)
        for (uint32_t e = threadIdx.x; e < G.dim; e += blockDim.x) own[e] = mine ? mine[e] : e == 0 ? T(1) : T(0);
        return;
    }
    if (WT > 0) bulk_stage_init(bar);
    join<T, WT>(G, own, also, suffix ? mine : other, suffix ? other : mine, bar, phase,
                reinterpret_cast<T*>(smem_raw + kBulkHeader));
}

template <typename T>
size_t join_smem(const Geometry& g) {
    return kBulkHeader + 2 * static_cast<size_t>(staged_elems<T>(g.dim)) * sizeof(T);
}

template <auto kernel, typename... Args>
cudaError_t join_launch(const DeviceInfo& dev, cudaStream_t s, dim3 grid, int threads, size_t smem, Args... args) {
    cudaError_t err = allow_large_smem<kernel>(dev);
    if (err != cudaSuccess) return err;
    kernel<<<grid, threads, smem, s>>>(args...);
    return cudaGetLastError();
}

// f(width with an instantiation whose operands are staged, or 0)
template <typename T, typename F>
cudaError_t with_join_width(const Geometry& g, const DeviceInfo& dev, F&& f) {
    if (column_width(g.width) &&
        join_smem<T>(g) <= std::min(kJoinSmemLimit, static_cast<size_t>(dev.max_smem_optin)))
        return with_width(g.width, f);
    return f(std::integral_constant<int, 0>{});
}

template <typename T, int W>
int join_threads(const Geometry& g) {
    if constexpr (W > 0) {
        const uint32_t tasks = tensor_tasks<T, W>(g, 0, g.depth);
        return std::min(kJoinThreads, std::max(64, static_cast<int>((tasks + 31) / 32 * 32)));
    } else {
        return threads_for(g.pw[g.depth]);
    }
}

// The scratch of the signature calls (pieces, ragged orders, workspaces) comes
// from a memory pool of the library's own, one a device, made with the device's first plan (so never inside a stream capture).
// The device's default pool gives its memory back at every synchronisation, and
// mapping it again cost the next call 100 to 250 us; this one keeps at most
// 256 MB while the device has a plan, and gives it back with the last one.
constexpr uint64_t kScratchKept = uint64_t{256} << 20;
std::mutex g_pool_lock;
cudaMemPool_t g_pool[kMaxDevices] = {};
int g_pool_users[kMaxDevices] = {};

void keep_at_most(cudaMemPool_t pool, uint64_t bytes) {
    cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &bytes);
}

}  // namespace

void scratch_retain(int device) {
    if (device < 0 || device >= kMaxDevices) return;
    std::lock_guard<std::mutex> guard(g_pool_lock);
    if (!g_pool[device]) {
        cudaMemPoolProps props{};
        props.allocType = cudaMemAllocationTypePinned;
        props.location.type = cudaMemLocationTypeDevice;
        props.location.id = device;
        if (cudaMemPoolCreate(&g_pool[device], &props) != cudaSuccess) {  // the default pool serves
            g_pool[device] = nullptr;
            cudaGetLastError();
        }
    }
    if (g_pool_users[device]++ == 0 && g_pool[device]) keep_at_most(g_pool[device], kScratchKept);
}

void scratch_release(int device) {
    if (device < 0 || device >= kMaxDevices) return;
    std::lock_guard<std::mutex> guard(g_pool_lock);
    if (--g_pool_users[device] == 0 && g_pool[device]) {
        keep_at_most(g_pool[device], 0);  // what is still in use goes when it is done
        cudaMemPoolTrimTo(g_pool[device], 0);
    }
}

cudaError_t scratch_alloc(int device, void** out, size_t bytes, cudaStream_t s) {
    cudaMemPool_t pool = nullptr;
    if (device >= 0 && device < kMaxDevices) {
        std::lock_guard<std::mutex> guard(g_pool_lock);
        pool = g_pool[device];
    }
    return pool ? cudaMallocFromPoolAsync(out, bytes, pool, s) : cudaMallocAsync(out, bytes, s);
}

// The rule.  Pieces are worth their joins where they put idle SMs to work and
// the chain they shorten is long: as many pieces per path as keep the GPU's
// CTA slots filled (four a SM, fewer where the state leaves room for fewer; two
// for the warp-per-letter kernels, whose steps are short against a join), of at
// least 8 increments (16 for those kernels), if the time taken off the chain
// is more than the joins cost.  A step's time is a fit to the kernels' measured
// chains (one path, 1 000 increments, FP64: W3 D2 0.87 us, W3 D5 2.7, W5 D5
// 4.0, W2 D10 6.4, W6 D5 5.8 forward, four times that with the reverse pass;
// warp-per-letter 0.13 and 0.7 us); a call's joins cost 50 us and each round 5
// at most (several launches of a call that is waited for), twice that with the
// reverse pass.  (The joins' cost was fitted to an earlier, slower form of them,
// so calls near the line still run whole that pieces would speed up.)
// Measured, forward + reverse, whole -> in pieces: FP64 W3 D5, 4 paths of 1 000,
// 10.13 -> 0.17 ms; W5 D5 1 path of 1 000 15.5 -> 0.27, 100 paths 15.6 -> 5.6;
// 64 increments, 8 paths 1.00 -> 0.18; W2 D10 FP32 1 path of 1 000 22.0 -> 0.26.
// Where SMs are not idle pieces lost: W5 D5 FP64, 1 000 paths of 64, 3.35 ms
// whole, 3.67 in four (with that earlier form).
template <typename T>
int64_t signature_chunks(const Geometry& g, const DeviceInfo& dev, int64_t batch, int64_t length, bool reverse) {
    const int D = g.depth;
    if (D < 1 || batch <= 0 || length < 16) return 1;
    const bool letters = std::is_same<T, float>::value && (reverse ? letter_reverse_supported(g.width, D)
                                                                   : letter_warps_supported(g.width, D));
    double fmas = 0.0, chains = 0.0;  // of a step; coefficients of its chains
    for (int j = 1; j <= D; ++j) fmas += static_cast<double>(D - j + 1) * g.pw[j];
    for (int j = 0; j < D; ++j) chains += static_cast<double>(D - j) * g.pw[j];
    const double step = letters ? (reverse ? 0.7 : 0.13) : (reverse ? 4.0 : 1.0) * (0.45 * D + 3e-4 * fmas);
    // CTAs of the shared-memory kernel that fit an SM
    const double state = (reverse ? 2.0 : 1.0) * (g.dim + chains) * sizeof(T);
    const int64_t fit = static_cast<int64_t>(dev.max_smem_optin / std::max(1.0, state));
    const int64_t per_sm = letters ? 2 : std::max<int64_t>(1, std::min<int64_t>(4, fit));
    int64_t chunks = std::min(per_sm * dev.sm_count / batch, length / (letters ? 16 : 8));
    // scratch: at most kScratchKept
    const int64_t row = static_cast<int64_t>((reverse ? 3 : 1) * sizeof(T)) * (g.dim + 32);
    chunks = std::min(chunks, static_cast<int64_t>(kScratchKept) / row / batch);
    if (chunks < 2) return 1;
    const int64_t piece = (length + chunks - 1) / chunks;
    chunks = (length + piece - 1) / piece;  // none empty
    int rounds = 0;
    while ((int64_t{1} << rounds) < chunks) ++rounds;
    return step * static_cast<double>(length - piece) > (reverse ? 2.0 : 1.0) * (50.0 + 5.0 * rounds) ? chunks : 1;
}

cudaError_t chunk_offsets(cudaStream_t s, int64_t* offsets, int64_t paths, int64_t length, int64_t chunks) {
    const unsigned blocks = static_cast<unsigned>((paths * chunks + 256) / 256);
    k_chunk_offsets<<<blocks, 256, 0, s>>>(offsets, paths, length, chunks, (length + chunks - 1) / chunks);
    return cudaGetLastError();
}

template <typename T>
cudaError_t chunk_reduce(const Geometry& g, const DeviceInfo& dev, cudaStream_t s, T* pieces, int64_t pitch,
                         int64_t paths, int64_t chunks, T* sig, int64_t sig_stride) {
    return with_join_width<T>(g, dev, [&](auto w) {
        constexpr int W = decltype(w)::value;
        cudaError_t err = cudaSuccess;
        for (int r = 0; (int64_t{1} << r) < chunks && err == cudaSuccess; ++r) {
            // pieces c = 0, 2^{r+1}, ... with a partner c + 2^r
            const int64_t pairs = (chunks - (int64_t{1} << r) + (int64_t{2} << r) - 1) >> (r + 1);
            err = join_launch<&k_chunk_reduce<T, W>>(dev, s, dim3(static_cast<unsigned>(paths * pairs)),
                                                     join_threads<T, W>(g), W > 0 ? join_smem<T>(g) : 0, g, pieces, pitch,
                                                     chunks, pairs, r, sig, sig_stride);
        }
        return err;
    });
}

template <typename T>
cudaError_t chunk_scan(const Geometry& g, const DeviceInfo& dev, cudaStream_t s, const T* pieces, T* p, T* q,
                       int64_t pitch, int64_t paths, int64_t chunks, T* sig, int64_t sig_stride) {
    return with_join_width<T>(g, dev, [&](auto w) {
        constexpr int W = decltype(w)::value;
        cudaError_t err = cudaSuccess;
        for (int r = 0; (int64_t{1} << r) < chunks && err == cudaSuccess; ++r)
            err = join_launch<&k_chunk_scan<T, W>>(dev, s, dim3(static_cast<unsigned>(paths * chunks), 2),
                                                   join_threads<T, W>(g), W > 0 ? join_smem<T>(g) : 0, g, pieces, p, q,
                                                   pitch, chunks, r, sig, sig_stride);
        return err;
    });
}

#define RPP_GB_INSTANTIATE_CHUNKS(T)                                                                              \
    template int64_t signature_chunks<T>(const Geometry&, const DeviceInfo&, int64_t, int64_t, bool);            \
    template cudaError_t chunk_reduce<T>(const Geometry&, const DeviceInfo&, cudaStream_t, T*, int64_t, int64_t, \
                                         int64_t, T*, int64_t);                                                   \
    template cudaError_t chunk_scan<T>(const Geometry&, const DeviceInfo&, cudaStream_t, const T*, T*, T*,       \
                                       int64_t, int64_t, int64_t, T*, int64_t);

RPP_GB_INSTANTIATE_CHUNKS(float)
RPP_GB_INSTANTIATE_CHUNKS(double)

}  // namespace rpp_gb

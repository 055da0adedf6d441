// shuffle_letters.cu -- the shuffle product (st_mul, st_fma, st_inplace_fma) and
// its adjoint (st_adj_mul) a letter at a time, for widths 2..8.
//
// The subset sums of shuffle.cu take 2^N terms for a word of N letters.  Dealing
// the letters of a word one by one to the two factors instead shares all but
// N^2 / 2 of them.  Adjoint: with
//     E_m^k[u, v, r] = sum over interleavings s of u and v of arg[s r],
// |u| = k, |v| = m - k, r the N - m letters not yet dealt,
//     E_{m+1}^k[u, v, r] = E_m^{k-1}[u', v, a r] + E_m^k[u, v', b r],
// u = u' a, v = v' b, and out[v] = sum_u op[u] E_N^k[u, v].  Stored as one array of
// W^N per k in the order u v r, the second term is the same place of the array
// (v takes in the letter beside it), so a step adds E^{k-1}, with the letter a
// moved past v, into E^k; E^0 and E^m are the argument itself.  At N = 5 that is
// 10 additions and 6 multiply-adds a word where the subsets take 32
// multiply-adds, at N = 8 28 and 9 against 256.
// The product is the transpose: E^k starts as L_k (x) R_{N-k} and every step adds
// E^k, the letter moved back, into E^{k-1}.
// A CTA owns a tensor and keeps the N arrays of one degree in shared memory, a
// barrier between the steps, which with the index instructions is what bounds it.
// Product / adjoint, by subsets -> by letters (us): FP64 W2 D8 batch 4096 652 ->
// 211 / 2570 -> 249, W3 D6 batch 3000 312 -> 203 / 661 -> 279, W4 D4 batch 1024
// 16.5 -> 15.7 / 43 -> 22; FP32 W2 D8 338 -> 118 / 2342 -> 156, W3 D6 172 -> 119 /
// 604 -> 181, W5 D5 batch 4096 496 -> 406 / 686 -> 644.
#include <algorithm>
#include <type_traits>

#include "common.cuh"
#include "ft_column.cuh"
#include "launch_util.cuh"
#include "ops.hpp"

namespace rpp_gb {
namespace {

using namespace ftcol;

constexpr size_t kLettersSmemLimit = 200 * 1024;
constexpr int kLettersMaxDepth = 12;

struct PowerDiv {
    FastDiv by[kLettersMaxDepth + 1];  // by W^j
};

// Place of (u' v a r) for i = (u' a v r): b letters in v, R in r; and back.
template <int W>
__device__ __forceinline__ uint32_t letter_past(const Geometry& G, const PowerDiv& pd, uint32_t i, int b, int R) {
    uint32_t t, r, u, v;
    pd.by[R].divmod(i, t, r);
    pd.by[b].divmod(t, u, v);
    const uint32_t up = u / W, a = u - up * W;
    return ((up * G.pw[b] + v) * W + a) * G.pw[R] + r;
}
template <int W>
__device__ __forceinline__ uint32_t letter_back(const Geometry& G, const PowerDiv& pd, uint32_t j, int b, int R) {
    uint32_t t, r, up, v;
    pd.by[R].divmod(j, t, r);
    const uint32_t t2 = t / W, a = t - t2 * W;
    pd.by[b].divmod(t2, up, v);
    return ((up * W + a) * G.pw[b] + v) * G.pw[R] + r;
}

// Coefficients of the degrees that a warp or less of lanes covers: their sums
// over u are shared by all warps and added up in warp order.
template <int W>
constexpr uint32_t kNarrow = W == 2 ? 31u : W == 3 ? 40u : W == 4 ? 21u : W == 5 ? 31u : W + 1u;

template <typename T, int W>
__global__ void __launch_bounds__(1024) k_shuffle_letters_adjoint(Geometry G, PowerDiv pd, TArg<T> out, TArg<T> op,
                                                                  TArg<T> arg, int64_t batch) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    T* g = reinterpret_cast<T*>(smem_raw);  // degree N of the argument, then E^1, E^2, ...
    const int D = G.depth, ohi = imin(out.hi, D);
    const int phi = imin(op.hi, D), ahi = imin(arg.hi, D);
    const uint32_t t0 = threadIdx.x, nt = blockDim.x, lane = t0 & 31u, warp = t0 >> 5, warps = nt >> 5;
    T* P = g + static_cast<uint32_t>(D) * G.pw[D];  // the op
    T* part = P + G.dim;                            // part[coefficient][warp]
    for (int64_t b = blockIdx.x; b < batch; b += gridDim.x) {
        const T* A = arg.at(b);
        T* o = out.at(b);
        if (op.lo <= phi) {
            const T* src = op.at(b);
            for (uint32_t i = G.db[op.lo] + t0; i < G.db[phi + 1]; i += nt) P[i] = src[i];
        }
        // every coefficient of the output is one thread's for all N
        for (int N = D; N >= 0; --N) {
            const uint32_t size = G.pw[N];
            const int kmax = imin(phi, N - out.lo), kmin = imax(op.lo, N - ohi);
            const bool any = N >= arg.lo && N <= ahi && kmin <= kmax;
            if (!any && N < D) continue;
            if (any) {
                for (uint32_t i = t0; i < size; i += nt) g[i] = A[G.db[N] + i];
                __syncthreads();
                for (int m = 1; m < N; ++m)
                    for (int k = imin(m, kmax); k >= 1; --k) {
                        T* E = g + static_cast<uint32_t>(k) * size;
                        const T* self = k == m ? g : E;
                        const T* prev = E - size;  // (k = 1: the argument)
                        const int bl = m + 1 - k, R = N - m - 1;
#pragma unroll 2
                        for (uint32_t i = t0; i < size; i += nt)
                            E[i] = self[i] + prev[letter_past<W>(G, pd, i, bl, R)];
                        __syncthreads();
                    }
            }
            // out[N-k][v] += sum_u op[k][u] E^k[u, v]; N = D stores (zeros where it
            // has no terms)
            for (int q = out.lo; q <= ohi; ++q) {
                const int k = N - q;
                const bool terms = any && k >= kmin && k <= kmax;
                if (!terms && N != D) continue;
                const uint32_t wq = G.pw[q], wk = terms ? G.pw[k] : 0u;
                const T* Pk = P + (terms ? G.db[k] : 0u);
                const T* E = (k == 0 || k == N || !terms) ? g : g + static_cast<uint32_t>(k) * size;
                if (wq >= 32u) {
                    T* oq = o + G.db[q];
                    for (uint32_t v = t0; v < wq; v += nt) {
                        T acc = N == D ? T(0) : oq[v];
#pragma unroll 4
                        for (uint32_t u = 0; u < wk; ++u) acc = fma(Pk[u], E[u * wq + v], acc);
                        oq[v] = acc;
                    }
                } else {
                    const uint32_t us = 32u / wq, u0 = lane / wq, v = lane - u0 * wq;
                    T acc = T(0);
                    if (u0 < us)
#pragma unroll 2
                        for (uint32_t u = warp * us + u0; u < wk; u += us * warps) acc = fma(Pk[u], E[u * wq + v], acc);
                    for (uint32_t off = wq; off < 32u; off *= 2u) {
                        const T x = __shfl_down_sync(0xffffffffu, acc, off);
                        if (lane + off < 32u) acc += x;
                    }
                    if (lane < wq) part[(G.db[q] + lane) * warps + warp] = acc;
                }
            }
            __syncthreads();
            // the narrow degrees' sums
            for (uint32_t c = t0; c < kNarrow<W> && c < G.dim; c += nt) {
                int q = 0;
                while (c >= G.db[q + 1]) ++q;
                const int k = N - q;
                const bool terms = any && k >= kmin && k <= kmax;
                if (q < out.lo || q > ohi || !(terms || N == D)) continue;
                T acc = N == D ? T(0) : o[c];
                const uint32_t used = terms ? warps : 0u;
                for (uint32_t w = 0; w < used; ++w) acc += part[c * warps + w];
                o[c] = acc;
            }
            __syncthreads();
        }
    }
}

template <typename T, int W>
__global__ void __launch_bounds__(1024) k_shuffle_letters_product(Geometry G, PowerDiv pd, int kind, TArg<T> out,
                                                                  TArg<T> add, TArg<T> lhs, TArg<T> rhs,
                                                                  int64_t batch, T alpha, T beta) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    T* g = reinterpret_cast<T*>(smem_raw);  // degree N of the product, then E^1, E^2, ...
    const int D = G.depth, ohi = imin(out.hi, D), lhi = imin(lhs.hi, D), rhi = imin(rhs.hi, D);
    const uint32_t t0 = threadIdx.x, nt = blockDim.x;
    for (int64_t b = blockIdx.x; b < batch; b += gridDim.x) {
        const T* L = lhs.at(b);
        const T* Rp = rhs.at(b);
        T* o = out.at(b);
        for (int N = ohi; N >= out.lo; --N) {
            const uint32_t size = G.pw[N];
            // the splits |u| = k of both ranges, and the arrays they reach
            const int kmin = imax(imax(lhs.lo, N - rhi), 0), kmax = imin(imin(lhi, N - rhs.lo), N);
            const int top = imin(kmax, N - 1);
            for (uint32_t i = t0; i < size; i += nt) {
                T v = T(0);
                if (kmin <= 0 && kmax >= 0) v = L[0] * Rp[G.db[N] + i];
                if (N > 0 && kmin <= N && kmax >= N) v = fma(L[G.db[N] + i], Rp[0], v);
                g[i] = v;
            }
            for (int k = 1; k <= top; ++k) {
                T* E = g + static_cast<uint32_t>(k) * size;
                for (uint32_t i = t0; i < size; i += nt) {
                    uint32_t u, v;
                    pd.by[N - k].divmod(i, u, v);
                    E[i] = k >= kmin ? L[G.db[k] + u] * Rp[G.db[N - k] + v] : T(0);
                }
            }
            __syncthreads();
            for (int m = N - 1; m >= 1; --m)
                for (int k = 1; k <= imin(m, top); ++k) {
                    const T* E = g + static_cast<uint32_t>(k) * size;
                    T* prev = g + static_cast<uint32_t>(k - 1) * size;  // (k = 1: the product)
                    const int bl = m + 1 - k, R = N - m - 1;
                    if (k == m && k > 1) {
                        // E^m ends here: it is the product's own share too
#pragma unroll 2
                        for (uint32_t i = t0; i < size; i += nt) {
                            prev[i] += E[letter_back<W>(G, pd, i, bl, R)];
                            g[i] += E[i];
                        }
                    } else if (k == m) {
                        for (uint32_t i = t0; i < size; i += nt) g[i] += E[letter_back<W>(G, pd, i, bl, R)] + E[i];
                    } else {
#pragma unroll 2
                        for (uint32_t i = t0; i < size; i += nt) prev[i] += E[letter_back<W>(G, pd, i, bl, R)];
                    }
                    __syncthreads();
                }
            T* oN = o + G.db[N];
            const T* aN = kind == static_cast<int>(ShuffleKind::InplaceFma) ? oN
                          : kind == static_cast<int>(ShuffleKind::Fma) && add.p && add.has(N) ? add.at(b) + G.db[N]
                                                                                              : nullptr;
            for (uint32_t i = t0; i < size; i += nt) {
                T v = g[i] * beta;
                if (aN) v = fma(alpha, aN[i], v);
                oN[i] = v;
            }
            __syncthreads();
        }
    }
}

template <typename T>
size_t letters_smem(const Geometry& g) {
    return static_cast<size_t>(std::max(1, g.depth)) * g.pw[g.depth] * sizeof(T);
}

template <typename T>
size_t letters_adjoint_smem(const Geometry& g, int threads) {
    return letters_smem<T>(g) + (g.dim + 40 * static_cast<size_t>(threads / 32)) * sizeof(T);
}

template <typename T>
bool apart(const Geometry& g, const TArg<T>& a, const TArg<T>& b, int64_t batch) {
    if (!a.p || !b.p || a.lo > a.hi || b.lo > b.hi) return true;
    auto begin = [&](const TArg<T>& t) { return t.p + g.db[t.lo]; };
    auto end = [&](const TArg<T>& t) { return t.p + (batch - 1) * t.stride + g.db[std::min(t.hi, g.depth) + 1]; };
    return end(a) <= begin(b) || end(b) <= begin(a);
}

// Four words of the widest degree a thread; an SM's worth of threads where one
// CTA fits it.
int letters_threads(const Geometry& g, size_t smem) {
    const int most = smem > 110 * 1024 ? 1024 : smem > 72 * 1024 ? 512 : 256;
    return std::max(32, std::min(most, static_cast<int>((g.pw[g.depth] / 4 + 31) / 32 * 32)));
}

PowerDiv power_div(const Geometry& g) {
    PowerDiv pd;
    for (int j = 0; j <= kLettersMaxDepth; ++j) pd.by[j] = FastDiv(j <= g.depth ? g.pw[j] : 1u);
    return pd;
}

// Where dealing letters is the faster way: the steps are barrier-separated, so
// three CTAs an SM are wanted (all in FP32 that fits), or operations that are
// three times fewer at least -- 2^D against D (D+1) / 2.  With one CTA an SM W5 D5
// FP64 took 1 007 us (product) and 1 500 (adjoint), the subsets 832 and 974.
template <typename T>
bool letters_fit(const Geometry& g, const DeviceInfo& dev) {
    const int D = g.depth;
    const size_t smem = letters_smem<T>(g);
    if (!column_width(g.width) || D < 3 || D > kLettersMaxDepth) return false;
    if (smem > std::min(kLettersSmemLimit, static_cast<size_t>(dev.max_smem_optin))) return false;
    return smem <= 66 * 1024 || (1u << D) >= 3u * static_cast<uint32_t>(D * (D + 1) / 2);
}

}  // namespace

// Operands are read as the result is written: the output must lie apart from
// both (the added term may be the output itself).
template <typename T>
bool shuffle_letters_product_fits(const Geometry& g, const DeviceInfo& dev, ShuffleKind kind, const TArg<T>& out,
                                  const TArg<T>& add, const TArg<T>& lhs, const TArg<T>& rhs, int64_t batch) {
    const bool same = add.p == out.p && (batch == 1 || add.stride == out.stride);
    // (degree 3 in FP64, 9 operations against 8: W4 D3 23 us, 20 by subsets)
    if (std::is_same<T, double>::value && g.depth < 4) return false;
    return kind != ShuffleKind::LeftHalf && out.lo <= out.hi && letters_fit<T>(g, dev) && apart(g, out, lhs, batch) &&
           apart(g, out, rhs, batch) && (kind != ShuffleKind::Fma || same || apart(g, out, add, batch));
}

template <typename T>
cudaError_t launch_shuffle_letters_product(const Geometry& g, const DeviceInfo& dev, cudaStream_t s, ShuffleKind kind,
                                           TArg<T> out, TArg<T> add, TArg<T> lhs, TArg<T> rhs, int64_t batch,
                                           double alpha, double beta) {
    const size_t smem = letters_smem<T>(g);
    return with_width(g.width, [&](auto w) {
        constexpr int W = decltype(w)::value;
        return run_column<&k_shuffle_letters_product<T, W>>(dev, s, letters_threads(g, smem), smem, batch, g,
                                                            power_div(g), static_cast<int>(kind), out, add, lhs, rhs,
                                                            batch, static_cast<T>(alpha), static_cast<T>(beta));
    });
}

template <typename T>
bool shuffle_letters_adjoint_fits(const Geometry& g, const DeviceInfo& dev, ShuffleAdjKind kind, const TArg<T>& out,
                                  const TArg<T>& op, const TArg<T>& arg, int64_t batch) {
    return kind == ShuffleAdjKind::Shuffle && out.lo <= out.hi && letters_fit<T>(g, dev) &&
           letters_adjoint_smem<T>(g, letters_threads(g, letters_smem<T>(g))) <= kLettersSmemLimit &&
           apart(g, out, op, batch) && apart(g, out, arg, batch);
}

template <typename T>
cudaError_t launch_shuffle_letters_adjoint(const Geometry& g, const DeviceInfo& dev, cudaStream_t s, TArg<T> out,
                                           TArg<T> op, TArg<T> arg, int64_t batch) {
    const int threads = letters_threads(g, letters_smem<T>(g));
    const size_t smem = letters_adjoint_smem<T>(g, threads);
    return with_width(g.width, [&](auto w) {
        constexpr int W = decltype(w)::value;
        return run_column<&k_shuffle_letters_adjoint<T, W>>(dev, s, threads, smem, batch, g, power_div(g), out, op, arg,
                                                            batch);
    });
}

#define RPP_GB_INSTANTIATE_LETTERS(T)                                                                               \
    template bool shuffle_letters_product_fits<T>(const Geometry&, const DeviceInfo&, ShuffleKind, const TArg<T>&,  \
                                                  const TArg<T>&, const TArg<T>&, const TArg<T>&, int64_t);         \
    template cudaError_t launch_shuffle_letters_product<T>(const Geometry&, const DeviceInfo&, cudaStream_t,        \
                                                           ShuffleKind, TArg<T>, TArg<T>, TArg<T>, TArg<T>,         \
                                                           int64_t, double, double);                                \
    template bool shuffle_letters_adjoint_fits<T>(const Geometry&, const DeviceInfo&, ShuffleAdjKind,               \
                                                  const TArg<T>&, const TArg<T>&, const TArg<T>&, int64_t);         \
    template cudaError_t launch_shuffle_letters_adjoint<T>(const Geometry&, const DeviceInfo&, cudaStream_t, TArg<T>, \
                                                           TArg<T>, TArg<T>, int64_t);

RPP_GB_INSTANTIATE_LETTERS(float)
RPP_GB_INSTANTIATE_LETTERS(double)

}  // namespace rpp_gb

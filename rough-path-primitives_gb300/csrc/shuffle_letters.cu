// shuffle_letters.cu -- the shuffle algebra a letter at a time, for widths 2..8:
// st_mul, st_fma, st_inplace_fma, left_hs_mul and their adjoints.
//
// The subset sums of shuffle.cu take 2^N terms for a word of N letters.  Dealing
// the letters of a word one by one to the two factors instead shares all but
// N^2 / 2 of them.  Adjoint: for a word c s of degree N = M + 1 and arrays over s,
//     E_m^k[r, v, u] = sum over interleavings t of u and v of arg[c r t],
// |u| = k, |v| = m - k, r the M - m letters not yet dealt (last letters first),
//     E_{m+1}^k[r, v, u] = E_m^k[r b, v', u] + E_m^{k-1}[r a, v, u'],
// v = b v', u = a u', and the first letter is dealt last,
//     out[v] += op[c u] E_M^k[v, u],   out[c v] += op[u] E_M^k[v, u],
// summed over u and c (the half-shuffle adjoints take one of the two).  Stored as
// one array of W^M per k in the order r v u, the first term of a step is the same
// place of the array (v takes in the letter beside it), so a step adds E^{k-1},
// with the letter a moved past v, into E^k; E^0 and E^m are the argument itself.
// At N = 5 that is 16 operations a word where the subsets take 32, at N = 8 37
// against 256.  The product is the transpose: E_M^k = L[c u] R[v] + L[u] R[c v]
// (the half-shuffle product: the first), and every step adds E^k, the letter
// moved back, into E^{k-1}.
// A CTA owns a tensor and keeps the arrays of one degree and one first letter (all
// first letters, where they fit) in shared memory, a barrier between the steps;
// these and the index instructions are what bounds it.  Subsets -> letters (us),
// batch 4096 unless said: st_mul FP64 W5 D5 832 -> 687, W6 D5 (2048) 1432 -> 911, W2
// D8 652 -> 181, FP32 W5 D5 496 -> 333, W8 D4 376 -> 262; st_adj_mul FP64 W2 D8 2570 ->
// 428, W3 D6 (3000) 661 -> 376, FP32 W5 D5 686 -> 479, W2 D8 2337 -> 167; left_hs_mul
// FP32 W4 D3 (8192) 17.7 -> 8.9; left_hs_adj_lmul / _rmul W2 D8 FP64 1033 -> 274 / 1773
// -> 312, FP32 937 -> 144 / 1632 -> 152.  What the adjoint's order costs: with whole
// degrees in the order u v r, lanes of a sum on consecutive v and a narrow sum over
// all warps, st_adj_mul alone took 249 at W2 D8 and 279 at W3 D6 in FP64; that order
// has no place for the half-shuffle forms.  It is not the banks: lanes that start at
// their own u, where W is a power of two, take 0.87 to 1.15 times as long, 1.05 in
// most cases; nor the one first letter at a time (all of them at W3 D6 FP64: 1.12).
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

// The letter step's arrays of `block` first letters (the argument or product,
// then E^1 ..), and what lies after them.
template <typename T>
size_t letters_smem(const Geometry& g, uint32_t block, int extras) {
    const int M = g.depth - 1;
    return (static_cast<size_t>(std::max(1, M)) * block * g.pw[M] + static_cast<size_t>(extras) * g.db[g.depth]) *
           sizeof(T);
}

template <typename T, int W>
__global__ void __launch_bounds__(512) k_deal_adjoint(Geometry G, PowerDiv pd, int kind, TArg<T> out, TArg<T> op,
                                                      TArg<T> arg, int64_t batch, T beta, uint32_t block) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    T* g = reinterpret_cast<T*>(smem_raw);
    const int D = G.depth, ohi = imin(out.hi, D), phi = imin(op.hi, D), ahi = imin(arg.hi, D);
    const uint32_t low = G.db[D];
    T* P = g + static_cast<uint32_t>(imax(1, D - 1)) * block * G.pw[D - 1];  // the op below its top degree
    T* sum_v = P + low;       // out[v]'s sums, and out[c v]'s: each updated once a block
    T* sum_cv = sum_v + low;
    const bool to_u = kind != static_cast<int>(ShuffleAdjKind::HalfR);
    const bool to_v = kind != static_cast<int>(ShuffleAdjKind::HalfL);
    const uint32_t t0 = threadIdx.x, nt = blockDim.x, lane = t0 & 31u, warp = t0 >> 5, warps = nt >> 5;
    for (int64_t b = blockIdx.x; b < batch; b += gridDim.x) {
        const T* A = arg.at(b);
        const T* Pg = op.at(b);
        T* o = out.at(b);
        for (uint32_t i = t0; i < low; i += nt) {
            sum_v[i] = sum_cv[i] = T(0);
            P[i] = op.lo <= phi && i >= G.db[op.lo] && i < G.db[phi + 1] ? Pg[i] : T(0);
        }
        __syncthreads();
        bool top = false;  // the top degree's coefficients are written
        for (int N = imin(ahi, D); N >= imax(arg.lo, 1); --N) {
            const int M = N - 1, kcap = imin(M, imin(phi, M + 1 - out.lo));
            if (kcap < 0) continue;
            const uint32_t S = G.pw[M];
            for (uint32_t c0 = 0; c0 < W; c0 += block) {
                const uint32_t size = block * S;
                for (uint32_t i = t0; i < size; i += nt) g[i] = A[G.db[N] + c0 * S + i];
                __syncthreads();
                for (int m = 1; m < M; ++m)
                    for (int k = imin(m, kcap); k >= 1; --k) {
                        T* E = g + static_cast<uint32_t>(k) * size;
                        const T* self = k == m ? g : E;
                        const T* prev = E - size;  // (k = 1: the argument)
#pragma unroll 2
                        for (uint32_t i = t0; i < size; i += nt)
                            E[i] = self[i] + prev[letter_back<W>(G, pd, i, m + 1 - k, k - 1)];
                        __syncthreads();
                    }
                for (int k = 0; k <= kcap; ++k) {
                    const int q = M - k;
                    const bool in_u = to_u && k + 1 >= op.lo && k + 1 <= phi && q >= out.lo && q <= ohi;
                    const bool in_v = to_v && k >= op.lo && k <= phi && q + 1 >= out.lo && q + 1 <= ohi;
                    if (!in_u && !in_v) continue;
                    const uint32_t wq = G.pw[q], wk = G.pw[k];
                    const T* E = (k == 0 || k == M) ? g : g + static_cast<uint32_t>(k) * size;
                    const T* Pu = k + 1 == D ? Pg + G.db[D] : P + G.db[k + 1];  // op[c u]
                    const T* Pv = P + G.db[k];                                   // op[u]
                    // (a warp's sums take five additions more; the barriers between the
                    // blocks order the sums' updates, whichever thread makes them)
                    if (wq >= 16u || wk < 64u) {
                        for (uint32_t v = t0; v < wq; v += nt) {
                            T s = T(0);
                            for (uint32_t c = 0; c < block; ++c) {
                                const T* row = E + (c * wq + v) * wk;
                                const T* pc = Pu + (c0 + c) * wk;
                                T d = T(0);
                                // two chains a long row, and the rows' sums in one: a chain
                                // through all rows rounds more than the subset sums (FP32
                                // st_adj_mul W5 D4 1.36 times, left adjoints 1.2 to 1.5; the
                                // two chains cost 10 to 25 % of the time, and in FP64, where
                                // only rows of 32 need them, 4 %)
                                constexpr uint32_t split = sizeof(T) == 8 ? 32u : 8u;
                                if (wk < split || (sizeof(T) == 4 && !in_u)) {
                                    if (in_u && in_v) {
#pragma unroll 4
                                        for (uint32_t u = 0; u < wk; ++u) {
                                            const T e = row[u];
                                            s = fma(pc[u], e, s);
                                            d = fma(Pv[u], e, d);
                                        }
                                    } else if (in_u) {
#pragma unroll 4
                                        for (uint32_t u = 0; u < wk; ++u) s = fma(pc[u], row[u], s);
                                    } else {
#pragma unroll 4
                                        for (uint32_t u = 0; u < wk; ++u) d = fma(Pv[u], row[u], d);
                                    }
                                } else {
                                    const uint32_t even = wk & ~1u;
                                    T s0 = T(0), s1 = T(0), d1 = T(0);
                                    if (in_u && in_v) {
#pragma unroll 2
                                        for (uint32_t u = 0; u < even; u += 2u) {
                                            const T e = row[u], f = row[u + 1u];
                                            s0 = fma(pc[u], e, s0);
                                            s1 = fma(pc[u + 1u], f, s1);
                                            d = fma(Pv[u], e, d);
                                            d1 = fma(Pv[u + 1u], f, d1);
                                        }
                                    } else if (in_u) {
#pragma unroll 2
                                        for (uint32_t u = 0; u < even; u += 2u) {
                                            s0 = fma(pc[u], row[u], s0);
                                            s1 = fma(pc[u + 1u], row[u + 1u], s1);
                                        }
                                    } else {
#pragma unroll 2
                                        for (uint32_t u = 0; u < even; u += 2u) {
                                            d = fma(Pv[u], row[u], d);
                                            d1 = fma(Pv[u + 1u], row[u + 1u], d1);
                                        }
                                    }
                                    if (even < wk) {
                                        if (in_u) s0 = fma(pc[even], row[even], s0);
                                        if (in_v) d = fma(Pv[even], row[even], d);
                                    }
                                    s += s0 + s1;
                                    d += d1;
                                }
                                if (in_v) {
                                    const uint32_t at = G.db[q + 1] + (c0 + c) * wq + v;
                                    if (q + 1 == D) o[at] = d * beta;
                                    else sum_cv[at] += d;
                                }
                            }
                            if (in_u) sum_v[G.db[q] + v] += s;
                        }
                    } else {
                        for (uint32_t v = warp; v < wq; v += warps) {
                            T s = T(0);
                            for (uint32_t c = 0; c < block; ++c) {
                                const T* row = E + (c * wq + v) * wk;
                                const T* pc = Pu + (c0 + c) * wk;
                                T d = T(0), part = T(0);
#pragma unroll 2
                                for (uint32_t u = lane; u < wk; u += 32u) {
                                    const T e = row[u];
                                    if (in_u) part = fma(pc[u], e, part);
                                    if (in_v) d = fma(Pv[u], e, d);
                                }
                                s += part;
                                if (in_v) {
#pragma unroll
                                    for (uint32_t off = 16u; off > 0u; off /= 2u) d += __shfl_down_sync(0xffffffffu, d, off);
                                    const uint32_t at = G.db[q + 1] + (c0 + c) * wq + v;
                                    if (lane == 0) {
                                        if (q + 1 == D) o[at] = d * beta;
                                        else sum_cv[at] += d;
                                    }
                                }
                            }
                            if (in_u) {
#pragma unroll
                                for (uint32_t off = 16u; off > 0u; off /= 2u) s += __shfl_down_sync(0xffffffffu, s, off);
                                if (lane == 0) sum_v[G.db[q] + v] += s;
                            }
                        }
                    }
                    top = top || (in_v && q + 1 == D);
                }
                __syncthreads();
            }
        }
        if (t0 == 0 && kind == static_cast<int>(ShuffleAdjKind::Shuffle) && arg.lo == 0 && ahi >= 0 && op.lo == 0 &&
            phi >= 0 && out.lo == 0)
            sum_v[0] = fma(P[0], A[0], sum_v[0]);
        __syncthreads();
        for (uint32_t i = G.db[out.lo] + t0; i < G.db[imin(ohi, D - 1) + 1]; i += nt) o[i] = (sum_v[i] + sum_cv[i]) * beta;
        if (ohi == D && !top)
            for (uint32_t i = low + t0; i < G.dim; i += nt) o[i] = T(0);
        __syncthreads();
    }
}

template <typename T, int W>
__global__ void __launch_bounds__(512) k_deal_product(Geometry G, PowerDiv pd, int kind, TArg<T> out, TArg<T> add,
                                                      TArg<T> lhs, TArg<T> rhs, int64_t batch, T alpha, T beta,
                                                      uint32_t block) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    T* g = reinterpret_cast<T*>(smem_raw);
    const int D = G.depth, ohi = imin(out.hi, D);
    const uint32_t low = G.db[D];
    T* sL = g + static_cast<uint32_t>(imax(1, D - 1)) * block * G.pw[D - 1];  // the factors below their top degree
    T* sR = sL + low;
    const bool both = kind != static_cast<int>(ShuffleKind::LeftHalf);
    const uint32_t t0 = threadIdx.x, nt = blockDim.x;
    for (int64_t b = blockIdx.x; b < batch; b += gridDim.x) {
        const T* Lg = lhs.at(b);
        const T* Rg = rhs.at(b);
        T* o = out.at(b);
        for (uint32_t i = t0; i < low; i += nt) {
            sL[i] = Lg[i];
            sR[i] = Rg[i];
        }
        __syncthreads();
        auto L = [&](int n, uint32_t i) -> T { return n < D ? sL[G.db[n] + i] : Lg[low + i]; };
        auto R = [&](int n, uint32_t i) -> T { return n < D ? sR[G.db[n] + i] : Rg[low + i]; };
        // the result of degree N, coefficient `at`, from its product
        auto finish = [&](int N, uint32_t at, T v) {
            v *= beta;
            T* dst = o + G.db[N] + at;
            if (kind == static_cast<int>(ShuffleKind::InplaceFma)) v = fma(alpha, *dst, v);
            else if (kind == static_cast<int>(ShuffleKind::Fma) && add.p && add.has(N)) v = fma(alpha, add.at(b)[G.db[N] + at], v);
            *dst = v;
        };
        for (int N = ohi; N >= imax(out.lo, 1); --N) {
            const int M = N - 1;
            const uint32_t S = G.pw[M];
            for (uint32_t c0 = 0; c0 < W; c0 += block) {
                const uint32_t size = block * S;
                for (uint32_t i = t0; i < size; i += nt) {
                    uint32_t c, j;
                    pd.by[M].divmod(i, c, j);
                    c += c0;
                    T v = L(1, c) * R(M, j);  // k = 0
                    if (both) v = fma(L(0, 0), R(N, c * S + j), v);
                    if (M > 0) {  // k = M
                        v = fma(L(N, c * S + j), R(0, 0), v);
                        if (both) v = fma(L(M, j), R(1, c), v);
                    }
                    if (M == 2) {  // k = 1, dealt here: no sum is rounded that one word alone needs
                        const uint32_t a = j / W, e = j - a * W;
                        v = fma(L(2, c * W + a), R(1, e), v);
                        v = fma(L(2, c * W + e), R(1, a), v);
                        if (both) {
                            v = fma(L(1, a), R(2, c * W + e), v);
                            v = fma(L(1, e), R(2, c * W + a), v);
                        }
                    }
                    g[i] = v;
                }
                for (int k = 1; k < M && M > 2; ++k) {
                    T* E = g + static_cast<uint32_t>(k) * size;
                    const T *Lc = sL + G.db[k + 1], *Lu = sL + G.db[k], *Rv = sR + G.db[M - k], *Rc = sR + G.db[M - k + 1];
                    const uint32_t wk = G.pw[k], wv = G.pw[M - k];
                    for (uint32_t i = t0; i < size; i += nt) {
                        uint32_t t, c, u, v;
                        pd.by[k].divmod(i, t, u);
                        pd.by[M - k].divmod(t, c, v);
                        c += c0;
                        T e = Lc[c * wk + u] * Rv[v];
                        if (both) e = fma(Lu[u], Rc[c * wv + v], e);
                        E[i] = e;
                    }
                }
                __syncthreads();
                for (int m = M - 1; m >= 1 && M > 2; --m)
                    for (int k = 1; k <= m; ++k) {
                        const T* E = g + static_cast<uint32_t>(k) * size;
                        T* prev = g + static_cast<uint32_t>(k - 1) * size;  // (k = 1: the product)
                        const int bl = m + 1 - k, r = k - 1;
                        if (k < m) {
#pragma unroll 2
                            for (uint32_t i = t0; i < size; i += nt) prev[i] += E[letter_past<W>(G, pd, i, bl, r)];
                        } else if (k > 1) {  // E^m ends here: it is the product's own share too
#pragma unroll 2
                            for (uint32_t i = t0; i < size; i += nt) {
                                prev[i] += E[letter_past<W>(G, pd, i, bl, r)];
                                g[i] += E[i];
                            }
                        } else {
                            for (uint32_t i = t0; i < size; i += nt) g[i] += E[letter_past<W>(G, pd, i, bl, r)] + E[i];
                        }
                        __syncthreads();
                    }
                for (uint32_t i = t0; i < size; i += nt) finish(N, c0 * S + i, g[i]);
                __syncthreads();
            }
        }
        if (out.lo == 0 && t0 == 0) {
            if (both) finish(0, 0, L(0, 0) * R(0, 0));
            else o[0] = T(0);
        }
        __syncthreads();
    }
}

// First letters at a time, shared memory and threads (four words each) of a
// launch: all first letters where six CTAs still fit an SM, else one.
template <typename T>
void letters_shape(const Geometry& g, int extras, uint32_t& block, size_t& smem, int& threads) {
    block = static_cast<uint32_t>(g.width);
    if (letters_smem<T>(g, block, extras) > 36 * 1024) block = 1;
    smem = letters_smem<T>(g, block, extras);
    const int most = smem > 100 * 1024 ? 512 : 256;
    threads = std::max(32, std::min(most, static_cast<int>((block * g.pw[g.depth - 1] / 4 + 31) / 32 * 32)));
}
constexpr int kAdjointExtras = 3, kProductExtras = 2;

PowerDiv power_div(const Geometry& g) {
    PowerDiv pd;
    for (int j = 0; j <= kLettersMaxDepth; ++j) pd.by[j] = FastDiv(j <= g.depth ? g.pw[j] : 1u);
    return pd;
}

template <typename T>
bool letters_fit(const Geometry& g, const DeviceInfo& dev, int extras) {
    if (!column_width(g.width) || g.depth < 3 || g.depth > kLettersMaxDepth) return false;
    uint32_t block;
    size_t smem;
    int threads;
    letters_shape<T>(g, extras, block, smem, threads);
    return smem <= std::min(kLettersSmemLimit, static_cast<size_t>(dev.max_smem_optin));
}

// Where dealing letters is the faster way: from how many tensors an SM on (kAny,
// kNone).  From degree 6 on it has a third of the operations or fewer.  Below, FP32
// gains from its plain loops, except where a half-shuffle adjoint of a wide tensor
// waits at its barriers (W6 D5 left 634 us, 360 by subsets); FP64 only where most of
// the operations are additions, the products (W4 D4 16.5 -> 13.6; but W8 D4 611, 558
// by subsets; left_hs_mul W5 D5 546, 467; st_adj_mul W5 D5 1263, 974).
// The steps are short and end in barriers, which an SM with a CTA or two waits at,
// where the subset sums have a thread per coefficient and none: six to eight an SM
// are needed (letters over subsets at batch 64, 608 and 1 300: st_adj_mul FP32 W7 D3
// 3.1, 1.5 and 1.0; st_mul FP64 W4 D5 2.5, 1.15 and 0.85; left_hs_mul FP64 W2 D7 2.4,
// 1.45 and 0.85), more for the smallest tensors, two or none where the operations
// saved outweigh the waits (W3 D6 st_mul FP64 0.9 at batch 64, 0.6 at 4 096).
// Measured at W 2..8, every depth from 3 to 6 000 coefficients.
enum : int { kAny = 0, kFew = 2, kSome = 6, kFull = 8, kMany = 20, kNone = 1 << 30 };

template <typename T>
int letters_need(const Geometry& g, ShuffleKind kind) {
    constexpr bool fp64 = std::is_same<T, double>::value;
    const int W = g.width, D = g.depth;
    const bool mid = !fp64 && g.dim >= 1000 && g.dim < 3500;
    if (kind == ShuffleKind::LeftHalf) {
        if (fp64 && D < 6 && g.dim > 1200) return kNone;
        if (D >= (fp64 ? 10 : 9) || (mid && W >= 4) || (D == 3 && (W == 4 || W == 8))) return kAny;
        if ((W == 2 && D == 5) || (fp64 && D == 4 && W <= 3)) return kNone;
        if (W == 2 && (D == 4 || D == 6 || (D == 7 && !fp64))) return kMany;
        if (fp64 && ((W == 3 && D == 5) || (W == 5 && D == 4))) return kMany;
        if ((W >= 3 && W <= 4 && D >= 6) || (W == 2 && D >= 8 && fp64) || (D == 3 && W >= 6) || (W == 5 && D == 4))
            return kFew;
    } else {
        if (fp64 && (D < 4 || (D == 4 && W > 6))) return kNone;
        if (D >= (fp64 ? 8 : 9) || (W >= 3 && D >= 6) || mid) return kAny;
        if (fp64 && D < 6 && W <= 3 && g.dim < 128) return kNone;  // W2 D4, D5, W3 D4
        if (!fp64 && W <= 3 && g.dim < 128) return kMany;
        if ((W == 2 && D == 8) || (W >= 5 && g.dim >= 500 && g.dim < 4000)) return kFew;
    }
    return g.dim < 256 ? kFull : kSome;
}

template <typename T>
int letters_need(const Geometry& g, ShuffleAdjKind kind) {
    constexpr bool fp64 = std::is_same<T, double>::value;
    const int W = g.width, D = g.depth;
    if (fp64 && D < 6) return kNone;
    // (FP64 W3 D6, left: 0.79 of the subsets' time, but 1.5 times their rounding error)
    if (fp64 && W == 3 && D == 6) return kind == ShuffleAdjKind::HalfL ? kNone : kSome;
    if (kind == ShuffleAdjKind::Shuffle) {
        if (W == 2 || D >= 6 || (W == 3 && D <= 4) || (W == 4 && D == 5)) return kAny;
        // (all first letters at once, in one long pass a degree: 1.3 times the subsets' time)
        if (W == 7 && D == 4) return kNone;
        if (D == 4 && (W == 5 || W == 6)) return kFew;
        return D == 3 && W >= 5 && W <= 7 ? kMany : 4;
    }
    if (W >= 4 && D >= 6) return kFew;
    if (kind == ShuffleAdjKind::HalfL) {
        if (D < 6 && g.dim > 700) return kNone;
        if ((W == 2 && D >= 4) || (W == 3 && (D == 4 || D >= 6))) return kAny;
        return W >= 5 && W <= 7 ? kMany : kFull;
    }
    if (D < 6 && (D < 4 || W == 6 || g.dim > 5000)) return kNone;
    if ((W <= 3 && D >= 5) || W == 7) return kAny;
    return W == 2 && D == 4 ? kMany : W == 4 ? 4 : kFull;
}

template <typename T, typename Kind>
bool letters_pay(const Geometry& g, const DeviceInfo& dev, Kind kind, int64_t batch) {
    return batch >= static_cast<int64_t>(letters_need<T>(g, kind)) * dev.sm_count;
}

}  // namespace

// Operands are read as the result is written: the output must lie apart from
// both (the added term may be the output itself).  The product's factors are
// whole tensors (degrees that a view lacks would be multiplied as zeros).
template <typename T>
bool shuffle_letters_product_fits(const Geometry& g, const DeviceInfo& dev, ShuffleKind kind, const TArg<T>& out,
                                  const TArg<T>& add, const TArg<T>& lhs, const TArg<T>& rhs, int64_t batch) {
    const bool same = add.p == out.p && (batch == 1 || add.stride == out.stride);
    const bool whole = lhs.lo == 0 && rhs.lo == 0 && lhs.hi >= g.depth && rhs.hi >= g.depth;
    return whole && out.lo <= out.hi && letters_pay<T>(g, dev, kind, batch) && letters_fit<T>(g, dev, kProductExtras) && apart(g, out, lhs, batch) &&
           apart(g, out, rhs, batch) && (kind != ShuffleKind::Fma || same || apart(g, out, add, batch));
}

template <typename T>
cudaError_t launch_shuffle_letters_product(const Geometry& g, const DeviceInfo& dev, cudaStream_t s, ShuffleKind kind,
                                           TArg<T> out, TArg<T> add, TArg<T> lhs, TArg<T> rhs, int64_t batch,
                                           double alpha, double beta) {
    uint32_t block;
    size_t smem;
    int threads;
    letters_shape<T>(g, kProductExtras, block, smem, threads);
    return with_width(g.width, [&](auto w) {
        constexpr int W = decltype(w)::value;
        return run_column<&k_deal_product<T, W>>(dev, s, threads, smem, batch, g, power_div(g), static_cast<int>(kind),
                                                 out, add, lhs, rhs, batch, static_cast<T>(alpha),
                                                 static_cast<T>(beta), block);
    });
}

template <typename T>
bool shuffle_letters_adjoint_fits(const Geometry& g, const DeviceInfo& dev, ShuffleAdjKind kind, const TArg<T>& out,
                                  const TArg<T>& op, const TArg<T>& arg, int64_t batch) {
    return out.lo <= out.hi && letters_pay<T>(g, dev, kind, batch) && letters_fit<T>(g, dev, kAdjointExtras) && apart(g, out, op, batch) &&
           apart(g, out, arg, batch);
}

template <typename T>
cudaError_t launch_shuffle_letters_adjoint(const Geometry& g, const DeviceInfo& dev, cudaStream_t s,
                                           ShuffleAdjKind kind, TArg<T> out, TArg<T> op, TArg<T> arg, int64_t batch,
                                           double beta) {
    uint32_t block;
    size_t smem;
    int threads;
    letters_shape<T>(g, kAdjointExtras, block, smem, threads);
    return with_width(g.width, [&](auto w) {
        constexpr int W = decltype(w)::value;
        return run_column<&k_deal_adjoint<T, W>>(dev, s, threads, smem, batch, g, power_div(g), static_cast<int>(kind),
                                                 out, op, arg, batch, static_cast<T>(beta), block);
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
    template cudaError_t launch_shuffle_letters_adjoint<T>(const Geometry&, const DeviceInfo&, cudaStream_t,        \
                                                           ShuffleAdjKind, TArg<T>, TArg<T>, TArg<T>, int64_t, double);

RPP_GB_INSTANTIATE_LETTERS(float)
RPP_GB_INSTANTIATE_LETTERS(double)

}  // namespace rpp_gb

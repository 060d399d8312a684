// Variants of one LP that differ only in their variable bounds, solved
// together with the matrix read once per iteration for all of them (included
// once, by engine.cu after batch.cuh).
//
// Branch and bound creates such LPs: every node of a round is the parent LP
// with a few bounds tightened (src/milp/milp_solver.cpp:401-447).  Packing K
// copies block-diagonally (batch.cuh) streams the matrix K times per
// iteration and turns every nonzero into K random 8-byte gathers.  Here the
// iterates are stored variant-minor -- element (j, k) of an n x K array at
// j * Kp + k, Kp = K rounded up to 32 -- and neighbouring lanes carry the
// variants of a line: a nonzero a_ij is loaded once per warp (a broadcast) and
// the gathered vector entry for 32 variants is one contiguous read.
//
// Every variant still runs the reference algorithm on its own
// (src/lp/first_order/pdlp.cpp:139-276): own step size, primal weight,
// restarts and termination, from its own DevState.  The shared setup (Ruiz
// scaling, norms, c, row bounds, the initial primal weight) depends only on
// A, c and the row bounds, which the variants share; their bounds are scaled
// and projected per variant.  Reductions are per variant: each block writes
// one partial per variant and a per-variant kernel sums them in a fixed
// order, so results are run-to-run deterministic.  Infeasible variants are
// certified as in the packed batch (crossed bounds, row activity, and the
// Farkas test of the dual ray candidate at every restart check).
#pragma once

#include "batch.cuh"

namespace mc {

constexpr int kVarWarps = kBlock / 32;  // warps per block, one line each per trip
constexpr int kVarGathers = 4;          // gathers in flight per lane (split_dot)
constexpr int kVarDualBlocks = 2;       // blocks per SM of the split dual kernels
constexpr int kVarLongColumn = 64;      // longest column above which kv_primal_wide asks for indices ahead (pack_dot)

// The base LP (scaled, shared by every variant).
struct VarBase {
    int m, n;
    const int* cs;        // CSC of the scaled A
    const int* ri;
    const double* cv;
    const int* rs;        // CSR of the scaled A
    const int* ci;
    const double* rv;
    const double* c;      // scaled objective (minimisation sign)
    const double* col_norm;
    const double* row_norm;
    const double* blo;    // scaled row bounds, sentinel form
    const double* bhi;
};

// The per-variant arrays (variant-minor, row stride Kp).
struct VarRefs {
    int K, Kp, nb;         // variants, padded count, blocks per grid row (partials per variant)
    DevState* st;          // [K]
    DevState* global;      // poll flag: every variant done
    double* lo;            // [n Kp] scaled bounds, sentinel form
    double* hi;
    double* olo;           // [n Kp] original bounds, sentinel form
    double* ohi;
    double* x;             // [n Kp]
    double* xb;            // [n Kp] x-bar (non-step iterations)
    double* xa;            // [n Kp] average
    double* xdx;           // [2 n Kp] (x-bar, dx) pairs (step-size iterations)
    double* y;             // [m Kp]
    double* ya;
    double* axb;           // [m Kp] A x-bar of a step-size iteration
    double* y_prev;        // [m Kp] dual average at the previous check (the start at setup)
    double* dray;          // [m Kp] the dual ray candidate of the current check
    double* partials;      // [NUM_SLOTS Kp nb]
    int* flags;            // [K] setup certificates: 1 crossed bounds, 2 row activity
    int* cert_idx;         // [2K] lowest crossed column, lowest failing row (INT_MAX if none)
};

__device__ __forceinline__ double* var_partial(const VarRefs& V, int slot, int k) {
    return V.partials + ((size_t)slot * V.Kp + k) * V.nb;
}

// Sum (or max) of one value per lane over the block's warps, in warp order;
// the result is valid in warp 0 (lane = variant).  Ends with a barrier.
template <class Op>
__device__ __forceinline__ double lanes_reduce(double v, double (*sm)[33], Op op) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    sm[warp][lane] = v;
    __syncthreads();
    if (warp == 0)
        for (int w = 1; w < kVarWarps; ++w) v = op(v, sm[w][lane]);
    __syncthreads();
    return v;
}

// The lane's variant; `live` when it exists and still runs.  Every block
// works on one group of 32 variants (blockIdx.y), so a block whose variants
// have all finished leaves as a whole.
#define MC_VARIANT_LANE(V, K_, LIVE)                                   \
    const int lane_ = threadIdx.x & 31;                                \
    const int K_ = blockIdx.y * 32 + lane_;                            \
    const bool LIVE = K_ < (V).K && !(V).st[K_].done;                  \
    if (!__syncthreads_or(LIVE)) return;

// Lines of the block's warps: line = blockIdx.x * warps + warp, strided over the grid.
#define MC_VARIANT_LINES(LINE, COUNT)                                                            \
    for (long long LINE = (long long)blockIdx.x * kVarWarps + (threadIdx.x >> 5); LINE < (COUNT); \
         LINE += (long long)gridDim.x * kVarWarps)

// Dot of CSR/CSC line `l` with the variant-minor vector v (column k), four
// gathers in flight; inactive lanes issue no loads.
__device__ __forceinline__ double variant_dot(const int* __restrict__ start, const int* __restrict__ idx,
                                              const double* __restrict__ val, const double* __restrict__ v,
                                              int Kp, long long l, int k, bool live, unsigned long long pol) {
    const int b = __ldg(start + l), e = __ldg(start + l + 1);
    double s0 = 0.0, s1 = 0.0, s2 = 0.0, s3 = 0.0;
    int p = b;
    for (; p + 4 <= e; p += 4) {
        const int i0 = __ldg(idx + p), i1 = __ldg(idx + p + 1), i2 = __ldg(idx + p + 2), i3 = __ldg(idx + p + 3);
        const double a0 = __ldg(val + p), a1 = __ldg(val + p + 1), a2 = __ldg(val + p + 2), a3 = __ldg(val + p + 3);
        if (live) {
            s0 = fma(a0, ld_keep(v + (size_t)i0 * Kp + k, pol), s0);
            s1 = fma(a1, ld_keep(v + (size_t)i1 * Kp + k, pol), s1);
            s2 = fma(a2, ld_keep(v + (size_t)i2 * Kp + k, pol), s2);
            s3 = fma(a3, ld_keep(v + (size_t)i3 * Kp + k, pol), s3);
        }
    }
    for (; p < e; ++p)
        if (live) s0 = fma(__ldg(val + p), ld_keep(v + (size_t)__ldg(idx + p) * Kp + k, pol), s0);
    return (s0 + s1) + (s2 + s3);
}

// ------------------------------------------------------------------ primal
// g = c + A^T y; x+ = clamp(x - tau g, l, u); x-bar; average; on step-size
// iterations dx and sum col_norm dx^2 per variant (pdlp.cpp:195-206, :226).
// This form, with the reduction, is that of a step-size iteration.
__global__ void __launch_bounds__(kBlock) kv_primal_step(VarBase Bs, VarRefs V, int kk) {
    __shared__ double sm[kVarWarps][33];
    MC_VARIANT_LANE(V, k, live);
    double step = 0.0, cnt = 1.0;
    if (live) {
        const DevState& s = V.st[k];
        step = s.eta / s.omega;
        cnt = (double)(s.avg_count + kk + 1);
    }
    const unsigned long long pol = policy_keep();
    double acc = 0.0;
    MC_VARIANT_LINES(j, Bs.n) {
        const double aty = variant_dot(Bs.cs, Bs.ri, Bs.cv, V.y, V.Kp, j, k, live, pol);
        if (live) {
            const size_t q = (size_t)j * V.Kp + k;
            const double cn = __ldg(Bs.col_norm + j);
            const double g = __dadd_rn(__ldg(Bs.c + j), aty);
            const double tau = __ddiv_rn(step, cn);
            const double xo = ld_stream(V.x + q);
            const double xp = clampv(__dsub_rn(xo, __dmul_rn(tau, g)), ld_stream(V.lo + q), ld_stream(V.hi + q));
            const double d = __dsub_rn(xp, xo);
            const double xbar = __dsub_rn(__dmul_rn(2.0, xp), xo);
            st_keep2(V.xdx + 2 * q, xbar, d, pol);
            acc += __dmul_rn(__dmul_rn(cn, d), d);
            st_stream(V.x + q, xp);
            const double xa = ld_stream(V.xa + q);
            st_stream(V.xa + q, __dadd_rn(xa, __ddiv_rn(__dsub_rn(xp, xa), cnt)));
        }
    }
    acc = lanes_reduce(acc, sm, OpSum());
    if ((threadIdx.x >> 5) == 0 && k < V.K) var_partial(V, SLOT_DX, k)[blockIdx.x] = acc;
}

// Step-size iteration: A x-bar (kept) and A dx from the (x-bar, dx) pairs,
// sum (A dx)_i^2 / row_norm_i per variant (pdlp.cpp:207-210)
__global__ void __launch_bounds__(kBlock) kv_dual_probe(VarBase Bs, VarRefs V) {
    __shared__ double sm[kVarWarps][33];
    MC_VARIANT_LANE(V, k, live);
    const unsigned long long pol = policy_keep();
    double acc = 0.0;
    MC_VARIANT_LINES(i, Bs.m) {
        const int b = __ldg(Bs.rs + i), e = __ldg(Bs.rs + i + 1);
        double sv0 = 0.0, sw0 = 0.0, sv1 = 0.0, sw1 = 0.0;
        int p = b;
        for (; p + 2 <= e; p += 2) {
            const int j0 = __ldg(Bs.ci + p), j1 = __ldg(Bs.ci + p + 1);
            const double a0 = __ldg(Bs.rv + p), a1 = __ldg(Bs.rv + p + 1);
            if (live) {
                double v0, w0, v1, w1;
                ld_keep2(V.xdx + 2 * ((size_t)j0 * V.Kp + k), pol, v0, w0);
                ld_keep2(V.xdx + 2 * ((size_t)j1 * V.Kp + k), pol, v1, w1);
                sv0 = fma(a0, v0, sv0);
                sw0 = fma(a0, w0, sw0);
                sv1 = fma(a1, v1, sv1);
                sw1 = fma(a1, w1, sw1);
            }
        }
        if (p < e && live) {
            double v0, w0;
            ld_keep2(V.xdx + 2 * ((size_t)__ldg(Bs.ci + p) * V.Kp + k), pol, v0, w0);
            const double a0 = __ldg(Bs.rv + p);
            sv0 = fma(a0, v0, sv0);
            sw0 = fma(a0, w0, sw0);
        }
        if (live) {
            V.axb[(size_t)i * V.Kp + k] = sv0 + sv1;
            const double adx = sw0 + sw1;
            acc += __ddiv_rn(__dmul_rn(adx, adx), __ldg(Bs.row_norm + i));
        }
    }
    acc = lanes_reduce(acc, sm, OpSum());
    if ((threadIdx.x >> 5) == 0 && k < V.K) var_partial(V, SLOT_ADX, k)[blockIdx.x] = acc;
}

// The adaptive eta rule per variant (pdlp.cpp:207-219), one block per variant.
__global__ void kv_step_size(VarRefs V, Controls ctl) {
    __shared__ double scratch[32];
    const int k = blockIdx.x;
    DevState* st = V.st + k;
    if (st->done) return;
    const double dxn = reduce_partials(var_partial(V, SLOT_DX, k), V.nb, scratch, OpSum());
    const double adx = reduce_partials(var_partial(V, SLOT_ADX, k), V.nb, scratch, OpSum());
    if (threadIdx.x == 0 && ctl.adaptive_step) st->eta = next_eta(st->eta, dxn, adx);
}

// ---------------------------------------------------------- pack kernels
// The iterations without a step-size probe reduce nothing over lines, so
// their kernels may share the work out in another way than a warp per line
// with one variant per lane.  That form waited: L2 was 11% busy, the issue
// slots 42%, and a column of 8 entries was a chain of 6 dependent reads.  Two
// forms replace it, both with the sums of variant_dot in the same order:
//  - packs (`*_wide`): a thread carries the variants of one 16-byte load (4
//    FP32, 2 FP64) of a line, `1 << lg` neighbouring threads (8 to 32) the
//    whole line or a 128-byte multiple of it.  One index, one address and one
//    gather serve the pack, the last 1-3 entries are loaded together, the
//    line's own vectors before the gathers are waited for.
//  - split rows (kv_dual, kvm_dual): see split_dot.
// us per launch, before -> now, 2000 x 6000 with 8 entries a column: primal
// (packs) FP32 18.8 -> 15.3, FP64 21.8 -> 20.1 at 128 variants, 60.5 -> 41.5 and
// 107 -> 79 at 512 (3000 x 9000); dual 16.8 -> 14.1 and 20.3 -> 14.8 (packs, 128),
// 12.7 -> 8.6 and 13.7 -> 10.7 (split, 32).  Columns are short, so the split
// form gains nothing there (FP32 12.7 against 10.7 for packs at 32 variants).
template <class T> struct PackOf;
template <> struct PackOf<float> { using type = float4; };
template <> struct PackOf<double> { using type = double2; };

template <class T>
struct alignas(16) Pack {
    static constexpr int W = 16 / sizeof(T);
    T v[W];
};
__device__ __forceinline__ Pack<float> ld_keep_pack(const float* a, unsigned long long pol) {
    Pack<float> r;
    asm("ld.global.nc.L1::no_allocate.L2::cache_hint.v4.f32 {%0, %1, %2, %3}, [%4], %5;"
        : "=f"(r.v[0]), "=f"(r.v[1]), "=f"(r.v[2]), "=f"(r.v[3]) : "l"(a), "l"(pol));
    return r;
}
__device__ __forceinline__ Pack<double> ld_keep_pack(const double* a, unsigned long long pol) {
    Pack<double> r;
    ld_keep2(a, pol, r.v[0], r.v[1]);
    return r;
}
__device__ __forceinline__ void st_keep_pack(float* a, const Pack<float>& r, unsigned long long pol) {
    asm volatile("st.global.L2::cache_hint.v4.f32 [%0], {%1, %2, %3, %4}, %5;" ::"l"(a), "f"(r.v[0]), "f"(r.v[1]),
                 "f"(r.v[2]), "f"(r.v[3]), "l"(pol) : "memory");
}
__device__ __forceinline__ void st_keep_pack(double* a, const Pack<double>& r, unsigned long long pol) {
    st_keep2(a, r.v[0], r.v[1], pol);
}
template <class T>
__device__ __forceinline__ Pack<T> ld_pack(const T* a) {
    using Q = typename PackOf<T>::type;
    Pack<T> r;
    *reinterpret_cast<Q*>(&r) = __ldcs(reinterpret_cast<const Q*>(a));
    return r;
}
template <class T>
__device__ __forceinline__ void st_pack(T* a, const Pack<T>& r) {
    using Q = typename PackOf<T>::type;
    __stcs(reinterpret_cast<Q*>(a), *reinterpret_cast<const Q*>(&r));
}

// The pack of this thread: its first variant, its lines (first, stride), and
// per variant the step factor and averaging count of this iteration.
template <class T>
struct VarPack {
    static constexpr int W = Pack<T>::W;
    int k;
    long long line, stride;
    bool any, live[W];
    T step[W], cnt[W];
    __device__ __forceinline__ VarPack(const VarRefs& V, int lg, int kk, bool dual) {
        k = W * ((blockIdx.y << lg) + (threadIdx.x & ((1 << lg) - 1)));
        line = (long long)blockIdx.x * (kBlock >> lg) + (threadIdx.x >> lg);
        stride = (long long)gridDim.x * (kBlock >> lg);
        any = false;
        // every state is read at once (no branch on `done` between the loads)
        double eta[W], omega[W];
        long long count[W];
        int done[W];
#pragma unroll
        for (int w = 0; w < W; ++w) {
            const DevState& s = V.st[min(k + w, V.K - 1)];
            done[w] = s.done;
            eta[w] = s.eta;
            omega[w] = s.omega;
            count[w] = s.avg_count;
        }
#pragma unroll
        for (int w = 0; w < W; ++w) {
            live[w] = k + w < V.K && !done[w];
            any |= live[w];
            step[w] = (T)(dual ? eta[w] * omega[w] : eta[w] / omega[w]);
            cnt[w] = (T)(double)(count[w] + kk + 1);
        }
    }
};

// variant_dot for a pack: v points at the pack of line 0.  A window adds entry
// q to sum q mod 4, the tail all of its entries to the first.
template <int N, class T>
__device__ __forceinline__ void pack_window(const int* __restrict__ idx, const T* __restrict__ val,
                                            const T* __restrict__ v, int Kp, int p, unsigned long long pol,
                                            T (&s)[4][Pack<T>::W], bool tail = false) {
    int i[N];
    T a[N];
    Pack<T> g[N];
#pragma unroll
    for (int q = 0; q < N; ++q) {
        i[q] = __ldg(idx + p + q);
        a[q] = __ldg(val + p + q);
    }
#pragma unroll
    for (int q = 0; q < N; ++q) g[q] = ld_keep_pack(v + (size_t)i[q] * Kp, pol);
#pragma unroll
    for (int q = 0; q < N; ++q)
#pragma unroll
        for (int w = 0; w < Pack<T>::W; ++w) {
            T& t = s[tail ? 0 : (q & 3)][w];
            t = fma(a[q], g[q].v[w], t);
        }
}
// AHEAD (rows): the indices of the next window are asked for before the
// gathers of this one are waited for: dual 18.7 -> 14.1 us (128 variants, FP32).
// Columns rarely fill one window, and the registers cost a block per SM; but a
// long one is a chain of windows, and all others wait for it, so FP64 columns
// are asked for ahead where the longest has more than kVarLongColumn entries: 120
// iterations of 4 variants of 2000 x 6000 with a column of 256 entries 7.5 -> 4.4 ms
// (7.2 with a warp per line), with one of 64 3.6 -> 2.9, of 32 2.95 either way.
template <bool AHEAD, class T>
__device__ __forceinline__ Pack<T> pack_dot(int b, int e, const int* __restrict__ idx, const T* __restrict__ val,
                                            const T* __restrict__ v, int Kp, unsigned long long pol) {
    T s[4][Pack<T>::W] = {};
    int p = b;
    if (!AHEAD) {
        for (; p + 8 <= e; p += 8) pack_window<8>(idx, val, v, Kp, p, pol, s);
    } else if (p + 8 <= e) {
        int i[8];
        T a[8];
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            i[q] = __ldg(idx + p + q);
            a[q] = __ldg(val + p + q);
        }
        for (; p + 8 <= e; p += 8) {
            Pack<T> g[8];
            T x[8];
#pragma unroll
            for (int q = 0; q < 8; ++q) {
                g[q] = ld_keep_pack(v + (size_t)i[q] * Kp, pol);
                x[q] = a[q];
            }
            if (p + 16 <= e) {
#pragma unroll
                for (int q = 0; q < 8; ++q) {
                    i[q] = __ldg(idx + p + 8 + q);
                    a[q] = __ldg(val + p + 8 + q);
                }
            }
#pragma unroll
            for (int q = 0; q < 8; ++q)
#pragma unroll
                for (int w = 0; w < Pack<T>::W; ++w) s[q & 3][w] = fma(x[q], g[q].v[w], s[q & 3][w]);
        }
    }
    if (p + 4 <= e) {
        pack_window<4>(idx, val, v, Kp, p, pol, s);
        p += 4;
    }
    if (e - p == 3) pack_window<3>(idx, val, v, Kp, p, pol, s, true);
    else if (e - p == 2) pack_window<2>(idx, val, v, Kp, p, pol, s, true);
    else if (e - p == 1) pack_window<1>(idx, val, v, Kp, p, pol, s, true);
    Pack<T> r;
#pragma unroll
    for (int w = 0; w < Pack<T>::W; ++w) r.v[w] = (s[0][w] + s[1][w]) + (s[2][w] + s[3][w]);
    return r;
}

// Grid of a pack kernel: 1 << lg threads per line, the largest power of two up
// to 32 that divides the packs of a line; one wave of resident blocks.
struct WideGrid {
    int lg;
    dim3 grid;
};
template <class T, class K>
WideGrid wide_grid(const Ctx& ctx, K kernel, long long lines, int Kp) {
    const int packs = Kp / Pack<T>::W;
    WideGrid g;
    for (g.lg = 3; g.lg < 5 && packs % (2 << g.lg) == 0;) ++g.lg;
    const int gy = packs >> g.lg;
    const long long per_block = kBlock >> g.lg;
    const long long wave = grid_for(ctx, kernel, 1LL << 30, 1);
    const long long x = std::min((lines + per_block - 1) / per_block, std::max<long long>(1, wave / gy));
    g.grid = dim3((unsigned)std::max<long long>(1, x), (unsigned)gy);
    return g;
}

// Grid of a split dual kernel: a warp per line and 32 variants, one wave of resident blocks.
template <class K>
dim3 dual_grid(const Ctx& ctx, K kernel, long long lines, int groups) {
    const long long wave = grid_for(ctx, kernel, 1LL << 30, 1);
    const long long x = std::min((lines + kVarWarps - 1) / kVarWarps, std::max<long long>(1, wave / groups));
    return dim3((unsigned)std::max<long long>(1, x), (unsigned)groups);
}

// From the pack of each of W neighbouring lanes, the sum over those lanes of
// the lane's own variant (lane mod W).  FP32: (s0 + s1) + (s2 + s3).
__device__ __forceinline__ float pack_fold(const float (&s)[1][4]) {
    const bool b0 = threadIdx.x & 1, b1 = threadIdx.x & 2;
    const float lo = (b0 ? s[0][1] : s[0][0]) + __shfl_xor_sync(0xffffffffu, b0 ? s[0][0] : s[0][1], 1);
    const float hi = (b0 ? s[0][3] : s[0][2]) + __shfl_xor_sync(0xffffffffu, b0 ? s[0][2] : s[0][3], 1);
    return (b1 ? hi : lo) + __shfl_xor_sync(0xffffffffu, b1 ? lo : hi, 2);
}
__device__ __forceinline__ double pack_fold(const double (&s)[2][2]) {
    const bool b0 = threadIdx.x & 1;
    const double u = (b0 ? s[0][1] : s[0][0]) + __shfl_xor_sync(0xffffffffu, b0 ? s[0][0] : s[0][1], 1);
    const double w = (b0 ? s[1][1] : s[1][0]) + __shfl_xor_sync(0xffffffffu, b0 ? s[1][0] : s[1][1], 1);
    return u + w;
}

// Whether a lane's pack holds a running variant.
template <class T>
__device__ __forceinline__ bool pack_any(bool live) {
    constexpr int W = Pack<T>::W;
    return (__ballot_sync(0xffffffffu, live) >> (threadIdx.x & 31 & ~(W - 1))) & ((1u << W) - 1u);
}

// variant_dot by the whole warp, for rows of many entries and few variants.
// W neighbouring lanes share the packs of their W variants: each gathers all W
// variants of its own one (FP64: two) of the four running sums, and pack_fold
// hands every lane its variant.  So a warp's load covers 4 (FP64: 2) entries,
// a row of 24 is two dependent gathers instead of six, and the next entries'
// indices are asked for before the gathers at hand are used.  `need`: the
// lane's pack has a running variant.
template <class T>
__device__ __forceinline__ T split_dot(int b, int e, const int* __restrict__ idx, const T* __restrict__ val,
                                         const T* __restrict__ v, int Kp, int k, bool need,
                                         unsigned long long pol) {
    constexpr int W = Pack<T>::W, C = 4 / W, U = kVarGathers / C;  // sums per lane, windows of four per turn
    const int q = threadIdx.x & (W - 1);
    v += k - q;
    const int nw = (e - b) >> 2, tail = b + 4 * nw, rest = e - tail;
    T s[C][W] = {};
    if (need) {
        T ta[3];
        Pack<T> tg[3];
        const bool first = q == 0;
#pragma unroll
        for (int u = 0; u < 3; ++u)
            if (u < rest && first) {
                ta[u] = __ldg(val + tail + u);
                tg[u] = ld_keep_pack(v + (size_t)__ldg(idx + tail + u) * Kp, pol);
            }
        int i[U][C];
        T a[U][C];
        const int p = b + q;
#pragma unroll
        for (int u = 0; u < U; ++u)
            if (u < nw)
#pragma unroll
                for (int c = 0; c < C; ++c) {
                    i[u][c] = __ldg(idx + p + 4 * u + W * c);
                    a[u][c] = __ldg(val + p + 4 * u + W * c);
                }
        for (int t = 0; t < nw; t += U) {
            Pack<T> g[U][C];
            T x[U][C];
#pragma unroll
            for (int u = 0; u < U; ++u)
                if (t + u < nw)
#pragma unroll
                    for (int c = 0; c < C; ++c) {
                        g[u][c] = ld_keep_pack(v + (size_t)i[u][c] * Kp, pol);
                        x[u][c] = a[u][c];
                    }
#pragma unroll
            for (int u = 0; u < U; ++u)
                if (t + U + u < nw)
#pragma unroll
                    for (int c = 0; c < C; ++c) {
                        i[u][c] = __ldg(idx + p + 4 * (t + U + u) + W * c);
                        a[u][c] = __ldg(val + p + 4 * (t + U + u) + W * c);
                    }
#pragma unroll
            for (int u = 0; u < U; ++u)
                if (t + u < nw)
#pragma unroll
                    for (int c = 0; c < C; ++c)
#pragma unroll
                        for (int w = 0; w < W; ++w) s[c][w] = fma(x[u][c], g[u][c].v[w], s[c][w]);
        }
#pragma unroll
        for (int u = 0; u < 3; ++u)
            if (u < rest && first)
#pragma unroll
                for (int w = 0; w < W; ++w) s[0][w] = fma(ta[u], tg[u].v[w], s[0][w]);
    }
    return pack_fold(s);
}

// The lane's variant in a dual kernel: no reduction over lines there, so a warp
// whose variants have all finished leaves by itself; the state is read at once.
struct DualLane {
    int k;
    bool live, need;
    double sg, cnt;
    template <class T>
    __device__ __forceinline__ static DualLane of(const VarRefs& V, int kk) {
        DualLane d;
        d.k = blockIdx.y * 32 + (threadIdx.x & 31);
        const DevState& s = V.st[min(d.k, V.K - 1)];
        d.live = d.k < V.K && !s.done;
        d.sg = s.eta * s.omega;
        d.cnt = (double)(s.avg_count + kk + 1);
        d.need = pack_any<T>(d.live);
        return d;
    }
};

// the primal step of an iteration without a probe (kv_primal_step has the formulas)
template <bool AHEAD>
__global__ void __launch_bounds__(kBlock) kv_primal_wide(VarBase Bs, VarRefs V, int lg, int kk) {
    const VarPack<double> me(V, lg, kk, false);
    if (!me.any) return;
    constexpr int W = Pack<double>::W;
    const unsigned long long pol = policy_keep();
    for (long long j = me.line; j < Bs.n; j += me.stride) {
        const size_t q = (size_t)j * V.Kp + me.k;
        const int b = __ldg(Bs.cs + j), e = __ldg(Bs.cs + j + 1);
        const double cn = __ldg(Bs.col_norm + j), cj = __ldg(Bs.c + j);
        Pack<double> x = ld_pack(V.x + q), xa = ld_pack(V.xa + q);
        const Pack<double> lo = ld_pack(V.lo + q), hi = ld_pack(V.hi + q);
        Pack<double> xb = pack_dot<AHEAD>(b, e, Bs.ri, Bs.cv, V.y + me.k, V.Kp, pol);
#pragma unroll
        for (int w = 0; w < W; ++w) {
            const double g = __dadd_rn(cj, xb.v[w]);
            const double tau = __ddiv_rn(me.step[w], cn);
            const double xp = clampv(__dsub_rn(x.v[w], __dmul_rn(tau, g)), lo.v[w], hi.v[w]);
            const double av = __dadd_rn(xa.v[w], __ddiv_rn(__dsub_rn(xp, xa.v[w]), me.cnt[w]));
            xb.v[w] = __dsub_rn(__dmul_rn(2.0, xp), x.v[w]);  // a finished variant's is not read
            x.v[w] = me.live[w] ? xp : x.v[w];
            xa.v[w] = me.live[w] ? av : xa.v[w];
        }
        st_keep_pack(V.xb + q, xb, pol);
        st_pack(V.x + q, x);
        st_pack(V.xa + q, xa);
    }
}

// v = y + sigma (A x-bar); y+ = v - sigma clamp(v/sigma, b_lo, b_hi); average
// (pdlp.cpp:220-227).  With APPLY A x-bar is the kept one of a probe iteration.
template <bool APPLY>
__global__ void __launch_bounds__(kBlock, kVarDualBlocks) kv_dual(VarBase Bs, VarRefs V, int kk) {
    const DualLane me = DualLane::of<double>(V, kk);
    if (!__any_sync(0xffffffffu, me.live)) return;
    const unsigned long long pol = policy_keep();
    MC_VARIANT_LINES(i, Bs.m) {
        const size_t q = (size_t)i * V.Kp + me.k;
        const double rn = __ldg(Bs.row_norm + i), bl = __ldg(Bs.blo + i), bh = __ldg(Bs.bhi + i);
        const double y = ld_stream(V.y + q), ya = ld_stream(V.ya + q);  // padding and finished variants included
        const double ax = APPLY ? ld_stream(V.axb + q)
                                : split_dot(__ldg(Bs.rs + i), __ldg(Bs.rs + i + 1), Bs.ci, Bs.rv, V.xb, V.Kp, me.k,
                                            me.need, pol);
        if (!me.live) continue;
        const double sigma = __ddiv_rn(me.sg, rn);
        const double v = __dadd_rn(y, __dmul_rn(sigma, ax));
        const double yn = __dsub_rn(v, __dmul_rn(sigma, clampv(__ddiv_rn(v, sigma), bl, bh)));
        st_keep(V.y + q, yn, pol);
        st_stream(V.ya + q, __dadd_rn(ya, __ddiv_rn(__dsub_rn(yn, ya), me.cnt)));
    }
}

// kv_dual for packs; with APPLY the dual update of a probe iteration, from the kept A x-bar
template <bool APPLY>
__global__ void __launch_bounds__(kBlock) kv_dual_wide(VarBase Bs, VarRefs V, int lg, int kk) {
    const VarPack<double> me(V, lg, kk, true);
    if (!me.any) return;
    constexpr int W = Pack<double>::W;
    const unsigned long long pol = policy_keep();
    for (long long i = me.line; i < Bs.m; i += me.stride) {
        const size_t q = (size_t)i * V.Kp + me.k;
        const int b = __ldg(Bs.rs + i), e = __ldg(Bs.rs + i + 1);
        const double rn = __ldg(Bs.row_norm + i), bl = __ldg(Bs.blo + i), bh = __ldg(Bs.bhi + i);
        Pack<double> y = ld_pack(V.y + q), ya = ld_pack(V.ya + q);
        const Pack<double> ax =
            APPLY ? ld_pack(V.axb + q) : pack_dot<true>(b, e, Bs.ci, Bs.rv, V.xb + me.k, V.Kp, pol);
#pragma unroll
        for (int w = 0; w < W; ++w) {
            const double sigma = __ddiv_rn(me.step[w], rn);
            const double v = __dadd_rn(y.v[w], __dmul_rn(sigma, ax.v[w]));
            const double yn = __dsub_rn(v, __dmul_rn(sigma, clampv(__ddiv_rn(v, sigma), bl, bh)));
            const double av = __dadd_rn(ya.v[w], __ddiv_rn(__dsub_rn(yn, ya.v[w]), me.cnt[w]));
            y.v[w] = me.live[w] ? yn : y.v[w];
            ya.v[w] = me.live[w] ? av : ya.v[w];
        }
        st_keep_pack(V.y + q, y, pol);
        st_pack(V.ya + q, ya);
    }
}

// --------------------------------------------------------------- residuals
// compute_unscaled_residuals (pdlp.cpp:62-135) of every variant's averages,
// with the Farkas test terms (RayTerms).
__global__ void __launch_bounds__(kBlock) kv_residual_rows(VarBase Bs, VarRefs V, Original O) {
    __shared__ double sm[kVarWarps][33];
    MC_VARIANT_LANE(V, k, live);
    const unsigned long long pol = policy_keep();
    RowTerms acc;
    RayTerms ray;
    MC_VARIANT_LINES(i, Bs.m) {
        const double s = variant_dot(Bs.rs, Bs.ci, Bs.rv, V.xa, V.Kp, i, k, live, pol);
        if (live) {
            const size_t q = (size_t)i * V.Kp + k;
            const double yv = V.ya[q];
            acc.add(O, (int)i, s, yv);
            const double d = RayTerms::candidate(O, (int)i, yv, V.y_prev + q);
            V.dray[q] = d;
            ray.add_row(O, (int)i, d);
        }
    }
    const double vmax = lanes_reduce(acc.vmax, sm, OpMax());
    const double dsum = lanes_reduce(acc.dsum, sm, OpSum());
    const double bad = lanes_reduce(acc.bad, sm, OpSum());
    const double ru = lanes_reduce(ray.u, sm, OpSum());
    const double rsc = lanes_reduce(ray.rscale, sm, OpSum());
    const double rinf = lanes_reduce(ray.rinf, sm, OpSum());
    if ((threadIdx.x >> 5) == 0 && k < V.K) {
        var_partial(V, SLOT_ROW_MAX, k)[blockIdx.x] = vmax;
        var_partial(V, SLOT_ROW_DOBJ, k)[blockIdx.x] = dsum;
        var_partial(V, SLOT_NAN, k)[blockIdx.x] = bad;
        var_partial(V, SLOT_RAY_U, k)[blockIdx.x] = ru;
        var_partial(V, SLOT_RAY_RSCALE, k)[blockIdx.x] = rsc;
        var_partial(V, SLOT_RAY_RINF, k)[blockIdx.x] = rinf;
    }
}

__global__ void __launch_bounds__(kBlock) kv_residual_cols(VarBase Bs, VarRefs V, Original O) {
    __shared__ double sm[kVarWarps][33];
    MC_VARIANT_LANE(V, k, live);
    const unsigned long long pol = policy_keep();
    ColTerms acc;
    RayTerms ray;
    MC_VARIANT_LINES(j, Bs.n) {
        const int b = __ldg(Bs.cs + j), e = __ldg(Bs.cs + j + 1);
        double s = 0.0, sd = 0.0, sa = 0.0;
        if (live) {
            for (int p = b; p < e; ++p) {
                const double a = __ldg(Bs.cv + p);
                const size_t qi = (size_t)__ldg(Bs.ri + p) * V.Kp + k;
                const double dv = V.dray[qi];
                s = fma(a, ld_keep(V.ya + qi, pol), s);
                sd = fma(a, dv, sd);
                sa = fma(fabs(a), fabs(dv), sa);
            }
            const size_t q = (size_t)j * V.Kp + k;
            acc.add_b(O, (int)j, s, V.xa[q], V.olo[q], V.ohi[q]);
            ray.add_col_b(O, (int)j, sd, sa, V.olo[q], V.ohi[q]);
        }
    }
    const double vmax = lanes_reduce(acc.vmax, sm, OpMax());
    const double dres = lanes_reduce(acc.dres, sm, OpSum());
    const double pobj = lanes_reduce(acc.pobj, sm, OpSum());
    const double dobj = lanes_reduce(acc.dobj, sm, OpSum());
    const double bad = lanes_reduce(acc.bad, sm, OpSum());
    const double rl = lanes_reduce(ray.l, sm, OpSum());
    const double rcs = lanes_reduce(ray.cscale, sm, OpSum());
    const double rci = lanes_reduce(ray.cinf, sm, OpSum());
    if ((threadIdx.x >> 5) == 0 && k < V.K) {
        var_partial(V, SLOT_COL_MAX, k)[blockIdx.x] = vmax;
        var_partial(V, SLOT_COL_DRES, k)[blockIdx.x] = dres;
        var_partial(V, SLOT_COL_POBJ, k)[blockIdx.x] = pobj;
        var_partial(V, SLOT_COL_DOBJ, k)[blockIdx.x] = dobj;
        var_partial(V, SLOT_B, k)[blockIdx.x] = bad;
        var_partial(V, SLOT_RAY_L, k)[blockIdx.x] = rl;
        var_partial(V, SLOT_RAY_CSCALE, k)[blockIdx.x] = rcs;
        var_partial(V, SLOT_RAY_CINF, k)[blockIdx.x] = rci;
    }
}

// One block per variant: KKT scalars, termination (optimal, or infeasible by
// the Farkas test), restart and primal weight (pdlp.cpp:229-261).
__global__ void kv_finalize(VarRefs V, double offset, long long span, int final_pass, Controls ctl) {
    __shared__ double scratch[32];
    const int k = blockIdx.x;
    DevState* st = V.st + k;
    if (st->done) return;
    const int nb = V.nb;
    const double row_max = reduce_partials(var_partial(V, SLOT_ROW_MAX, k), nb, scratch, OpMax());
    const double row_dobj = reduce_partials(var_partial(V, SLOT_ROW_DOBJ, k), nb, scratch, OpSum());
    const double bad_r = reduce_partials(var_partial(V, SLOT_NAN, k), nb, scratch, OpSum());
    const double col_max = reduce_partials(var_partial(V, SLOT_COL_MAX, k), nb, scratch, OpMax());
    const double col_dres = reduce_partials(var_partial(V, SLOT_COL_DRES, k), nb, scratch, OpSum());
    const double col_pobj = reduce_partials(var_partial(V, SLOT_COL_POBJ, k), nb, scratch, OpSum());
    const double col_dobj = reduce_partials(var_partial(V, SLOT_COL_DOBJ, k), nb, scratch, OpSum());
    const double bad_c = reduce_partials(var_partial(V, SLOT_B, k), nb, scratch, OpSum());
    const double ray_l = reduce_partials(var_partial(V, SLOT_RAY_L, k), nb, scratch, OpSum());
    const double ray_cs = reduce_partials(var_partial(V, SLOT_RAY_CSCALE, k), nb, scratch, OpSum());
    const double ray_ci = reduce_partials(var_partial(V, SLOT_RAY_CINF, k), nb, scratch, OpSum());
    const double ray_rs = reduce_partials(var_partial(V, SLOT_RAY_RSCALE, k), nb, scratch, OpSum());
    const double ray_ri = reduce_partials(var_partial(V, SLOT_RAY_RINF, k), nb, scratch, OpSum());
    const double ray_u = reduce_partials(var_partial(V, SLOT_RAY_U, k), nb, scratch, OpSum());
    if (threadIdx.x != 0) return;
    const double primal = maxv(row_max, col_max);
    const double dual = sqrt(col_dres) / st->c_scale;
    const double pobj = offset + col_pobj;
    const double dobj = (offset + row_dobj) + col_dobj;
    const double gap = fabs(pobj - dobj) / (1.0 + fabs(pobj) + fabs(dobj));
    const double score = maxv(maxv(primal, dual), gap);
    const double margin = ray_l - ray_u;
    const bool farkas = ray_ci == 0.0 && ray_ri == 0.0 && margin > 0.0 && margin > 1e-9 * (ray_cs + ray_rs);
    st->primal_infeas = primal;
    st->dual_infeas = dual;
    st->gap = gap;
    st->objective = pobj;
    st->dual_objective = dobj;
    st->score = score;
    st->restart_pending = 0;
    const long long isr = st->iters_since_restart + span;
    if (bad_r + bad_c > 0.0 || !isfinite(score)) {
        st->nonfinite = 1;
        st->done = 1;
        st->status = 3;
    } else if (!final_pass && primal <= ctl.primal_tol && dual <= ctl.dual_tol && gap <= ctl.gap_tol) {
        st->done = 1;
        st->status = 0;
    } else if (farkas) {
        st->done = 1;
        st->status = 2;
        st->cert = MC_CERT_DUAL_RAY;
    } else if (!final_pass) {
        const bool do_restart =
            ctl.strategy == 2 ||
            (ctl.strategy == 1 && (score <= ctl.restart_reduction * st->last_restart_score ||
                                   (isr >= 5 * ctl.restart_every && score < st->last_restart_score)));
        if (do_restart) {
            if (ctl.adaptive_weight && primal > 1e-12 && dual > 1e-12) {
                const double ratio = clampv(sqrt(primal / dual), 0.05, 20.0);
                st->omega = clampv(st->omega * pow(ratio, ctl.weight_smoothing), 1e-6, 1e6);
            }
            st->restart_pending = 1;
            st->avg_count = 0;
            st->iters_since_restart = 0;
            st->last_restart_score = score;
            st->restarts += 1;
        } else {
            st->avg_count += span;
            st->iters_since_restart = isr;
        }
    }
    st->iter += span;
    if (!final_pass) st->checks += 1;
}

// restart to the average (pdlp.cpp:257-258) of the variants that restart
__global__ void __launch_bounds__(kBlock) kv_restart_copy(VarBase Bs, VarRefs V) {
    const int k = blockIdx.y * 32 + (threadIdx.x & 31);
    if (k >= V.K) return;
    const DevState& s = V.st[k];
    if (!s.restart_pending || s.done) return;
    MC_VARIANT_LINES(l, (long long)Bs.n + Bs.m) {
        if (l < Bs.n) {
            const size_t q = (size_t)l * V.Kp + k;
            V.x[q] = V.xa[q];
        } else {
            const size_t q = (size_t)(l - Bs.n) * V.Kp + k;
            V.y[q] = V.ya[q];
        }
    }
}

// the poll flag: done once every variant is
__global__ void kv_poll(VarRefs V) {
    __shared__ int running;
    if (threadIdx.x == 0) running = 0;
    __syncthreads();
    int mine = 0;
    for (int k = threadIdx.x; k < V.K; k += blockDim.x) mine += V.st[k].done ? 0 : 1;
    if (mine) atomicAdd(&running, mine);
    __syncthreads();
    if (threadIdx.x == 0) {
        V.global->done = running == 0 ? 1 : 0;
        V.global->active_tiles[0] = running;
    }
}

// ------------------------------------------------------------------ setup
// Variant bounds (given [K][n], original units) into the variant-minor
// arrays: scaled and sentinel forms, the crossed-bound certificate, and the
// start x = proj(given start or 0) (pdlp.cpp:186-191).  Padding lanes get
// zeros, so that gathers over them read finite values.
__global__ void __launch_bounds__(kBlock) kv_setup_cols(VarBase Bs, VarRefs V, const int* __restrict__ perm,
                                                        const double* __restrict__ lo_in,
                                                        const double* __restrict__ hi_in,
                                                        const double* __restrict__ warm_x,
                                                        const int* __restrict__ has_warm_x,
                                                        const double* __restrict__ col_scale) {
    const int k = blockIdx.y * 32 + (threadIdx.x & 31);
    const bool real = k < V.K;
    MC_VARIANT_LINES(j, Bs.n) {
        const size_t q = (size_t)j * V.Kp + k;
        if (!real) {
            V.lo[q] = V.hi[q] = V.olo[q] = V.ohi[q] = 0.0;
            V.x[q] = V.xa[q] = V.xb[q] = 0.0;
            V.xdx[2 * q] = V.xdx[2 * q + 1] = 0.0;
            continue;
        }
        const int b = perm[k];  // the caller's variant in slot k
        const size_t g = (size_t)b * Bs.n + j;
        const double s = col_scale[j];
        const double inv = 1.0 / s;
        const double l0 = lo_in[g], h0 = hi_in[g];
        const double ls = isfinite(l0) ? __dmul_rn(l0, inv) : l0;
        const double hs = isfinite(h0) ? __dmul_rn(h0, inv) : h0;
        const double lsent = isinf(ls) ? -kBig : ls;
        const double hsent = isinf(hs) ? kBig : hs;
        V.lo[q] = lsent;
        V.hi[q] = hsent;
        V.olo[q] = isinf(l0) ? -kBig : l0;
        V.ohi[q] = isinf(h0) ? kBig : h0;
        if (l0 > h0) {
            atomicOr(V.flags + k, 1);
            atomicMin(V.cert_idx + k, (int)j);
        }
        const double start = (has_warm_x && has_warm_x[b]) ? __dmul_rn(warm_x[g], inv) : 0.0;
        const double x0 = clampv(start, lsent, hsent);
        V.x[q] = x0;
        V.xa[q] = x0;
        V.xb[q] = x0;
        V.xdx[2 * q] = x0;
        V.xdx[2 * q + 1] = 0.0;
    }
}

// Row-activity certificate per variant (the packed batch's kb_setup_rows
// test on the variant's box) and the dual start.
__global__ void __launch_bounds__(kBlock) kv_setup_rows(VarBase Bs, VarRefs V, const int* __restrict__ perm,
                                                        const double* __restrict__ rlo_in,
                                                        const double* __restrict__ rhi_in,
                                                        const double* __restrict__ row_scale,
                                                        const double* __restrict__ col_scale,
                                                        const double* __restrict__ warm_y,
                                                        const int* __restrict__ has_warm_y) {
    const int k = blockIdx.y * 32 + (threadIdx.x & 31);
    const bool real = k < V.K;
    MC_VARIANT_LINES(i, Bs.m) {
        const size_t q = (size_t)i * V.Kp + k;
        if (!real) {
            V.y[q] = V.ya[q] = V.axb[q] = V.y_prev[q] = V.dray[q] = 0.0;
            continue;
        }
        const double s = row_scale[i];
        const double l0 = rlo_in[i], h0 = rhi_in[i];
        double amin = 0.0, amax = 0.0, mag = 0.0;
        for (int p = Bs.rs[i]; p < Bs.rs[i + 1]; ++p) {
            const int j = Bs.ci[p];
            const double a = Bs.rv[p] / (s * col_scale[j]);
            const size_t qj = (size_t)j * V.Kp + k;
            const double lj = V.olo[qj], hj = V.ohi[qj];
            const double t1 = fabs(lj) >= 1e299 ? copysign(INFINITY, lj) * a : a * lj;
            const double t2 = fabs(hj) >= 1e299 ? copysign(INFINITY, hj) * a : a * hj;
            amin += (a > 0) ? t1 : t2;
            amax += (a > 0) ? t2 : t1;
            mag += fabs(a) * maxv(fabs(lj) < 1e299 ? fabs(lj) : 0.0, fabs(hj) < 1e299 ? fabs(hj) : 0.0);
        }
        const double slack =
            1e-9 * (1.0 + mag + maxv(isfinite(l0) ? fabs(l0) : 0.0, isfinite(h0) ? fabs(h0) : 0.0));
        if ((isfinite(l0) && amax < l0 - slack) || (isfinite(h0) && amin > h0 + slack)) {
            atomicOr(V.flags + k, 2);
            atomicMin(V.cert_idx + V.K + k, (int)i);
        }
        const int b = perm[k];
        const double y0 = (has_warm_y && has_warm_y[b]) ? __dmul_rn(warm_y[(size_t)b * Bs.m + i], 1.0 / s) : 0.0;
        V.y[q] = y0;
        V.ya[q] = y0;
        V.axb[q] = 0.0;
        V.y_prev[q] = y0;
        V.dray[q] = 0.0;
    }
}

// every variant starts from the base LP's scalars (pdlp.cpp:153-185): the
// norms, the initial primal weight and eta depend on A, c and the row bounds only
__global__ void kv_setup_state(VarRefs V, const DevState* __restrict__ base) {
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < V.K; k += gridDim.x * blockDim.x) {
        DevState s = *base;
        s.iter = s.avg_count = s.iters_since_restart = s.restarts = s.checks = 0;
        s.restart_pending = 0;
        s.nonfinite = 0;
        s.last_restart_score = 1e300;
        s.primal_infeas = s.dual_infeas = s.gap = 1e300;
        if (V.flags[k]) {
            s.done = 1;
            s.status = 2;
            s.cert = (V.flags[k] & 1) ? MC_CERT_CROSSED_BOUNDS : MC_CERT_ROW_ACTIVITY;
        } else {
            s.done = 0;
            s.status = 1;
            s.cert = MC_CERT_NONE;
        }
        V.st[k] = s;
    }
}

// unscaled averages of every variant into [K][n] and [K][m] staging
__global__ void __launch_bounds__(kBlock) kv_unscale_out(VarBase Bs, VarRefs V, const double* __restrict__ col_scale,
                                                         const double* __restrict__ row_scale, double* __restrict__ xo,
                                                         double* __restrict__ yo) {
    const int k = blockIdx.y * 32 + (threadIdx.x & 31);
    if (k >= V.K) return;
    // a variant proven infeasible by a dual ray returns the ray as its dual
    const bool ray = V.st[k].status == 2 && V.st[k].cert == MC_CERT_DUAL_RAY;
    const double* yv = ray ? V.dray : V.ya;
    MC_VARIANT_LINES(l, (long long)Bs.n + Bs.m) {
        if (l < Bs.n) {
            xo[(size_t)k * Bs.n + l] = __dmul_rn(V.xa[(size_t)l * V.Kp + k], col_scale[l]);
        } else {
            const long long i = l - Bs.n;
            yo[(size_t)k * Bs.m + i] = __dmul_rn(yv[(size_t)i * V.Kp + k], row_scale[i]);
        }
    }
}

// ------------------------------------------------------------ the engine
struct EngineVariants {
    VarBase Bs;
    VarRefs V;
    Original O;
    dim3 grid;
    WideGrid cols, wide;  // packs of columns, of rows
    dim3 rows;
    bool rows_wide, long_cols;
    int shape_class(const DevState&) const { return 0; }
    void use_class(int) const {}

    int iteration(Ctx& ctx, int k, bool step, const Controls& ctl) const {
        cudaStream_t s = ctx.stream;
        ctx.begin_launch(MC_KERNEL_PRIMAL);
        if (step) kv_primal_step<<<grid, kBlock, 0, s>>>(Bs, V, k);
        else if (long_cols) kv_primal_wide<true><<<cols.grid, kBlock, 0, s>>>(Bs, V, cols.lg, k);
        else kv_primal_wide<false><<<cols.grid, kBlock, 0, s>>>(Bs, V, cols.lg, k);
        ctx.end_launch();
        if (step) {
            ctx.begin_launch(MC_KERNEL_DUAL_STEP);
            kv_dual_probe<<<grid, kBlock, 0, s>>>(Bs, V);
            ctx.end_launch();
            ctx.begin_launch(MC_KERNEL_OTHER);
            kv_step_size<<<V.K, 256, 0, s>>>(V, ctl);
            ctx.end_launch();
            ctx.begin_launch(MC_KERNEL_DUAL_STEP);
            if (rows_wide) kv_dual_wide<true><<<wide.grid, kBlock, 0, s>>>(Bs, V, wide.lg, k);
            else kv_dual<true><<<rows, kBlock, 0, s>>>(Bs, V, k);
            ctx.end_launch();
        } else {
            ctx.begin_launch(MC_KERNEL_DUAL);
            if (rows_wide) kv_dual_wide<false><<<wide.grid, kBlock, 0, s>>>(Bs, V, wide.lg, k);
            else kv_dual<false><<<rows, kBlock, 0, s>>>(Bs, V, k);
            ctx.end_launch();
        }
        return ctx.launch_check("variant iteration");
    }

    int check(Ctx& ctx, long long span, int final_pass, const Controls& ctl, const TraceBuf&) const {
        cudaStream_t s = ctx.stream;
        ctx.begin_launch(MC_KERNEL_RESIDUAL);
        kv_residual_rows<<<grid, kBlock, 0, s>>>(Bs, V, O);
        ctx.end_launch();
        ctx.begin_launch(MC_KERNEL_RESIDUAL);
        kv_residual_cols<<<grid, kBlock, 0, s>>>(Bs, V, O);
        ctx.end_launch();
        ctx.begin_launch(MC_KERNEL_RESIDUAL);
        kv_finalize<<<V.K, 256, 0, s>>>(V, O.offset, span, final_pass, ctl);
        ctx.end_launch();
        if (!final_pass) {
            ctx.begin_launch(MC_KERNEL_OTHER);
            kv_restart_copy<<<grid, kBlock, 0, s>>>(Bs, V);
            ctx.end_launch();
        }
        ctx.begin_launch(MC_KERNEL_OTHER);
        kv_poll<<<1, 1024, 0, s>>>(V);
        ctx.end_launch();
        return ctx.launch_check("variant check");
    }
};

// ----------------------------------------------------- the FP32 form
// The mixed-precision form of mixed.cuh per variant: each variant's iterate
// is an FP64 base plus an FP32 correction, x = xh + dx, y = yh + dy; FP32 PDHG
// runs on the correction LP (FP32 matrix, FP32 variant-minor vectors); the
// residual pass, gap, restart test and primal weight are FP64 on xh + dx_avg
// with the FP64 matrix; at every restart a variant's base moves to its average
// and its correction LP is rebuilt from the residual pass's FP64 products.
struct VarMixed {
    const int* cs;          // the base's CSC / CSR structure (shared with the FP64 data)
    const int* ri;
    const float* cv;        // FP32 matrix values
    const int* rs;
    const int* ci;
    const float* rv;
    const float* col_norm;  // FP32 norms
    const float* row_norm;
    const double* c64;      // scaled c, FP64
    const double* blo64;    // scaled row bounds, sentinel form, FP64
    const double* bhi64;
    double* xh;             // [n Kp] FP64 bases
    double* yh;             // [m Kp]
    double* axf;            // [m Kp] A (xh + dx_avg) from the residual pass
    double* atyf;           // [n Kp] A^T (yh + dy_avg)
    float* x;               // [n Kp] dx
    float* xb;              // [n Kp] dx-bar
    float* xa;              // [n Kp] dx average
    float* xdx;             // [2 n Kp] (dx-bar, d dx) pairs
    float* g;               // [n Kp] float(c + A^T yh)
    float* lo;              // [n Kp] float(lo - xh), +-inf when unbounded
    float* hi;
    float* y;               // [m Kp] dy
    float* ya;              // [m Kp] dy average
    float* axb;             // [m Kp] A dx-bar of a step-size iteration
    float* yb;              // [m Kp] float(yh)
    float* rlo;             // [m Kp] float(A xh - b_lo), +inf when unbounded
    float* rhi;             // [m Kp] float(A xh - b_hi), -inf when unbounded
};

__device__ __forceinline__ float variant_dot_f(const int* __restrict__ start, const int* __restrict__ idx,
                                               const float* __restrict__ val, const float* __restrict__ v, int Kp,
                                               long long l, int k, bool live, unsigned long long pol) {
    const int b = __ldg(start + l), e = __ldg(start + l + 1);
    float s0 = 0.f, s1 = 0.f, s2 = 0.f, s3 = 0.f;
    int p = b;
    for (; p + 4 <= e; p += 4) {
        const int i0 = __ldg(idx + p), i1 = __ldg(idx + p + 1), i2 = __ldg(idx + p + 2), i3 = __ldg(idx + p + 3);
        const float a0 = __ldg(val + p), a1 = __ldg(val + p + 1), a2 = __ldg(val + p + 2), a3 = __ldg(val + p + 3);
        if (live) {
            s0 = fmaf(a0, ld_keep(v + (size_t)i0 * Kp + k, pol), s0);
            s1 = fmaf(a1, ld_keep(v + (size_t)i1 * Kp + k, pol), s1);
            s2 = fmaf(a2, ld_keep(v + (size_t)i2 * Kp + k, pol), s2);
            s3 = fmaf(a3, ld_keep(v + (size_t)i3 * Kp + k, pol), s3);
        }
    }
    for (; p < e; ++p)
        if (live) s0 = fmaf(__ldg(val + p), ld_keep(v + (size_t)__ldg(idx + p) * Kp + k, pol), s0);
    return (s0 + s1) + (s2 + s3);
}

__global__ void __launch_bounds__(kBlock) kvm_primal_step(int n, VarRefs V, VarMixed M, int kk) {
    __shared__ double sm[kVarWarps][33];
    MC_VARIANT_LANE(V, k, live);
    float step = 0.f, cnt = 1.f;
    if (live) {
        const DevState& s = V.st[k];
        step = (float)(s.eta / s.omega);
        cnt = (float)(double)(s.avg_count + kk + 1);
    }
    const unsigned long long pol = policy_keep();
    double acc = 0.0;
    MC_VARIANT_LINES(j, n) {
        const float aty = variant_dot_f(M.cs, M.ri, M.cv, M.y, V.Kp, j, k, live, pol);
        if (live) {
            const size_t q = (size_t)j * V.Kp + k;
            const float cn = __ldg(M.col_norm + j);
            const float g = __fadd_rn(ld_stream(M.g + q), aty);
            const float tau = __fdiv_rn(step, cn);
            const float xo = ld_stream(M.x + q);
            const float xp = clampv(__fsub_rn(xo, __fmul_rn(tau, g)), ld_stream(M.lo + q), ld_stream(M.hi + q));
            const float d = __fsub_rn(xp, xo);
            const float xbar = __fsub_rn(__fmul_rn(2.f, xp), xo);
            st_keep2(M.xdx + 2 * q, xbar, d, pol);
            acc += __dmul_rn(__dmul_rn((double)cn, (double)d), (double)d);
            st_stream(M.x + q, xp);
            const float xa = ld_stream(M.xa + q);
            st_stream(M.xa + q, __fadd_rn(xa, __fdiv_rn(__fsub_rn(xp, xa), cnt)));
        }
    }
    acc = lanes_reduce(acc, sm, OpSum());
    if ((threadIdx.x >> 5) == 0 && k < V.K) var_partial(V, SLOT_DX, k)[blockIdx.x] = acc;
}

__global__ void __launch_bounds__(kBlock) kvm_dual_probe(int m, VarRefs V, VarMixed M) {
    __shared__ double sm[kVarWarps][33];
    MC_VARIANT_LANE(V, k, live);
    const unsigned long long pol = policy_keep();
    double acc = 0.0;
    MC_VARIANT_LINES(i, m) {
        const int b = __ldg(M.rs + i), e = __ldg(M.rs + i + 1);
        float sv0 = 0.f, sw0 = 0.f, sv1 = 0.f, sw1 = 0.f;
        int p = b;
        for (; p + 2 <= e; p += 2) {
            const int j0 = __ldg(M.ci + p), j1 = __ldg(M.ci + p + 1);
            const float a0 = __ldg(M.rv + p), a1 = __ldg(M.rv + p + 1);
            if (live) {
                float v0, w0, v1, w1;
                ld_keep2(M.xdx + 2 * ((size_t)j0 * V.Kp + k), pol, v0, w0);
                ld_keep2(M.xdx + 2 * ((size_t)j1 * V.Kp + k), pol, v1, w1);
                sv0 = fmaf(a0, v0, sv0);
                sw0 = fmaf(a0, w0, sw0);
                sv1 = fmaf(a1, v1, sv1);
                sw1 = fmaf(a1, w1, sw1);
            }
        }
        if (p < e && live) {
            float v0, w0;
            ld_keep2(M.xdx + 2 * ((size_t)__ldg(M.ci + p) * V.Kp + k), pol, v0, w0);
            const float a0 = __ldg(M.rv + p);
            sv0 = fmaf(a0, v0, sv0);
            sw0 = fmaf(a0, w0, sw0);
        }
        if (live) {
            M.axb[(size_t)i * V.Kp + k] = sv0 + sv1;
            const double adx = (double)(sw0 + sw1);
            acc += __ddiv_rn(__dmul_rn(adx, adx), (double)__ldg(M.row_norm + i));
        }
    }
    acc = lanes_reduce(acc, sm, OpSum());
    if ((threadIdx.x >> 5) == 0 && k < V.K) var_partial(V, SLOT_ADX, k)[blockIdx.x] = acc;
}

// The FP32 divisions of a pack without branches, so that those of its four
// variants overlap (primal 18.9 -> 15.6 us at 128 variants): a / b =
// float(a * recip_wide(b)), correctly rounded.  For floats a, b and a rounding
// boundary c (25 bits), |a - c b| is 0 or at least one unit of its last place,
// so a / b differs from c by 0 or at least 2^-49 of itself, eight times the
// error of the FP64 product; and FP64 has room for every float quotient.  (A
// tie, |a - c b| = 0, exists only among quotients below 2^-126, where the last
// bit may differ from the divide's.)  The reciprocal starts from the hardware's
// approximation (about 2^-23) and takes one third-order step (e -> e^3); a b
// whose approximation is no good (zero, tiny, huge, not finite) is divided.
__device__ __forceinline__ double recip_wide(float b) {
    const double y = (double)__fdividef(1.f, b), e = fma(-(double)b, y, 1.0);
    if (!(fabs(e) < 1e-6)) return __ddiv_rn(1.0, (double)b);
    return fma(y, fma(e, e, e), y);
}
__device__ __forceinline__ float div_wide(float a, double y) { return (float)__dmul_rn((double)a, y); }

// the primal step of an iteration without a probe, on the correction
__global__ void __launch_bounds__(kBlock) kvm_primal_wide(int n, VarRefs V, VarMixed M, int lg, int kk) {
    const VarPack<float> me(V, lg, kk, false);
    if (!me.any) return;
    constexpr int W = Pack<float>::W;
    double rcnt[W];
#pragma unroll
    for (int w = 0; w < W; ++w) rcnt[w] = recip_wide(me.cnt[w]);
    const unsigned long long pol = policy_keep();
    for (long long j = me.line; j < n; j += me.stride) {
        const size_t q = (size_t)j * V.Kp + me.k;
        const int b = __ldg(M.cs + j), e = __ldg(M.cs + j + 1);
        const float cn = __ldg(M.col_norm + j);
        Pack<float> x = ld_pack(M.x + q), xa = ld_pack(M.xa + q);
        const Pack<float> g = ld_pack(M.g + q), lo = ld_pack(M.lo + q), hi = ld_pack(M.hi + q);
        const double rcn = recip_wide(cn);
        Pack<float> xb = pack_dot<false>(b, e, M.ri, M.cv, M.y + me.k, V.Kp, pol);
#pragma unroll
        for (int w = 0; w < W; ++w) {
            const float gw = __fadd_rn(g.v[w], xb.v[w]);
            const float tau = div_wide(me.step[w], rcn);
            const float xp = clampv(__fsub_rn(x.v[w], __fmul_rn(tau, gw)), lo.v[w], hi.v[w]);
            const float av = __fadd_rn(xa.v[w], div_wide(__fsub_rn(xp, xa.v[w]), rcnt[w]));
            xb.v[w] = __fsub_rn(__fmul_rn(2.f, xp), x.v[w]);  // a finished variant's is not read
            x.v[w] = me.live[w] ? xp : x.v[w];
            xa.v[w] = me.live[w] ? av : xa.v[w];
        }
        st_keep_pack(M.xb + q, xb, pol);
        st_pack(M.x + q, x);
        st_pack(M.xa + q, xa);
    }
}

// the dual step on the correction (dual_update_mx of mixed.cuh, per variant)
template <bool APPLY>
__global__ void __launch_bounds__(kBlock, kVarDualBlocks) kvm_dual(int m, VarRefs V, VarMixed M, int kk) {
    const DualLane me = DualLane::of<float>(V, kk);
    if (!__any_sync(0xffffffffu, me.live)) return;
    const float sg = (float)me.sg, cnt = (float)me.cnt;
    const unsigned long long pol = policy_keep();
    MC_VARIANT_LINES(i, m) {
        const size_t q = (size_t)i * V.Kp + me.k;
        const float rn = __ldg(M.row_norm + i);
        const float dy = ld_stream(M.y + q), dya = ld_stream(M.ya + q), yb = ld_stream(M.yb + q);
        const float rl = ld_stream(M.rlo + q), rh = ld_stream(M.rhi + q);
        const float ax = APPLY ? ld_stream(M.axb + q)
                               : split_dot(__ldg(M.rs + i), __ldg(M.rs + i + 1), M.ci, M.rv, M.xb, V.Kp, me.k,
                                           me.need, pol);
        if (!me.live) continue;
        const float sigma = __fdiv_rn(sg, rn);
        const float base = __fdiv_rn(__fadd_rn(yb, dy), sigma);
        const float tl = __fadd_rn(rl, ax), th = __fadd_rn(rh, ax);
        const bool below = __fadd_rn(base, tl) < 0.f, above = __fadd_rn(base, th) > 0.f;
        const float moved = __fadd_rn(dy, __fmul_rn(sigma, below ? tl : th));
        const float dyn = (below || above) ? moved : -yb;
        st_keep(M.y + q, dyn, pol);
        st_stream(M.ya + q, __fadd_rn(dya, __fdiv_rn(__fsub_rn(dyn, dya), cnt)));
    }
}

// kvm_dual for packs; with APPLY the dual update of a probe iteration, from the kept A dx-bar
template <bool APPLY>
__global__ void __launch_bounds__(kBlock) kvm_dual_wide(int m, VarRefs V, VarMixed M, int lg, int kk) {
    const VarPack<float> me(V, lg, kk, true);
    if (!me.any) return;
    constexpr int W = Pack<float>::W;
    double rcnt[W];
#pragma unroll
    for (int w = 0; w < W; ++w) rcnt[w] = recip_wide(me.cnt[w]);
    const unsigned long long pol = policy_keep();
    for (long long i = me.line; i < m; i += me.stride) {
        const size_t q = (size_t)i * V.Kp + me.k;
        const int b = __ldg(M.rs + i), e = __ldg(M.rs + i + 1);
        const float rn = __ldg(M.row_norm + i);
        Pack<float> y = ld_pack(M.y + q), ya = ld_pack(M.ya + q);
        const Pack<float> yb = ld_pack(M.yb + q), rl = ld_pack(M.rlo + q), rh = ld_pack(M.rhi + q);
        const double rrn = recip_wide(rn);
        const Pack<float> ax =
            APPLY ? ld_pack(M.axb + q) : pack_dot<true>(b, e, M.ci, M.rv, M.xb + me.k, V.Kp, pol);
#pragma unroll
        for (int w = 0; w < W; ++w) {
            // the dual step on the correction (dual_update_mx of mixed.cuh)
            const float dy = y.v[w];
            const float sigma = div_wide(me.step[w], rrn);
            const float base = div_wide(__fadd_rn(yb.v[w], dy), recip_wide(sigma));
            const float tl = __fadd_rn(rl.v[w], ax.v[w]), th = __fadd_rn(rh.v[w], ax.v[w]);
            const bool below = __fadd_rn(base, tl) < 0.f, above = __fadd_rn(base, th) > 0.f;
            const float moved = __fadd_rn(dy, __fmul_rn(sigma, below ? tl : th));
            const float dyn = (below || above) ? moved : -yb.v[w];
            const float av = __fadd_rn(ya.v[w], div_wide(__fsub_rn(dyn, ya.v[w]), rcnt[w]));
            y.v[w] = me.live[w] ? dyn : dy;
            ya.v[w] = me.live[w] ? av : ya.v[w];
        }
        st_keep_pack(M.y + q, y, pol);
        st_pack(M.ya + q, ya);
    }
}

// FP64 residual pass on xh + dx_avg, yh + dy_avg (FP64 matrix of the base),
// keeping A x and A^T y of that point for the recentring; Farkas terms.
__global__ void __launch_bounds__(kBlock) kvm_residual_rows(VarBase Bs, VarRefs V, VarMixed M, Original O) {
    __shared__ double sm[kVarWarps][33];
    MC_VARIANT_LANE(V, k, live);
    RowTerms acc;
    RayTerms ray;
    MC_VARIANT_LINES(i, Bs.m) {
        double s = 0.0;
        if (live) {
            for (int p = __ldg(Bs.rs + i); p < __ldg(Bs.rs + i + 1); ++p) {
                const size_t qj = (size_t)__ldg(Bs.ci + p) * V.Kp + k;
                s = fma(__ldg(Bs.rv + p), M.xh[qj] + (double)M.xa[qj], s);
            }
            const size_t q = (size_t)i * V.Kp + k;
            M.axf[q] = s;
            const double yv = M.yh[q] + (double)M.ya[q];
            acc.add(O, (int)i, s, yv);
            const double d = RayTerms::candidate(O, (int)i, yv, V.y_prev + q);
            V.dray[q] = d;
            ray.add_row(O, (int)i, d);
        }
    }
    const double vmax = lanes_reduce(acc.vmax, sm, OpMax());
    const double dsum = lanes_reduce(acc.dsum, sm, OpSum());
    const double bad = lanes_reduce(acc.bad, sm, OpSum());
    const double ru = lanes_reduce(ray.u, sm, OpSum());
    const double rsc = lanes_reduce(ray.rscale, sm, OpSum());
    const double rinf = lanes_reduce(ray.rinf, sm, OpSum());
    if ((threadIdx.x >> 5) == 0 && k < V.K) {
        var_partial(V, SLOT_ROW_MAX, k)[blockIdx.x] = vmax;
        var_partial(V, SLOT_ROW_DOBJ, k)[blockIdx.x] = dsum;
        var_partial(V, SLOT_NAN, k)[blockIdx.x] = bad;
        var_partial(V, SLOT_RAY_U, k)[blockIdx.x] = ru;
        var_partial(V, SLOT_RAY_RSCALE, k)[blockIdx.x] = rsc;
        var_partial(V, SLOT_RAY_RINF, k)[blockIdx.x] = rinf;
    }
}

__global__ void __launch_bounds__(kBlock) kvm_residual_cols(VarBase Bs, VarRefs V, VarMixed M, Original O) {
    __shared__ double sm[kVarWarps][33];
    MC_VARIANT_LANE(V, k, live);
    ColTerms acc;
    RayTerms ray;
    MC_VARIANT_LINES(j, Bs.n) {
        double s = 0.0, sd = 0.0, sa = 0.0;
        if (live) {
            for (int p = __ldg(Bs.cs + j); p < __ldg(Bs.cs + j + 1); ++p) {
                const double a = __ldg(Bs.cv + p);
                const size_t qi = (size_t)__ldg(Bs.ri + p) * V.Kp + k;
                const double dv = V.dray[qi];
                s = fma(a, M.yh[qi] + (double)M.ya[qi], s);
                sd = fma(a, dv, sd);
                sa = fma(fabs(a), fabs(dv), sa);
            }
            const size_t q = (size_t)j * V.Kp + k;
            M.atyf[q] = s;
            acc.add_b(O, (int)j, s, M.xh[q] + (double)M.xa[q], V.olo[q], V.ohi[q]);
            ray.add_col_b(O, (int)j, sd, sa, V.olo[q], V.ohi[q]);
        }
    }
    const double vmax = lanes_reduce(acc.vmax, sm, OpMax());
    const double dres = lanes_reduce(acc.dres, sm, OpSum());
    const double pobj = lanes_reduce(acc.pobj, sm, OpSum());
    const double dobj = lanes_reduce(acc.dobj, sm, OpSum());
    const double bad = lanes_reduce(acc.bad, sm, OpSum());
    const double rl = lanes_reduce(ray.l, sm, OpSum());
    const double rcs = lanes_reduce(ray.cscale, sm, OpSum());
    const double rci = lanes_reduce(ray.cinf, sm, OpSum());
    if ((threadIdx.x >> 5) == 0 && k < V.K) {
        var_partial(V, SLOT_COL_MAX, k)[blockIdx.x] = vmax;
        var_partial(V, SLOT_COL_DRES, k)[blockIdx.x] = dres;
        var_partial(V, SLOT_COL_POBJ, k)[blockIdx.x] = pobj;
        var_partial(V, SLOT_COL_DOBJ, k)[blockIdx.x] = dobj;
        var_partial(V, SLOT_B, k)[blockIdx.x] = bad;
        var_partial(V, SLOT_RAY_L, k)[blockIdx.x] = rl;
        var_partial(V, SLOT_RAY_CSCALE, k)[blockIdx.x] = rcs;
        var_partial(V, SLOT_RAY_CINF, k)[blockIdx.x] = rci;
    }
}

// Restart of a variant to its average: its base moves there and its
// correction LP is rebuilt from the residual pass's FP64 products
// (k_recenter_mx per variant).  `force` rebuilds every running variant.
__global__ void __launch_bounds__(kBlock) kvm_recenter(int m, int n, VarRefs V, VarMixed M, int force) {
    const int k = blockIdx.y * 32 + (threadIdx.x & 31);
    if (k >= V.K) return;
    const DevState& s = V.st[k];
    if (s.done || (!force && !s.restart_pending)) return;
    const float inf = __int_as_float(0x7f800000);
    MC_VARIANT_LINES(l, (long long)n + m) {
        if (l < n) {
            const size_t q = (size_t)l * V.Kp + k;
            const double xh = M.xh[q] + (double)M.xa[q];
            M.xh[q] = xh;
            M.x[q] = 0.f;
            M.xa[q] = 0.f;
            M.g[q] = (float)(M.c64[l] + M.atyf[q]);
            const double lo = V.lo[q], hi = V.hi[q];
            M.lo[q] = (lo <= -1e299) ? -inf : (float)(lo - xh);
            M.hi[q] = (hi >= 1e299) ? inf : (float)(hi - xh);
        } else {
            const long long i = l - n;
            const size_t q = (size_t)i * V.Kp + k;
            const double yh = M.yh[q] + (double)M.ya[q];
            M.yh[q] = yh;
            M.y[q] = 0.f;
            M.ya[q] = 0.f;
            M.yb[q] = (float)yh;
            const double ax = M.axf[q], lo = M.blo64[i], hi = M.bhi64[i];
            M.rlo[q] = (lo <= -1e299) ? inf : (float)(ax - lo);
            M.rhi[q] = (hi >= 1e299) ? -inf : (float)(ax - hi);
        }
    }
}

// unscaled outputs of the FP32 form: x = (xh + dx_avg) D_C, y = (yh + dy_avg) D_R
// (the ray for a variant proven infeasible by one)
__global__ void __launch_bounds__(kBlock) kvm_unscale_out(int m, int n, VarRefs V, VarMixed M,
                                                          const double* __restrict__ col_scale,
                                                          const double* __restrict__ row_scale,
                                                          double* __restrict__ xo, double* __restrict__ yo) {
    const int k = blockIdx.y * 32 + (threadIdx.x & 31);
    if (k >= V.K) return;
    const bool ray = V.st[k].status == 2 && V.st[k].cert == MC_CERT_DUAL_RAY;
    MC_VARIANT_LINES(l, (long long)n + m) {
        if (l < n) {
            const size_t q = (size_t)l * V.Kp + k;
            xo[(size_t)k * n + l] = __dmul_rn(M.xh[q] + (double)M.xa[q], col_scale[l]);
        } else {
            const long long i = l - n;
            const size_t q = (size_t)i * V.Kp + k;
            const double yv = ray ? V.dray[q] : M.yh[q] + (double)M.ya[q];
            yo[(size_t)k * m + i] = __dmul_rn(yv, row_scale[i]);
        }
    }
}

struct EngineVariantsMixed {
    VarBase Bs;
    VarRefs V;
    VarMixed M;
    Original O;
    dim3 grid;
    WideGrid cols, wide;  // packs of columns, of rows
    dim3 rows;
    bool rows_wide;
    int shape_class(const DevState&) const { return 0; }
    void use_class(int) const {}

    int iteration(Ctx& ctx, int k, bool step, const Controls& ctl) const {
        cudaStream_t s = ctx.stream;
        ctx.begin_launch(MC_KERNEL_PRIMAL);
        if (step) kvm_primal_step<<<grid, kBlock, 0, s>>>(Bs.n, V, M, k);
        else kvm_primal_wide<<<cols.grid, kBlock, 0, s>>>(Bs.n, V, M, cols.lg, k);
        ctx.end_launch();
        if (step) {
            ctx.begin_launch(MC_KERNEL_DUAL_STEP);
            kvm_dual_probe<<<grid, kBlock, 0, s>>>(Bs.m, V, M);
            ctx.end_launch();
            ctx.begin_launch(MC_KERNEL_OTHER);
            kv_step_size<<<V.K, 256, 0, s>>>(V, ctl);
            ctx.end_launch();
            ctx.begin_launch(MC_KERNEL_DUAL_STEP);
            if (rows_wide) kvm_dual_wide<true><<<wide.grid, kBlock, 0, s>>>(Bs.m, V, M, wide.lg, k);
            else kvm_dual<true><<<rows, kBlock, 0, s>>>(Bs.m, V, M, k);
            ctx.end_launch();
        } else {
            ctx.begin_launch(MC_KERNEL_DUAL);
            if (rows_wide) kvm_dual_wide<false><<<wide.grid, kBlock, 0, s>>>(Bs.m, V, M, wide.lg, k);
            else kvm_dual<false><<<rows, kBlock, 0, s>>>(Bs.m, V, M, k);
            ctx.end_launch();
        }
        return ctx.launch_check("variant iteration (FP32)");
    }

    int residual_pass(Ctx& ctx) const {
        ctx.begin_launch(MC_KERNEL_RESIDUAL);
        kvm_residual_rows<<<grid, kBlock, 0, ctx.stream>>>(Bs, V, M, O);
        ctx.end_launch();
        ctx.begin_launch(MC_KERNEL_RESIDUAL);
        kvm_residual_cols<<<grid, kBlock, 0, ctx.stream>>>(Bs, V, M, O);
        ctx.end_launch();
        return ctx.launch_check("variant residual (FP32)");
    }

    int recenter(Ctx& ctx, int force) const {
        ctx.begin_launch(MC_KERNEL_OTHER);
        kvm_recenter<<<grid, kBlock, 0, ctx.stream>>>(Bs.m, Bs.n, V, M, force);
        ctx.end_launch();
        return ctx.launch_check("variant recenter");
    }

    int check(Ctx& ctx, long long span, int final_pass, const Controls& ctl, const TraceBuf&) const {
        TRY(residual_pass(ctx));
        ctx.begin_launch(MC_KERNEL_RESIDUAL);
        kv_finalize<<<V.K, 256, 0, ctx.stream>>>(V, O.offset, span, final_pass, ctl);
        ctx.end_launch();
        if (!final_pass) TRY(recenter(ctx, 0));
        ctx.begin_launch(MC_KERNEL_OTHER);
        kv_poll<<<1, 1024, 0, ctx.stream>>>(V);
        ctx.end_launch();
        return ctx.launch_check("variant check (FP32)");
    }
};

// Host driver: the base LP's setup as a single solve's (upload, validation,
// transpose, Ruiz, norms), then the variants' bounds, starts and
// certificates, the PDHG loop in chunk graphs, and per-variant outputs.
int solve_variants(Ctx& ctx, const mc_lp* base, int count, const double* const* var_lower,
                   const double* const* var_upper, const mc_pdlp_options* o, const double* const* x0,
                   const double* const* y0, double* const* x_out, double* const* y_out, mc_pdlp_result* results) {
    ctx.drop_session();  // reuses the arena
    const double t_begin = now_ms();
    if (!base || count <= 0 || !results) return set_error(MC_ERR_INVALID_ARGUMENT, "no variants");
    TRY(validate_options(o));
    TRY(validate_lp(base));
    const bool mixed = o->precision == MC_PRECISION_FP32_REFINE;
    const int m = base->num_rows, n = base->num_cols;
    const long long nnz = base->nnz;
    for (int b = 0; b < count; ++b) {
        std::memset(&results[b], 0, sizeof(mc_pdlp_result));
        std::snprintf(results[b].backend_actually_used, sizeof results[b].backend_actually_used, "cuda");
        results[b].tolerance = o->primal_tolerance;
        results[b].certificate_index = -1;
    }
    if (m == 0 || n == 0) {  // pdlp.cpp:144-149, for every variant
        for (int b = 0; b < count; ++b) {
            results[b].status = MC_PDLP_OPTIMAL;
            fill_message(&results[b], "trivial");
            results[b].total_ms = now_ms() - t_begin;
        }
        return MC_OK;
    }
    const int Kp = (count + 31) / 32 * 32;
    const int groups = Kp / 32;
    if (groups > 65535) return set_error(MC_ERR_RESOURCE_LIMIT, "too many variants (%d)", count);
    cudaStream_t s = ctx.stream;
    for (int q = 0; q < MC_KERNEL_KINDS; ++q) {
        ctx.launches[q] = 0;
        ctx.kernel_ms[q] = 0.0;
    }
    ctx.profiling = o->profile_kernels != 0;
    ctx.pending.clear();
    ctx.prof_used = 0;
    ctx.release_graphs();

    // grid: (blocks per variant group, variant groups), about two waves of resident blocks
    int per_sm = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kv_residual_cols, kBlock, 0) != cudaSuccess ||
        per_sm < 1)
        per_sm = 1;
    const long long lines = std::max<long long>(n, m);
    long long nbx = std::max<long long>(1, (long long)ctx.sm_count * per_sm * 2 / groups);
    nbx = std::min<long long>(nbx, (lines + kVarWarps - 1) / kVarWarps);
    nbx = std::max<long long>(1, std::min<long long>(nbx, kMaxPartials));

    // ---- arena
    const bool dev_in = base->memory == MC_MEMORY_DEVICE;
    bool any_wx = false, any_wy = false;
    for (int b = 0; b < count; ++b) {
        any_wx = any_wx || (x0 && x0[b]);
        any_wy = any_wy || (y0 && y0[b]);
    }
    Layout L;
    const size_t o_cs = L.add<int>(n + 1), o_ri = L.add<int>(nnz + 16), o_cv = L.add<double>(nnz + 16);
    const size_t o_rs = L.add<int>(m + 1), o_ci = L.add<int>(nnz + 16), o_rv = L.add<double>(nnz + 16);
    const size_t o_cursor = L.add<int>(m), o_long = L.add<int>(m), o_counters = L.add<int>(4);
    const size_t o_scan = L.add<int>((m + 1) / kScanTile + 4096);
    size_t o_n[12], o_m[9];
    for (auto& v : o_n) v = L.add<double>(n);
    for (auto& v : o_m) v = L.add<double>(m);
    const size_t o_part1 = L.add<double>((long long)NUM_SLOTS * kMaxPartials);
    const size_t o_state = L.add<DevState>(count + 2);
    const long long nk = (long long)n * Kp, mk = (long long)m * Kp;
    size_t o_vn[7], o_vm[5];
    for (auto& v : o_vn) v = L.add<double>(nk);
    const size_t o_vxdx = L.add<double>(2 * nk);
    for (auto& v : o_vm) v = L.add<double>(mk);
    const size_t o_vpart = L.add<double>((long long)NUM_SLOTS * Kp * nbx);
    const size_t o_flags = L.add<int>(count), o_cert = L.add<int>(2LL * count);
    const size_t o_lo_in = L.add<double>((long long)count * n), o_hi_in = L.add<double>((long long)count * n);
    const size_t o_wx = any_wx ? L.add<double>((long long)count * n) : 0;
    const size_t o_wy = any_wy ? L.add<double>((long long)count * m) : 0;
    const size_t o_hw = L.add<int>(2LL * count);
    const size_t o_perm = L.add<int>(count);
    const size_t o_xo = L.add<double>((long long)count * n), o_yo = L.add<double>((long long)count * m);
    // FP32 form: FP32 matrix copies and norms, FP32 variant-minor correction data
    size_t o_f_cv = 0, o_f_rv = 0, o_f_cn = 0, o_f_rn = 0, o_fn[7] = {}, o_fxdx = 0, o_fm[6] = {};
    if (mixed) {
        o_f_cv = L.add<float>(nnz + 16);
        o_f_rv = L.add<float>(nnz + 16);
        o_f_cn = L.add<float>(n);
        o_f_rn = L.add<float>(m);
        for (auto& v : o_fn) v = L.add<float>(nk);
        o_fxdx = L.add<float>(2 * nk);
        for (auto& v : o_fm) v = L.add<float>(mk);
    }
    TRY(ctx.arena.reserve(L.offset));
    char* A = static_cast<char*>(ctx.arena.base);
    auto at = [&](size_t off) { return static_cast<void*>(A + off); };
    int* cs = static_cast<int*>(at(o_cs));
    int* ri = static_cast<int*>(at(o_ri));
    double* cv = static_cast<double*>(at(o_cv));
    int* rs = static_cast<int*>(at(o_rs));
    int* ci = static_cast<int*>(at(o_ci));
    double* rv = static_cast<double*>(at(o_rv));
    double* obj_in = static_cast<double*>(at(o_n[0]));
    double* base_lo_in = static_cast<double*>(at(o_n[1]));  // base variable bounds (base setup only)
    double* base_hi_in = static_cast<double*>(at(o_n[2]));
    double* c = static_cast<double*>(at(o_n[3]));
    double* lo_b = static_cast<double*>(at(o_n[4]));
    double* hi_b = static_cast<double*>(at(o_n[5]));
    double* c_orig = static_cast<double*>(at(o_n[6]));
    double* lo_orig = static_cast<double*>(at(o_n[7]));
    double* hi_orig = static_cast<double*>(at(o_n[8]));
    double* col_norm = static_cast<double*>(at(o_n[9]));
    double* col_scale = static_cast<double*>(at(o_n[10]));
    double* x_scratch = static_cast<double*>(at(o_n[11]));
    double* rlo_in = static_cast<double*>(at(o_m[0]));
    double* rhi_in = static_cast<double*>(at(o_m[1]));
    double* blo = static_cast<double*>(at(o_m[2]));
    double* bhi = static_cast<double*>(at(o_m[3]));
    double* blo_orig = static_cast<double*>(at(o_m[4]));
    double* bhi_orig = static_cast<double*>(at(o_m[5]));
    double* row_norm = static_cast<double*>(at(o_m[6]));
    double* row_scale = static_cast<double*>(at(o_m[7]));
    double* y_scratch = static_cast<double*>(at(o_m[8]));
    double* part1 = static_cast<double*>(at(o_part1));
    DevState* st = static_cast<DevState*>(at(o_state));  // [0] base, [1] poll, [2..] variants
    int* has_warm = static_cast<int*>(at(o_hw));

    // ---- uploads and validation of the base
    CU(cudaEventRecord(ctx.ev_a, s));
    const cudaMemcpyKind in_kind = dev_in ? cudaMemcpyDeviceToDevice : cudaMemcpyHostToDevice;
    CU(cudaMemcpyAsync(cs, base->col_start, sizeof(int) * (size_t)(n + 1), in_kind, s));
    if (nnz) {
        CU(cudaMemcpyAsync(ri, base->row_index, sizeof(int) * (size_t)nnz, in_kind, s));
        CU(cudaMemcpyAsync(cv, base->value, sizeof(double) * (size_t)nnz, in_kind, s));
    }
    CU(cudaMemsetAsync(ri + nnz, 0, sizeof(int) * 16, s));
    CU(cudaMemsetAsync(cv + nnz, 0, sizeof(double) * 16, s));
    CU(cudaMemsetAsync(ci + nnz, 0, sizeof(int) * 16, s));
    CU(cudaMemsetAsync(rv + nnz, 0, sizeof(double) * 16, s));
    CU(cudaMemcpyAsync(obj_in, base->objective, sizeof(double) * n, in_kind, s));
    CU(cudaMemcpyAsync(base_lo_in, base->var_lower, sizeof(double) * n, in_kind, s));
    CU(cudaMemcpyAsync(base_hi_in, base->var_upper, sizeof(double) * n, in_kind, s));
    CU(cudaMemcpyAsync(rlo_in, base->row_lower, sizeof(double) * m, in_kind, s));
    CU(cudaMemcpyAsync(rhi_in, base->row_upper, sizeof(double) * m, in_kind, s));
    double* lo_in = static_cast<double*>(at(o_lo_in));
    double* hi_in = static_cast<double*>(at(o_hi_in));
    double* wx = any_wx ? static_cast<double*>(at(o_wx)) : nullptr;
    double* wy = any_wy ? static_cast<double*>(at(o_wy)) : nullptr;
    std::vector<int> hw(2 * (size_t)count, 0);
    Staging& up = ctx.staging;
    up.begin();
    for (int b = 0; b < count; ++b)
        TRY(up.put(s, lo_in + (size_t)b * n, (var_lower && var_lower[b]) ? var_lower[b] : base->var_lower, sizeof(double) * n));
    for (int b = 0; b < count; ++b)
        TRY(up.put(s, hi_in + (size_t)b * n, (var_upper && var_upper[b]) ? var_upper[b] : base->var_upper, sizeof(double) * n));
    for (int b = 0; b < count; ++b)
        if (x0 && x0[b]) {
            hw[b] = 1;
            TRY(up.put(s, wx + (size_t)b * n, x0[b], sizeof(double) * n));
        }
    for (int b = 0; b < count; ++b)
        if (y0 && y0[b]) {
            hw[count + b] = 1;
            TRY(up.put(s, wy + (size_t)b * m, y0[b], sizeof(double) * m));
        }
    TRY(up.flush(s));
    CU(cudaMemcpyAsync(has_warm, hw.data(), sizeof(int) * hw.size(), cudaMemcpyHostToDevice, s));
    CU(cudaEventRecord(ctx.ev_b, s));
    int* counters = static_cast<int*>(at(o_counters));
    CU(cudaMemsetAsync(counters, 0, sizeof(int) * 4, s));
    ctx.begin_launch(MC_KERNEL_SETUP);
    k_validate_csc<<<(n + kBlock - 1) / kBlock, kBlock, 0, s>>>(m, n, nnz, cs, ri, cv, counters + 2);
    ctx.end_launch();
    int bad = 0;
    CU(cudaMemcpyAsync(&bad, counters + 2, sizeof(int), cudaMemcpyDeviceToHost, s));
    CU(cudaStreamSynchronize(s));
    TRY(ctx.drain_profile());
    if (bad) return set_error(MC_ERR_INVALID_ARGUMENT, "invalid CSC matrix in the base LP (flags %d)", bad);

    // ---- the base LP's setup (shared by every variant)
    CU(cudaMemsetAsync(st, 0, sizeof(DevState) * (count + 2), s));
    int longest[2];  // entries of a row, of a column
    TRY(build_csr(ctx, m, n, nnz, cs, ri, cv, rs, ci, rv, static_cast<int*>(at(o_cursor)),
                  static_cast<int*>(at(o_long)), counters, static_cast<int*>(at(o_scan)), longest));
    TRY(ruiz(ctx, m, n, nnz, cs, ri, cv, rs, ci, rv, row_scale, col_scale, y_scratch, row_norm, x_scratch,
             col_norm, part1, st,
             o->ruiz_scaling ? o->ruiz_iterations : 0));
    const double obj_sign = (base->objective_sense == MC_MAXIMIZE) ? -1.0 : 1.0;
    const int nbc = blocks_for(ctx, n, kBlock), nbr = blocks_for(ctx, m, kBlock);
    ctx.begin_launch(MC_KERNEL_SETUP);
    k_setup_cols<<<nbc, kBlock, 0, s>>>(n, cs, cv, obj_in, base_lo_in, base_hi_in, col_scale, nullptr, obj_sign, c,
                                        lo_b, hi_b, c_orig, lo_orig, hi_orig, col_norm, x_scratch, x_scratch, part1);
    ctx.end_launch();
    ctx.begin_launch(MC_KERNEL_SETUP);
    k_setup_rows<<<nbr, kBlock, 0, s>>>(m, rs, rv, rlo_in, rhi_in, row_scale, nullptr, blo, bhi, blo_orig, bhi_orig,
                                        row_norm, y_scratch, y_scratch, part1);
    ctx.end_launch();
    ctx.begin_launch(MC_KERNEL_SETUP);
    k_setup_scalars<<<1, 1024, 0, s>>>(part1, nbc, nbr, o->initial_primal_weight, o->step_size_reduction, st);
    ctx.end_launch();

    // ---- the variants
    VarBase Bs{m, n, cs, ri, cv, rs, ci, rv, c, col_norm, row_norm, blo, bhi};
    VarRefs V;
    V.K = count;
    V.Kp = Kp;
    V.nb = (int)nbx;
    V.st = st + 2;
    V.global = st + 1;
    V.lo = static_cast<double*>(at(o_vn[0]));
    V.hi = static_cast<double*>(at(o_vn[1]));
    V.olo = static_cast<double*>(at(o_vn[2]));
    V.ohi = static_cast<double*>(at(o_vn[3]));
    V.x = static_cast<double*>(at(o_vn[4]));
    V.xb = static_cast<double*>(at(o_vn[5]));
    V.xa = static_cast<double*>(at(o_vn[6]));
    V.xdx = static_cast<double*>(at(o_vxdx));
    V.y = static_cast<double*>(at(o_vm[0]));
    V.ya = static_cast<double*>(at(o_vm[1]));
    V.axb = static_cast<double*>(at(o_vm[2]));
    V.y_prev = static_cast<double*>(at(o_vm[3]));
    V.dray = static_cast<double*>(at(o_vm[4]));
    V.partials = static_cast<double*>(at(o_vpart));
    V.flags = static_cast<int*>(at(o_flags));
    V.cert_idx = static_cast<int*>(at(o_cert));
    CU(cudaMemsetAsync(V.partials, 0, sizeof(double) * (size_t)NUM_SLOTS * Kp * nbx, s));
    const dim3 grid((unsigned)nbx, (unsigned)groups);
    // Slots: variant b of the caller sits in slot k with perm[k] = b.  The
    // variants certified infeasible at setup go last, so that the groups of
    // 32 slots that hold only finished variants leave every kernel at once;
    // the certificates are found with the identity order first.
    int* perm_dev = static_cast<int*>(at(o_perm));
    std::vector<int> perm(count);
    for (int b = 0; b < count; ++b) perm[b] = b;
    auto setup_slots = [&]() -> int {
        CU(cudaMemcpyAsync(perm_dev, perm.data(), sizeof(int) * count, cudaMemcpyHostToDevice, s));
        CU(cudaMemsetAsync(V.flags, 0, sizeof(int) * count, s));
        CU(cudaMemsetAsync(V.cert_idx, 0x7f, sizeof(int) * 2 * (size_t)count, s));  // "none" above any index
        ctx.begin_launch(MC_KERNEL_SETUP);
        kv_setup_cols<<<grid, kBlock, 0, s>>>(Bs, V, perm_dev, lo_in, hi_in, wx, any_wx ? has_warm : nullptr,
                                              col_scale);
        ctx.end_launch();
        ctx.begin_launch(MC_KERNEL_SETUP);
        kv_setup_rows<<<grid, kBlock, 0, s>>>(Bs, V, perm_dev, rlo_in, rhi_in, row_scale, col_scale, wy,
                                              any_wy ? has_warm + count : nullptr);
        ctx.end_launch();
        return ctx.launch_check("variant slots");
    };
    TRY(setup_slots());
    {
        std::vector<int> hflags(count);
        CU(cudaMemcpyAsync(hflags.data(), V.flags, sizeof(int) * count, cudaMemcpyDeviceToHost, s));
        CU(cudaStreamSynchronize(s));
        TRY(ctx.drain_profile());
        std::vector<int> order;
        order.reserve(count);
        for (int b = 0; b < count; ++b)
            if (!hflags[b]) order.push_back(b);
        for (int b = 0; b < count; ++b)
            if (hflags[b]) order.push_back(b);
        if (order != perm) {
            perm = order;
            TRY(setup_slots());
        }
    }
    ctx.begin_launch(MC_KERNEL_SETUP);
    kv_setup_state<<<(count + 255) / 256, 256, 0, s>>>(V, st);
    ctx.end_launch();
    ctx.begin_launch(MC_KERNEL_SETUP);
    kv_poll<<<1, 1024, 0, s>>>(V);
    ctx.end_launch();
    TRY(ctx.launch_check("variant setup"));

    Original O{c_orig, obj_in, lo_orig, hi_orig, blo_orig, bhi_orig, col_scale, row_scale, base->objective_offset};
    Controls ctl{o->primal_tolerance, o->dual_tolerance, o->gap_tolerance, o->restart_reduction_factor,
                 o->primal_weight_smoothing, o->restart_every, o->restart_strategy, o->adaptive_step_size,
                 o->adaptive_primal_weight};
    TraceBuf tr{0, nullptr, nullptr, nullptr, nullptr, nullptr, nullptr, nullptr};
    const int poll_every = o->check_every_chunks > 0 ? o->check_every_chunks : 1;
    VarMixed M{};
    // Rows go to the split form while one wave of its warps takes them all,
    // else to packs, which issue fewer instructions: us per dual launch split /
    // packs / one variant per lane, 8 entries a column: 8.6 / 17.2 / 12.7 (32 x
    // 2000 rows, FP32), 10.6 / 12.6 / 13.7 (FP64); 18.1 / 14.1 / 16.8 (128 x 2000,
    // FP32), 20.9 / 14.8 / 20.3 (FP64).
    const bool rows_wide = (long long)m * groups > (long long)ctx.sm_count * kVarDualBlocks * kVarWarps;
    if (!mixed) {
        EngineVariants eng;
        eng.Bs = Bs;
        eng.V = V;
        eng.O = O;
        eng.grid = grid;
        eng.long_cols = longest[1] > kVarLongColumn;
        eng.cols = eng.long_cols ? wide_grid<double>(ctx, kv_primal_wide<true>, n, Kp)
                                 : wide_grid<double>(ctx, kv_primal_wide<false>, n, Kp);
        eng.rows = dual_grid(ctx, kv_dual<false>, m, groups);
        eng.wide = wide_grid<double>(ctx, kv_dual_wide<false>, m, Kp);
        eng.rows_wide = rows_wide;
        TRY(run_chunks(ctx, eng, V.global, o->max_iterations, o->restart_every, poll_every, ctl, tr));
    } else {
        float* f_cv = static_cast<float*>(at(o_f_cv));
        float* f_rv = static_cast<float*>(at(o_f_rv));
        float* f_cn = static_cast<float*>(at(o_f_cn));
        float* f_rn = static_cast<float*>(at(o_f_rn));
        const int nbz = blocks_for(ctx, nnz + 16, kBlock) * 4;
        ctx.begin_launch(MC_KERNEL_SETUP);
        k_to_float<<<nbz, kBlock, 0, s>>>(nnz + 16, cv, f_cv);
        ctx.end_launch();
        ctx.begin_launch(MC_KERNEL_SETUP);
        k_to_float<<<nbz, kBlock, 0, s>>>(nnz + 16, rv, f_rv);
        ctx.end_launch();
        ctx.begin_launch(MC_KERNEL_SETUP);
        k_to_float<<<blocks_for(ctx, n, kBlock), kBlock, 0, s>>>(n, col_norm, f_cn);
        ctx.end_launch();
        ctx.begin_launch(MC_KERNEL_SETUP);
        k_to_float<<<blocks_for(ctx, m, kBlock), kBlock, 0, s>>>(m, row_norm, f_rn);
        ctx.end_launch();
        M.cs = cs;
        M.ri = ri;
        M.cv = f_cv;
        M.rs = rs;
        M.ci = ci;
        M.rv = f_rv;
        M.col_norm = f_cn;
        M.row_norm = f_rn;
        M.c64 = c;
        M.blo64 = blo;
        M.bhi64 = bhi;
        M.xh = V.x;       // the FP64 start point is every variant's first base
        M.yh = V.y;
        M.axf = V.axb;
        M.atyf = V.xb;
        float* fn[7];
        for (int q = 0; q < 7; ++q) fn[q] = static_cast<float*>(at(o_fn[q]));
        float* fm[6];
        for (int q = 0; q < 6; ++q) fm[q] = static_cast<float*>(at(o_fm[q]));
        M.x = fn[0];
        M.xb = fn[1];
        M.xa = fn[2];
        M.g = fn[3];
        M.lo = fn[4];
        M.hi = fn[5];
        M.xdx = static_cast<float*>(at(o_fxdx));
        M.y = fm[0];
        M.ya = fm[1];
        M.axb = fm[2];
        M.yb = fm[3];
        M.rlo = fm[4];
        M.rhi = fm[5];
        // corrections start at zero (padding lanes included: gathers read them)
        for (int q = 0; q < 7; ++q) CU(cudaMemsetAsync(fn[q], 0, sizeof(float) * (size_t)nk, s));
        CU(cudaMemsetAsync(M.xdx, 0, sizeof(float) * 2 * (size_t)nk, s));
        for (int q = 0; q < 6; ++q) CU(cudaMemsetAsync(fm[q], 0, sizeof(float) * (size_t)mk, s));
        EngineVariantsMixed eng;
        eng.Bs = Bs;
        eng.V = V;
        eng.M = M;
        eng.O = O;
        eng.grid = grid;
        eng.cols = wide_grid<float>(ctx, kvm_primal_wide, n, Kp);
        eng.rows = dual_grid(ctx, kvm_dual<false>, m, groups);
        eng.wide = wide_grid<float>(ctx, kvm_dual_wide<false>, m, Kp);
        eng.rows_wide = rows_wide;
        // the first correction LP of every running variant, around its start
        TRY(eng.residual_pass(ctx));
        TRY(eng.recenter(ctx, 1));
        TRY(run_chunks(ctx, eng, V.global, o->max_iterations, o->restart_every, poll_every, ctl, tr));
    }
    CU(cudaEventRecord(ctx.ev_c, s));

    // ---- outputs
    double* xo = static_cast<double*>(at(o_xo));
    double* yo = static_cast<double*>(at(o_yo));
    ctx.begin_launch(MC_KERNEL_OTHER);
    if (mixed) kvm_unscale_out<<<grid, kBlock, 0, s>>>(m, n, V, M, col_scale, row_scale, xo, yo);
    else kv_unscale_out<<<grid, kBlock, 0, s>>>(Bs, V, col_scale, row_scale, xo, yo);
    ctx.end_launch();
    TRY(ctx.launch_check("variant unscale"));
    std::vector<Staging::Piece> x_pieces, y_pieces;
    for (int k = 0; k < count; ++k) {  // slot k holds variant perm[k]
        const int b = perm[k];
        const size_t xb = sizeof(double) * (size_t)n, yb = sizeof(double) * (size_t)m;
        if (x_out && x_out[b]) x_pieces.push_back({x_out[b], (size_t)k * xb, xb});
        if (y_out && y_out[b]) y_pieces.push_back({y_out[b], (size_t)k * yb, yb});
    }
    TRY(up.get(s, xo, x_pieces));
    TRY(up.get(s, yo, y_pieces));
    std::vector<DevState> hs(count + 2);
    CU(cudaMemcpyAsync(hs.data(), st, sizeof(DevState) * (count + 2), cudaMemcpyDeviceToHost, s));
    std::vector<int> hcert(2 * (size_t)count);
    CU(cudaMemcpyAsync(hcert.data(), V.cert_idx, sizeof(int) * hcert.size(), cudaMemcpyDeviceToHost, s));
    CU(cudaEventRecord(ctx.ev_d, s));
    CU(cudaStreamSynchronize(s));
    if (hs[0].fault) return set_error(MC_ERR_CUDA, "a wait of a cooperative kernel timed out");
    TRY(ctx.drain_profile());
    float h2d = 0.f, kern = 0.f, d2h = 0.f;
    CU(cudaEventElapsedTime(&h2d, ctx.ev_a, ctx.ev_b));
    CU(cudaEventElapsedTime(&kern, ctx.ev_b, ctx.ev_c));
    CU(cudaEventElapsedTime(&d2h, ctx.ev_c, ctx.ev_d));
    long long total = 0;
    for (int q = 0; q < MC_KERNEL_KINDS; ++q) total += ctx.launches[q];
    const double total_ms = now_ms() - t_begin;
    for (int k = 0; k < count; ++k) {
        const int b = perm[k];
        mc_pdlp_result& r = results[b];
        const DevState& S = hs[2 + k];
        r.status = S.status;
        r.objective = S.objective;
        r.primal_infeasibility = S.primal_infeas;
        r.dual_infeasibility = S.dual_infeas;
        r.duality_gap = S.gap;
        r.iterations = S.iter;
        r.certificate = S.status == MC_PDLP_INFEASIBLE_OR_UNBOUNDED ? S.cert : MC_CERT_NONE;
        r.certificate_index = r.certificate == MC_CERT_CROSSED_BOUNDS ? hcert[k]
                              : r.certificate == MC_CERT_ROW_ACTIVITY ? hcert[count + k]
                                                                      : -1;
        fill_message(&r, S.status == MC_PDLP_OPTIMAL ? "PDLP converged"
                         : r.certificate == MC_CERT_CROSSED_BOUNDS ? "infeasible: crossed variable bounds"
                         : r.certificate == MC_CERT_ROW_ACTIVITY ? "infeasible: row activity outside its bounds"
                         : r.certificate == MC_CERT_DUAL_RAY ? "infeasible: dual ray (Farkas certificate in dual)"
                         : S.status == MC_PDLP_NUMERICAL_FAILURE ? "non-finite iterate or residual"
                                                                 : "iteration limit reached");
        r.h2d_ms = dev_in ? 0.0 : h2d;
        r.kernel_ms = kern + (dev_in ? h2d : 0.0);
        r.d2h_ms = d2h;
        r.total_ms = total_ms;
        r.ruiz_iterations_executed = o->ruiz_scaling ? hs[0].ruiz_passes : 0;
        r.restarts = S.restarts;
        r.final_primal_weight = S.omega;
        r.final_step_size = S.eta;
        r.kernel_launches = total;
        r.refinement_rounds = mixed ? S.restarts : 0;  // each restart re-centres the variant's FP64 base
        r.inner_iterations = mixed ? S.iter : 0;
        for (int q = 0; q < MC_KERNEL_KINDS; ++q) {
            r.launches_by_kind[q] = ctx.launches[q];
            r.kernel_ms_by_kind[q] = ctx.kernel_ms[q];
        }
    }
    return MC_OK;
}

}  // namespace mc

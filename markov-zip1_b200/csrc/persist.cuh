// The PDHG loop of small and medium LPs as one persistent kernel
// (src/lp/first_order/pdlp.cpp:194-275): whole restart chunks -- iterations,
// step-size rule, KKT check, restart -- run inside one launch, the phases of
// an iteration separated by a barrier instead of a kernel boundary.
//
// Why: below about a million nonzeros an iteration of the streaming kernels
// (iter_kernels.cuh) is two launches of 4-5 us each whatever the size, because
// a launch, its ramp and its drain cost more than the work.
//
// Every group of G lanes owns one column and one row for the whole launch and
// keeps their vector entries (bounds, step, iterate, average) in registers;
// the block's slice of the matrix lies in shared memory where it fits.  Two
// forms:
//   * CL (cluster): one thread-block cluster of 1..16 blocks.  Every block has
//     a full copy of the gathered vectors (x-bar, dx, y) in shared memory; new
//     entries go to the other blocks' copies through distributed shared
//     memory.  The barrier is the hardware cluster barrier.
//   * grid: one block per SM (cooperative launch), the gathered vectors in
//     global memory (L2).  An entry is stored together with the number of the
//     iteration that wrote it, in one 16-byte word, and a gather repeats its
//     load until the number is the one it needs: no barrier at all (one at
//     148 blocks costs 2 us, an iteration with four of them 7 us against 3.3
//     on the smallest LPs).  The entries are updated in place: x-bar_j is read
//     by the rows of column j only, and its owner overwrites it only after
//     gathering the new duals of those rows, which they wrote after reading it
//     (and the same with rows and columns exchanged).  The reductions
//     (step-size rule, KKT check) exchange their partials the same way.
// The averages are updated after the new entries are on their way, off the
// chain gather -> update -> store that sets the time of an iteration.
//
// Arithmetic: every line's dot runs over the same lanes in the same order as
// line_dot / line_dot2 of the streaming kernels, and the element-wise updates
// are the same operations, so the iterates agree bit for bit with those
// kernels' (FP64 and FP32); only the block partials of the reductions that
// feed the step-size rule and the KKT check are grouped differently.
#pragma once

#include "common.cuh"
#include "iter_kernels.cuh"
#include "mixed.cuh"

#include <cooperative_groups.h>
#include <cstddef>

namespace mc {

constexpr int kPersistMaxBlocks = 160;
constexpr int kPersistPartials = 2 * 2 * 8 * kPersistMaxBlocks;  // tagged partials and sums of the reductions

// ---- gathered vectors
// Grid form: an entry and the number of the iteration that wrote it, in one
// 16-byte word that is read and written whole (FP32 entries as doubles: 8-byte
// words put four owners into a sector, 8.8 us an iteration against 7.5 at 400k
// nonzeros).  Every bit of the word is used: a load of which only parts are
// used may be narrowed and is then no longer one access.
using Tag = unsigned long long;
constexpr Tag kFailed = 1ull << 63;  // in the tag of a reduction's partial or sum: a wait has run out
template <class T>
struct alignas(16) Tagged {
    unsigned long long value;
    Tag tag;
};
__device__ __forceinline__ void ld_tagged(const Tagged<double>* p, double& v, Tag& tag) {
    unsigned long long a;
    asm volatile("{\n .reg .b128 q;\n ld.relaxed.gpu.global.b128 q, [%2];\n mov.b128 {%0, %1}, q;\n}"
                 : "=l"(a), "=l"(tag)
                 : "l"(p)
                 : "memory");
    v = __longlong_as_double((long long)a);
}
__device__ __forceinline__ void st_tagged(Tagged<double>* p, double v, Tag tag) {
    asm volatile("{\n .reg .b128 q;\n mov.b128 q, {%1, %2};\n st.relaxed.gpu.global.b128 [%0], q;\n}" ::"l"(p),
                 "l"(__double_as_longlong(v)), "l"(tag)
                 : "memory");
}
__device__ __forceinline__ void ld_tagged(const Tagged<float>* p, float& v, Tag& tag) {
    double d;
    ld_tagged(reinterpret_cast<const Tagged<double>*>(p), d, tag);
    v = (float)d;
}
__device__ __forceinline__ void st_tagged(Tagged<float>* p, float v, Tag tag) {
    st_tagged(reinterpret_cast<Tagged<double>*>(p), (double)v, tag);
}

// Where a dot gathers from: the block's shared copy (CL), or tagged entries,
// of which a thread waits for tag `want`.  All loads of a step are out before
// the first is waited for, and every round repeats the missing ones together;
// `bad` is set once a wait has run out (no further wait then).
template <class T>
struct FromShared {
    const T* v;
    __device__ static T scalar();
    template <int N>
    __device__ __forceinline__ void get(const int (&i)[N], T (&a)[N]) {
#pragma unroll
        for (int q = 0; q < N; ++q) a[q] = v[i[q]];
    }
};
template <class T>
struct FromBase {  // mixed form, CL: base plus averaged correction from global memory
    const double* base;
    const T* corr;
    __device__ static double scalar();
    template <int N>
    __device__ __forceinline__ void get(const int (&i)[N], double (&a)[N]) {
#pragma unroll
        for (int q = 0; q < N; ++q) a[q] = __ldcg(base + i[q]) + (double)__ldcg(corr + i[q]);
    }
};
template <class T, int STRIDE, bool REDUCTION = false>
struct FromTagged {
    const Tagged<T>* v;
    Tag want;
    unsigned limit;
    bool& bad;
    __device__ static T scalar();
    template <int N>
    __device__ __forceinline__ void get(const int (&i)[N], T (&a)[N]) {
        Tag tag[N];
#pragma unroll
        for (int q = 0; q < N; ++q) ld_tagged(v + (long long)STRIDE * i[q], a[q], tag[q]);
        unsigned spins = 0;
        while (true) {
            bool all = true;
#pragma unroll
            for (int q = 0; q < N; ++q) all = all && (REDUCTION ? tag[q] & ~kFailed : tag[q]) == want;
            if (REDUCTION && all) {
#pragma unroll
                for (int q = 0; q < N; ++q) bad = bad || (tag[q] & kFailed);
            }
            if (all || bad) return;
#pragma unroll
            for (int q = 0; q < N; ++q)
                if (tag[q] != want) ld_tagged(v + (long long)STRIDE * i[q], a[q], tag[q]);
            bad = ++spins > limit;
        }
    }
};

// line_dot's lanes and order over entries [b, e) of a slice.  The up to three
// entries left over are gathered together too: those that do not exist repeat
// the first one.
template <class T, class From>
__device__ __forceinline__ T slice_dot(const int* idx, const T* val, From from, int b, int e, int G, int sub) {
    T s0 = T(0), s1 = T(0), s2 = T(0), s3 = T(0);
    int p = b + sub;
    for (; p + 3 * G < e; p += 4 * G) {
        const int i[4] = {idx[p], idx[p + G], idx[p + 2 * G], idx[p + 3 * G]};
        T v[4];
        from.get(i, v);
        s0 = fma(val[p], v[0], s0);
        s1 = fma(val[p + G], v[1], s1);
        s2 = fma(val[p + 2 * G], v[2], s2);
        s3 = fma(val[p + 3 * G], v[3], s3);
    }
    if (p < e) {
        const int p1 = p + G < e ? p + G : p, p2 = p + 2 * G < e ? p + 2 * G : p;
        const int i[3] = {idx[p], idx[p1], idx[p2]};
        T v[3];
        from.get(i, v);
        s0 = fma(val[p], v[0], s0);
        if (p1 != p) s0 = fma(val[p1], v[1], s0);
        if (p2 != p) s0 = fma(val[p2], v[2], s0);
    }
    return (s0 + s1) + (s2 + s3);
}

// line_dot2's lanes and order: x-bar and dx, from two shared copies or from
// tagged pairs (one gather of four for two entries)
template <class T>
struct PairsFromShared {
    const T *x, *d;
    __device__ __forceinline__ void get(int i0, int i1, T (&v)[2], T (&w)[2]) {
        v[0] = x[i0];
        w[0] = d[i0];
        v[1] = x[i1];
        w[1] = d[i1];
    }
};
template <class T>
struct PairsFromTagged {
    FromTagged<T, 1> pairs;
    __device__ __forceinline__ void get(int i0, int i1, T (&v)[2], T (&w)[2]) {
        const int i[4] = {2 * i0, 2 * i0 + 1, 2 * i1, 2 * i1 + 1};
        T a[4];
        pairs.get(i, a);
        v[0] = a[0];
        w[0] = a[1];
        v[1] = a[2];
        w[1] = a[3];
    }
};
template <class T, class Pairs>
__device__ __forceinline__ void slice_dot2(const int* idx, const T* val, Pairs from, int b, int e, int G, int sub,
                                           T& out_v, T& out_w) {
    T sv0 = T(0), sw0 = T(0), sv1 = T(0), sw1 = T(0);
    for (int p = b + sub; p < e; p += 2 * G) {
        const bool two = p + G < e;
        const int p1 = two ? p + G : p;
        T v[2], w[2];
        from.get(idx[p], idx[p1], v, w);
        sv0 = fma(val[p], v[0], sv0);
        sw0 = fma(val[p], w[0], sw0);
        if (two) {
            sv1 = fma(val[p1], v[1], sv1);
            sw1 = fma(val[p1], w[1], sw1);
        }
    }
    out_v = sv0 + sv1;
    out_w = sw0 + sw1;
}

// The residual pass's lanes and order (one accumulator per lane), FP64
template <class From>
__device__ __forceinline__ double slice_dot_plain(const int* idx, const double* val, From from, int b, int e, int G,
                                                  int sub) {
    double s = 0.0;
    for (int p = b + sub; p < e; p += 4 * G) {
        const int p1 = p + G < e ? p + G : p, p2 = p + 2 * G < e ? p + 2 * G : p, p3 = p + 3 * G < e ? p + 3 * G : p;
        const int i[4] = {idx[p], idx[p1], idx[p2], idx[p3]};
        decltype(from.scalar()) v[4];
        from.get(i, v);
        s = fma(val[p], (double)v[0], s);
        if (p1 != p) s = fma(val[p1], (double)v[1], s);
        if (p2 != p) s = fma(val[p2], (double)v[2], s);
        if (p3 != p) s = fma(val[p3], (double)v[3], s);
    }
    return s;
}

// a / b, correctly rounded, from y = 1 / b (correctly rounded): Markstein's
// corrections (P. Markstein, IBM J. Res. Dev. 34, 1990).  a y is within 1.5
// units of the last place of a / b; the first correction brings it within
// one, the second rounds it correctly, as every remainder a - q b is then
// exact.  Holds while no intermediate under- or overflows: outside a safe
// range of |a| and y it divides.  (b is an iteration count or a step size; a
// step size of an unscaled model can be anything, 0 and infinity included.)
__device__ __forceinline__ double div_recip(double a, double b, double y) {
    const double m = fabs(a);
    if (!(y > 1e-100 && y < 1e150) || !(m < 1e150) || (m < 1e-150 && m != 0.0)) return __ddiv_rn(a, b);
    double q = __dmul_rn(a, y);
    q = fma(fma(-q, b, a), y, q);
    return fma(fma(-q, b, a), y, q);
}
__device__ __forceinline__ float div_recip(float a, float b, float y) {
    const float m = fabsf(a);
    if (!(y > 1e-15f && y < 1e15f) || !(m < 1e15f) || (m < 1e-15f && m != 0.f)) return __fdiv_rn(a, b);
    float q = __fmul_rn(a, y);
    q = fmaf(fmaf(-q, b, a), y, q);
    return fmaf(fmaf(-q, b, a), y, q);
}

struct PersistArgs {
    Original O;
    Controls ctl;
    TraceBuf tr;
    int chunks;         // whole restart chunks to run, each with its check
    int R;              // iterations per chunk
    int skip;           // iterations of the first chunk that earlier launches ran
    int rem;            // then the iterations of another chunk up to this one,
    int final_pass;     // evaluated as the loop's last (1), or left for the next launch (0)
    int g_col, g_row, g_probe;  // lanes per line
    int smem_bytes;     // dynamic shared memory of the launch
    unsigned* counter;  // arrivals at the grid barrier, zeroed before the launch
    WaitLimits limits;
    int fail_block;     // -1, or a block whose waits run out at once (tests)
    // grid form: tagged (x-bar, dx) pairs [2n] and y [2m, every other one used]:
    // one 32-byte sector per column and row, whose owner is its only writer
    void *tx, *ty;
    Tagged<double>*ax, *ay;  // grid form: tagged averages [n], [m] of a KKT check
    Tagged<double>* tp;      // grid form: [2][8][kPersistMaxBlocks] tagged block partials, [2][kPersistMaxBlocks][8] sums
    int stage_y;        // grid form: the whole y is copied to shared memory per iteration
};

// Sum or maximum over a warp.
__device__ __forceinline__ double warp_fold(double t, bool mx) {
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
        const double o = __shfl_xor_sync(0xffffffffu, t, off);
        t = mx ? maxv(t, o) : t + o;
    }
    return t;
}

// One group's column and row, in registers.  All lanes of a group hold the
// same values.
template <class T>
struct ColState {
    int b = 0, e = 0;  // entries within the block's slice
    T c, lo, hi, tau, x, xa;
};
template <class T>
struct RowState {
    int b = 0, e = 0;
    bool fixed;
    T sigma, rsigma, b0, b1, y, ya, yb;  // b0, b1: row bounds, or the correction's A x_hat - b
};

template <class T, bool CL, int NT>
__global__ void __launch_bounds__(NT, 1) k_persist(Iterates<T> P, MixedState M, PersistArgs A) {
    constexpr bool MX = sizeof(T) == 4;  // the correction LP of the mixed form
    constexpr int WMAX = NT / 32;
    const int nt = blockDim.x, W = nt >> 5;
    extern __shared__ __align__(16) char dyn[];
    __shared__ DevState S;
    __shared__ double red[8][WMAX];
    __shared__ double parts[8][16];  // CL: every block's partials
    __shared__ double sums[8];
    __shared__ T rcnts[64];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int b = blockIdx.x, nb = gridDim.x;
    namespace cg = cooperative_groups;
    if (tid == 0) S = *P.st;
    __syncthreads();
    if (S.done) return;  // every block reads the same state
    const int Gc = A.g_col, Gr = A.g_row, Gp = A.g_probe;
    const int sub_c = tid & (Gc - 1), sub_r = tid & (Gr - 1);
    // the block's lines: equal runs, at most blockDim / G of them (the launch's rule)
    const int npb = (P.n + nb - 1) / nb, mpb = (P.m + nb - 1) / nb;
    const int c0 = min(P.n, b * npb), nc = min(npb, P.n - c0);
    const int r0 = min(P.m, b * mpb), nr = min(mpb, P.m - r0);
    const int j = c0 + tid / Gc, i = r0 + tid / Gr;  // the group's column and row
    const bool vc = tid / Gc < nc, vr = tid / Gr < nr;
    const bool own_c = vc && sub_c == 0, own_r = vr && sub_r == 0;

    // ---- shared memory: the gathered vectors (CL), then the matrix slices
    char* at = dyn;
    auto take = [&](long long bytes) -> char* {
        bytes = (bytes + 15) & ~15LL;
        if (at + bytes > dyn + A.smem_bytes) return nullptr;
        char* p = at;
        at += bytes;
        return p;
    };
    T* xbuf = reinterpret_cast<T*>(dyn);
    T* dbuf = xbuf + P.n;
    T* ybuf = dbuf + P.n;
    if (CL) take((2LL * P.n + P.m) * (long long)sizeof(T));
    const bool stage_y = !CL && A.stage_y;
    if (stage_y) ybuf = reinterpret_cast<T*>(take(2LL * P.m * (long long)sizeof(T)));  // two copies, in turn
    const int pc = P.csc_start[c0], pr = P.csr_start[r0];
    const int zc = P.csc_start[c0 + nc] - pc, zr = P.csr_start[r0 + nr] - pr;
    int* ri_s = nullptr;
    int* ci_s = nullptr;
    T* cv_s = reinterpret_cast<T*>(take((long long)zc * sizeof(T)));
    if (cv_s) ri_s = reinterpret_cast<int*>(take((long long)zc * sizeof(int)));
    T* rv_s = reinterpret_cast<T*>(take((long long)zr * sizeof(T)));
    if (rv_s) ci_s = reinterpret_cast<int*>(take((long long)zr * sizeof(int)));
    const bool cs_sh = ri_s != nullptr, rs_sh = ci_s != nullptr;
    const int* ri_g = P.csc_row + pc;
    const int* ci_g = P.csr_col + pr;
    const T* cv_g = P.csc_val + pc;
    const T* rv_g = P.csr_val + pr;
    if (cs_sh)
        for (int q = tid; q < zc; q += nt) {
            cv_s[q] = cv_g[q];
            ri_s[q] = ri_g[q];
        }
    if (rs_sh)
        for (int q = tid; q < zr; q += nt) {
            rv_s[q] = rv_g[q];
            ci_s[q] = ci_g[q];
        }
    if (CL)
        for (int q = tid; q < P.m; q += nt) ybuf[q] = P.y[q];
    Tagged<T>* tx = static_cast<Tagged<T>*>(A.tx);
    Tagged<T>* ty = static_cast<Tagged<T>*>(A.ty);
    Tag now = 0;  // number of the iteration within the launch (a check counts as one)
    Tag rnum = 0;  // number of the reduction
    bool bad = !CL && b == A.fail_block;
    // dots of the group's lines against the gathered vectors
    auto from = [&](T* shared, Tagged<T>* tagged, Tag want) {
        if constexpr (CL) return FromShared<T>{shared};
        else return FromTagged<T, 2>{tagged, want, A.limits.entry, bad};
    };
    auto pairs = [&]() {
        if constexpr (CL) return PairsFromShared<T>{xbuf, dbuf};
        else return PairsFromTagged<T>{{tx, now, A.limits.entry, bad}};
    };
    // The whole of a short vector into shared memory.  Entries that no line of
    // this block needs may already be ahead of `want`: any tag from it on ends
    // the wait.  The copy of the iteration before may still be read by slower
    // warps of the block, so there are two (one barrier per phase).
    auto stage = [&](T* to, const Tagged<T>* tagged, int len, Tag want) {
        for (int q = tid; q < len; q += nt) {
            T v;
            Tag tag;
            unsigned spins = 0;
            ld_tagged(tagged + 2LL * q, v, tag);
            while (tag < want && !bad) {
                ld_tagged(tagged + 2LL * q, v, tag);
                bad = ++spins > A.limits.entry;
            }
            to[q] = v;
        }
        __syncthreads();
    };

    ColState<T> C{};
    RowState<T> Q{};
    // probe lanes: twice the row's, so a block's rows take up to two trips there
    const int sub_p = tid & (Gp - 1);
    if (vc) {
        C.b = P.csc_start[j] - pc;
        C.e = P.csc_start[j + 1] - pc;
        C.c = P.c[j];
        C.lo = P.lo[j];
        C.hi = P.hi[j];
        C.x = P.x[j];
        C.xa = P.x_avg[j];
    }
    if (vr) {
        Q.b = P.csr_start[i] - pr;
        Q.e = P.csr_start[i + 1] - pr;
        Q.b0 = MX ? T(M.r_lo[i]) : P.blo[i];
        Q.b1 = MX ? T(M.r_hi[i]) : P.bhi[i];
        Q.y = P.y[i];
        Q.ya = P.y_avg[i];
        if (MX) Q.yb = T(M.yb[i]);
    }
    // step sizes, after every change of eta or omega
    auto set_steps = [&]() {
        if (vc) C.tau = div_rn(T(S.eta / S.omega), P.col_norm[j]);
        if (vr) {
            Q.sigma = div_rn(T(S.eta * S.omega), P.row_norm[i]);
            Q.rsigma = div_rn(T(1), Q.sigma);
            // an equality row's clamp gives its bound whatever v / sigma is, unless
            // that can be 0 / 0 or inf / inf
            Q.fixed = !MX && Q.b0 == Q.b1 && Q.rsigma > T(0) && Q.rsigma < T(INFINITY);
        }
    };
    set_steps();
    // whole warps without a line of one kind skip that phase
    const bool wc = (tid & ~31) / Gc < nc, wr = (tid & ~31) / Gr < nr;
    if (!CL) {
        if (own_c) {
            st_tagged(tx + 2LL * j, T(0), Tag(0));
            st_tagged(tx + 2LL * j + 1, T(0), Tag(0));
            st_tagged(A.ax + j, 0.0, Tag(0));
        }
        if (own_r) {
            st_tagged(ty + 2LL * i, Q.y, Tag(0));
            st_tagged(A.ay + i, 0.0, Tag(0));
        }
        if (tid < 16) st_tagged(A.tp + tid * kPersistMaxBlocks + b, 0.0, Tag(0));
        if (tid < 16)
            st_tagged(A.tp + (16 + (tid & 8)) * kPersistMaxBlocks + b * 8 + (tid & 7), 0.0, Tag(0));
    }
    BlockBarrier<CL> bar{A.counter, 0u, A.limits.barrier, nb == 1};
    // an entry of a gathered vector to every block's copy, the group's lanes
    // sharing the blocks
    auto spread = [&](T* buf, int at_, T v, int sub, int G) {
        if (nb == 1) {
            if (sub == 0) buf[at_] = v;
            return;
        }
        for (int q = sub; q < nb; q += G) *cg::this_cluster().map_shared_rank(buf + at_, q) = v;
    };
    // sums[q] of the per-thread values v[q] over all blocks (max for q < NMAX)
    auto reduce_all = [&](auto& v, auto count_, auto nmax_) -> bool {
        constexpr int COUNT = decltype(count_)::value, NMAX = decltype(nmax_)::value;
#pragma unroll
        for (int q = 0; q < COUNT; ++q) {
            const double t = warp_fold(v[q], q < NMAX);
            if (lane == 0) red[q][warp] = t;
        }
        if constexpr (CL) {
            __syncthreads();
            for (int q = warp; q < COUNT; q += W) {
                const double t = warp_fold(lane < W ? red[q][lane] : 0.0, q < NMAX);
                if (nb == 1) {
                    if (lane == 0) sums[q] = t;
                } else if (lane < nb) {
                    *cg::this_cluster().map_shared_rank(&parts[q][b], lane) = t;
                }
            }
            bar.sync();
            if (nb > 1)
                for (int q = warp; q < COUNT; q += W) {
                    const double t = warp_fold(lane < nb ? parts[q][lane] : 0.0, q < NMAX);
                    if (lane == 0) sums[q] = t;
                }
        } else {
            // tagged with the reduction's number, two sets in turn: a block
            // reuses a set only after every block has read it (they all have
            // contributed to the reduction in between)
            ++rnum;
            // A block in which a wait has run out says so with its partials, and
            // block 0 with the sums: no block goes on with what it computed
            // from entries that had not come.
            bad = __syncthreads_or(bad);
            const Tag mark = bad ? rnum | kFailed : rnum;
            Tagged<double>* set = A.tp + (size_t)(rnum & 1) * 8 * kPersistMaxBlocks;
            for (int q = warp; q < COUNT; q += W) {
                const double t = warp_fold(lane < W ? red[q][lane] : 0.0, q < NMAX);
                if (lane == 0) st_tagged(set + q * kPersistMaxBlocks + b, t, mark);
            }
            // Block 0 adds them up and puts the sums in front of every block,
            // a 128-byte line each: lines polled by many blocks at once keep
            // their writer waiting (30,000 cycles for 8 sums on one line).
            Tagged<double>* result = A.tp + 16 * kPersistMaxBlocks + (size_t)(rnum & 1) * 8 * kPersistMaxBlocks;
            for (int q = warp; q < COUNT; q += W) {
                double t = 0.0;
                if (b == 0) {
                    constexpr int N = kPersistMaxBlocks / 32;
                    double o[N];
                    int r_[N];
#pragma unroll
                    for (int r = 0; r < N; ++r) r_[r] = min(r * 32 + lane, nb - 1);
                    FromTagged<double, 1, true>{set + q * kPersistMaxBlocks, rnum, A.limits.entry, bad}.get(r_, o);
#pragma unroll
                    for (int r = 0; r < N; ++r)
                        if (r * 32 + lane < nb) t = q < NMAX ? maxv(t, o[r]) : t + o[r];
                    t = warp_fold(t, q < NMAX);
                    bad = __any_sync(0xffffffffu, bad);
                    for (int r = lane; r < nb; r += 32) st_tagged(result + r * 8 + q, t, bad ? rnum | kFailed : rnum);
                } else if (lane == 0) {
                    const int at_[1] = {q};
                    double o[1];
                    FromTagged<double, 1, true>{result + b * 8, rnum, A.limits.entry, bad}.get(at_, o);
                    t = o[0];
                }
                if (lane == 0) sums[q] = t;
            }
        }
        return __syncthreads_or(bad) == 0;
    };
    // y+ of the group's row from (A x-bar), stored where it is gathered
    auto dual_step = [&](T ax) {
        if (!vr) return;
        T yn;
        if (MX) {
            const T base = div_recip(add_rn(Q.yb, Q.y), Q.sigma, Q.rsigma);
            const T tl = add_rn(Q.b0, ax), th = add_rn(Q.b1, ax);
            if (add_rn(base, tl) < T(0)) yn = add_rn(Q.y, mul_rn(Q.sigma, tl));
            else if (add_rn(base, th) > T(0)) yn = add_rn(Q.y, mul_rn(Q.sigma, th));
            else yn = -Q.yb;
        } else {
            const T v = add_rn(Q.y, mul_rn(Q.sigma, ax));
            const T cl = Q.fixed ? Q.b0 : clampv(div_recip(v, Q.sigma, Q.rsigma), Q.b0, Q.b1);
            yn = sub_rn(v, mul_rn(Q.sigma, cl));
        }
        Q.y = yn;
        if (CL) spread(ybuf, i, yn, sub_r, Gr);
        else if (sub_r == 0) st_tagged(ty + 2LL * i, yn, now);
    };

    if (!bar.sync()) {
        if (tid == 0) atomicExch(&P.st->fault, 1);
        return;
    }
    bool ok = true;
    const int passes = A.chunks + ((A.rem > 0 || A.final_pass) ? 1 : 0);
    for (int pass = 0; pass < passes && ok; ++pass) {
        const bool last = pass == A.chunks;  // the partial chunk and the final evaluation
        const int span = last ? A.rem : A.R;
        const int skip = pass == 0 ? A.skip : 0;
        int phase10 = (int)((S.iter + skip) % 10);
        long long count = S.avg_count + skip;
        const int steps = span - skip;
        for (int k = 0; k < steps; ++k) {
            const bool step_it = A.ctl.adaptive_step && phase10 == 0;
            phase10 = phase10 == 9 ? 0 : phase10 + 1;
            const T cnt = T((double)(++count));
            if ((k & 63) == 0) {  // 1 / cnt of the next 64 iterations
                __syncthreads();
                if (tid < 64) rcnts[tid] = div_rn(T(1), T((double)(count + tid)));
                __syncthreads();
            }
            const T rcnt = rcnts[k & 63];
            double v2[2] = {0.0, 0.0};
            ++now;
            if (stage_y) stage(ybuf + (now & 1) * P.m, ty, P.m, now - 1);
            if (wc) {  // primal step (k_primal)
                T aty = T(0);
                if (vc && stage_y) {
                    FromShared<T> Y{ybuf + (now & 1) * P.m};
                    aty = cs_sh ? slice_dot(ri_s, cv_s, Y, C.b, C.e, Gc, sub_c)
                                : slice_dot(ri_g, cv_g, Y, C.b, C.e, Gc, sub_c);
                } else if (vc) {
                    auto Y = from(ybuf, ty, now - 1);
                    aty = cs_sh ? slice_dot(ri_s, cv_s, Y, C.b, C.e, Gc, sub_c)
                                : slice_dot(ri_g, cv_g, Y, C.b, C.e, Gc, sub_c);
                }
                aty = group_sum_n(aty, Gc);
                const T xp = clampv(sub_rn(C.x, mul_rn(C.tau, add_rn(C.c, aty))), C.lo, C.hi);
                const T d = sub_rn(xp, C.x);
                const T xb = sub_rn(mul_rn(T(2), xp), C.x);
                C.x = xp;
                if (CL) {
                    if (vc) spread(xbuf, j, xb, sub_c, Gc);
                    if (vc && step_it) spread(dbuf, j, d, sub_c, Gc);
                } else if (own_c) {
                    st_tagged(tx + 2LL * j, xb, now);
                    if (step_it) st_tagged(tx + 2LL * j + 1, d, now);
                }
                if (CL) bar.arrive();
                C.xa = add_rn(C.xa, div_recip(sub_rn(xp, C.xa), cnt, rcnt));
                if (step_it && own_c) v2[0] = __dmul_rn(__dmul_rn((double)P.col_norm[j], (double)d), (double)d);
            } else if (CL) {
                bar.arrive();
            }
            if (CL) bar.wait();
            if (!step_it) {  // dual step (k_dual, k_dual_mx)
                if (wr) {
                    T ax = T(0);
                    if (vr) {
                        auto X = from(xbuf, tx, now);
                        ax = rs_sh ? slice_dot(ci_s, rv_s, X, Q.b, Q.e, Gr, sub_r)
                                   : slice_dot(ci_g, rv_g, X, Q.b, Q.e, Gr, sub_r);
                    }
                    dual_step(group_sum_n(ax, Gr));
                }
            } else {  // k_dual_probe, k_step_size, k_dual_apply
                T ax = T(0);
                for (int l0 = 0; l0 < nr; l0 += nt / Gp) {
                    const int l = l0 + tid / Gp;
                    T av = T(0), aw = T(0);
                    if (l < nr) {
                        const int bb = P.csr_start[r0 + l] - pr, ee = P.csr_start[r0 + l + 1] - pr;
                        auto XD = pairs();
                        if (rs_sh) slice_dot2(ci_s, rv_s, XD, bb, ee, Gp, sub_p, av, aw);
                        else slice_dot2(ci_g, rv_g, XD, bb, ee, Gp, sub_p, av, aw);
                    }
                    av = group_sum_n(av, Gp);
                    aw = group_sum_n(aw, Gp);
                    if (l < nr && sub_p == 0) {
                        P.ax_bar[r0 + l] = av;
                        const double a = (double)aw;
                        v2[1] += __ddiv_rn(__dmul_rn(a, a), (double)P.row_norm[r0 + l]);
                    }
                }
                ok = reduce_all(v2, std::integral_constant<int, 2>(), std::integral_constant<int, 0>());
                if (!ok) break;
                const double eta = S.eta;
                __syncthreads();
                if (tid == 0) S.eta = next_eta(eta, sums[0], sums[1]);
                __syncthreads();
                if (S.eta != eta) set_steps();
                if (vr) ax = P.ax_bar[i];  // this block's write, before the barrier
                dual_step(ax);
            }
            if (CL) bar.arrive();
            if (wr) Q.ya = add_rn(Q.ya, div_recip(sub_rn(Q.y, Q.ya), cnt, rcnt));
            if (CL) bar.wait();
        }
        if (!ok) break;
        if (last && !A.final_pass) {  // no check, and so no reduction that tells of a wait that ran out
            if (!CL) ok = __syncthreads_or(bad) == 0;
            break;
        }
        // ---- the KKT check on the averages (k_residual_rows/cols[_mx], k_finalize)
        // the averages (base plus averaged correction in the mixed form) in
        // FP64, gathered by the block's lines
        const double xh = MX && vc ? M.x_hat[j] : 0.0, yh = MX && vr ? M.y_hat[i] : 0.0;
        const double xv = MX ? xh + (double)C.xa : (double)C.xa, yv = MX ? yh + (double)Q.ya : (double)Q.ya;
        constexpr bool SH = CL && !MX;  // gathered from the shared copies
        ++now;
        if constexpr (SH) {
            if (vc) spread(xbuf, j, C.xa, sub_c, Gc);
            if (vr) spread(ybuf, i, Q.ya, sub_r, Gr);
            bar.sync();
        } else if constexpr (CL) {
            if (own_c) P.x_avg[j] = C.xa;
            if (own_r) P.y_avg[i] = Q.ya;
            bar.sync();
        } else {
            if (own_c) st_tagged(A.ax + j, xv, now);
            if (own_r) st_tagged(A.ay + i, yv, now);
        }
        auto averages = [&](T* shared, const double* base, const T* corr, const Tagged<double>* tagged) {
            if constexpr (SH) return FromShared<T>{shared};
            else if constexpr (CL) return FromBase<T>{base, corr};
            else return FromTagged<double, 1>{tagged, now, A.limits.entry, bad};
        };
        RowTerms rt;
        ColTerms ct;
        double s_row = 0.0, s_col = 0.0;
        if (vr) s_row = slice_dot_plain(rs_sh ? ci_s : ci_g, MX ? M.csr_val64 + pr : reinterpret_cast<const double*>(rs_sh ? rv_s : rv_g),
                                        averages(xbuf, M.x_hat, P.x_avg, A.ax), Q.b, Q.e, Gr, sub_r);
        s_row = group_sum_n(s_row, Gr);
        if (own_r) rt.add(A.O, i, s_row, yv);
        if (vc) s_col = slice_dot_plain(cs_sh ? ri_s : ri_g, MX ? M.csc_val64 + pc : reinterpret_cast<const double*>(cs_sh ? cv_s : cv_g),
                                        averages(ybuf, M.y_hat, P.y_avg, A.ay), C.b, C.e, Gc, sub_c);
        s_col = group_sum_n(s_col, Gc);
        if (own_c) ct.add(A.O, j, s_col, xv);
        double v8[8] = {rt.vmax, ct.vmax, rt.dsum, rt.bad, ct.dres, ct.pobj, ct.dobj, ct.bad};
        ok = reduce_all(v8, std::integral_constant<int, 8>(), std::integral_constant<int, 2>());
        if (!ok) break;
        if (tid == 0) {  // every block computes the same state
            const CheckSums q{sums[0], sums[2], sums[3], sums[1], sums[4], sums[5], sums[6], sums[7]};
            const bool restarted = apply_check(&S, q, span, last, A.O.offset, A.ctl);
            if (!last && b == 0) trace_check(A.tr, &S, restarted);
        }
        __syncthreads();
        if (S.restart_pending && !S.done) {
            if (!MX) {  // k_restart_copy
                C.x = C.xa;
                Q.y = Q.ya;
            } else {  // k_recenter_mx
                const T inf = T(__int_as_float(0x7f800000));
                if (vc) {
                    const double xn = xv;
                    if (sub_c == 0) M.x_hat[j] = xn;
                    C.x = C.xa = T(0);
                    C.c = (T)(M.c64[j] + s_col);
                    const double a = M.lo64[j], h = M.hi64[j];
                    C.lo = (a <= -1e299) ? -inf : (T)(a - xn);
                    C.hi = (h >= 1e299) ? inf : (T)(h - xn);
                }
                if (vr) {
                    const double yn = yv;
                    if (sub_r == 0) M.y_hat[i] = yn;
                    Q.y = Q.ya = T(0);
                    Q.yb = (T)yn;
                    const double a = M.blo64[i], h = M.bhi64[i];
                    Q.b0 = (a <= -1e299) ? inf : (T)(s_row - a);
                    Q.b1 = (h >= 1e299) ? -inf : (T)(s_row - h);
                }
            }
            set_steps();
        }
        if (CL) {
            if (vr) spread(ybuf, i, Q.y, sub_r, Gr);
            bar.sync();
        } else if (own_r) {
            st_tagged(ty + 2LL * i, Q.y, now);  // the next iteration waits for the check's number
        }
        if (S.done) break;
    }
    if (!ok) {
        if (tid == 0) atomicExch(&P.st->fault, 1);
        return;
    }
    // ---- the state of the next launch and of the output stage
    if (own_c) {
        P.x[j] = C.x;
        P.x_avg[j] = C.xa;
        if (MX) {
            M.g[j] = (float)C.c;
            M.lo[j] = (float)C.lo;
            M.hi[j] = (float)C.hi;
        }
    }
    if (own_r) {
        P.y[i] = Q.y;
        P.y_avg[i] = Q.ya;
        if (MX) {
            M.yb[i] = (float)Q.yb;
            M.r_lo[i] = (float)Q.b0;
            M.r_hi[i] = (float)Q.b1;
        }
    }
    if (b == 0) {  // all but the fault, which a block sets by itself
        constexpr int words = sizeof(DevState) / sizeof(int), skip = offsetof(DevState, fault) / sizeof(int);
        for (int q = tid; q < words; q += nt)
            if (q != skip) reinterpret_cast<int*>(P.st)[q] = reinterpret_cast<const int*>(&S)[q];
    }
}

}  // namespace mc

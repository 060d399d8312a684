// One-time kernels of a solve: input validation, CSC -> CSR transpose,
// Ruiz equilibration, L1 norms and the initial iterate.  All run in FP64;
// none is on the per-iteration path.
#pragma once

#include "common.cuh"

namespace mc {

template <class T>
__global__ void k_fill(T* __restrict__ a, long long n, T v) {
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
         i += (long long)gridDim.x * blockDim.x)
        a[i] = v;
}

// longest row (for the long-row sort path) and longest column
__global__ void k_max_line(int m, const int* __restrict__ row_start, int n, const int* __restrict__ col_start,
                           int* __restrict__ longest) {
    int mx[2] = {0, 0};
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < m; i += gridDim.x * blockDim.x)
        mx[0] = max(mx[0], row_start[i + 1] - row_start[i]);
    for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < n; j += gridDim.x * blockDim.x)
        mx[1] = max(mx[1], col_start[j + 1] - col_start[j]);
#pragma unroll
    for (int q = 0; q < 2; ++q) {
        for (int off = 16; off > 0; off >>= 1) mx[q] = max(mx[q], __shfl_xor_sync(0xffffffffu, mx[q], off));
        if ((threadIdx.x & 31) == 0) atomicMax(longest + q, mx[q]);
    }
}

// ---------------------------------------------------------------- validation
// Flags what SparseMatrixCSC::validate rejects (src/model/model.cpp:41-66):
// bad pointers, row index out of range, rows not strictly increasing, zero or
// non-finite values.  Guarding device-resident input keeps every later gather
// in bounds.
__global__ void k_validate_csc(int m, int n, long long nnz, const int* __restrict__ col_start,
                               const int* __restrict__ row_index, const double* __restrict__ value,
                               int* __restrict__ bad) {
    const int j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= n) return;
    const int b = col_start[j], e = col_start[j + 1];
    if (j == 0 && b != 0) atomicOr(bad, 1);
    if (j == n - 1 && (long long)e != nnz) atomicOr(bad, 1);
    if (b > e || b < 0 || (long long)e > nnz) { atomicOr(bad, 1); return; }
    int prev = -1;
    for (int p = b; p < e; ++p) {
        const int r = row_index[p];
        const double v = value[p];
        if (r < 0 || r >= m) { atomicOr(bad, 2); return; }
        if (r <= prev) { atomicOr(bad, 4); return; }
        if (!isfinite(v) || v == 0.0) { atomicOr(bad, 8); return; }
        prev = r;
    }
}

// ----------------------------------------------------------------- transpose
// counts[r + 1] += 1 for every entry of row r
__global__ void k_count_rows(long long nnz, const int* __restrict__ row_index, int* __restrict__ counts) {
    for (long long p = blockIdx.x * (long long)blockDim.x + threadIdx.x; p < nnz;
         p += (long long)gridDim.x * blockDim.x)
        atomicAdd(&counts[row_index[p] + 1], 1);
}

// In-place inclusive scan of int32 in tiles of kScanTile per block; the
// tile totals go to `totals` (one per block).
constexpr int kScanThreads = 1024;
constexpr int kScanItems = 4;
constexpr int kScanTile = kScanThreads * kScanItems;

__global__ void __launch_bounds__(kScanThreads) k_scan_tiles(int* __restrict__ data, long long n, int* __restrict__ totals) {
    __shared__ int warp_sums[32];
    const long long base = (long long)blockIdx.x * kScanTile + (long long)threadIdx.x * kScanItems;
    int v[kScanItems];
    int run = 0;
#pragma unroll
    for (int q = 0; q < kScanItems; ++q) {
        const long long i = base + q;
        run += (i < n) ? data[i] : 0;
        v[q] = run;
    }
    // exclusive scan of per-thread totals across the block
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int t = run;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
        const int o = __shfl_up_sync(0xffffffffu, t, off);
        if (lane >= off) t += o;
    }
    if (lane == 31) warp_sums[warp] = t;
    __syncthreads();
    if (warp == 0) {
        int w = warp_sums[lane];
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
            const int o = __shfl_up_sync(0xffffffffu, w, off);
            if (lane >= off) w += o;
        }
        warp_sums[lane] = w;
    }
    __syncthreads();
    const int before = (t - run) + (warp > 0 ? warp_sums[warp - 1] : 0);
#pragma unroll
    for (int q = 0; q < kScanItems; ++q) {
        const long long i = base + q;
        if (i < n) data[i] = v[q] + before;
    }
    if (threadIdx.x == kScanThreads - 1) totals[blockIdx.x] = before + run;
}

// adds the scanned total of all previous tiles to every element of a tile
__global__ void k_scan_add(int* __restrict__ data, long long n, const int* __restrict__ scanned_totals) {
    if (blockIdx.x == 0) return;
    const int add = scanned_totals[blockIdx.x - 1];
    const long long base = (long long)blockIdx.x * kScanTile;
    for (int q = threadIdx.x; q < kScanTile; q += blockDim.x) {
        const long long i = base + q;
        if (i < n) data[i] += add;
    }
}

// Unordered scatter of CSC entries into their CSR rows (thread per column).
__global__ void k_scatter_rows(int n, const int* __restrict__ col_start, const int* __restrict__ row_index,
                               const double* __restrict__ value, const int* __restrict__ row_start,
                               int* __restrict__ cursor, int* __restrict__ col_index,
                               double* __restrict__ csr_value) {
    const int j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= n) return;
    for (int p = col_start[j]; p < col_start[j + 1]; ++p) {
        const int r = row_index[p];
        const int pos = row_start[r] + atomicAdd(&cursor[r], 1);
        col_index[pos] = j;
        csr_value[pos] = value[p];
    }
}

constexpr int kShortRow = 32;     // rows up to this length: sorted by a warp in registers, or by one thread
constexpr int kSmemSortRow = 4096;  // rows up to this length: shared-memory bitonic sort

// Sort short rows by column and list the long rows for the block-level sort:
// by a warp per row, or (k_sort_short_rows_thread) by a thread per row where the
// rows fill the chip's threads and are short (build_csr has the rule).
//
// A warp per row, an entry per lane: the row is read once, each entry counts
// the smaller ones by shuffles and goes to that place.  (An insertion sort by
// one thread per row is a chain of dependent loads and stores: 51 us for 1000
// rows of 18 entries, 77 us for 4001 of 27, on B200; a warp per row takes 3.9
// and 4.6, and 51 us for 200,000 rows of 20, where its loads are coalesced.)
__global__ void k_sort_short_rows(int m, const int* __restrict__ row_start, int* __restrict__ col_index,
                                  double* __restrict__ value, int* __restrict__ long_rows,
                                  int* __restrict__ long_count) {
    const long long i = (blockIdx.x * (long long)blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (i >= m) return;
    const int b = row_start[i], len = row_start[i + 1] - b;
    if (len > kShortRow) {
        if (lane == 0) long_rows[atomicAdd(long_count, 1)] = (int)i;
        return;
    }
    const bool in = lane < len;
    const int key = in ? col_index[b + lane] : 0;
    const double v = in ? value[b + lane] : 0.0;
    int place = 0;
    for (int q = 0; q < len; ++q) {
        const int other = __shfl_sync(0xffffffffu, key, q);
        place += other < key || (other == key && q < lane);
    }
    __syncwarp();  // every lane has read before any writes
    if (in) {
        col_index[b + place] = key;
        value[b + place] = v;
    }
}

// An entry moves down past the larger ones before it.
__global__ void k_sort_short_rows_thread(int m, const int* __restrict__ row_start, int* __restrict__ col_index,
                                         double* __restrict__ value, int* __restrict__ long_rows,
                                         int* __restrict__ long_count) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= m) return;
    const int b = row_start[i], e = row_start[i + 1];
    if (e - b > kShortRow) {
        long_rows[atomicAdd(long_count, 1)] = i;
        return;
    }
    for (int p = b + 1; p < e; ++p) {
        const int key = col_index[p];
        const double v = value[p];
        int q = p;
        for (; q > b && col_index[q - 1] > key; --q) {
            col_index[q] = col_index[q - 1];
            value[q] = value[q - 1];
        }
        if (q == p) continue;
        col_index[q] = key;
        value[q] = v;
    }
}

// One block per long row.  Rows up to kSmemSortRow: bitonic sort in shared
// memory.  Longer rows: each element's final slot is its rank (columns are
// distinct within a row), written to scratch and copied back.
__global__ void __launch_bounds__(1024) k_sort_long_rows(const int* __restrict__ long_rows,
                                                         const int* __restrict__ row_start,
                                                         int* __restrict__ col_index,
                                                         double* __restrict__ value,
                                                         int* __restrict__ tmp_col,
                                                         double* __restrict__ tmp_val) {
    extern __shared__ unsigned char smem_raw[];
    const int i = long_rows[blockIdx.x];
    const int b = row_start[i], e = row_start[i + 1];
    const int len = e - b;
    if (len <= kSmemSortRow) {
        int pow2 = 1;
        while (pow2 < len) pow2 <<= 1;
        int* keys = reinterpret_cast<int*>(smem_raw);
        double* vals = reinterpret_cast<double*>(smem_raw + kSmemSortRow * sizeof(int));
        for (int q = threadIdx.x; q < pow2; q += blockDim.x) {
            keys[q] = (q < len) ? col_index[b + q] : 0x7fffffff;
            vals[q] = (q < len) ? value[b + q] : 0.0;
        }
        __syncthreads();
        for (int size = 2; size <= pow2; size <<= 1) {
            for (int stride = size >> 1; stride > 0; stride >>= 1) {
                for (int q = threadIdx.x; q < pow2; q += blockDim.x) {
                    const int partner = q ^ stride;
                    if (partner > q) {
                        const bool up = (q & size) == 0;
                        const int a = keys[q], c = keys[partner];
                        if ((a > c) == up) {
                            keys[q] = c;
                            keys[partner] = a;
                            const double tv = vals[q];
                            vals[q] = vals[partner];
                            vals[partner] = tv;
                        }
                    }
                }
                __syncthreads();
            }
        }
        for (int q = threadIdx.x; q < len; q += blockDim.x) {
            col_index[b + q] = keys[q];
            value[b + q] = vals[q];
        }
    } else {
        for (int q = threadIdx.x; q < len; q += blockDim.x) {
            const int key = col_index[b + q];
            int rank = 0;
            for (int t = 0; t < len; ++t) rank += (col_index[b + t] < key) ? 1 : 0;
            tmp_col[b + rank] = key;
            tmp_val[b + rank] = value[b + q];
        }
        __syncthreads();
        for (int q = threadIdx.x; q < len; q += blockDim.x) {
            col_index[b + q] = tmp_col[b + q];
            value[b + q] = tmp_val[b + q];
        }
    }
}

// ---------------------------------------------------------------------- Ruiz
// equilibrate_model, src/scale/ruiz_scaling.cpp:167-218, all passes (up to 64)
// in one cooperative launch, for one LP or for a packed batch.  Maxima are
// exact in any order, and the rescale computes value * (delta_r[i] * delta_c[j])
// exactly as :215, so the scaled matrix equals the reference's bit for bit.
//
// A pass reads and writes both copies of the matrix once: while a line is
// rescaled by the pass' deltas its new maximum is taken and the next pass'
// delta written, so that one grid barrier separates two passes.  G lanes share
// a line as in the SpMV kernels (the gather of the other side's delta is one
// request per entry, which bounds the pass: 0.26 ms per copy at 40M nonzeros).
// Before, a pass was seven launches with a thread per line: per call 12.9 ms
// of rescales and 1.7 ms of maxima at 40M nonzeros, 350 us at 600.
// A short line is one chain start -> index -> delta -> value, so the chain is what
// a pass waits for: a line's last one to three entries go together, the next
// line's ends and delta come meanwhile, and where both sides have a thread a line
// (SHORT: fewer than 8 entries on average) the lanes are a constant and four blocks
// share an SM.  mc_ruiz_equilibrate, 10 passes, ms, seven launches a pass / the
// general form entry by entry / now: rows of 1 on average, 3M x 1M 1.84 / 2.95 / 1.77;
// rows of 0.8, 10M x 4M 5.64 / 10.0 / 5.74; seven launches / now: rows of 3, 1M x 3M
// 1.85 / 1.77; of 4, 2M x 2M 2.99 / 2.51; of 7 4.58 / 3.80; of 20, 2M x 5M 16.1 / 10.4.
// The first four in the general form of now 1.99, 6.7, 1.96 and 2.65; in windows
// of two entries at six blocks an SM 2.43, 7.7, 2.58 and 5.2.
struct RuizSide {
    const int* start;
    const int* inner;
    double* value;
    double* scale;     // product of the deltas
    double* delta[2];  // of this pass and the next, in turn
    int lanes;         // per line
    // tiles of lines of one LP each; lp == NULL: one LP, `per` lines a tile
    const int *lp, *l0, *l1;
    int ntiles, lines, per;
};

// W entries of a line from p, those before e, together: rescaled, and the
// maximum of |a|.
template <bool FIRST, int W, bool ALL>
__device__ __forceinline__ double ruiz_window(const RuizSide& S, const double* __restrict__ delta_in, double dout, int p,
                                              int e, int G, double mx) {
    double v[W];
    bool in[W];
#pragma unroll
    for (int q = 0; q < W; ++q) {
        in[q] = ALL || p + q * G < e;
        v[q] = in[q] ? ld_stream(S.value + p + q * G) : 0.0;
    }
    if (!FIRST) {
        double d[W];
#pragma unroll
        for (int q = 0; q < W; ++q) d[q] = in[q] ? __ldcg(delta_in + ld_stream(S.inner + p + q * G)) : 0.0;
#pragma unroll
        for (int q = 0; q < W; ++q) {
            v[q] = __dmul_rn(v[q], __dmul_rn(dout, d[q]));
            if (in[q]) st_stream(S.value + p + q * G, v[q]);
        }
    }
#pragma unroll
    for (int q = 0; q < W; ++q) mx = in[q] ? maxv(mx, fabs(v[q])) : mx;
    return mx;
}

// Entries [b, e) of line j: maximum of |a| after this pass' rescale.
template <bool FIRST, bool SHORT>
__device__ __forceinline__ double ruiz_line(const RuizSide& S, const double* __restrict__ delta_in, double dout, int b,
                                            int e, int sub) {
    const int G = SHORT ? 1 : S.lanes;
    double mx = 0.0;
    int p = b + sub;
    for (; p + 3 * G < e; p += 4 * G) mx = ruiz_window<FIRST, 4, true>(S, delta_in, dout, p, e, G, mx);
    if (p < e) mx = ruiz_window<FIRST, 3, false>(S, delta_in, dout, p, e, G, mx);
    if (!SHORT)
        for (int off = G >> 1; off > 0; off >>= 1) mx = maxv(mx, __shfl_xor_sync(0xffffffffu, mx, off));
    return mx;
}

// errs: [3][2][nlp] maxima of |1 - norm| (as bits: they order like the
// values), zeroed before the launch; a pass reads one set (rows, columns),
// writes the next and clears the third.
__device__ __forceinline__ bool ruiz_converged(const unsigned long long* errs, int set, int nlp, int lp, double tolerance) {
    const double r = __longlong_as_double((long long)__ldcg(errs + (size_t)(2 * set) * nlp + lp));
    const double c = __longlong_as_double((long long)__ldcg(errs + (size_t)(2 * set + 1) * nlp + lp));
    return r < tolerance && c < tolerance;
}

template <bool FIRST, bool SHORT>
__device__ __forceinline__ void ruiz_side(const RuizSide& S, const double* delta_in, int cur, unsigned long long* errs,
                                          int read_set, int write_set, int side, int nlp, double tolerance,
                                          double* scratch) {
    const int G = SHORT ? 1 : S.lanes, sub = threadIdx.x & (G - 1);
    const double* own = cur ? S.delta[1] : S.delta[0];
    double* next = (FIRST ? cur : !cur) ? S.delta[1] : S.delta[0];
    double err = 0.0;
    int lp = 0;
    auto flush = [&]() {
        err = block_reduce(err, scratch, OpMax());
        if (threadIdx.x == 0 && err > 0.0)
            atomicMax(errs + (size_t)(2 * write_set + side) * nlp + lp, (unsigned long long)__double_as_longlong(err));
        err = 0.0;
    };
    // line j with maximum mx: the next pass' delta
    auto finish = [&](int j, double mx, double dout) {
        if (mx == 0.0) mx = 1.0;
        next[j] = 1.0 / sqrt(mx);
        err = maxv(err, fabs(1.0 - mx));
        S.scale[j] = FIRST ? 1.0 : S.scale[j] * dout;
    };
    if (!S.lp) {  // one LP: the next line's ends and delta come while this line's entries do
        const int step = (int)gridDim.x * S.per;
        int j = (int)blockIdx.x * S.per + (int)threadIdx.x / G, b = 0, e = 0;
        double dout = 1.0;
        if (j < S.lines) {
            b = __ldg(S.start + j);
            e = __ldg(S.start + j + 1);
            if (!FIRST) dout = own[j];
        }
        for (int t = blockIdx.x; t < S.ntiles; t += gridDim.x) {
            const int jn = t + (int)gridDim.x < S.ntiles ? j + step : S.lines;
            int bn = 0, en = 0;
            double dn = 1.0;
            if (jn < S.lines) {
                bn = __ldg(S.start + jn);
                en = __ldg(S.start + jn + 1);
                if (!FIRST) dn = own[jn];
            }
            const double mx = ruiz_line<FIRST, SHORT>(S, delta_in, dout, b, e, sub);
            if (j < S.lines && sub == 0) finish(j, mx, dout);
            j = jn, b = bn, e = en, dout = dn;
        }
        flush();
        return;
    }
    for (int t = blockIdx.x; t < S.ntiles; t += gridDim.x) {
        const int l0 = S.l0[t], l1 = S.l1[t], tile_lp = S.lp[t];
        if (tile_lp != lp) {
            flush();
            lp = tile_lp;
        }
        if (!FIRST && ruiz_converged(errs, read_set, nlp, lp, tolerance)) continue;
        for (int base = l0; base < l1; base += kBlock / G) {
            const int j = base + threadIdx.x / G;
            const bool valid = j < l1;
            int b = 0, e = 0;
            double dout = 1.0;
            if (valid) {
                b = __ldg(S.start + j);
                e = __ldg(S.start + j + 1);
                if (!FIRST) dout = own[j];
            }
            const double mx = ruiz_line<FIRST, SHORT>(S, delta_in, dout, b, e, sub);
            if (valid && sub == 0) finish(j, mx, dout);
        }
    }
    flush();
}

// Passes [pass0, pass1); pass 0 begins with the maxima of the matrix as given.
// counter[1] is set when there is nothing left to do after them.
template <bool SHORT>
__global__ void __launch_bounds__(kBlock, SHORT ? 4 : 3)
    k_ruiz(RuizSide C, RuizSide R, long long pass0, long long pass1, double tolerance, int nlp,
           unsigned long long* errs, unsigned* counter, unsigned limit, DevState* st) {
    __shared__ double scratch[32];
    BlockBarrier<false> bar{counter, 0u, limit, false};
    if (pass0 == 0) {
        ruiz_side<true, SHORT>(C, nullptr, 0, errs, 0, 0, 1, nlp, tolerance, scratch);
        ruiz_side<true, SHORT>(R, nullptr, 0, errs, 0, 0, 0, nlp, tolerance, scratch);
    }
    int set = (int)(pass0 % 3);
    for (long long pass = pass0; pass < pass1; ++pass, set = set == 2 ? 0 : set + 1) {
        if (!bar.sync()) {
            if (threadIdx.x == 0) {
                atomicExch(&st->fault, 1);
                atomicExch(counter + 1, 1u);
            }
            return;
        }
        // convergence test (:185-197); a converged LP's later passes are no-ops
        const int write_set = set == 2 ? 0 : set + 1, clear_set = write_set == 2 ? 0 : write_set + 1;
        int all = 1;
        for (int lp = threadIdx.x; lp < nlp; lp += kBlock) {
            const bool done = ruiz_converged(errs, set, nlp, lp, tolerance);
            all &= done;
            if (blockIdx.x == 0) {
                if (done) st[lp].ruiz_done = 1;
                else st[lp].ruiz_passes += 1;
                errs[(size_t)(2 * clear_set) * nlp + lp] = 0ull;
                errs[(size_t)(2 * clear_set + 1) * nlp + lp] = 0ull;
            }
        }
        if (__syncthreads_and(all)) {
            if (blockIdx.x == 0 && threadIdx.x == 0) counter[1] = 1u;
            return;
        }
        const int cur = (int)(pass & 1);
        ruiz_side<false, SHORT>(C, cur ? R.delta[1] : R.delta[0], cur, errs, set, write_set, 1, nlp, tolerance, scratch);
        ruiz_side<false, SHORT>(R, cur ? C.delta[1] : C.delta[0], cur, errs, set, write_set, 0, nlp, tolerance, scratch);
    }
}

// ------------------------------------------------------------ problem setup
// Column data (:153-159, :168-176, :186-191 and the Ruiz bound/objective
// scaling :238-244).  Writes the scaled c, bounds (sentinel form), the
// original bounds (sentinel form), L1 column norms, the starting x.
// Partials: SLOT_A max|c|, SLOT_B max|c_orig| (residual scale).
__global__ void k_setup_cols(int n, const int* __restrict__ col_start, const double* __restrict__ value,
                             const double* __restrict__ obj_in, const double* __restrict__ lo_in,
                             const double* __restrict__ hi_in, const double* __restrict__ col_scale,
                             const double* __restrict__ warm_x, double obj_sign,
                             double* __restrict__ c, double* __restrict__ lo, double* __restrict__ hi,
                             double* __restrict__ c_orig, double* __restrict__ lo_orig,
                             double* __restrict__ hi_orig, double* __restrict__ col_norm,
                             double* __restrict__ x, double* __restrict__ x_avg,
                             double* __restrict__ partials) {
    __shared__ double scratch[32];
    double cmax = 0.0, comax = 0.0;
    for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < n; j += gridDim.x * blockDim.x) {
        const double s = col_scale[j];
        const double inv = 1.0 / s;
        const double l0 = lo_in[j], h0 = hi_in[j];
        const double ls = isfinite(l0) ? __dmul_rn(l0, inv) : l0;
        const double hs = isfinite(h0) ? __dmul_rn(h0, inv) : h0;
        const double lsent = isinf(ls) ? -kBig : ls;
        const double hsent = isinf(hs) ? kBig : hs;
        lo[j] = lsent;
        hi[j] = hsent;
        lo_orig[j] = isinf(l0) ? -kBig : l0;
        hi_orig[j] = isinf(h0) ? kBig : h0;
        const double cj = obj_sign * __dmul_rn(obj_in[j], s);
        c[j] = cj;
        cmax = maxv(cmax, fabs(cj));
        const double co = obj_sign * obj_in[j];
        c_orig[j] = co;
        comax = maxv(comax, fabs(co));
        double nrm = 0.0;
        for (int p = col_start[j]; p < col_start[j + 1]; ++p) nrm += fabs(value[p]);
        col_norm[j] = (nrm < 1e-12) ? 1.0 : nrm;
        const double start = warm_x ? __dmul_rn(warm_x[j], inv) : 0.0;
        const double x0 = clampv(start, lsent, hsent);
        x[j] = x0;
        x_avg[j] = x0;
    }
    cmax = block_reduce(cmax, scratch, OpMax());
    if (threadIdx.x == 0) partials[SLOT_A * kMaxPartials + blockIdx.x] = cmax;
    comax = block_reduce(comax, scratch, OpMax());
    if (threadIdx.x == 0) partials[SLOT_B * kMaxPartials + blockIdx.x] = comax;
}

// Row data (:160-167, :168-176, Ruiz row-bound scaling :229-236).
// Partial SLOT_C: max finite |b|.
__global__ void k_setup_rows(int m, const int* __restrict__ row_start, const double* __restrict__ value,
                             const double* __restrict__ rlo_in, const double* __restrict__ rhi_in,
                             const double* __restrict__ row_scale, const double* __restrict__ warm_y,
                             double* __restrict__ blo, double* __restrict__ bhi,
                             double* __restrict__ blo_orig, double* __restrict__ bhi_orig,
                             double* __restrict__ row_norm, double* __restrict__ y,
                             double* __restrict__ y_avg, double* __restrict__ partials) {
    __shared__ double scratch[32];
    double bmax = 0.0;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < m; i += gridDim.x * blockDim.x) {
        const double s = row_scale[i];
        const double l0 = rlo_in[i], h0 = rhi_in[i];
        const double ls = isfinite(l0) ? __dmul_rn(l0, s) : l0;
        const double hs = isfinite(h0) ? __dmul_rn(h0, s) : h0;
        const double lsent = isinf(ls) ? -kBig : ls;
        const double hsent = isinf(hs) ? kBig : hs;
        blo[i] = lsent;
        bhi[i] = hsent;
        blo_orig[i] = isinf(l0) ? -kBig : l0;
        bhi_orig[i] = isinf(h0) ? kBig : h0;
        if (fabs(lsent) < 1e299) bmax = maxv(bmax, fabs(lsent));
        if (fabs(hsent) < 1e299) bmax = maxv(bmax, fabs(hsent));
        double nrm = 0.0;
        for (int p = row_start[i]; p < row_start[i + 1]; ++p) nrm += fabs(value[p]);
        row_norm[i] = (nrm < 1e-12) ? 1.0 : nrm;
        const double y0 = warm_y ? __dmul_rn(warm_y[i], 1.0 / s) : 0.0;
        y[i] = y0;
        y_avg[i] = y0;
    }
    bmax = block_reduce(bmax, scratch, OpMax());
    if (threadIdx.x == 0) partials[SLOT_C * kMaxPartials + blockIdx.x] = bmax;
}

// Scalars (:155-159, :165-166, :177-179) and counters (:192-193).
__global__ void k_setup_scalars(const double* __restrict__ partials, int ncol_parts, int nrow_parts,
                                double initial_primal_weight, double step_size_reduction,
                                DevState* __restrict__ st) {
    __shared__ double scratch[32];
    const double cmax = reduce_partials(partials + SLOT_A * kMaxPartials, ncol_parts, scratch, OpMax());
    const double comax = reduce_partials(partials + SLOT_B * kMaxPartials, ncol_parts, scratch, OpMax());
    const double bmax = reduce_partials(partials + SLOT_C * kMaxPartials, nrow_parts, scratch, OpMax());
    if (threadIdx.x == 0) {
        const double c_norm = maxv(1.0, cmax);
        const double b_norm = maxv(1.0, bmax);
        st->c_norm_inf = c_norm;
        st->b_norm_inf = b_norm;
        st->c_scale = maxv(1.0, comax);
        st->omega = (initial_primal_weight > 0.0) ? initial_primal_weight
                                                  : clampv(sqrt(c_norm / b_norm), 0.01, 100.0);
        st->eta = clampv(step_size_reduction, 0.1, 0.99);
        st->last_restart_score = 1e300;
        st->primal_infeas = st->dual_infeas = st->gap = 1e300;
        st->iter = 0;
        st->avg_count = 0;
        st->iters_since_restart = 0;
        st->restarts = 0;
        st->checks = 0;
        st->done = 0;
        st->status = 1;  // iteration_limit until proven otherwise
        st->restart_pending = 0;
        st->nonfinite = 0;
    }
}

// Unscaled averages out (pdlp.cpp:76-79): x = x_avg * D_C, y = y_avg * D_R.
__global__ void k_unscale_out(int n, int m, const double* __restrict__ x_avg, const double* __restrict__ y_avg,
                              const double* __restrict__ col_scale, const double* __restrict__ row_scale,
                              double* __restrict__ x_out, double* __restrict__ y_out) {
    for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < n + m; t += gridDim.x * blockDim.x) {
        if (t < n) {
            if (x_out) x_out[t] = __dmul_rn(x_avg[t], col_scale[t]);
        } else {
            const int i = t - n;
            if (y_out) y_out[i] = __dmul_rn(y_avg[i], row_scale[i]);
        }
    }
}

}  // namespace mc

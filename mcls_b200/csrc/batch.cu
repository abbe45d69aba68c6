// batch.cu -- many systems and many right-hand sides in one MCSA loop.
//
// m systems A_s (uneven sizes) with R_s right-hand sides each are solved
// together: the block-diagonal operator S = diag(A_1..A_m) carries one
// point-Jacobi domain H = I - D^-1 S (walks never leave a block).  System s
// gets W_s = R_s rounded up to a power of two columns; the systems are
// grouped by W_s into five width classes (1, 2, 4, 8, 16 columns), each a
// contiguous range of rows whose vectors are row-major [rows][W] blocks of
// the element arrays (BatchClasses), so a system with one right-hand side
// costs one column, not the widest system's sixteen.  Forward walks do not
// depend on the source, so one set of histories per iteration serves every
// right-hand side of every system: each history carries one tally per column
// of its row's class (walk32_batch).  Every (system, rhs) pair has its own
// convergence test |rp_{s,r}|_2 <= tol |D^-1 b_{s,r}|_2 (the
// MCSASolverManager criterion, src/MCLS_MCSASolverManager_impl.hpp:299-318);
// a system whose pairs have all met it stops (its rows and walks are
// skipped), and the loop ends when every pair has met it or at the iteration
// limit.  One iteration is four kernels in a CUDA graph whose WHILE node the
// last one controls: the residual at the smoothed iterate, the tally source,
// the shared walk -- which adds the correction to it (with several histories
// per row, a pass of its own does) -- and residual + per-pair norms + the next
// smoothed iterate, whose last block to finish runs the convergence test.
//
// The passes over the elements take them in units: one row by two
// consecutive columns per thread (one 16-byte access), the entries from rows of
// fixed width.  What bounds them is the chain of dependent loads: with one
// column per thread and the CSR row walked entry by entry (row bounds, column,
// value) they ran at a third of the HBM rate (128 systems, 5M elements: 109, 57
// and 164 us).  Fixed rows need no bounds, the gathers of a row are in flight
// together, and the next tile's column indices are loaded meanwhile, which
// leaves one memory latency per tile.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <numeric>
#include <type_traits>
#include <vector>

#include "internal.h"

namespace mclsgpu {
namespace {

struct BatchState {
    int iter;
    int done;
    int max_iters;
    int check_freq;
    double tol;
    int converged;  // pairs converged
    int pairs;      // pairs in the batch
};

constexpr int kThreads = 256;
constexpr int kRowBlocks = 3;  // blocks per SM of the row passes (their registers)

// Rows for the element passes: the first 8 entries at a fixed width, entry-major
// (entry k of row i at k * n + i, columns ascending; padding entries repeat the
// row's own index with value 0), the others from the CSR rows they came from.
// Only systems with longer rows look for those, so neither the time nor the
// memory of a system depends on the rows of another.  10 iterations on 64
// systems: 1,545 us on 5- and 7-point ones, 1,733 with a 9-point one among them
// and 1,952 on 9-point ones; at the width of the longest row of all, read entry
// by entry past the eighth, 3,348 and 3,385.
constexpr int kRowChunk = 8;
struct BatchRows {
    int n = 0;
    int* col = nullptr;
    double* val = nullptr;
    const int* rp = nullptr;
    const int* ci = nullptr;
    const double* v = nullptr;
};

struct BatchArgs {
    int nsys;
    int pw;              // per-pair row width: pair (s, r) is s * pw + r
    int per;             // histories per row
    BatchRows S;         // the operator
    const double* dinv;  // D^-1
    BatchRows H;         // H rows (forward domain, FP64)
    // Per system: first row, first element, log2 of its width, rows.
    const int* srow0;
    const long long* seoff;
    const int* slog;
    const int* slong;    // some row has more than kRowChunk entries
    const int* sn;
    const int* sorder;   // the systems in placement order
    // The systems this launch works on: lsys[k] for k < *lcount, their tiles of
    // kThreads units at [ltcum[k], ltcum[k+1]) of the launch's tiles.
    const int* lsys;
    const int* ltcum;
    const int* lcount;
    // The active list the convergence test rebuilds (the iteration's list).
    int* act_sys;
    int* act_tcum;
    int* act_hcum;
    int* act_count;
    const double* B;
    double* X;
    double* X2;          // smoothed iterate x + w rp
    double* RP2;
    double* Y;
    float* cR;
    double* norm2;       // [nsys][pw]
    double* bnorm2;
    int* conv_iter;      // [nsys][pw]
    const int* nrhs;
    int* sys_done;       // per system: every right-hand side converged
    BatchState* st;
    unsigned* blocks_done;
    double omega;        // Richardson relaxation
    double nomega;       // Neumann relaxation (1 when absent)
    double inv_per;      // 1 / histories per state
    int ev;              // expected-value estimator
    unsigned long long* d_epoch;
    unsigned long long* d_tim;
    int* status;
};

// Columns of a unit of width class c, and the units of a row.
__host__ __device__ constexpr int unit_cols(int c) { return c >= 1 ? 2 : 1; }
__host__ __device__ constexpr int unit_log(int c) { return c >= 1 ? c - 1 : 0; }

// Tiles of a system: kThreads units each, the last one partial.
__host__ __device__ constexpr long long system_tiles(int n, int c) {
    return (((long long)n << unit_log(c)) + kThreads - 1) / kThreads;
}

// One thread's unit: its system s with log2 width c, first row row0 and first
// element eoff; its row (in the operator: i, in the system: rl) and the index
// of its first column inside the system's elements.
struct Unit {
    int s, c, row0, i, g;
    int tail;          // the system's rows may go on past kRowChunk entries
    unsigned col0;     // g * unit_cols(c)
    long long eoff;
    __device__ __forceinline__ size_t elem() const {
        return size_t(eoff) + ((size_t(i - row0) << c) + col0);
    }
};

// The list entry k with ltcum[k] <= t < ltcum[k+1] (count >= 1 entries).
__device__ __forceinline__ int tile_entry(const int* ltcum, int count, int t) {
    int lo = 0, hi = count - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (ltcum[mid] <= t) lo = mid; else hi = mid - 1;
    }
    return lo;
}

// Loop over the launch's tiles: each block takes one contiguous range.  A tile
// lies in one system, so the system's fields are uniform in the block and
// reloaded only when it moves on to the next.  body(live, q, next) runs on every
// thread of the block for every tile, enter(q, live, row) before the first tile
// of each system (so both may use warp collectives); next: the thread's row in
// the next tile if that has one in the same system, else -1.
template <class Enter, class Body>
__device__ __forceinline__ void for_tiles(const BatchArgs& a, Enter enter, Body body) {
    __shared__ int s_k0;
    const int count = *a.lcount;
    const int total = count > 0 ? a.ltcum[count] : 0;
    const int span = (total + int(gridDim.x) - 1) / int(gridDim.x);
    const int beg = blockIdx.x * span;
    const int end = min(beg + span, total);
    if (beg >= end) return;  // the whole block
    if (threadIdx.x == 0) s_k0 = tile_entry(a.ltcum, count, beg);
    __syncthreads();
    int k = s_k0 - 1, lo = 0, hi = -1, units = 0;
    Unit q;
#pragma unroll 1
    for (int t = beg; t < end; ++t) {
        if (t >= hi) {
            ++k;
            q.s = a.lsys[k];
            q.c = a.slog[q.s];
            q.tail = a.slong[q.s];
            q.row0 = a.srow0[q.s];
            q.eoff = a.seoff[q.s];
            units = a.sn[q.s] << unit_log(q.c);
            lo = a.ltcum[k];
            hi = a.ltcum[k + 1];
            q.g = threadIdx.x & ((1 << unit_log(q.c)) - 1);
            q.col0 = unsigned(q.g * unit_cols(q.c));
            const int u0 = (t - lo) * kThreads + threadIdx.x;
            enter(q, u0 < units, q.row0 + (u0 >> unit_log(q.c)));
        }
        const int u = (t - lo) * kThreads + threadIdx.x, un = u + kThreads;
        q.i = q.row0 + (u >> unit_log(q.c));
        body(u < units, q, t + 1 < hi && un < units ? q.row0 + (un >> unit_log(q.c)) : -1);
    }
}
struct NoEnter {
    __device__ __forceinline__ void operator()(const Unit&, bool, int) const {}
};

// N consecutive doubles (one access of 8 or 16 bytes; the element arrays are
// aligned to 128 bytes and a unit to its own size).
template <int N>
struct Cols {
    double v[N];
};
template <int N>
__device__ __forceinline__ Cols<N> ldn(const double* p) {
    Cols<N> r;
    if constexpr (N == 2) {
        const double2 t = *reinterpret_cast<const double2*>(p);
        r.v[0] = t.x;
        r.v[1] = t.y;
    } else
        r.v[0] = *p;
    return r;
}
template <int N>
__device__ __forceinline__ void stn(double* p, const Cols<N>& r) {
    if constexpr (N == 2)
        *reinterpret_cast<double2*>(p) = make_double2(r.v[0], r.v[1]);
    else
        *p = r.v[0];
}

// f(integral_constant<int, columns>) for the unit's class.
template <class F>
__device__ __forceinline__ void with_cols(int c, F f) {
    if (c >= 1) f(std::integral_constant<int, 2>{});
    else f(std::integral_constant<int, 1>{});
}

// The column indices of the first chunk of a thread's row, loaded one tile
// ahead (the body of a tile starts the next tile's loads after its gathers).
struct Ahead {
    int col[kRowChunk];
    __device__ __forceinline__ void load(const BatchRows& M, int i) {
#pragma unroll
        for (int m = 0; m < kRowChunk; ++m) col[m] = M.col[size_t(m) * M.n + i];
    }
};

// Entries past the fixed width that are loaded at a time.
constexpr int kTail = 4;

// The unit's row of M times the columns of x, entries in ascending column
// order; `next`: the row whose indices to load into h meanwhile (or -1).  TAIL:
// some system has rows that go on past the fixed width (in batches without one the
// look for them costs 3 %).
template <int N, bool TAIL>
__device__ __forceinline__ Cols<N> row_times(const BatchRows& M, const Unit& q, const double* x,
                                             Ahead& h, int next) {
    const double* xs = x + q.eoff + q.col0;
    Cols<N> acc;
#pragma unroll
    for (int n = 0; n < N; ++n) acc.v[n] = 0.0;
    int p = 0, end = 0;
    if (TAIL && q.tail) {
        p = M.rp[q.i] + kRowChunk;
        end = M.rp[q.i + 1];
    }
    Cols<N> xv[kRowChunk];
    double val[kRowChunk];
#pragma unroll
    for (int m = 0; m < kRowChunk; ++m) {
        xv[m] = ldn<N>(xs + (size_t(unsigned(h.col[m] - q.row0)) << q.c));
        val[m] = M.val[size_t(m) * M.n + q.i];
    }
    if (next >= 0) h.load(M, next);
#pragma unroll
    for (int m = 0; m < kRowChunk; ++m) {
#pragma unroll
        for (int n = 0; n < N; ++n) acc.v[n] = fma(val[m], xv[m].v[n], acc.v[n]);
    }
#pragma unroll 1
    for (; TAIL && p < end; p += kTail) {
        int col[kTail];
        double v[kTail];
#pragma unroll
        for (int t = 0; t < kTail; ++t) {  // past the end: the last entry again, not added
            const int at = min(p + t, end - 1);
            col[t] = M.ci[at];
            v[t] = M.v[at];
        }
        Cols<N> xk[kTail];
#pragma unroll
        for (int t = 0; t < kTail; ++t)
            xk[t] = ldn<N>(xs + (size_t(unsigned(col[t] - q.row0)) << q.c));
#pragma unroll
        for (int t = 0; t < kTail; ++t)
            if (p + t < end) {
#pragma unroll
                for (int n = 0; n < N; ++n) acc.v[n] = fma(v[t], xk[t].v[n], acc.v[n]);
            }
    }
    return acc;
}

// rp2 = D^-1 (b - S x2) at the smoothed iterate x2 = x + w rp (RichardsonIteration::
// doOneIteration then updatePrecResidual, src/MCLS_RichardsonIteration_impl.hpp:
// 134-147); Y (not null: the walk adds into it) is cleared for this
// iteration's walk.
template <bool TAIL>
__global__ void __launch_bounds__(kThreads, kRowBlocks) k_b_smoothed_residual(BatchArgs a) {
    Ahead h;
    auto enter = [&](const Unit&, bool live, int i) {
        if (live) h.load(a.S, i);
    };
    for_tiles(a, enter, [&](bool live, const Unit& q, int next) {
        if (!live) return;
        const size_t e = q.elem();
        with_cols(q.c, [&](auto nt) {
            constexpr int N = decltype(nt)::value;
            const Cols<N> bv = ldn<N>(a.B + e);
            const double di = a.dinv[q.i];
            Cols<N> t = row_times<N, TAIL>(a.S, q, a.X2, h, next);
#pragma unroll
            for (int n = 0; n < N; ++n) t.v[n] = di * (bv.v[n] - t.v[n]);
            stn<N>(a.RP2 + e, t);
            if (a.Y) {
#pragma unroll
                for (int n = 0; n < N; ++n) t.v[n] = 0.0;
                stn<N>(a.Y + e, t);
            }
        });
    });
}

// Tally source of every right-hand side: expected value c = H (w rp2),
// collision c = w rp2 (FP32).
template <bool TAIL>
__global__ void __launch_bounds__(kThreads, kRowBlocks) k_b_source(BatchArgs a) {
    Ahead h;
    auto enter = [&](const Unit&, bool live, int i) {
        if (live && a.ev) h.load(a.H, i);
    };
    for_tiles(a, enter, [&](bool live, const Unit& q, int next) {
        if (!live) return;
        const size_t e = q.elem();
        with_cols(q.c, [&](auto nt) {
            constexpr int N = decltype(nt)::value;
            const Cols<N> t = a.ev ? row_times<N, TAIL>(a.H, q, a.RP2, h, next)
                                   : ldn<N>(a.RP2 + e);
            float f[N];
#pragma unroll
            for (int n = 0; n < N; ++n) f[n] = __double2float_rn(a.nomega * t.v[n]);
            float* c = a.cR + e;
            if constexpr (N == 2)
                *reinterpret_cast<float2*>(c) = make_float2(f[0], f[1]);
            else
                *c = f[0];
        });
    });
}

// x = x2 + Y / per (+ w rp2 for the expected value, the estimator's source
// term; ForwardTally::finalize, src/MCLS_ForwardTally_impl.hpp:180-209), when
// the walk's rows have several histories.
__global__ void __launch_bounds__(kThreads, 4) k_b_correct(BatchArgs a) {
    for_tiles(a, NoEnter{}, [&](bool live, const Unit& q, int) {
        if (!live) return;
        const size_t e = q.elem();
        with_cols(q.c, [&](auto nt) {
            constexpr int N = decltype(nt)::value;
            Cols<N> x = ldn<N>(a.X2 + e);
            const Cols<N> r2 = ldn<N>(a.RP2 + e), y = ldn<N>(a.Y + e);
#pragma unroll
            for (int n = 0; n < N; ++n)
                x.v[n] = batch_corrected(x.v[n], r2.v[n], y.v[n], a.nomega, a.inv_per, a.ev);
            stn<N>(a.X + e, x);
        });
    });
}

// The active list from sys_done, in placement order, by one block: each
// thread counts a contiguous run of systems, a block scan places the runs.
__device__ void build_active(const BatchArgs& a) {
    __shared__ int s_cnt[1024];
    __shared__ int s_el[1024];
    __shared__ int s_h[1024];
    const int T = blockDim.x, tid = threadIdx.x;
    const int seg = (a.nsys + T - 1) / T;
    const int j0 = min(tid * seg, a.nsys), j1 = min(j0 + seg, a.nsys);
    int cnt = 0, hs = 0, el = 0;
    for (int j = j0; j < j1; ++j) {
        const int s = a.sorder[j];
        if (a.sys_done[s]) continue;
        ++cnt;
        el += int(system_tiles(a.sn[s], a.slog[s]));
        hs += a.sn[s] * a.per;
    }
    s_cnt[tid] = cnt;
    s_el[tid] = el;
    s_h[tid] = hs;
    __syncthreads();
    for (int d = 1; d < T; d <<= 1) {  // inclusive scan (Hillis-Steele)
        int c2 = 0, h2 = 0, e2 = 0;
        if (tid >= d) {
            c2 = s_cnt[tid - d];
            e2 = s_el[tid - d];
            h2 = s_h[tid - d];
        }
        __syncthreads();
        s_cnt[tid] += c2;
        s_el[tid] += e2;
        s_h[tid] += h2;
        __syncthreads();
    }
    int k = s_cnt[tid] - cnt;
    int eo = s_el[tid] - el;
    int ho = s_h[tid] - hs;
    for (int j = j0; j < j1; ++j) {
        const int s = a.sorder[j];
        if (a.sys_done[s]) continue;
        a.act_sys[k] = s;
        a.act_tcum[k] = eo;
        a.act_hcum[k] = ho;
        eo += int(system_tiles(a.sn[s], a.slog[s]));
        ho += a.sn[s] * a.per;
        ++k;
    }
    if (tid == T - 1) {
        *a.act_count = s_cnt[tid];
        a.act_tcum[s_cnt[tid]] = s_el[tid];
        a.act_hcum[s_cnt[tid]] = s_h[tid];
    }
}

// Per-pair convergence, loop control and the per-iteration bookkeeping (new
// stream epoch, walk timing, norms cleared, the active list rebuilt), run by
// one block.
__device__ void batch_check(const BatchArgs& a, int use_cond, cudaGraphConditionalHandle handle) {
    __shared__ int s_conv;
    if (threadIdx.x == 0) s_conv = 0;
    __syncthreads();
    int changed = 0;
    BatchState st = *a.st;
    const int it = st.iter + 1;
    const bool check = (it % st.check_freq) == 0 || it >= st.max_iters;
    // The pw lanes of a system are neighbours in a warp (pw is a power of two, at
    // most 16), so a ballot tells whether all its pairs have converged.  A few
    // pairs per thread are loaded before the first is stored; pair after pair and
    // with rp written besides, k_b_update took 74 us on 128 systems, 67 us so.
    int conv = 0;
    const int total = a.nsys * a.pw;
    const int lane = threadIdx.x & 31;
    const unsigned group = ((1u << a.pw) - 1u) << (lane & ~(a.pw - 1));
    constexpr int kAhead = 4;
    for (int base = 0; base < total; base += kAhead * int(blockDim.x)) {
        double nr[kAhead], bn[kAhead];
        int since[kAhead], done[kAhead];
        bool pair[kAhead];
#pragma unroll
        for (int u = 0; u < kAhead; ++u) {
            const int q = base + u * int(blockDim.x) + int(threadIdx.x), s = q / a.pw;
            pair[u] = q < total && q % a.pw < a.nrhs[s];
            done[u] = q < total ? a.sys_done[s] : 1;
            nr[u] = pair[u] ? __ldcg(&a.norm2[q]) : 0.0;
            bn[u] = pair[u] ? a.bnorm2[q] : 0.0;
            since[u] = pair[u] ? a.conv_iter[q] : 0;
        }
#pragma unroll
        for (int u = 0; u < kAhead; ++u) {
            const int q = base + u * int(blockDim.x) + int(threadIdx.x), s = q / a.pw;
            if (pair[u]) {
                if (!isfinite(nr[u])) atomicOr(a.status, DEV_ERR_NONFINITE);
                if (since[u] < 0 && check && sqrt(nr[u]) <= st.tol * sqrt(bn[u]))
                    a.conv_iter[q] = since[u] = it;
                if (since[u] >= 0) ++conv;
                a.norm2[q] = 0.0;
            }
            // Systems whose every right-hand side has converged stop iterating.
            const int all = (__ballot_sync(0xffffffffu, since[u] < 0) & group) == 0u;
            if (q < total && q % a.pw == 0 && done[u] != all) {
                a.sys_done[s] = all;
                changed = 1;
            }
        }
    }
    atomicAdd(&s_conv, conv);
    __syncthreads();
    // The list stands while no system finishes.
    if (__syncthreads_or(changed)) build_active(a);
    if (threadIdx.x == 0) {
        st.iter = it;
        st.converged = s_conv;
        const int keep = (s_conv < st.pairs) && (it < st.max_iters) && (*a.status == 0);
        st.done = !keep;
        *a.st = st;
        *a.d_epoch += 1;
        unsigned long long* t = a.d_tim;
        if (t[1] > t[0]) t[2] += t[1] - t[0];
        t[3] += 1;
        t[0] = ~0ULL;
        t[1] = 0;
        if (use_cond) cudaGraphSetConditional(handle, keep ? 1u : 0u);
    }
}

// Per-(system, column) sums of squares: a thread's columns stay the same from
// tile to tile of its system, so it keeps their sums in registers; when the
// block leaves the system the lanes of each column group add them with
// shuffles and the first of them adds into the global sums.
struct PairSums {
    double* sums;   // [nsys][pw]
    int pw;
    int s = -1, c = 0, g = 0;
    double v[2] = {0.0, 0.0};
    __device__ __forceinline__ void flush() {  // the whole warp
        if (s >= 0) {
            const int ul = unit_log(c), cols = unit_cols(c);
            for (int d = 16; d >= (1 << ul); d >>= 1) {
                v[0] += __shfl_xor_sync(0xffffffffu, v[0], d);
                v[1] += __shfl_xor_sync(0xffffffffu, v[1], d);
            }
            if ((threadIdx.x & 31) < (1 << ul))
                for (int n = 0; n < cols; ++n)
                    if (v[n] != 0.0) atomicAdd(&sums[size_t(s) * pw + g * cols + n], v[n]);
        }
        v[0] = v[1] = 0.0;
    }
    __device__ __forceinline__ void enter(const Unit& q) {
        flush();
        s = q.s;
        c = q.c;
        g = q.g;
    }
};

// rp = D^-1 (b - S x): the next smoothed iterate x2 = x + w rp and the
// per-(system, rhs) sums of squares (rp itself is not kept).  CHECK: the last
// block to finish runs the convergence test (the other blocks' sums are complete
// and visible by then).
template <bool CHECK, bool TAIL>
__global__ void __launch_bounds__(kThreads, kRowBlocks) k_b_update(BatchArgs a, int use_cond,
                                                         cudaGraphConditionalHandle handle) {
    PairSums ps{a.norm2, a.pw};
    Ahead h;
    auto enter = [&](const Unit& q, bool live, int i) {
        ps.enter(q);
        if (live) h.load(a.S, i);
    };
    for_tiles(a, enter, [&](bool live, const Unit& q, int next) {
        if (!live) return;
        const size_t e = q.elem();
        with_cols(q.c, [&](auto nt) {
            constexpr int N = decltype(nt)::value;
            const Cols<N> bv = ldn<N>(a.B + e);
            const double di = a.dinv[q.i];
            Cols<N> t = row_times<N, TAIL>(a.S, q, a.X, h, next);
            Cols<N> x = ldn<N>(a.X + e);
#pragma unroll
            for (int n = 0; n < N; ++n) {
                t.v[n] = di * (bv.v[n] - t.v[n]);
                ps.v[n] += t.v[n] * t.v[n];
                x.v[n] = __dadd_rn(x.v[n], __dmul_rn(a.omega, t.v[n]));
            }
            stn<N>(a.X2 + e, x);
        });
    });
    ps.flush();
    if (CHECK) {
        __shared__ bool s_last;
        __threadfence();
        __syncthreads();
        if (threadIdx.x == 0) s_last = atomicAdd(a.blocks_done, 1u) == gridDim.x - 1;
        __syncthreads();
        if (s_last) {
            __threadfence();
            batch_check(a, use_cond, handle);
            if (threadIdx.x == 0) *a.blocks_done = 0u;
        }
    }
}

// Before the loop: sums of squares of D^-1 b per pair (every system).
__global__ void __launch_bounds__(kThreads) k_b_init_norms(BatchArgs a) {
    PairSums ps{a.bnorm2, a.pw};
    auto enter = [&](const Unit& q, bool, int) { ps.enter(q); };
    for_tiles(a, enter, [&](bool live, const Unit& q, int) {
        if (!live) return;
        const size_t e = q.elem();
        with_cols(q.c, [&](auto nt) {
            constexpr int N = decltype(nt)::value;
            const Cols<N> bv = ldn<N>(a.B + e);
            const double di = a.dinv[q.i];
#pragma unroll
            for (int n = 0; n < N; ++n) {
                const double v = di * bv.v[n];
                ps.v[n] += v * v;
            }
        });
    });
    ps.flush();
}

// The fixed-width part of CSR rows.
__global__ void k_b_rows(const int* rp, const int* ci, const double* v, BatchRows M) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < M.n; i += gridDim.x * blockDim.x) {
        const int p0 = rp[i], len = rp[i + 1] - p0;
        for (int k = 0; k < kRowChunk; ++k) {
            M.col[size_t(k) * M.n + i] = k < len ? ci[p0 + k] : i;
            M.val[size_t(k) * M.n + i] = k < len ? v[p0 + k] : 0.0;
        }
    }
}

// Loop state, per-pair bookkeeping and the active list (every system), by
// one block.
__global__ void k_b_state_init(BatchArgs a, int max_iters, int check_freq, double tol,
                               int pairs) {
    const int count = a.nsys * a.pw;
    for (int q = threadIdx.x; q < count; q += blockDim.x) {
        a.conv_iter[q] = -1;
        a.norm2[q] = 0.0;
    }
    for (int q = threadIdx.x; q < a.nsys; q += blockDim.x) a.sys_done[q] = 0;
    __syncthreads();
    build_active(a);
    if (threadIdx.x == 0) {
        BatchState s{};
        s.max_iters = max_iters;
        s.check_freq = check_freq;
        s.tol = tol;
        s.pairs = pairs;
        *a.st = s;
    }
}

}  // namespace
}  // namespace mclsgpu


struct mclsgpu_batch {
    mclsgpu_context* ctx = nullptr;
    int nsys = 0;
    int pw = 1;                    // widest system's width (per-pair arrays)
    int n = 0;                     // rows
    long long ne = 0;              // elements (padding included)
    mclsgpu::BatchClasses cls{};
    std::vector<int64_t> row0;     // system -> its first row (placement order)
    std::vector<int64_t> eoff;     // system -> its first element
    std::vector<int> width;        // system -> its width (power of two)
    std::vector<int> nrhs;
    mclsgpu_operator* op = nullptr;
    mclsgpu_precond* pc = nullptr;
    mclsgpu_domain* dom = nullptr;
    mclsgpu::BatchRows S, H;       // the operator and H in rows of fixed width
    int* d_nrhs = nullptr;
    // Per system (device): first row, first element, log2 width, rows, and
    // the systems in placement order.
    int* d_srow0 = nullptr;
    long long* d_seoff = nullptr;
    int* d_slog = nullptr;
    int* d_slong = nullptr;
    bool tail = false;             // some row goes on past the fixed width
    int* d_sn = nullptr;
    int* d_sorder = nullptr;
    // The active list (rebuilt every iteration) and the list of every system.
    int* act_sys = nullptr;
    int* act_tcum = nullptr;
    int* act_hcum = nullptr;
    int* act_count = nullptr;
    int* all_sys = nullptr;
    int* all_tcum = nullptr;
    int* all_count = nullptr;
    double *X = nullptr, *X2 = nullptr, *RP2 = nullptr, *B = nullptr, *Y = nullptr;
    float* cR = nullptr;
    double* norm2 = nullptr;
    double* bnorm2 = nullptr;
    int* conv_iter = nullptr;
    int* sys_done = nullptr;
    unsigned* blocks_done = nullptr;
    mclsgpu::BatchState* d_state = nullptr;
    mclsgpu::BatchState* h_state = nullptr;
    cudaGraphExec_t graph = nullptr;
    mclsgpu::LoopKey graph_key;
    uint64_t graph_seed = 0;       // the domain seed the captured walks carry
    int body_kernels = 0;
    int per = 1;
    int grab = 1;                  // 32-history chunks that a walk's warp takes at a time
    // Grids of the element kernels: every block resident at once (each block
    // takes one contiguous range, so a second wave would double the time).
    int g_rich = 1, g_src = 1, g_cor = 1, g_upd = 1, g_upd0 = 1, g_init = 1;
};

namespace mclsgpu {
namespace {

void batch_release(mclsgpu_batch* b) {
    if (b->graph) cudaGraphExecDestroy(b->graph);
    if (b->dom) mclsgpu_domain_destroy(b->dom);
    if (b->pc) mclsgpu_precond_destroy(b->pc);
    if (b->op) mclsgpu_operator_destroy(b->op);
    dfree(b->S.col);
    dfree(b->S.val);
    dfree(b->H.col);
    dfree(b->H.val);
    dfree(b->d_nrhs);
    dfree(b->d_srow0);
    dfree(b->d_seoff);
    dfree(b->d_slog);
    dfree(b->d_slong);
    dfree(b->d_sn);
    dfree(b->d_sorder);
    dfree(b->act_sys);
    dfree(b->act_tcum);
    dfree(b->act_hcum);
    dfree(b->act_count);
    dfree(b->all_sys);
    dfree(b->all_tcum);
    dfree(b->all_count);
    dfree(b->X);
    dfree(b->X2);
    dfree(b->RP2);
    dfree(b->B);
    dfree(b->Y);
    dfree(b->cR);
    dfree(b->norm2);
    dfree(b->bnorm2);
    dfree(b->conv_iter);
    dfree(b->sys_done);
    dfree(b->blocks_done);
    dfree(b->d_state);
    if (b->h_state) cudaFreeHost(b->h_state);
    delete b;
}

int fixed_rows(mclsgpu_context* ctx, const DevCsr& A, BatchRows& M) {
    M.n = A.n;
    M.rp = A.rp;
    M.ci = A.ci;
    M.v = A.v;
    const size_t entries = size_t(M.n) * kRowChunk;
    cudaError_t e;
    if ((e = dmalloc(&M.col, entries)) != cudaSuccess ||
        (e = dmalloc(&M.val, entries)) != cudaSuccess)
        return cuda_fail(ctx, e, "cudaMalloc batch rows");
    const int grid = std::min((M.n + kThreads - 1) / kThreads, ctx->num_sms * 8);
    drop_stale_error();
    k_b_rows<<<grid, kThreads, 0, ctx->stream>>>(A.rp, A.ci, A.v, M);
    e = cudaGetLastError();
    return e == cudaSuccess ? MCLSGPU_OK : cuda_fail(ctx, e, "batch rows");
}

// Kernel arguments over the active list (all = false) or every system.
BatchArgs batch_args(mclsgpu_batch* b, const mclsgpu_mcsa_params* mp, bool all) {
    const mclsgpu_mc_params& p = b->dom->p;
    BatchArgs a{};
    a.nsys = b->nsys;
    a.pw = b->pw;
    a.per = b->per;
    a.S = b->S;
    a.dinv = b->pc->diag;
    a.H = b->H;
    a.srow0 = b->d_srow0;
    a.seoff = b->d_seoff;
    a.slog = b->d_slog;
    a.slong = b->d_slong;
    a.sn = b->d_sn;
    a.sorder = b->d_sorder;
    a.lsys = all ? b->all_sys : b->act_sys;
    a.ltcum = all ? b->all_tcum : b->act_tcum;
    a.lcount = all ? b->all_count : b->act_count;
    a.act_sys = b->act_sys;
    a.act_tcum = b->act_tcum;
    a.act_hcum = b->act_hcum;
    a.act_count = b->act_count;
    a.B = b->B;
    a.X = b->X;
    a.X2 = b->X2;
    a.RP2 = b->RP2;
    a.Y = b->Y;
    a.cR = b->cR;
    a.norm2 = b->norm2;
    a.bnorm2 = b->bnorm2;
    a.conv_iter = b->conv_iter;
    a.nrhs = b->d_nrhs;
    a.sys_done = b->sys_done;
    a.st = b->d_state;
    a.blocks_done = b->blocks_done;
    a.omega = mp ? mp->richardson_omega : 1.0;
    a.nomega = p.neumann_relaxation > 0.0 ? p.neumann_relaxation : 1.0;
    a.inv_per = 1.0 / double(b->per);
    a.ev = p.estimator == MCLSGPU_EXPECTED_VALUE;
    a.d_epoch = b->dom->d_epoch;
    a.d_tim = b->dom->d_tim;
    a.status = b->ctx->d_status;
    return a;
}

template <class K>
int resident_grid(K kernel, int sms) {
    int b = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, kernel, kThreads, 0);
    return sms * (b > 0 ? b : 1);
}

// One batched MCSA iteration (4 kernels; 5 with several histories per row)
// over the active systems.
int enqueue_batch_iteration(mclsgpu_batch* b, const mclsgpu_mcsa_params* mp, int use_cond,
                            cudaGraphConditionalHandle handle) {
    cudaStream_t s = b->ctx->stream;
    BatchArgs a = batch_args(b, mp, false);
    auto residual = b->tail ? k_b_smoothed_residual<true> : k_b_smoothed_residual<false>;
    auto source = b->tail ? k_b_source<true> : k_b_source<false>;
    auto update = b->tail ? k_b_update<true, true> : k_b_update<true, false>;
    residual<<<b->g_rich, kThreads, 0, s>>>(a);
    source<<<b->g_src, kThreads, 0, s>>>(a);
    const BatchList list{b->act_sys, b->act_hcum, b->act_count, b->d_srow0};
    const BatchFinish fin{b->X, b->X2, b->RP2, a.nomega, a.inv_per, a.ev};
    int rc = launch_walk_batch(b->dom, b->cls, list, b->cR, b->Y, fin, b->grab);
    if (rc) return rc;
    if (b->Y) k_b_correct<<<b->g_cor, kThreads, 0, s>>>(a);
    update<<<b->g_upd, kThreads, 0, s>>>(a, use_cond, handle);
    return MCLSGPU_OK;
}

int build_batch_graph(mclsgpu_batch* b, const mclsgpu_mcsa_params* mp) {
    mclsgpu_context* ctx = b->ctx;
    if (b->graph) {
        cudaGraphExecDestroy(b->graph);
        b->graph = nullptr;
    }
    int red = MCLSGPU_OK;
    const int rc = build_while_graph(
        ctx, [&](cudaGraphConditionalHandle h) { red = enqueue_batch_iteration(b, mp, 1, h); },
        &b->graph, &b->body_kernels);
    return rc ? rc : red;
}

}  // namespace
}  // namespace mclsgpu

using namespace mclsgpu;

extern "C" {

int mclsgpu_batch_build(mclsgpu_context* ctx, int nsys, const int64_t* n,
                        const int64_t* const* rowptr, const int64_t* const* colind,
                        const double* const* values, const int32_t* nrhs,
                        const mclsgpu_mc_params* params, mclsgpu_batch** out) {
    if (!ctx || nsys < 1 || !n || !rowptr || !colind || !values || !nrhs || !params || !out)
        return MCLSGPU_ERR_INVALID_ARG;
    *out = nullptr;
    if (params->size < sizeof(mclsgpu_mc_params))
        return set_error(ctx, MCLSGPU_ERR_INVALID_ARG, "mc params: size mismatch");
    if (params->direction != MCLSGPU_FORWARD || params->precision != MCLSGPU_FP32 ||
        params->weight_cutoff > 0.0)
        return set_error(ctx, MCLSGPU_ERR_UNSUPPORTED,
                         "batched MCSA runs forward FP32 walks of fixed length");
    // Width classes: system s gets W_s = nrhs_s rounded up to a power of two;
    // the systems are placed class by class (in argument order within a class).
    std::vector<int> width(nsys), cls_of(nsys);
    int pw = 1;
    for (int s = 0; s < nsys; ++s) {
        if (n[s] < 1 || !rowptr[s] || !colind[s] || !values[s] || nrhs[s] < 1 || nrhs[s] > 16)
            return set_error(ctx, MCLSGPU_ERR_INVALID_ARG,
                             "batch system %d: empty, missing arrays or 1..16 right-hand sides", s);
        int c = 0;
        while ((1 << c) < nrhs[s]) ++c;
        cls_of[s] = c;
        width[s] = 1 << c;
        if (width[s] > pw) pw = width[s];
    }
    std::vector<int> order;
    for (int c = 0; c < 5; ++c)
        for (int s = 0; s < nsys; ++s)
            if (cls_of[s] == c) order.push_back(s);
    BatchClasses cls{};
    std::vector<int64_t> row0(nsys), eoff(nsys);
    int64_t N = 0, NE = 0;
    size_t k = 0;
    for (int c = 0; c < 5; ++c) {
        cls.crow[c] = int(std::min<int64_t>(N, int64_t(1) << 30));
        NE = (NE + 15) / 16 * 16;  // class blocks start on 16-element boundaries
        cls.cel[c] = NE;
        for (; k < order.size() && cls_of[order[k]] == c; ++k) {
            const int s = order[k];
            row0[s] = N;
            eoff[s] = NE;
            N += n[s];
            NE += n[s] << c;
        }
    }
    cls.crow[5] = int(std::min<int64_t>(N, int64_t(1) << 30));
    NE = (NE + 15) / 16 * 16;
    cls.cel[5] = NE;
    if (N >= (int64_t(1) << 30))
        return set_error(ctx, MCLSGPU_ERR_UNSUPPORTED, "batch too large (%lld rows)", (long long)N);
    int64_t nnz = 0;
    for (int s = 0; s < nsys; ++s) nnz += rowptr[s][n[s]] - rowptr[s][0];
    if (nnz >= (int64_t(1) << 31) - 1)
        return set_error(ctx, MCLSGPU_ERR_UNSUPPORTED, "batch too large (%lld entries)", (long long)nnz);
    // The block-diagonal operator in placement order.
    std::vector<int64_t> rp(N + 1), ci(nnz);
    std::vector<double> v(nnz);
    int64_t pos = 0;
    for (int s : order) {
        const int64_t o = row0[s];
        for (int64_t i = 0; i < n[s]; ++i) {
            rp[o + i] = pos;
            for (int64_t p = rowptr[s][i]; p < rowptr[s][i + 1]; ++p, ++pos) {
                if (colind[s][p] < 0 || colind[s][p] >= n[s])
                    return set_error(ctx, MCLSGPU_ERR_INVALID_ARG,
                                     "batch system %d: column index out of range", s);
                ci[pos] = colind[s][p] + o;
                v[pos] = values[s][p];
            }
        }
    }
    rp[N] = pos;
    mclsgpu_batch* b = new mclsgpu_batch;
    b->ctx = ctx;
    b->nsys = nsys;
    b->pw = pw;
    b->n = int(N);
    b->ne = NE;
    b->cls = cls;
    b->row0 = row0;
    b->eoff = eoff;
    b->width = width;
    b->nrhs.assign(nrhs, nrhs + nsys);
    b->per = params->sample_ratio > 0.0 ? int(std::ceil(params->sample_ratio)) : 1;
    if (double(N) * b->per >= double(int64_t(1) << 31)) {
        delete b;
        return set_error(ctx, MCLSGPU_ERR_UNSUPPORTED, "batch too large (histories per iteration)");
    }
    // Per-system tables and the list of every system (placement order).
    std::vector<int> srow0(nsys), sn(nsys), all_count(1, nsys);
    std::vector<long long> seoff(nsys);
    std::vector<int> all_tcum(nsys + 1, 0);
    for (int s = 0; s < nsys; ++s) {
        srow0[s] = int(row0[s]);
        seoff[s] = eoff[s];
        sn[s] = int(n[s]);
    }
    for (int k = 0; k < nsys; ++k) {
        const int s = order[k];
        all_tcum[k + 1] = all_tcum[k] + int(system_tiles(int(n[s]), cls_of[s]));
    }
    int rc = mclsgpu_operator_upload(ctx, N, rp.data(), ci.data(), v.data(), &b->op);
    mclsgpu_precond_params pp{};
    pp.size = sizeof(pp);
    pp.kind = MCLSGPU_PREC_POINT_JACOBI;
    if (!rc) rc = mclsgpu_precond_build(ctx, b->op, &pp, &b->pc);
    if (!rc) rc = mclsgpu_domain_build(ctx, b->op, b->pc, nullptr, params, &b->dom);
    if (!rc && b->dom->stencil_k && b->dom->slots > 8) {
        // The shared walk takes stencil records of at most 64 bytes.
        mclsgpu_domain_destroy(b->dom);
        b->dom = nullptr;
        mclsgpu_mc_params pk = *params;
        pk.record_format = MCLSGPU_RECORD_PACKED;
        rc = mclsgpu_domain_build(ctx, b->op, b->pc, nullptr, &pk, &b->dom);
    }
    if (!rc && (b->dom->slots > 16 || b->dom->rec_q16))
        rc = set_error(ctx, MCLSGPU_ERR_UNSUPPORTED,
                       "batched walks: rows of at most 15 retained entries");
    // The rows of the element passes.
    std::vector<int> slong(nsys, 0);
    int longest = 0;
    for (int k = 0; k < nsys; ++k)
        for (int64_t i = 0; i < n[k]; ++i) {
            const int64_t len = rowptr[k][i + 1] - rowptr[k][i];
            longest = std::max(longest, int(len));
            if (len > kRowChunk) slong[k] = 1;
        }
    // H's rows are parts of the operator's, unless one lacks its diagonal.
    if (!rc && b->dom->max_row > longest) std::fill(slong.begin(), slong.end(), 1);
    b->tail = std::count(slong.begin(), slong.end(), 1) > 0;
    if (!rc) rc = fixed_rows(ctx, b->op->A, b->S);
    if (!rc && params->estimator == MCLSGPU_EXPECTED_VALUE) rc = fixed_rows(ctx, b->dom->D, b->H);
    const size_t PR = size_t(nsys) * pw;
    cudaError_t e = cudaSuccess;
    if (!rc &&
        ((e = dmalloc(&b->d_nrhs, nsys)) != cudaSuccess ||
         (e = dmalloc(&b->d_srow0, nsys)) != cudaSuccess ||
         (e = dmalloc(&b->d_seoff, nsys)) != cudaSuccess ||
         (e = dmalloc(&b->d_slog, nsys)) != cudaSuccess ||
         (e = dmalloc(&b->d_slong, nsys)) != cudaSuccess || (e = dmalloc(&b->d_sn, nsys)) != cudaSuccess ||
         (e = dmalloc(&b->d_sorder, nsys)) != cudaSuccess ||
         (e = dmalloc(&b->act_sys, nsys)) != cudaSuccess ||
         (e = dmalloc(&b->act_tcum, nsys + 1)) != cudaSuccess ||
         (e = dmalloc(&b->act_hcum, nsys + 1)) != cudaSuccess ||
         (e = dmalloc(&b->act_count, 1)) != cudaSuccess ||
         (e = dmalloc(&b->all_sys, nsys)) != cudaSuccess ||
         (e = dmalloc(&b->all_tcum, nsys + 1)) != cudaSuccess ||
         (e = dmalloc(&b->all_count, 1)) != cudaSuccess ||
         (e = dmalloc(&b->X, NE)) != cudaSuccess || (e = dmalloc(&b->X2, NE)) != cudaSuccess ||
         (e = dmalloc(&b->RP2, NE)) != cudaSuccess ||
         (e = dmalloc(&b->B, NE)) != cudaSuccess ||
         (b->per > 1 && (e = dmalloc(&b->Y, NE)) != cudaSuccess) ||
         (e = dmalloc(&b->cR, NE)) != cudaSuccess || (e = dmalloc(&b->norm2, PR)) != cudaSuccess ||
         (e = dmalloc(&b->bnorm2, PR)) != cudaSuccess ||
         (e = dmalloc(&b->conv_iter, PR)) != cudaSuccess || (e = dmalloc(&b->sys_done, nsys)) != cudaSuccess ||
         (e = dmalloc(&b->blocks_done, 1)) != cudaSuccess || (e = dmalloc(&b->d_state, 1)) != cudaSuccess ||
         (e = cudaMallocHost(reinterpret_cast<void**>(&b->h_state), sizeof(BatchState))) != cudaSuccess))
        rc = cuda_fail(ctx, e, "cudaMalloc batch");
    if (!rc) {
        const int sms = ctx->num_sms;
        const bool tail = b->tail;
        b->g_rich = resident_grid(
            tail ? k_b_smoothed_residual<true> : k_b_smoothed_residual<false>, sms);
        b->g_src = resident_grid(tail ? k_b_source<true> : k_b_source<false>, sms);
        b->g_cor = resident_grid(k_b_correct, sms);
        b->g_upd = resident_grid(tail ? k_b_update<true, true> : k_b_update<true, false>, sms);
        b->g_upd0 = resident_grid(tail ? k_b_update<false, true> : k_b_update<false, false>, sms);
        b->g_init = resident_grid(k_b_init_norms, sms);
        cudaStream_t s = ctx->stream;
        cudaMemcpyAsync(b->d_nrhs, b->nrhs.data(), sizeof(int) * nsys, cudaMemcpyHostToDevice, s);
        cudaMemcpyAsync(b->d_srow0, srow0.data(), sizeof(int) * nsys, cudaMemcpyHostToDevice, s);
        cudaMemcpyAsync(b->d_seoff, seoff.data(), sizeof(long long) * nsys, cudaMemcpyHostToDevice,
                        s);
        cudaMemcpyAsync(b->d_slog, cls_of.data(), sizeof(int) * nsys, cudaMemcpyHostToDevice, s);
        cudaMemcpyAsync(b->d_slong, slong.data(), sizeof(int) * nsys, cudaMemcpyHostToDevice, s);
        cudaMemcpyAsync(b->d_sn, sn.data(), sizeof(int) * nsys, cudaMemcpyHostToDevice, s);
        cudaMemcpyAsync(b->d_sorder, order.data(), sizeof(int) * nsys, cudaMemcpyHostToDevice, s);
        cudaMemcpyAsync(b->all_sys, order.data(), sizeof(int) * nsys, cudaMemcpyHostToDevice, s);
        cudaMemcpyAsync(b->all_tcum, all_tcum.data(), sizeof(int) * (nsys + 1),
                        cudaMemcpyHostToDevice, s);
        cudaMemcpyAsync(b->all_count, all_count.data(), sizeof(int), cudaMemcpyHostToDevice, s);
        // Padding elements are never written by the loop: zero every array once.
        cudaMemsetAsync(b->X, 0, sizeof(double) * NE, s);
        cudaMemsetAsync(b->X2, 0, sizeof(double) * NE, s);
        cudaMemsetAsync(b->RP2, 0, sizeof(double) * NE, s);
        if (b->Y) cudaMemsetAsync(b->Y, 0, sizeof(double) * NE, s);
        cudaMemsetAsync(b->cR, 0, sizeof(float) * NE, s);
        cudaMemsetAsync(b->blocks_done, 0, sizeof(unsigned), s);
        e = cudaStreamSynchronize(s);
        if (e != cudaSuccess) rc = cuda_fail(ctx, e, "batch build");
    }
    if (rc) {
        batch_release(b);
        return rc;
    }
    *out = b;
    return MCLSGPU_OK;
}

int mclsgpu_batch_destroy(mclsgpu_batch* b) {
    if (!b) return MCLSGPU_OK;
    batch_release(b);
    return MCLSGPU_OK;
}

int mclsgpu_batch_layout(mclsgpu_batch* b, int64_t* elem_offsets, int32_t* widths,
                         int64_t* elements, int32_t* max_width) {
    if (!b) return MCLSGPU_ERR_INVALID_ARG;
    for (int s = 0; s < b->nsys; ++s) {
        if (elem_offsets) elem_offsets[s] = b->eoff[s];
        if (widths) widths[s] = b->width[s];
    }
    if (elements) *elements = b->ne;
    if (max_width) *max_width = b->pw;
    return MCLSGPU_OK;
}

int mclsgpu_batch_domain(mclsgpu_batch* b, mclsgpu_domain** dom) {
    if (!b || !dom) return MCLSGPU_ERR_INVALID_ARG;
    *dom = b->dom;
    return MCLSGPU_OK;
}

int mclsgpu_batch_set_launch(mclsgpu_batch* b, int block_size, int grab) {
    if (!b || (block_size != 128 && block_size != 256) || grab < 1 || grab > 8)
        return MCLSGPU_ERR_INVALID_ARG;
    b->dom->walk_block = block_size;
    b->grab = grab;
    return MCLSGPU_OK;
}

int mclsgpu_batch_autotune(mclsgpu_batch* b, const double* b_dev, double* x_dev, int reps,
                           int* block_size, int* grab, double* walk_ms) {
    if (!b || !b_dev || !x_dev || reps < 1) return MCLSGPU_ERR_INVALID_ARG;
    mclsgpu_mcsa_params p{};
    p.size = sizeof(p);
    p.max_iters = reps;
    p.tolerance = 0.0;
    p.check_freq = 1;
    p.smoother_steps = 1;
    p.richardson_omega = 1.0;
    p.host_loop = 1;
    const int blocks[2] = {256, 128};
    const int grabs[3] = {1, 2, 4};
    int best_b = 256, best_g = 1;
    double best_ms = 1e300;
    for (int blk : blocks)
        for (int g : grabs) {
            b->dom->walk_block = blk;
            b->grab = g;
            cudaMemsetAsync(x_dev, 0, sizeof(double) * size_t(b->ne), b->ctx->stream);
            mclsgpu_stats st{};
            st.size = sizeof(st);
            int rc = mclsgpu_batch_mcsa_solve_dev(b, b_dev, x_dev, &p, nullptr, nullptr, &st);
            if (rc) return rc;
            const double per = st.walk_launches ? st.walk_ms / double(st.walk_launches) : 1e300;
            if (per < best_ms) {
                best_ms = per;
                best_b = blk;
                best_g = g;
            }
        }
    b->dom->walk_block = best_b;
    b->grab = best_g;
    if (block_size) *block_size = best_b;
    if (grab) *grab = best_g;
    if (walk_ms) *walk_ms = best_ms;
    return MCLSGPU_OK;
}

int mclsgpu_batch_mcsa_solve_dev(mclsgpu_batch* b, const double* b_dev, double* x_dev,
                                 const mclsgpu_mcsa_params* params, int32_t* conv_iters,
                                 double* rel_resid, mclsgpu_stats* stats) {
    if (!b || !b_dev || !x_dev || !params) return MCLSGPU_ERR_INVALID_ARG;
    mclsgpu_context* ctx = b->ctx;
    if (params->size < sizeof(mclsgpu_mcsa_params) || params->max_iters < 1 ||
        params->check_freq < 1 || !(params->tolerance >= 0.0) || params->smoother_steps != 1)
        return set_error(ctx, MCLSGPU_ERR_INVALID_ARG,
                         "batch mcsa params out of range (one smoother step)");
    cudaStream_t s = ctx->stream;
    const size_t NE = size_t(b->ne), PR = size_t(b->nsys) * b->pw;
    int pairs = 0;
    for (int q = 0; q < b->nsys; ++q) pairs += b->nrhs[q];
    const LoopKey key{params->richardson_omega, b->grab, b->dom->walk_block};
    if (!params->host_loop && (!b->graph || b->graph_key != key || b->graph_seed != b->dom->seed)) {
        int rc = build_batch_graph(b, params);
        if (rc) return rc;
        b->graph_key = key;
        b->graph_seed = b->dom->seed;
    }
    cudaEvent_t e0, e1;
    cudaEventCreate(&e0);
    cudaEventCreate(&e1);
    cudaMemsetAsync(ctx->d_status, 0, sizeof(int), s);
    cudaMemsetAsync(b->dom->d_steps, 0, sizeof(unsigned long long), s);
    cudaMemsetAsync(b->blocks_done, 0, sizeof(unsigned), s);
    {
        unsigned long long tim0[4] = {~0ULL, 0ULL, 0ULL, 0ULL};
        cudaMemcpyAsync(b->dom->d_tim, tim0, sizeof(tim0), cudaMemcpyHostToDevice, s);
    }
    cudaEventRecord(e0, s);
    cudaMemcpyAsync(b->B, b_dev, sizeof(double) * NE, cudaMemcpyDeviceToDevice, s);
    cudaMemcpyAsync(b->X, x_dev, sizeof(double) * NE, cudaMemcpyDeviceToDevice, s);
    cudaMemsetAsync(b->bnorm2, 0, sizeof(double) * PR, s);
    BatchArgs a = batch_args(b, params, true);  // every system
    k_b_state_init<<<1, 1024, 0, s>>>(a, params->max_iters, params->check_freq,
                                       params->tolerance, pairs);
    k_b_init_norms<<<b->g_init, kThreads, 0, s>>>(a);
    auto norms = b->tail ? k_b_update<false, true> : k_b_update<false, false>;
    norms<<<b->g_upd0, kThreads, 0, s>>>(a, 0, cudaGraphConditionalHandle(0));
    cudaMemsetAsync(b->norm2, 0, sizeof(double) * PR, s);
    cudaError_t e = cudaSuccess;
    int rc = MCLSGPU_OK;
    if (!params->host_loop) {
        e = cudaGraphLaunch(b->graph, s);
    } else {
        for (int it = 0; it < params->max_iters && e == cudaSuccess && !rc; ++it) {
            rc = enqueue_batch_iteration(b, params, 0, cudaGraphConditionalHandle(0));
            cudaMemcpyAsync(b->h_state, b->d_state, sizeof(BatchState), cudaMemcpyDeviceToHost, s);
            e = cudaStreamSynchronize(s);
            if (e == cudaSuccess && b->h_state->done) break;
        }
    }
    cudaEventRecord(e1, s);
    if (e == cudaSuccess) {
        cudaMemcpyAsync(x_dev, b->X, sizeof(double) * NE, cudaMemcpyDeviceToDevice, s);
        cudaMemcpyAsync(b->h_state, b->d_state, sizeof(BatchState), cudaMemcpyDeviceToHost, s);
        e = cudaStreamSynchronize(s);
    }
    float ms = 0.f;
    cudaEventElapsedTime(&ms, e0, e1);
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    if (rc) return rc;
    if (e != cudaSuccess) return cuda_fail(ctx, e, "batch mcsa");
    if ((rc = check_device_status(ctx))) return rc;
    const BatchState st = *b->h_state;
    if (conv_iters || rel_resid) {
        // Final per-pair residuals: one more residual pass on the result.
        std::vector<double> nr(PR), bn(PR);
        std::vector<int> ci(PR);
        cudaMemsetAsync(b->norm2, 0, sizeof(double) * PR, s);
        norms<<<b->g_upd0, kThreads, 0, s>>>(a, 0, cudaGraphConditionalHandle(0));
        cudaMemcpyAsync(nr.data(), b->norm2, sizeof(double) * PR, cudaMemcpyDeviceToHost, s);
        cudaMemcpyAsync(bn.data(), b->bnorm2, sizeof(double) * PR, cudaMemcpyDeviceToHost, s);
        cudaMemcpyAsync(ci.data(), b->conv_iter, sizeof(int) * PR, cudaMemcpyDeviceToHost, s);
        e = cudaStreamSynchronize(s);
        if (e != cudaSuccess) return cuda_fail(ctx, e, "batch residuals");
        for (size_t q = 0; q < PR; ++q) {
            const bool valid = int(q % b->pw) < b->nrhs[q / b->pw];
            if (conv_iters) conv_iters[q] = valid ? ci[q] : -1;
            if (rel_resid)
                rel_resid[q] = valid ? (bn[q] > 0.0 ? std::sqrt(nr[q] / bn[q]) : std::sqrt(nr[q])) : 0.0;
        }
    }
    if (stats) {
        if (stats->size < sizeof(mclsgpu_stats))
            return set_error(ctx, MCLSGPU_ERR_INVALID_ARG, "stats: size mismatch");
        mclsgpu_stats out{};
        out.size = sizeof(out);
        unsigned long long steps = 0, tim[4] = {0, 0, 0, 0};
        cudaMemcpy(&steps, b->dom->d_steps, sizeof(steps), cudaMemcpyDeviceToHost);
        cudaMemcpy(tim, b->dom->d_tim, sizeof(tim), cudaMemcpyDeviceToHost);
        out.iterations = st.iter;
        out.converged = st.converged == st.pairs;
        out.walk_steps = int64_t(steps);
        out.histories = int64_t(st.iter) * int64_t(b->n) * b->per;
        out.solve_ms = ms;
        out.walk_ms = double(tim[2]) * 1e-6;
        out.walk_launches = int64_t(tim[3]);
        out.kernel_launches = int64_t(b->body_kernels ? b->body_kernels : 4) * st.iter + 3;
        out.rho = -1.0;
        *stats = out;
    }
    return MCLSGPU_OK;
}

}  // extern "C"

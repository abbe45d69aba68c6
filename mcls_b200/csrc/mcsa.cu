// mcsa.cu -- Monte Carlo solve and the MCSA Richardson/correction loop.
//
// MC solve (MonteCarloSolverManager::solve + MCSolver::solve,
// src/MCLS_MonteCarloSolverManager_impl.hpp:199-235, 346-380,
// src/MCLS_MCSolver_impl.hpp:82-112): source from the (left preconditioned
// unless internal, Neumann-relaxed) right-hand side, transport, normalise by
// the number of histories, right-preconditioner recovery unless internal.
//
// Estimators.  Collision: x = y / Nh with y the collision tally.
// Expected value (no counterpart in this reference snapshot): every step adds
// w * h_{s,j} to x_j for all j of the current row; summed over a history
// this equals H applied to the history's collision tally, so the kernel
// computes x = b_src + (D^T y) / Nh with one gather over the transposed
// domain instead of k scattered updates per step (forward: the tally source
// is H b_src instead of b_src).
//
// MCSA (MCSASolverManager::solve, src/MCLS_MCSASolverManager_impl.hpp:
// 278-432): each iteration runs Richardson smoothing (x += w rp, then
// rp = PL(b - A PR x)), zeroes the correction, solves the residual problem by
// MC (internal), adds the correction and recomputes the residual; the loop
// stops when |rp|_2 <= tol * |PL b|_2 or the iteration limit is reached,
// checked every "Iteration Check Frequency" iterations.  The whole loop is one
// CUDA graph: a WHILE conditional node whose body is one iteration and whose
// condition is set on the device by the convergence check, so a solve makes
// no host round trip per iteration.
#include <algorithm>
#include <array>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <vector>

#include <cooperative_groups.h>

#include "internal.h"
#include "ops.cuh"
#include "rng.cuh"

namespace mclsgpu {

void launch_adjoint_source(mclsgpu_domain* dom, const double* v, double omega, int has_omega);
void launch_forward_source(mclsgpu_domain* dom, const double* v, double omega, int has_omega,
                           bool fused);
void launch_advance_walk_pos(mclsgpu_domain* dom);
void prepare_walk(mclsgpu_domain* dom);
bool walks_from_shared(const mclsgpu_domain* dom);
void launch_walk(mclsgpu_domain* dom, const RowFinish& fin, long long max_trace,
                 long long* tr_states, double* tr_w, int* tr_ev, long long* tr_start, bool fused);

namespace {

inline int grid_for(long long work, int threads = 256, int cap = 148 * 16) {
    long long g = (work + threads - 1) / threads;
    if (g < 1) g = 1;
    return int(g > cap ? cap : g);
}

// rp = (b - A x) [* dinv]   (LinearProblem::updatePrecResidual, :410-442)
template <class Op>
__global__ void __launch_bounds__(256) k_residual(Op A, const double* x, const double* b,
                                                  const double* dinv, double* out) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < A.n; i += gridDim.x * blockDim.x) {
        const double s = A.dot(i, [&](int j) { return x[j]; });
        double r = b[i] - s;
        out[i] = dinv ? dinv[i] * r : r;
    }
}

// out = [dinv *] A x   (the A and PL factors of LinearProblem::apply, :251-279)
template <class Op>
__global__ void __launch_bounds__(256) k_matvec(Op A, const double* x, const double* dinv,
                                                double* out) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < A.n; i += gridDim.x * blockDim.x) {
        const double s = A.dot(i, [&](int j) { return x[j]; });
        out[i] = dinv ? dinv[i] * s : s;
    }
}

// x += w * r  (RichardsonIteration::doOneIteration, :134-147)
__global__ void k_richardson(double* x, const double* r, int n, double w) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        x[i] = __dadd_rn(x[i], __dmul_rn(w, r[i]));
}

// The words a solve's counters and report live in.
struct Counters {
    int* status;
    unsigned long long* steps;
    unsigned long long* hist;
    unsigned long long* tim;
    const McsaState* st;
    const double* src_sumsq;
};

__device__ __forceinline__ void write_report(const Counters& c, SolveReport* r) {
    SolveReport v;
    v.st = *c.st;
    v.src_sumsq = *c.src_sumsq;
    v.steps = *c.steps;
    v.hist = *c.hist;
    v.walk_ns = c.tim[2];
    v.launches = c.tim[3];
    v.status = *c.status;
    v.pad = 0;
    *r = v;
}

__global__ void k_report(Counters c, SolveReport* r) { write_report(c, r); }

// Start of a solve: the device error word and the walk statistics cleared.
__global__ void k_solve_begin(Counters c) {
    *c.status = 0;
    *c.steps = 0;
    *c.hist = 0;
    c.tim[2] = 0;
    c.tim[3] = 0;
}

// End of a Monte Carlo solve (one thread): the stream epoch, the history count,
// the walk timing, and the host's report (may be null).
__device__ __forceinline__ void end_mc(unsigned long long* epoch, const int* d_nh,
                                       const Counters& c, SolveReport* report) {
    const unsigned long long e = *epoch, h = *c.hist;
    const int nh = *d_nh;
    *epoch = e + 1ULL;
    *c.hist = h + (unsigned long long)nh;
    add_walk_time(c.tim);
    if (report) write_report(c, report);
}

__global__ void k_mc_end(unsigned long long* epoch, const int* d_nh, Counters c,
                         SolveReport* report) {
    end_mc(epoch, d_nh, c, report);
}

struct FinalizeArgs {
    int n;
    int mode;            // 0 adjoint collision, 1 adjoint EV, 2 forward
    int ev;
    int base;            // kBase*: out = delta, out + delta, or xin + delta
    int fp32;
    double per;          // forward histories per state
    const double* xin;
    const double* sc;    // [2] = 1/nh
    const double* src;   // MC source vector before scaling
    double omega;
    int has_omega;
    const double* y64;
    const int* dtrp;
    const int* dtci;
    const float* dth32;
    const double* dth64;
    double* out;
    // A Monte Carlo solve of its own ends here (null epoch: its caller ends it).
    unsigned long long* epoch;
    const int* d_nh;
    Counters c;
    SolveReport* report;
    unsigned int* ticket;
};

// The walks' tallies into the solution; for a Monte Carlo solve of its own the
// last block also ends the solve (a launch of its own took 4.2 us of the 66 us of
// a 32^2 solve with host vectors, the ticket 3).
__global__ void __launch_bounds__(256) k_finalize(FinalizeArgs a) {
    const double inv = a.sc[2];
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < a.n; i += gridDim.x * blockDim.x) {
        double d;
        const double srci = a.has_omega ? a.src[i] * a.omega : a.src[i];
        if (a.mode == 0) {
            // AdjointTally::normalize: x *= 1/nh  (src/MCLS_AdjointTally_impl.hpp:68-72)
            d = __dmul_rn(a.y64[i], inv);
        } else if (a.mode == 1) {
            double t = 0.0;
            if (a.fp32) {
                for (int k = a.dtrp[i]; k < a.dtrp[i + 1]; ++k)
                    t = fma(double(a.dth32[k]), a.y64[a.dtci[k]], t);
            } else {
                for (int k = a.dtrp[i]; k < a.dtrp[i + 1]; ++k)
                    t = fma(a.dth64[k], a.y64[a.dtci[k]], t);
            }
            d = __dadd_rn(__dmul_rn(t, inv), srci);
        } else {
            // ForwardTally::finalize: sum / count  (src/MCLS_ForwardTally_impl.hpp:194-208)
            d = __ddiv_rn(a.y64[i], a.per);
            if (a.ev) d = __dadd_rn(d, srci);
        }
        if (a.base == kBaseOut)
            d = __dadd_rn(a.out[i], d);
        else if (a.base == kBaseIn)
            d = __dadd_rn(a.xin[i], d);
        a.out[i] = d;
    }
    if (!a.epoch) return;
    __syncthreads();
    if (threadIdx.x != 0) return;
    __threadfence();
    if (atomicAdd(a.ticket, 1u) != gridDim.x - 1) return;
    *a.ticket = 0u;
    end_mc(a.epoch, a.d_nh, a.c, a.report);
}

// Convergence check of one MCSA iteration (src/MCLS_MCSASolverManager_impl.hpp:380-394).
// s: the loop state and `status` the device error word, as loaded.
__device__ __forceinline__ int mcsa_check(McsaState s, int status, McsaState* st, double sumsq,
                                          double* hist, int hist_cap, int* d_status) {
    s.iter += 1;
    s.rnorm = sqrt(sumsq);
    if (hist && s.iter <= hist_cap) hist[s.iter - 1] = s.rnorm;
    int keep = 1;
    if (s.iter % s.check_freq == 0) keep = (s.rnorm > s.crit) && (s.iter < s.max_iters);
    // A non-finite residual norm ends the loop as a divergence.
    if (!isfinite(s.rnorm)) {
        atomicOr(d_status, DEV_ERR_NONFINITE);
        keep = 0;
    }
    if (status) keep = 0;
    s.done = !keep;
    s.converged = s.rnorm <= s.crit;
    *st = s;
    return keep;
}

__global__ void k_mcsa_check(McsaState* st, const double* sumsq, double* hist, int hist_cap,
                             int* status, cudaGraphConditionalHandle handle) {
    const int keep = mcsa_check(*st, *status, st, *sumsq, hist, hist_cap, status);
    cudaGraphSetConditional(handle, keep ? 1u : 0u);
}

__global__ void k_mcsa_check_host(McsaState* st, const double* sumsq, double* hist, int hist_cap,
                                  int* status) {
    mcsa_check(*st, *status, st, *sumsq, hist, hist_cap, status);
}

// ---- fused iteration kernels (smoother_steps == 1, PL in {I, point Jacobi}) ----
constexpr int kFusedThreads = 256;

// Richardson smoothing fused with the residual: x2 = x + w rp (rounded as the
// separate update would be) and rp2 = PL (b - A x2), reading x + w rp at the
// neighbours on the fly (Anderson steps and adjoint domains; a forward MCSA
// loop has x2 from the last iteration's k_residual_norm).
template <class Op>
__global__ void __launch_bounds__(kFusedThreads) k_smoothed_residual(
    Op A, const double* b, const double* dinv, const double* x, const double* r, double w,
    double* x2, double* r2) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < A.n; i += gridDim.x * blockDim.x) {
        const double s = A.dot(i, [&](int j) { return __dadd_rn(x[j], __dmul_rn(w, r[j])); });
        const double res = b[i] - s;
        r2[i] = dinv ? dinv[i] * res : res;
        x2[i] = __dadd_rn(x[i], __dmul_rn(w, r[i]));
    }
}

struct ResidArgs {
    int n;
    const double* b;
    const double* dinv;       // null: no left preconditioner
    double* x;                // the corrected iterate
    double* rout;
    double* x2;               // the smoothed iterate: read (FOLD) or the next x + w rp
    double w;
    const double* y;          // FOLD: the walk's tallies and 1 / histories
    const double* inv_nh;
    double* part;
    unsigned int* ticket;
    McsaState* st;
    double* hist;
    int hist_cap;
    int* status;
    unsigned long long* d_epoch;
    unsigned long long* d_tim;
    int* d_counter;
    unsigned long long* d_hist;
    const int* d_nh;
    cudaGraphConditionalHandle handle;
    int use_cond;
};

// The words that the end of an iteration reads and updates (one thread), loaded
// together: one after the other they cost 2 us of a small system's iteration.
struct IterationWords {
    McsaState st;
    int status, nh;
    unsigned long long epoch, histories, tim[4];
    __device__ __forceinline__ void load(const ResidArgs& a) {
        st = *a.st;
        status = *a.status;
        nh = *a.d_nh;
        epoch = *a.d_epoch;
        histories = *a.d_hist;
        for (int k = 0; k < 4; ++k) tim[k] = a.d_tim[k];
    }
};

// The MCSA convergence check, the stream epoch, the walk timing, the work-queue
// reset and the loop condition (one thread).
__device__ __forceinline__ void end_iteration(const ResidArgs& a, IterationWords& w,
                                              double sumsq) {
    const int keep = mcsa_check(w.st, w.status, a.st, sumsq, a.hist, a.hist_cap, a.status);
    *a.d_epoch = w.epoch + 1ULL;
    *a.d_hist = w.histories + (unsigned long long)w.nh;
    add_walk_time(w.tim);
    for (int k = 0; k < 4; ++k) a.d_tim[k] = w.tim[k];
    *a.d_counter = 0;
    if (a.use_cond) cudaGraphSetConditional(a.handle, keep ? 1u : 0u);
}

// Block sum of the threads' acc, then (last block to finish) the end of the
// iteration.
__device__ __forceinline__ void norm_and_check(const ResidArgs& a, double acc) {
    __shared__ double warp_sum[32];
    const int warps = int(blockDim.x >> 5);
    __shared__ bool last;
    for (int d = 16; d > 0; d >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, d);
    if ((threadIdx.x & 31) == 0) warp_sum[threadIdx.x >> 5] = acc;
    __syncthreads();
    if (threadIdx.x == 0) {
        double t = 0.0;
        for (int w = 0; w < warps; ++w) t += warp_sum[w];
        a.part[blockIdx.x] = t;
        __threadfence();
        last = atomicAdd(a.ticket, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    IterationWords words;
    if (threadIdx.x == 0) words.load(a);
    double t = 0.0;
    for (int i = threadIdx.x; i < gridDim.x; i += blockDim.x) t += a.part[i];
    for (int d = 16; d > 0; d >>= 1) t += __shfl_down_sync(0xffffffffu, t, d);
    __syncthreads();
    if ((threadIdx.x & 31) == 0) warp_sum[threadIdx.x >> 5] = t;
    __syncthreads();
    if (threadIdx.x == 0) {
        double sumsq = 0.0;
        for (int w = 0; w < warps; ++w) sumsq += warp_sum[w];
        end_iteration(a, words, sumsq);
        *a.ticket = 0u;
    }
}

// The same for a system whose rows one cluster takes: the blocks' sums meet in
// the first block's shared memory, and its first thread has loaded the words
// before the rows.  Another block's shared memory may be written only once that
// block has started: every thread arrives at the cluster's barrier on entry
// (cluster_enter) and waits before the store, so the rows hide the wait.
constexpr int kClusterCtas = 8, kClusterThreads = 1024;
__device__ __forceinline__ void cluster_enter() {
    cooperative_groups::this_cluster().barrier_arrive();
}
__device__ __forceinline__ void norm_and_check_cluster(const ResidArgs& a, IterationWords& words,
                                                       double acc) {
    namespace cg = cooperative_groups;
    cg::cluster_group cluster = cg::this_cluster();
    __shared__ double warp_sum[kClusterThreads / 32];
    __shared__ double block_sum[kClusterCtas];
    for (int d = 16; d > 0; d >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, d);
    if ((threadIdx.x & 31) == 0) warp_sum[threadIdx.x >> 5] = acc;
    __syncthreads();
    cluster.barrier_wait();  // of cluster_enter
    if (threadIdx.x < 32) {
        double t = warp_sum[threadIdx.x];
        for (int d = 16; d > 0; d >>= 1) t += __shfl_down_sync(0xffffffffu, t, d);
        if (threadIdx.x == 0) *cluster.map_shared_rank(&block_sum[blockIdx.x], 0) = t;
    }
    cluster.sync();
    if (blockIdx.x != 0 || threadIdx.x != 0) return;
    double sumsq = 0.0;
    for (int r = 0; r < kClusterCtas; ++r) sumsq += block_sum[r];
    end_iteration(a, words, sumsq);
}

// (256, 8): eight blocks an SM, the grid's size, must be resident; with the 46
// registers that the one thread's check asks for five were, and the pass took
// 33 us at 128^3 instead of 28.9 us (k_mcsa_begin: 43 and 32.3 us).
//
// FOLD: the collision tallies of adjoint walks are normalised and added here
// (x = x2 + y / nh, formed at the neighbours as well), which saves the pass
// that did it (5 us at 64^3, 3 us at 10^4 states); the next smoothed iterate is
// then left to the next smoothing pass, since x2 is read at the neighbours.
template <bool FOLD, class Op>
__device__ __forceinline__ double residual_rows(const Op& A, const ResidArgs& a) {
    const double inv = FOLD ? *a.inv_nh : 0.0;
    auto x = [&](int j) {
        // AdjointTally::normalize: x *= 1/nh  (src/MCLS_AdjointTally_impl.hpp:68-72)
        if constexpr (FOLD) return __dadd_rn(a.x2[j], __dmul_rn(a.y[j], inv));
        else return a.x[j];
    };
    double acc = 0.0;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < a.n; i += gridDim.x * blockDim.x) {
        const double s = A.dot(i, x);
        const double res = a.b[i] - s;
        const double r = a.dinv ? a.dinv[i] * res : res;
        a.rout[i] = r;
        if constexpr (FOLD) a.x[i] = x(i);
        else a.x2[i] = __dadd_rn(x(i), __dmul_rn(a.w, r));
        acc = fma(r, r, acc);
    }
    return acc;
}
template <class Op>
__global__ void __launch_bounds__(kFusedThreads, Op::kMinBlocks) k_residual_norm(Op A, ResidArgs a) {
    norm_and_check(a, residual_rows<false>(A, a));
}
template <class Op>
__global__ void __launch_bounds__(kFusedThreads, Op::kMinBlocks) k_finalize_norm(Op A, ResidArgs a) {
    norm_and_check(a, residual_rows<true>(A, a));
}

// Small stencil systems: one cluster of eight 1024-thread CTAs.  The ticket, the
// partial sums and the words are three trips to L2 after the rows; without them
// an iteration takes 16.3 instead of 17.7 us at 77^2, 18.2 instead of 20 us at
// 90^2, 15.9 instead of 16.6 us at 18^3.  At 25^3 (two rows per thread) both
// take the same, and unstructured rows, whose gathers want more SMs, take
// longer at any size (21.3 to 22.7 us at 1500 rows).
constexpr int kClusterRows = 3 * kClusterCtas * kClusterThreads / 2;
template <class Op>
__global__ void __cluster_dims__(kClusterCtas, 1, 1) __launch_bounds__(kClusterThreads)
    k_residual_norm_cluster(Op A, ResidArgs a) {
    cluster_enter();
    IterationWords words;
    if (blockIdx.x == 0 && threadIdx.x == 0) words.load(a);
    norm_and_check_cluster(a, words, residual_rows<false>(A, a));
}
template <class Op>
__global__ void __cluster_dims__(kClusterCtas, 1, 1) __launch_bounds__(kClusterThreads)
    k_finalize_norm_cluster(Op A, ResidArgs a) {
    cluster_enter();
    IterationWords words;
    if (blockIdx.x == 0 && threadIdx.x == 0) words.load(a);
    norm_and_check_cluster(a, words, residual_rows<true>(A, a));
}

// A left preconditioner M stored on A's diagonals (learned SPAI): out = M v.
template <class Op>
__global__ void __launch_bounds__(kFusedThreads) k_dia_apply(Op M, const double* v, double* out) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < M.n; i += gridDim.x * blockDim.x)
        out[i] = M.dot(i, [&](int j) { return v[j]; });
}

// M (b - A x) in one pass, M held on A's diagonals: a block (a row per thread)
// forms the raw residual of its rows and of a halo of H = max |offset| rows on
// each side in shared memory and applies M from there.  The halo's rows are
// formed by two blocks, with the same sums, so the result is that of the two
// passes, which are launch latency while one wave of blocks holds the system.
// NORM: with the norm and the end of the iteration.  Learned SPAI on 9-point
// grids, a solve of 20 iterations: 704 -> 666 us at 128^2, 799 -> 766 at 256^2,
// 1017 -> 978 at 384^2; with a second wave slower (1271 -> 1323 at 450^2).
constexpr int kPairRows = 1024, kPairHalo = 512;
template <bool NORM, class Op>
__device__ __forceinline__ void residual_pair(const Op& A, const double* mdia, const double* x,
                                              const double* b, double* out, int halo,
                                              const ResidArgs& a) {
    __shared__ double raw[kPairRows + 2 * kPairHalo];
    const int rows = blockDim.x, r0 = blockIdx.x * rows, r1 = min(r0 + rows, A.n);
    const int lo = max(r0 - halo, 0), hi = min(r1 + halo, A.n);
#pragma unroll 2
    for (int j = lo + int(threadIdx.x); j < hi; j += rows)
        raw[j - lo] = b[j] - A.dot(j, [&](int c) { return x[c]; });
    __syncthreads();
    const int i = r0 + int(threadIdx.x);
    double acc = 0.0;
    if (i < r1) {
        const double r = dot_on_diagonals(A, mdia, i, [&](int c) { return raw[c - lo]; });
        out[i] = r;
        if (NORM) {
            a.x2[i] = __dadd_rn(x[i], __dmul_rn(a.w, r));
            acc = r * r;
        }
    }
    if (NORM) norm_and_check(a, acc);
}
template <class Op>
__global__ void __launch_bounds__(kPairRows) k_residual_pair(Op A, const double* mdia,
                                                                const double* x, const double* b,
                                                                double* out, int halo) {
    residual_pair<false>(A, mdia, x, b, out, halo, ResidArgs{});
}
template <class Op>
__global__ void __launch_bounds__(kPairRows) k_residual_pair_norm(Op A, const double* mdia,
                                                                     int halo, ResidArgs a) {
    residual_pair<true>(A, mdia, a.x, a.b, a.rout, halo, a);
}

// rp = M (b - A x) from the raw residual, its norm and the convergence check.
template <class Op>
__global__ void __launch_bounds__(kFusedThreads, 8) k_precond_norm(Op M, ResidArgs a,
                                                               const double* raw) {
    double acc = 0.0;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < a.n; i += gridDim.x * blockDim.x) {
        const double r = M.dot(i, [&](int j) { return raw[j]; });
        a.rout[i] = r;
        a.x2[i] = __dadd_rn(a.x[i], __dmul_rn(a.w, r));
        acc = fma(r, r, acc);
    }
    norm_and_check(a, acc);
}

__device__ __forceinline__ McsaState initial_state(double src_sumsq, double r_sumsq, double tol,
                                                  int check_freq, int max_iters) {
    McsaState s{};
    double sn = sqrt(src_sumsq);
    s.pad = 0;
    // Homogeneous case (:312-316)
    double crit_norm = fabs(sn) < 10.0 * 2.220446049250313e-16 ? 1.0 : sn;
    s.crit = tol * crit_norm;
    s.check_freq = check_freq > 0 ? check_freq : 1;
    s.max_iters = max_iters;
    s.iter = 0;
    s.done = 0;
    s.rnorm = sqrt(r_sumsq);
    s.converged = 0;
    return s;
}

__global__ void k_mcsa_init(McsaState* st, const double* src_sumsq, double tol, int check_freq,
                            int max_iters, const double* r_sumsq) {
    *st = initial_state(*src_sumsq, *r_sumsq, tol, check_freq, max_iters);
}

// The start of an MCSA solve with no left preconditioner or a diagonal one in
// one pass: b and x copied to the loop's vectors, rp = PL (b - A x), the
// smoothed iterate, |PL b|^2 and |rp|^2, and (last block) the loop state, the
// counters and the forward walk's history count.  Apart these were twelve
// launches and copies, 30 us of a small system's solve.
struct BeginArgs {
    const double* b_in;
    const double* x_in;
    double* b;
    double* x;
    double* x2;               // x + w rp
    double w;
    double* rp;
    const double* dinv;
    double* part;             // 2 per block
    unsigned int* ticket;
    double* sc;               // [0] and [2] forward walk, [5] |rp|^2, [6] |PL b|^2
    McsaState* st;
    double tol;
    int check_freq;
    int max_iters;
    int forward_nh;           // > 0: the forward walk's histories
    int* d_nh;
    int* d_counter;
    Counters c;
};

__device__ __forceinline__ double fused_block_sum(double v, double* sh) {
    for (int d = 16; d > 0; d >>= 1) v += __shfl_down_sync(0xffffffffu, v, d);
    __syncthreads();
    if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = v;
    __syncthreads();
    double t = 0.0;
    if (threadIdx.x == 0)
        for (int w = 0; w < kFusedThreads / 32; ++w) t += sh[w];
    return t;
}

template <class Op>
__global__ void __launch_bounds__(kFusedThreads, Op::kMinBlocks) k_mcsa_begin(Op A, BeginArgs a) {
    __shared__ double sh[kFusedThreads / 32];
    __shared__ bool last;
    double sb = 0.0, sr = 0.0;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < A.n; i += gridDim.x * blockDim.x) {
        const double s = A.dot(i, [&](int j) { return a.x_in[j]; });
        const double bi = a.b_in[i];
        const double di = a.dinv ? a.dinv[i] : 1.0;
        const double r = a.dinv ? di * (bi - s) : bi - s;
        const double pb = a.dinv ? di * bi : bi;
        a.rp[i] = r;
        if (a.b != a.b_in) a.b[i] = bi;
        const double xi = a.x_in[i];
        if (a.x != a.x_in) a.x[i] = xi;
        a.x2[i] = __dadd_rn(xi, __dmul_rn(a.w, r));
        sb = fma(pb, pb, sb);
        sr = fma(r, r, sr);
    }
    const double tb = fused_block_sum(sb, sh), tr = fused_block_sum(sr, sh);
    if (threadIdx.x == 0) {
        a.part[2 * blockIdx.x] = tb;
        a.part[2 * blockIdx.x + 1] = tr;
        __threadfence();
        last = atomicAdd(a.ticket, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    double ub = 0.0, ur = 0.0;
    for (int k = threadIdx.x; k < int(gridDim.x); k += blockDim.x) {
        ub += __ldcg(&a.part[2 * k]);
        ur += __ldcg(&a.part[2 * k + 1]);
    }
    const double src = fused_block_sum(ub, sh), res = fused_block_sum(ur, sh);
    if (threadIdx.x != 0) return;
    *a.ticket = 0u;
    a.sc[5] = res;
    a.sc[6] = src;
    *a.st = initial_state(src, res, a.tol, a.check_freq, a.max_iters);
    if (a.forward_nh > 0) {
        *a.d_nh = a.forward_nh;
        a.sc[0] = 1.0;
        a.sc[2] = 1.0 / double(a.forward_nh);
    }
    *a.d_counter = 0;
    *a.c.status = 0;
    *a.c.steps = 0;
    *a.c.hist = 0;
    a.c.tim[2] = 0;
    a.c.tim[3] = 0;
}

}  // namespace

// ---------------------------------------------------------------------------
// rp = PL (b - A PR x)
static void update_prec_residual(mclsgpu_domain* dom, const double* x, const double* b,
                                 double* rp_out) {
    cudaStream_t s = dom->ctx->stream;
    const mclsgpu_operator* op = dom->op;
    const int grid = grid_for(op->A.n, 256, 148 * 8);
    const double* xin = x;
    if (dom->right) {
        spmv(s, dom->right->P, x, dom->tmp2);
        xin = dom->tmp2;
    }
    mclsgpu_precond* L = dom->left;
    if (!L) {
        MCLSGPU_LAUNCH_OP(op, grid, 256, s, k_residual, xin, b, nullptr, rp_out);
    } else if (L->kind == MCLSGPU_PREC_POINT_JACOBI) {
        MCLSGPU_LAUNCH_OP(op, grid, 256, s, k_residual, xin, b, L->diag, rp_out);
    } else {
        MCLSGPU_LAUNCH_OP(op, grid, 256, s, k_residual, xin, b, nullptr, dom->tmp);
        spmv(s, L->P, dom->tmp, rp_out);
    }
}

void prec_residual(mclsgpu_domain* dom, const double* x, const double* b, double* rp_out) {
    update_prec_residual(dom, x, b, rp_out);
}

// y = PL A PR x  (LinearProblem::apply, src/MCLS_LinearProblem_impl.hpp:251-279)
void composite_apply(mclsgpu_domain* dom, const double* x, double* y) {
    cudaStream_t s = dom->ctx->stream;
    const mclsgpu_operator* op = dom->op;
    const int grid = grid_for(op->A.n, 256, 148 * 8);
    const double* xin = x;
    if (dom->right) {
        spmv(s, dom->right->P, x, dom->tmp2);
        xin = dom->tmp2;
    }
    mclsgpu_precond* L = dom->left;
    if (!L) {
        MCLSGPU_LAUNCH_OP(op, grid, 256, s, k_matvec, xin, nullptr, y);
    } else if (L->kind == MCLSGPU_PREC_POINT_JACOBI) {
        MCLSGPU_LAUNCH_OP(op, grid, 256, s, k_matvec, xin, L->diag, y);
    } else {
        MCLSGPU_LAUNCH_OP(op, grid, 256, s, k_matvec, xin, nullptr, dom->tmp);
        spmv(s, L->P, dom->tmp, y);
    }
}

static Counters counters(const mclsgpu_domain* dom) {
    return Counters{dom->ctx->d_status, dom->d_steps,  dom->d_hist,
                    dom->d_tim,         dom->d_state, dom->d_scalars + 6};
}

void mcsa_solve_begin(mclsgpu_domain* dom) {
    k_solve_begin<<<1, 1, 0, dom->ctx->stream>>>(counters(dom));
}

void mcsa_enqueue_report(mclsgpu_domain* dom) {
    k_report<<<1, 1, 0, dom->ctx->stream>>>(counters(dom), dom->ctx->h_report);
}

int mcsa_finish_report(mclsgpu_domain* dom, mclsgpu_stats* st) {
    const SolveReport& r = *dom->ctx->h_report;
    if (int rc = status_error(dom->ctx, r.status)) return rc;
    if (st) {
        st->walk_steps = (int64_t)r.steps;
        st->histories = (int64_t)r.hist;
        st->walk_ms = double(r.walk_ns) * 1e-6;
        st->walk_launches = (int64_t)r.launches;
    }
    return MCLSGPU_OK;
}

// One MC solve of the source vector `v` (device, already left preconditioned
// when required) into out: out = delta, out + delta or x2 + delta (`base`).
// Walks that finish their rows themselves write out; the others' tallies are
// normalised and added by k_finalize (base kBaseTally: by the caller's next
// pass).  `fused`: inside the fused MCSA iteration the epoch increment and the
// walk bookkeeping are done by k_residual_norm.
static void enqueue_mc(mclsgpu_domain* dom, const double* v, double* out, int base,
                       long long max_trace, long long* tr_states, double* tr_w, int* tr_ev,
                       long long* tr_start, bool fused = false, bool report = false) {
    const mclsgpu_mc_params& p = dom->p;
    const double omega = p.neumann_relaxation;
    const int has_omega = p.neumann_relaxation > 0.0;
    const double per = p.sample_ratio > 0.0 ? std::ceil(p.sample_ratio) : 1.0;
    const int ev = p.estimator == MCLSGPU_EXPECTED_VALUE;
    RowFinish fin;
    fin.out = out;
    fin.src = v;
    fin.xin = dom->x2;
    fin.omega = omega;
    fin.has_omega = has_omega;
    int ex = 0;
    fin.per_pow2 = std::frexp(per, &ex) == 0.5;  // per = 2^(ex-1)
    fin.inv_per = 1.0 / per;
    fin.ev = ev;
    fin.base = base;
    if (p.direction == MCLSGPU_ADJOINT)
        launch_adjoint_source(dom, v, omega, has_omega);
    else
        launch_forward_source(dom, v, omega, has_omega, fused);
    launch_walk(dom, fin, max_trace, tr_states, tr_w, tr_ev, tr_start, fused);
    launch_advance_walk_pos(dom);
    cudaStream_t s = dom->ctx->stream;
    SolveReport* const host = report ? dom->ctx->h_report : nullptr;
    if (!walk_finishes(dom) && base != kBaseTally) {
        FinalizeArgs f{};
        f.n = dom->n;
        f.mode = p.direction == MCLSGPU_FORWARD ? 2 : (ev ? 1 : 0);
        f.ev = ev;
        f.base = base;
        f.xin = dom->x2;
        f.fp32 = p.precision == MCLSGPU_FP32;
        f.per = per;
        f.sc = dom->d_scalars;
        f.src = v;
        f.omega = omega;
        f.has_omega = has_omega;
        f.y64 = dom->y64;
        f.dtrp = dom->DT.rp;
        f.dtci = dom->DT.ci;
        f.dth32 = dom->dt_h32;
        f.dth64 = dom->DT.v;
        f.out = out;
        if (!fused) {
            f.epoch = dom->d_epoch;
            f.d_nh = dom->d_nh;
            f.c = counters(dom);
            f.report = host;
            f.ticket = dom->d_ticket;
        }
        k_finalize<<<grid_for(dom->n, 256, 148 * 8), 256, 0, s>>>(f);
    } else if (!fused) {
        k_mc_end<<<1, 1, 0, s>>>(dom->d_epoch, dom->d_nh, counters(dom), host);
    }
}

// MC solve with device vectors.  host_x (may be null): pinned memory that
// receives x too.
static int mc_solve_device(mclsgpu_domain* dom, const double* rhs_dev, double* x_dev, int internal,
                           long long max_trace, long long* tr_states, double* tr_w, int* tr_ev,
                           long long* tr_start, mclsgpu_stats* stats, double* host_x = nullptr) {
    mclsgpu_context* ctx = dom->ctx;
    cudaStream_t s = ctx->stream;
    drop_stale_error();
    mcsa_solve_begin(dom);
    const double* v = rhs_dev;
    if (dom->left && !internal) {
        spmv(s, dom->left->P, rhs_dev, dom->tmp);
        v = dom->tmp;
    }
    cudaEventRecord(ctx->ev[0], s);
    // The walk's report is the last word of a solve without right recovery.
    if (dom->right && !internal) {
        // v is rhs_dev or tmp, so tmp2 is free for the unrecovered result.
        enqueue_mc(dom, v, dom->tmp2, kBaseNone, max_trace, tr_states, tr_w, tr_ev, tr_start,
                   false, true);
        spmv(s, dom->right->P, dom->tmp2, x_dev);
    } else {
        enqueue_mc(dom, v, x_dev, kBaseNone, max_trace, tr_states, tr_w, tr_ev, tr_start,
                   false, true);
    }
    cudaEventRecord(ctx->ev[1], s);
    if (host_x)
        cudaMemcpyAsync(host_x, x_dev, size_t(dom->n) * sizeof(double), cudaMemcpyDeviceToHost, s);
    cudaError_t e = cudaStreamSynchronize(s);
    if (e == cudaSuccess) e = cudaGetLastError();
    if (e != cudaSuccess) return cuda_fail(ctx, e, "mc solve");
    if (int rc = mcsa_finish_report(dom, stats)) return rc;
    if (stats) {
        float ms = 0.f;
        cudaEventElapsedTime(&ms, ctx->ev[0], ctx->ev[1]);
        stats->solve_ms = ms;
        stats->iterations = 0;
        stats->converged = 1;
    }
    return MCLSGPU_OK;
}

// x2 = x + w r (rounded as the reference's vector update)
__global__ void k_axpy_to(const double* x, const double* r, double w, double* x2, int n) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        x2[i] = __dadd_rn(x[i], __dmul_rn(w, r[i]));
}

void mc_correction(mclsgpu_domain* dom, const double* v, double* out, bool fused) {
    enqueue_mc(dom, v, out, kBaseNone, 0, nullptr, nullptr, nullptr, nullptr, fused);
}

// The fused iteration covers one smoothing step, no right preconditioner and
// a left preconditioner that is the identity or point Jacobi.
static bool fused_iteration(const mclsgpu_domain* dom, const mclsgpu_mcsa_params* mp) {
    return mp->smoother_steps == 1 && mp->fixed_point_type == MCLSGPU_FIXED_POINT_RICHARDSON &&
           !dom->right &&
           (!dom->left || dom->left->kind == MCLSGPU_PREC_POINT_JACOBI ||
            (dom->left->mdia && dom->op->dia_k > 0));
}

// The halo of residual_pair for this domain; 0: two passes.
static int pair_halo(const mclsgpu_domain* dom) {
    const mclsgpu_operator* op = dom->op;
    if (!dom->left || !dom->left->mdia || op->dia_k == 0 ||
        dom->n > dom->ctx->num_sms * kPairRows)
        return 0;
    int h = 1;
    for (int j = 0; j < op->dia_k; ++j) h = std::max(h, std::abs(op->dia_off[j]));
    return h <= kPairHalo ? h : 0;
}

// At most 8 blocks per SM: the per-block partial sums (two of them in
// k_mcsa_begin) go to dom->part, sized for that many blocks.
static int fused_grid(const mclsgpu_domain* dom) {
    return grid_for(dom->n, kFusedThreads, dom->ctx->num_sms * 8);
}

void richardson_residual(mclsgpu_domain* dom, const double* x, const double* r, double w,
                         double* x2, double* r2) {
    cudaStream_t s = dom->ctx->stream;
    const mclsgpu_operator* op = dom->op;
    const int grid = fused_grid(dom);
    const mclsgpu_precond* L = dom->left;
    if (!dom->right && (!L || L->kind == MCLSGPU_PREC_POINT_JACOBI)) {
        MCLSGPU_LAUNCH_OP(op, grid, kFusedThreads, s, k_smoothed_residual, dom->b,
                          L ? L->diag : nullptr, x, r, w, x2, r2);
    } else if (!dom->right && L->mdia && op->dia_k > 0) {
        MCLSGPU_LAUNCH_OP(op, grid, kFusedThreads, s, k_smoothed_residual, dom->b, nullptr, x, r, w,
                          x2, dom->tmp);
        MCLSGPU_LAUNCH_M(op, L->mdia, grid, kFusedThreads, s, k_dia_apply, dom->tmp, r2);
    } else {
        k_axpy_to<<<grid, kFusedThreads, 0, s>>>(x, r, w, x2, dom->n);
        update_prec_residual(dom, x2, dom->b, r2);
    }
}

// One MCSA iteration including its convergence check.  The fused form: the
// residual rp2 at the smoothed iterate x2, the source build (forward: tally
// sources into the records), the walk, which makes x = x2 + the correction (or
// k_finalize does), and residual + norm + check, which also makes the next
// iteration's x2 = x + w rp where x and rp are at hand: the smoothing pass then
// gathers one vector at the neighbours, not two, and x2 is read once.  At 128^3
// the smoothing pass takes 23.6 us (32 us with x + w rp formed at the
// neighbours) and the last pass, with x2's store, 28.9 us.  A recurrence rp2 =
// rp - w PL A rp would save 2 us more but rounds rp2 differently, which moves
// FP32 tally sources and, in adjoint domains, the history count.
static void enqueue_iteration(mclsgpu_domain* dom, const mclsgpu_mcsa_params* mp,
                              cudaGraphConditionalHandle handle, int use_cond) {
    mclsgpu_context* ctx = dom->ctx;
    cudaStream_t s = ctx->stream;
    const int n = dom->n;
    if (!fused_iteration(dom, mp)) {
        for (int l = 0; l < mp->smoother_steps; ++l)
            enqueue_fixed_point_step(dom, mp->fixed_point_type, mp->richardson_omega);
        enqueue_mc(dom, dom->rp, dom->x, kBaseOut, 0, nullptr, nullptr, nullptr, nullptr);
        update_prec_residual(dom, dom->x, dom->b, dom->rp);
        sum_sq(s, dom->rp, n, dom->part, dom->d_scalars + 5);
        if (use_cond)
            k_mcsa_check<<<1, 1, 0, s>>>(dom->d_state, dom->d_scalars + 5, dom->d_resid,
                                         dom->resid_cap, ctx->d_status, handle);
        else
            k_mcsa_check_host<<<1, 1, 0, s>>>(dom->d_state, dom->d_scalars + 5, dom->d_resid,
                                               dom->resid_cap, ctx->d_status);
        return;
    }
    const mclsgpu_operator* op = dom->op;
    const double* dinv = dom->left ? dom->left->diag : nullptr;
    // A left preconditioner on A's diagonals (learned SPAI): the raw residual
    // goes to tmp and a second pass applies M.
    const double* mdia = dom->left ? dom->left->mdia : nullptr;
    const int grid = fused_grid(dom);
    // The last pass can add the tallies itself when it needs nothing but them.
    const bool fold = !mdia && dom->p.direction == MCLSGPU_ADJOINT &&
                      dom->p.estimator == MCLSGPU_COLLISION;
    const int halo = pair_halo(dom);
    // Fewer rows per block where there are few, so that most SMs take part.
    const int pair_rows = n >= 100 * kPairRows  ? kPairRows
                          : n >= 25 * kPairRows ? kPairRows / 2
                                                : kPairRows / 4;
    const int pairs = (n + pair_rows - 1) / pair_rows;
    if (fold) {
        richardson_residual(dom, dom->x, dom->rp, mp->richardson_omega, dom->x2, dom->rp2);
    } else if (halo > 0) {
        MCLSGPU_LAUNCH_DIA(op, pairs, pair_rows, s, k_residual_pair, mdia, dom->x2, dom->b, dom->rp2,
                          halo);
    } else if (mdia) {
        MCLSGPU_LAUNCH_OP(op, grid, kFusedThreads, s, k_residual, dom->x2, dom->b, nullptr,
                          dom->tmp);
        MCLSGPU_LAUNCH_M(op, mdia, grid, kFusedThreads, s, k_dia_apply, dom->tmp, dom->rp2);
    } else {
        MCLSGPU_LAUNCH_OP(op, grid, kFusedThreads, s, k_residual, dom->x2, dom->b, dinv, dom->rp2);
    }
    enqueue_mc(dom, dom->rp2, dom->x, fold ? kBaseTally : kBaseIn, 0, nullptr, nullptr, nullptr,
               nullptr, true);
    ResidArgs a{};
    a.n = n;
    a.b = dom->b;
    a.dinv = dinv;
    a.x = dom->x;
    a.rout = dom->rp;
    a.x2 = dom->x2;
    a.w = mp->richardson_omega;
    a.y = dom->y64;
    a.inv_nh = dom->d_scalars + 2;
    a.part = dom->part;
    a.ticket = dom->d_ticket;
    a.st = dom->d_state;
    a.hist = dom->d_resid;
    a.hist_cap = dom->resid_cap;
    a.status = ctx->d_status;
    a.d_epoch = dom->d_epoch;
    a.d_tim = dom->d_tim;
    a.d_counter = dom->d_counter;
    a.d_hist = dom->d_hist;
    a.d_nh = dom->d_nh;
    a.handle = handle;
    a.use_cond = use_cond;
    if (halo > 0) {
        MCLSGPU_LAUNCH_DIA(op, pairs, pair_rows, s, k_residual_pair_norm, mdia, halo, a);
    } else if (mdia) {
        MCLSGPU_LAUNCH_OP(op, grid, kFusedThreads, s, k_residual, dom->x, dom->b, nullptr,
                          dom->tmp);
        MCLSGPU_LAUNCH_M(op, mdia, grid, kFusedThreads, s, k_precond_norm, a, dom->tmp);
    } else if (op->dia_k > 0 && n <= kClusterRows) {
        if (fold)
            MCLSGPU_LAUNCH_DIA(op, kClusterCtas, kClusterThreads, s, k_finalize_norm_cluster, a);
        else
            MCLSGPU_LAUNCH_DIA(op, kClusterCtas, kClusterThreads, s, k_residual_norm_cluster, a);
    } else if (fold) {
        MCLSGPU_LAUNCH_OP(op, grid, kFusedThreads, s, k_finalize_norm, a);
    } else {
        MCLSGPU_LAUNCH_OP(op, grid, kFusedThreads, s, k_residual_norm, a);
    }
}

void drop_loops(mclsgpu_domain* dom) {
    if (dom->graph) cudaGraphExecDestroy(dom->graph);
    dom->graph = nullptr;
    if (dom->set_graph) cudaGraphExecDestroy(dom->set_graph);
    dom->set_graph = nullptr;
    anderson_drop_graph(dom);
}

int grow_history(mclsgpu_domain* dom, int iters) {
    if (iters <= dom->resid_cap) return MCLSGPU_OK;
    cudaStreamSynchronize(dom->ctx->stream);
    drop_loops(dom);
    dom->resid_cap = 0;
    dfree(dom->d_resid);
    cudaError_t e = dmalloc(&dom->d_resid, size_t(iters));
    if (e != cudaSuccess) return cuda_fail(dom->ctx, e, "cudaMalloc residual history");
    dom->resid_cap = iters;
    return MCLSGPU_OK;
}

// Build the CUDA graph of the MCSA loop (WHILE node, one iteration per body).
static int build_mcsa_graph(mclsgpu_domain* dom, const mclsgpu_mcsa_params* mp) {
    mclsgpu_context* ctx = dom->ctx;
    cudaStream_t s = ctx->stream;
    if (dom->graph) {
        cudaGraphExecDestroy(dom->graph);
        dom->graph = nullptr;
    }
    cudaGraph_t g;
    cudaError_t e = cudaGraphCreate(&g, 0);
    if (e != cudaSuccess) return cuda_fail(ctx, e, "cudaGraphCreate");
    cudaGraphConditionalHandle handle;
    e = cudaGraphConditionalHandleCreate(&handle, g, 1, cudaGraphCondAssignDefault);
    if (e != cudaSuccess) {
        cudaGraphDestroy(g);
        return cuda_fail(ctx, e, "cudaGraphConditionalHandleCreate");
    }
    cudaGraphNodeParams np = {};
    np.type = cudaGraphNodeTypeConditional;
    np.conditional.handle = handle;
    np.conditional.type = cudaGraphCondTypeWhile;
    np.conditional.size = 1;
    cudaGraphNode_t node;
    e = cudaGraphAddNode(&node, g, nullptr, 0, &np);
    if (e != cudaSuccess) {
        cudaGraphDestroy(g);
        return cuda_fail(ctx, e, "cudaGraphAddNode(conditional)");
    }
    cudaGraph_t body = np.conditional.phGraph_out[0];
    e = cudaStreamBeginCaptureToGraph(s, body, nullptr, nullptr, 0, cudaStreamCaptureModeThreadLocal);
    if (e != cudaSuccess) {
        cudaGraphDestroy(g);
        return cuda_fail(ctx, e, "cudaStreamBeginCaptureToGraph");
    }
    enqueue_iteration(dom, mp, handle, 1);
    cudaGraph_t captured = body;
    e = cudaStreamEndCapture(s, &captured);
    if (e != cudaSuccess) {
        cudaGraphDestroy(g);
        return cuda_fail(ctx, e, "cudaStreamEndCapture");
    }
    size_t nn = 0;
    cudaGraphGetNodes(body, nullptr, &nn);
    std::vector<cudaGraphNode_t> nodes(nn);
    if (nn) cudaGraphGetNodes(body, nodes.data(), &nn);
    dom->body_kernels = 0;
    for (size_t k = 0; k < nn; ++k) {
        cudaGraphNodeType t;
        if (cudaGraphNodeGetType(nodes[k], &t) == cudaSuccess && t == cudaGraphNodeTypeKernel)
            ++dom->body_kernels;
    }
    e = cudaGraphInstantiate(&dom->graph, g, 0);
    cudaGraphDestroy(g);
    if (e != cudaSuccess) {
        dom->graph = nullptr;
        return cuda_fail(ctx, e, "cudaGraphInstantiate");
    }
    return MCLSGPU_OK;
}

// b, x0, the initial residual, the norms and the loop state; counters cleared.
// Returns the launches made.
static int mcsa_begin(mclsgpu_domain* dom, const double* b_dev, const double* x_dev,
                      const mclsgpu_mcsa_params* mp) {
    mclsgpu_context* ctx = dom->ctx;
    cudaStream_t s = ctx->stream;
    const int n = dom->n;
    const mclsgpu_operator* op = dom->op;
    const mclsgpu_precond* L = dom->left;
    const bool forward = dom->p.direction == MCLSGPU_FORWARD;
    if (fused_iteration(dom, mp) && (!L || L->kind == MCLSGPU_PREC_POINT_JACOBI)) {
        BeginArgs a{};
        a.b_in = b_dev;
        a.x_in = x_dev;
        a.b = dom->b;
        a.x = dom->x;
        a.x2 = dom->x2;
        a.w = mp->richardson_omega;
        a.rp = dom->rp;
        a.dinv = L ? L->diag : nullptr;
        a.part = dom->part;
        a.ticket = dom->d_ticket;
        a.sc = dom->d_scalars;
        a.st = dom->d_state;
        a.tol = mp->tolerance;
        a.check_freq = mp->check_freq;
        a.max_iters = mp->max_iters;
        const int per = dom->p.sample_ratio > 0.0 ? int(std::ceil(dom->p.sample_ratio)) : 1;
        a.forward_nh = forward ? n * per : 0;
        a.d_nh = dom->d_nh;
        a.d_counter = dom->d_counter;
        a.c = counters(dom);
        const int grid = fused_grid(dom);  // two partial sums per block
        MCLSGPU_LAUNCH_OP(op, grid, kFusedThreads, s, k_mcsa_begin, a);
        return 1;
    }
    mcsa_solve_begin(dom);
    // The fused iteration expects a zero work-queue counter on entry (it
    // resets it itself at the end of every iteration).
    cudaMemsetAsync(dom->d_counter, 0, sizeof(int), s);
    if (b_dev != dom->b)
        cudaMemcpyAsync(dom->b, b_dev, size_t(n) * sizeof(double), cudaMemcpyDeviceToDevice, s);
    if (x_dev != dom->x)
        cudaMemcpyAsync(dom->x, x_dev, size_t(n) * sizeof(double), cudaMemcpyDeviceToDevice, s);
    // Source norm |PL b|_2 (:299-318) and the initial preconditioned residual.
    const double* pb = dom->b;
    if (L) {
        spmv(s, L->P, dom->b, dom->tmp);
        pb = dom->tmp;
    }
    sum_sq(s, pb, n, dom->part, dom->d_scalars + 6);
    update_prec_residual(dom, dom->x, dom->b, dom->rp);
    sum_sq(s, dom->rp, n, dom->part, dom->d_scalars + 5);
    k_mcsa_init<<<1, 1, 0, s>>>(dom->d_state, dom->d_scalars + 6, mp->tolerance, mp->check_freq,
                                mp->max_iters, dom->d_scalars + 5);
    if (fused_iteration(dom, mp)) {
        k_axpy_to<<<fused_grid(dom), kFusedThreads, 0, s>>>(dom->x, dom->rp, mp->richardson_omega,
                                                            dom->x2, n);
        if (forward) launch_forward_setup(dom);
    }
    return 11;
}

static int mcsa_solve_device(mclsgpu_domain* dom, const double* b_dev, double* x_dev,
                             const mclsgpu_mcsa_params* mp, mclsgpu_stats* stats,
                             double* host_x = nullptr) {
    mclsgpu_context* ctx = dom->ctx;
    cudaStream_t s = ctx->stream;
    const int n = dom->n;
    if (int rc = grow_history(dom, mp->max_iters)) return rc;
    drop_stale_error();
    const LoopKey key{mp->richardson_omega, mp->smoother_steps, mp->fixed_point_type};
    if (int rc = prepare_fixed_point(dom, mp->fixed_point_type)) return rc;
    // Variable-length reference-stream walks synchronise with the host.
    const bool host_loop = mp->host_loop || walk_needs_rounds(dom);
    if (!host_loop && (!dom->graph || dom->graph_key != key)) {
        if (int rc = build_mcsa_graph(dom, mp)) return rc;
        dom->graph_key = key;
    }
    cudaEventRecord(ctx->ev[0], s);
    const int setup = mcsa_begin(dom, b_dev, x_dev, mp);
    cudaError_t e = cudaSuccess;
    if (!host_loop) {
        e = cudaGraphLaunch(dom->graph, s);
    } else {
        // Host-driven loop: the same iteration, one state read-back each.
        for (int it = 0; it < mp->max_iters && e == cudaSuccess; ++it) {
            enqueue_iteration(dom, mp, cudaGraphConditionalHandle(0), 0);
            cudaMemcpyAsync(dom->h_state, dom->d_state, sizeof(McsaState), cudaMemcpyDeviceToHost, s);
            e = cudaStreamSynchronize(s);
            if (e == cudaSuccess && dom->h_state->done) break;
        }
    }
    cudaEventRecord(ctx->ev[1], s);
    if (e == cudaSuccess) {
        // Right preconditioner recovery (:410-418).
        const double* xr = dom->x;
        if (dom->right) {
            spmv(s, dom->right->P, dom->x, dom->tmp);
            xr = dom->tmp;
        }
        const size_t bytes = size_t(n) * sizeof(double);
        if (x_dev != xr) cudaMemcpyAsync(x_dev, xr, bytes, cudaMemcpyDeviceToDevice, s);
        if (host_x) cudaMemcpyAsync(host_x, xr, bytes, cudaMemcpyDeviceToHost, s);
        mcsa_enqueue_report(dom);
        e = cudaStreamSynchronize(s);
    }
    if (e == cudaSuccess) e = cudaGetLastError();
    if (e != cudaSuccess) return cuda_fail(ctx, e, "mcsa graph");
    if (int rc = mcsa_finish_report(dom, stats)) return rc;
    const double src_sumsq = dom->ctx->h_report->src_sumsq;
    const McsaState st = dom->ctx->h_report->st;
    if (mp->verbose) {
        std::vector<double> hist(st.iter < dom->resid_cap ? st.iter : dom->resid_cap);
        if (!hist.empty())
            cudaMemcpy(hist.data(), dom->d_resid, hist.size() * sizeof(double), cudaMemcpyDeviceToHost);
        const double sn = std::sqrt(src_sumsq) > 0.0 ? std::sqrt(src_sumsq) : 1.0;
        std::printf("\n**************************************************\n");
        std::printf("*       MCLS: Monte Carlo Linear Solvers         *\n");
        std::printf("**************************************************\n\n");
        std::printf("                     MCSA                         \n\n");
        std::printf("%18s%18s\n", "Iteration", "|r|_2 / |b|_2");
        const int pf = mp->print_freq > 0 ? mp->print_freq : 10;
        for (int i = 0; i < (int)hist.size(); ++i)
            if ((i + 1) % pf == 0 || i + 1 == st.iter)
                std::printf("%18d%18.4e\n", i + 1, hist[i] / sn);
        std::printf("\n**************************************************\n\n");
    }
    if (stats) {
        float ms = 0.f;
        cudaEventElapsedTime(&ms, ctx->ev[0], ctx->ev[1]);
        stats->iterations = st.iter;
        stats->converged = st.converged;
        stats->residual_norm = st.rnorm;
        const double sn = std::sqrt(src_sumsq);
        stats->achieved_tol = sn > 0.0 ? st.rnorm / sn : st.rnorm;  // achievedTol (:142-173)
        stats->solve_ms = ms;
        stats->fallback_taken = dom->left ? dom->left->fallback : 0;
        // kernels of the captured iterations plus the set-up launches and the
        // report
        stats->kernel_launches = int64_t(dom->body_kernels) * st.iter + setup + 1;
        stats->rho = dom->left ? dom->left->rho : -1.0;
    }
    return MCLSGPU_OK;
}

// ---- multi-set loop pieces (multiset.cu) ------------------------------------
// Start of an MCSA loop on dom->x and dom->b: |PL b|_2, the initial
// preconditioned residual and its norm, the loop state.
void mcsa_loop_begin(mclsgpu_domain* dom, const double* b_dev, const double* x_dev,
                     const mclsgpu_mcsa_params* mp) {
    mclsgpu_context* ctx = dom->ctx;
    cudaStream_t s = ctx->stream;
    const int n = dom->n;
    mcsa_solve_begin(dom);
    if (b_dev != dom->b)
        cudaMemcpyAsync(dom->b, b_dev, size_t(n) * sizeof(double), cudaMemcpyDeviceToDevice, s);
    if (x_dev != dom->x)
        cudaMemcpyAsync(dom->x, x_dev, size_t(n) * sizeof(double), cudaMemcpyDeviceToDevice, s);
    const double* pb = dom->b;
    if (dom->left) {
        spmv(s, dom->left->P, dom->b, dom->tmp);
        pb = dom->tmp;
    }
    sum_sq(s, pb, n, dom->part, dom->d_scalars + 6);
    update_prec_residual(dom, dom->x, dom->b, dom->rp);
    sum_sq(s, dom->rp, n, dom->part, dom->d_scalars + 5);
    k_mcsa_init<<<1, 1, 0, s>>>(dom->d_state, dom->d_scalars + 6, mp->tolerance, mp->check_freq,
                                mp->max_iters, dom->d_scalars + 5);
}

// The convergence check on |rp|_2 (d_scalars[5]), ending a device-side loop
// through `handle` when use_cond.
void mcsa_loop_check(mclsgpu_domain* dom, cudaGraphConditionalHandle handle, int use_cond) {
    cudaStream_t s = dom->ctx->stream;
    if (use_cond)
        k_mcsa_check<<<1, 1, 0, s>>>(dom->d_state, dom->d_scalars + 5, dom->d_resid,
                                     dom->resid_cap, dom->ctx->d_status, handle);
    else
        k_mcsa_check_host<<<1, 1, 0, s>>>(dom->d_state, dom->d_scalars + 5, dom->d_resid,
                                           dom->resid_cap, dom->ctx->d_status);
}

// End of the loop: x_dev = PR x, the loop state and the statistics.
int mcsa_loop_finish(mclsgpu_domain* dom, double* x_dev, float ms, int kernels_per_iter,
                     mclsgpu_stats* stats) {
    mclsgpu_context* ctx = dom->ctx;
    cudaStream_t s = ctx->stream;
    const size_t bytes = size_t(dom->n) * sizeof(double);
    if (dom->right) {
        spmv(s, dom->right->P, dom->x, dom->tmp);
        cudaMemcpyAsync(x_dev, dom->tmp, bytes, cudaMemcpyDeviceToDevice, s);
    } else if (x_dev != dom->x) {
        cudaMemcpyAsync(x_dev, dom->x, bytes, cudaMemcpyDeviceToDevice, s);
    }
    mcsa_enqueue_report(dom);
    cudaError_t e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) return cuda_fail(ctx, e, "mcsa loop");
    if (int rc = mcsa_finish_report(dom, stats)) return rc;
    const McsaState st = dom->ctx->h_report->st;
    const double src_sumsq = dom->ctx->h_report->src_sumsq;
    if (stats) {
        stats->iterations = st.iter;
        stats->converged = st.converged;
        stats->residual_norm = st.rnorm;
        const double sn = std::sqrt(src_sumsq);
        stats->achieved_tol = sn > 0.0 ? st.rnorm / sn : st.rnorm;
        stats->solve_ms = ms;
        stats->fallback_taken = dom->left ? dom->left->fallback : 0;
        stats->kernel_launches = int64_t(kernels_per_iter) * st.iter;
        stats->rho = dom->left ? dom->left->rho : -1.0;
    }
    return MCLSGPU_OK;
}

}  // namespace mclsgpu

using namespace mclsgpu;

static int check_mcsa_params(mclsgpu_domain* dom, const mclsgpu_mcsa_params* p,
                             mclsgpu_mcsa_params* out);

namespace mclsgpu {
int mcsa_check_params(mclsgpu_domain* dom, const mclsgpu_mcsa_params* p,
                      mclsgpu_mcsa_params* out) {
    return check_mcsa_params(dom, p, out);
}
}  // namespace mclsgpu

static int check_mcsa_params(mclsgpu_domain* dom, const mclsgpu_mcsa_params* p,
                             mclsgpu_mcsa_params* out) {
    mclsgpu_mcsa_params d{};
    d.size = sizeof(d);
    d.max_iters = 1000;
    d.tolerance = 1.0;
    d.check_freq = 1;
    d.smoother_steps = 1;
    d.richardson_omega = 1.0;
    d.print_freq = 10;
    if (p) {
        if (p->size < sizeof(mclsgpu_mcsa_params))
            return set_error(dom->ctx, MCLSGPU_ERR_INVALID_ARG, "mcsa params: size mismatch");
        d = *p;
    }
    if (d.max_iters < 1 || d.check_freq < 1 || d.smoother_steps < 0 || !(d.tolerance >= 0.0))
        return set_error(dom->ctx, MCLSGPU_ERR_INVALID_ARG, "mcsa params out of range");
    if (d.fixed_point_type < MCLSGPU_FIXED_POINT_RICHARDSON ||
        d.fixed_point_type > MCLSGPU_FIXED_POINT_RNSD)
        return set_error(dom->ctx, MCLSGPU_ERR_INVALID_ARG, "Iteration type not supported!");
    *out = d;
    return MCLSGPU_OK;
}

extern "C" {

int mclsgpu_mc_solve_dev(mclsgpu_domain* dom, const double* rhs_dev, double* x_dev, int internal,
                         mclsgpu_stats* stats) {
    if (!dom || !rhs_dev || !x_dev) return MCLSGPU_ERR_INVALID_ARG;
    return mc_solve_device(dom, rhs_dev, x_dev, internal, 0, nullptr, nullptr, nullptr, nullptr,
                           stats);
}

int mclsgpu_mc_solve(mclsgpu_domain* dom, const double* rhs, double* x, int internal,
                     mclsgpu_stats* stats) {
    if (!dom || !rhs || !x) return MCLSGPU_ERR_INVALID_ARG;
    cudaStream_t s = dom->ctx->stream;
    const size_t bytes = size_t(dom->n) * sizeof(double);
    cudaMemcpyAsync(dom->b, rhs, bytes, cudaMemcpyHostToDevice, s);
    double* stage = dom->n <= kStageMax ? dom->ctx->h_stage : nullptr;
    int rc = mc_solve_device(dom, dom->b, dom->x, internal, 0, nullptr, nullptr, nullptr, nullptr,
                             stats, stage);
    if (rc) return rc;
    if (stage) {
        std::memcpy(x, stage, bytes);
        return MCLSGPU_OK;
    }
    cudaError_t e = cudaMemcpyAsync(x, dom->x, bytes, cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    return e == cudaSuccess ? MCLSGPU_OK : cuda_fail(dom->ctx, e, "mc_solve copy-out");
}

int mclsgpu_mc_trace(mclsgpu_domain* dom, const double* rhs, double* x, int internal,
                     int64_t max_trace, int64_t* states, double* final_weight, int32_t* events,
                     int64_t* start_state, int64_t* num_histories) {
    if (!dom || !rhs || !x || max_trace < 0) return MCLSGPU_ERR_INVALID_ARG;
    if (dom->p.precision != MCLSGPU_FP64)
        return set_error(dom->ctx, MCLSGPU_ERR_UNSUPPORTED, "trace needs the FP64 walk");
    mclsgpu_context* ctx = dom->ctx;
    cudaStream_t s = ctx->stream;
    const int L = dom->p.history_length;
    const size_t bytes = size_t(dom->n) * sizeof(double);
    long long *d_states = nullptr, *d_start = nullptr;
    double* d_w = nullptr;
    int* d_ev = nullptr;
    cudaError_t e;
    if (max_trace > 0) {
        if ((e = dmalloc(&d_states, size_t(max_trace) * (L + 1))) != cudaSuccess ||
            (e = dmalloc(&d_start, size_t(max_trace))) != cudaSuccess ||
            (e = dmalloc(&d_w, size_t(max_trace))) != cudaSuccess ||
            (e = dmalloc(&d_ev, size_t(max_trace))) != cudaSuccess) {
            dfree(d_states); dfree(d_start); dfree(d_w); dfree(d_ev);
            return cuda_fail(ctx, e, "cudaMalloc trace");
        }
    }
    cudaMemcpyAsync(dom->b, rhs, bytes, cudaMemcpyHostToDevice, s);
    int rc = mc_solve_device(dom, dom->b, dom->x, internal, max_trace, d_states, d_w, d_ev, d_start,
                             nullptr);
    if (!rc) {
        int nh = 0;
        cudaMemcpyAsync(&nh, dom->d_nh, sizeof(int), cudaMemcpyDeviceToHost, s);
        cudaMemcpyAsync(x, dom->x, bytes, cudaMemcpyDeviceToHost, s);
        e = cudaStreamSynchronize(s);
        if (e != cudaSuccess) rc = cuda_fail(ctx, e, "trace copy-out");
        if (!rc) {
            long long k = nh < max_trace ? nh : max_trace;
            if (num_histories) *num_histories = nh;
            if (k > 0) {
                if (states)
                    cudaMemcpy(states, d_states, size_t(k) * (L + 1) * sizeof(long long),
                               cudaMemcpyDeviceToHost);
                if (start_state)
                    cudaMemcpy(start_state, d_start, size_t(k) * sizeof(long long),
                               cudaMemcpyDeviceToHost);
                if (final_weight)
                    cudaMemcpy(final_weight, d_w, size_t(k) * sizeof(double), cudaMemcpyDeviceToHost);
                if (events) cudaMemcpy(events, d_ev, size_t(k) * sizeof(int), cudaMemcpyDeviceToHost);
            }
        }
    }
    dfree(d_states); dfree(d_start); dfree(d_w); dfree(d_ev);
    return rc;
}

int mclsgpu_mcsa_solve_dev(mclsgpu_domain* dom, const double* b_dev, double* x_dev,
                           const mclsgpu_mcsa_params* params, mclsgpu_stats* stats) {
    if (!dom || !b_dev || !x_dev) return MCLSGPU_ERR_INVALID_ARG;
    mclsgpu_mcsa_params p;
    int rc = check_mcsa_params(dom, params, &p);
    if (rc) return rc;
    return mcsa_solve_device(dom, b_dev, x_dev, &p, stats);
}

int mclsgpu_mcsa_begin(mclsgpu_domain* dom, const double* b_dev, const double* x0_dev,
                       const mclsgpu_mcsa_params* params, double* rnorm, double* bnorm) {
    if (!dom || !b_dev || !x0_dev) return MCLSGPU_ERR_INVALID_ARG;
    mclsgpu_mcsa_params p;
    int rc = check_mcsa_params(dom, params, &p);
    if (rc) return rc;
    mclsgpu_context* ctx = dom->ctx;
    cudaStream_t s = ctx->stream;
    const int n = dom->n;
    if ((rc = prepare_fixed_point(dom, p.fixed_point_type))) return rc;
    mcsa_solve_begin(dom);
    cudaMemsetAsync(dom->d_ticket, 0, sizeof(unsigned int), s);
    if (b_dev != dom->b) cudaMemcpyAsync(dom->b, b_dev, size_t(n) * sizeof(double), cudaMemcpyDeviceToDevice, s);
    if (x0_dev != dom->x) cudaMemcpyAsync(dom->x, x0_dev, size_t(n) * sizeof(double), cudaMemcpyDeviceToDevice, s);
    // |PL b|_2 and the initial preconditioned residual
    // (src/MCLS_MCSASolverManager_impl.hpp:299-346).
    const double* pb = dom->b;
    if (dom->left) {
        spmv(s, dom->left->P, dom->b, dom->tmp);
        pb = dom->tmp;
    }
    sum_sq(s, pb, n, dom->part, dom->d_scalars + 6);
    update_prec_residual(dom, dom->x, dom->b, dom->rp);
    sum_sq(s, dom->rp, n, dom->part, dom->d_scalars + 5);
    double h[2] = {0.0, 0.0};
    cudaMemcpyAsync(h, dom->d_scalars + 5, 2 * sizeof(double), cudaMemcpyDeviceToHost, s);
    cudaError_t e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) return cuda_fail(ctx, e, "mcsa begin");
    if ((rc = check_device_status(ctx))) return rc;
    if (rnorm) *rnorm = std::sqrt(h[0]);
    if (bnorm) *bnorm = std::sqrt(h[1]);
    dom->step_p = p;
    dom->step_ready = 1;
    return MCLSGPU_OK;
}

int mclsgpu_mcsa_correction(mclsgpu_domain* dom, double* delta_dev) {
    if (!dom || !delta_dev) return MCLSGPU_ERR_INVALID_ARG;
    mclsgpu_context* ctx = dom->ctx;
    if (!dom->step_ready)
        return set_error(ctx, MCLSGPU_ERR_INVALID_ARG, "mclsgpu_mcsa_begin first");
    cudaStream_t s = ctx->stream;
    const mclsgpu_mcsa_params& p = dom->step_p;
    for (int l = 0; l < p.smoother_steps; ++l)
        enqueue_fixed_point_step(dom, p.fixed_point_type, p.richardson_omega);
    // The residual problem's source is already left preconditioned.
    enqueue_mc(dom, dom->rp, delta_dev, kBaseNone, 0, nullptr, nullptr, nullptr, nullptr);
    cudaError_t e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) return cuda_fail(ctx, e, "mcsa correction");
    return check_device_status(ctx);
}

int mclsgpu_mcsa_apply(mclsgpu_domain* dom, const double* delta_dev, double scale,
                       double* rnorm) {
    if (!dom || !delta_dev) return MCLSGPU_ERR_INVALID_ARG;
    mclsgpu_context* ctx = dom->ctx;
    if (!dom->step_ready)
        return set_error(ctx, MCLSGPU_ERR_INVALID_ARG, "mclsgpu_mcsa_begin first");
    cudaStream_t s = ctx->stream;
    const int n = dom->n;
    k_richardson<<<grid_for(n, 256, 148 * 8), 256, 0, s>>>(dom->x, delta_dev, n, scale);
    update_prec_residual(dom, dom->x, dom->b, dom->rp);
    sum_sq(s, dom->rp, n, dom->part, dom->d_scalars + 5);
    double h = 0.0;
    cudaMemcpyAsync(&h, dom->d_scalars + 5, sizeof(double), cudaMemcpyDeviceToHost, s);
    cudaError_t e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) return cuda_fail(ctx, e, "mcsa apply");
    int rc = check_device_status(ctx);
    if (rc) return rc;
    if (!std::isfinite(h)) return set_error(ctx, MCLSGPU_ERR_DIVERGED, "non-finite residual");
    if (rnorm) *rnorm = std::sqrt(h);
    return MCLSGPU_OK;
}

int mclsgpu_mcsa_finish(mclsgpu_domain* dom, double* x_dev, mclsgpu_stats* stats) {
    if (!dom || !x_dev) return MCLSGPU_ERR_INVALID_ARG;
    mclsgpu_context* ctx = dom->ctx;
    if (!dom->step_ready)
        return set_error(ctx, MCLSGPU_ERR_INVALID_ARG, "mclsgpu_mcsa_begin first");
    cudaStream_t s = ctx->stream;
    const size_t bytes = size_t(dom->n) * sizeof(double);
    if (dom->right) {
        spmv(s, dom->right->P, dom->x, dom->tmp);  // right-preconditioner recovery
        cudaMemcpyAsync(x_dev, dom->tmp, bytes, cudaMemcpyDeviceToDevice, s);
    } else if (x_dev != dom->x) {
        cudaMemcpyAsync(x_dev, dom->x, bytes, cudaMemcpyDeviceToDevice, s);
    }
    mcsa_enqueue_report(dom);
    cudaError_t e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) return cuda_fail(ctx, e, "mcsa finish");
    dom->step_ready = 0;
    return stats ? mcsa_finish_report(dom, stats) : MCLSGPU_OK;
}

int mclsgpu_domain_residual(mclsgpu_domain* dom, double* rp_dev) {
    if (!dom || !rp_dev || !dom->rp) return MCLSGPU_ERR_INVALID_ARG;
    mclsgpu_context* ctx = dom->ctx;
    cudaError_t e = cudaMemcpyAsync(rp_dev, dom->rp, size_t(dom->n) * sizeof(double),
                                    cudaMemcpyDeviceToDevice, ctx->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(ctx->stream);
    return e == cudaSuccess ? MCLSGPU_OK : cuda_fail(ctx, e, "domain residual");
}

int mclsgpu_domain_set_launch(mclsgpu_domain* dom, int histories_per_lane, int block_size) {
    if (!dom ||
        (histories_per_lane != 1 && histories_per_lane != 2 && histories_per_lane != 4 &&
         histories_per_lane != 8) ||
        (block_size != 128 && block_size != 256))
        return MCLSGPU_ERR_INVALID_ARG;
    dom->walk_ilp = histories_per_lane;
    dom->walk_block = block_size;
    prepare_walk(dom);
    drop_loops(dom);  // the launch shape is baked into them
    return MCLSGPU_OK;
}

int mclsgpu_domain_set_record_cache(mclsgpu_domain* dom, int allocate_l1) {
    if (!dom || (allocate_l1 != 0 && allocate_l1 != 1)) return MCLSGPU_ERR_INVALID_ARG;
    dom->walk_l1 = allocate_l1;
    prepare_walk(dom);
    drop_loops(dom);  // baked into them
    return MCLSGPU_OK;
}

int mclsgpu_domain_autotune(mclsgpu_domain* dom, const double* rhs_dev, int reps,
                            int* histories_per_lane, int* block_size, double* walk_ms) {
    if (!dom || !rhs_dev || reps < 1) return MCLSGPU_ERR_INVALID_ARG;
    if (dom->p.precision != MCLSGPU_FP32)
        return set_error(dom->ctx, MCLSGPU_ERR_UNSUPPORTED, "autotune applies to FP32 walks");
    cudaStream_t s = dom->ctx->stream;
    unsigned long long saved[2] = {0, 0};
    cudaMemcpyAsync(&saved[0], dom->d_epoch, sizeof(saved[0]), cudaMemcpyDeviceToHost, s);
    cudaMemcpyAsync(&saved[1], dom->d_pos, sizeof(saved[1]), cudaMemcpyDeviceToHost, s);
    cudaError_t e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) return cuda_fail(dom->ctx, e, "autotune");
    // The shapes that differ for this domain: records in shared memory have one;
    // forward histories and those ended by a cutoff walk one per lane, and four
    // per lane apply to 32-byte records only.  Each with the record loads
    // bypassing L1 and allocated in it.
    const bool fixed = !(dom->p.weight_cutoff > 0.0);
    const bool adjoint = dom->p.direction == MCLSGPU_ADJOINT;
    const int most = !fixed || !adjoint ? 1 : dom->slots == 4 ? 4 : dom->slots == 8 ? 2 : 1;
    std::vector<std::array<int, 3>> shapes;
    for (int l1 = 0; l1 < 2; ++l1)
        for (int h = 1; h <= most; h *= 2)
            for (int block : {256, 128}) shapes.push_back({h, block, l1});
    if (walks_from_shared(dom)) shapes.resize(1);
    double best = 1e300;
    int bh = 1, bb = 256, bl = 0;
    for (const auto& sh : shapes) {
        int rc = mclsgpu_domain_set_launch(dom, sh[0], sh[1]);
        if (!rc) rc = mclsgpu_domain_set_record_cache(dom, sh[2]);
        if (rc) return rc;
        mclsgpu_stats st{};
        st.size = sizeof(st);
        rc = mc_solve_device(dom, rhs_dev, dom->tmp2, 1, 0, nullptr, nullptr, nullptr, nullptr,
                             &st);  // warm-up
        double tot = 0.0;
        for (int r = 0; r < reps && !rc; ++r) {
            rc = mc_solve_device(dom, rhs_dev, dom->tmp2, 1, 0, nullptr, nullptr, nullptr,
                                 nullptr, &st);
            tot += st.walk_ms;
        }
        if (rc) return rc;
        if (tot / reps < best) {
            best = tot / reps;
            bh = sh[0];
            bb = sh[1];
            bl = sh[2];
        }
    }
    int rc = mclsgpu_domain_set_launch(dom, bh, bb);
    if (!rc) rc = mclsgpu_domain_set_record_cache(dom, bl);
    cudaMemcpyAsync(dom->d_epoch, &saved[0], sizeof(saved[0]), cudaMemcpyHostToDevice, s);
    cudaMemcpyAsync(dom->d_pos, &saved[1], sizeof(saved[1]), cudaMemcpyHostToDevice, s);
    e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) return cuda_fail(dom->ctx, e, "autotune");
    if (histories_per_lane) *histories_per_lane = bh;
    if (block_size) *block_size = bb;
    if (walk_ms) *walk_ms = best;
    return rc;
}

int mclsgpu_mcsa_solve(mclsgpu_domain* dom, const double* b, double* x,
                       const mclsgpu_mcsa_params* params, mclsgpu_stats* stats) {
    if (!dom || !b || !x) return MCLSGPU_ERR_INVALID_ARG;
    mclsgpu_mcsa_params p;
    int rc = check_mcsa_params(dom, params, &p);
    if (rc) return rc;
    cudaStream_t s = dom->ctx->stream;
    const size_t bytes = size_t(dom->n) * sizeof(double);
    cudaMemcpyAsync(dom->b, b, bytes, cudaMemcpyHostToDevice, s);
    cudaMemcpyAsync(dom->x, x, bytes, cudaMemcpyHostToDevice, s);
    double* stage = dom->n <= kStageMax ? dom->ctx->h_stage : nullptr;
    rc = mcsa_solve_device(dom, dom->b, dom->x, &p, stats, stage);
    if (rc) return rc;
    if (stage) {
        std::memcpy(x, stage, bytes);
        return MCLSGPU_OK;
    }
    cudaError_t e = cudaMemcpyAsync(x, dom->x, bytes, cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    return e == cudaSuccess ? MCLSGPU_OK : cuda_fail(dom->ctx, e, "mcsa copy-out");
}

}  // extern "C"

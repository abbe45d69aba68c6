// source.cu -- device build of the Monte Carlo source.
//
// Adjoint (UniformAdjointSource, src/MCLS_UniformAdjointSource_impl.hpp:58-263):
//   weight = |b|_1; random sampling draws nh = int(Nh * cdf.back() / |b|_1)
//   starting states from the CDF of |b| (whose first element is the signed
//   b[0], :185) with lower_bound; stratified sampling takes
//   ceil(|b_i| * nh_local / sum|b|) histories per state.  Histories are
//   emitted from the highest state down (the LIFO stack of :157-175); the
//   emission order fixes which uniforms each history consumes in the
//   reference stream.
// Forward (UniformForwardSource, src/MCLS_UniformForwardSource_impl.hpp:60-148):
//   ceil(Sample Ratio) histories per state in state order, weight 1.
//
// Sampling uses a guide table over the FP64 CDF, one entry per 16 states:
// guide[t] is the first state whose cdf*G reaches t, so the lower_bound of u
// lies in [guide[t], guide[t+1]] with t = floor(u*G); a short binary search in
// that window returns std::lower_bound's answer.
//
// The random adjoint source of a large system is four launches: tile sums and
// the history count, CDF and guide, draws, emission.  Apart (a reduction, a
// scan of its partials and a copy for each sum, memsets, a separate
// normalisation, guide marks and a maximum scan, a pass for the tile counts)
// they were nineteen, 80 of the 107 us of an MCSA iteration at 64^3.
#include <cfloat>
#include <climits>

#include <cooperative_groups.h>

#include <mutex>

#include "internal.h"
#include "rng.cuh"
#include "scan.cuh"

namespace mclsgpu {
namespace {

using namespace scan;

inline int grid_for(long long work, int threads = 256, int cap = 148 * 16) {
    long long g = (work + threads - 1) / threads;
    if (g < 1) g = 1;
    return int(g > cap ? cap : g);
}

__device__ __forceinline__ double load_src(const double* v, int i, double omega, int has) {
    return has ? v[i] * omega : v[i];
}

// The history count nh = int(Nh_total * cdf.back() / norm1)  (:198); *error is
// set when the source sums are not finite or, since total <= norm1 in exact
// arithmetic and so nh <= nh_req <= cap, have lost all precision (a diverging
// iteration).  A zero source (an exact iterate) gets no histories.
__device__ __forceinline__ int history_count(int nh_req, double norm1, double total, int cap,
                                             bool* error) {
    const double r = __ddiv_rn(__dmul_rn(double(nh_req), total), norm1);
    int nh = (r >= 0.0 && r < 2147483647.0) ? int(r) : (r >= 2147483647.0 ? INT_MAX : 0);
    const bool finite = isfinite(norm1) && isfinite(total);
    if (!finite || !(norm1 > 0.0)) nh = 0;
    *error = !finite || nh > cap;
    return nh > cap ? cap : nh;
}

// The same with the starting weight norm1 (:67) into the solve's scalars, by
// one thread.
__device__ __forceinline__ void random_count(int nh_req, double norm1, double total, int cap,
                                             double* sc, int* d_nh, int* status) {
    bool error;
    const int nh = history_count(nh_req, norm1, total, cap, &error);
    if (error) atomicOr(status, DEV_ERR_NONFINITE);
    sc[0] = norm1;
    sc[1] = total;
    sc[2] = nh > 0 ? 1.0 / double(nh) : 0.0;
    *d_nh = nh;
}

__global__ void k_random_count(int nh_req, double* sc, int* d_nh, int cap, int* status) {
    random_count(nh_req, sc[0], sc[1], cap, sc, d_nh, status);
}

// Stratified: nh_local = ceil(Nh * local_sum / weight) (:241), and the factor
// nh_local / local_sum of the counts (:246-262) in sc[3].
__device__ __forceinline__ void strat_factor(int nh_req, double norm1, double* sc) {
    sc[0] = norm1;
    if (!(norm1 > 0.0)) {  // zero source: no histories (non-finite sums are flagged elsewhere)
        sc[3] = 0.0;
        return;
    }
    const double nh_local = ceil(__ddiv_rn(__dmul_rn(double(nh_req), norm1), norm1));
    sc[3] = __ddiv_rn(double(int(nh_local)), norm1);
}

__global__ void k_strat_prep(int nh_req, double* sc) { strat_factor(nh_req, sc[0], sc); }

// Totals of the nb tile partials with part[0] (a) and with `abs0` in its place
// (b), and the exclusive scan of the first in place.  One block.
__device__ __forceinline__ Pair scan_tiles(double* part, int nb, double abs0, Pair* warp_tot) {
    __shared__ Pair chunk;
    Pair carry{0.0, 0.0};
    for (int base = 0; base < nb; base += kThreads) {
        const int i = base + threadIdx.x;
        const double x = i < nb ? __ldcg(&part[i]) : 0.0;
        Pair excl;
        const Pair incl =
            block_scan(Pair{x, i == 0 ? abs0 : x}, AddOp(), Pair{0.0, 0.0}, warp_tot, &excl);
        if (i < nb) part[i] = carry.a + excl.a;
        if (threadIdx.x == kThreads - 1) chunk = incl;
        __syncthreads();
        carry = carry + chunk;
        __syncthreads();
    }
    return carry;
}

// True in the block that finishes last, which then sees the others' partials.
__device__ __forceinline__ bool last_block(unsigned int* ticket) {
    __shared__ bool last;
    if (threadIdx.x == 0) {
        __threadfence();
        last = atomicAdd(ticket, 1u) == gridDim.x - 1;
        if (last) *ticket = 0u;
    }
    __syncthreads();
    if (last) __threadfence();
    return last;
}

// Tile sums of the source CDF's terms (signed first element, :185) and, in the
// last block, their exclusive scan, |b|_1 (with the CDF's association, so that
// the two totals agree when b[0] >= 0), the history count or the stratified
// factor.  part has tiles + 2 entries.  Bound by latency (one tile a block,
// two round trips and the last block's scan): 5.9 us at 64^3, 11 us when the
// threads read their 8 elements from the same banks and the last block made
// two scans.
__global__ void __launch_bounds__(kThreads) k_src_reduce(const double* v, int n, double omega,
                                                         int has, int strat, int nh_req, int cap,
                                                         double* part, unsigned int* ticket,
                                                         double* sc, int* d_nh, int* status) {
    __shared__ double stage[kTile];
    __shared__ Pair warp_tot[32];
    double* const warp_totd = &warp_tot[0].a;
    const int base = blockIdx.x * kTile, nb = gridDim.x;
#pragma unroll
    for (int q = 0; q < kItems; ++q) {
        const int k = threadIdx.x + q * kThreads, i = base + k;
        const double x = i < n ? load_src(v, i, omega, has) : 0.0;
        stage[swz<8>(k)] = i == 0 ? x : fabs(x);
    }
    __syncthreads();
    const double v0 = stage[0];  // signed in block 0
    double acc = stage[swz<8>(threadIdx.x * kItems)];
#pragma unroll
    for (int k = 1; k < kItems; ++k) acc = acc + stage[swz<8>(threadIdx.x * kItems + k)];
    double excl;
    double incl = block_scan(acc, AddOp(), 0.0, warp_totd, &excl);
    if (threadIdx.x == kThreads - 1) part[blockIdx.x] = incl;
    if (blockIdx.x == 0) {
        // The first tile's sum of magnitudes.
        if (threadIdx.x == 0) {
            acc = fabs(v0);
            for (int k = 1; k < kItems; ++k) acc = acc + stage[swz<8>(k)];
        }
        incl = block_scan(acc, AddOp(), 0.0, warp_totd, &excl);
        if (threadIdx.x == kThreads - 1) part[nb + 1] = incl;
    }
    __syncthreads();
    if (!last_block(ticket)) return;
    const Pair t = scan_tiles(part, nb, __ldcg(&part[nb + 1]), warp_tot);
    if (threadIdx.x != 0) return;
    const double total = t.a, norm1 = t.b;
    part[nb] = total;
    if (strat) {
        strat_factor(nh_req, norm1, sc);
    } else {
        random_count(nh_req, norm1, total, cap, sc, d_nh, status);
    }
}

inline int guide_size(int n) { return (n + 15) / 16; }

// The CDF of a tile (cdf[i] /= cdf.back(), :201-205; the last element is set
// to exactly 1), its states' counts cleared, and the guide entries that fall
// into the tile: from the first t its lower boundary reaches to the last one
// before the next tile's.  RESCAN false: the CDF is there already (the
// reference's sequential order).  6.6 us at 64^3; 13 us with bank conflicts
// and one warp searching a tile's 128 guide entries.
template <bool RESCAN>
__global__ void __launch_bounds__(kThreads) k_src_cdf(const double* v, int n, double omega, int has,
                                                      const double* part, const double* sc,
                                                      double* cdf, int* counts, int* guide, int G,
                                                      unsigned long long* emitted) {
    __shared__ double stage[kTile];
    __shared__ double warp_tot[32];
    const int base = blockIdx.x * kTile;
    const int len = min(kTile, n - base);
    double lower, upper;  // the tile's range of the CDF
    if (threadIdx.x == 0) emitted[blockIdx.x] = 0ULL;
    if constexpr (RESCAN) {
        const double total = sc[1];
#pragma unroll
        for (int q = 0; q < kItems; ++q) {
            const int k = threadIdx.x + q * kThreads, i = base + k;
            const double x = i < n ? load_src(v, i, omega, has) : 0.0;
            stage[swz<8>(k)] = i == 0 ? x : fabs(x);
        }
        __syncthreads();
        double loc[kItems];
        loc[0] = stage[swz<8>(threadIdx.x * kItems)];
#pragma unroll
        for (int k = 1; k < kItems; ++k)
            loc[k] = loc[k - 1] + stage[swz<8>(threadIdx.x * kItems + k)];
        double excl;
        block_scan(loc[kItems - 1], AddOp(), 0.0, warp_tot, &excl);
        const double carry = part[blockIdx.x];
#pragma unroll
        for (int k = 0; k < kItems; ++k) {
            const int i = base + threadIdx.x * kItems + k;
            stage[swz<8>(threadIdx.x * kItems + k)] =
                i >= n - 1 ? 1.0 : (carry + (excl + loc[k])) / total;
        }
        __syncthreads();
        for (int k = threadIdx.x; k < len; k += kThreads) {
            cdf[base + k] = stage[swz<8>(k)];
            counts[base + k] = 0;
        }
        lower = carry / total;
        upper = part[blockIdx.x + 1] / total;
    } else {
        for (int k = threadIdx.x; k < len; k += kThreads) {
            stage[swz<8>(k)] = cdf[base + k];
            counts[base + k] = 0;
        }
        __syncthreads();
        lower = base > 0 ? cdf[base - 1] : 0.0;
        upper = stage[swz<8>(len - 1)];
    }
    // Guide entries t0..t1 of this tile (0..G over all tiles).
    const double g = double(G);
    int t0 = 0, t1 = G;
    if (blockIdx.x > 0) t0 = min(max(int(floor(lower * g)) + 1, 0), G + 1);
    if (blockIdx.x + 1 < gridDim.x) t1 = min(max(int(floor(upper * g)), -1), G);
    // First k in [lo, hi] with stage[k] * G >= t (hi when there is none).
    auto first = [&](int t, int lo, int hi) {
        while (lo < hi) {
            const int mid = (lo + hi) >> 1;
            if (stage[swz<8>(mid)] * g < double(t)) lo = mid + 1; else hi = mid;
        }
        return lo;
    };
    // One search per entry and thread; where a source is concentrated in few
    // states and the tile has many entries a warp takes 256, and a run of
    // entries inside one state is filled without searching.
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (t1 - t0 < 8 * kThreads) {
        for (int t = t0 + threadIdx.x; t <= t1; t += kThreads)
            guide[t] = base + first(t, 0, len - 1);
        return;
    }
    for (int ta = t0 + 256 * warp; ta <= t1; ta += 256 * (kThreads / 32)) {
        const int tb = min(ta + 255, t1);
        const int ka = first(ta, 0, len - 1), kb = first(tb, ka, len - 1);
        for (int t = ta + lane; t <= tb; t += 32)
            guide[t] = base + (ka == kb ? ka : first(t, ka, kb));
    }
}

// std::lower_bound(cdf, u) through the guide.
__device__ __forceinline__ int guided_lower_bound(const double* cdf, const int* guide, int n,
                                                  int G, double u) {
    int t = int(floor(u * double(G)));
    t = t < 0 ? 0 : (t > G - 1 ? G - 1 : t);
    int lo = guide[t], hi = guide[t + 1];
    if (hi < lo) hi = lo;
    while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (cdf[mid] < u) lo = mid + 1; else hi = mid;
    }
    // A tile boundary's rounding can put the window one state off.
    while (lo < n - 1 && cdf[lo] < u) ++lo;
    while (lo > 0 && cdf[lo - 1] >= u) --lo;
    return lo;
}

// Random sampling: draw k in [0, nh) -> counts[lower_bound(cdf, u_k)]++.
// Reference stream: each thread owns a contiguous run of draws and jumps once.
__global__ void k_sample(const double* cdf, const int* guide, int n, int G, const int* d_nh,
                         int rng_mode, uint64_t seed, const unsigned long long* d_epoch,
                         const uint64_t* jump, const unsigned long long* d_pos, int* counts) {
    const int nh = *d_nh;
    const uint64_t ekey = epoch_key(seed, *d_epoch);
    const int tid = blockIdx.x * blockDim.x + threadIdx.x;
    const int nthreads = gridDim.x * blockDim.x;
    if (rng_mode == MCLSGPU_RNG_COUNTER) {
        for (int k = tid; k < nh; k += nthreads) {
            uint64_t x = xs_step(counter_state(ekey, 1, uint64_t(k)));
            int j = guided_lower_bound(cdf, guide, n, G, canonical64(x));
            atomicAdd(&counts[j], 1);
        }
    } else {
        const int per = (nh + nthreads - 1) / nthreads;
        const long long k0 = (long long)tid * per;
        if (k0 >= nh) return;
        const long long k1 = k0 + per < nh ? k0 + per : nh;
        uint64_t x = xs_jump(jump, seed, *d_pos + uint64_t(k0));
        for (long long k = k0; k < k1; ++k) {
            x = xs_step(x);
            int j = guided_lower_bound(cdf, guide, n, G, canonical64(x));
            atomicAdd(&counts[j], 1);
        }
    }
}

__global__ void k_advance_pos(unsigned long long* d_pos, const int* d_nh, int mult) {
    *d_pos += (unsigned long long)(*d_nh) * (unsigned long long)mult;
}

// Stratified counts_i = ceil(|b_i| * (nh_local / local_sum)) (:246-262).
__global__ void k_strat_counts(const double* v, int n, double omega, int has, const double* sc,
                               int* counts, unsigned long long* emitted) {
    const double num_over_sum = sc[3];
    if (threadIdx.x == 0)
        for (int t = blockIdx.x; t * kTile < n; t += gridDim.x) emitted[t] = 0ULL;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        double c = ceil(__dmul_rn(fabs(load_src(v, i, omega, has)), num_over_sum));
        counts[i] = c > 0.0 ? int(c) : 0;
    }
}

// The histories of the tiles before `tile` (a warp's look-back): every tile
// publishes its own count first and, once it knows it, the count up to and
// including itself.  Tiles are numbered in the order their blocks start, so
// the ones waited for run or have run; a wait that expires all the same is
// reported and its tile's histories keep within the buffer.
constexpr unsigned long long kOwnCount = 1ULL << 62, kUpTo = 2ULL << 62;
constexpr unsigned long long kCountMask = kOwnCount - 1;

__device__ __forceinline__ long long look_back(const unsigned long long* emitted, int tile,
                                               int* status) {
    const int lane = threadIdx.x & 31;
    long long sum = 0;
    for (int at = tile - 1; at >= 0; at -= 32) {
        const int t = at - lane;
        unsigned long long w = 0ULL;
        for (int spin = 0; spin < (1 << 20); ++spin) {
            w = t >= 0 ? *reinterpret_cast<const volatile unsigned long long*>(&emitted[t])
                       : kUpTo;
            if (__all_sync(kFull, w != 0ULL)) break;
        }
        if (w == 0ULL) atomicOr(status, DEV_ERR_TIMEOUT);
        const unsigned upto = __ballot_sync(kFull, (w >> 62) == 2ULL);
        const int last = upto ? __ffs(upto) - 1 : 31;
        long long x = lane <= last ? (long long)(w & kCountMask) : 0;
#pragma unroll
        for (int d = 16; d > 0; d >>= 1) x += __shfl_xor_sync(kFull, x, d);
        sum += x;
        if (upto) break;
    }
    return sum;
}

// Emission order (highest state first, the LIFO stack of :157-175) and step-0
// collision tally in one pass over the counts: start[o_i + t] = i | sign with
// o_i the histories of the higher states, y_i = counts_i * w0_i (the tally
// every history makes at its first state).  Stratified sampling takes its
// history count from the total.  A tile's counts and sources are loaded before
// anything is stored.  Bound by the latency of those loads and of the
// look-back: 10 us at 64^3; a pass for the tile counts and one that read
// counts and sources one after the other between its stores took 9 and 13 us.
__global__ void __launch_bounds__(kThreads) k_src_emit(const double* v, int n, double omega,
                                                       int has, int strat, const int* counts,
                                                       unsigned long long* emitted,
                                                       unsigned int* ticket, double* sc, int cap,
                                                       int* start, double* y, int* d_nh,
                                                       int* status) {
    __shared__ int stage[kTile];
    __shared__ int warp_tot[32];
    __shared__ int s_tile;
    __shared__ long long s_before;
    if (threadIdx.x == 0) {
        s_tile = int(atomicAdd(ticket, 1u));
        if (s_tile == int(gridDim.x) - 1) *ticket = 0u;  // the last one to take a number
    }
    __syncthreads();
    const int tile = s_tile, base = tile * kTile;
    const double weight = sc[0];
    int ci[kItems];
    double b[kItems];
#pragma unroll
    for (int q = 0; q < kItems; ++q) {
        const int i = n - 1 - (base + int(threadIdx.x) + q * kThreads);
        ci[q] = i >= 0 ? counts[i] : 0;
        b[q] = i >= 0 ? load_src(v, i, omega, has) : 0.0;
    }
#pragma unroll
    for (int q = 0; q < kItems; ++q) stage[swz<4>(threadIdx.x + q * kThreads)] = ci[q];
    __syncthreads();
    int c[kItems], acc = 0;
#pragma unroll
    for (int k = 0; k < kItems; ++k) {
        c[k] = stage[swz<4>(threadIdx.x * kItems + k)];
        acc += c[k];
    }
    int excl;
    const int incl = block_scan(acc, AddOp(), 0, warp_tot, &excl);
    if (threadIdx.x == kThreads - 1) {
        *reinterpret_cast<volatile unsigned long long*>(&emitted[tile]) =
            (tile == 0 ? kUpTo : kOwnCount) | (unsigned long long)incl;
        warp_tot[0] = incl;
    }
    int o = excl;
#pragma unroll
    for (int k = 0; k < kItems; ++k) {
        stage[swz<4>(threadIdx.x * kItems + k)] = o;
        o += c[k];
    }
    __syncthreads();
    if (threadIdx.x < 32) {
        const long long before = tile > 0 ? look_back(emitted, tile, status) : 0;
        if (threadIdx.x == 0) {
            const long long upto = before + warp_tot[0];
            if (tile > 0)
                *reinterpret_cast<volatile unsigned long long*>(&emitted[tile]) =
                    kUpTo | (unsigned long long)upto;
            s_before = before;
            if (strat && tile == int(gridDim.x) - 1) {
                if (upto > cap) atomicOr(status, DEV_ERR_CAPACITY);
                const int nh = upto > cap ? cap : int(upto);
                *d_nh = nh;
                sc[2] = nh > 0 ? 1.0 / double(nh) : 0.0;
            }
        }
    }
    __syncthreads();
    const long long before = s_before;
#pragma unroll
    for (int q = 0; q < kItems; ++q) {
        const int k = threadIdx.x + q * kThreads, i = n - 1 - (base + k);
        if (i < 0) break;
        const unsigned sign = b[q] > 0.0 ? 0u : 0x80000000u;  // weight_sign (:169)
        double yi = 0.0;
        if (ci[q] > 0) {
            const long long at = before + stage[swz<4>(k)];
            if (at + ci[q] > cap) {
                atomicOr(status, DEV_ERR_CAPACITY);
            } else {
                for (int t = 0; t < ci[q]; ++t) start[at + t] = int(unsigned(i) | sign);
            }
            yi = double(ci[q]) * (sign ? -weight : weight);
        }
        y[i] = yi;
    }
}

// Forward tally source: c = src (collision) or H src (expected value).
template <class TC>
__global__ void k_forward_c(const double* v, int n, double omega, int has, int ev, const int* rp,
                            const int* ci, const double* h, TC* c) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        double s;
        if (!ev) {
            s = load_src(v, i, omega, has);
        } else {
            s = 0.0;
            for (int k = rp[i]; k < rp[i + 1]; ++k)
                s = fma(h[k], load_src(v, ci[k], omega, has), s);
        }
        c[i] = TC(s);
    }
}

// FP32 forward walk: the tally source of each state goes into its record's
// header word (slot 0, second word) so that a step reads one record only;
// the history-sum tallies are cleared in the same pass.
__global__ void __launch_bounds__(256) k_forward_rec(const double* v, int n, int row0,
                                                     double omega, int has, int ev,
                                                     const int* off, const int* col,
                                                     const double* h, int slots, uint2* rec,
                                                     double* y) {
    // H over SELL-32: a warp owns one slice, every entry column is one
    // coalesced access.
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        double c;
        if (!ev) {
            c = load_src(v, row0 + i, omega, has);
        } else {
            c = 0.0;
            const int o = off[i >> 5] + (i & 31), w = (off[(i >> 5) + 1] - off[i >> 5]) >> 5;
            for (int k = 0; k < w; ++k)
                c = fma(h[o + 32 * k], load_src(v, col[o + 32 * k], omega, has), c);
        }
        rec[size_t(i) * slots].y = __float_as_uint(__double2float_rn(c));
        if (y) y[i] = 0.0;
    }
}

struct StencilOffsets {
    int off[32];
};

// Stencil records: the tally source H b is rebuilt from the record itself,
// |h_j| = W * (cdf_j - cdf_prev), so the pass reads 32 bytes per row instead
// of the FP64 domain.
// Tally source of one stencil record of WORDS 32-bit words: c = sum_j h_j
// v[i + off_j] with |h_j| = W (|cdf_j| - |cdf_prev|) and the sign of slot j.
// The record is read with 256-bit loads and its first 32 bytes (W, c and the
// first CDF slots) written back with one 256-bit store.
// The source at the stencil neighbours of state i, loaded before the record
// so that both round trips overlap (an index outside [0, n) -- a neighbour
// the row does not have -- is clamped and its value never used).
template <int SLOTS>
__device__ __forceinline__ void prefetch_neighbours(const double* v, int i, int n, double omega,
                                                    int has, int K, const StencilOffsets& so,
                                                    double (&vs)[SLOTS]) {
    // Every slot is loaded (a slot past K has offset 0: the state itself), so
    // the loop unrolls and vs stays in registers.
#pragma unroll
    for (int j = 0; j < SLOTS; ++j) {
        int g = i + so.off[j];
        g = g < 0 ? 0 : (g >= n ? n - 1 : g);
        vs[j] = load_src(v, g, omega, has);
    }
}

template <int WORDS>
__device__ __forceinline__ void rec_stencil_source(uint32_t* r, int i, int n, const double* v,
                                                   double omega, int has, int K,
                                                   const StencilOffsets& so) {
    // 32-byte records: the neighbours' source loaded before the record; larger
    // records load it slot by slot after the record (their slot counts would
    // cost the registers of several resident blocks).
    constexpr bool kPre = WORDS == 8;
    double vs[kPre ? WORDS - 2 : 1];
    if constexpr (kPre) prefetch_neighbours<WORDS - 2>(v, i, n, omega, has, K, so, vs);
    uint32_t q[WORDS];
#pragma unroll
    for (int t = 0; t < WORDS / 8; ++t)
        asm volatile("ld.global.v8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                     : "=r"(q[8 * t]), "=r"(q[8 * t + 1]), "=r"(q[8 * t + 2]), "=r"(q[8 * t + 3]),
                       "=r"(q[8 * t + 4]), "=r"(q[8 * t + 5]), "=r"(q[8 * t + 6]),
                       "=r"(q[8 * t + 7])
                     : "l"(r + 8 * t));
    const float W = __uint_as_float(q[0]);
    float prev = 0.f;
    double c = 0.0;
#pragma unroll
    for (int j = 0; j < WORDS - 2; ++j) {
        if (j >= K) break;
        const float qv = __uint_as_float(q[2 + j]);
        if (isnan(qv)) continue;
        const float a = fabsf(qv);
        const float h = W * (a - prev);
        prev = a;
        double src;
        if constexpr (kPre) src = vs[j];
        else src = load_src(v, i + so.off[j], omega, has);
        c = fma(double(qv < 0.f ? -h : h), src, c);
    }
    q[1] = __float_as_uint(__double2float_rn(c));
    asm volatile("st.global.v8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"l"(r), "r"(q[0]),
                 "r"(q[1]), "r"(q[2]), "r"(q[3]), "r"(q[4]), "r"(q[5]), "r"(q[6]), "r"(q[7])
                 : "memory");
}

// The same for a stencil16 record: slot j carries |h_j| = W (t_j - t_prev) /
// 65536 (the last entry's 65535 standing for 65536), the transition
// probabilities the walk samples, and the sign in bit j of word 2.
template <int WORDS>
__device__ __forceinline__ void rec_stencil16_source(uint32_t* r, int i, int n, const double* v,
                                                     double omega, int has, int K,
                                                     const StencilOffsets& so) {
    constexpr bool kPre = WORDS == 8;
    double vs[kPre ? 2 * (WORDS - 3) : 1];
    if constexpr (kPre) prefetch_neighbours<2 * (WORDS - 3)>(v, i, n, omega, has, K, so, vs);
    uint32_t q[WORDS];
#pragma unroll
    for (int t = 0; t < WORDS / 8; ++t)
        asm volatile("ld.global.v8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                     : "=r"(q[8 * t]), "=r"(q[8 * t + 1]), "=r"(q[8 * t + 2]), "=r"(q[8 * t + 3]),
                       "=r"(q[8 * t + 4]), "=r"(q[8 * t + 5]), "=r"(q[8 * t + 6]),
                       "=r"(q[8 * t + 7])
                     : "l"(r + 8 * t));
    const float W = __uint_as_float(q[0]);
    unsigned prev = 0u;
    double c = 0.0;
#pragma unroll
    for (int j = 0; j < 2 * (WORDS - 3); ++j) {
        if (j >= K) break;
        unsigned t = (q[3 + j / 2] >> (16 * (j & 1))) & 0xffffu;
        if (t == 0u) continue;
        if (t == 65535u) t = 65536u;
        const float h = W * (float(t - prev) * 0x1p-16f);
        prev = t;
        double src;
        if constexpr (kPre) src = vs[j];
        else src = load_src(v, i + so.off[j], omega, has);
        c = fma(double(((q[2] >> j) & 1u) ? -h : h), src, c);
    }
    q[1] = __float_as_uint(__double2float_rn(c));
    asm volatile("st.global.v8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"l"(r), "r"(q[0]),
                 "r"(q[1]), "r"(q[2]), "r"(q[3]), "r"(q[4]), "r"(q[5]), "r"(q[6]), "r"(q[7])
                 : "memory");
}

// One kernel per record layout (WORDS 32-bit words, Q16: 16-bit
// thresholds), so that each keeps only its own slots' prefetched source in
// registers.
template <int WORDS, bool Q16>
__global__ void __launch_bounds__(256) k_forward_rec_stencil(const double* v, int nv, int n,
                                                             int row0, double omega, int has,
                                                             int ev, int K, StencilOffsets so,
                                                             uint32_t* rec, double* y) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        uint32_t* r = rec + size_t(i) * WORDS;
        const int g = row0 + i;  // the state's index in v
        if (!ev)
            r[1] = __float_as_uint(__double2float_rn(load_src(v, g, omega, has)));
        else if constexpr (Q16)
            rec_stencil16_source<WORDS>(r, g, nv, v, omega, has, K, so);
        else
            rec_stencil_source<WORDS>(r, g, nv, v, omega, has, K, so);
        if (y) y[i] = 0.0;
    }
}

__global__ void k_forward_nh(int* d_nh, int nh, double* sc) {
    *d_nh = nh;
    sc[0] = 1.0;
    sc[2] = 1.0 / double(nh);
}

// ---- small systems: the whole adjoint source in one cluster --------------
// For a few thousand states the multi-kernel source build is all launch
// latency.  One cluster of 8 CTAs does the same steps: every CTA forms the
// whole CDF in its shared memory (|v|_1, the reference's signed first element,
// the history count), the CTAs share the counter-stream draws and search them
// with lower_bound (the guide table only narrows that search), each CTA owns
// an eighth of the states, whose counts the others reach through distributed
// shared memory, and expands it into starting states behind the eighths above
// it (LIFO emission order).
//
// What bounds it: the chain of barriers and shared-memory round trips.  The
// warps scan 32 states at a time for all chunks of 1,024 at once and only the
// chunks' carries are serial; the searches' power-of-two probes are spread
// over the banks by a swizzle (70 us without).  The sums' association is
// fixed: it decides the truncated history count.  At 100^2 it takes 13 us of a 42 us MCSA iteration;
// one CTA with a scan per 1,024 states took 44 of 72 us.  Up to kSmallSlice
// states one CTA does it all (C = 1): the draws are then few and a cluster of 8
// costs 4 us more than it saves (a solve of 1,024 states 63 against 67 us).
constexpr int kSmallThreads = 1024;
constexpr int kSmallSourceMax = 16384;
constexpr int kSmallCtas = 8;
constexpr int kSmallSlice = kSmallSourceMax / kSmallCtas;

__device__ __forceinline__ int swizzle(int i) {
    return i ^ (((i >> 4) ^ (i >> 8) ^ (i >> 12)) & 15);
}

// Exclusive block scan of one value per thread (all 1024 threads call it);
// *total receives the sum.
template <class T>
__device__ __forceinline__ T block_scan_excl(T x, T* warp_tot, T* total) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const T y = __shfl_up_sync(0xffffffffu, x, d);
        if (lane >= d) x += y;
    }
    if (lane == 31) warp_tot[w] = x;
    __syncthreads();
    if (w == 0) {
        T t = warp_tot[lane];
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const T y = __shfl_up_sync(0xffffffffu, t, d);
            if (lane >= d) t += y;
        }
        warp_tot[lane] = t;
    }
    __syncthreads();
    T r = __shfl_up_sync(0xffffffffu, x, 1);
    if (lane == 0) r = T(0);
    if (w > 0) r += warp_tot[w - 1];
    *total = warp_tot[31];
    __syncthreads();
    return r;
}

// Inclusive scan of one value per lane.
__device__ __forceinline__ double warp_scan(double x, int lane) {
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const double y = __shfl_up_sync(0xffffffffu, x, d);
        if (lane >= d) x += y;
    }
    return x;
}

// Shared memory: the CDF (n doubles, swizzled) and the counts of the CTA's
// states (the state's sign in the top bit).
constexpr int kSmallSmem = kSmallSourceMax * sizeof(double) + kSmallSlice * sizeof(int);

template <int C>
__global__ void __cluster_dims__(C, 1, 1) __launch_bounds__(kSmallThreads)
    k_small_adjoint_source(const double* v, int n, double omega, int has, int nh_req, int cap,
                           uint64_t seed, const unsigned long long* d_epoch, int* start,
                           double* y, double* sc, int* d_nh, int* status) {
    extern __shared__ __align__(16) unsigned char smem_src[];
    double* cdf = reinterpret_cast<double*>(smem_src);
    int* counts = reinterpret_cast<int*>(smem_src + sizeof(double) * kSmallSourceMax);
    constexpr int kChunks = kSmallSourceMax / kSmallThreads;
    __shared__ double wsum[kChunks][32];   // a chunk's warp sums, then their scan
    __shared__ double wabs[32];            // chunk 0's with |v[0]|
    __shared__ double carry[kChunks + 1];
    __shared__ double s_norm1;
    __shared__ int wtoti[32];
    __shared__ int s_slice[C];
    cooperative_groups::cluster_group cluster = cooperative_groups::this_cluster();
    const int tid = threadIdx.x, rank = int(cluster.block_rank());
    const int lane = tid & 31, wid = tid >> 5;
    const int slice = (n + C - 1) / C;
    const int j0 = min(rank * slice, n), j1 = min(j0 + slice, n);  // this CTA's states
    const unsigned long long epoch = *d_epoch;
    const int chunks = (n + kSmallThreads - 1) / kSmallThreads;
    // 1. Terms of the CDF (signed first element), scanned within each warp of
    //    32 states, and the states' signs.
    constexpr int kAhead = 4;
    for (int c0 = 0; c0 < chunks; c0 += kAhead) {
        double b[kAhead];
#pragma unroll
        for (int q = 0; q < kAhead; ++q) {
            const int i = (c0 + q) * kSmallThreads + tid;
            b[q] = i < n ? load_src(v, i, omega, has) : 0.0;
        }
#pragma unroll
        for (int q = 0; q < kAhead; ++q) {
            const int c = c0 + q, i = c * kSmallThreads + tid;
            if (c >= chunks) break;
            if (i >= j0 && i < j1) counts[i - j0] = b[q] > 0.0 ? 0 : INT_MIN;
            const double x = warp_scan(i == 0 ? b[q] : fabs(b[q]), lane);
            cdf[swizzle(i)] = x;
            if (lane == 31) wsum[c][wid] = x;
            if (c == 0) {
                // The first warp's sum of magnitudes.
                const double xa = wid == 0 ? warp_scan(fabs(b[q]), lane) : x;
                if (lane == 31) wabs[wid] = xa;
            }
        }
    }
    __syncthreads();
    // 2. Scan of each chunk's warp sums, one warp per chunk.
    if (wid < chunks) wsum[wid][lane] = warp_scan(wsum[wid][lane], lane);
    if (wid == 31) wabs[lane] = warp_scan(wabs[lane], lane);
    __syncthreads();
    // 3. The chunks' carries, |v|_1 with the same association (so that it
    //    equals the CDF's total when v[0] >= 0), and the history count.
    if (tid == 0) {
        double signed_sum = 0.0, abs_sum = 0.0;
        for (int c = 0; c < chunks; ++c) {
            const double last = cdf[swizzle(c * kSmallThreads + kSmallThreads - 1)];
            carry[c] = signed_sum;
            signed_sum = (last + wsum[c][30]) + signed_sum;
            abs_sum = (last + (c == 0 ? wabs[30] : wsum[c][30])) + abs_sum;
        }
        carry[chunks] = signed_sum;
        s_norm1 = abs_sum;
        if (rank == 0) random_count(nh_req, abs_sum, signed_sum, cap, sc, d_nh, status);
    }
    __syncthreads();
    const double total = carry[chunks], norm1 = s_norm1;
    bool error;
    const int nh = history_count(nh_req, norm1, total, cap, &error);
    // 4. Normalise (cdf[n-1] = 1 exactly).
#pragma unroll 4
    for (int c = 0; c < chunks; ++c) {
        const int i = c * kSmallThreads + tid;
        if (i >= n) break;
        double x = cdf[swizzle(i)];
        if (wid > 0) x += wsum[c][wid - 1];
        x += carry[c];
        cdf[swizzle(i)] = i == n - 1 ? 1.0 : x / total;
    }
    cluster.sync();  // every CTA's counts are set
    // 5. Draw the starting states (counter stream, kind 1), two searches in
    //    flight per thread.
    const uint64_t ekey = epoch_key(seed, epoch);
    const int top = n > 1 ? 1 << (31 - __clz(n - 1)) : 0;
    constexpr int kDraws = 2, kStride = C * kSmallThreads;
    for (int k = rank * kSmallThreads + tid; k < nh; k += kDraws * kStride) {
        double u[kDraws];
        int lo[kDraws];
#pragma unroll
        for (int q = 0; q < kDraws; ++q) {
            u[q] = canonical64(xs_step(counter_state(ekey, 1, uint64_t(k + q * kStride))));
            lo[q] = 0;
        }
        // lower_bound over [0, n-1]: lo is the count of elements known < u.
        for (int half = top; half > 0; half >>= 1) {
#pragma unroll
            for (int q = 0; q < kDraws; ++q) {
                const int m = lo[q] + half;
                if (m <= n - 1 && cdf[swizzle(m - 1)] < u[q]) lo[q] = m;
            }
        }
#pragma unroll
        for (int q = 0; q < kDraws; ++q)
            if (k + q * kStride < nh) {
                const int owner = lo[q] / slice;
                atomicAdd(cluster.map_shared_rank(counts, owner) + (lo[q] - owner * slice), 1);
            }
    }
    cluster.sync();
    // 6. Emission (highest state first): a thread's run of states starts after
    //    the histories of the runs above it, a CTA's after the CTAs above it.
    constexpr int kOwn = kSmallSlice / kSmallThreads;
    const int t0 = min(j0 + tid * kOwn, j1), t1 = min(t0 + kOwn, j1);
    int mine = 0;
    for (int i = t0; i < t1; ++i) mine += counts[i - j0] & INT_MAX;
    int all;
    const int before = block_scan_excl(mine, wtoti, &all);
    if (tid < C) *cluster.map_shared_rank(&s_slice[rank], tid) = all;
    cluster.sync();
    int o = all - before - mine;
    for (int q = rank + 1; q < C; ++q) o += s_slice[q];
    for (int i = t1 - 1; i >= t0; --i) {
        const int ci = counts[i - j0], c = ci & INT_MAX;
        if (o + c > cap) {
            if (c > 0) atomicOr(status, DEV_ERR_CAPACITY);
        } else {
            for (int t = 0; t < c; ++t) start[o + t] = i | (ci & INT_MIN);
        }
        o += c;
        // Step-0 tally.
        y[i] = c > 0 ? double(c) * (ci < 0 ? -norm1 : norm1) : 0.0;
    }
}

// Dynamic shared memory opt-in for k_small_adjoint_source, once per device.
std::mutex g_small_mutex;
bool g_small_set[64] = {false};

bool small_source_ready(mclsgpu_context* ctx) {
    std::lock_guard<std::mutex> lock(g_small_mutex);
    const int d = ctx->device;
    if (d >= 0 && d < 64 && g_small_set[d]) return true;
    if (cudaFuncSetAttribute(k_small_adjoint_source<kSmallCtas>,
                             cudaFuncAttributeMaxDynamicSharedMemorySize,
                             kSmallSmem) != cudaSuccess ||
        cudaFuncSetAttribute(k_small_adjoint_source<1>,
                             cudaFuncAttributeMaxDynamicSharedMemorySize,
                             kSmallSmem) != cudaSuccess) {
        cudaGetLastError();
        return false;  // keep the multi-kernel path
    }
    if (d >= 0 && d < 64) g_small_set[d] = true;
    return true;
}

}  // namespace

// Set-up time (outside any stream capture): the small-system source kernel's
// shared-memory opt-in.
void prepare_source(mclsgpu_domain* dom) {
    if (dom->n <= kSmallSourceMax && dom->p.direction == MCLSGPU_ADJOINT)
        small_source_ready(dom->ctx);
}

// Build the adjoint source from v*omega (omega applied when has_omega).
void launch_adjoint_source(mclsgpu_domain* dom, const double* v, double omega, int has_omega) {
    mclsgpu_context* ctx = dom->ctx;
    cudaStream_t s = ctx->stream;
    const int n = dom->n;
    const mclsgpu_mc_params& p = dom->p;
    // The reproducible mode (FP64 walks on the reference stream) is the parity
    // template: |b|_1 and the source CDF follow the reference's left-to-right
    // summation order (one thread).  Every other mode uses the parallel tree
    // order, which can differ in the last bits of |b|_1 and the CDF.
    const bool parity = p.precision == MCLSGPU_FP64 && p.rng_mode == MCLSGPU_RNG_REFERENCE;
    const int nh_req = p.sample_ratio > 0.0 ? int(double(n) * p.sample_ratio) : n;
    const int cap = int(dom->nh_cap);
    if (!parity && p.rng_mode == MCLSGPU_RNG_COUNTER &&
        p.source_sampling == MCLSGPU_SOURCE_RANDOM && n <= kSmallSourceMax &&
        small_source_ready(ctx)) {
        const bool one = n <= kSmallSlice;
        auto kernel = one ? k_small_adjoint_source<1> : k_small_adjoint_source<kSmallCtas>;
        kernel<<<one ? 1 : kSmallCtas, kSmallThreads, kSmallSmem, s>>>(
            v, n, omega, has_omega, nh_req, cap, dom->seed, dom->d_epoch, dom->start, dom->y64,
            dom->d_scalars, dom->d_nh, ctx->d_status);
        return;
    }
    const bool strat = p.source_sampling != MCLSGPU_SOURCE_RANDOM;
    const int nb = tiles(n), G = guide_size(n);
    if (!parity) {
        k_src_reduce<<<nb, kThreads, 0, s>>>(v, n, omega, has_omega, strat, nh_req, cap, dom->part,
                                             dom->d_ticket, dom->d_scalars, dom->d_nh,
                                             ctx->d_status);
    } else if (strat) {
        abs_sum_sequential(s, v, n, omega, has_omega, dom->d_scalars + 0);
        k_strat_prep<<<1, 1, 0, s>>>(nh_req, dom->d_scalars);
    } else {
        source_sequential(s, v, n, omega, has_omega, dom->d_scalars + 0, dom->scdf,
                          dom->d_scalars + 1);
        k_random_count<<<1, 1, 0, s>>>(nh_req, dom->d_scalars, dom->d_nh, cap, ctx->d_status);
    }
    if (!strat) {
        auto cdf = parity ? k_src_cdf<false> : k_src_cdf<true>;
        cdf<<<nb, kThreads, 0, s>>>(v, n, omega, has_omega, dom->part, dom->d_scalars, dom->scdf,
                                    dom->counts, dom->guide, G, dom->emitted);
        const int sample_grid = p.rng_mode == MCLSGPU_RNG_COUNTER ? ctx->num_sms * 8 : 64;
        k_sample<<<sample_grid, 256, 0, s>>>(dom->scdf, dom->guide, n, G, dom->d_nh, p.rng_mode,
                                             dom->seed, dom->d_epoch, dom->d_jump, dom->d_pos,
                                             dom->counts);
        if (p.rng_mode == MCLSGPU_RNG_REFERENCE) k_advance_pos<<<1, 1, 0, s>>>(dom->d_pos, dom->d_nh, 1);
    } else {
        k_strat_counts<<<grid_for(n), 256, 0, s>>>(v, n, omega, has_omega, dom->d_scalars,
                                                   dom->counts, dom->emitted);
    }
    k_src_emit<<<nb, kThreads, 0, s>>>(v, n, omega, has_omega, strat, dom->counts, dom->emitted,
                                       dom->d_ticket, dom->d_scalars, cap, dom->start, dom->y64,
                                       dom->d_nh, ctx->d_status);
}

void launch_forward_setup(mclsgpu_domain* dom) {
    const mclsgpu_mc_params& p = dom->p;
    const int per = p.sample_ratio > 0.0 ? int(ceil(p.sample_ratio)) : 1;
    k_forward_nh<<<1, 1, 0, dom->ctx->stream>>>(dom->d_nh, dom->n * per, dom->d_scalars);
}

void launch_forward_records(mclsgpu_domain* dom, const double* v, int nv, double omega,
                            int has_omega, int row0, double* y) {
    cudaStream_t s = dom->ctx->stream;
    const int n = dom->n;
    const int ev = dom->p.estimator == MCLSGPU_EXPECTED_VALUE;
    if (dom->stencil_k) {
        StencilOffsets so{};
        for (int j = 0; j < 32; ++j) so.off[j] = dom->stencil_off[j];
        const int grid = grid_for(n, 256, 148 * 8);
        uint32_t* rec = reinterpret_cast<uint32_t*>(dom->rec);
        const int K = dom->stencil_k, words = 2 * dom->slots;
#define MCLSGPU_SRC(W, Q)                                                                 \
    k_forward_rec_stencil<W, Q><<<grid, 256, 0, s>>>(v, nv, n, row0, omega, has_omega, ev, K, \
                                                     so, rec, y)
        if (dom->rec_q16) {
            if (words == 8) MCLSGPU_SRC(8, true);
            else MCLSGPU_SRC(16, true);
        } else if (words == 8) {
            MCLSGPU_SRC(8, false);
        } else if (words == 16) {
            MCLSGPU_SRC(16, false);
        } else {
            MCLSGPU_SRC(32, false);
        }
#undef MCLSGPU_SRC
    } else {
        k_forward_rec<<<grid_for(n, 256, 148 * 8), 256, 0, s>>>(v, n, row0, omega, has_omega, ev,
                                                               dom->DS.off, dom->DS.col,
                                                               dom->DS.val, dom->slots, dom->rec,
                                                               y);
    }
}

// `fused`: the history count was set once by launch_forward_setup.
void launch_forward_source(mclsgpu_domain* dom, const double* v, double omega, int has_omega,
                           bool fused) {
    mclsgpu_context* ctx = dom->ctx;
    cudaStream_t s = ctx->stream;
    const int n = dom->n;
    const mclsgpu_mc_params& p = dom->p;
    const int per = p.sample_ratio > 0.0 ? int(ceil(p.sample_ratio)) : 1;
    const int ev = p.estimator == MCLSGPU_EXPECTED_VALUE;
    if (!fused) k_forward_nh<<<1, 1, 0, s>>>(dom->d_nh, n * per, dom->d_scalars);
    if (p.precision == MCLSGPU_FP32) {
        // Walks that finish their rows themselves read no tallies.
        launch_forward_records(dom, v, n, omega, has_omega, 0,
                               walk_finishes(dom) ? nullptr : dom->y64);
    } else {
        k_forward_c<double><<<grid_for(n), 256, 0, s>>>(v, n, omega, has_omega, ev, dom->D.rp,
                                                        dom->D.ci, dom->D.v, dom->c64);
        cudaMemsetAsync(dom->y64, 0, size_t(n) * sizeof(double), s);
    }
}

void launch_advance_walk_pos(mclsgpu_domain* dom) {
    // Variable-length histories advance the stream by their summed lengths
    // in the walk itself.
    if (dom->p.rng_mode == MCLSGPU_RNG_REFERENCE && !walk_needs_rounds(dom))
        k_advance_pos<<<1, 1, 0, dom->ctx->stream>>>(dom->d_pos, dom->d_nh, dom->p.history_length);
}

}  // namespace mclsgpu

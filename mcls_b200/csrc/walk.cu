// walk.cu -- Neumann-Ulam random-walk kernels.
//
// One history restates DomainTransporter::transport
// (src/MCLS_DomainTransporter_impl.hpp:70-119): tally at the pre-transition
// state, then AlmostOptimalDomain::processTransition
// (src/MCLS_AlmostOptimalDomain.hpp:254-284): u ~ U[0,1),
// j = lower_bound(cdf_row, u), state <- col_j, w *= W_row * sign(h_j), and
// termination once the history has taken "History Length" steps
// (:135-136) or, with the legacy "Weight Cutoff", once |w| < cutoff * |w0|.
//
// walk32_*: the production kernels.  A step reads one packed FP32 record
// (slots * 8 bytes, 32-byte vector loads), selects the first entry whose CDF
// value is >= u with predicated compares (the records' padding entries hold
// 2.0 and are never selected) and carries the weight in FP32; tallies reduce
// into FP64.  Forward histories of fixed length (walk32_rows) keep a Kahan-
// compensated FP32 sum each and the lanes of a row finish its estimate;
// adjoint histories (walk32_adjoint) tally with a fire-and-forget FP64
// reduction per step, the step-0 tally being made by the source build (counts
// * w0), so walks tally from step 1; histories ended by a weight cutoff
// (walk32_cutoff) are pulled from a work queue.  Fixed-length walks of domains
// whose records fit shared memory read them there (walk32_small).
//
// walk64: the parity kernel.  FP64 domain, std::lower_bound's selection, FP64
// weights and tallies, optional trajectory trace.  With the reference stream it
// reproduces the reference's trajectories bit for bit.
#include <algorithm>
#include <climits>

#include "internal.h"
#include "rng.cuh"

namespace mclsgpu {

struct WalkArgs {
    int n;
    int L;
    int per;                    // forward: histories per state
    int rng_mode;
    const int* d_nh;
    int* d_counter;
    const int* start;           // adjoint: state | sign<<31
    const double* sc;           // [0] weight
    float cutoff;               // relative weight cutoff (0 = off)
    double cutoff64;
    uint64_t seed;
    const unsigned long long* d_epoch;
    const uint64_t* jump;
    const unsigned long long* d_pos;
    // FP32 records
    const uint2* rec;
    // FP64 records (walk64, PACKED) and domain
    const Record64* rec64;
    const int* rp;
    const int* col;
    const double* h;
    const double* cdf;
    const double* W;
    // tallies
    double* y64;
    const double* c64;
    unsigned long long* d_steps;
    unsigned long long* d_tim;  // [0] first warp start, [1] last warp end (ns)
    int* status;
    int l1;                     // record loads allocate in L1
    int stoff[32];              // stencil records: column offset of each slot
    // variable-length histories on the reference stream (FP64 only): history
    // e's first draw is *d_pos + hoff[e]; hlen[e] receives its length
    const int* hoff;
    int* hlen;
    // trace (FP64 only)
    long long max_trace;
    long long* tr_states;
    double* tr_w;
    int* tr_ev;
    long long* tr_start;
};

namespace {

constexpr unsigned kFull = 0xffffffffu;

// 256-bit read-only load of half a record, not allocated in L1 (records are
// read once per step and reused across steps only through L2).
__device__ __forceinline__ void ld_record256(const void* p, uint32_t* r) {
    asm volatile(
        "ld.global.nc.L1::no_allocate.v8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
          "=r"(r[7])
        : "l"(p));
}
// The same load allocated in L1: histories of one block start at neighbouring
// states and step to neighbours, so their records are often fetched again by
// the block's other warps.
__device__ __forceinline__ void ld_record256_l1(const void* p, uint32_t* r) {
    asm volatile(
        "ld.global.nc.v8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
          "=r"(r[7])
        : "l"(p));
}

__device__ __forceinline__ unsigned long long global_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

__device__ __forceinline__ uint64_t history_state(const WalkArgs& a, uint64_t ekey, long long e) {
    if (a.rng_mode == MCLSGPU_RNG_COUNTER) return counter_state(ekey, 2, uint64_t(e));
    const uint64_t off = a.hoff ? uint64_t(a.hoff[e]) : uint64_t(e) * uint64_t(a.L);
    return xs_jump(a.jump, a.seed, *a.d_pos + off);
}

// Small records (up to 8 slots) run at full occupancy: 8 blocks of 256 threads
// per SM, i.e. at most 32 registers per thread; packed ones up to 16 slots,
// read in halves, at six blocks.  The per-launch constants
// that are only needed when a lane takes a new history (history count,
// stream key, starting weight) live in shared memory, not registers.
template <int S, int ST>
struct WalkOccupancy {
    static constexpr int kMinBlocks = S <= 8 ? 8 : (S <= 16 && ST == 0) ? 6 : (S <= 24 ? 4 : 2);
};

// Record kinds of the FP32 walk (template parameter ST).
//   0 packed:      slot 0 = {W, len or tally source}, slots 1.. = {cdf (f32),
//                  column | sign << 31}, padding CDF 2.0
//   1 stencil:     word 0 = W, word 1 = tally source, word 2 + j = the CDF at
//                  column offset off[j] with the sign of h_j in its sign bit,
//                  NaN where the row has no entry at that offset
//   2 stencil16:   word 0 = W, word 1 = tally source, word 2 = the signs of
//                  h_j (bit j), then 16-bit thresholds t_j two to a word
//                  (slot j in word 3 + j/2, bits 16 (j % 2)..): t_j =
//                  round(65536 cdf_j), 65535 for the row's last entry, 0 where
//                  the row has no entry at off[j]
constexpr int kPacked = 0, kStencil = 1, kStencil16 = 2;

// Selection in one FP32 record (the S-slot words q of state s) for the draw
// x: the first entry whose CDF value is >= u (sampleDiscreteCDF's
// lower_bound) with u the draw's 24-bit uniform, or for stencil16 the first
// slot with u16 < t_j, u16 = min(top 16 bits, 65534).  s becomes the selected
// column; neg is the sign bit of the selected h.  The slots are scanned from
// the last to the first, each match overwriting the one before, so a slot
// costs a compare and a predicated move and no "found" flag.  POS: the domain
// has no negative h, so the sign is not read.  soff: the column offsets of the
// stencil slots in shared memory, soff[kNoSlot] = 0 (no slot matched: a NaN
// record, reported by the residual check).
constexpr int kNoSlot = 31;
// Slots A .. B-1 of a packed record: the selected entry's column and sign.
template <int A, int B>
__device__ __forceinline__ unsigned select_packed(const uint32_t* q, float u) {
    unsigned sel = 0u;
#pragma unroll
    for (int t = B - 1; t >= A; --t)
        if (__uint_as_float(q[2 * t]) >= u) sel = q[2 * t + 1];
    return sel;
}
template <int S, int ST, bool POS = false>
__device__ __forceinline__ void select32(const int* soff, const uint32_t* q, uint64_t x, int& s,
                                         unsigned& neg) {
    if constexpr (ST == kPacked) {
        const unsigned sel = select_packed<1, S>(q, canonical32(x));
        neg = sel & 0x80000000u;
        s = int(sel & 0x7fffffffu);
    } else if constexpr (ST == kStencil) {
        // Stencil slots: first |cdf_j| >= u (NaN slots never match); the next
        // state is s + offset_j, the sign of h_j is the sign bit of the slot.
        const float u = canonical32(x);
        int jsel = kNoSlot;
        unsigned ng = 0u;
#pragma unroll
        for (int j = 2 * S - 3; j >= 0; --j)
            if (fabsf(__uint_as_float(q[2 + j])) >= u) {
                jsel = j;
                if constexpr (!POS) ng = q[2 + j];
            }
        neg = ng & 0x80000000u;
        s += soff[jsel];
    } else {
        // A slot's threshold is compared inside its word: the high half
        // against (u16 << 16 | 0xffff), the low half after a shift.
        const unsigned u16 = min(unsigned(x >> 48), 65534u);
        const unsigned top = (u16 << 16) | 0xffffu;
        int jsel = kNoSlot;
#pragma unroll
        for (int j = 2 * (2 * S - 3) - 1; j >= 0; --j) {
            const unsigned word = q[3 + j / 2];
            if ((j & 1) ? word > top : (word << 16) > top) jsel = j;
        }
        neg = POS ? 0u : ((q[2] >> jsel) & 1u) << 31;
        s += soff[jsel];
    }
}

// Selection in the FP64 domain row of state s for the uniform u
// (std::lower_bound over the row's CDF, as the reference samples it).
// Returns the entry index within the row; the caller checks it is < len.
__device__ __forceinline__ int select64(const WalkArgs& a, int s, double u, int& r0, int& len) {
    r0 = a.rp[s];
    len = a.rp[s + 1] - r0;
    int lo = 0, hi = len;
    while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (a.cdf[r0 + mid] < u) lo = mid + 1; else hi = mid;
    }
    return lo;
}

// The same transition from a packed record: the CDF does not fall along a row,
// so std::lower_bound's position is the number of values below u.
__device__ __forceinline__ void select_record64(const Record64* rec, int s, double u, double& Ws,
                                                int& col, int* status) {
    uint32_t q[24];
#pragma unroll
    for (int t = 0; t < 3; ++t)
        ld_record256(reinterpret_cast<const char*>(rec + s) + 32 * t, q + 8 * t);
    int lo = 0;
#pragma unroll
    for (int j = 0; j < Record64::kEntries; ++j)
        lo += __hiloint2double(int(q[3 + 2 * j]), int(q[2 + 2 * j])) < u;
    const int len = int(q[23] & 0xffu);
    if (lo >= len) {
        atomicOr(status, DEV_ERR_BOUNDS);
        lo = len - 1;
    }
    col = int(q[16]);
#pragma unroll
    for (int j = 1; j < Record64::kEntries; ++j) col = lo == j ? int(q[16 + j]) : col;
    const double W = __hiloint2double(int(q[1]), int(q[0]));
    Ws = (q[23] >> (8 + lo)) & 1u ? -W : W;
}

// Slots of a record that every step reads.  Packed records longer than 64 bytes
// are read in two parts: the walk is bound by the sectors it requests, so what
// lies past the seventh entry is read only by the lanes whose draw lies there (the
// CDF does not fall along a row and its padding holds 2.0), and with the
// registers this frees six blocks are resident instead of four.  It gives the
// more the fewer rows are long, and costs nothing where all are: solves of 8
// iterations on 60,007 rows of 8, 12, 16, 24 and 30 entries each take 293, 337,
// 398, 528 and 568 us, with whole records 323, 382, 464, 567 and 572; 2 x 10^5
// histories on 10^5 rows of 7 entries on average and 16 at most 22 and 34.4 us.
template <int S, int ST>
constexpr int first_slots() {
    return ST == kPacked && S > 8 ? 8 : S;
}

// Where a step finds the records: global memory past L1 or allocating in it, or
// the block's copy in shared memory.
enum : int { kBypass = 0, kCached = 1, kShared = 2 };

template <int S, int MEM>
__device__ __forceinline__ void load_slots(const char* r, uint32_t* q) {
#pragma unroll
    for (int t = 0; t < S / 4; ++t) {
        if constexpr (MEM == kShared) {
            const uint4 u = *reinterpret_cast<const uint4*>(r + 32 * t);
            const uint4 v = *reinterpret_cast<const uint4*>(r + 32 * t + 16);
            q[8 * t] = u.x, q[8 * t + 1] = u.y, q[8 * t + 2] = u.z, q[8 * t + 3] = u.w;
            q[8 * t + 4] = v.x, q[8 * t + 5] = v.y, q[8 * t + 6] = v.z, q[8 * t + 7] = v.w;
        } else if constexpr (MEM == kCached) {
            ld_record256_l1(r + 32 * t, q + 8 * t);
        } else {
            ld_record256(r + 32 * t, q + 8 * t);
        }
    }
}

// One transition of a history at state s (DomainTransporter::transport's
// loop body): tally at the pre-transition state, read the state's record,
// draw u, select the first entry whose CDF value is >= u, update the state
// and the weight.
//
template <int S, int DIR, int ST, int MEM, bool POS = false>
__device__ __forceinline__ void walk_step(const char* rec, double* y, const int* soff, int& s,
                                          float& w, uint64_t& x, float& acc, float& comp, int k) {
    // One record: S/4 256-bit loads.  rec and y point at global row 0.  Long
    // packed records: the first 64 bytes (7 entries), the others only when u lies
    // past them.
    constexpr int kFirst = first_slots<S, ST>();
    const char* r = rec + size_t(unsigned(s)) * (S * 8);
    uint32_t q[2 * kFirst];
    load_slots<kFirst, MEM>(r, q);
    if (DIR == MCLSGPU_ADJOINT) {
        // FP32 weight, FP64 reduction (fire-and-forget RED.ADD.F64).
        if (k > 0) atomicAdd(&y[s], double(w));
    } else {
        // Kahan-compensated FP32 history sum; the tally source of the state
        // rides in the record header (slot 0, second word).
        const float term = w * __uint_as_float(q[1]) - comp;
        const float t = acc + term;
        comp = (t - acc) - term;
        acc = t;
    }
    x = xs_step(x);
    const float Wt = __uint_as_float(q[0]);
    unsigned neg;
    if constexpr (kFirst < S) {
        const float u = canonical32(x);
        unsigned sel;
        if (__uint_as_float(q[2 * (kFirst - 1)]) >= u) {
            sel = select_packed<1, kFirst>(q, u);
        } else {
            uint32_t z[2 * (S - kFirst)];
            load_slots<S - kFirst, MEM>(r + kFirst * 8, z);
            sel = select_packed<0, S - kFirst>(z, u);
        }
        neg = sel & 0x80000000u;
        s = int(sel & 0x7fffffffu);
    } else {
        select32<S, ST, POS>(soff, q, x, s, neg);
    }
    w = __uint_as_float(__float_as_uint(w * Wt) ^ neg);
}

// Starting state, weight and stream of history e.
template <int DIR>
__device__ __forceinline__ void walk_start(const WalkArgs& a, int e, uint64_t ekey, float wnorm,
                                           int& s, float& w, uint64_t& x) {
    if (DIR == MCLSGPU_ADJOINT) {
        const int sv = a.start[e];
        s = sv & 0x7fffffff;
        w = sv < 0 ? -wnorm : wnorm;
    } else {
        s = e / a.per;
        w = 1.f;
    }
    x = history_state(a, ekey, e);
}

// The column offsets of the record's slots in shared memory.
__device__ __forceinline__ void stage_offsets(const int* stoff, int* soff) {
    if (threadIdx.x < 32) soff[threadIdx.x] = threadIdx.x < kNoSlot ? stoff[threadIdx.x] : 0;
}

// First block start and last block end of a walk launch (d_tim): one atomic
// each per block, not per warp, because they all meet at the same address.
__device__ __forceinline__ void walk_begin_time(const WalkArgs& a) {
    if (threadIdx.x == 0) atomicMin(&a.d_tim[0], global_ns());
}
__device__ __forceinline__ void walk_end_time(const WalkArgs& a) {
    __syncthreads();
    if (threadIdx.x == 0) atomicMax(&a.d_tim[1], global_ns());
}

// All of a small domain's records in the block's shared memory, fetched with
// bulk copies.
struct RecordCopy {
    const char* rec;
    uint32_t bar;  // mbarrier (shared-memory address)

    // One thread: start the copies (dst: 16-byte aligned shared memory).
    __device__ __forceinline__ void start(const void* src, int bytes) const {
        const uint32_t dst = uint32_t(__cvta_generic_to_shared(rec));
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar),
                     "r"(bytes)
                     : "memory");
        constexpr int kChunk = 16 * 1024;
        for (int at = 0; at < bytes; at += kChunk)
            asm volatile(
                "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, "
                "[%3];" ::"r"(dst + at),
                "l"(reinterpret_cast<const char*>(src) + at), "r"(min(kChunk, bytes - at)), "r"(bar)
                : "memory");
    }
    // True once the records are there; false (and reported) when the wait
    // expires.
    __device__ __forceinline__ bool wait(int* status) const {
        for (int spin = 0; spin < (1 << 22); ++spin) {
            uint32_t done;
            asm volatile(
                "{\n.reg .pred p;\n"
                "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], 0;\n"
                "selp.u32 %0, 1, 0, p;\n}"
                : "=r"(done)
                : "r"(bar)
                : "memory");
            if (done) return true;
        }
        atomicOr(status, DEV_ERR_TIMEOUT);
        return false;
    }
};

// What bounds it: 8,850 warp steps per SM for 41.9M steps (128^3, two
// histories per row), and the loads' L1TEX cycles -- a warp's 32 records lie in
// up to 32 different lines, one request to L2 each.  So the lanes of a warp
// start in a brick of neighbouring rows (RowOrder) and the two histories of a
// row sit in the same warp, which keeps them in fewer lines for longer: 26.8
// lines per request for 32 rows along x, 20.3 for 4 x 2 x 2 rows with two
// histories each, and 124 against 114 us for the launch.  Loads that allocate
// in L1 hit 80 % of the time and are slower (139 us): their data-stage
// wavefronts then bind.  Further histories per lane add no speed (137 us with
// one, 145 with two and four before the bricks): 64 resident warps already
// cover the latency.  With the work queue, the per-warp timing atomics and
// the tallies in memory the launch took 145 us at its tuned shape (213 us at
// the default one), and 15 us instead of 4.8 for a 20^3 grid.
//
// Forward histories of fixed length, one per thread at a time.  2^f.hlog
// neighbouring lanes share a row and split its `per` histories; they add
// their sums with shuffles and the first of them finishes the row's estimate,
// out = [base +] sum / per [+ source], so a row's sum needs no atomics, no
// cleared tally and no pass of its own.  The histories are assigned
// statically: they all take the same number of steps, and a work queue costs
// one contended atomic per warp.  The histories from m0 on in steps of `step`.
template <int S, int ST, bool POS, int MEM>
__device__ __forceinline__ double row_histories(const WalkArgs& a, int m0, int step,
                                                const int* soff, uint64_t ekey, int row,
                                                const RecordCopy& copy) {
    const char* rec = reinterpret_cast<const char*>(a.rec);
    const int L = a.L;
    double sum = 0.0;
    for (int m = m0; m < a.per; m += step) {
        int s = row, k = 0;
        float w = 1.f, acc = 0.f, comp = 0.f;
        uint64_t x = history_state(a, ekey, (long long)row * a.per + m);
        if constexpr (MEM == kShared) {
            // The first record from memory, while the others are on their way.
            walk_step<S, MCLSGPU_FORWARD, ST, kBypass, POS>(rec, nullptr, soff, s, w, x, acc, comp,
                                                            k++);
            if (!copy.wait(a.status)) return 0.0;
        }
        const char* from = MEM == kShared ? copy.rec : rec;
        for (; k < L; ++k)
            walk_step<S, MCLSGPU_FORWARD, ST, MEM, POS>(from, nullptr, soff, s, w, x, acc, comp, k);
        sum += double(acc) - double(comp);
    }
    return sum;
}

// The row's estimate from its histories' sums (one per lane of the row).
__device__ __forceinline__ void finish_row(const WalkArgs& a, const RowFinish& f, double sum, int i,
                                           bool live) {
    for (int d = 1; d < (1 << f.hlog); d <<= 1) sum += __shfl_xor_sync(kFull, sum, d);
    if (!live || (threadIdx.x & ((1 << f.hlog) - 1)) != 0) return;
    // sum / count (ForwardTally::finalize, src/MCLS_ForwardTally_impl.hpp:
    // 194-208); for a power-of-two count the product with its reciprocal
    // is the same number.
    double d = f.per_pow2 ? sum * f.inv_per : __ddiv_rn(sum, double(a.per));
    if (f.ev) d = __dadd_rn(d, f.has_omega ? f.src[i] * f.omega : f.src[i]);
    if (f.base == kBaseOut)
        d = __dadd_rn(f.out[i], d);
    else if (f.base == kBaseIn)
        d = __dadd_rn(f.xin[i], d);
    f.out[i] = d;
}

template <int S, int ST, bool POS>
__global__ void __launch_bounds__(256, WalkOccupancy<S, ST>::kMinBlocks)
    walk32_rows(WalkArgs a, RowFinish f) {
    static_assert(S % 4 == 0, "records are whole 32-byte halves");
    __shared__ uint64_t s_ekey;
    __shared__ int s_off[32];
    stage_offsets(a.stoff, s_off);
    if (threadIdx.x == 0) s_ekey = epoch_key(a.seed, *a.d_epoch);
    walk_begin_time(a);
    __syncthreads();
    const unsigned pos = (blockIdx.x * blockDim.x + threadIdx.x) >> f.hlog;
    // A position past the end walks the last row's histories and drops the
    // result, so every lane takes part in the shuffles.
    const bool live = pos < unsigned(a.n);
    const unsigned p = live ? pos : unsigned(a.n) - 1u;
    const int i = f.order ? f.order[p] : int(p);
    const RecordCopy none{};
    const int H = 1 << f.hlog, m0 = threadIdx.x & (H - 1);
    const double sum = a.l1 ? row_histories<S, ST, POS, kCached>(a, m0, H, s_off, s_ekey, i, none)
                            : row_histories<S, ST, POS, kBypass>(a, m0, H, s_off, s_ekey, i, none);
    finish_row(a, f, sum, i, live);
    if (blockIdx.x == 0 && threadIdx.x == 0)
        atomicAdd(a.d_steps, (unsigned long long)(a.n) * a.per * a.L);
    walk_end_time(a);
}

// The same where a warp per row leaves the chip idle (few rows, many histories
// each): f.split warps share a row and add their sums into its tally, which
// the finalizing pass reads.
template <int S, int ST>
__global__ void __launch_bounds__(256, WalkOccupancy<S, ST>::kMinBlocks)
    walk32_split(WalkArgs a, RowFinish f) {
    __shared__ uint64_t s_ekey;
    __shared__ int s_off[32];
    stage_offsets(a.stoff, s_off);
    if (threadIdx.x == 0) s_ekey = epoch_key(a.seed, *a.d_epoch);
    walk_begin_time(a);
    __syncthreads();
    const unsigned warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int i = int(warp / unsigned(f.split));
    if (i < a.n) {  // the same in every lane of a warp
        const RecordCopy none{};
        const int lane = threadIdx.x & 31, m0 = int(warp % unsigned(f.split)) * 32 + lane;
        const int step = 32 * f.split;
        double sum =
            a.l1 ? row_histories<S, ST, false, kCached>(a, m0, step, s_off, s_ekey, i, none)
                 : row_histories<S, ST, false, kBypass>(a, m0, step, s_off, s_ekey, i, none);
        for (int d = 16; d > 0; d >>= 1) sum += __shfl_xor_sync(kFull, sum, d);
        if (lane == 0) atomicAdd(&a.y64[i], sum);
    }
    if (blockIdx.x == 0 && threadIdx.x == 0)
        atomicAdd(a.d_steps, (unsigned long long)(a.n) * a.per * a.L);
    walk_end_time(a);
}

// Adjoint histories of fixed length, ILP per lane, assigned statically (see
// walk32_rows); they tally where they stand.
template <int S, int ST, bool POS, int MEM, int ILP>
__device__ __forceinline__ void adjoint_histories(const WalkArgs& a, const int* soff,
                                                  uint64_t ekey, float wnorm, long long e0,
                                                  int nh, const RecordCopy& copy) {
    const char* rec = reinterpret_cast<const char*>(a.rec);
    const int L = a.L;
    int s[ILP];
    float w[ILP];
    uint64_t x[ILP];
#pragma unroll
    for (int m = 0; m < ILP; ++m) {
        const long long e = e0 + (long long)m * blockDim.x;
        s[m] = 0;
        w[m] = 0.f;
        x[m] = 0;
        if (e < nh) walk_start<MCLSGPU_ADJOINT>(a, int(e), ekey, wnorm, s[m], w[m], x[m]);
    }
    int k = 0;
    if constexpr (MEM == kShared) {
        static_assert(ILP == 1, "one history per lane");
        float acc = 0.f, comp = 0.f;
        walk_step<S, MCLSGPU_ADJOINT, ST, kBypass, POS>(rec, a.y64, soff, s[0], w[0], x[0], acc,
                                                        comp, k++);
        if (!copy.wait(a.status)) return;
        rec = copy.rec;
    }
    for (; k < L; ++k) {
#pragma unroll
        for (int m = 0; m < ILP; ++m) {
            float acc = 0.f, comp = 0.f;
            if (e0 + (long long)m * blockDim.x < nh)
                walk_step<S, MCLSGPU_ADJOINT, ST, MEM, POS>(rec, a.y64, soff, s[m], w[m], x[m],
                                                            acc, comp, k);
        }
    }
}

template <int S, int ST, bool POS, int ILP>
__global__ void __launch_bounds__(256, ILP == 1 ? WalkOccupancy<S, ST>::kMinBlocks
                                       : ILP == 2 ? 5
                                                  : 4)
    walk32_adjoint(WalkArgs a) {
    __shared__ uint64_t s_ekey;
    __shared__ int s_nh;
    __shared__ float s_wnorm;
    __shared__ int s_off[32];
    stage_offsets(a.stoff, s_off);
    if (threadIdx.x == 0) {
        s_ekey = epoch_key(a.seed, *a.d_epoch);
        s_nh = *a.d_nh;
        s_wnorm = float(a.sc[0]);
    }
    walk_begin_time(a);
    __syncthreads();
    // The launch has a thread for every history the domain was sized for.
    const long long e0 = (long long)blockIdx.x * (blockDim.x * ILP) + threadIdx.x;
    const RecordCopy none{};
    if (e0 < s_nh) {
        if (a.l1)
            adjoint_histories<S, ST, POS, kCached, ILP>(a, s_off, s_ekey, s_wnorm, e0, s_nh, none);
        else
            adjoint_histories<S, ST, POS, kBypass, ILP>(a, s_off, s_ekey, s_wnorm, e0, s_nh, none);
    }
    if (blockIdx.x == 0 && threadIdx.x == 0)
        atomicAdd(a.d_steps, (unsigned long long)s_nh * a.L);
    walk_end_time(a);
}

// The fixed-length walks of a domain whose records fit a block's shared memory.
// Their time is a chain of L dependent reads of a record, which the other warps
// of so few histories cannot hide: every block copies the records once (190 KB
// take about two microseconds, during which the first step is made) and the
// other steps read shared memory.  77^2, two histories per row: 6.6 us, 8.9 us
// from global memory.  Blocks are small, so that all SMs take part.
constexpr int kSmallBlock = 128;
constexpr int kSmallRecords = 200 * 1024;  // bytes

template <int S, int ST, bool POS, int DIR>
__global__ void __launch_bounds__(kSmallBlock) walk32_small(WalkArgs a, RowFinish f) {
    extern __shared__ __align__(128) char s_rec[];
    __shared__ __align__(8) uint64_t s_bar;
    __shared__ uint64_t s_ekey;
    __shared__ int s_off[32];
    RecordCopy copy{s_rec, uint32_t(__cvta_generic_to_shared(&s_bar))};
    stage_offsets(a.stoff, s_off);
    if (threadIdx.x == 0) {
        copy.start(a.rec, a.n * (S * 8));
        s_ekey = epoch_key(a.seed, *a.d_epoch);
    }
    walk_begin_time(a);
    __syncthreads();
    const unsigned at = blockIdx.x * blockDim.x + threadIdx.x;
    unsigned long long histories;
    if constexpr (DIR == MCLSGPU_FORWARD) {
        const unsigned pos = at >> f.hlog;
        const bool live = pos < unsigned(a.n);
        const int i = int(live ? pos : unsigned(a.n) - 1u);
        const int H = 1 << f.hlog;
        const double sum = row_histories<S, ST, POS, kShared>(a, int(threadIdx.x) & (H - 1), H,
                                                              s_off, s_ekey, i, copy);
        finish_row(a, f, sum, i, live);
        histories = (unsigned long long)a.n * a.per;
    } else {
        const int nh = *a.d_nh;
        if (at < unsigned(nh))
            adjoint_histories<S, ST, POS, kShared, 1>(a, s_off, s_ekey, float(a.sc[0]), at, nh,
                                                      copy);
        histories = (unsigned long long)nh;
    }
    if (at == 0) atomicAdd(a.d_steps, histories * a.L);
    copy.wait(a.status);  // no block ends with its copies in flight
    walk_end_time(a);
}

// Histories ended by the weight cutoff: persistent warps whose lanes refill
// one by one from the work queue as their histories terminate.
template <int S, int DIR, int ST, int MEM>
__global__ void __launch_bounds__(256, WalkOccupancy<S, ST>::kMinBlocks) walk32_cutoff(WalkArgs a) {
    static_assert(S % 4 == 0, "records are whole 32-byte halves");
    __shared__ uint64_t s_ekey;
    __shared__ int s_nh;
    __shared__ float s_wnorm;
    __shared__ int s_off[32];
    const int lane = threadIdx.x & 31;
    stage_offsets(a.stoff, s_off);
    if (threadIdx.x == 0) {
        s_ekey = epoch_key(a.seed, *a.d_epoch);
        s_nh = *a.d_nh;
        s_wnorm = float(a.sc[0]);
    }
    walk_begin_time(a);
    __syncthreads();
    const char* rec = reinterpret_cast<const char*>(a.rec);
    unsigned steps = 0;
    int s = 0, s0 = 0, k = 0;
    float w = 0.f, wcut = 0.f, acc = 0.f, comp = 0.f;
    uint64_t x = 0;
    bool alive = false, drained = false;
    while (true) {
        const unsigned need = __ballot_sync(kFull, !alive);
        if (need && !drained) {
            const int leader = __ffs(need) - 1;
            const int cnt = __popc(need);
            const int nh = s_nh;
            int base = 0;
            if (lane == leader) base = atomicAdd(a.d_counter, cnt);
            base = __shfl_sync(kFull, base, leader);
            if (base + cnt >= nh) drained = true;
            if (!alive) {
                const int e = base + __popc(need & ((1u << lane) - 1));
                if (e < nh) {
                    walk_start<DIR>(a, e, s_ekey, s_wnorm, s, w, x);
                    acc = 0.f;
                    comp = 0.f;
                    s0 = s;
                    wcut = a.cutoff * fabsf(w);
                    k = 0;
                    alive = true;
                }
            }
        }
        if (!__any_sync(kFull, alive)) break;
        if (alive) {
            walk_step<S, DIR, ST, MEM>(rec, a.y64, s_off, s, w, x, acc, comp, k);
            ++k;
            ++steps;
            if (k >= a.L || fabsf(w) < wcut) {
                alive = false;
                if (DIR == MCLSGPU_FORWARD) atomicAdd(&a.y64[s0], double(acc) - double(comp));
            }
        }
    }
    // Step count: one reduction per warp.
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) steps += __shfl_down_sync(kFull, steps, d);
    if (lane == 0 && steps) atomicAdd(a.d_steps, (unsigned long long)steps);
    walk_end_time(a);
}

// Bound by the latency of a step's loads.  PACKED: rows of at most 7 entries, one
// record of three sectors per step, 12.3 us for 10^4 histories; the
// general form follows row pointers, CDF (a binary search), weight and column
// one after the other, 18.7 us there.
template <int DIR, bool PACKED>
__global__ void __launch_bounds__(128) walk64(WalkArgs a) {
    const int nh = *a.d_nh;
    const double weight = a.sc[0];
    const int L = a.L;
    const uint64_t ekey = epoch_key(a.seed, *a.d_epoch);
    unsigned long long steps = 0;
    for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < nh;
         e += (long long)gridDim.x * blockDim.x) {
        int s;
        double w;
        if (DIR == MCLSGPU_ADJOINT) {
            const int sv = a.start[e];
            s = sv & 0x7fffffff;
            w = sv < 0 ? -weight : weight;
        } else {
            s = int(e / a.per);
            w = 1.0;
        }
        const int s0 = s;
        const double wcut = a.cutoff64 * fabs(w);
        uint64_t x = history_state(a, ekey, e);
        double acc = 0.0;
        const bool tr = a.tr_states && e < a.max_trace;
        if (tr) {
            for (int t = 0; t <= L; ++t) a.tr_states[e * (L + 1) + t] = -1;
            a.tr_states[e * (L + 1)] = s;
        }
        int k = 0;
        while (true) {
            if (DIR == MCLSGPU_ADJOINT) {
                if (k > 0) atomicAdd(&a.y64[s], w);
            } else {
                acc = __dadd_rn(acc, __dmul_rn(w, a.c64[s]));
            }
            x = xs_step(x);
            const double u = canonical64(x);
            double Ws;
            if constexpr (PACKED) {
                select_record64(a.rec64, s, u, Ws, s, a.status);
            } else {
                int r0, len;
                int lo = select64(a, s, u, r0, len);
                if (lo >= len) {
                    atomicOr(a.status, DEV_ERR_BOUNDS);
                    lo = len - 1;
                }
                Ws = a.h[r0 + lo] > 0.0 ? a.W[s] : -a.W[s];
                s = a.col[r0 + lo];
            }
            w = __dmul_rn(w, Ws);
            ++k;
            ++steps;
            if (tr) a.tr_states[e * (L + 1) + k] = s;
            if (k >= L || fabs(w) < wcut) break;
        }
        if (!isfinite(w)) atomicOr(a.status, DEV_ERR_NONFINITE);
        if (a.hlen) a.hlen[e] = k;
        if (DIR == MCLSGPU_FORWARD) atomicAdd(&a.y64[s0], acc);
        if (e < a.max_trace) {
            if (a.tr_w) a.tr_w[e] = w;
            if (a.tr_ev) a.tr_ev[e] = 2;  // Event::CUTOFF
            if (a.tr_start) a.tr_start[e] = s0;
        }
    }
    // Step count: one atomic per warp (one per thread serialises on the
    // counter when most threads have no history).
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) steps += __shfl_down_sync(kFull, steps, d);
    if ((threadIdx.x & 31) == 0 && steps) atomicAdd(a.d_steps, steps);
}

// Resident blocks per SM of a cutoff walk (a persistent grid).
template <int S, int DIR, int ST, int MEM>
int cutoff_blocks_per_sm(int block) {
    static int cached[2] = {0, 0};
    int& c = cached[block == 128 ? 0 : 1];
    if (!c) {
        int b = 0;
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, walk32_cutoff<S, DIR, ST, MEM>, block, 0);
        c = b > 0 ? b : 1;
    }
    return c;
}

struct WalkLaunch {
    const mclsgpu_domain* dom;
    WalkArgs a;
    RowFinish fin;
    bool launch;   // false: only cache the occupancy
};

template <int S, int ST, bool POS>
void launch_rows(const WalkLaunch& l) {
    const mclsgpu_domain* d = l.dom;
    const int T = d->walk_block;
    if (l.fin.split > 1) {
        const long long threads = ((long long)d->n * l.fin.split) << 5;
        walk32_split<S, ST><<<int((threads + T - 1) / T), T, 0, d->ctx->stream>>>(l.a, l.fin);
        return;
    }
    const long long threads = (long long)d->n << l.fin.hlog;
    walk32_rows<S, ST, POS><<<int((threads + T - 1) / T), T, 0, d->ctx->stream>>>(l.a, l.fin);
}

template <int S, int ST, bool POS, int ILP>
void launch_adj(const WalkLaunch& l) {
    const mclsgpu_domain* d = l.dom;
    const long long per_block = (long long)d->walk_block * ILP;
    long long grid = (d->nh_cap + per_block - 1) / per_block;
    if (grid < 1) grid = 1;
    walk32_adjoint<S, ST, POS, ILP><<<int(grid), d->walk_block, 0, d->ctx->stream>>>(l.a);
}

template <int S, int ST, bool POS, int DIR>
void launch_small(const WalkLaunch& l) {
    const mclsgpu_domain* d = l.dom;
    const int bytes = d->n * S * 8;
    if (!l.launch) {
        cudaFuncSetAttribute(walk32_small<S, ST, POS, DIR>,
                             cudaFuncAttributeMaxDynamicSharedMemorySize, kSmallRecords);
        return;
    }
    const long long threads = DIR == MCLSGPU_FORWARD ? (long long)d->n << l.fin.hlog : d->nh_cap;
    const long long grid = (threads + kSmallBlock - 1) / kSmallBlock;
    walk32_small<S, ST, POS, DIR><<<int(grid < 1 ? 1 : grid), kSmallBlock, bytes,
                                    d->ctx->stream>>>(l.a, l.fin);
}

// Records in shared memory: they must fit, and the blocks must run at once, one
// per SM.  MCSA solves of 24^2 to 80^2 grids take 5 to 9 % less time than from
// global memory, adjoint ones 4 to 6 %; nothing on this side of the line is
// slower.
bool small_walk(const mclsgpu_domain* d) {
    if (d->p.weight_cutoff > 0.0 || d->slots > 16 || d->walk_split > 1 ||
        (long long)d->n * d->slots * 8 > kSmallRecords)
        return false;
    const long long threads = d->p.direction == MCLSGPU_FORWARD
                                  ? (long long)d->n << d->walk_hlog
                                  : (long long)d->nh_cap;
    return threads <= (long long)d->ctx->num_sms * kSmallBlock;
}

template <int S, int ST, bool POS>
void launch32_fixed(const WalkLaunch& l) {
    const mclsgpu_domain* d = l.dom;
    if constexpr (S <= 16)
        if (small_walk(d)) {
            if (d->p.direction == MCLSGPU_ADJOINT)
                return launch_small<S, ST, POS, MCLSGPU_ADJOINT>(l);
            return launch_small<S, ST, POS, MCLSGPU_FORWARD>(l);
        }
    if (!l.launch) return;
    if (d->p.direction == MCLSGPU_ADJOINT) {
        // Several histories per lane: two on records of at most 64 bytes,
        // four on 32-byte records (the register budget).
        const int ilp = d->walk_ilp;
        if constexpr (S == 4)
            if (ilp >= 4) return launch_adj<S, ST, POS, 4>(l);
        if constexpr (S <= 8)
            if (ilp >= 2) return launch_adj<S, ST, POS, 2>(l);
        return launch_adj<S, ST, POS, 1>(l);
    }
    launch_rows<S, ST, POS>(l);
}

template <int S, int DIR, int ST, int MEM>
void launch_cutoff(const WalkLaunch& l) {
    const mclsgpu_domain* d = l.dom;
    const int T = d->walk_block;
    const long long fit =
        (long long)d->ctx->num_sms * cutoff_blocks_per_sm<S, DIR, ST, MEM>(T);
    if (!l.launch) return;
    // No more blocks than the histories need, at most what fits at once.
    const long long need = std::max((d->nh_cap + T - 1) / T, int64_t(1));
    walk32_cutoff<S, DIR, ST, MEM><<<int(std::min(need, fit)), T, 0, d->ctx->stream>>>(l.a);
}

template <int S, int ST>
void launch32_case(const WalkLaunch& l) {
    const mclsgpu_domain* d = l.dom;
    if (d->p.weight_cutoff > 0.0) {
        if (d->p.direction == MCLSGPU_ADJOINT)
            return d->walk_l1 ? launch_cutoff<S, MCLSGPU_ADJOINT, ST, kCached>(l)
                              : launch_cutoff<S, MCLSGPU_ADJOINT, ST, kBypass>(l);
        return d->walk_l1 ? launch_cutoff<S, MCLSGPU_FORWARD, ST, kCached>(l)
                          : launch_cutoff<S, MCLSGPU_FORWARD, ST, kBypass>(l);
    }
    if constexpr (ST == kStencil)
        if (!d->neg_h) return launch32_fixed<S, ST, true>(l);
    launch32_fixed<S, ST, false>(l);
}

// Dispatch on the record layout; `launch` false only caches the occupancy.
void dispatch_walk32(const WalkLaunch& l) {
    const int slots = l.dom->slots;
    if (l.dom->stencil_k && l.dom->rec_q16) {
        if (slots == 4) launch32_case<4, kStencil16>(l);
        else launch32_case<8, kStencil16>(l);
    } else if (l.dom->stencil_k) {
        if (slots == 4) launch32_case<4, kStencil>(l);
        else if (slots == 8) launch32_case<8, kStencil>(l);
        else launch32_case<16, kStencil>(l);
    } else {
        switch (slots) {
            case 4: launch32_case<4, kPacked>(l); break;
            case 8: launch32_case<8, kPacked>(l); break;
            case 12: launch32_case<12, kPacked>(l); break;
            case 16: launch32_case<16, kPacked>(l); break;
            case 24: launch32_case<24, kPacked>(l); break;
            default: launch32_case<32, kPacked>(l);
        }
    }
}

}  // namespace

namespace {

__device__ __forceinline__ unsigned fdiv(unsigned x, unsigned d, unsigned& rem) {
    const unsigned q = x / d;
    rem = x - q * d;
    return q;
}

// order[pos] = the row at position pos of a RowOrder.
__global__ void k_fill_order(RowOrder o, int n, int* order) {
    for (int pos = blockIdx.x * blockDim.x + threadIdx.x; pos < n;
         pos += gridDim.x * blockDim.x) {
        unsigned r, x, y, line;
        const unsigned zg = fdiv(pos, o.bz * o.X * o.Y, r);
        const unsigned nz = min(o.bz, o.Z - zg * o.bz);
        const unsigned yg = fdiv(r, o.by * o.X * nz, r);
        const unsigned ny = min(o.by, o.Y - yg * o.by);
        const unsigned strip = fdiv(r, o.bx * nz * ny, r);
        const unsigned wx = min(o.bx, o.X - strip * o.bx);
        line = fdiv(r, wx, x);
        const unsigned z = fdiv(line, ny, y);
        order[pos] = int(x + strip * o.bx + o.X * (y + yg * o.by + o.Y * (z + zg * o.bz)));
    }
}

}  // namespace

bool walks_from_shared(const mclsgpu_domain* dom) { return small_walk(dom); }

// How a row's histories are shared out (set-up time).  Up to four lanes when
// they get the same number; where the chip would not be full, as many as there
// are histories, up to a warp, then several warps that tally.  A lane's
// histories follow one another: 8 iterations on 32^2 rows with 1,000 histories
// each take 439 us, with four lanes a row at most 2,430; 101 on the same rows 233
// and 1,127; 33 on 100^2 rows 310 and 890; 4,000 on 10^2 rows 563 and 8,900.
void prepare_walk_lanes(mclsgpu_domain* dom) {
    if (!walks_rows(dom)) return;
    const int per = dom->p.sample_ratio > 0.0 ? int(ceil(dom->p.sample_ratio)) : 1;
    int hlog = per % 4 == 0 ? 2 : per % 2 == 0 ? 1 : 0;
    const long long fit = (long long)dom->ctx->num_sms * 2048, n = dom->n;
    while (hlog < 5 && (1 << hlog) < per && (n << (hlog + 1)) <= fit) ++hlog;
    dom->walk_hlog = hlog;
    const long long most = std::min(fit / (n << 5), (long long)(per + 31) / 32);
    dom->walk_split = hlog == 5 && most > 1 ? int(most) : 1;
}

// The row order of the forward walk (set-up time).  Records in shared memory are
// walked in any order, and more lanes than four share a row only where there are
// few rows.  Without the memory for it the walk takes the rows as they come.
void prepare_walk_order(mclsgpu_domain* dom) {
    if (!walk_finishes(dom) || dom->walk_hlog > 2 || small_walk(dom)) return;
    const RowOrder o = row_order(dom->n, dom->op->dia_k, dom->op->dia_off, 32 >> dom->walk_hlog);
    if (o.X <= 1) return;
    if (dmalloc(&dom->walk_order, size_t(dom->n)) != cudaSuccess) {
        cudaGetLastError();
        dom->walk_order = nullptr;
        return;
    }
    const int grid = (dom->n + 255) / 256;
    k_fill_order<<<grid < 2368 ? grid : 2368, 256, 0, dom->ctx->stream>>>(o, dom->n,
                                                                        dom->walk_order);
}

// Cache the occupancy of the walk kernel this domain will launch (set-up time,
// outside any stream capture).
void prepare_walk(mclsgpu_domain* dom) {
    if (dom->p.precision != MCLSGPU_FP32) return;
    dispatch_walk32(WalkLaunch{dom, WalkArgs{}, RowFinish{}, false});
}

namespace {

// Forward walks shared by the right-hand sides of a batch (batched MCSA): the
// walk does not depend on the source, so each history carries one
// Kahan-compensated FP32 sum of w * c_r(state) per column r of its start
// row's width class (cR holds the tally source of every column at every
// state, in the batch's element layout) and adds them into Y at the start
// row's elements in FP64.  Fixed-length histories only; a history never
// leaves its system, so every state it visits has its start row's width.
struct BatchWalk {
    const float* cR;
    double* Y;
    BatchFinish fin;
    BatchList list;
    BatchClasses cls;
    int grab;
    int per;
};

// The list entry k with hcum[k] <= h < hcum[k+1] (count entries).
__device__ __forceinline__ int list_entry(const int* hcum, int count, int h) {
    int lo = 0, hi = count - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (hcum[mid] <= h) lo = mid; else hi = mid - 1;
    }
    return lo;
}

// The tally-source row of state s in class c (W = 2^c columns).
template <int W>
__device__ __forceinline__ void load_source_row(const float* p, float (&c)[W]) {
    if constexpr (W >= 8) {
#pragma unroll
        for (int r = 0; r < W; r += 8) {
            uint32_t q[8];
            ld_record256_l1(p + r, q);
#pragma unroll
            for (int t = 0; t < 8; ++t) c[r + t] = __uint_as_float(q[t]);
        }
    } else if constexpr (W == 4) {
        const float4 q = __ldg(reinterpret_cast<const float4*>(p));
        c[0] = q.x;
        c[1] = q.y;
        c[2] = q.z;
        c[3] = q.w;
    } else if constexpr (W == 2) {
        const float2 q = __ldg(reinterpret_cast<const float2*>(p));
        c[0] = q.x;
        c[1] = q.y;
    } else {
        c[0] = __ldg(p);
    }
}

// One history of a row of class C (2^C columns), returns its steps.
template <int S, bool ST, int C>
__device__ __forceinline__ unsigned batch_history(const WalkArgs& a, const char* rec,
                                                  const int* soff, const BatchWalk& m, int s,
                                                  float w, uint64_t x, double* stage) {
    constexpr int W = 1 << C;
    const int r0 = m.cls.crow[C];
    const float* cbase = m.cR + m.cls.cel[C];
    const int s0 = s;
    float acc[W], comp[W];
#pragma unroll
    for (int r = 0; r < W; ++r) acc[r] = comp[r] = 0.f;
    const int L = a.L;
    for (int k = 0; k < L; ++k) {
        float c[W];
        load_source_row<W>(cbase + size_t(s - r0) * W, c);
#pragma unroll
        for (int r = 0; r < W; ++r) {
            const float term = w * c[r] - comp[r];
            const float t = acc[r] + term;
            comp[r] = (t - acc[r]) - term;
            acc[r] = t;
        }
        float da = 0.f, dc = 0.f;  // the record header's own tally is unused here
        walk_step<S, MCLSGPU_FORWARD, ST ? kStencil : kPacked, kBypass>(rec, nullptr, soff, s, w, x, da, dc,
                                                                 k);
    }
    if (!m.Y) {
        // The row's only history: its sums go to the warp's finishing pass.
#pragma unroll
        for (int r = 0; r < W; ++r) stage[r] = double(acc[r]) - double(comp[r]);
        return unsigned(L);
    }
    double* y = m.Y + m.cls.cel[C] + size_t(s0 - r0) * W;
#pragma unroll
    for (int r = 0; r < W; ++r)
        if (acc[r] != 0.f || comp[r] != 0.f) atomicAdd(&y[r], double(acc[r]) - double(comp[r]));
    return unsigned(L);
}

// Sums of one lane in the warp's stage: 16 columns and a word of padding, so
// that the lanes' writes spread over the banks.
constexpr int kBatchStage = 17;

// The iterate of the warp's 32 rows from their staged sums.  The rows of a
// warp inside one class and one run of rows are consecutive elements, which
// the lanes take in order (a lane writing its own row's columns would touch 32
// lines per column: 450 us for a walk of 97); otherwise row by row.
__device__ __forceinline__ void finish_rows(const BatchWalk& m, const double* stage, int row,
                                            int c, bool live) {
    const BatchFinish& f = m.fin;
    const int lane = threadIdx.x & 31;
    __syncwarp();
    const int row0 = __shfl_sync(kFull, row, 0), c0 = __shfl_sync(kFull, c, 0);
    auto finish = [&](size_t e, double y) {
        f.X[e] = batch_corrected(f.X2[e], f.RP2[e], y, f.nomega, f.inv_per, f.ev);
    };
    if (__all_sync(kFull, live && c == c0 && row == row0 + lane)) {
        const size_t e0 = size_t(m.cls.cel[c0]) + (size_t(row0 - m.cls.crow[c0]) << c0);
        for (int t = lane; t < (32 << c0); t += 32)
            finish(e0 + t, stage[(t >> c0) * kBatchStage + (t & ((1 << c0) - 1))]);
    } else if (live) {
        const size_t e0 = size_t(m.cls.cel[c]) + (size_t(row - m.cls.crow[c]) << c);
        for (int r = 0; r < (1 << c); ++r) finish(e0 + r, stage[lane * kBatchStage + r]);
    }
    __syncwarp();
}

template <int S, bool ST>
__global__ void __launch_bounds__(256, 3) walk32_batch(WalkArgs a, BatchWalk m) {
    static_assert(S % 4 == 0, "records are whole 32-byte halves");
    __shared__ uint64_t s_ekey;
    __shared__ int s_nh, s_count;
    __shared__ int s_off[32];
    // One history per row: the warps' sums, kBatchStage doubles per lane.
    extern __shared__ double s_stage[];
    stage_offsets(a.stoff, s_off);
    const int lane = threadIdx.x & 31;
    double* warp_stage = s_stage + (threadIdx.x >> 5) * (32 * kBatchStage);
    double* mine = warp_stage + lane * kBatchStage;
    if (threadIdx.x == 0) {
        s_ekey = epoch_key(a.seed, *a.d_epoch);
        s_count = *m.list.lcount;
        s_nh = s_count > 0 ? m.list.hcum[s_count] : 0;
    }
    __syncthreads();
    walk_begin_time(a);
    const char* rec = reinterpret_cast<const char*>(a.rec);
    unsigned steps = 0;
    // Every history takes the same number of steps: the warps take their
    // chunks statically (a shared counter is one contended atomic per chunk).
    const int chunk = 32 * m.grab, warps = gridDim.x * (blockDim.x >> 5);
    const int count = s_count, nh = s_nh;
    const int w0 = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    for (long long first = (long long)w0 * chunk; first < nh; first += (long long)warps * chunk) {
        const int base = int(first);
        // The list entry of the grab's first history (one search per warp);
        // the lanes step forward from it.
        int k0 = 0;
        if (lane == 0) k0 = list_entry(m.list.hcum, count, base);
        k0 = __shfl_sync(kFull, k0, 0);
        for (int g = 0; g < m.grab; ++g) {
            const int h = base + 32 * g + lane;
            if (base + 32 * g >= nh) break;  // the whole warp
            // A lane past the end walks the last history and drops its sums.
            const bool live = h < nh;
            const int hh = live ? h : nh - 1;
            int k = k0;
            while (k + 1 < count && hh >= m.list.hcum[k + 1]) ++k;
            const int sys = m.list.lsys[k];
            const int e = m.list.srow0[sys] * m.per + (hh - m.list.hcum[k]);
            int s;
            float w;
            uint64_t x;
            walk_start<MCLSGPU_FORWARD>(a, e, s_ekey, 1.f, s, w, x);
            int c = 0;
            while (c < 4 && s >= m.cls.crow[c + 1]) ++c;
            const int row = s;
            if (!live && m.Y) continue;  // (per > 1: no warp-wide pass follows)
            switch (c) {
                case 0: steps += batch_history<S, ST, 0>(a, rec, s_off, m, s, w, x, mine); break;
                case 1: steps += batch_history<S, ST, 1>(a, rec, s_off, m, s, w, x, mine); break;
                case 2: steps += batch_history<S, ST, 2>(a, rec, s_off, m, s, w, x, mine); break;
                case 3: steps += batch_history<S, ST, 3>(a, rec, s_off, m, s, w, x, mine); break;
                default: steps += batch_history<S, ST, 4>(a, rec, s_off, m, s, w, x, mine); break;
            }
            if (m.Y) continue;
            if (!live) steps -= unsigned(a.L);
            finish_rows(m, warp_stage, row, c, live);
        }
    }
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) steps += __shfl_down_sync(kFull, steps, d);
    if (lane == 0 && steps) atomicAdd(a.d_steps, (unsigned long long)steps);
    walk_end_time(a);
}

template <int S, bool ST>
void launch_batch_s(const WalkArgs& a, const BatchWalk& m, int sms, int block, cudaStream_t st) {
    static int cached[2] = {0, 0};
    const int slot = block == 128 ? 0 : 1;
    const size_t smem = size_t(block) * kBatchStage * sizeof(double);  // at most 34 KB
    if (!cached[slot]) {
        int b = 0;
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, walk32_batch<S, ST>, block, smem);
        cached[slot] = b > 0 ? b : 1;
    }
    walk32_batch<S, ST><<<sms * cached[slot], block, smem, st>>>(a, m);
}

}  // namespace

// Fill the walk arguments of a domain (shared by the single- and the
// multi-right-hand-side walks).
static void fill_walk_args(mclsgpu_domain* dom, WalkArgs& a) {
    mclsgpu_context* ctx = dom->ctx;
    const mclsgpu_mc_params& p = dom->p;
    a.n = dom->n;
    a.L = p.history_length;
    a.per = p.sample_ratio > 0.0 ? int(ceil(p.sample_ratio)) : 1;
    a.rng_mode = p.rng_mode;
    a.d_nh = dom->d_nh;
    a.d_counter = dom->d_counter;
    a.start = dom->start;
    a.sc = dom->d_scalars;
    a.seed = dom->seed;
    a.d_epoch = dom->d_epoch;
    a.jump = dom->d_jump;
    a.d_pos = dom->d_pos;
    a.rec = dom->rec;
    a.rec64 = dom->rec64;
    a.d_steps = dom->d_steps;
    a.d_tim = dom->d_tim;
    a.status = ctx->d_status;
    a.l1 = dom->walk_l1;
    for (int j = 0; j < 32; ++j) a.stoff[j] = dom->stencil_off[j];
}

// Batched forward walks over the domain's FP32 records (records of at most
// 16 slots; see launch_walk_batch in internal.h).
int launch_walk_batch(mclsgpu_domain* dom, const BatchClasses& cls, const BatchList& list,
                      const float* cR, double* Y, const BatchFinish& fin, int grab) {
    mclsgpu_context* ctx = dom->ctx;
    if (dom->p.precision != MCLSGPU_FP32 || dom->p.direction != MCLSGPU_FORWARD || !dom->slots ||
        dom->rec_q16)
        return set_error(ctx, MCLSGPU_ERR_UNSUPPORTED,
                         "batched walks need FP32 forward packed or stencil records");
    if (grab < 1 || grab > 8)
        return set_error(ctx, MCLSGPU_ERR_INVALID_ARG, "batched walks: grab %d not in 1..8", grab);
    WalkArgs a{};
    fill_walk_args(dom, a);
    const int sms = ctx->num_sms;
    const int block = dom->walk_block;
    cudaStream_t st = ctx->stream;
    const BatchWalk m{cR, Y, fin, list, cls, grab, a.per};
    bool ok = true;
    if (dom->stencil_k) {
        switch (dom->slots) {
            case 4: launch_batch_s<4, true>(a, m, sms, block, st); break;
            case 8: launch_batch_s<8, true>(a, m, sms, block, st); break;
            default: ok = false;
        }
    } else {
        switch (dom->slots) {
            case 4: launch_batch_s<4, false>(a, m, sms, block, st); break;
            case 8: launch_batch_s<8, false>(a, m, sms, block, st); break;
            case 12: launch_batch_s<12, false>(a, m, sms, block, st); break;
            case 16: launch_batch_s<16, false>(a, m, sms, block, st); break;
            default: ok = false;
        }
    }
    if (!ok)
        return set_error(ctx, MCLSGPU_ERR_UNSUPPORTED, "batched walks: %d-slot records not supported",
                         dom->slots);
    return MCLSGPU_OK;
}

__global__ void k_fill_offsets(int* hoff, const int* d_nh, int L) {
    const int nh = *d_nh;
    for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < nh; e += gridDim.x * blockDim.x)
        hoff[e] = e * L;
}

// hoff2 (exclusive prefix of the lengths) against hoff: *changed = 1 when
// any offset moved; hoff takes the new offsets.
__global__ void k_update_offsets(int* hoff, const int* hoff2, const int* d_nh, int* changed) {
    const int nh = *d_nh;
    int c = 0;
    for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < nh; e += gridDim.x * blockDim.x) {
        if (hoff[e] != hoff2[e]) {
            c = 1;
            hoff[e] = hoff2[e];
        }
    }
    if (__syncthreads_or(c) && threadIdx.x == 0) atomicOr(changed, 1);
}

__global__ void k_advance_pos_by(unsigned long long* d_pos, long long draws) { *d_pos += draws; }

static void launch_walk64(const mclsgpu_domain* dom, const WalkArgs& a, int grid) {
    cudaStream_t st = dom->ctx->stream;
    const bool adjoint = dom->p.direction == MCLSGPU_ADJOINT;
    auto kernel = dom->rec64 ? (adjoint ? walk64<MCLSGPU_ADJOINT, true> : walk64<MCLSGPU_FORWARD, true>)
                             : (adjoint ? walk64<MCLSGPU_ADJOINT, false>
                                        : walk64<MCLSGPU_FORWARD, false>);
    kernel<<<grid, 128, 0, st>>>(a);
}

// Variable-length histories on the reference stream (a Weight Cutoff with
// "Reproducible MC Mode"): the reference draws history e's uniforms right
// after history e-1's, so e's first draw depends on every earlier length.
// Round 1 walks with offsets e * L; each later round walks again with the
// offsets the previous round's lengths give, until no offset moves.  The
// histories before the first moved offset are final after each round, so the
// rounds end (at most one more than the histories); in practice lengths
// repeat and a few rounds suffice.  Tallies and the step count are restored
// before each repeated round.  Host-synchronous.
static void walk_reference_rounds(mclsgpu_domain* dom, WalkArgs a, int grid) {
    mclsgpu_context* ctx = dom->ctx;
    cudaStream_t st = ctx->stream;
    const int n = dom->n;
    const int L = dom->p.history_length;
    int nh = 0;
    unsigned long long steps0 = 0;
    cudaMemcpyAsync(&nh, dom->d_nh, sizeof(int), cudaMemcpyDeviceToHost, st);
    cudaMemcpyAsync(&steps0, dom->d_steps, sizeof(steps0), cudaMemcpyDeviceToHost, st);
    cudaMemcpyAsync(dom->y_save, dom->y64, size_t(n) * sizeof(double), cudaMemcpyDeviceToDevice,
                    st);
    k_fill_offsets<<<grid, 128, 0, st>>>(dom->hoff, dom->d_nh, L);
    a.hoff = dom->hoff;
    a.hlen = dom->hlen;
    int* changed = reinterpret_cast<int*>(dom->hoff2 + dom->nh_cap + 1);
    long long total = 0;
    int rounds = 0;
    for (;;) {
        ++rounds;
        launch_walk64(dom, a, grid);
        if (nh == 0 || exclusive_scan_counts_dev(ctx, dom->hlen, nh, dom->hoff2, &total)) break;
        cudaMemsetAsync(changed, 0, sizeof(int), st);
        k_update_offsets<<<grid, 128, 0, st>>>(dom->hoff, dom->hoff2, dom->d_nh, changed);
        int h_changed = 0;
        cudaMemcpyAsync(&h_changed, changed, sizeof(int), cudaMemcpyDeviceToHost, st);
        if (cudaStreamSynchronize(st) != cudaSuccess || !h_changed || rounds > nh) break;
        cudaMemcpyAsync(dom->y64, dom->y_save, size_t(n) * sizeof(double),
                        cudaMemcpyDeviceToDevice, st);
        cudaMemcpyAsync(dom->d_steps, &steps0, sizeof(steps0), cudaMemcpyHostToDevice, st);
    }
    dom->walk_rounds = rounds;
    k_advance_pos_by<<<1, 1, 0, st>>>(dom->d_pos, total);
}

// Launch the walks of the current source.  Trace arrays only with FP64.
// `fused`: the work-queue counter is reset by the fused residual kernel that
// follows the walk (MCSA loop).
// `fin`: how forward fixed-length FP32 walks finish each row (walk_finishes).
void launch_walk(mclsgpu_domain* dom, const RowFinish& fin, long long max_trace,
                 long long* tr_states, double* tr_w, int* tr_ev, long long* tr_start, bool fused) {
    mclsgpu_context* ctx = dom->ctx;
    const mclsgpu_mc_params& p = dom->p;
    WalkArgs a{};
    fill_walk_args(dom, a);
    a.cutoff = float(p.weight_cutoff > 0.0 ? p.weight_cutoff : 0.0);
    a.cutoff64 = p.weight_cutoff > 0.0 ? p.weight_cutoff : 0.0;
    a.rp = dom->D.rp;
    a.col = dom->D.ci;
    a.h = dom->D.v;
    a.cdf = dom->cdf;
    a.W = dom->w;
    a.y64 = dom->y64;
    a.c64 = dom->c64;
    a.max_trace = max_trace;
    a.tr_states = tr_states;
    a.tr_w = tr_w;
    a.tr_ev = tr_ev;
    a.tr_start = tr_start;
    cudaStream_t st = ctx->stream;
    if (p.precision == MCLSGPU_FP32) {
        if (!fused && p.weight_cutoff > 0.0)
            cudaMemsetAsync(dom->d_counter, 0, sizeof(int), st);
        WalkLaunch l{dom, a, fin, true};
        l.fin.hlog = dom->walk_hlog;
        l.fin.split = dom->walk_split;
        l.fin.order = dom->walk_order;
        dispatch_walk32(l);
    } else {
        // One thread per history up to 8 blocks per SM (the kernel strides
        // beyond that); no more blocks than the history capacity needs.
        long long g = (dom->nh_cap + 127) / 128;
        if (g < 1) g = 1;
        const int grid = int(g < ctx->num_sms * 8 ? g : ctx->num_sms * 8);
        if (walk_needs_rounds(dom))
            walk_reference_rounds(dom, a, grid);
        else
            launch_walk64(dom, a, grid);
    }
}

// ---- row-partitioned domains (domain-decomposed transport) -----------------
//
// One part holds the records and tallies of rows [row0, row0 + n).  A
// history walks while its state stays in the part; when a transition takes
// it to another part's row and the history goes on (steps left, weight above
// the cutoff), it is written to that part's outbox (HistoryWire: Xorshift
// state, state, step, weight and, forward, its running sum) and continues
// there in a later round, on the same random stream.  An adjoint history
// tallies where it stands, so its tallies land in the parts it visits.  A
// forward history's sum belongs to its start row: when it ends outside the
// part that owns that row, the sum travels there as a tally return (state
// -1).  Every transition and tally is therefore the one the whole-domain walk
// would make.
namespace {

__device__ __forceinline__ int part_owner(const int* sb, int nparts, int s) {
    int lo = 0, up = nparts;  // sb[lo] <= s < sb[lo + 1]
    while (up - lo > 1) {
        const int mid = (lo + up) >> 1;
        if (sb[mid] <= s) lo = mid; else up = mid;
    }
    return lo;
}

__device__ __forceinline__ void part_send(const PartWalk& p, int q, const HistoryWire& h) {
    const unsigned long long slot = atomicAdd(&p.out_cnt[q], 1ULL);
    if (slot < (unsigned long long)p.cap)
        p.out[size_t(q) * size_t(p.cap) + slot] = h;
    else
        atomicOr(p.status, DEV_ERR_CAPACITY);
}

template <int S, int DIR, int ST>
__global__ void __launch_bounds__(256) walk32_part(PartWalk p) {
    __shared__ int sb[kMaxParts + 1];
    __shared__ int s_off[32];
    for (int t = threadIdx.x; t <= p.nparts; t += blockDim.x) sb[t] = p.bounds[t];
    stage_offsets(p.stoff, s_off);
    __syncthreads();
    const uint64_t ekey = epoch_key(p.seed, *p.d_epoch);
    const float wnorm = DIR == MCLSGPU_ADJOINT ? float(p.sc[0]) : 1.f;
    const float wcut = p.cutoff * wnorm;
    const long long nwork = p.in ? p.n_in : p.e_end - p.e_begin;
    // walk_step indexes records and tallies by the global state.
    const char* rec = reinterpret_cast<const char*>(p.rec) - ptrdiff_t(p.row0) * (S * 8);
    double* y = p.y - p.row0;
    const int hi = p.row0 + p.n;
    unsigned steps = 0;
    for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < nwork;
         t += (long long)gridDim.x * blockDim.x) {
        int s, k, id;
        float w, acc = 0.f, comp = 0.f;
        uint64_t x;
        if (p.in) {
            const HistoryWire h = p.in[t];
            if (DIR == MCLSGPU_FORWARD && h.state < 0) {  // a tally return
                const int s0 = h.id / p.per;
                if (s0 < p.row0 || s0 >= hi)
                    atomicOr(p.status, DEV_ERR_BOUNDS);
                else
                    atomicAdd(&p.y[s0 - p.row0], double(h.acc) - double(h.comp));
                continue;
            }
            s = h.state;
            k = h.step;
            w = h.weight;
            x = h.rng;
            id = h.id;
            acc = h.acc;
            comp = h.comp;
        } else {
            const long long e = p.e_begin + t;
            if (DIR == MCLSGPU_ADJOINT) {
                const int sv = p.start[e];
                s = sv & 0x7fffffff;
                w = sv < 0 ? -wnorm : wnorm;
            } else {
                s = int(e / p.per);
                w = 1.f;
            }
            x = counter_state(ekey, 2, uint64_t(e));
            k = 0;
            id = int(e);
        }
        if (s < p.row0 || s >= hi) {  // not this part's history
            atomicOr(p.status, DEV_ERR_BOUNDS);
            continue;
        }
        while (true) {
            walk_step<S, DIR, ST, kBypass>(rec, y, s_off, s, w, x, acc, comp, k);
            ++k;
            ++steps;
            if (k >= p.L || fabsf(w) < wcut) {
                if (DIR == MCLSGPU_FORWARD) {
                    const int s0 = id / p.per;
                    if (s0 >= p.row0 && s0 < hi) {
                        atomicAdd(&p.y[s0 - p.row0], double(acc) - double(comp));
                    } else {
                        HistoryWire h;
                        h.rng = 0;
                        h.state = -1;
                        h.step = k;
                        h.weight = w;
                        h.id = id;
                        h.acc = acc;
                        h.comp = comp;
                        part_send(p, part_owner(sb, p.nparts, s0), h);
                    }
                }
                break;
            }
            if (s < p.row0 || s >= hi) {
                HistoryWire h;
                h.rng = x;
                h.state = s;
                h.step = k;
                h.weight = w;
                h.id = id;
                h.acc = acc;
                h.comp = comp;
                part_send(p, part_owner(sb, p.nparts, s), h);
                break;
            }
        }
    }
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) steps += __shfl_down_sync(kFull, steps, d);
    if ((threadIdx.x & 31) == 0 && steps) atomicAdd(p.d_steps, (unsigned long long)steps);
}

// FP32-versus-FP64 transition agreement.  History e starts at state e mod n
// on its counter stream and walks `L` transitions along the FP64 domain
// (walk64's selection with u = canonical64(x)); at every transition the FP32
// record of the same state is searched with u = canonical32(x) of the same
// draw (walk32's selection).  A transition disagrees when the two select a
// different column or sign; out[0] += histories with at least one
// disagreement, out[1] += disagreeing transitions.
template <int S, int ST>
__global__ void __launch_bounds__(256) k_walk_agreement(WalkArgs a, long long nh, uint64_t ekey,
                                                        unsigned long long* out) {
    __shared__ int s_off[32];
    stage_offsets(a.stoff, s_off);
    __syncthreads();
    const char* rec = reinterpret_cast<const char*>(a.rec);
    unsigned long long hd = 0, td = 0;
    for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < nh;
         e += (long long)gridDim.x * blockDim.x) {
        int s = int(e % a.n);
        uint64_t x = counter_state(ekey, 2, uint64_t(e));
        bool differ = false;
        for (int k = 0; k < a.L; ++k) {
            uint32_t q[2 * S];
            const char* r = rec + size_t(s) * (S * 8);
#pragma unroll
            for (int t = 0; t < S / 4; ++t) ld_record256(r + 32 * t, q + 8 * t);
            x = xs_step(x);
            int s32 = s;
            unsigned neg32;
            select32<S, ST>(s_off, q, x, s32, neg32);
            int r0, len;
            int j = select64(a, s, canonical64(x), r0, len);
            if (j >= len) {
                atomicOr(a.status, DEV_ERR_BOUNDS);
                j = len - 1;
            }
            const int s64 = a.col[r0 + j];
            const bool neg64 = !(a.h[r0 + j] > 0.0);
            if (s32 != s64 || (neg32 != 0u) != neg64) {
                ++td;
                differ = true;
            }
            s = s64;
        }
        hd += differ ? 1 : 0;
    }
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) {
        hd += __shfl_down_sync(kFull, hd, d);
        td += __shfl_down_sync(kFull, td, d);
    }
    if ((threadIdx.x & 31) == 0) {
        if (hd) atomicAdd(&out[0], hd);
        if (td) atomicAdd(&out[1], td);
    }
}

}  // namespace

int walk_agreement(mclsgpu_domain* dom, long long histories, uint64_t seed, long long* hist_diff,
                   long long* trans_diff) {
    mclsgpu_context* ctx = dom->ctx;
    if (dom->p.precision != MCLSGPU_FP32 || !dom->rec)
        return set_error(ctx, MCLSGPU_ERR_INVALID_ARG, "walk agreement needs FP32 records");
    if (histories < 1) return set_error(ctx, MCLSGPU_ERR_INVALID_ARG, "histories < 1");
    WalkArgs a{};
    fill_walk_args(dom, a);
    a.rp = dom->D.rp;
    a.col = dom->D.ci;
    a.h = dom->D.v;
    a.cdf = dom->cdf;
    a.W = dom->w;
    unsigned long long* d_out = nullptr;
    cudaError_t e = dmalloc(&d_out, 2);
    if (e != cudaSuccess) return cuda_fail(ctx, e, "cudaMalloc");
    cudaStream_t st = ctx->stream;
    cudaMemsetAsync(d_out, 0, 2 * sizeof(unsigned long long), st);
    const long long g = (histories + 255) / 256;
    const int grid = int(g < ctx->num_sms * 8 ? g : ctx->num_sms * 8);
    const uint64_t ekey = epoch_key(seed, 0);
    drop_stale_error();
    bool ok = true;
#define MCLSGPU_AGREE(SL, STV) k_walk_agreement<SL, STV><<<grid, 256, 0, st>>>(a, histories, ekey, d_out)
    if (dom->stencil_k && dom->rec_q16) {
        switch (dom->slots) {
            case 4: MCLSGPU_AGREE(4, kStencil16); break;
            case 8: MCLSGPU_AGREE(8, kStencil16); break;
            default: ok = false;
        }
    } else if (dom->stencil_k) {
        switch (dom->slots) {
            case 4: MCLSGPU_AGREE(4, kStencil); break;
            case 8: MCLSGPU_AGREE(8, kStencil); break;
            case 16: MCLSGPU_AGREE(16, kStencil); break;
            default: ok = false;
        }
    } else {
        switch (dom->slots) {
            case 4: MCLSGPU_AGREE(4, kPacked); break;
            case 8: MCLSGPU_AGREE(8, kPacked); break;
            case 12: MCLSGPU_AGREE(12, kPacked); break;
            case 16: MCLSGPU_AGREE(16, kPacked); break;
            case 24: MCLSGPU_AGREE(24, kPacked); break;
            case 32: MCLSGPU_AGREE(32, kPacked); break;
            default: ok = false;
        }
    }
#undef MCLSGPU_AGREE
    unsigned long long h[2] = {0, 0};
    e = cudaGetLastError();
    if (e == cudaSuccess) e = cudaMemcpyAsync(h, d_out, sizeof(h), cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    dfree(d_out);
    if (!ok) return set_error(ctx, MCLSGPU_ERR_UNSUPPORTED, "walk agreement: %d-slot records",
                              dom->slots);
    if (e != cudaSuccess) return cuda_fail(ctx, e, "walk agreement");
    int rc = check_device_status(ctx);
    if (rc) return rc;
    *hist_diff = (long long)h[0];
    *trans_diff = (long long)h[1];
    return MCLSGPU_OK;
}

void launch_walk_part(const PartWalk& p, mclsgpu_context* ctx) {
    const long long nwork = p.in ? p.n_in : p.e_end - p.e_begin;
    if (nwork <= 0) return;
    long long g = (nwork + 255) / 256;
    const int grid = int(g < ctx->num_sms * 8 ? g : ctx->num_sms * 8);
    cudaStream_t st = ctx->stream;
#define MCLSGPU_PART_SLOTS(D)                                                 \
    if (p.kind == kStencil16) {                                               \
        if (p.slots == 4) walk32_part<4, D, kStencil16><<<grid, 256, 0, st>>>(p);  \
        else walk32_part<8, D, kStencil16><<<grid, 256, 0, st>>>(p);            \
    } else if (p.kind == kStencil) {                                          \
        switch (p.slots) {                                                    \
            case 4: walk32_part<4, D, kStencil><<<grid, 256, 0, st>>>(p); break;   \
            case 8: walk32_part<8, D, kStencil><<<grid, 256, 0, st>>>(p); break;   \
            default: walk32_part<16, D, kStencil><<<grid, 256, 0, st>>>(p); break; \
        }                                                                     \
    } else {                                                                  \
        switch (p.slots) {                                                    \
            case 4: walk32_part<4, D, kPacked><<<grid, 256, 0, st>>>(p); break;   \
            case 8: walk32_part<8, D, kPacked><<<grid, 256, 0, st>>>(p); break;   \
            case 12: walk32_part<12, D, kPacked><<<grid, 256, 0, st>>>(p); break; \
            case 16: walk32_part<16, D, kPacked><<<grid, 256, 0, st>>>(p); break; \
            case 24: walk32_part<24, D, kPacked><<<grid, 256, 0, st>>>(p); break; \
            default: walk32_part<32, D, kPacked><<<grid, 256, 0, st>>>(p); break; \
        }                                                                     \
    }
    if (p.dir == MCLSGPU_FORWARD) {
        MCLSGPU_PART_SLOTS(MCLSGPU_FORWARD)
    } else {
        MCLSGPU_PART_SLOTS(MCLSGPU_ADJOINT)
    }
#undef MCLSGPU_PART_SLOTS
}

}  // namespace mclsgpu

// spai.cu -- learned sparse-approximate-inverse (SPAI) preconditioner.
//
// A per-row MLP maps the local stencil of row i of A to the values of row i
// of M, a sparse approximate inverse on A's own pattern, which replaces the
// Jacobi M^-1 = diag(A)^-1 in H = I - M A.  There is no counterpart in the
// reference (its closest relative is the ParaSails preconditioner slot).
//
// Stencil slots.  The operator must be stored by diagonal offsets (K <= 9
// offsets, ascending, the centre among them); slot s is the s-th offset.
// Features of row i (16, BF16): for each non-centre slot s in order,
//   a_s = A[i,i+o_s] / A[i,i]                  (0 where A has no entry)
//   d_s = log(A[j,j] / A[i,i]), j = i + o_s    (0 where A has no entry)
// zero-padded to 16.  Outputs (16, FP32): slot s of row i gives
//   M[i, i+o_s] = (delta(o_s, 0) + out_s) / A[i,i]
// on A's pattern, so a network whose last layer is zero is exactly Jacobi.
//
// Network: 16 -> 64 (ReLU) -> 64 (ReLU) -> 16, BF16 operands with FP32
// accumulation on the tensor cores (tcgen05.mma kind::f16, accumulators in
// tensor memory), FP32 master parameters and Adam moments in HBM.  Flat
// parameter order: W1[64][16], b1[64], W2[64][64], b2[64], W3[16][64], b3[16]
// (weights stored out x in).
//
// Training loss on an operator A and vectors v_1..v_R (residual snapshots
// of MCSA and random vectors):
//   L = (1/R) sum_v |v - M A v|_2^2 / |v|_2^2
// whose gradient with respect to out_{i,s} is
//   G[i,s] = -(2/R) sum_v e_i (A v)_{i+o_s} / (A[i,i] |v|^2),  e = v - M A v.
// The backward kernel propagates G through the network on the tensor cores.
#include <cuda_bf16.h>

#include <algorithm>
#include <cmath>
#include <mutex>
#include <cstring>
#include <random>
#include <type_traits>
#include <utility>
#include <vector>

#include "internal.h"

namespace mclsgpu {
namespace {

constexpr int kF = 16;      // features
constexpr int kH = 64;      // hidden width
constexpr int kO = 16;      // outputs (stencil slots, padded)
constexpr int kMaxSlots = 9;
constexpr int kTileRows = 128;
constexpr int kThreads = 128;
// Flat parameter offsets.
constexpr int kW1 = 0;
constexpr int kB1 = kW1 + kH * kF;
constexpr int kW2 = kB1 + kH;
constexpr int kB2 = kW2 + kH * kH;
constexpr int kW3 = kB2 + kH;
constexpr int kB3 = kW3 + kO * kH;
constexpr int kParams = kB3 + kO;  // 6288

// ---- shared-memory operand layout ------------------------------------------
// K-major, no swizzle: a tile of R rows (the M or N extent) by C columns (the
// K extent) of BF16 is stored as 8x8 core matrices of 128 contiguous bytes
// (8 rows x 16 bytes); core matrix (r/8, c/8) sits at
// ((c/8) * (R/8) + r/8) * 128.  The same bytes read with the roles of rows
// and columns exchanged form an MN-major operand (rows become K), which the
// weight-gradient products use.
__device__ __forceinline__ uint32_t kmaj_off(int r, int c, int R) {
    return uint32_t((((c >> 3) * (R >> 3)) + (r >> 3)) * 128 + (r & 7) * 16 + (c & 7) * 2);
}

// Shared-memory matrix descriptor (tcgen05), no swizzle.  Fields: start
// address >> 4 in bits 0-13, leading-dimension byte offset >> 4 in 16-29,
// stride-dimension byte offset >> 4 in 32-45, descriptor version 1 in 46-47,
// layout type 0 (no swizzle) in 61-63.
__device__ __forceinline__ uint64_t smem_desc(uint32_t saddr, uint32_t lbo, uint32_t sbo) {
    return uint64_t((saddr >> 4) & 0x3FFF) | (uint64_t((lbo >> 4) & 0x3FFF) << 16) |
           (uint64_t((sbo >> 4) & 0x3FFF) << 32) | (uint64_t(1) << 46);
}
// K-major operand: the two 8-column K chunks of one K=16 step are one
// column-chunk stride apart (leading offset); 8-row groups are 128 B apart.
__device__ __forceinline__ uint64_t desc_kmajor(uint32_t tile, int R, int kstep) {
    const uint32_t chunk = uint32_t(R / 8) * 128;
    return smem_desc(tile + uint32_t(2 * kstep) * chunk, chunk, 128);
}
// MN-major view of a tile stored K-major with R rows: MN = the stored
// columns (8-column groups one chunk stride apart: stride offset), K = the
// stored rows (8-row groups 128 B apart: leading offset); K step t covers
// stored rows 16t..16t+15.
__device__ __forceinline__ uint64_t desc_mnmajor(uint32_t tile, int R, int kstep) {
    const uint32_t chunk = uint32_t(R / 8) * 128;
    return smem_desc(tile + uint32_t(2 * kstep) * 128, 128, chunk);
}
// Instruction descriptor of kind::f16: FP32 accumulate (bits 4-5 = 1), BF16
// A and B (bits 7-9, 10-12 = 1), majors in bits 15/16 (1 = MN-major),
// N >> 3 in bits 17-22, M >> 4 in bits 24-28.
__host__ __device__ constexpr uint32_t idesc_bf16(int M, int N, int a_mn, int b_mn) {
    return (1u << 4) | (1u << 7) | (1u << 10) | (uint32_t(a_mn) << 15) | (uint32_t(b_mn) << 16) |
           (uint32_t(N >> 3) << 17) | (uint32_t(M >> 4) << 24);
}

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
    return uint32_t(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ void mma_bf16(uint32_t tmem_d, uint64_t da, uint64_t db, uint32_t idesc,
                                         uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}\n"
        :
        : "r"(tmem_d), "l"(da), "l"(db), "r"(idesc), "r"(accumulate)
        : "memory");
}
__device__ __forceinline__ void mma_commit(uint32_t mbar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];"
                 :
                 : "r"(mbar)
                 : "memory");
}
__device__ __forceinline__ void fence_before_sync() {
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void fence_after_sync() {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void fence_async_smem() {
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}
__device__ __forceinline__ void mbar_init(uint32_t mbar) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(mbar) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
// Polls a bounded mbarrier wait makes before it gives up (host-settable
// through mclsgpu_set_wait_limit; 0 makes every such wait give up at once).
constexpr int kDefaultWaitPolls = 1 << 20;
__device__ int g_wait_polls = kDefaultWaitPolls;

// Bounded wait for the phase `parity` of an mbarrier to complete, at most
// `polls` polls.
__device__ __forceinline__ bool mbar_wait_n(uint32_t mbar, uint32_t parity, int polls) {
    for (int it = 0; it < polls; ++it) {
        uint32_t ok;
        asm volatile(
            "{\n\t.reg .pred P1;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 P1, [%1], %2;\n\t"
            "selp.b32 %0, 1, 0, P1;\n\t}\n"
            : "=r"(ok)
            : "r"(mbar), "r"(parity)
            : "memory");
        if (ok) return true;
    }
    return false;
}
// The bound in force, read once per kernel (a load per wait is on the chain).
__device__ __forceinline__ int wait_polls() {
    return *reinterpret_cast<volatile int*>(&g_wait_polls);
}
// After a wait gave up, the MMAs of the phase it waited for may still be
// writing tensor memory.  The thread that issued them waits for that phase
// (with the default bound, whatever the host limit) before the columns are
// released.
__device__ __forceinline__ void mbar_drain(uint32_t mbar, uint32_t parity) {
    mbar_wait_n(mbar, parity, kDefaultWaitPolls);
}
__device__ __forceinline__ void tmem_alloc(uint32_t slot, uint32_t ncols) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(slot),
                 "r"(ncols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t base, uint32_t ncols) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(base), "r"(ncols)
                 : "memory");
}
// 16 consecutive FP32 columns of this thread's TMEM lane (32x32b shape).
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, float* v) {
    uint32_t r[16];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
        "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
          "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
          "=r"(r[14]), "=r"(r[15])
        : "r"(taddr)
        : "memory");
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int k = 0; k < 16; ++k) v[k] = __uint_as_float(r[k]);
}

// 32 consecutive columns.
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, float* v) {
    uint32_t r[32];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
        "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
        "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
          "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
          "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]),
          "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]),
          "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr)
        : "memory");
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int k = 0; k < 32; ++k) v[k] = __uint_as_float(r[k]);
}

__device__ __forceinline__ float bf16_round(float x) {
    return __bfloat162float(__float2bfloat16_rn(x));
}
// 8 values -> one 16-byte store of BF16 at a K-major tile position.
__device__ __forceinline__ void store8(unsigned char* tile, int r, int c0, int R, const float* v) {
    __align__(16) __nv_bfloat16 h[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) h[k] = __float2bfloat16_rn(v[k]);
    *reinterpret_cast<uint4*>(tile + kmaj_off(r, c0, R)) = *reinterpret_cast<const uint4*>(h);
}
__device__ __forceinline__ void load8(const unsigned char* tile, int r, int c0, int R, float* v) {
    __align__(16) __nv_bfloat16 h[8];
    *reinterpret_cast<uint4*>(h) = *reinterpret_cast<const uint4*>(tile + kmaj_off(r, c0, R));
#pragma unroll
    for (int k = 0; k < 8; ++k) v[k] = __bfloat162float(h[k]);
}

struct SlotTable {
    int off[kMaxSlots];
    int K;
    int centre;
    // Two-step offsets o_s + o_t of H = I - M A: distinct values in
    // ascending order, pair[s][t] their index, pcentre the index of 0.
    unsigned char pair[kMaxSlots][kMaxSlots];
    int npair;
    int pcentre;
};

// Features of row i from the diagonal-offset storage of A (FP64 values,
// features formed in FP32: the network reads them in BF16).  KT slots when
// KT > 0, t.K otherwise.  Every load is issued before the first division, so
// a row costs one memory round trip, not one per slot.
template <int KT>
__device__ __forceinline__ void row_features(const double* dia, int n, const SlotTable& t, int i,
                                             float* f) {
    constexpr int kMax = KT > 0 ? KT : kMaxSlots;
    const int K = KT > 0 ? KT : t.K;
#pragma unroll
    for (int k = 0; k < kF; ++k) f[k] = 0.f;
    if (i >= n) return;
    const double* centre = dia + size_t(t.centre) * n;
    double a[kMax], d[kMax];
    const float aii = float(centre[i]);
#pragma unroll
    for (int s = 0; s < kMax; ++s) {
        a[s] = 0.0;
        d[s] = 1.0;
        if (s < K) {
            const int j = i + t.off[s];
            a[s] = dia[size_t(s) * n + i];
            if (j >= 0 && j < n) d[s] = centre[j];
            else a[s] = 0.0;
        }
    }
    // Pair q: the q-th slot without the centre.
#pragma unroll
    for (int q = 0; q < kMax - 1; ++q) {
        const double av = q < t.centre ? a[q] : a[q + 1];
        const double dv = q < t.centre ? d[q] : d[q + 1];
        if (av != 0.0) {
            f[2 * q] = float(av) / aii;
            f[2 * q + 1] = logf(float(dv) / aii);
        }
    }
}

// Stage W (rows x cols, FP32, row-major out x in) as a K-major BF16 tile.
__device__ void stage_weights(unsigned char* tile, const float* W, int rows, int cols) {
    for (int idx = threadIdx.x; idx < rows * (cols / 8); idx += blockDim.x) {
        const int r = idx / (cols / 8), c0 = (idx % (cols / 8)) * 8;
        float v[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) v[k] = W[r * cols + c0 + k];
        store8(tile, r, c0, rows, v);
    }
}

struct SpaiFwdArgs {
    const float* params;
    const double* dia;     // A by diagonal offsets
    const int* rp;         // A's CSR pattern (M shares it)
    const int* ci;
    SlotTable slots;
    int n;
    double* mval;          // M values on A's pattern (may be null)
    double* mdia;          // M by diagonal offsets, 0 off the pattern (may be null)
    unsigned short* mask;  // with mdia: bit s = slot s is on the pattern
    float* out;            // raw outputs [n][16] (may be null)
    int out_align;         // alignment of out, bytes: 32, 16 or its elements' 4
    int* status;
};

// Shared memory of the forward kernel (dynamic, 1024-byte aligned base).
constexpr int kFwdW1 = 0;                          // 64 x 16
constexpr int kFwdW2 = kFwdW1 + kH * kF * 2;       // 64 x 64
constexpr int kFwdW3 = kFwdW2 + kH * kH * 2;       // 16 x 64
constexpr int kFwdX = kFwdW3 + kO * kH * 2;        // 128 x 16
constexpr int kFwdH = kFwdX + kTileRows * kF * 2;  // 128 x 64, then the tile's M values
constexpr int kFwdBias = kFwdH + kTileRows * kH * 2;  // b1, b2, b3 (FP32)
constexpr int kFwdBar = kFwdBias + (2 * kH + kO) * 4;
constexpr int kFwdSmem = kFwdBar + 64;
// CTAs per SM: the registers' and shared memory's limit; their tensor-memory
// columns (64 each) are within the SM's 512.
constexpr int kFwdCtas = 6;
constexpr int kFwdCols = 64;
static_assert(kTileRows * kMaxSlots * 8 <= kTileRows * kH * 2, "the tile's M values fit H");
static_assert(kFwdCtas * (kFwdSmem + 1024) <= 227 * 1024 && kFwdCtas * kFwdCols <= 512,
              "forward kernel residency");

// One hidden layer's epilogue for this thread's row: 64 accumulator columns
// plus bias, ReLU, to BF16 as the next layer's K-major operand.
__device__ __forceinline__ void hidden_epilogue(uint32_t taddr, const float* bias,
                                                unsigned char* H, int row) {
#pragma unroll 1
    for (int c = 0; c < kH; c += 32) {
        float z[32];
        tmem_ld32(taddr + c, z);
#pragma unroll
        for (int k = 0; k < 32; k += 4) {
            const float4 b = *reinterpret_cast<const float4*>(bias + c + k);
            z[k] = fmaxf(z[k] + b.x, 0.f);
            z[k + 1] = fmaxf(z[k + 1] + b.y, 0.f);
            z[k + 2] = fmaxf(z[k + 2] + b.z, 0.f);
            z[k + 3] = fmaxf(z[k + 3] + b.w, 0.f);
        }
#pragma unroll
        for (int k = 0; k < 32; k += 8) store8(H, row, c + k, kTileRows, z + k);
    }
}

// The backward epilogue: dZ = dH where the activation is positive, to BF16.
__device__ __forceinline__ void masked_epilogue(uint32_t taddr, const unsigned char* H,
                                                unsigned char* dZ, int row) {
#pragma unroll 1
    for (int c = 0; c < kH; c += 32) {
        float d[32];
        tmem_ld32(taddr + c, d);
#pragma unroll
        for (int k = 0; k < 32; k += 8) {
            float h[8];
            load8(H, row, c + k, kTileRows, h);
#pragma unroll
            for (int j = 0; j < 8; ++j) d[k + j] = h[j] > 0.f ? d[k + j] : 0.f;
            store8(dZ, row, c + k, kTileRows, d + k);
        }
    }
}

// Row `row` of M from its outputs: on A's pattern into `stage` (the tile's
// entries in order, from tile entry e0) and/or by diagonal offset.
template <int KT>
__device__ __forceinline__ void emit_m(const SpaiFwdArgs& a, int row, const float* o,
                                       double* stage, int e0) {
    constexpr int kMax = KT > 0 ? KT : kMaxSlots;
    const int K = KT > 0 ? KT : a.slots.K;
    const int p0 = a.rp[row], len = a.rp[row + 1] - p0;
    const double inv = 1.0 / a.dia[size_t(a.slots.centre) * a.n + row];
    double m[kMax];
#pragma unroll
    for (int s = 0; s < kMax; ++s)
        m[s] = ((s == a.slots.centre ? 1.0 : 0.0) + double(o[s])) * inv;
    // A full row's entries are its slots in order (columns are sorted).
    unsigned mask = (1u << K) - 1u;
    if (len == K) {
        if (stage) {
#pragma unroll
            for (int s = 0; s < kMax; ++s)
                if (s < K) stage[p0 - e0 + s] = m[s];
        }
    } else {
        mask = 0u;
        for (int p = p0; p < p0 + len; ++p) {
            const int d = a.ci[p] - row;
            double v = 0.0;
#pragma unroll
            for (int s = 0; s < kMax; ++s)
                if (s < K && a.slots.off[s] == d) {
                    v = m[s];
                    mask |= 1u << s;
                }
            if (stage) stage[p - e0] = v;
        }
    }
    if (a.mdia) {
#pragma unroll
        for (int s = 0; s < kMax; ++s)
            if (s < K) a.mdia[size_t(s) * a.n + row] = (mask >> s) & 1u ? m[s] : 0.0;
        a.mask[row] = (unsigned short)mask;
    }
}

// Forward pass: one CTA (4 warps, one row per thread) per 128-row tile,
// persistent over tiles; every layer accumulates in the same 64 TMEM columns.
//
// What bounds it: the chain of one tile (features, MMA, TMEM load, ReLU to
// BF16, next MMA, ...), hidden by running six CTAs per SM.  At 128^3 (16,384
// tiles, 376 MB in and out, 58 us at the copy rate) it took 804 us with three
// CTAs of 162 registers, dependent loads slot by slot in the features, biases
// read from global memory and M stored entry by entry; those are now one batch
// of loads, shared memory, and a tile's M values staged in shared memory and
// written in order: 172 to 176 us.
template <int KT>
__global__ void __launch_bounds__(kThreads, kFwdCtas) k_spai_forward(SpaiFwdArgs a) {
    extern __shared__ __align__(1024) unsigned char smem[];
    const int tid = threadIdx.x, warp = tid >> 5;
    uint64_t* bar = reinterpret_cast<uint64_t*>(smem + kFwdBar);
    uint32_t* tslot = reinterpret_cast<uint32_t*>(smem + kFwdBar + 16);
    float* bias = reinterpret_cast<float*>(smem + kFwdBias);
    const uint32_t mbar = smem_u32(bar);
    stage_weights(smem + kFwdW1, a.params + kW1, kH, kF);
    stage_weights(smem + kFwdW2, a.params + kW2, kH, kH);
    stage_weights(smem + kFwdW3, a.params + kW3, kO, kH);
    if (tid < kH) {
        bias[tid] = a.params[kB1 + tid];
        bias[kH + tid] = a.params[kB2 + tid];
    }
    if (tid < kO) bias[2 * kH + tid] = a.params[kB3 + tid];
    if (tid == 0) mbar_init(mbar);
    if (warp == 0) tmem_alloc(smem_u32(tslot), kFwdCols);
    const int polls = wait_polls();
    fence_async_smem();
    fence_before_sync();
    __syncthreads();
    fence_after_sync();
    const uint32_t tmem = *tslot;
    const uint32_t lane_base = tmem + (uint32_t(warp * 32) << 16);
    const uint32_t sX = smem_u32(smem + kFwdX), sH = smem_u32(smem + kFwdH);
    const uint32_t sW1 = smem_u32(smem + kFwdW1), sW2 = smem_u32(smem + kFwdW2),
                   sW3 = smem_u32(smem + kFwdW3);
    uint32_t phase = 0;
    bool ok = true;
    // Thread 0 issues the MMAs, and only while its own waits succeed, so at
    // most one committed phase is outstanding when a wait gives up.
    bool pend = false;
    uint32_t pend_parity = 0;
    auto wait_mma = [&]() {
        const bool got = ok && mbar_wait_n(mbar, phase, polls);
        if (ok && !got) {
            pend = true;
            pend_parity = phase;
        }
        ok = got;
        phase ^= 1;
        fence_after_sync();
    };
    auto stage_sync = [&]() {
        fence_async_smem();
        fence_before_sync();
        __syncthreads();
    };
    const int ntiles = (a.n + kTileRows - 1) / kTileRows;
    for (int tile = blockIdx.x; tile < ntiles && ok; tile += gridDim.x) {
        const int row = tile * kTileRows + tid;
        {
            float f[kF];
            row_features<KT>(a.dia, a.n, a.slots, row, f);
            store8(smem + kFwdX, tid, 0, kTileRows, f);
            store8(smem + kFwdX, tid, 8, kTileRows, f + 8);
        }
        stage_sync();
        // Layer 1: Z1 = X W1^T  (M 128, N 64, K 16).
        if (tid == 0 && ok) {
            fence_after_sync();
            mma_bf16(tmem, desc_kmajor(sX, kTileRows, 0), desc_kmajor(sW1, kH, 0),
                     idesc_bf16(128, kH, 0, 0), 0);
            mma_commit(mbar);
        }
        wait_mma();
        hidden_epilogue(lane_base, bias, smem + kFwdH, tid);
        stage_sync();
        // Layer 2: Z2 = H1 W2^T  (M 128, N 64, K 64), over Z1, which every
        // thread has read before the barrier above.
        if (tid == 0 && ok) {
            fence_after_sync();
            for (int ks = 0; ks < kH / 16; ++ks)
                mma_bf16(tmem, desc_kmajor(sH, kTileRows, ks), desc_kmajor(sW2, kH, ks),
                         idesc_bf16(128, kH, 0, 0), ks > 0);
            mma_commit(mbar);
        }
        wait_mma();
        // H2 overwrites H1: layer 2's operands are consumed (its MMAs are
        // complete once the barrier phase has flipped).
        hidden_epilogue(lane_base, bias + kH, smem + kFwdH, tid);
        stage_sync();
        // Layer 3: out = H2 W3^T  (M 128, N 16, K 64).
        if (tid == 0 && ok) {
            fence_after_sync();
            for (int ks = 0; ks < kH / 16; ++ks)
                mma_bf16(tmem, desc_kmajor(sH, kTileRows, ks), desc_kmajor(sW3, kO, ks),
                         idesc_bf16(128, kO, 0, 0), ks > 0);
            mma_commit(mbar);
        }
        wait_mma();
        float o[kO];
        tmem_ld16(lane_base, o);
        fence_before_sync();
        // The next tile's layer 1 reuses these columns; a timed-out wait on
        // any thread ends the loop on all of them.
        ok = __syncthreads_and(ok);
        if (!ok) break;
#pragma unroll
        for (int k = 0; k < kO; ++k) o[k] += bias[2 * kH + k];
        if (a.out && row < a.n) {
            float* dst = a.out + size_t(row) * kO;
            if (a.out_align == 32) {
#pragma unroll
                for (int k = 0; k < kO; k += 8)
                    asm volatile("st.global.v8.f32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"l"(dst + k),
                                 "f"(o[k]), "f"(o[k + 1]), "f"(o[k + 2]), "f"(o[k + 3]),
                                 "f"(o[k + 4]), "f"(o[k + 5]), "f"(o[k + 6]), "f"(o[k + 7])
                                 : "memory");
            } else if (a.out_align == 16) {
#pragma unroll
                for (int k = 0; k < kO; k += 4)
                    *reinterpret_cast<float4*>(dst + k) =
                        make_float4(o[k], o[k + 1], o[k + 2], o[k + 3]);
            } else {
#pragma unroll
                for (int k = 0; k < kO; ++k) dst[k] = o[k];
            }
        }
        if (a.mval) {
            // Layer 3 has read H: the tile's M entries take its place.
            double* stage = reinterpret_cast<double*>(smem + kFwdH);
            const int last = min(a.n, (tile + 1) * kTileRows);
            const int e0 = a.rp[tile * kTileRows], e1 = a.rp[last];
            if (row < a.n) emit_m<KT>(a, row, o, stage, e0);
            __syncthreads();
            for (int e = tid; e < e1 - e0; e += kThreads) a.mval[e0 + e] = stage[e];
        } else if (a.mdia && row < a.n) {
            emit_m<KT>(a, row, o, nullptr, 0);
        }
    }
    if (!ok && tid == 0) atomicExch(a.status, MCLSGPU_ERR_TIMEOUT);
    if (tid == 0 && pend) mbar_drain(mbar, pend_parity);
    fence_before_sync();
    __syncthreads();
    if (warp == 0) {
        fence_after_sync();
        tmem_dealloc(tmem, kFwdCols);
    }
}

struct SpaiBwdArgs {
    const float* params;
    const double* dia;
    SlotTable slots;
    int n;
    const float* G;        // dL/dout [n][16]
    float* grad;           // parameter gradient (accumulated)
    int* status;
};

// Shared memory of the backward kernel.  The H1 and X tiles carry an extra
// 8-column group whose first column is 1 and the rest 0, so that the
// weight-gradient products also produce the bias gradients of layers 2 and 1
// (sum over rows of dZ = dZ^T * ones).
constexpr int kXC = 24;   // X tile columns: 16 features + ones group
constexpr int kH1C = 72;  // H1 tile columns: 64 + ones group
constexpr int kBwW1 = 0;                                // 64 x 16
constexpr int kBwW2 = kBwW1 + kH * kF * 2;              // 64 x 64
constexpr int kBwW3 = kBwW2 + kH * kH * 2;              // 16 x 64
constexpr int kBwX = kBwW3 + kO * kH * 2;               // 128 x 24
constexpr int kBwH1 = kBwX + kTileRows * kXC * 2;       // 128 x 72
constexpr int kBwH2 = kBwH1 + kTileRows * kH1C * 2;     // 128 x 64
constexpr int kBwG = kBwH2 + kTileRows * kH * 2;        // 128 x 16
constexpr int kBwDZ2 = kBwG + kTileRows * kO * 2;       // 128 x 64
constexpr int kBwDZ1 = kBwDZ2 + kTileRows * kH * 2;     // 128 x 64
constexpr int kBwB3 = kBwDZ1 + kTileRows * kH * 2;      // 16 floats
constexpr int kBwBias = kBwB3 + 64;                     // b1, b2 (FP32)
constexpr int kBwBar = kBwBias + 2 * kH * 4;
constexpr int kBwSmem = kBwBar + 64;
// Two CTAs per SM, 256 tensor-memory columns each: a training sample of 32^3
// rows (256 tiles) is then one tile per CTA instead of two in sequence.
constexpr int kBwCtas = 2;
constexpr int kBwCols = 256;
static_assert(kBwCtas * (kBwSmem + 1024) <= 227 * 1024 && kBwCtas * kBwCols <= 512,
              "backward kernel residency");
// TMEM columns of the backward kernel.  One 64-column buffer serves Z1, Z2,
// dH2 and dH1 in turn: each is read before the barrier that precedes the
// MMAs of the next.
constexpr uint32_t kTA = 0;      // Z1, Z2, dH2, dH1 (M 128 x 64)
constexpr uint32_t kTdW3 = 64;   // dW3^T: rows h2, cols o     (M 64 x 16)
constexpr uint32_t kTdW2 = 96;   // dW2: rows h2, cols h1 | db2 (M 64 x 72, read as 80)
constexpr uint32_t kTdW1 = 192;  // dW1: rows h1, cols in | db1 (M 64 x 24, read as 32)

// 16 consecutive sums (16-byte aligned) in four 16-byte reductions.  One by one
// almost every one of a CTA's 6,288 sums was a reduction in a sector of its own:
// 43 us for the kernel at 32^3 (256 CTAs), 20 us so.
__device__ __forceinline__ void red16(float* p, const float (&v)[16]) {
#pragma unroll
    for (int k = 0; k < 16; k += 4)
        asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(p + k), "f"(v[k]),
                     "f"(v[k + 1]), "f"(v[k + 2]), "f"(v[k + 3])
                     : "memory");
}
static_assert(kW1 % 4 == 0 && kW2 % 4 == 0 && kF == 16 && kH % 16 == 0, "aligned rows");

// Backward pass: the forward activations of each tile are recomputed, the
// output gradient G is propagated to dZ2 and dZ1, and the weight and bias
// gradients accumulate in TMEM across the CTA's tiles; at the end each CTA
// adds its sums into `grad`.  Bound by the chain of a tile (five MMA steps, each
// waiting for an epilogue) at two CTAs per SM: 20 us at 32^3.
template <int KT>
__global__ void __launch_bounds__(kThreads, kBwCtas) k_spai_backward(SpaiBwdArgs a) {
    extern __shared__ __align__(1024) unsigned char smem[];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    uint64_t* bar = reinterpret_cast<uint64_t*>(smem + kBwBar);
    uint32_t* tslot = reinterpret_cast<uint32_t*>(smem + kBwBar + 16);
    float* db3 = reinterpret_cast<float*>(smem + kBwB3);
    float* bias = reinterpret_cast<float*>(smem + kBwBias);
    const uint32_t mbar = smem_u32(bar);
    stage_weights(smem + kBwW1, a.params + kW1, kH, kF);
    stage_weights(smem + kBwW2, a.params + kW2, kH, kH);
    stage_weights(smem + kBwW3, a.params + kW3, kO, kH);
    if (tid < kO) db3[tid] = 0.f;
    if (tid < kH) {
        bias[tid] = a.params[kB1 + tid];
        bias[kH + tid] = a.params[kB2 + tid];
    }
    {
        // Ones groups (column 16 of X, column 64 of H1) for every row.
        float one[8] = {1.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
        store8(smem + kBwX, tid, 16, kTileRows, one);
        store8(smem + kBwH1, tid, 64, kTileRows, one);
    }
    if (tid == 0) mbar_init(mbar);
    if (warp == 0) tmem_alloc(smem_u32(tslot), kBwCols);
    const int polls = wait_polls();
    fence_async_smem();
    fence_before_sync();
    __syncthreads();
    fence_after_sync();
    const uint32_t tmem = *tslot;
    const uint32_t lane_base = tmem + (uint32_t(warp * 32) << 16);
    const uint32_t sW1 = smem_u32(smem + kBwW1), sW2 = smem_u32(smem + kBwW2),
                   sW3 = smem_u32(smem + kBwW3), sX = smem_u32(smem + kBwX),
                   sH1 = smem_u32(smem + kBwH1), sH2 = smem_u32(smem + kBwH2),
                   sG = smem_u32(smem + kBwG), sDZ2 = smem_u32(smem + kBwDZ2),
                   sDZ1 = smem_u32(smem + kBwDZ1);
    uint32_t phase = 0;
    bool ok = true;
    int done = 0;
    // Thread 0 issues the MMAs only while its own waits succeed (at most one
    // committed phase outstanding when a wait gives up).
    bool pend = false;
    uint32_t pend_parity = 0;
    const int ntiles = (a.n + kTileRows - 1) / kTileRows;
    auto stage_sync = [&]() {
        fence_async_smem();
        fence_before_sync();
        __syncthreads();
    };
    auto wait_mma = [&]() {
        const bool got = ok && mbar_wait_n(mbar, phase, polls);
        if (ok && !got) {
            pend = true;
            pend_parity = phase;
        }
        ok = got;
        phase ^= 1;
        fence_after_sync();
    };
    for (int tile = blockIdx.x; tile < ntiles && ok; tile += gridDim.x, ++done) {
        const int row = tile * kTileRows + tid;
        {
            float f[kF];
            row_features<KT>(a.dia, a.n, a.slots, row, f);
            store8(smem + kBwX, tid, 0, kTileRows, f);
            store8(smem + kBwX, tid, 8, kTileRows, f + 8);
        }
        stage_sync();
        if (tid == 0 && ok) {
            fence_after_sync();
            mma_bf16(tmem + kTA, desc_kmajor(sX, kTileRows, 0), desc_kmajor(sW1, kH, 0),
                     idesc_bf16(128, kH, 0, 0), 0);
            mma_commit(mbar);
        }
        wait_mma();
        hidden_epilogue(lane_base + kTA, bias, smem + kBwH1, tid);
        stage_sync();
        if (tid == 0 && ok) {
            fence_after_sync();
            for (int ks = 0; ks < kH / 16; ++ks)
                mma_bf16(tmem + kTA, desc_kmajor(sH1, kTileRows, ks), desc_kmajor(sW2, kH, ks),
                         idesc_bf16(128, kH, 0, 0), ks > 0);
            mma_commit(mbar);
        }
        wait_mma();
        hidden_epilogue(lane_base + kTA, bias + kH, smem + kBwH2, tid);
        {
            float g[kO];
#pragma unroll
            for (int k = 0; k < kO; ++k) g[k] = 0.f;
            if (row < a.n) {
                const float4* src = reinterpret_cast<const float4*>(a.G + size_t(row) * kO);
#pragma unroll
                for (int k = 0; k < kO; k += 4) {
                    const float4 q = src[k / 4];
                    g[k] = q.x;
                    g[k + 1] = q.y;
                    g[k + 2] = q.z;
                    g[k + 3] = q.w;
                }
            }
            store8(smem + kBwG, tid, 0, kTileRows, g);
            store8(smem + kBwG, tid, 8, kTileRows, g + 8);
            // db3: sum over rows of the BF16-rounded G.
#pragma unroll
            for (int k = 0; k < kO; ++k) {
                float s = bf16_round(g[k]);
#pragma unroll
                for (int d = 16; d > 0; d >>= 1) s += __shfl_xor_sync(0xffffffffu, s, d);
                if (lane == 0) atomicAdd(&db3[k], s);
            }
        }
        stage_sync();
        // dH2 = G W3 (B = W3 read MN-major: N 64 = h2, K 16 = o) and
        // dW3^T += H2^T G (A = H2 MN-major, B = G MN-major; K = 128 rows).
        if (tid == 0 && ok) {
            fence_after_sync();
            mma_bf16(tmem + kTA, desc_kmajor(sG, kTileRows, 0), desc_mnmajor(sW3, kO, 0),
                     idesc_bf16(128, kH, 0, 1), 0);
            for (int ks = 0; ks < kTileRows / 16; ++ks)
                mma_bf16(tmem + kTdW3, desc_mnmajor(sH2, kTileRows, ks),
                         desc_mnmajor(sG, kTileRows, ks), idesc_bf16(64, kO, 1, 1),
                         (done > 0 || ks > 0));
            mma_commit(mbar);
        }
        wait_mma();
        masked_epilogue(lane_base + kTA, smem + kBwH2, smem + kBwDZ2, tid);
        stage_sync();
        // dH1 = dZ2 W2 (B = W2 MN-major: N 64 = h1, K 64 = h2) and
        // [dW2 | db2] += dZ2^T [H1 | 1] (K = 128 rows).
        if (tid == 0 && ok) {
            fence_after_sync();
            for (int ks = 0; ks < kH / 16; ++ks)
                mma_bf16(tmem + kTA, desc_kmajor(sDZ2, kTileRows, ks), desc_mnmajor(sW2, kH, ks),
                         idesc_bf16(128, kH, 0, 1), ks > 0);
            for (int ks = 0; ks < kTileRows / 16; ++ks)
                mma_bf16(tmem + kTdW2, desc_mnmajor(sDZ2, kTileRows, ks),
                         desc_mnmajor(sH1, kTileRows, ks), idesc_bf16(64, kH1C, 1, 1),
                         (done > 0 || ks > 0));
            mma_commit(mbar);
        }
        wait_mma();
        masked_epilogue(lane_base + kTA, smem + kBwH1, smem + kBwDZ1, tid);
        stage_sync();
        // [dW1 | db1] += dZ1^T [X | 1] (K = 128 rows).
        if (tid == 0 && ok) {
            fence_after_sync();
            for (int ks = 0; ks < kTileRows / 16; ++ks)
                mma_bf16(tmem + kTdW1, desc_mnmajor(sDZ1, kTileRows, ks),
                         desc_mnmajor(sX, kTileRows, ks), idesc_bf16(64, kXC, 1, 1),
                         (done > 0 || ks > 0));
            mma_commit(mbar);
        }
        wait_mma();
        fence_before_sync();
        // TMEM columns A/B and every tile are reused next; a timed-out wait
        // on any thread ends the loop on all of them.
        ok = __syncthreads_and(ok);
    }
    if (!ok && tid == 0) atomicExch(a.status, MCLSGPU_ERR_TIMEOUT);
    if (tid == 0 && pend) mbar_drain(mbar, pend_parity);
    if (ok && done > 0) {
        fence_after_sync();
        // M = 64 accumulators: row 16w + t of the product sits in lane
        // 32w + t (t < 16) of TMEM.
        const int r = 16 * warp + lane;
        float v[16];
        tmem_ld16(lane_base + kTdW3, v);
        if (lane < 16)
            for (int o = 0; o < kO; ++o) atomicAdd(&a.grad[kW3 + o * kH + r], v[o]);
        for (int c = 0; c < 80; c += 16) {
            tmem_ld16(lane_base + kTdW2 + c, v);
            if (lane < 16) {
                if (c < kH) red16(&a.grad[kW2 + r * kH + c], v);
                else atomicAdd(&a.grad[kB2 + r], v[0]);
            }
        }
        for (int c = 0; c < 32; c += 16) {
            tmem_ld16(lane_base + kTdW1 + c, v);
            if (lane < 16) {
                if (c < kF) red16(&a.grad[kW1 + r * kF + c], v);
                else atomicAdd(&a.grad[kB1 + r], v[0]);
            }
        }
        __syncthreads();
        if (tid < kO) atomicAdd(&a.grad[kB3 + tid], db3[tid]);
    }
    fence_before_sync();
    __syncthreads();
    if (warp == 0) {
        fence_after_sync();
        tmem_dealloc(tmem, kBwCols);
    }
}

// z_v = A v for every training vector (blockIdx.y) and, in the vector's block
// that finishes last, wv[v] = 1 / (nvec |v|^2) (block sums in block order).
template <int KT>
__global__ void __launch_bounds__(256) k_spai_vectors(int n, int nvec, const double* dia,
                                                      SlotTable slots, const double* V, double* Z,
                                                      double* part, unsigned* tickets,
                                                      double* wv) {
    constexpr int kMax = KT > 0 ? KT : kMaxSlots;
    const int K = KT > 0 ? KT : slots.K;
    __shared__ double sh[8];
    __shared__ bool last;
    const int v = blockIdx.y;
    const double* x = V + size_t(v) * n;
    double sq = 0.0;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        double z = 0.0;
#pragma unroll
        for (int s = 0; s < kMax; ++s) {
            const int j = i + slots.off[s];
            if (s < K && j >= 0 && j < n) z = fma(dia[size_t(s) * n + i], x[j], z);
        }
        Z[size_t(v) * n + i] = z;
        sq = fma(x[i], x[i], sq);
    }
    for (int d = 16; d > 0; d >>= 1) sq += __shfl_down_sync(0xffffffffu, sq, d);
    if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = sq;
    __syncthreads();
    double* vp = part + size_t(v) * gridDim.x;
    if (threadIdx.x == 0) {
        double t = 0.0;
        for (int w = 0; w < 8; ++w) t += sh[w];
        vp[blockIdx.x] = t;
        __threadfence();
        last = atomicAdd(&tickets[v], 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    double t = 0.0;
    for (int k = threadIdx.x; k < int(gridDim.x); k += blockDim.x) t += __ldcg(&vp[k]);
    for (int d = 16; d > 0; d >>= 1) t += __shfl_down_sync(0xffffffffu, t, d);
    if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = t;
    __syncthreads();
    if (threadIdx.x == 0) {
        t = 0.0;
        for (int w = 0; w < 8; ++w) t += sh[w];
        wv[v] = t > 0.0 ? 1.0 / (double(nvec) * t) : 0.0;
    }
}

// The row-sum penalty's part of the loss and of row i's output gradient:
// pen_w/n * max(0, W_i - pen_c)^2, W_i the row sum of |H| for H = I - M A (the
// factor by which a forward walk's weight grows at state i), from row i of M
// and the rows of A at its neighbours.
__device__ double penalty_row(int n, int i, const double* m, unsigned mask, const double* dia,
                              const SlotTable& slots, double inv, double pen_w, double pen_c,
                              double* g) {
    double h[kMaxSlots * kMaxSlots];
    for (int q = 0; q < slots.npair; ++q) h[q] = 0.0;
    h[slots.pcentre] = 1.0;
    for (int s = 0; s < slots.K; ++s) {
        const int k = i + slots.off[s];
        if (!((mask >> s) & 1u) || k < 0 || k >= n) continue;
        for (int t = 0; t < slots.K; ++t) h[slots.pair[s][t]] -= m[s] * dia[size_t(t) * n + k];
    }
    double W = 0.0;
    for (int q = 0; q < slots.npair; ++q) W += fabs(h[q]);
    const double pen = W - pen_c;
    if (!(pen > 0.0)) return 0.0;
    const double coef = 2.0 * pen_w * pen / double(n) * inv;
    for (int s = 0; s < slots.K; ++s) {
        const int k = i + slots.off[s];
        if (!((mask >> s) & 1u) || k < 0 || k >= n) continue;
        double dW = 0.0;
        for (int t = 0; t < slots.K; ++t) {
            const double hv = h[slots.pair[s][t]];
            const double sg = hv > 0.0 ? 1.0 : (hv < 0.0 ? -1.0 : 0.0);
            dW -= sg * dia[size_t(t) * n + k];
        }
        g[s] += coef * dW;
    }
    return pen_w * pen * pen / double(n);
}

// e_v = v - M (A v) per row; loss and the output gradient G.  PEN: with the
// row-sum penalty.  A block is 32 rows by kLossGroups groups of vectors (a
// 32^3 sample alone has too few rows to fill the chip); the groups' gradients
// are added in shared memory in group order.
constexpr int kLossGroups = 8;
template <int KT, bool PEN>
__global__ void __launch_bounds__(32 * kLossGroups)
    k_spai_loss_grad(int n, int nvec, const double* mdia, const unsigned short* mask,
                     const double* dia, SlotTable slots, const double* V, const double* Z,
                     const double* wv, double pen_w, double pen_c, float* G, double* loss) {
    constexpr int kMax = KT > 0 ? KT : kMaxSlots;
    const int K = KT > 0 ? KT : slots.K;
    __shared__ double sg[kLossGroups][kMax][32];
    const int lane = threadIdx.x & 31, grp = threadIdx.x >> 5;
    const int i = blockIdx.x * 32 + lane;
    const bool live = i < n;
    double part = 0.0;
    double g[kMax];
#pragma unroll
    for (int s = 0; s < kMax; ++s) g[s] = 0.0;
    if (live) {
        const double inv = 1.0 / dia[size_t(slots.centre) * n + i];
        const unsigned msk = mask[i];
        double m[kMax];
#pragma unroll
        for (int s = 0; s < kMax; ++s) m[s] = s < K ? mdia[size_t(s) * n + i] : 0.0;
        if constexpr (PEN)
            if (grp == 0)
                part += penalty_row(n, i, m, msk, dia, slots, inv, pen_w, pen_c, g);
        for (int v = grp; v < nvec; v += kLossGroups) {
            const double* z = Z + size_t(v) * n;
            double zs[kMax];
            double mz = 0.0;
#pragma unroll
            for (int s = 0; s < kMax; ++s) {
                // A slot off the row's pattern has no neighbour.
                zs[s] = s < K && ((msk >> s) & 1u) ? z[i + slots.off[s]] : 0.0;
                mz += m[s] * zs[s];
            }
            const double e = V[size_t(v) * n + i] - mz;
            part += e * e * wv[v];
            const double c = -2.0 * e * wv[v] * inv;
#pragma unroll
            for (int s = 0; s < kMax; ++s) g[s] += c * zs[s];
        }
    }
#pragma unroll
    for (int s = 0; s < kMax; ++s) sg[grp][s][lane] = g[s];
    __syncthreads();
    // Group grp sums slots 2 grp and 2 grp + 1 of the 16 outputs.
    if (live) {
        float o[2] = {0.f, 0.f};
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            const int s = 2 * grp + q;
            if (s < K) {
                double t = 0.0;
                for (int w = 0; w < kLossGroups; ++w) t += sg[w][s][lane];
                o[q] = float(t);
            }
        }
        *reinterpret_cast<float2*>(G + size_t(i) * kO + 2 * grp) = make_float2(o[0], o[1]);
    }
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) part += __shfl_xor_sync(0xffffffffu, part, d);
    __shared__ double sl[kLossGroups];
    if (lane == 0) sl[grp] = part;
    __syncthreads();
    if (threadIdx.x == 0) {
        double t = 0.0;
        for (int w = 0; w < kLossGroups; ++w) t += sl[w];
        atomicAdd(loss, t);
    }
}

__global__ void k_adam(float* p, float* m, float* v, const float* g, int count, float lr,
                       float b1, float b2, float eps, float c1, float c2, float clip) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= count) return;
    float gi = g[i];
    if (clip > 0.f) gi = fminf(fmaxf(gi, -clip), clip);
    const float mi = b1 * m[i] + (1.f - b1) * gi;
    const float vi = b2 * v[i] + (1.f - b2) * gi * gi;
    m[i] = mi;
    v[i] = vi;
    p[i] -= lr * (mi / c1) / (sqrtf(vi / c2) + eps);
}

// y = v - M (A v) for the power iteration on H = I - M A.
__global__ void k_sub(int n, const double* v, const double* u, double* y) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        y[i] = v[i] - u[i];
}
__global__ void k_scale_by_norm(int n, double* v, const double* sq) {
    const double s = *sq > 0.0 ? 1.0 / sqrt(*sq) : 0.0;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        v[i] *= s;
}

inline int grid_for(long long work, int threads = 256, int cap = 148 * 16) {
    long long g = (work + threads - 1) / threads;
    if (g < 1) g = 1;
    return int(g > cap ? cap : g);
}

}  // namespace
}  // namespace mclsgpu

struct mclsgpu_spai {
    mclsgpu_context* ctx = nullptr;
    int slots = 0;
    float* params = nullptr;  // FP32 master parameters
    float* grad = nullptr;
    float* m = nullptr;       // Adam moments
    float* v = nullptr;
    long long step = 0;
    double pen_w = 0.0;       // row-sum penalty weight (0 = off)
    double pen_c = 1.0;       // row-sum threshold
    // Scratch of the training gradient, kept between calls up to kScratchKeep
    // bytes (released with the network).
    unsigned char* scratch = nullptr;
    size_t scratch_bytes = 0;
};

namespace mclsgpu {
namespace {

// Slot table of an operator stored by diagonal offsets.
int slot_table(mclsgpu_context* ctx, const mclsgpu_operator* op, int want, SlotTable& t) {
    if (op->dia_k <= 0 || !op->dia_val)
        return set_error(ctx, MCLSGPU_ERR_UNSUPPORTED,
                         "learned SPAI needs an operator with a fixed stencil (diagonal-offset "
                         "storage)");
    if (op->dia_k > kMaxSlots)
        return set_error(ctx, MCLSGPU_ERR_UNSUPPORTED,
                         "learned SPAI: %d stencil offsets, at most %d supported", op->dia_k,
                         kMaxSlots);
    if (want > 0 && op->dia_k != want)
        return set_error(ctx, MCLSGPU_ERR_INVALID_ARG,
                         "learned SPAI network has %d slots, operator has %d stencil offsets",
                         want, op->dia_k);
    t.K = op->dia_k;
    t.centre = -1;
    for (int s = 0; s < t.K; ++s) {
        t.off[s] = op->dia_off[s];
        if (op->dia_off[s] == 0) t.centre = s;
    }
    for (int s = t.K; s < kMaxSlots; ++s) t.off[s] = 0;  // never selected (s < K)
    if (t.centre < 0)
        return set_error(ctx, MCLSGPU_ERR_UNSUPPORTED, "learned SPAI: operator has no diagonal");
    std::vector<int> sums;
    for (int a = 0; a < t.K; ++a)
        for (int b = 0; b < t.K; ++b) sums.push_back(t.off[a] + t.off[b]);
    std::sort(sums.begin(), sums.end());
    sums.erase(std::unique(sums.begin(), sums.end()), sums.end());
    t.npair = int(sums.size());
    std::memset(t.pair, 0, sizeof(t.pair));
    for (int a = 0; a < t.K; ++a)
        for (int b = 0; b < t.K; ++b)
            t.pair[a][b] = (unsigned char)(std::lower_bound(sums.begin(), sums.end(),
                                                            t.off[a] + t.off[b]) -
                                           sums.begin());
    t.pcentre = int(std::lower_bound(sums.begin(), sums.end(), 0) - sums.begin());
    return MCLSGPU_OK;
}

// Calls f(integral_constant<int, K>) with the operator's slot count when it
// is one of the unrolled ones (5-, 7- and 9-point stencils), else with 0.
template <class F>
void with_slots(int K, F f) {
    switch (K) {
        case 5: f(std::integral_constant<int, 5>{}); break;
        case 7: f(std::integral_constant<int, 7>{}); break;
        case 9: f(std::integral_constant<int, 9>{}); break;
        default: f(std::integral_constant<int, 0>{});
    }
}

// The kernels' dynamic shared memory exceeds the 48 KB default: opt in once
// per device (the attribute belongs to the device's context).
std::mutex g_attr_mutex;
bool g_attr_set[64] = {false};

int set_smem_attributes(mclsgpu_context* ctx) {
    std::lock_guard<std::mutex> lock(g_attr_mutex);
    const int d = ctx->device;
    if (d >= 0 && d < 64 && g_attr_set[d]) return MCLSGPU_OK;
    cudaError_t e = cudaSuccess;
    for (int K : {0, 5, 7, 9})
        with_slots(K, [&](auto k) {
            constexpr int KT = decltype(k)::value;
            if (e == cudaSuccess)
                e = cudaFuncSetAttribute(k_spai_forward<KT>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, kFwdSmem);
            if (e == cudaSuccess)
                e = cudaFuncSetAttribute(k_spai_backward<KT>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, kBwSmem);
        });
    if (e != cudaSuccess) return cuda_fail(ctx, e, "spai shared-memory opt-in");
    if (d >= 0 && d < 64) g_attr_set[d] = true;
    return MCLSGPU_OK;
}

int launch_forward(mclsgpu_spai* net, mclsgpu_operator* op, const SlotTable& t, double* mval,
                   float* out, double* mdia = nullptr, unsigned short* mask = nullptr) {
    mclsgpu_context* ctx = net->ctx;
    int rc = set_smem_attributes(ctx);
    if (rc) return rc;
    SpaiFwdArgs a{};
    a.params = net->params;
    a.dia = op->dia_val;
    a.rp = op->A.rp;
    a.ci = op->A.ci;
    a.slots = t;
    a.n = op->A.n;
    a.mval = mval;
    a.mdia = mdia;
    a.mask = mask;
    a.out = out;
    const uintptr_t at = reinterpret_cast<uintptr_t>(out);
    a.out_align = at % 32 == 0 ? 32 : at % 16 == 0 ? 16 : 4;
    a.status = ctx->d_status;
    const int ntiles = (op->A.n + kTileRows - 1) / kTileRows;
    const int fit = ctx->num_sms * kFwdCtas;
    const int grid = ntiles < fit ? ntiles : fit;
    drop_stale_error();
    with_slots(t.K, [&](auto k) {
        k_spai_forward<decltype(k)::value><<<grid, kThreads, kFwdSmem, ctx->stream>>>(a);
    });
    cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? MCLSGPU_OK : cuda_fail(ctx, e, "spai forward launch");
}

// Scratch of one gradient: sub-arrays of one allocation.
constexpr size_t kScratchKeep = size_t(256) << 20;
struct GradScratch {
    double* mdia;
    double* Z;
    double* part;
    double* wv;
    float* G;
    unsigned short* mask;
    double* loss;         // loss, then the tickets: cleared together
    unsigned* tickets;
    size_t clear;         // bytes from loss on
};

size_t grad_layout(unsigned char* base, int n, int nvec, int K, int blocks, GradScratch* g) {
    size_t at = 0;
    auto take = [&](size_t bytes) {
        unsigned char* p = base + at;
        at += (bytes + 255) & ~size_t(255);
        return p;
    };
    g->mdia = reinterpret_cast<double*>(take(sizeof(double) * n * K));
    g->Z = reinterpret_cast<double*>(take(sizeof(double) * n * nvec));
    g->part = reinterpret_cast<double*>(take(sizeof(double) * nvec * blocks));
    g->wv = reinterpret_cast<double*>(take(sizeof(double) * nvec));
    g->G = reinterpret_cast<float*>(take(sizeof(float) * n * kO));
    g->mask = reinterpret_cast<unsigned short*>(take(sizeof(unsigned short) * n));
    g->clear = sizeof(double) + sizeof(unsigned) * nvec;
    g->loss = reinterpret_cast<double*>(take(g->clear));
    g->tickets = reinterpret_cast<unsigned*>(g->loss + 1);
    return at;
}

// Zero the gradient, then loss + gradient of the parameters on (op, V).
//
// A 32^3 sample with 15 vectors took 0.4 ms in 65 launches (A v and |v|^2 one
// vector at a time, the loss with one thread per row walking the CSR row
// twice per vector) and 2 to 22 ms in the seven allocations and releases of
// each call.  Now: one pass over all vectors, the network's pass (M by
// diagonals), the loss pass, the backward pass, and scratch that is kept.
int gradient(mclsgpu_spai* net, mclsgpu_operator* op, const double* V, int nvec, double* loss_out) {
    mclsgpu_context* ctx = net->ctx;
    cudaStream_t s = ctx->stream;
    SlotTable t;
    int rc = slot_table(ctx, op, net->slots, t);
    if (rc) return rc;
    if (nvec < 1 || nvec > 1024)
        return set_error(ctx, MCLSGPU_ERR_INVALID_ARG, "spai gradient: 1..1024 vectors");
    const int n = op->A.n;
    const int blocks = grid_for(n, 256, 4 * ctx->num_sms);
    GradScratch g;
    const size_t bytes = grad_layout(nullptr, n, nvec, t.K, blocks, &g);
    unsigned char* mem = net->scratch;
    cudaError_t e = cudaSuccess;
    if (bytes > net->scratch_bytes) {
        const bool keep = bytes <= kScratchKeep;
        if (keep) {
            dfree(net->scratch);
            net->scratch_bytes = 0;
        }
        if ((e = dmalloc(&mem, bytes)) != cudaSuccess) return cuda_fail(ctx, e, "cudaMalloc");
        if (keep) {
            net->scratch = mem;
            net->scratch_bytes = bytes;
        }
    }
    grad_layout(mem, n, nvec, t.K, blocks, &g);
    cudaMemsetAsync(net->grad, 0, sizeof(float) * kParams, s);
    cudaMemsetAsync(g.loss, 0, g.clear, s);
    rc = launch_forward(net, op, t, nullptr, nullptr, g.mdia, g.mask);
    if (!rc) {
        SpaiBwdArgs b{};
        b.params = net->params;
        b.dia = op->dia_val;
        b.slots = t;
        b.n = n;
        b.G = g.G;
        b.grad = net->grad;
        b.status = ctx->d_status;
        const int ntiles = (n + kTileRows - 1) / kTileRows;
        const int fit = ctx->num_sms * kBwCtas;
        const int grid = ntiles < fit ? ntiles : fit;
        with_slots(t.K, [&](auto k) {
            constexpr int KT = decltype(k)::value;
            k_spai_vectors<KT><<<dim3(blocks, nvec), 256, 0, s>>>(
                n, nvec, op->dia_val, t, V, g.Z, g.part, g.tickets, g.wv);
            auto loss_grad = net->pen_w > 0.0 ? k_spai_loss_grad<KT, true>
                                              : k_spai_loss_grad<KT, false>;
            loss_grad<<<(n + 31) / 32, 32 * kLossGroups, 0, s>>>(
                n, nvec, g.mdia, g.mask, op->dia_val, t, V, g.Z, g.wv, net->pen_w, net->pen_c,
                g.G, g.loss);
            k_spai_backward<KT><<<grid, kThreads, kBwSmem, s>>>(b);
        });
        e = cudaGetLastError();
        if (e != cudaSuccess) rc = cuda_fail(ctx, e, "spai backward launch");
    }
    if (!rc) {
        double l = 0.0;
        e = cudaMemcpyAsync(&l, g.loss, sizeof(double), cudaMemcpyDeviceToHost, s);
        if (e == cudaSuccess) e = cudaStreamSynchronize(s);
        if (e != cudaSuccess) rc = cuda_fail(ctx, e, "spai gradient");
        if (!rc) rc = check_device_status(ctx);
        if (loss_out) *loss_out = l;
    }
    if (mem != net->scratch) dfree(mem);
    return rc;
}

// Power-iteration estimate of rho(I - M A) (M as CSR on any pattern).
int rho_estimate(mclsgpu_context* ctx, const DevCsr& A, const DevCsr& M, int iters, uint64_t seed,
                 double* rho) {
    const int n = A.n;
    cudaStream_t s = ctx->stream;
    double *v = nullptr, *w = nullptr, *u = nullptr, *part = nullptr, *sq = nullptr;
    cudaError_t e;
    if ((e = dmalloc(&v, n)) != cudaSuccess || (e = dmalloc(&w, n)) != cudaSuccess ||
        (e = dmalloc(&u, n)) != cudaSuccess ||
        (e = dmalloc(&part, size_t(scan_partials_needed(n)))) != cudaSuccess ||
        (e = dmalloc(&sq, size_t(iters + 1))) != cudaSuccess) {
        dfree(v); dfree(w); dfree(u); dfree(part); dfree(sq);
        return cuda_fail(ctx, e, "cudaMalloc");
    }
    std::vector<double> h(n);
    std::mt19937_64 gen(seed);
    std::uniform_real_distribution<double> U(-1.0, 1.0);
    for (int i = 0; i < n; ++i) h[i] = U(gen);
    cudaMemcpyAsync(v, h.data(), sizeof(double) * n, cudaMemcpyHostToDevice, s);
    sum_sq(s, v, n, part, sq);
    k_scale_by_norm<<<grid_for(n), 256, 0, s>>>(n, v, sq);
    for (int k = 0; k < iters; ++k) {
        spmv(s, A, v, w);
        spmv(s, M, w, u);
        k_sub<<<grid_for(n), 256, 0, s>>>(n, v, u, w);
        sum_sq(s, w, n, part, sq + 1 + k);
        k_scale_by_norm<<<grid_for(n), 256, 0, s>>>(n, w, sq + 1 + k);
        std::swap(v, w);
    }
    std::vector<double> hs(iters + 1);
    cudaMemcpyAsync(hs.data(), sq, sizeof(double) * (iters + 1), cudaMemcpyDeviceToHost, s);
    e = cudaStreamSynchronize(s);
    dfree(v); dfree(w); dfree(u); dfree(part); dfree(sq);
    if (e != cudaSuccess) return cuda_fail(ctx, e, "power iteration");
    // Geometric mean of the last growth factors.
    const int tail = iters < 10 ? iters : 10;
    double lg = 0.0;
    for (int k = iters - tail; k < iters; ++k) lg += 0.5 * std::log(hs[1 + k]);
    *rho = std::exp(lg / tail);
    return MCLSGPU_OK;
}

}  // namespace

// LEARNED_SPAI preconditioner: M from the network on A's pattern, then the
// spectral-radius gate.  The learned M is kept unless rho(I - M A) reaches
// both `rho_fallback` and the point-Jacobi rho, in which case (or when the
// operator has no fixed stencil) point Jacobi is built instead and
// `fallback` is set.
int spai_build(mclsgpu_context* ctx, mclsgpu_operator* op, const mclsgpu_precond_params* p,
               mclsgpu_precond* pc) {
    mclsgpu_spai* net = static_cast<mclsgpu_spai*>(const_cast<void*>(p->spai_net));
    const double thresh = p->rho_fallback > 0.0 ? p->rho_fallback : 0.95;
    SlotTable t;
    int rc = MCLSGPU_OK;
    const bool usable = net && net->ctx == ctx && slot_table(ctx, op, net->slots, t) == MCLSGPU_OK;
    // Point Jacobi: the fallback and the gate's yardstick.
    DevCsr J;
    double* dinv = nullptr;
    cudaError_t e;
    if ((e = dmalloc(&dinv, op->A.n)) != cudaSuccess) return cuda_fail(ctx, e, "cudaMalloc");
    rc = reciprocal_diagonal(ctx, op->A, dinv);
    if (!rc) rc = point_jacobi_csr(ctx, op->A.n, dinv, J);
    if (rc) {
        dfree(dinv);
        J.release();
        return rc;
    }
    double rho_j = 1.0, rho_l = 1.0;
    bool keep = false;
    if (usable) {
        rc = csr_copy(ctx, op->A, pc->P);
        if (!rc) rc = launch_forward(net, op, t, pc->P.v, nullptr);
        if (!rc) {
            e = cudaStreamSynchronize(ctx->stream);
            if (e != cudaSuccess) rc = cuda_fail(ctx, e, "spai inference");
        }
        if (!rc) rc = check_device_status(ctx);
        if (!rc) rc = rho_estimate(ctx, op->A, pc->P, 200, 0x5eed5eedull, &rho_l);
        if (!rc) rc = rho_estimate(ctx, op->A, J, 200, 0x5eed5eedull, &rho_j);
        if (rc) {
            dfree(dinv);
            J.release();
            pc->P.release();
            return rc;
        }
        keep = std::isfinite(rho_l) && !(rho_l >= thresh && rho_l >= rho_j);
    }
    if (keep) {
        J.release();
        dfree(dinv);
        // M on A's diagonals too, for the fused MCSA iteration.
        rc = csr_to_dia(ctx, pc->P, op->dia_k, op->dia_off, &pc->mdia);
        if (rc) {
            pc->P.release();
            return rc;
        }
        pc->kind = MCLSGPU_PREC_LEARNED_SPAI;
        pc->rho = rho_l;
        pc->fallback = 0;
    } else {
        pc->P.release();
        pc->P = J;
        pc->diag = dinv;
        pc->kind = MCLSGPU_PREC_POINT_JACOBI;
        pc->rho = usable ? rho_l : -1.0;
        pc->fallback = 1;
    }
    return MCLSGPU_OK;
}

}  // namespace mclsgpu

using namespace mclsgpu;

extern "C" {

int mclsgpu_set_wait_limit(mclsgpu_context* ctx, int32_t polls) {
    if (!ctx) return MCLSGPU_ERR_INVALID_ARG;
    const int v = polls < 0 ? kDefaultWaitPolls : polls;
    cudaError_t e = cudaSetDevice(ctx->device);
    if (e == cudaSuccess)
        e = cudaMemcpyToSymbolAsync(g_wait_polls, &v, sizeof(int), 0, cudaMemcpyHostToDevice,
                                    ctx->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(ctx->stream);
    return e == cudaSuccess ? MCLSGPU_OK : cuda_fail(ctx, e, "set wait limit");
}

int mclsgpu_spai_num_params(void) { return kParams; }

int mclsgpu_spai_create(mclsgpu_context* ctx, int slots, uint64_t seed, mclsgpu_spai** out) {
    if (!ctx || !out) return MCLSGPU_ERR_INVALID_ARG;
    *out = nullptr;
    if (slots < 3 || slots > kMaxSlots)
        return set_error(ctx, MCLSGPU_ERR_INVALID_ARG, "spai: 3..%d stencil slots", kMaxSlots);
    mclsgpu_spai* net = new mclsgpu_spai;
    net->ctx = ctx;
    net->slots = slots;
    cudaError_t e;
    if ((e = dmalloc(&net->params, kParams)) != cudaSuccess ||
        (e = dmalloc(&net->grad, kParams)) != cudaSuccess ||
        (e = dmalloc(&net->m, kParams)) != cudaSuccess ||
        (e = dmalloc(&net->v, kParams)) != cudaSuccess) {
        dfree(net->params); dfree(net->grad); dfree(net->m); dfree(net->v);
        delete net;
        return cuda_fail(ctx, e, "cudaMalloc");
    }
    // He-uniform hidden layers, zero biases, zero output layer (= Jacobi).
    std::vector<float> h(kParams, 0.f);
    std::mt19937_64 gen(seed);
    std::uniform_real_distribution<float> U(-1.f, 1.f);
    const float a1 = std::sqrt(6.f / kF), a2 = std::sqrt(6.f / kH);
    for (int i = 0; i < kH * kF; ++i) h[kW1 + i] = a1 * U(gen);
    for (int i = 0; i < kH * kH; ++i) h[kW2 + i] = a2 * U(gen);
    cudaMemcpyAsync(net->params, h.data(), sizeof(float) * kParams, cudaMemcpyHostToDevice,
                    ctx->stream);
    cudaMemsetAsync(net->m, 0, sizeof(float) * kParams, ctx->stream);
    cudaMemsetAsync(net->v, 0, sizeof(float) * kParams, ctx->stream);
    cudaMemsetAsync(net->grad, 0, sizeof(float) * kParams, ctx->stream);
    e = cudaStreamSynchronize(ctx->stream);
    if (e != cudaSuccess) {
        dfree(net->params); dfree(net->grad); dfree(net->m); dfree(net->v);
        delete net;
        return cuda_fail(ctx, e, "spai create");
    }
    *out = net;
    return MCLSGPU_OK;
}

int mclsgpu_spai_destroy(mclsgpu_spai* net) {
    if (!net) return MCLSGPU_OK;
    dfree(net->params);
    dfree(net->grad);
    dfree(net->m);
    dfree(net->v);
    dfree(net->scratch);
    delete net;
    return MCLSGPU_OK;
}

int mclsgpu_spai_set_penalty(mclsgpu_spai* net, double weight, double threshold) {
    if (!net || !(weight >= 0.0) || !(threshold > 0.0)) return MCLSGPU_ERR_INVALID_ARG;
    net->pen_w = weight;
    net->pen_c = threshold;
    return MCLSGPU_OK;
}

int mclsgpu_spai_get_params(mclsgpu_spai* net, float* host) {
    if (!net || !host) return MCLSGPU_ERR_INVALID_ARG;
    cudaError_t e = cudaMemcpyAsync(host, net->params, sizeof(float) * kParams,
                                    cudaMemcpyDeviceToHost, net->ctx->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(net->ctx->stream);
    return e == cudaSuccess ? MCLSGPU_OK : cuda_fail(net->ctx, e, "spai get params");
}

int mclsgpu_spai_set_params(mclsgpu_spai* net, const float* host) {
    if (!net || !host) return MCLSGPU_ERR_INVALID_ARG;
    cudaError_t e = cudaMemcpyAsync(net->params, host, sizeof(float) * kParams,
                                    cudaMemcpyHostToDevice, net->ctx->stream);
    cudaMemsetAsync(net->m, 0, sizeof(float) * kParams, net->ctx->stream);
    cudaMemsetAsync(net->v, 0, sizeof(float) * kParams, net->ctx->stream);
    net->step = 0;
    if (e == cudaSuccess) e = cudaStreamSynchronize(net->ctx->stream);
    return e == cudaSuccess ? MCLSGPU_OK : cuda_fail(net->ctx, e, "spai set params");
}

int mclsgpu_spai_infer(mclsgpu_spai* net, mclsgpu_operator* op, float* out, double* mvals) {
    if (!net || !op || (!out && !mvals)) return MCLSGPU_ERR_INVALID_ARG;
    mclsgpu_context* ctx = net->ctx;
    SlotTable t;
    int rc = slot_table(ctx, op, net->slots, t);
    if (rc) return rc;
    const int n = op->A.n;
    float* dout = nullptr;
    double* dm = nullptr;
    cudaError_t e;
    if ((e = dmalloc(&dout, size_t(n) * kO)) != cudaSuccess ||
        (e = dmalloc(&dm, size_t(op->A.nnz))) != cudaSuccess) {
        dfree(dout);
        return cuda_fail(ctx, e, "cudaMalloc");
    }
    rc = launch_forward(net, op, t, dm, dout);
    if (!rc) {
        if (out)
            cudaMemcpyAsync(out, dout, sizeof(float) * n * kO, cudaMemcpyDeviceToHost, ctx->stream);
        if (mvals)
            cudaMemcpyAsync(mvals, dm, sizeof(double) * op->A.nnz, cudaMemcpyDeviceToHost,
                            ctx->stream);
        e = cudaStreamSynchronize(ctx->stream);
        if (e != cudaSuccess) rc = cuda_fail(ctx, e, "spai infer");
        if (!rc) rc = check_device_status(ctx);
    }
    dfree(dout);
    dfree(dm);
    return rc;
}

int mclsgpu_spai_infer_dev(mclsgpu_spai* net, mclsgpu_operator* op, float* out_dev,
                           double* mvals_dev, float* ms) {
    if (!net || !op || (!out_dev && !mvals_dev)) return MCLSGPU_ERR_INVALID_ARG;
    mclsgpu_context* ctx = net->ctx;
    SlotTable t;
    int rc = slot_table(ctx, op, net->slots, t);
    if (rc) return rc;
    cudaEvent_t e0 = nullptr, e1 = nullptr;
    if (ms) {
        cudaEventCreate(&e0);
        cudaEventCreate(&e1);
        cudaEventRecord(e0, ctx->stream);
    }
    rc = launch_forward(net, op, t, mvals_dev, out_dev);
    if (ms) cudaEventRecord(e1, ctx->stream);
    cudaError_t e = cudaStreamSynchronize(ctx->stream);
    if (!rc && e != cudaSuccess) rc = cuda_fail(ctx, e, "spai infer");
    if (ms) {
        *ms = 0.f;
        if (!rc) cudaEventElapsedTime(ms, e0, e1);
        cudaEventDestroy(e0);
        cudaEventDestroy(e1);
    }
    if (!rc) rc = check_device_status(ctx);
    return rc;
}

int mclsgpu_spai_gradient(mclsgpu_spai* net, mclsgpu_operator* op, const double* v_dev, int nvec,
                          double* loss, float* grad) {
    if (!net || !op || !v_dev) return MCLSGPU_ERR_INVALID_ARG;
    int rc = gradient(net, op, v_dev, nvec, loss);
    if (rc || !grad) return rc;
    cudaError_t e = cudaMemcpyAsync(grad, net->grad, sizeof(float) * kParams,
                                    cudaMemcpyDeviceToHost, net->ctx->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(net->ctx->stream);
    return e == cudaSuccess ? MCLSGPU_OK : cuda_fail(net->ctx, e, "spai gradient copy");
}

int mclsgpu_spai_train_step(mclsgpu_spai* net, mclsgpu_operator* op, const double* v_dev, int nvec,
                            const mclsgpu_spai_adam* opt, double* loss) {
    if (!net || !op || !v_dev || !opt) return MCLSGPU_ERR_INVALID_ARG;
    if (opt->size < sizeof(mclsgpu_spai_adam))
        return set_error(net->ctx, MCLSGPU_ERR_INVALID_ARG, "adam params: size mismatch");
    int rc = gradient(net, op, v_dev, nvec, loss);
    if (rc) return rc;
    ++net->step;
    const float c1 = 1.f - std::pow(float(opt->beta1), float(net->step));
    const float c2 = 1.f - std::pow(float(opt->beta2), float(net->step));
    k_adam<<<(kParams + 255) / 256, 256, 0, net->ctx->stream>>>(
        net->params, net->m, net->v, net->grad, kParams, float(opt->lr), float(opt->beta1),
        float(opt->beta2), float(opt->eps), c1, c2, float(opt->grad_clip));
    cudaError_t e = cudaStreamSynchronize(net->ctx->stream);
    return e == cudaSuccess ? MCLSGPU_OK : cuda_fail(net->ctx, e, "spai adam");
}

int mclsgpu_spai_smooth_vectors(mclsgpu_spai* net, mclsgpu_operator* op, double* v_dev, int nvec,
                                int iters) {
    if (!net || !op || !v_dev || nvec < 1 || iters < 0) return MCLSGPU_ERR_INVALID_ARG;
    mclsgpu_context* ctx = net->ctx;
    cudaStream_t s = ctx->stream;
    SlotTable t;
    int rc = slot_table(ctx, op, net->slots, t);
    if (rc) return rc;
    const int n = op->A.n;
    DevCsr M;
    double *w = nullptr, *u = nullptr, *part = nullptr, *sq = nullptr;
    cudaError_t e;
    if ((e = dmalloc(&w, n)) != cudaSuccess || (e = dmalloc(&u, n)) != cudaSuccess ||
        (e = dmalloc(&part, size_t(scan_partials_needed(n)))) != cudaSuccess ||
        (e = dmalloc(&sq, 1)) != cudaSuccess) {
        dfree(w); dfree(u); dfree(part); dfree(sq);
        return cuda_fail(ctx, e, "cudaMalloc");
    }
    rc = csr_copy(ctx, op->A, M);
    if (!rc) rc = launch_forward(net, op, t, M.v, nullptr);
    if (!rc) {
        for (int k = 0; k < nvec; ++k) {
            double* v = v_dev + size_t(k) * n;
            for (int it = 0; it < iters; ++it) {
                spmv(s, op->A, v, w);
                spmv(s, M, w, u);
                k_sub<<<grid_for(n), 256, 0, s>>>(n, v, u, v);
                sum_sq(s, v, n, part, sq);
                k_scale_by_norm<<<grid_for(n), 256, 0, s>>>(n, v, sq);
            }
        }
        e = cudaStreamSynchronize(s);
        if (e != cudaSuccess) rc = cuda_fail(ctx, e, "spai smooth vectors");
    }
    M.release();
    dfree(w); dfree(u); dfree(part); dfree(sq);
    return rc;
}

int mclsgpu_spai_rho(mclsgpu_spai* net, mclsgpu_operator* op, int iters, double* rho_learned,
                     double* rho_jacobi) {
    if (!net || !op) return MCLSGPU_ERR_INVALID_ARG;
    mclsgpu_context* ctx = net->ctx;
    SlotTable t;
    int rc = slot_table(ctx, op, net->slots, t);
    if (rc) return rc;
    DevCsr M, J;
    double* dinv = nullptr;
    cudaError_t e = dmalloc(&dinv, op->A.n);
    if (e != cudaSuccess) return cuda_fail(ctx, e, "cudaMalloc");
    rc = csr_copy(ctx, op->A, M);
    if (!rc) rc = launch_forward(net, op, t, M.v, nullptr);
    if (!rc && rho_learned) rc = rho_estimate(ctx, op->A, M, iters, 0x5eed5eedull, rho_learned);
    if (!rc && rho_jacobi) {
        rc = reciprocal_diagonal(ctx, op->A, dinv);
        if (!rc) rc = point_jacobi_csr(ctx, op->A.n, dinv, J);
        if (!rc) rc = rho_estimate(ctx, op->A, J, iters, 0x5eed5eedull, rho_jacobi);
    }
    M.release();
    J.release();
    dfree(dinv);
    return rc;
}

}  // extern "C"

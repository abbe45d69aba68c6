// scan.cuh -- block scan and tile geometry of the scan and source kernels:
// tiles of 2048 elements, 8 consecutive ones per thread, staged through shared
// memory.  The association order is fixed, so results are reproducible run to
// run.
#pragma once

namespace mclsgpu {
namespace scan {

constexpr int kThreads = 256;
constexpr int kItems = 8;
constexpr int kTile = kThreads * kItems;
constexpr unsigned kFull = 0xffffffffu;

struct AddOp {
    template <class T>
    __device__ __forceinline__ T operator()(T a, T b) const { return a + b; }
};

// Place of element e of a tile of 8-byte (Swz<8>) or 4-byte elements in shared
// memory: 8 consecutive elements per thread, read one by one, would hit the
// same banks from 16 (8) lanes; permuted within groups of 16 (8) elements each
// access takes the fewest wavefronts, and consecutive elements still do.
template <int BYTES>
__device__ __forceinline__ int swz(int e) {
    return BYTES == 8 ? e ^ ((e >> 4) & 15) : e ^ ((e >> 5) & 7);
}

// Two sums scanned together.
struct Pair {
    double a, b;
    __device__ __forceinline__ Pair operator+(const Pair& o) const { return {a + o.a, b + o.b}; }
};
template <class T>
__device__ __forceinline__ T shfl_up(T v, int d) {
    return __shfl_up_sync(kFull, v, d);
}
__device__ __forceinline__ Pair shfl_up(Pair v, int d) {
    return {__shfl_up_sync(kFull, v.a, d), __shfl_up_sync(kFull, v.b, d)};
}

// Inclusive block scan of one value per thread (256 threads).  On return
// *excl holds the exclusive value of this thread.
template <class T, class Op>
__device__ __forceinline__ T block_scan(T v, Op op, T identity, T* warp_tot, T* excl) {
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        T o = shfl_up(v, d);
        if (lane >= d) v = op(o, v);
    }
    if (lane == 31) warp_tot[wid] = v;
    __syncthreads();
    if (wid == 0) {
        T t = lane < kThreads / 32 ? warp_tot[lane] : identity;
#pragma unroll
        for (int d = 1; d < 8; d <<= 1) {
            T o = shfl_up(t, d);
            if (lane >= d) t = op(o, t);
        }
        if (lane < kThreads / 32) warp_tot[lane] = t;
    }
    __syncthreads();
    if (wid > 0) v = op(warp_tot[wid - 1], v);
    T prev = shfl_up(v, 1);
    if (lane == 0) prev = wid > 0 ? warp_tot[wid - 1] : identity;
    *excl = prev;
    __syncthreads();
    return v;
}

inline int tiles(int n) { return (n + kTile - 1) / kTile; }

}  // namespace scan
}  // namespace mclsgpu

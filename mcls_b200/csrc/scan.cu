// scan.cu -- deterministic reductions (tiles staged through shared memory, a
// single-block scan of the tile partials) and the reference's left-to-right
// source sums.
#include "internal.h"
#include "scan.cuh"

namespace mclsgpu {
namespace {

using namespace scan;

// Loaders ---------------------------------------------------------------------
struct CdfLoad {  // source CDF input: signed first element, |.| after
    const double* v;
    double scale;
    int has_scale;
    __device__ __forceinline__ double operator()(int i) const {
        double x = has_scale ? v[i] * scale : v[i];
        return i == 0 ? x : fabs(x);
    }
};
struct AbsLoad {
    const double* v;
    double scale;
    int has_scale;
    __device__ __forceinline__ double operator()(int i) const {
        double x = has_scale ? v[i] * scale : v[i];
        return fabs(x);
    }
};
struct SqLoad {
    const double* v;
    __device__ __forceinline__ double operator()(int i) const { return v[i] * v[i]; }
};
template <class T, class Load>
__device__ __forceinline__ void stage_tile(Load ld, int n, T identity, T* stage) {
    const int base = blockIdx.x * kTile;
    for (int k = threadIdx.x; k < kTile; k += kThreads) {
        int i = base + k;
        stage[k] = i < n ? ld(i) : identity;
    }
    __syncthreads();
}

template <class T, class Op, class Load>
__global__ void __launch_bounds__(kThreads) tile_reduce(Load ld, int n, Op op, T identity,
                                                        T* part) {
    __shared__ T stage[kTile];
    __shared__ T warp_tot[32];
    stage_tile(ld, n, identity, stage);
    T acc = stage[threadIdx.x * kItems];
#pragma unroll
    for (int k = 1; k < kItems; ++k) acc = op(acc, stage[threadIdx.x * kItems + k]);
    T excl;
    T incl = block_scan(acc, op, identity, warp_tot, &excl);
    if (threadIdx.x == kThreads - 1) part[blockIdx.x] = incl;
}

// Exclusive scan of the tile partials in one block; part[nb] = total.
template <class T, class Op>
__global__ void __launch_bounds__(kThreads) partial_scan(T* part, int nb, Op op, T identity) {
    __shared__ T warp_tot[32];
    __shared__ T carry_s;
    if (threadIdx.x == 0) carry_s = identity;
    __syncthreads();
    for (int base = 0; base < nb; base += kThreads) {
        int i = base + threadIdx.x;
        T v = i < nb ? part[i] : identity;
        T excl;
        T incl = block_scan(v, op, identity, warp_tot, &excl);
        T carry = carry_s;
        if (i < nb) part[i] = op(carry, excl);
        __syncthreads();
        if (threadIdx.x == kThreads - 1) carry_s = op(carry, incl);
        __syncthreads();
    }
    if (threadIdx.x == 0) part[nb] = carry_s;
}

__global__ void seq_source_cdf(CdfLoad ld, int n, double* cdf, double* total) {
    // buildRandomSource left-to-right order (src/MCLS_UniformAdjointSource_impl.hpp:184-204)
    double c = ld(0);
    cdf[0] = c;
    for (int i = 1; i < n; ++i) {
        c = c + ld(i);
        cdf[i] = c;
    }
    const double back = c;
    for (int i = 0; i < n; ++i) cdf[i] = cdf[i] / back;
    *total = back;
}

__global__ void seq_abs_sum(AbsLoad ld, int n, double* out) {
    double s = 0.0;
    for (int i = 0; i < n; ++i) s = s + ld(i);
    *out = s;
}

template <class T>
__global__ void copy_total(const T* part, int nb, T* out) {
    *out = part[nb];
}

}  // namespace

int scan_partials_needed(int n) { return tiles(n) + 2; }

void source_sequential(cudaStream_t s, const double* v, int n, double scale, int has_scale,
                       double* norm1, double* cdf, double* total) {
    seq_abs_sum<<<1, 1, 0, s>>>(AbsLoad{v, scale, has_scale}, n, norm1);
    seq_source_cdf<<<1, 1, 0, s>>>(CdfLoad{v, scale, has_scale}, n, cdf, total);
}

void abs_sum_sequential(cudaStream_t s, const double* v, int n, double scale, int has_scale,
                        double* norm1) {
    seq_abs_sum<<<1, 1, 0, s>>>(AbsLoad{v, scale, has_scale}, n, norm1);
}

void sum_sq(cudaStream_t s, const double* v, int n, double* part, double* out) {
    SqLoad ld{v};
    int nb = tiles(n);
    tile_reduce<double><<<nb, kThreads, 0, s>>>(ld, n, AddOp(), 0.0, part);
    partial_scan<double><<<1, kThreads, 0, s>>>(part, nb, AddOp(), 0.0);
    copy_total<double><<<1, 1, 0, s>>>(part, nb, out);
}

}  // namespace mclsgpu

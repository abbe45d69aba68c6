// ops.cuh -- the operator layouts that the residual passes read, and the launch
// of a kernel on an operator's fastest one.
#pragma once
#include "internal.h"

namespace mclsgpu {

// Row dot products A(r,:) . f(col) over the two operator layouts.  Both visit
// a row's entries in ascending column order with FMA accumulation, and their
// padding entries contribute a product with 0 (which adds exactly nothing),
// so both return the CSR sum bit for bit.
struct SellView {  // SELL-32
    // A row's entries are loaded kBatch at a time, then the vector at their
    // columns: with one row per thread and few warps per SM the round trips
    // must overlap (entry by entry 13.5 us for the residual of 10^5 rows of an
    // unstructured operator, 11.5 us so).  The registers cost resident blocks.
    static constexpr int kMinBlocks = 4;
    static constexpr int kBatch = 8;
    const int* off;
    const int* col;
    const double* val;
    int n;
    template <class F>
    __device__ __forceinline__ double dot(int r, F f) const {
        const int a = off[r >> 5];
        const int o = a + (r & 31), w = (off[(r >> 5) + 1] - a) >> 5;
        double s = 0.0;
        for (int k0 = 0; k0 < w; k0 += kBatch) {
            int c[kBatch];
            double v[kBatch];
#pragma unroll
            for (int q = 0; q < kBatch; ++q) {
                // Past the slice's width: its last column again, not added.
                const int k = k0 + q < w ? k0 + q : w - 1;
                c[q] = col[o + 32 * k];
                v[q] = val[o + 32 * k];
            }
            double x[kBatch];
#pragma unroll
            for (int q = 0; q < kBatch; ++q) x[q] = f(c[q]);
#pragma unroll
            for (int q = 0; q < kBatch; ++q)
                if (k0 + q < w) s = fma(v[q], x[q], s);
        }
        return s;
    }
};

// Stencil operator stored by diagonal offset (no indices).  KK > 0 fixes the
// number of offsets at compile time so the row loop unrolls and every load of
// the row is issued before the first product.
template <int KK>
struct DiaViewT {
    static constexpr int kMinBlocks = 8;
    static constexpr int kDiags = KK > 0 ? KK : 16;  // at most
    const double* val;
    int n;
    int k;
    int off[16];
    __device__ __forceinline__ int diags() const { return KK > 0 ? KK : k; }
    __device__ __forceinline__ int offset(int j) const { return off[j]; }
    template <class F>
    __device__ __forceinline__ double dot(int r, F f) const {
        constexpr int kmax = KK > 0 ? KK : 16;
        const int kk = KK > 0 ? KK : k;
        double s = 0.0;
#pragma unroll
        for (int j = 0; j < kmax; ++j) {
            if (j >= kk) break;
            const int c = r + off[j];
            if (unsigned(c) < unsigned(n)) s = fma(val[size_t(j) * n + r], f(c), s);
        }
        return s;
    }
};
using DiaView = DiaViewT<0>;

// Symmetric stencil operator (A(r, r - o) == A(r - o, r)): only the diagonal
// and the H positive-offset diagonals are read; A(r, r - o_h) is taken as
// A(r - o_h, r).  The products are the same as DiaViewT's, in the same
// (ascending column) order, so the sums are bit for bit the same with
// (1 + H) / (1 + 2H) of the matrix bytes.
template <int H>
struct DiaSymView {
    static constexpr int kMinBlocks = 8;
    static constexpr int kDiags = 2 * H + 1;
    const double* val;  // [(1 + H) * n]: diagonal, then positive offsets ascending
    int n;
    int off[H];
    __device__ __forceinline__ int diags() const { return kDiags; }
    // Diagonal j in ascending order.
    __device__ __forceinline__ int offset(int j) const {
        return j < H ? -off[H - 1 - j] : j == H ? 0 : off[j - H - 1];
    }
    template <class F>
    __device__ __forceinline__ double dot(int r, F f) const {
        double s = 0.0;
#pragma unroll
        for (int h = H - 1; h >= 0; --h) {
            const int c = r - off[h];
            if (c >= 0) s = fma(val[size_t(1 + h) * n + c], f(c), s);
        }
        s = fma(val[r], f(r), s);
#pragma unroll
        for (int h = 0; h < H; ++h) {
            const int c = r + off[h];
            if (c < n) s = fma(val[size_t(1 + h) * n + r], f(c), s);
        }
        return s;
    }
};

// Row r of another matrix on A's diagonals (values vals) times f: the sum that
// DiaViewT's dot gives for it.
template <class Op, class F>
__device__ __forceinline__ double dot_on_diagonals(const Op& A, const double* vals, int r, F f) {
    double s = 0.0;
#pragma unroll
    for (int j = 0; j < Op::kDiags; ++j) {
        if (j >= A.diags()) break;
        const int c = r + A.offset(j);
        if (unsigned(c) < unsigned(A.n)) s = fma(vals[size_t(j) * A.n + r], f(c), s);
    }
    return s;
}

inline SellView sell_view(const mclsgpu_operator* op) {
    return SellView{op->S.off, op->S.col, op->S.val, op->S.n};
}

template <int H>
inline DiaSymView<H> sym_view(const mclsgpu_operator* op) {
    DiaSymView<H> v{};
    v.val = op->sym_val;
    v.n = op->A.n;
    for (int h = 0; h < H; ++h) v.off[h] = op->sym_off[h];
    return v;
}

template <int KK>
inline DiaViewT<KK> dia_view(const mclsgpu_operator* op) {
    DiaViewT<KK> v{};
    v.val = op->dia_val;
    v.n = op->A.n;
    v.k = op->dia_k;
    for (int j = 0; j < 16; ++j) v.off[j] = op->dia_off[j];
    return v;
}

// The diagonal-offset view of another matrix on the operator's offsets.
template <int KK>
inline DiaViewT<KK> dia_view_vals(const mclsgpu_operator* op, const double* vals) {
    DiaViewT<KK> v = dia_view<KK>(op);
    v.val = vals;
    return v;
}

#define MCLSGPU_LAUNCH_M(op, vals, grid, threads, stream, kern, ...)                         \
    do {                                                                                     \
        switch ((op)->dia_k) {                                                               \
            case 5:                                                                          \
                kern<DiaViewT<5>><<<grid, threads, 0, stream>>>(dia_view_vals<5>(op, vals),  \
                                                                __VA_ARGS__);                \
                break;                                                                       \
            case 7:                                                                          \
                kern<DiaViewT<7>><<<grid, threads, 0, stream>>>(dia_view_vals<7>(op, vals),  \
                                                                __VA_ARGS__);                \
                break;                                                                       \
            case 9:                                                                          \
                kern<DiaViewT<9>><<<grid, threads, 0, stream>>>(dia_view_vals<9>(op, vals),  \
                                                                __VA_ARGS__);                \
                break;                                                                       \
            default:                                                                         \
                kern<DiaView><<<grid, threads, 0, stream>>>(dia_view_vals<0>(op, vals),      \
                                                            __VA_ARGS__);                    \
        }                                                                                    \
    } while (0)

// Launch `kern<Op>` on a stencil operator's fastest layout (dia_k > 0):
// diagonal-offset values, unrolled for the 5-, 7- and 9-point stencils; only the
// diagonal and upper diagonals when the values are symmetric.
#define MCLSGPU_LAUNCH_DIA(op, grid, threads, stream, kern, ...)                             \
    do {                                                                                     \
        switch ((op)->dia_k) {                                                               \
            case 5:                                                                          \
                if ((op)->sym_h == 2)                                                        \
                    kern<DiaSymView<2>><<<grid, threads, 0, stream>>>(sym_view<2>(op),       \
                                                                      __VA_ARGS__);          \
                else                                                                         \
                    kern<DiaViewT<5>><<<grid, threads, 0, stream>>>(dia_view<5>(op),         \
                                                                    __VA_ARGS__);            \
                break;                                                                       \
            case 7:                                                                          \
                if ((op)->sym_h == 3)                                                        \
                    kern<DiaSymView<3>><<<grid, threads, 0, stream>>>(sym_view<3>(op),       \
                                                                      __VA_ARGS__);          \
                else                                                                         \
                    kern<DiaViewT<7>><<<grid, threads, 0, stream>>>(dia_view<7>(op),         \
                                                                    __VA_ARGS__);            \
                break;                                                                       \
            case 9:                                                                          \
                if ((op)->sym_h == 4)                                                        \
                    kern<DiaSymView<4>><<<grid, threads, 0, stream>>>(sym_view<4>(op),       \
                                                                      __VA_ARGS__);          \
                else                                                                         \
                    kern<DiaViewT<9>><<<grid, threads, 0, stream>>>(dia_view<9>(op),         \
                                                                    __VA_ARGS__);            \
                break;                                                                       \
            default:                                                                         \
                kern<DiaView><<<grid, threads, 0, stream>>>(dia_view<0>(op), __VA_ARGS__);   \
        }                                                                                    \
    } while (0)

// The same, or on SELL-32 where the operator is no stencil.
#define MCLSGPU_LAUNCH_OP(op, grid, threads, stream, kern, ...)                              \
    do {                                                                                     \
        if ((op)->dia_k == 0)                                                                \
            kern<SellView><<<grid, threads, 0, stream>>>(sell_view(op), __VA_ARGS__);        \
        else                                                                                 \
            MCLSGPU_LAUNCH_DIA(op, grid, threads, stream, kern, __VA_ARGS__);                \
    } while (0)

}  // namespace mclsgpu

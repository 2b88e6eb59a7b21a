// SpMV with several right-hand sides in 16-byte aligned row-major blocks:
// the column-slice kernel shared by the SpMV entry points and the solvers.
#pragma once

#include <type_traits>

#include "common.cuh"

namespace b2s {

constexpr int kLanesBlock = 256;

// ---------------------------------------------------------------------------
// Four or more right-hand sides: KL = K / VW lanes share one row and each
// owns VW consecutive columns (one 16-byte vector), so the lanes of a row
// read one contiguous stretch of b(col, :) and write one of c(row, :); the
// row's values and column indices are broadcast loads.  Used for Csr, Ell
// and Sellp; needs 16-byte aligned b/c rows.
// ---------------------------------------------------------------------------
template <typename T>
struct Vec16;
template <>
struct Vec16<double> {
    using type = double2;
    static constexpr int width = 2;
};
template <>
struct Vec16<float> {
    using type = float4;
    static constexpr int width = 4;
};

template <typename T>
__device__ __forceinline__ void fma_vec(typename Vec16<T>::type& acc, T a,
                                        const T* p)
{
    const auto x = __ldg(reinterpret_cast<const typename Vec16<T>::type*>(p));
    if constexpr (Vec16<T>::width == 2) {
        acc.x += a * x.x;
        acc.y += a * x.y;
    } else {
        acc.x += a * x.x;
        acc.y += a * x.y;
        acc.z += a * x.z;
        acc.w += a * x.w;
    }
}

template <typename T>
__device__ __forceinline__ void store_vec(T* dst, const typename Vec16<T>::type& acc,
                                          const T* alpha, const T* beta)
{
    constexpr int W = Vec16<T>::width;
    const T* a = reinterpret_cast<const T*>(&acc);
    T out[W];
#pragma unroll
    for (int u = 0; u < W; ++u) out[u] = combine(a[u], alpha, beta, dst + u);
    *reinterpret_cast<typename Vec16<T>::type*>(dst) =
        *reinterpret_cast<const typename Vec16<T>::type*>(out);
}

// FMT 0: Csr, 1: Ell, 2: Sellp.  skip: when non-null and set, the whole
// grid returns (a solver whose columns have all stopped).
template <typename T, int K, int FMT>
__global__ void __launch_bounds__(kLanesBlock)
    rhs_lanes_kernel(int64_t n, const int32_t* __restrict__ rp,
                     int64_t width_or_slice, int64_t stride,
                     const uint64_t* __restrict__ slice_sets,
                     const uint64_t* __restrict__ slice_lengths,
                     const int32_t* __restrict__ ci, const T* __restrict__ v,
                     const T* __restrict__ b, int64_t ldb, T* __restrict__ c,
                     int64_t ldc, const T* __restrict__ alpha,
                     const T* __restrict__ beta, const int* __restrict__ skip = nullptr)
{
    if (skip != nullptr && *skip) return;
    using V = typename Vec16<T>::type;
    constexpr int VW = Vec16<T>::width;
    constexpr int KL = K / VW;
    const int64_t g = blockIdx.x * int64_t(kLanesBlock) + threadIdx.x;
    const int64_t row = g / KL;
    if (row >= n) return;
    const int sub = int(g % KL);
    const T* bc = b + sub * VW;
    V acc;
    {
        T* a = reinterpret_cast<T*>(&acc);
#pragma unroll
        for (int u = 0; u < VW; ++u) a[u] = T(0);
    }
    int64_t first, step, len;
    if constexpr (FMT == 0) {
        first = rp[row];
        len = rp[row + 1] - first;
        step = 1;
    } else if constexpr (FMT == 1) {
        first = row;
        len = width_or_slice;
        step = stride;
    } else {
        const int64_t s = row / width_or_slice;
        first = int64_t(slice_sets[s]) * width_or_slice + (row - s * width_or_slice);
        len = int64_t(slice_lengths[s]);
        step = width_or_slice;
    }
    int64_t i = 0;
    for (; i + 4 <= len; i += 4) {
        int32_t col[4];
        T val[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            col[u] = __ldg(ci + first + (i + u) * step);
            val[u] = __ldg(v + first + (i + u) * step);
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            if (FMT == 0 || col[u] != -1) fma_vec<T>(acc, val[u], bc + int64_t(col[u]) * ldb);
        }
    }
    for (; i < len; ++i) {
        const int32_t col = __ldg(ci + first + i * step);
        const T val = __ldg(v + first + i * step);
        if (FMT == 0 || col != -1) fma_vec<T>(acc, val, bc + int64_t(col) * ldb);
    }
    store_vec<T>(c + row * ldc + sub * VW, acc, alpha, beta);
}

// The same products with a warp per ROWS consecutive rows (4 to 32).  The
// warp loads the column indices and values of E = 32 / ROWS entries of every
// row at once, lane e * ROWS + r taking entry e of row r, one load step
// ahead of their use; the rows then pass in S = ROWS / (32 / KL) steps, the
// index and value handed to the row's KL = K / VW lanes by shuffles, so that
// the S * E = KL gathers of b (512 bytes each) of a load step are in flight
// together.  rhs_lanes_kernel has the gathers of four entries in flight and
// loads every index and value KL times, one sector for 8 or 16 useful bytes
// in the column-major formats.
template <typename T, int K, int FMT, int ROWS, typename Store>
__device__ __forceinline__ void rhs_rows(int64_t n, int64_t r0, const int32_t* __restrict__ rp,
                                         int64_t width_or_slice, int64_t stride,
                                         const uint64_t* __restrict__ slice_sets,
                                         const uint64_t* __restrict__ slice_lengths,
                                         const int32_t* __restrict__ ci,
                                         const T* __restrict__ v, const T* __restrict__ b,
                                         int64_t ldb, Store&& store)
{
    using V = typename Vec16<T>::type;
    constexpr int VW = Vec16<T>::width;
    constexpr int KL = K / VW;           // lanes per row
    constexpr int RPW = kWarp / KL;      // rows per step
    constexpr int S = ROWS / RPW;        // steps
    constexpr int E = kWarp / ROWS;      // entries per load
    static_assert(S >= 1 && S * RPW == ROWS && E * ROWS == kWarp, "whole steps and loads");
    constexpr unsigned kFull = 0xffffffffu;
    const int lane = threadIdx.x % kWarp;
    const int64_t row = r0 + lane % ROWS;
    int64_t first = 0, step = 1;
    int len = 0;
    if (row < n) {
        if constexpr (FMT == 0) {
            first = rp[row];
            len = int(rp[row + 1] - first);
        } else if constexpr (FMT == 1) {
            first = row;
            len = int(width_or_slice);
            step = stride;
        } else {
            const int64_t s = row / width_or_slice;
            first = int64_t(slice_sets[s]) * width_or_slice + (row - s * width_or_slice);
            len = int(slice_lengths[s]);
            step = width_or_slice;
        }
    }
    const int wlen = __reduce_max_sync(kFull, len);
    const T* bc = b + (lane % KL) * VW;
    V acc[S];
#pragma unroll
    for (int s = 0; s < S; ++s) {
        T* a = reinterpret_cast<T*>(&acc[s]);
#pragma unroll
        for (int u = 0; u < VW; ++u) a[u] = T(0);
    }
    const int e0 = lane / ROWS;
    const int32_t* pc = ci + first + e0 * step;
    const T* pv = v + first + e0 * step;
    int32_t col = e0 < len ? __ldg(pc) : -1;
    T val = e0 < len ? __ldg(pv) : T(0);
    for (int i = 0; i < wlen; i += E) {
        int32_t ncol = -1;
        T nval = T(0);
        if (i + E + e0 < len) {
            pc += E * step;
            pv += E * step;
            ncol = __ldg(pc);
            nval = __ldg(pv);
        }
        V x[KL];
        T a[KL];
#pragma unroll
        for (int g = 0; g < KL; ++g) {
            const int src = (g / S) * ROWS + (g % S) * RPW + lane / KL;
            const int32_t cc = KL == 1 ? col : __shfl_sync(kFull, col, src);
            const T vv = KL == 1 ? val : __shfl_sync(kFull, val, src);
            T* z = reinterpret_cast<T*>(&x[g]);
#pragma unroll
            for (int u = 0; u < VW; ++u) z[u] = T(0);
            a[g] = T(0);
            if (cc != -1) {  // padding adds nothing, whatever its value
                a[g] = vv;
                x[g] = __ldg(reinterpret_cast<const V*>(bc + int64_t(cc) * ldb));
            }
        }
#pragma unroll
        for (int g = 0; g < KL; ++g) {
            T* q = reinterpret_cast<T*>(&acc[g % S]);
            const T* z = reinterpret_cast<const T*>(&x[g]);
#pragma unroll
            for (int u = 0; u < VW; ++u) q[u] += a[g] * z[u];
        }
        col = ncol;
        val = nval;
    }
#pragma unroll
    for (int s = 0; s < S; ++s) {
        const int64_t orow = r0 + s * RPW + lane / KL;
        if (orow < n) store(orow, (lane % KL) * VW, acc[s]);
    }
}

template <typename T, int K, int FMT, int ROWS>
__global__ void __launch_bounds__(kLanesBlock)
    rhs_rows_kernel(int64_t n, const int32_t* __restrict__ rp, int64_t width_or_slice,
                    int64_t stride, const uint64_t* __restrict__ slice_sets,
                    const uint64_t* __restrict__ slice_lengths, const int32_t* __restrict__ ci,
                    const T* __restrict__ v, const T* __restrict__ b, int64_t ldb,
                    T* __restrict__ c, int64_t ldc, const T* __restrict__ alpha,
                    const T* __restrict__ beta, const int* __restrict__ skip = nullptr)
{
    if (skip != nullptr && *skip) return;
    const int64_t r0 =
        (blockIdx.x * int64_t(kLanesBlock / kWarp) + threadIdx.x / kWarp) * ROWS;
    if (r0 >= n) return;  // whole warp
    rhs_rows<T, K, FMT, ROWS>(n, r0, rp, width_or_slice, stride, slice_sets, slice_lengths, ci,
                              v, b, ldb,
                              [&](int64_t row, int col0, const typename Vec16<T>::type& acc) {
                                  store_vec<T>(c + row * ldc + col0, acc, alpha, beta);
                              });
}

// Rows a warp of rhs_rows_kernel takes, 0 where rhs_lanes_kernel stays.
// `longest`: the longest row (Csr, Ell) or slice (Sellp), 0 when not known.
//
// Rows differ in length inside a warp in Csr and Sellp, and a warp runs to
// its longest: matrices with rows over 64 entries keep rhs_lanes_kernel (one
// long row holds up the other rows of its warp; the power-law matrix's
// longest slices have 1,805 entries).  Few rows: the fewest rows per warp,
// for the most warps (3d 27-point 24^3, 16 FP64 columns, Sellp: 6.9 us with
// 4 rows, 15.7 with 32).  Many short rows (up to 8 entries, two load steps
// at most): 32 rows, the longest coalesced loads and stores, except at 16
// FP64 columns, whose 8 accumulators of 32 rows need 102 registers (267
// against 231 us with 16 rows, 7-point 128^3).  Longer rows: 16 per warp, so
// that each load step brings two entries per row (27-point 77^3, 4 FP64
// columns, Sellp: 55.1 against 65.0 us with 32 rows).
// 7-point 128^3, 4 / 8 / 16 columns, before -> after: Sellp FP64 141 / 263 /
// 476 -> 89 / 115 / 231 us, FP32 68 / 133 / 248 -> 47 / 69 / 110 us; Ell FP64
// 90 / 168 / 318 -> 78 / 128 / 209 us.  Csr's entries of a row already sit
// together and its reloads hit L1, so there the kernel pays only from four
// lanes per row on short rows (FP64 117 -> 96 us at 8 columns, 224 -> 204 at
// 16; FP32 105 -> 85 at 16; at 4 FP64 columns 66 against 69) and on few rows
// longer than 8 (27-point 24^3, 8 FP64 columns: 7.9 -> 5.5 us).
constexpr int64_t kRowsMaxLen = 64;
constexpr int64_t kRowsFew = int64_t(1) << 14;
constexpr int64_t kRowsShort = 8;

inline int rhs_rows_per_warp(int fmt, int lanes, int64_t n, int64_t longest)
{
    // (Ell's rows are all as long as its width)
    if (longest <= 0 || longest > (fmt == 1 ? int64_t(1) << 30 : kRowsMaxLen)) return 0;
    const int fewest = kWarp / lanes;
    const bool few = n < kRowsFew, short_rows = longest <= kRowsShort;
    if (fmt == 0 && !(few ? !short_rows : short_rows && lanes >= 4)) return 0;
    if (few) return fewest;
    const int rows = short_rows && lanes < 8 ? 32 : 16;
    return rows > fewest ? rows : fewest;
}

// Calls f(std::integral_constant<int, ROWS>) for a value of
// rhs_rows_per_warp.
template <int KL, typename F>
void with_rows_per_warp(int rows, F&& f)
{
    constexpr int kFewest = kWarp / KL;
    if (rows == kFewest) {
        f(std::integral_constant<int, kFewest>());
    } else if (rows == 32) {
        if constexpr (KL > 1 && KL < 8) f(std::integral_constant<int, 32>());
    } else {
        if constexpr (KL > 2) f(std::integral_constant<int, 16>());
    }
}

// Products of K columns (K >= 4 and a multiple of the 16-byte vector width;
// b and c rows 16-byte aligned) with the kernel that the sizes call for.
template <typename T, int K, int FMT>
void launch_rhs_lanes(int64_t n, const int32_t* rp, int64_t w_or_s, int64_t stride,
                      const uint64_t* sets, const uint64_t* lens, const int32_t* ci, const T* v,
                      const T* b, int64_t ldb, T* c, int64_t ldc, const T* alpha, const T* beta,
                      int64_t longest, cudaStream_t st, const int* skip = nullptr)
{
    static_assert(K >= 4 && K % Vec16<T>::width == 0, "column slices of 16 bytes");
    constexpr int KL = K / Vec16<T>::width;
    const int rows = rhs_rows_per_warp(FMT, KL, n, longest);
    if (rows > 0) {
        with_rows_per_warp<KL>(rows, [&](auto rc) {
            constexpr int ROWS = decltype(rc)::value;
            const int64_t grid = ceildiv(ceildiv(n, ROWS), kLanesBlock / kWarp);
            rhs_rows_kernel<T, K, FMT, ROWS><<<grid, kLanesBlock, 0, st>>>(
                n, rp, w_or_s, stride, sets, lens, ci, v, b, ldb, c, ldc, alpha, beta, skip);
        });
        return;
    }
    rhs_lanes_kernel<T, K, FMT><<<ceildiv(n * KL, kLanesBlock), kLanesBlock, 0, st>>>(
        n, rp, w_or_s, stride, sets, lens, ci, v, b, ldb, c, ldc, alpha, beta, skip);
}

}  // namespace b2s

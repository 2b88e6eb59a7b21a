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
                    const T* __restrict__ beta)
{
    const int64_t r0 =
        (blockIdx.x * int64_t(kLanesBlock / kWarp) + threadIdx.x / kWarp) * ROWS;
    if (r0 >= n) return;  // whole warp
    rhs_rows<T, K, FMT, ROWS>(n, r0, rp, width_or_slice, stride, slice_sets, slice_lengths, ci,
                              v, b, ldb,
                              [&](int64_t row, int col0, const typename Vec16<T>::type& acc) {
                                  store_vec<T>(c + row * ldc + col0, acc, alpha, beta);
                              });
}

// Ell with two neighbouring rows per lane slot: the rows' column indices and
// values at each entry are one 8- or 16-byte vector load (the layout is
// column-major, so rows r and r + 1 sit next to each other), and each slot
// gathers two 16-byte pieces of b per entry, eight in flight.  Needs an even
// stride, vector-aligned indices and values and 16-byte aligned b and c rows;
// a pair whose second row lies past the matrix computes the first alone.
template <typename T, int K>
__global__ void __launch_bounds__(kLanesBlock)
    rhs_pairs_kernel(int64_t n, int64_t width, int64_t stride, const int32_t* __restrict__ ci,
                     const T* __restrict__ v, const T* __restrict__ b, int64_t ldb,
                     T* __restrict__ c, int64_t ldc, const T* __restrict__ alpha,
                     const T* __restrict__ beta)
{
    using V = typename Vec16<T>::type;
    using V2 = typename std::conditional<sizeof(T) == 8, double2, float2>::type;
    constexpr int VW = Vec16<T>::width;
    constexpr int KL = K / VW;
    const int64_t g = blockIdx.x * int64_t(kLanesBlock) + threadIdx.x;
    const int64_t r0 = 2 * (g / KL);
    if (r0 >= n) return;
    const int sub = int(g % KL);
    const T* bc = b + sub * VW;
    V acc0, acc1;
    {
        T* a0 = reinterpret_cast<T*>(&acc0);
        T* a1 = reinterpret_cast<T*>(&acc1);
#pragma unroll
        for (int u = 0; u < VW; ++u) a0[u] = a1[u] = T(0);
    }
    const int64_t first = r0, len = width, step = stride;
    // always so with an even stride; without the test the compiler issues the
    // gathers one by one (34 registers in place of 62; 27-point 32^3, 16 FP32
    // columns: 13.1 in place of 8.2 us)
    const bool pair = r0 + 1 < stride;
    const bool second = r0 + 1 < n;
    if (pair) {
        // four entries' index and value pairs in flight before their gathers
        int64_t i = 0;
        for (; i + 4 <= len; i += 4) {
            int2 cc[4];
            V2 vv[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int64_t e = first + (i + u) * step;
                cc[u] = __ldg(reinterpret_cast<const int2*>(ci + e));
                vv[u] = __ldg(reinterpret_cast<const V2*>(v + e));
            }
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                if (cc[u].x != -1) fma_vec<T>(acc0, vv[u].x, bc + int64_t(cc[u].x) * ldb);
                if (second && cc[u].y != -1) {
                    fma_vec<T>(acc1, vv[u].y, bc + int64_t(cc[u].y) * ldb);
                }
            }
        }
        for (; i < len; ++i) {
            const int64_t e = first + i * step;
            const int2 cc = __ldg(reinterpret_cast<const int2*>(ci + e));
            const V2 vv = __ldg(reinterpret_cast<const V2*>(v + e));
            if (cc.x != -1) fma_vec<T>(acc0, vv.x, bc + int64_t(cc.x) * ldb);
            if (second && cc.y != -1) fma_vec<T>(acc1, vv.y, bc + int64_t(cc.y) * ldb);
        }
    } else {
        for (int64_t i = 0; i < len; ++i) {
            const int64_t e = first + i * step;
            const int32_t col = __ldg(ci + e);
            if (col != -1) fma_vec<T>(acc0, __ldg(v + e), bc + int64_t(col) * ldb);
        }
    }
    store_vec<T>(c + r0 * ldc + sub * VW, acc0, alpha, beta);
    if (second) store_vec<T>(c + (r0 + 1) * ldc + sub * VW, acc1, alpha, beta);
}

// Rows a warp of rhs_rows_kernel takes; 0 where rhs_lanes_kernel stays, and
// kRowPairs for rhs_pairs_kernel (Ell, when its alignment allows).
// `longest`: the longest row (Csr, Ell) or slice (Sellp), 0 when not known.
//
// Rows differ in length inside a warp in Csr and Sellp, and a warp runs to
// its longest: matrices with rows over 64 entries keep rhs_lanes_kernel (one
// long row holds up the other rows of its warp; the power-law matrix's
// longest slices have 1,805 entries).  Ell's rows are all as long as its
// width.
//
// A warp of many rows makes the longest coalesced loads and stores, which
// pays once the matrix and the vectors come from HBM: 32 rows when they are
// short (up to 8 entries, two load steps at most), except at eight lanes per
// row, whose 8 accumulators of 32 rows need 102 registers (267 against 231 us
// with 16 rows, 7-point 128^3); 16 longer ones, so that each load step brings
// two entries per row (27-point 77^3, 4 FP64 columns, Sellp: 55.1 against
// 65.0 us with 32 rows).  7-point 128^3, 4 / 8 / 16 columns, one row per lane
// slot (Csr, FP32 4 columns) or two (Ell, Sellp) -> many rows per warp: Sellp
// FP64 141 / 263 / 474 -> 89 / 115 / 207 us, FP32 67 / 133 / 248 -> 47 / 69 /
// 110 us; Ell FP64 90 / 167 / 319 -> 78 / 128 / 207 us; Csr (whose entries of
// a row already sit together and whose reloads hit L1) FP64 115 -> 95 us at 8
// columns, 224 -> 205 at 16, FP32 104 -> 84 at 16.
//
// With fewer rows there are then too few warps to hide the gathers, and the
// lines below are where the measured sides cross (us, us):
// - four and eight lanes, Ell and Sellp, few rows: the fewest rows per warp,
//   which loads several entries of each row per step.  Sellp 27-point 24^3,
//   16 FP64 columns: 4 rows 6.2, one row per slot 6.4, 16 rows 9.2; 7-point
//   32^3, 16 FP32 columns: 8 rows 3.5, 32 rows 5.6.
// - then, for Ell, two rows per lane slot.  27-point 32^3, 16 FP64 columns:
//   10.2, 16 rows 11.8; 40^3 17.7 and 21.9.  On 2^17 rows the sides meet
//   (5-point 360^2 9.8, 9.9; 27-point 50^3 37.8, 36.7).
// - one and two lanes: one row per slot.  27-point 50^3, 4 FP64 columns, Ell:
//   11.9, 16 rows 14.3.
// - Csr, short rows: one row per slot up to 2^18 rows at four lanes (7-point
//   40^3, 16 FP32 columns 4.8, 32 rows 5.3; 64^3 12.2, 11.7) and 2^19 at
//   eight (7-point 50^3 11.3, 16 rows 12.8; 80^3 55.3, 54.5).
// - Csr, longer rows: the fewest rows per warp on few rows (27-point 24^3, 8
//   FP64 columns: 7.9 -> 5.5).
constexpr int64_t kRowsMaxLen = 64;
constexpr int64_t kRowsShort = 8;
constexpr int kRowPairs = -1;

inline int rhs_rows_per_warp(int fmt, int lanes, int64_t n, int64_t longest)
{
    constexpr int64_t k14 = int64_t(1) << 14, k17 = int64_t(1) << 17;
    if (longest <= 0 || (fmt != 1 && longest > kRowsMaxLen)) return 0;
    const bool short_rows = longest <= kRowsShort;
    const int fewest = kWarp / lanes;
    const int many = lanes < 8 && (short_rows || lanes == 1) ? 32 : 16;
    if (fmt == 0) {
        if (!short_rows) return n < k14 ? fewest : 0;
        return lanes == 4 && n >= 2 * k17 ? many : lanes == 8 && n >= 4 * k17 ? many : 0;
    }
    if (lanes <= 2) {
        if (fmt == 1 && lanes == 2 && !short_rows) return 0;
        return n < (lanes == 2 && short_rows ? k17 / 2 : k17) ? 0 : many;
    }
    if (fmt == 1) return n * lanes < k17 ? fewest : n < k17 ? kRowPairs : many;
    if (lanes == 8 && short_rows) return n < k14 ? fewest : n < 2 * k14 ? 0 : many;
    return n < k17 / 2 ? fewest : many;
}

// Calls f(std::integral_constant<int, ROWS>) for a positive value of
// rhs_rows_per_warp<FMT>; instances that the rule never picks are not made.
template <int FMT, int KL, typename F>
void with_rows_per_warp(int rows, F&& f)
{
    constexpr int kFewest = kWarp / KL;
    if (rows == kFewest) {
        if constexpr (FMT != 1 || KL != 2) f(std::integral_constant<int, kFewest>());
    } else if (rows == 32) {
        if constexpr (KL == 4 || (KL == 2 && FMT != 0)) f(std::integral_constant<int, 32>());
    } else {
        if constexpr (KL == 8 || (KL == 4 && FMT != 0)) f(std::integral_constant<int, 16>());
    }
}

// Products of K columns (K >= 4 and a multiple of the 16-byte vector width;
// b and c rows 16-byte aligned) with the kernel that the sizes call for.
template <typename T, int K, int FMT>
void launch_rhs_lanes(int64_t n, const int32_t* rp, int64_t w_or_s, int64_t stride,
                      const uint64_t* sets, const uint64_t* lens, const int32_t* ci, const T* v,
                      const T* b, int64_t ldb, T* c, int64_t ldc, const T* alpha, const T* beta,
                      int64_t longest, cudaStream_t st)
{
    static_assert(K >= 4 && K % Vec16<T>::width == 0, "column slices of 16 bytes");
    constexpr int KL = K / Vec16<T>::width;
    const int rows = rhs_rows_per_warp(FMT, KL, n, longest);
    if (rows > 0) {
        with_rows_per_warp<FMT, KL>(rows, [&](auto rc) {
            constexpr int ROWS = decltype(rc)::value;
            const int64_t grid = ceildiv(ceildiv(n, ROWS), kLanesBlock / kWarp);
            rhs_rows_kernel<T, K, FMT, ROWS><<<grid, kLanesBlock, 0, st>>>(
                n, rp, w_or_s, stride, sets, lens, ci, v, b, ldb, c, ldc, alpha, beta);
        });
        return;
    }
    if constexpr (FMT == 1 && KL >= 4) {
        if (rows == kRowPairs && stride % 2 == 0 && reinterpret_cast<uintptr_t>(ci) % 8 == 0 &&
            reinterpret_cast<uintptr_t>(v) % (2 * sizeof(T)) == 0) {
            rhs_pairs_kernel<T, K><<<ceildiv(ceildiv(n, 2) * KL, kLanesBlock), kLanesBlock, 0,
                                     st>>>(n, w_or_s, stride, ci, v, b, ldb, c, ldc, alpha, beta);
            return;
        }
    }
    rhs_lanes_kernel<T, K, FMT><<<ceildiv(n * KL, kLanesBlock), kLanesBlock, 0, st>>>(
        n, rp, w_or_s, stride, sets, lens, ci, v, b, ldb, c, ldc, alpha, beta);
}

}  // namespace b2s

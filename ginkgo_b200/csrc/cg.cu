// Fused preconditioned CG (scalar Jacobi, block Jacobi or identity), the loop of
// core/solver/cg.cpp:91-189 with the kernels of
// common/unified/solver/cg_kernels.cpp:23-107 regrouped into two passes per
// iteration and no host synchronisation inside the loop:
//
//   spmv pass   p' = z + (rho / prev_rho) p  with z = D^-1 r, formed on the
//               fly for every column index the SpMV touches (p is double
//               buffered, so every row reads the old p); q = A p';
//               dot(p', q) reduced in-kernel; the last block sets
//               alpha = rho / dot(p', q)  (step_1 + SpMV + dot)
//   update pass x += alpha p', r -= alpha q; rho' = dot(r, D^-1 r) and
//               ||r||^2 reduced in-kernel; the last block advances the
//               iteration, swaps rho, and applies the Iteration and
//               ResidualNorm(rhs_norm) checks  (step_2 + precond + 2 dots +
//               residual_norm check)
//
// With four or more right-hand sides (FP64; eight or more in FP32) the same
// two passes run with lanes owning 16-byte column slices of each row.  Large
// systems run a split iteration of three passes (cg_direction_kernel, an
// SpMV with the dot as its epilogue, cg_residual_kernel) that gathers p
// alone.
//
// With scalar Jacobi z is never stored.  A block Jacobi preconditioner
// stores z = M^-1 r, formed in the update pass (see cg_block_kernel), and
// the SpMV passes read it in place of D^-1 r.  Per-column stopping status
// uses the reference's bit
// layout; stopped columns are frozen as in the reference.  The host replays
// a CUDA graph of `check_every` iterations and reads the stop flag once per
// replay.
#include <cstring>
#include <type_traits>

#include "csr_async.cuh"
#include "grid_exchange.cuh"
#include "jacobi_scheme.cuh"
#include "rhs_lanes.cuh"
#include "solver_common.cuh"

namespace b2s {
namespace {

template <typename T>
struct CgScalars {
    T rho[kMaxRhs], prev_rho[kMaxRhs], alpha[kMaxRhs], tau[kMaxRhs],
        start[kMaxRhs];
    int pending[kMaxRhs];  // split passes: x still lacks alpha p
};

template <typename T>
__device__ __forceinline__ T cg_p(T d, T r, T beta, T p, bool from_z)
{
    const T z = mul_rn(d, r);
    return from_z ? z : add_rn(z, mul_rn(beta, p));
}

// The last block's part of the initial pass (its first warp, lane j taking
// column j): tot holds ||b||^2, rho = dot(r, z) and ||r||^2 of every column
// (K each); sets the starting norms, rho and the initial stopping status.
template <typename T, int K>
__device__ void cg_init_finish(const T* tot, int k, SolveCtl* ctl, CgScalars<T>* sc)
{
    const int j = threadIdx.x;
    bool stopped = true;
    if (j < K) {
        const bool none = ctl->max_iters <= 0;
        uint8_t s = 0;
        if (j >= k) {
            stop_status(s, kIterationId, true);  // padding column
        }
        const T tau = sqrt(tot[2 * K + j]), rho = tot[K + j];
        const T start = start_norm(ctl, T(sqrt(tot[j])), tau);
        if (none) stop_status(s, kIterationId, true);
        if (residual_met(ctl, tau, rho, start)) converge_status(s, kResidualId, true);
        sc->start[j] = start;
        sc->rho[j] = rho;
        sc->prev_rho[j] = T(1);
        sc->alpha[j] = T(0);
        sc->pending[j] = 0;
        sc->tau[j] = tau;
        ctl->status[j] = s;
        stopped = has_stopped(s);
    }
    const bool all = __all_sync(0xffffffffu, stopped);
    if (j == 0) {
        ctl->ticket = 0;
        ctl->iter = 0;
        ctl->all_stopped = all;
    }
}

// The last block's part of the update pass (its first warp, lane j taking
// column j): tot holds the new rho = dot(r, z) and ||r||^2 per column;
// advances the iteration, swaps rho and applies the Iteration and residual
// checks.  Every load is issued before the first store and the columns run
// side by side: one thread walking them waited for a dozen L2 round trips
// per column, 20 us of each iteration with 16 columns.
template <typename T, int K>
__device__ void cg_update_finish(const T* tot, SolveCtl* ctl, CgScalars<T>* sc)
{
    const int j = threadIdx.x;
    const int iter = ctl->iter + 1, max_iters = ctl->max_iters;
    bool stopped = true;
    if (j < K) {
        uint8_t s = ctl->status[j];
        const T old_rho = sc->rho[j], start = sc->start[j];
        const T rho = tot[j], tau = sqrt(tot[K + j]);
        const bool met = residual_met(ctl, tau, rho, start);
        if (!has_stopped(s)) {
            if (met) converge_status(s, kResidualId, true);
            if (iter >= max_iters) stop_status(s, kIterationId, true);
            sc->prev_rho[j] = old_rho;
            sc->rho[j] = rho;
            sc->tau[j] = tau;
            ctl->status[j] = s;
        }
        stopped = has_stopped(s);
    }
    const bool all = __all_sync(0xffffffffu, stopped);
    if (j == 0) {
        ctl->ticket = 0;
        ctl->iter = iter;
        ctl->all_stopped = all;
    }
}

template <typename T, int K>
__global__ void __launch_bounds__(kSolverBlock)
    cg_init_kernel(int64_t n, const T* __restrict__ dinv,
                   const T* __restrict__ b, int64_t ldb, int k,
                   const T* __restrict__ r, T* __restrict__ p_old,
                   SolveCtl* ctl, CgScalars<T>* sc, T* __restrict__ partials)
{
    __shared__ T red[kSolverBlock / kWarp * 3 * K];
    __shared__ T tot[3 * K];
    __shared__ int last;
    T acc[3 * K];
#pragma unroll
    for (int j = 0; j < 3 * K; ++j) acc[j] = T(0);
    for (int64_t i = blockIdx.x * int64_t(kSolverBlock) + threadIdx.x; i < n;
         i += int64_t(gridDim.x) * kSolverBlock) {
        const T d = dinv ? dinv[i] : T(1);
#pragma unroll
        for (int j = 0; j < K; ++j) {
            const T rr = r[i * K + j];
            const T bb = j < k ? b[i * ldb + j] : T(0);
            p_old[i * K + j] = T(0);
            acc[j] += bb * bb;
            acc[K + j] += rr * mul_rn(d, rr);
            acc[2 * K + j] += rr * rr;
        }
    }
    block_partials<T, 3 * K>(acc, partials, red);
    if (last_block_done(&ctl->ticket, &last)) {
        sum_partials<T, 3 * K>(partials, gridDim.x, tot, red);
        if (threadIdx.x < kWarp) cg_init_finish<T, K>(tot, k, ctl, sc);
    }
}

template <typename T, int SW, int K>
__global__ void __launch_bounds__(kSolverBlock)
    cg_spmv_kernel(int64_t n, const int32_t* __restrict__ rp,
                   const int32_t* __restrict__ ci, const T* __restrict__ v,
                   const T* __restrict__ dinv, const T* __restrict__ r,
                   const T* __restrict__ p_old, T* __restrict__ p_new,
                   T* __restrict__ q, SolveCtl* ctl, CgScalars<T>* sc,
                   T* __restrict__ partials)
{
    __shared__ T red[kSolverBlock / kWarp * K];
    __shared__ T tot[K];
    __shared__ int last;
    if (ctl->all_stopped) return;
    bool active[K], from_z[K];
    T beta[K];
#pragma unroll
    for (int j = 0; j < K; ++j) {
        active[j] = !has_stopped(ctl->status[j]);
        const T pr = sc->prev_rho[j];
        from_z[j] = pr == T(0);
        beta[j] = from_z[j] ? T(0) : sc->rho[j] / pr;
    }
    T dot[K];
#pragma unroll
    for (int j = 0; j < K; ++j) dot[j] = T(0);
    const int lane = threadIdx.x % SW;
    const int64_t nsub = int64_t(gridDim.x) * kSolverBlock / SW;
    // warp-uniform trip count: all lanes of a warp run every iteration, so
    // the subwarp shuffles below always see the whole warp
    for (int64_t wbase = (blockIdx.x * int64_t(kSolverBlock) + threadIdx.x) /
                         kWarp * (kWarp / SW);
         wbase < n; wbase += nsub) {
        const int64_t row = wbase + (threadIdx.x % kWarp) / SW;
        const bool valid = row < n;
        T acc[K];
#pragma unroll
        for (int j = 0; j < K; ++j) acc[j] = T(0);
        const int end = valid ? rp[row + 1] : 0;
        for (int e = (valid ? rp[row] : end) + lane; e < end; e += SW) {
            const T a = v[e];
            const int64_t c = ci[e];
            const T d = dinv ? dinv[c] : T(1);
#pragma unroll
            for (int j = 0; j < K; ++j) {
                if (active[j]) {
                    acc[j] += a * cg_p(d, r[c * K + j], beta[j], p_old[c * K + j],
                                       from_z[j]);
                }
            }
        }
#pragma unroll
        for (int j = 0; j < K; ++j) acc[j] = subwarp_sum<SW>(acc[j]);
        if (valid && lane == 0) {
            const T d = dinv ? dinv[row] : T(1);
#pragma unroll
            for (int j = 0; j < K; ++j) {
                if (active[j]) {
                    const T pn = cg_p(d, r[row * K + j], beta[j],
                                      p_old[row * K + j], from_z[j]);
                    p_new[row * K + j] = pn;
                    q[row * K + j] = acc[j];
                    dot[j] += pn * acc[j];
                }
            }
        }
    }
    block_partials<T, K>(dot, partials, red);
    if (last_block_done(&ctl->ticket, &last)) {
        sum_partials<T, K>(partials, gridDim.x, tot, red);
        if (threadIdx.x < K) {
            const T pq = tot[threadIdx.x];
            // step_2 skips the update when dot(p, q) == 0
            sc->alpha[threadIdx.x] = pq != T(0) ? sc->rho[threadIdx.x] / pq : T(0);
        }
        if (threadIdx.x == 0) ctl->ticket = 0;
    }
}

template <typename T, int K>
__global__ void __launch_bounds__(kSolverBlock)
    cg_update_kernel(int64_t n, const T* __restrict__ dinv, T* __restrict__ x,
                     int64_t ldx, T* __restrict__ r, const T* __restrict__ p,
                     const T* __restrict__ q, SolveCtl* ctl, CgScalars<T>* sc,
                     T* __restrict__ partials)
{
    __shared__ T red[kSolverBlock / kWarp * 2 * K];
    __shared__ T tot[2 * K];
    __shared__ int last;
    if (ctl->all_stopped) return;
    bool active[K];
    T alpha[K];
#pragma unroll
    for (int j = 0; j < K; ++j) {
        active[j] = !has_stopped(ctl->status[j]);
        alpha[j] = sc->alpha[j];
    }
    T acc[2 * K];
#pragma unroll
    for (int j = 0; j < 2 * K; ++j) acc[j] = T(0);
    for (int64_t i = blockIdx.x * int64_t(kSolverBlock) + threadIdx.x; i < n;
         i += int64_t(gridDim.x) * kSolverBlock) {
        const T d = dinv ? dinv[i] : T(1);
#pragma unroll
        for (int j = 0; j < K; ++j) {
            if (active[j]) {
                x[i * ldx + j] += alpha[j] * p[i * K + j];
                const T rr = r[i * K + j] - alpha[j] * q[i * K + j];
                r[i * K + j] = rr;
                acc[j] += rr * mul_rn(d, rr);
                acc[K + j] += rr * rr;
            }
        }
    }
    block_partials<T, 2 * K>(acc, partials, red);
    if (last_block_done(&ctl->ticket, &last)) {
        sum_partials<T, 2 * K>(partials, gridDim.x, tot, red);
        if (threadIdx.x < kWarp) cg_update_finish<T, K>(tot, ctl, sc);
    }
}

// ---------------------------------------------------------------------------
// Four or more right-hand sides: lanes own columns.  A row's KL = K / VW
// lanes each hold VW = 16 / sizeof(T) consecutive columns (one 16-byte
// vector of the row-major n x K blocks), so the gathers of r(c, :) and
// p(c, :) are contiguous 16-byte loads across the row's lanes and no
// shuffle reduction runs per row.  Stopped columns are computed along
// (their results are never used: the update pass freezes them).
// ---------------------------------------------------------------------------

template <typename T, int K>
__global__ void __launch_bounds__(kSolverBlock)
    cg_spmv_lanes_kernel(int64_t n, const int32_t* __restrict__ rp,
                         const int32_t* __restrict__ ci, const T* __restrict__ v,
                         const T* __restrict__ dinv, const T* __restrict__ r,
                         const T* __restrict__ p_old, T* __restrict__ p_new,
                         T* __restrict__ q, SolveCtl* ctl, CgScalars<T>* sc,
                         T* __restrict__ partials)
{
    constexpr int VW = int(16 / sizeof(T));
    constexpr int KL = K / VW;         // lanes per row
    constexpr int RPW = kWarp / KL;    // rows per warp
    constexpr int W = kSolverBlock / kWarp;
    __shared__ T red[W][K];
    __shared__ T tot[K];
    __shared__ int last;
    if (ctl->all_stopped) return;
    const int lane = threadIdx.x % kWarp, wid = threadIdx.x / kWarp;
    const int col0 = (lane % KL) * VW;
    bool from_z[VW];
    T beta[VW];
#pragma unroll
    for (int u = 0; u < VW; ++u) {
        const T pr = sc->prev_rho[col0 + u];
        from_z[u] = pr == T(0);
        beta[u] = from_z[u] ? T(0) : sc->rho[col0 + u] / pr;
    }
    T dot[VW];
#pragma unroll
    for (int u = 0; u < VW; ++u) dot[u] = T(0);
    const int64_t nwarps = int64_t(gridDim.x) * W;
    for (int64_t g = blockIdx.x * int64_t(W) + wid; g * RPW < n; g += nwarps) {
        const int64_t row = g * RPW + lane / KL;
        if (row < n) {
            T acc[VW];
#pragma unroll
            for (int u = 0; u < VW; ++u) acc[u] = T(0);
            const int end = rp[row + 1];
            for (int e = rp[row]; e < end; ++e) {
                const T a = v[e];
                const int64_t c = ci[e];
                const T d = dinv ? dinv[c] : T(1);
                T rr[VW], pp[VW];
                ld_vec<T, VW>(r + c * K + col0, rr);
                ld_vec<T, VW>(p_old + c * K + col0, pp);
#pragma unroll
                for (int u = 0; u < VW; ++u) acc[u] += a * cg_p(d, rr[u], beta[u], pp[u], from_z[u]);
            }
            const T d = dinv ? dinv[row] : T(1);
            T rr[VW], pp[VW], pn[VW];
            ld_vec<T, VW>(r + row * K + col0, rr);
            ld_vec<T, VW>(p_old + row * K + col0, pp);
#pragma unroll
            for (int u = 0; u < VW; ++u) {
                pn[u] = cg_p(d, rr[u], beta[u], pp[u], from_z[u]);
                dot[u] += pn[u] * acc[u];
            }
            st_vec<T, VW>(p_new + row * K + col0, pn);
            st_vec<T, VW>(q + row * K + col0, acc);
        }
    }
    // lanes with the same columns: xor over the row bits of the lane index
#pragma unroll
    for (int off = KL; off < kWarp; off *= 2) {
#pragma unroll
        for (int u = 0; u < VW; ++u) dot[u] += __shfl_xor_sync(0xffffffffu, dot[u], off);
    }
    if (lane < KL) {
#pragma unroll
        for (int u = 0; u < VW; ++u) red[wid][col0 + u] = dot[u];
    }
    __syncthreads();
    if (threadIdx.x < K) {
        T s = T(0);
        for (int k = 0; k < W; ++k) s += red[k][threadIdx.x];
        partials[blockIdx.x * K + threadIdx.x] = s;
    }
    if (last_block_done(&ctl->ticket, &last)) {
        fold_columns<T, K, 1>(partials, gridDim.x, tot);
        if (threadIdx.x < K) {
            const T pq = tot[threadIdx.x];
            sc->alpha[threadIdx.x] = pq != T(0) ? sc->rho[threadIdx.x] / pq : T(0);
        }
        if (threadIdx.x == 0) ctl->ticket = 0;
    }
}

// x += alpha p, r -= alpha q over the row-major n x K blocks as one flat
// array of 16-byte vectors (a thread keeps the same VW columns: the grid
// stride is a multiple of K); rho' = dot(r, D^-1 r) and ||r||^2 per column.
template <typename T, int K>
__global__ void __launch_bounds__(kSolverBlock)
    cg_update_lanes_kernel(int64_t n, const T* __restrict__ dinv, T* __restrict__ x,
                           int64_t ldx, T* __restrict__ r, const T* __restrict__ p,
                           const T* __restrict__ q, SolveCtl* ctl, CgScalars<T>* sc,
                           T* __restrict__ partials)
{
    constexpr int VW = int(16 / sizeof(T));
    constexpr int KL = K / VW;
    constexpr int W = kSolverBlock / kWarp;
    __shared__ T red[W][2 * K];
    __shared__ T tot[2 * K];
    __shared__ int last;
    if (ctl->all_stopped) return;
    const int lane = threadIdx.x % kWarp, wid = threadIdx.x / kWarp;
    const int64_t t0 = blockIdx.x * int64_t(kSolverBlock) + threadIdx.x;
    const int col0 = int((t0 * VW) % K);
    bool active[VW];
    T alpha[VW];
#pragma unroll
    for (int u = 0; u < VW; ++u) {
        active[u] = !has_stopped(ctl->status[col0 + u]);
        alpha[u] = sc->alpha[col0 + u];
    }
    T acc[2 * VW];
#pragma unroll
    for (int u = 0; u < 2 * VW; ++u) acc[u] = T(0);
    const int64_t nvec = n * K / VW;
    for (int64_t t = t0; t < nvec; t += int64_t(gridDim.x) * kSolverBlock) {
        const int64_t i = t * VW / K;
        const T d = dinv ? dinv[i] : T(1);
        T pv[VW], qv[VW], rv[VW];
        ld_vec<T, VW>(p + t * VW, pv);
        ld_vec<T, VW>(q + t * VW, qv);
        ld_vec<T, VW>(r + t * VW, rv);
#pragma unroll
        for (int u = 0; u < VW; ++u) {
            if (active[u]) {
                x[i * ldx + col0 + u] += alpha[u] * pv[u];
                const T rr = rv[u] - alpha[u] * qv[u];
                rv[u] = rr;
                acc[u] += rr * mul_rn(d, rr);
                acc[VW + u] += rr * rr;
            }
        }
        st_vec<T, VW>(r + t * VW, rv);
    }
#pragma unroll
    for (int off = KL; off < kWarp; off *= 2) {
#pragma unroll
        for (int u = 0; u < 2 * VW; ++u) acc[u] += __shfl_xor_sync(0xffffffffu, acc[u], off);
    }
    if (lane < KL) {
#pragma unroll
        for (int u = 0; u < VW; ++u) {
            red[wid][col0 + u] = acc[u];
            red[wid][K + col0 + u] = acc[VW + u];
        }
    }
    __syncthreads();
    // partials: rho parts [block][K], then ||r||^2 parts [block][K] (two
    // K-wide sums keep the last block's register use low)
    if (threadIdx.x < 2 * K) {
        T s = T(0);
        for (int k = 0; k < W; ++k) s += red[k][threadIdx.x];
        const int j = threadIdx.x % K;
        partials[(threadIdx.x < K ? 0 : int64_t(gridDim.x) * K) + blockIdx.x * K + j] = s;
    }
    if (last_block_done(&ctl->ticket, &last)) {
        fold_columns<T, K, 2>(partials, gridDim.x, tot);
        if (threadIdx.x < kWarp) cg_update_finish<T, K>(tot, ctl, sc);
    }
}

// ---------------------------------------------------------------------------
// Split iteration, for systems whose vectors do not stay in L1 between the
// gathers: forming p' = D^-1 r + beta p at every gathered column (the fused
// pass above) costs three gathers per stored entry.  Three passes instead:
//   cg_direction_kernel  x += alpha p of the iteration before, then
//                        p = D^-1 r + beta p in place (the fused pass's
//                        rounding): r, p, x read once, p, x written once
//   SpMV with epilogue   q = A p and dot(p, q) from the finished rows, no
//                        pass of its own for the dot; last block: alpha
//   cg_residual_kernel   r -= alpha q, dot(r, D^-1 r) and ||r||^2; last
//                        block: the iteration's end
// ten vector passes and the matrix per iteration, the least this loop can
// do with its two reduction points.  7-point 128^3: 16.7 + 44.6 + 17.5 us;
// 64^3 with 16 columns: 25.3 + 37.5 + 22.2 us (the fused passes 78.7 + 47.4).  The x update is applied one pass late;
// `pending` marks the columns that still need it and cg_last_step_kernel
// closes the loop.
// ---------------------------------------------------------------------------
//
// From 2^17 rows with one column (us per iteration, fused -> split: 5-point
// 360^2 21.0 -> 19.9, 7-point 48^3 21.3 -> 21.0, 64^3 26.9 -> 22.9, 27-point
// 64^3 66.5 -> 38.5, 7-point 128^3 118 -> 79).  With 16-byte column slices
// from 393,216 vector entries (7-point 32^3, 4 columns 19.3 -> 21.1, 16
// columns 30.1 -> 25.5; 48^3, 4 columns 26.0 -> 24.1; 128^3, 16 columns 728
// -> 617), or an eighth of that where rows are longer than 8 entries, each a
// gather (27-point 24^3, 4 columns 25.8 -> 23.0).
constexpr int64_t kCgSplitRows = int64_t(1) << 17;
constexpr int64_t kCgSplitEntries = int64_t(3) << 17;

// K columns as one flat array of VW-wide vectors (VW = 1 for one column);
// a thread keeps the same columns: the grid stride is a multiple of K.
template <typename T, int K>
struct CgSlice {
    static constexpr int VW = K * sizeof(T) >= 32 ? int(16 / sizeof(T)) : 1;
    static_assert(VW > 1 || K == 1, "one column or 16-byte column slices");
};

template <typename T, int VW>
__device__ __forceinline__ void cg_load(const T* p, T (&o)[VW])
{
    if constexpr (VW == 1) {
        o[0] = *p;
    } else {
        ld_vec<T, VW>(p, o);
    }
}
template <typename T, int VW>
__device__ __forceinline__ void cg_store(T* p, const T (&o)[VW])
{
    if constexpr (VW == 1) {
        *p = o[0];
    } else {
        st_vec<T, VW>(p, o);
    }
}

// Vectors of a thread in flight in the streaming passes.
constexpr int kCgUnroll = 4;

// x: null when the caller keeps x itself (block Jacobi).  xvec: x's rows
// are K wide and 16-byte aligned.
template <typename T, int K>
__global__ void __launch_bounds__(kSolverBlock)
    cg_direction_kernel(int64_t n, const T* __restrict__ dinv, const T* __restrict__ r,
                        T* __restrict__ p, T* __restrict__ x, int64_t ldx, bool xvec,
                        SolveCtl* ctl, CgScalars<T>* sc)
{
    constexpr int VW = CgSlice<T, K>::VW;
    if (ctl->all_stopped) return;
    const int64_t t0 = blockIdx.x * int64_t(kSolverBlock) + threadIdx.x;
    const int col0 = int((t0 * VW) % K);
    bool active[VW], from_z[VW], pend[VW];
    T beta[VW], alpha[VW];
    bool all = true;
#pragma unroll
    for (int u = 0; u < VW; ++u) {
        active[u] = !has_stopped(ctl->status[col0 + u]);
        pend[u] = x != nullptr && sc->pending[col0 + u];
        all = all && active[u] && pend[u];
        alpha[u] = sc->alpha[col0 + u];
        const T pr = sc->prev_rho[col0 + u];
        from_z[u] = pr == T(0);
        beta[u] = from_z[u] ? T(0) : sc->rho[col0 + u] / pr;
    }
    const int64_t nvec = n * K / VW;
    const int64_t step = int64_t(gridDim.x) * kSolverBlock;
    for (int64_t tb = t0; tb < nvec; tb += kCgUnroll * step) {
        T d[kCgUnroll], pv[kCgUnroll][VW], rv[kCgUnroll][VW], xv[kCgUnroll][VW];
#pragma unroll
        for (int w = 0; w < kCgUnroll; ++w) {
            const int64_t t = tb + w * step, i = t * VW / K;
            if (t < nvec) {
                d[w] = dinv ? dinv[i] : T(1);
                cg_load<T, VW>(p + t * VW, pv[w]);
                cg_load<T, VW>(r + t * VW, rv[w]);
                T* xp = x + i * ldx + col0;
                if (all && xvec) {
                    cg_load<T, VW>(xp, xv[w]);
                } else {
#pragma unroll
                    for (int u = 0; u < VW; ++u) xv[w][u] = pend[u] ? xp[u] : T(0);
                }
            }
        }
#pragma unroll
        for (int w = 0; w < kCgUnroll; ++w) {
            const int64_t t = tb + w * step, i = t * VW / K;
            if (t < nvec) {
                T* xp = x + i * ldx + col0;
#pragma unroll
                for (int u = 0; u < VW; ++u) xv[w][u] += alpha[u] * pv[w][u];
                if (all && xvec) {
                    cg_store<T, VW>(xp, xv[w]);
                } else {
#pragma unroll
                    for (int u = 0; u < VW; ++u) {
                        if (pend[u]) xp[u] = xv[w][u];
                    }
                }
#pragma unroll
                for (int u = 0; u < VW; ++u) {
                    if (active[u]) pv[w][u] = cg_p(d[w], rv[w][u], beta[u], pv[w][u], from_z[u]);
                }
                cg_store<T, VW>(p + t * VW, pv[w]);
            }
        }
    }
}

// x += alpha p for the columns still pending after the loop.
template <typename T, int K>
__global__ void __launch_bounds__(kSolverBlock)
    cg_last_step_kernel(int64_t n, const T* __restrict__ p, T* __restrict__ x, int64_t ldx,
                        const CgScalars<T>* sc)
{
    for (int64_t t = blockIdx.x * int64_t(kSolverBlock) + threadIdx.x; t < n * K;
         t += int64_t(gridDim.x) * kSolverBlock) {
        const int64_t i = t / K;
        const int j = int(t % K);
        if (sc->pending[j]) x[i * ldx + j] += sc->alpha[j] * p[t];
    }
}

// The last block of an SpMV with dot(p, q): alpha of the active columns.
template <typename T>
__device__ __forceinline__ void cg_alpha(int j, T pq, const SolveCtl* ctl, CgScalars<T>* sc)
{
    // step_2 skips the update when dot(p, q) == 0
    const bool active = !has_stopped(ctl->status[j]);
    if (active) sc->alpha[j] = pq != T(0) ? sc->rho[j] / pq : T(0);
    sc->pending[j] = active;
}

// Epilogue of csr_async_epi_kernel: dot(p, q) of the rows as they finish.
template <typename T>
struct CgDotEpilogue {
    static constexpr bool kOn = true;
    const T* p;
    T* partials;
    SolveCtl* ctl;
    CgScalars<T>* sc;
    T sum[1] = {T(0)};
    __device__ __forceinline__ void row(int64_t i, T q) { sum[0] += p[i] * q; }
    // sm: the block's stages, no longer used
    __device__ __forceinline__ void finish(void* sm)
    {
        static_assert(kAsyncBlock == kSolverBlock, "one block size");
        T* red = static_cast<T*>(sm);
        T* tot = red + kSolverBlock / kWarp;
        int* last = reinterpret_cast<int*>(tot + 1);
        block_partials<T, 1>(sum, partials, red);
        if (last_block_done(&ctl->ticket, last)) {
            sum_partials<T, 1>(partials, gridDim.x, tot, red);
            if (threadIdx.x == 0) {
                cg_alpha(0, tot[0], ctl, sc);
                ctl->ticket = 0;
            }
        }
    }
};

// q = A p for K columns, a warp per 16 or 32 rows (rhs_rows), with dot(p, q) per
// column from the finished rows.
template <typename T, int K, int ROWS>
__global__ void __launch_bounds__(kSolverBlock)
    cg_spmv_rows_kernel(int64_t n, const int32_t* __restrict__ rp,
                        const int32_t* __restrict__ ci, const T* __restrict__ v,
                        const T* __restrict__ p, T* __restrict__ q, SolveCtl* ctl,
                        CgScalars<T>* sc, T* __restrict__ partials)
{
    constexpr int VW = CgSlice<T, K>::VW;
    constexpr int KL = K / VW;
    constexpr int W = kSolverBlock / kWarp;
    __shared__ T red[W][K];
    __shared__ T tot[K];
    __shared__ int last;
    if (ctl->all_stopped) return;
    const int lane = threadIdx.x % kWarp, wid = threadIdx.x / kWarp;
    T dot[VW];
#pragma unroll
    for (int u = 0; u < VW; ++u) dot[u] = T(0);
    for (int64_t r0 = (blockIdx.x * int64_t(W) + wid) * ROWS; r0 < n;
         r0 += int64_t(gridDim.x) * W * ROWS) {
        rhs_rows<T, K, 0, ROWS>(n, r0, rp, 0, 0, nullptr, nullptr, ci, v, p, K,
                          [&](int64_t row, int col0, const typename Vec16<T>::type& acc) {
                              T pv[VW], a[VW];
                              memcpy(a, &acc, 16);
                              ld_vec<T, VW>(p + row * K + col0, pv);
#pragma unroll
                              for (int u = 0; u < VW; ++u) dot[u] += pv[u] * a[u];
                              st_vec<T, VW>(q + row * K + col0, a);
                          });
    }
    // lanes with the same columns
#pragma unroll
    for (int off = KL; off < kWarp; off *= 2) {
#pragma unroll
        for (int u = 0; u < VW; ++u) dot[u] += __shfl_xor_sync(0xffffffffu, dot[u], off);
    }
    if (lane < KL) {
#pragma unroll
        for (int u = 0; u < VW; ++u) red[wid][lane * VW + u] = dot[u];
    }
    __syncthreads();
    if (threadIdx.x < K) {
        T s = T(0);
        for (int k = 0; k < W; ++k) s += red[k][threadIdx.x];
        partials[blockIdx.x * K + threadIdx.x] = s;
    }
    if (last_block_done(&ctl->ticket, &last)) {
        fold_columns<T, K, 1>(partials, gridDim.x, tot);
        if (threadIdx.x < K) cg_alpha(threadIdx.x, tot[threadIdx.x], ctl, sc);
        if (threadIdx.x == 0) ctl->ticket = 0;
    }
}

// r -= alpha q; rho' = dot(r, D^-1 r) and ||r||^2 per column.
template <typename T, int K>
__global__ void __launch_bounds__(kSolverBlock)
    cg_residual_kernel(int64_t n, const T* __restrict__ dinv, T* __restrict__ r,
                       const T* __restrict__ q, SolveCtl* ctl, CgScalars<T>* sc,
                       T* __restrict__ partials)
{
    constexpr int VW = CgSlice<T, K>::VW;
    constexpr int KL = K / VW;
    constexpr int W = kSolverBlock / kWarp;
    __shared__ T red[W][2 * K];
    __shared__ T tot[2 * K];
    __shared__ int last;
    if (ctl->all_stopped) return;
    const int lane = threadIdx.x % kWarp, wid = threadIdx.x / kWarp;
    const int64_t t0 = blockIdx.x * int64_t(kSolverBlock) + threadIdx.x;
    const int col0 = int((t0 * VW) % K);
    bool active[VW];
    T alpha[VW];
#pragma unroll
    for (int u = 0; u < VW; ++u) {
        active[u] = !has_stopped(ctl->status[col0 + u]);
        alpha[u] = sc->alpha[col0 + u];
    }
    T acc[2 * VW];
#pragma unroll
    for (int u = 0; u < 2 * VW; ++u) acc[u] = T(0);
    const int64_t nvec = n * K / VW;
    const int64_t step = int64_t(gridDim.x) * kSolverBlock;
    for (int64_t tb = t0; tb < nvec; tb += kCgUnroll * step) {
        T d[kCgUnroll], qv[kCgUnroll][VW], rv[kCgUnroll][VW];
#pragma unroll
        for (int w = 0; w < kCgUnroll; ++w) {
            const int64_t t = tb + w * step;
            if (t < nvec) {
                d[w] = dinv ? dinv[t * VW / K] : T(1);
                cg_load<T, VW>(q + t * VW, qv[w]);
                cg_load<T, VW>(r + t * VW, rv[w]);
            }
        }
#pragma unroll
        for (int w = 0; w < kCgUnroll; ++w) {
            const int64_t t = tb + w * step;
            if (t < nvec) {
#pragma unroll
                for (int u = 0; u < VW; ++u) {
                    if (active[u]) {
                        const T rr = rv[w][u] - alpha[u] * qv[w][u];
                        rv[w][u] = rr;
                        acc[u] += rr * mul_rn(d[w], rr);
                        acc[VW + u] += rr * rr;
                    }
                }
                cg_store<T, VW>(r + t * VW, rv[w]);
            }
        }
    }
#pragma unroll
    for (int off = KL; off < kWarp; off *= 2) {
#pragma unroll
        for (int u = 0; u < 2 * VW; ++u) acc[u] += __shfl_xor_sync(0xffffffffu, acc[u], off);
    }
    if (lane < KL) {
#pragma unroll
        for (int u = 0; u < VW; ++u) {
            red[wid][lane * VW + u] = acc[u];
            red[wid][K + lane * VW + u] = acc[VW + u];
        }
    }
    __syncthreads();
    // partials: rho parts [block][K], then ||r||^2 parts [block][K] (two
    // K-wide sums keep the last block's register use low)
    if (threadIdx.x < 2 * K) {
        T s = T(0);
        for (int k = 0; k < W; ++k) s += red[k][threadIdx.x];
        const int j = threadIdx.x % K;
        partials[(threadIdx.x < K ? 0 : int64_t(gridDim.x) * K) + blockIdx.x * K + j] = s;
    }
    if (last_block_done(&ctl->ticket, &last)) {
        fold_columns<T, K, 2>(partials, gridDim.x, tot);
        if (threadIdx.x < kWarp) cg_update_finish<T, K>(tot, ctl, sc);
    }
}

// ---------------------------------------------------------------------------
// One right-hand side on a small system: the whole loop in one cooperative
// kernel, one block per SM.  At these sizes an iteration's data sits in L1,
// L2 and registers and the time goes to launches and to the drain and fill
// of each pass; here the passes are separated by grid_exchange, which also
// carries the dots.  A thread (SW lanes when there are fewer rows than
// threads) owns RPT rows and keeps their r, x, p, q and D^-1 in registers;
// r and p go to global memory only for the other rows' gathers, which read
// L2 (__ldcg), p double buffered as in the fused passes.
// 5-point 256^2 to 1e-10 (710 iterations): 11.3 -> 6.0 ms.
// ---------------------------------------------------------------------------
constexpr int kCgResidentBlock = 512;
constexpr int kCgResidentIters = 1 << 13;  // iterations per launch
// Status of the loop when the device cannot hold its blocks at once (a
// limited share of the SMs) or a block's entries exceed its stage (rows
// longer than max_row_nnz): nothing has run, the passes take the solve.
constexpr int kCgNotResident = 1;

template <typename T, int SW, int RPT>
__global__ void __launch_bounds__(kCgResidentBlock, 1)
    cg_resident_kernel(int64_t n, const int32_t* __restrict__ rp,
                       const int32_t* __restrict__ ci, const T* __restrict__ v,
                       const T* __restrict__ dinv, T* __restrict__ x, int64_t ldx, T* r, T* p0,
                       T* p1, SolveCtl* ctl, CgScalars<T>* sc, ExchangeSlot* slots, int capacity,
                       int polls)
{
    extern __shared__ __align__(16) unsigned char stage_raw[];
    __shared__ double red[kExchangeShared];
    if (ctl->all_stopped) return;
    const int sub = threadIdx.x % SW;
    // the block's rows are consecutive, about n / gridDim.x of them
    const int64_t row0 = n * blockIdx.x / gridDim.x, row1 = n * (blockIdx.x + 1) / gridDim.x;
    const int64_t first = row0 + threadIdx.x / SW;
    constexpr int step = kCgResidentBlock / SW;
    int rs[RPT], re[RPT];
    T rr[RPT], xx[RPT], pp[RPT], qq[RPT], dd[RPT];
    T* pa = ctl->iter % 2 ? p1 : p0;  // p of the iteration before
    T* pb = ctl->iter % 2 ? p0 : p1;
#pragma unroll
    for (int m = 0; m < RPT; ++m) {
        const int64_t row = first + m * step;
        rs[m] = re[m] = 0;  // (both minus e0 below: still no entries)
        rr[m] = xx[m] = pp[m] = T(0);
        dd[m] = T(1);
        if (row < row1) {
            rs[m] = rp[row];
            re[m] = rp[row + 1];
            rr[m] = r[row];
            xx[m] = x[row * ldx];
            pp[m] = pa[row];
            if (dinv) dd[m] = dinv[row];
        }
    }
    // the block's entries: staged once (the exchanges' fences empty L1, so
    // they would come from L2 in every iteration)
    const int e0 = rp[row0], cnt = rp[row1] - e0;
    T* mv = reinterpret_cast<T*>(stage_raw);
    int32_t* mc = reinterpret_cast<int32_t*>(mv + capacity);
    unsigned epoch = 0;
    // rows longer than the caller said: all blocks leave together, nothing
    // written
    T over[1] = {threadIdx.x == 0 && cnt > capacity ? T(1) : T(0)};
    if (!grid_exchange<T, 1>(over, slots, ++epoch, red, polls)) {
        if (threadIdx.x == 0) ctl->failed = 1;
        return;
    }
    if (over[0] != T(0)) {
        if (blockIdx.x == 0 && threadIdx.x == 0) ctl->failed = 2;
        return;
    }
    for (int e = threadIdx.x; e < cnt; e += kCgResidentBlock) {
        mv[e] = v[e0 + e];
        mc[e] = ci[e0 + e];
    }
#pragma unroll
    for (int m = 0; m < RPT; ++m) {
        rs[m] -= e0;
        re[m] -= e0;
    }
    __syncthreads();
    int iter = ctl->iter;
    const int max_iters = ctl->max_iters, last = iter + kCgResidentIters;
    SolveCtl crit;  // the criterion's fields, out of the loop
    crit.implicit = ctl->implicit;
    crit.reduction = ctl->reduction;
    uint8_t status = ctl->status[0];
    T rho = sc->rho[0], prev_rho = sc->prev_rho[0], tau = sc->tau[0];
    const T start = sc->start[0];
    while (!has_stopped(status) && iter < last) {
        const bool from_z = prev_rho == T(0);
        const T beta = from_z ? T(0) : rho / prev_rho;
        T pq[1] = {T(0)};
#pragma unroll
        for (int m = 0; m < RPT; ++m) {
            const int64_t row = first + m * step;
            T acc = T(0);
#pragma unroll 8
            for (int e = rs[m] + sub; e < re[m]; e += SW) {
                const int c = mc[e];
                const T d = dinv ? __ldg(dinv + c) : T(1);
                acc += mv[e] * cg_p(d, __ldcg(r + c), beta, __ldcg(pa + c), from_z);
            }
            acc = subwarp_sum<SW>(acc);
            pp[m] = cg_p(dd[m], rr[m], beta, pp[m], from_z);
            qq[m] = acc;
            if (row < row1 && sub == 0) {
                __stcg(pb + row, pp[m]);
                pq[0] += pp[m] * acc;
            }
        }
        if (!grid_exchange<T, 1>(pq, slots, ++epoch, red, polls)) {
            if (threadIdx.x == 0) ctl->failed = 1;
            return;
        }
        const T alpha = pq[0] != T(0) ? rho / pq[0] : T(0);
        T sums[2] = {T(0), T(0)};
#pragma unroll
        for (int m = 0; m < RPT; ++m) {
            const int64_t row = first + m * step;
            xx[m] += alpha * pp[m];
            rr[m] -= alpha * qq[m];
            if (row < row1 && sub == 0) {
                __stcg(r + row, rr[m]);
                sums[0] += rr[m] * mul_rn(dd[m], rr[m]);
                sums[1] += rr[m] * rr[m];
            }
        }
        if (!grid_exchange<T, 2>(sums, slots, ++epoch, red, polls)) {
            if (threadIdx.x == 0) ctl->failed = 1;
            return;
        }
        ++iter;
        prev_rho = rho;
        rho = sums[0];
        tau = sqrt(sums[1]);
        if (residual_met(&crit, tau, rho, start)) converge_status(status, kResidualId, true);
        if (iter >= max_iters) stop_status(status, kIterationId, true);
        T* t = pa;
        pa = pb;
        pb = t;
    }
#pragma unroll
    for (int m = 0; m < RPT; ++m) {
        const int64_t row = first + m * step;
        if (row < row1 && sub == 0) x[row * ldx] = xx[m];
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        // every block is past its reads of these: they precede the exchanges
        ctl->iter = iter;
        ctl->status[0] = status;
        ctl->all_stopped = has_stopped(status);
        sc->rho[0] = rho;
        sc->prev_rho[0] = prev_rho;
        sc->tau[0] = tau;
    }
}

// Blocks of the resident kernel, and its rows per thread with SW lanes per
// row (a block has at most ceil(n / blocks) rows).
inline int64_t cg_resident_blocks(int64_t n)
{
    return std::max<int64_t>(1, std::min<int64_t>(ceildiv(n, kWarp),
                                                  std::min(num_sms(), kExchangeBlocks)));
}
inline int64_t cg_resident_rpt(int64_t n, int sw)
{
    return ceildiv(ceildiv(n, cg_resident_blocks(n)) * sw, kCgResidentBlock);
}
// Shared memory a block may use for its matrix entries.
constexpr int64_t kCgStageBytes = 224 * 1024;
template <typename T>
int64_t cg_stage_bytes(int64_t n, int64_t max_row_nnz)
{
    return ceildiv(n, cg_resident_blocks(n)) * max_row_nnz * int64_t(sizeof(T) + 4);
}

// Runs the loop with the resident kernel; the host looks in between launches
// of kCgResidentIters iterations.
template <typename T>
int cg_resident_loop(int64_t n, const int32_t* rp, const int32_t* ci, const T* v, const T* dinv,
                     T* x, int64_t ldx, T* r, T* p0, T* p1, SolveCtl* ctl, CgScalars<T>* sc,
                     ExchangeSlot* slots, int64_t max_row_nnz, int max_iters, int polls,
                     cudaStream_t st, SolveCtl* host_ctl)
{
    // lanes per row while a block's rows still fit its threads: short rows
    // take all their gathers at once
    int sw = 1;
    while (sw < 8 && sw * 2 <= max_row_nnz && cg_resident_rpt(n, sw * 2) == 1) sw *= 2;
    const int64_t rpt = cg_resident_rpt(n, sw);
    const int64_t grid = cg_resident_blocks(n);
    const int64_t need = cg_stage_bytes<T>(n, max_row_nnz);
    using Kern = decltype(&cg_resident_kernel<T, 1, 1>);
    const Kern kernel = sw == 8    ? cg_resident_kernel<T, 8, 1>
                        : sw == 4  ? cg_resident_kernel<T, 4, 1>
                        : sw == 2  ? cg_resident_kernel<T, 2, 1>
                        : rpt == 1 ? cg_resident_kernel<T, 1, 1>
                        : rpt == 2 ? cg_resident_kernel<T, 1, 2>
                                   : cg_resident_kernel<T, 1, 4>;
    const size_t smem = size_t(need);
    B2S_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      int(kCgStageBytes)));
    int capacity = int(need / int64_t(sizeof(T) + 4));  // entries of a block's stage
    void* args[] = {&n,  &rp, &ci,  &v,  &dinv,  &x,       &ldx, &r,
                    &p0, &p1, &ctl, &sc, &slots, &capacity, &polls};
    const int64_t max_launches = int64_t(max_iters) / kCgResidentIters + 2;
    for (int64_t l = 0; l < max_launches; ++l) {
        B2S_CUDA_TRY(cudaMemsetAsync(slots, 0, kExchangeSlots * sizeof(ExchangeSlot), st));
        const cudaError_t e = cudaLaunchCooperativeKernel(
            reinterpret_cast<const void*>(kernel), dim3(unsigned(grid)), dim3(kCgResidentBlock),
            args, smem, st);
        if (e != cudaSuccess && l == 0) {
            (void)cudaGetLastError();
            return kCgNotResident;
        }
        B2S_CUDA_TRY(e);
        B2S_CUDA_TRY(cudaMemcpyAsync(host_ctl, ctl, sizeof(SolveCtl), cudaMemcpyDeviceToHost, st));
        B2S_CUDA_TRY(cudaStreamSynchronize(st));
        if (host_ctl->failed == 2) return kCgNotResident;
        if (host_ctl->failed) {
            set_error("CG: the blocks of the resident kernel did not meet");
            return B2S_ERR_CUDA;
        }
        if (host_ctl->all_stopped) break;
    }
    return B2S_OK;
}

// ---------------------------------------------------------------------------
// Block Jacobi: z = M^-1 r is no longer a row-wise scale, so it is stored.
// The SpMV passes above run with z in place of r and no diagonal
// (p' = z + beta p); the update pass below (and the initial one, INIT)
// runs one warp per group of the block-interleaved storage, lane (sub, i)
// owning row i of block sub of the group: r -= alpha q and x += alpha p'
// for the lane's row, then z of the row from the block's new residual,
// which the block's lanes pass along by shuffles (inverse columns in the
// order of apply_block, reference/preconditioner/jacobi_kernels.cpp:
// 419-445), and dot(r, z), ||r||^2.  INIT additionally zeroes p and sums
// ||b||^2 (cg::initialize and the first z = M r, core/solver/cg.cpp:
// 122-149).
// ---------------------------------------------------------------------------
// How the last block ends an iteration in the FP64 passes whose registers lie
// at the edge of two blocks per SM.  kInline is cg_update_finish in place.  In
// the forms below it pushed the pass past 128 registers, to one block, or into
// spills: out of line, with two blocks stated, or one thread walking the four
// columns leaves the pass at 128 (40 iterations, in line -> chosen: 7-point
// 64^3, blocks of 32 rows, 4 columns 4.08 -> 3.40 ms; 16 rows, 8 columns 4.84
// -> 4.37 ms; 5-point 1000^2, 16 rows of mixed precisions, 4 columns 6.72 ->
// 6.45 ms).
enum CgBlockTail { kInline, kOutOfLine, kOneThread };

template <typename T, int MB2, int K, bool INIT, int SK>
constexpr CgBlockTail cg_block_tail()
{
    if (INIT || sizeof(T) != 8) return kInline;
    if (K == 8 && (MB2 == 8 || (MB2 == 16 && SK == kSkFull))) return kOutOfLine;
    if (K == 4 && ((MB2 == 32 && SK == kSkFull) || (MB2 == 16 && SK == kSkMixed))) {
        return kOneThread;
    }
    return kInline;
}

template <typename T, int K>
__device__ __noinline__ void cg_block_end(const T* partials, T* tot, T* red, SolveCtl* ctl,
                                          CgScalars<T>* sc)
{
    sum_partials<T, 2 * K>(partials, gridDim.x, tot, red);
    if (threadIdx.x < kWarp) cg_update_finish<T, K>(tot, ctl, sc);
}

// cg_update_finish by one thread.
template <typename T, int K>
__device__ __forceinline__ void cg_update_finish_serial(const T* tot, SolveCtl* ctl,
                                                        CgScalars<T>* sc)
{
    ctl->ticket = 0;
    const int iter = ctl->iter + 1;
    ctl->iter = iter;
    int all = 1;
    for (int j = 0; j < K; ++j) {
        uint8_t s = ctl->status[j];
        if (!has_stopped(s)) {
            sc->prev_rho[j] = sc->rho[j];
            sc->rho[j] = tot[j];
            sc->tau[j] = sqrt(tot[K + j]);
            if (residual_met(ctl, sc->tau[j], sc->rho[j], sc->start[j])) {
                converge_status(s, kResidualId, true);
            }
            if (iter >= ctl->max_iters) stop_status(s, kIterationId, true);
            ctl->status[j] = s;
        }
        all &= has_stopped(s);
    }
    ctl->all_stopped = all;
}

// A fixed storage kind widens its loads in registers; holding those
// instances to five blocks per SM keeps them at the full-precision pass's 48
// registers (64 otherwise); a minimum of 0 leaves the others unconstrained.
template <typename T, int MB2, int K, bool INIT, int SK>
constexpr int cg_block_min_blocks()
{
    constexpr CgBlockTail tail = cg_block_tail<T, MB2, K, INIT, SK>();
    if (tail == kOutOfLine || (tail == kOneThread && SK == kSkFull)) return 2;
    return MB2 > 8 ? 0 : SK == kF16 ? 6 : SK >= 0 ? 5 : 0;
}

template <typename T, int MB2, int K, bool INIT, int SK>
__global__ void __launch_bounds__(kSolverBlock, (cg_block_min_blocks<T, MB2, K, INIT, SK>()))
    cg_block_kernel(int64_t n, BlockPrec<T> bp, const T* __restrict__ b, int64_t ldb, int k,
                    T* __restrict__ x, int64_t ldx, T* __restrict__ r, T* __restrict__ z,
                    T* __restrict__ p, const T* __restrict__ q, SolveCtl* ctl,
                    CgScalars<T>* sc, T* __restrict__ partials)
{
    constexpr int NS = INIT ? 3 : 2;  // sums per column
    constexpr unsigned kFull = 0xffffffffu;
    __shared__ T red[kSolverBlock / kWarp * NS * K];
    __shared__ T tot[NS * K];
    __shared__ int last;
    if (!INIT && ctl->all_stopped) return;
    bool active[K];
    T alpha[K];
#pragma unroll
    for (int j = 0; j < K; ++j) {
        active[j] = INIT || !has_stopped(ctl->status[j]);
        alpha[j] = INIT ? T(0) : sc->alpha[j];
    }
    T acc[NS * K];
#pragma unroll
    for (int j = 0; j < NS * K; ++j) acc[j] = T(0);
    const BlockScheme bsc = block_scheme(bp.max_bs);
    const int lane = threadIdx.x % kWarp;
    const int sub = lane / bp.max_bs, i = lane % bp.max_bs;
    const bool in_group = lane < bsc.gs * bp.max_bs;
    const int base = sub * bp.max_bs;  // first lane of this lane's block
    const int64_t ngroups = (bp.num_blocks + bsc.gs - 1) / bsc.gs;
    const int64_t nwarps = int64_t(gridDim.x) * (kSolverBlock / kWarp);
    for (int64_t grp = blockIdx.x * int64_t(kSolverBlock / kWarp) + threadIdx.x / kWarp;
         grp < ngroups; grp += nwarps) {
        const int64_t blk = grp * bsc.gs + sub;
        int s = 0, bs = 0;
        const bool in_block = in_group && blk < bp.num_blocks &&
                              block_extent(bp.ptrs, blk, n, bp.max_bs, s, bs);
        const bool act = in_block && i < bs;
        const int64_t row = s + i;
        BlockRow<SK, MB2, T> inv;
        inv.load(bp, bsc, grp, lane, in_group);
#pragma unroll
        for (int j = 0; j < K; ++j) {
            T rn = T(0);
            if (act) {
                if (INIT) {
                    rn = r[row * K + j];
                    p[row * K + j] = T(0);
                    const T bb = j < k ? b[row * ldb + j] : T(0);
                    acc[j] += bb * bb;
                } else if (active[j]) {
                    x[row * ldx + j] += alpha[j] * p[row * K + j];
                    rn = r[row * K + j] - alpha[j] * q[row * K + j];
                    r[row * K + j] = rn;
                }
            }
            if (!active[j]) continue;  // uniform: a frozen column keeps its z
            T zz = T(0);
#pragma unroll
            for (int c = 0; c < MB2; ++c) {
                if (c < bp.max_bs) {
                    const T rc = __shfl_sync(kFull, rn, (base + c) % kWarp);
                    if (act && c < bs) zz += inv[c] * rc;
                }
            }
            if (act) {
                z[row * K + j] = zz;
                acc[(NS - 2) * K + j] += rn * zz;
                acc[(NS - 1) * K + j] += rn * rn;
            }
        }
    }
    block_partials<T, NS * K>(acc, partials, red);
    if (last_block_done(&ctl->ticket, &last)) {
        constexpr CgBlockTail tail = cg_block_tail<T, MB2, K, INIT, SK>();
        if constexpr (tail == kOutOfLine) {
            cg_block_end<T, K>(partials, tot, red, ctl, sc);
        } else {
            sum_partials<T, NS * K>(partials, gridDim.x, tot, red);
            if constexpr (INIT) {
                if (threadIdx.x < kWarp) cg_init_finish<T, K>(tot, k, ctl, sc);
            } else if constexpr (tail == kOneThread) {
                if (threadIdx.x == 0) cg_update_finish_serial<T, K>(tot, ctl, sc);
            } else {
                if (threadIdx.x < kWarp) cg_update_finish<T, K>(tot, ctl, sc);
            }
        }
    }
}

// Launches cg_block_kernel for the block size class of bp.
template <typename T, int K, bool INIT>
void launch_cg_block(int64_t n, const BlockPrec<T>& bp, const T* b, int64_t ldb, int k, T* x,
                     int64_t ldx, T* r, T* z, T* p, const T* q, SolveCtl* ctl,
                     CgScalars<T>* sc, T* partials, cudaStream_t st)
{
    const BlockScheme bsc = block_scheme(bp.max_bs);
    const int64_t ngroups = ceildiv(bp.num_blocks, bsc.gs);
    const int grid = int(std::min<int64_t>(
        std::max<int64_t>(1, ceildiv(ngroups, kSolverBlock / kWarp)), solver_grid()));
    const int mb2 = kMaxBs / bsc.gs;
#define B2S_CG_BLOCK(MB)                                                           \
    case MB:                                                                       \
        with_pass_kind<T, K == 1>(bp, [&](auto sk) {                               \
            auto kernel = cg_block_kernel<T, MB, K, INIT, decltype(sk)::value>;    \
            kernel<<<pgrid(kernel, grid), kSolverBlock, 0, st>>>(                  \
                n, bp, b, ldb, k, x, ldx, r, z, p, q, ctl, sc, partials);          \
        });                                                                        \
        break;
    switch (mb2) {
        B2S_CG_BLOCK(2)
        B2S_CG_BLOCK(4)
        B2S_CG_BLOCK(8)
        B2S_CG_BLOCK(16)
        B2S_CG_BLOCK(32)
    default: B2S_CG_BLOCK(1)
    }
#undef B2S_CG_BLOCK
}

// Whether one column runs the resident kernel: four rows per thread at most
// (303,104 rows on 148 SMs) and the entries of a block's rows in its shared
// memory.  100 iterations, passes -> resident, us per iteration: 5-point 64^2
// 16.5 -> 8.0, 256^2 18.5 -> 8.8, 512^2 25.6 -> 13.1; 7-point 20^3 16.3 ->
// 10.4, 67^3 (the largest) 28.7 -> 16.6; 27-point 40^3 27.2 -> 12.5.  With the
// entries left in L2 the 27-point 64^3 system took 53.6 us against 38.4 in
// the split passes.
template <typename T>
bool cg_resident_ok(int64_t n, int64_t max_row_nnz)
{
    return n >= 1 && cg_resident_rpt(n, 1) <= 4 &&
           cg_stage_bytes<T>(n, max_row_nnz) <= kCgStageBytes;
}

// Whether K >= 4 columns run the split iteration.
inline bool cg_split_lanes(int64_t n, int K, int64_t max_row_nnz)
{
    const int64_t least = max_row_nnz > kRowsShort ? kCgSplitEntries / 8 : kCgSplitEntries;
    return n * K >= least && max_row_nnz >= 1 && max_row_nnz <= kRowsMaxLen;
}

struct CgLayout {
    int64_t bytes;
    int64_t off_ctl, off_sc, off_r, off_p0, off_p1, off_q, off_partials, off_z, off_slots;
};

// with_z: the stored z = M^-1 r of a block preconditioner
template <typename T>
CgLayout cg_layout(int64_t n, int K, bool with_z = false)
{
    Carver c{nullptr};
    CgLayout l;
    l.off_ctl = c.take<SolveCtl>(1);
    l.off_sc = c.take<CgScalars<T>>(1);
    l.off_r = c.take<T>(n * K);
    l.off_p0 = c.take<T>(n * K);
    l.off_p1 = c.take<T>(n * K);
    l.off_q = c.take<T>(n * K);
    l.off_partials = c.take<T>(int64_t(kSolverGrid) * 3 * K);
    l.off_z = with_z ? c.take<T>(n * K) : 0;
    l.off_slots = c.take<ExchangeSlot>(kExchangeSlots);
    l.bytes = c.used;
    return l;
}

// bp: a block Jacobi preconditioner (dinv then null), or null.  max_polls:
// the resident kernel's limit on a wait of its blocks
template <typename T>
int cg_solve(int64_t n, const int32_t* rp, const int32_t* ci, const T* v,
             int64_t max_row_nnz, const T* dinv, const BlockPrec<T>* bp, const T* b,
             int64_t ldb, T* x, int64_t ldx, int64_t k, int64_t max_iters, double reduction,
             int residual_mode, int64_t check_every, void* workspace,
             int64_t workspace_bytes,
             int64_t* iterations, double* residual_norms, uint8_t* status,
             void* stream, int64_t max_polls = kExchangePolls)
{
    B2S_CHECK_ARG(max_polls >= 0 && max_polls < (int64_t(1) << 31), "max_polls out of range");
    B2S_CHECK_ARG(n >= 0 && k >= 1 && k <= kMaxRhs, "num_rhs must be 1..16");
    B2S_CHECK_ARG(ldb >= k && ldx >= k, "leading dimension < num_rhs");
    B2S_CHECK_ARG(max_iters >= 0 && max_iters < (int64_t(1) << 30),
                  "max_iters out of range");
    B2S_CHECK_ARG(valid_residual_mode(residual_mode), "unknown residual mode %d",
                  residual_mode);
    if (bp) {
        B2S_CHECK_ARG(bp->max_bs >= 1 && bp->max_bs <= kMaxBs,
                      "max_block_size must be 1..32");
        B2S_CHECK_ARG(bp->num_blocks >= 1 && bp->ptrs && bp->blocks,
                      "block preconditioner without blocks");
    }
    const int K = rhs_bucket(k);
    const CgLayout lay = cg_layout<T>(n, K, bp != nullptr);
    if (workspace_bytes < lay.bytes) {
        set_error("workspace of %lld bytes < %lld", (long long)workspace_bytes,
                  (long long)lay.bytes);
        return B2S_ERR_WORKSPACE;
    }
    B2S_CHECK_ARG(workspace != nullptr && b && x && rp, "null pointer");
    cudaStream_t st = as_stream(stream);
    char* w = static_cast<char*>(workspace);
    auto* ctl = reinterpret_cast<SolveCtl*>(w + lay.off_ctl);
    auto* sc = reinterpret_cast<CgScalars<T>*>(w + lay.off_sc);
    T* r = reinterpret_cast<T*>(w + lay.off_r);
    T* p[2] = {reinterpret_cast<T*>(w + lay.off_p0),
               reinterpret_cast<T*>(w + lay.off_p1)};
    T* q = reinterpret_cast<T*>(w + lay.off_q);
    T* partials = reinterpret_cast<T*>(w + lay.off_partials);
    // block preconditioner: the SpMV passes read the stored z in place of r
    T* z = bp ? reinterpret_cast<T*>(w + lay.off_z) : nullptr;
    T* zr = bp ? z : r;

    SolveCtl h{};
    h.max_iters = int(max_iters);
    h.reduction = reduction;
    h.baseline = residual_mode & ~B2S_STOP_IMPLICIT;
    h.implicit = (residual_mode & B2S_STOP_IMPLICIT) != 0;
    B2S_CUDA_TRY(cudaMemcpyAsync(ctl, &h, sizeof(h), cudaMemcpyHostToDevice, st));
    const int sw = solver_subwarp(max_row_nnz);
    const int64_t row_blocks = std::max<int64_t>(1, ceildiv(n * sw, kSolverBlock));
    const int grid_spmv = int(std::min<int64_t>(row_blocks, solver_grid()));
    const int grid_vec = int(std::min<int64_t>(
        std::max<int64_t>(1, ceildiv(n, kSolverBlock)), solver_grid()));
    // iterations per replay, even; a solve of fewer records no more than it
    // runs (7-point 60^3, 4 columns, one iteration: 391 -> 339 us)
    const int64_t most = std::min<int64_t>(std::max<int64_t>(check_every, 1), max_iters);
    const int chunk = int(std::max<int64_t>(2, (most + 1) / 2 * 2));

    B2S_DISPATCH_RHS(K, {
        B2S_DISPATCH_SW(sw, {
            residual_kernel<T, SW, K><<<pgrid(residual_kernel<T, SW, K>, grid_spmv), kSolverBlock, 0, st>>>(
                n, rp, ci, v, x, ldx, b, ldb, int(k), r);
        });
        B2S_LAUNCH_CHECK();
        if (bp) {
            launch_cg_block<T, K, true>(n, *bp, b, ldb, int(k), x, ldx, r, z, p[0], nullptr,
                                        ctl, sc, partials, st);
        } else {
            cg_init_kernel<T, K><<<pgrid(cg_init_kernel<T, K>, grid_vec), kSolverBlock, 0, st>>>(
                n, dinv, b, ldb, int(k), r, p[0], ctl, sc, partials);
        }
        B2S_LAUNCH_CHECK();
    });
    // the split iteration: one column of a large system, or four and more
    // (16-byte column slices) whose rows are short enough for a warp to
    // walk 16 or 32 of them together
    const int lpr = async_lanes_per_row(max_row_nnz);
    const int64_t async_need = ceildiv(ceildiv(n, kWarp / lpr), kAsyncBlock / kWarp);
    const bool split1 = K == 1 && n >= kCgSplitRows;
    const bool split_k = K * int(sizeof(T)) >= 32 && cg_split_lanes(n, K, max_row_nnz);
    const bool split = split1 || split_k;
    auto launch_split = [&](auto kc, cudaStream_t cs) {
        constexpr int KC = decltype(kc)::value;
        constexpr int VW = CgSlice<T, KC>::VW;
        const bool xvec = VW == 1 || (k == KC && ldx * int64_t(sizeof(T)) % 16 == 0 &&
                                      reinterpret_cast<uintptr_t>(x) % 16 == 0);
        const int gv = int(std::min<int64_t>(
            std::max<int64_t>(1, ceildiv(n * KC / VW, kSolverBlock)), solver_grid()));
        T* xd = bp ? nullptr : x;
        cg_direction_kernel<T, KC><<<pgrid(cg_direction_kernel<T, KC>, gv), kSolverBlock, 0, cs>>>(
            n, dinv, zr, p[0], xd, ldx, xvec, ctl, sc);
        if constexpr (KC == 1) {
            CgDotEpilogue<T> epi{p[0], partials, ctl, sc};
            with_async_epi_kernel<T, CgDotEpilogue<T>>(lpr, [&](auto kernel) {
                const int64_t grid = std::min<int64_t>(
                    std::min<int64_t>(async_need, async_resident_blocks(kernel)), kSolverGrid);
                kernel<<<grid, kAsyncBlock, 0, cs>>>(n, rp, ci, v, p[0], q, &ctl->all_stopped,
                                                     epi);
            });
        } else {
            // 32 rows per warp where a row is at most two load steps and the
            // accumulators leave room (see rhs_rows_per_warp), else 16
            constexpr int KL = KC / VW;
            auto spmv = [&](auto rc) {
                constexpr int ROWS = decltype(rc)::value;
                auto kernel = cg_spmv_rows_kernel<T, KC, ROWS>;
                const int gs = int(std::min<int64_t>(
                    ceildiv(ceildiv(n, ROWS), kSolverBlock / kWarp), kSolverGrid));
                kernel<<<pgrid(kernel, gs), kSolverBlock, 0, cs>>>(n, rp, ci, v, p[0], q, ctl, sc,
                                                                   partials);
            };
            if (KL < 8 && max_row_nnz <= kRowsShort) {
                spmv(std::integral_constant<int, KL < 8 ? 32 : 16>());
            } else {
                spmv(std::integral_constant<int, 16>());
            }
        }
        if (bp) {
            launch_cg_block<T, KC, false>(n, *bp, nullptr, 0, int(k), x, ldx, r, z, p[0], q,
                                          ctl, sc, partials, cs);
        } else {
            cg_residual_kernel<T, KC><<<pgrid(cg_residual_kernel<T, KC>, gv), kSolverBlock, 0, cs>>>(
                n, dinv, r, q, ctl, sc, partials);
        }
    };
    auto capture = [&](cudaStream_t cs) -> int {
        for (int it = 0; it < chunk; ++it) {
            T* po = p[it % 2];
            T* pn = p[(it + 1) % 2];
            if (split) {
                B2S_DISPATCH_RHS(K, {
                    if constexpr (K == 1 || K * sizeof(T) >= 32) {
                        launch_split(std::integral_constant<int, K>(), cs);
                    }
                });
                B2S_LAUNCH_CHECK();
                continue;
            }
            B2S_DISPATCH_RHS(K, {
                if constexpr (K * sizeof(T) >= 32) {
                    // lanes own 16-byte column slices of a row
                    constexpr int VW = int(16 / sizeof(T));
                    constexpr int RPW = kWarp / (K / VW);
                    const int gs = int(std::min<int64_t>(
                        std::max<int64_t>(1, ceildiv(n, RPW * (kSolverBlock / kWarp))),
                        solver_grid()));
                    const int gu = int(std::min<int64_t>(
                        std::max<int64_t>(1, ceildiv(n * K / VW, kSolverBlock)), solver_grid()));
                    cg_spmv_lanes_kernel<T, K><<<pgrid(cg_spmv_lanes_kernel<T, K>, gs), kSolverBlock, 0, cs>>>(
                        n, rp, ci, v, dinv, zr, po, pn, q, ctl, sc, partials);
                    if (bp) {
                        launch_cg_block<T, K, false>(n, *bp, nullptr, 0, int(k), x, ldx, r, z,
                                                     pn, q, ctl, sc, partials, cs);
                    } else {
                        cg_update_lanes_kernel<T, K><<<pgrid(cg_update_lanes_kernel<T, K>, gu), kSolverBlock, 0, cs>>>(
                            n, dinv, x, ldx, r, pn, q, ctl, sc, partials);
                    }
                } else {
                    B2S_DISPATCH_SW(sw, {
                        cg_spmv_kernel<T, SW, K><<<pgrid(cg_spmv_kernel<T, SW, K>, grid_spmv), kSolverBlock, 0, cs>>>(
                            n, rp, ci, v, dinv, zr, po, pn, q, ctl, sc, partials);
                    });
                    if (bp) {
                        launch_cg_block<T, K, false>(n, *bp, nullptr, 0, int(k), x, ldx, r, z,
                                                     pn, q, ctl, sc, partials, cs);
                    } else {
                        cg_update_kernel<T, K><<<pgrid(cg_update_kernel<T, K>, grid_vec), kSolverBlock, 0, cs>>>(
                            n, dinv, x, ldx, r, pn, q, ctl, sc, partials);
                    }
                }
            });
            B2S_LAUNCH_CHECK();
        }
        return B2S_OK;
    };
    // the graph always runs an even number of iterations, so p[0] holds the
    // current direction at every replay boundary
    bool resident = K == 1 && !bp && cg_resident_ok<T>(n, max_row_nnz);
    int rc = B2S_OK;
    if (resident) {
        rc = cg_resident_loop<T>(n, rp, ci, v, dinv, x, ldx, r, p[0], p[1], ctl, sc,
                                 reinterpret_cast<ExchangeSlot*>(w + lay.off_slots),
                                 max_row_nnz, int(max_iters), int(max_polls), st, &h);
        resident = rc != kCgNotResident;
    }
    if (!resident) rc = run_graph_loop(st, ctl, int(max_iters), chunk, capture, &h);
    if (rc != B2S_OK) return rc;
    if (split && !bp && !resident) {
        B2S_DISPATCH_RHS(K, {
            const int gl = int(std::min<int64_t>(
                std::max<int64_t>(1, ceildiv(n * K, kSolverBlock)), solver_grid()));
            cg_last_step_kernel<T, K><<<gl, kSolverBlock, 0, st>>>(n, p[0], x, ldx, sc);
        });
        B2S_LAUNCH_CHECK();
    }
    CgScalars<T> hs;
    B2S_CUDA_TRY(cudaMemcpyAsync(&hs, sc, sizeof(hs), cudaMemcpyDeviceToHost, st));
    B2S_CUDA_TRY(cudaMemcpyAsync(&h, ctl, sizeof(h), cudaMemcpyDeviceToHost, st));
    B2S_CUDA_TRY(cudaStreamSynchronize(st));
    if (iterations) *iterations = h.iter;
    for (int64_t j = 0; j < k; ++j) {
        if (residual_norms) residual_norms[j] = double(hs.tau[j]);
        if (status) status[j] = h.status[j];
    }
    return B2S_OK;
}

}  // namespace
}  // namespace b2s

using namespace b2s;

extern "C" {

int64_t b2s_cg_workspace_bytes(int64_t num_rows, int64_t num_rhs,
                               int value_bytes)
{
    const int K = rhs_bucket(num_rhs);
    if (K < 0 || num_rows < 0) return -1;
    return value_bytes == 8 ? cg_layout<double>(num_rows, K).bytes
                            : cg_layout<float>(num_rows, K).bytes;
}

int64_t b2s_cg_block_workspace_bytes(int64_t num_rows, int64_t num_rhs,
                                     int value_bytes)
{
    const int K = rhs_bucket(num_rhs);
    if (K < 0 || num_rows < 0) return -1;
    return value_bytes == 8 ? cg_layout<double>(num_rows, K, true).bytes
                            : cg_layout<float>(num_rows, K, true).bytes;
}

#define B2S_CG_ENTRY(T, S)                                                    \
    int b2s_cg_solve_##S(int64_t num_rows, const int32_t* row_ptrs,           \
                         const int32_t* col_idxs, const T* values,            \
                         int64_t max_row_nnz, const T* inv_diag, const T* b,  \
                         int64_t ldb, T* x, int64_t ldx, int64_t num_rhs,     \
                         int64_t max_iters, double reduction_factor,          \
                         int residual_mode, int64_t check_every,              \
                         void* workspace,                                     \
                         int64_t workspace_bytes, int64_t* iterations,        \
                         double* residual_norms, uint8_t* status,             \
                         void* stream)                                        \
    {                                                                         \
        return cg_solve<T>(num_rows, row_ptrs, col_idxs, values, max_row_nnz, \
                           inv_diag, nullptr, b, ldb, x, ldx, num_rhs,        \
                           max_iters, reduction_factor, residual_mode,        \
                           check_every, workspace,                            \
                           workspace_bytes, iterations, residual_norms,       \
                           status, stream);                                   \
    }                                                                         \
    int b2s_cg_solve_waiting_##S(                                             \
        int64_t num_rows, const int32_t* row_ptrs, const int32_t* col_idxs,   \
        const T* values, int64_t max_row_nnz, const T* inv_diag, const T* b,  \
        int64_t ldb, T* x, int64_t ldx, int64_t num_rhs, int64_t max_iters,   \
        double reduction_factor, int residual_mode, int64_t check_every,      \
        void* workspace, int64_t workspace_bytes, int64_t* iterations,        \
        double* residual_norms, uint8_t* status, void* stream,                \
        int64_t max_polls)                                                    \
    {                                                                         \
        return cg_solve<T>(num_rows, row_ptrs, col_idxs, values, max_row_nnz, \
                           inv_diag, nullptr, b, ldb, x, ldx, num_rhs,        \
                           max_iters, reduction_factor, residual_mode,        \
                           check_every, workspace, workspace_bytes,           \
                           iterations, residual_norms, status, stream,        \
                           max_polls);                                        \
    }                                                                         \
    int b2s_cg_block_solve_##S(                                               \
        int64_t num_rows, const int32_t* row_ptrs, const int32_t* col_idxs,  \
        const T* values, int64_t max_row_nnz, int64_t num_blocks,            \
        const int32_t* block_ptrs, int max_block_size,                        \
        const uint8_t* block_precisions, const T* blocks,       \
        const T* b, int64_t ldb, T* x, int64_t ldx, int64_t num_rhs,          \
        int64_t max_iters, double reduction_factor, int residual_mode,        \
        int64_t check_every, void* workspace, int64_t workspace_bytes,        \
        int64_t* iterations, double* residual_norms, uint8_t* status,         \
        void* stream)                                                         \
    {                                                                         \
        BlockPrec<T> bp;                                                      \
        bp.num_blocks = num_blocks;                                           \
        bp.ptrs = block_ptrs;                                                 \
        bp.max_bs = max_block_size;                                           \
        bp.blocks = blocks;                                                   \
        bp.prec = block_precisions;                                           \
        if (bp.prec && workspace && workspace_bytes >= int64_t(sizeof(int))) { \
            /* the workspace's first word as scratch, before the solve */       \
            B2S_CUDA_TRY(resolve_storage_kind(bp, static_cast<int*>(workspace), \
                                              as_stream(stream)));        \
        }                                                                 \
        return cg_solve<T>(num_rows, row_ptrs, col_idxs, values, max_row_nnz, \
                           nullptr, &bp, b, ldb, x, ldx, num_rhs, max_iters,  \
                           reduction_factor, residual_mode, check_every,      \
                           workspace, workspace_bytes, iterations,            \
                           residual_norms, status, stream);                   \
    }

B2S_CG_ENTRY(double, f64)
B2S_CG_ENTRY(float, f32)

}  // extern "C"

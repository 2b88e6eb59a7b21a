// Sums over all blocks of a cooperative launch, the synchronisation of the
// solvers that keep a whole iteration loop inside one kernel.
#pragma once

#include "common.cuh"

namespace b2s {

// Blocks per exchange: one per SM.
constexpr int kExchangeBlocks = kMaxSMs;
// Polls after which a block gives up where the caller does not say (each
// takes a trip to L2, so this is on the order of a second); the kernel then
// reports the failure and ends.
constexpr int kExchangePolls = 1 << 21;

// A block's value and the exchange it belongs to, in two 8-byte words that
// are each written and read whole: a reader that finds the exchange's number
// in both words has the whole value, so one trip to L2 carries the arrival
// and the data.
struct __align__(16) ExchangeSlot {
    unsigned lo, epoch_lo, hi, epoch_hi;
};

constexpr int kExchangeShared = 2 * 32 + 4;

// Slots for exchanges of up to two values: exchange e uses buffer e % 2 (a
// block can be one exchange ahead of another, not two).
constexpr int64_t kExchangeSlots = int64_t(2) * 2 * (kExchangeBlocks + 1);

__device__ __forceinline__ void exchange_put(ExchangeSlot* s, double v, unsigned epoch)
{
    const unsigned long long b = __double_as_longlong(v);
    const unsigned long long e = static_cast<unsigned long long>(epoch) << 32;
    asm volatile("st.relaxed.gpu.global.b64 [%0], %1;" ::"l"(s), "l"((b & 0xffffffffull) | e)
                 : "memory");
    asm volatile("st.relaxed.gpu.global.b64 [%0], %1;" ::"l"(&s->hi), "l"((b >> 32) | e)
                 : "memory");
}

// The slot's value if it holds exchange `epoch`.
__device__ __forceinline__ bool exchange_get(const ExchangeSlot* s, unsigned epoch, double& v)
{
    unsigned long long a, b;
    asm volatile("ld.relaxed.gpu.global.b64 %0, [%1];" : "=l"(a) : "l"(s) : "memory");
    asm volatile("ld.relaxed.gpu.global.b64 %0, [%1];" : "=l"(b) : "l"(&s->hi) : "memory");
    v = __longlong_as_double((long long)((a & 0xffffffffull) | (b << 32)));
    return unsigned(a >> 32) == epoch && unsigned(b >> 32) == epoch;
}

__device__ __forceinline__ void exchange_fence() { asm volatile("fence.acq_rel.gpu;" ::: "memory"); }

// Adds M (1 or 2) values over every thread of every block; all threads get
// the totals, the same bits in every block (fixed order).  On return all
// global writes that any thread of the grid made before the call are visible
// to L2 reads (__ldcg) of every thread.  `epoch` counts the exchanges of the
// launch from 1; the slots are zero at launch.  False when a block did not
// arrive within `polls` polls: the caller ends the kernel.  Threads must be a
// multiple of 32, up to 1024, at least 64; red holds kExchangeShared values.
//
// Block 0 collects the values and publishes the total, so a waiting block
// polls one slot.  With every block polling all the others' slots (one hop
// less) the polls of 148 blocks met in the few L2 slices that hold the slots
// and an exchange took 4.5 to 5 us.
template <typename T, int M>
__device__ __forceinline__ bool grid_exchange(T (&v)[M], ExchangeSlot* slots, unsigned epoch,
                                              double* red, int polls)
{
    static_assert(M == 1 || M == 2, "one or two values");
    const int lane = threadIdx.x % kWarp, wid = threadIdx.x / kWarp;
    const int nw = blockDim.x / kWarp;
    double* tot = red + 2 * 32;
#pragma unroll
    for (int m = 0; m < M; ++m) {
        const T s = warp_sum(v[m]);
        if (lane == 0) red[m * 32 + wid] = double(s);
    }
    __syncthreads();
    if (wid < M) {
        T s = lane < nw ? T(red[wid * 32 + lane]) : T(0);
        s = warp_sum(s);
        ExchangeSlot* buf = slots + (int64_t(epoch % 2) * 2 + wid) * (kExchangeBlocks + 1);
        ExchangeSlot* total = buf + kExchangeBlocks;
        bool all = true;
        T sum = T(0);
        if (blockIdx.x != 0) {
            if (lane == 0) {
                // release the block's writes, which the barrier ordered before
                exchange_fence();
                exchange_put(buf + blockIdx.x, double(s), epoch);
                double got = 0.0;
                all = false;
                for (int poll = 0; poll < polls && !all; ++poll) {
                    all = exchange_get(total, epoch, got);
                }
                sum = T(got);
                exchange_fence();
            }
        } else {
            // block 0 collects: lane l the blocks l, l + 32, ...
            constexpr int kPer = (kExchangeBlocks + kWarp - 1) / kWarp;
            double got[kPer] = {};
            all = false;
            for (int poll = 0; poll < polls && !all; ++poll) {
                bool mine = true;
#pragma unroll
                for (int q = 0; q < kPer; ++q) {
                    const int b = lane + q * kWarp;
                    got[q] = 0.0;
                    if (b == 0) {
                        got[q] = double(s);
                    } else if (b < int(gridDim.x)) {
                        mine &= exchange_get(buf + b, epoch, got[q]);
                    }
                }
                all = __all_sync(0xffffffffu, mine);
            }
            // Every lane acquires the writes behind the slots it read (ahead
            // of the sum, which then runs beside the fence), and lane 0
            // releases them all with the total: shuffles and votes order no
            // memory between lanes, __syncwarp does.  CG on 5-point 256^2,
            // 710 iterations: 5.8 ms without that order, 6.0 with it.
            exchange_fence();
#pragma unroll
            for (int q = 0; q < kPer; ++q) sum += T(got[q]);
            sum = warp_sum(sum);
            __syncwarp();
            if (lane == 0 && all) {
                exchange_fence();
                exchange_put(total, double(sum), epoch);
            }
        }
        if (lane == 0) {
            tot[wid] = double(sum);
            tot[2 + wid] = all ? 1.0 : 0.0;
        }
    }
    __syncthreads();
    bool ok = true;
#pragma unroll
    for (int m = 0; m < M; ++m) {
        v[m] = T(tot[m]);
        ok = ok && tot[2 + m] != 0.0;
    }
    return ok;
}

}  // namespace b2s

// Grid-wide exchange of inner products for the persistent solvers: barrier and
// reduction in one, with bounded waits.
#pragma once

#include "pvof_device.cuh"
#include "pvof_kernels.cuh"

namespace pvof {

constexpr unsigned long long BARRIER_SPIN_LIMIT = 1ull << 26;   // polls of one wait

// Grid-wide sum and barrier in one: every block publishes its partial sums in
// a slot of its own, tagged with the number of the exchange (the epoch).  On
// at most 32 blocks every block polls all slots until they carry that tag; on
// more, the first does and publishes the totals in one more slot, which the
// other blocks poll (all blocks polling all slots crowds the few L2 lines the
// slots lie in).  One or two one-way trips through L2; a barrier that counts
// arrivals and a load of the partials behind it take three.  Measured, B200,
// us per exchange without and with PUBLISH: 9 blocks of 512 threads 0.97 and
// 1.9, counting barrier and partials 2.5; 227 blocks 2.1 and 3.2, every block
// polling 4.4 and 5.3, counting 6.3.
// A slot holds each double as two words of 32 value bits and the 32-bit
// epoch, so a word is valid by itself and the two need not arrive together.
// Two buffers alternate: a block writes epoch e + 2 only after it has the
// totals of e + 1, which need every block's e + 1, published after it read e.
// Both begin at the same place whatever NV is (slots are NV doubles apart
// inside), so an exchange of two sums right behind one of one sum does not
// write over slots that are still read.
// The host zeroes the slots before each launch; epochs start at 1.  The sums
// are taken in a fixed order (a tree in the block, then the blocks by lane), so
// every block has the same totals and runs repeat bit for bit.
// PUBLISH: the block's earlier stores to global memory are visible to every
// block after the exchange (else only the sums are exchanged): a fence before
// the block's slot is written, acquiring loads once a slot has been seen, and
// a fence in the first block before the totals.  False, in every thread of the block,
// when the bounded wait gave up.
struct Slots {
    unsigned long long *w;   // two buffers of nb + 1 slots of up to SLOT_SUMS sums
    int *error;
    unsigned nb, rank;       // blocks that exchange with one another, this block's number among them
    int code;                // what DevScalars::error says when a wait gives up
    unsigned epoch;
};

constexpr unsigned ALL_POLL_BLOCKS = 32;

__device__ __forceinline__ void slot_put(unsigned long long *p, double v, unsigned e)
{
    const unsigned long long x = (unsigned long long)__double_as_longlong(v), tag = (unsigned long long)e << 32;
    asm volatile("st.relaxed.gpu.global.v2.b64 [%0], {%1, %2};" ::"l"(p), "l"((x & 0xffffffffull) | tag), "l"((x >> 32) | tag)
                 : "memory");
}

// waits (bounded) for epoch e in slot p
template <bool ACQUIRE>
__device__ __forceinline__ bool slot_get(const unsigned long long *p, unsigned e, double &v, int *error, int code)
{
    unsigned long long lo, hi, spins = 0;
    for (;;) {
        asm volatile("ld.relaxed.gpu.global.v2.b64 {%0, %1}, [%2];" : "=l"(lo), "=l"(hi) : "l"(p) : "memory");
        if ((unsigned)(lo >> 32) == e && (unsigned)(hi >> 32) == e) break;
        ++spins;
        if ((spins & 1023ull) == 0 && (*(volatile int *)error != 0 || spins > BARRIER_SPIN_LIMIT)) {
            atomicCAS(error, 0, code);
            return false;
        }
        if (spins > 4096) __nanosleep(64);
    }
    if (ACQUIRE) {
        unsigned long long seen;
        asm volatile("ld.acquire.gpu.global.b64 %0, [%1];" : "=l"(seen) : "l"(p) : "memory");
    }
    v = __longlong_as_double((long long)((lo & 0xffffffffull) | (hi << 32)));
    return true;
}

template <int NV>
struct ExchangeSums {
    double wsum[32][NV], vals[NV][SLOT_BLOCKS], total[NV];
};
// one set per kernel and NV, whether PUBLISH or not (block barriers separate the
// uses of consecutive exchanges)
template <int NV>
__device__ __forceinline__ ExchangeSums<NV> &exchange_sums()
{
    __shared__ ExchangeSums<NV> s;
    return s;
}

template <int NV, bool PUBLISH>
__device__ __forceinline__ bool grid_exchange(Slots &sl, double (&v)[NV])
{
    ExchangeSums<NV> &S = exchange_sums<NV>();
    auto &wsum = S.wsum;
    auto &vals = S.vals;
    auto &total = S.total;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const unsigned nb = sl.nb, rank = sl.rank, e = ++sl.epoch;
    static_assert(NV <= SLOT_SUMS, "a slot buffer holds SLOT_SUMS sums per block");
    unsigned long long *buf = sl.w + (size_t)(e & 1u) * (nb + 1) * 2 * SLOT_SUMS;
    int good = 1;
#pragma unroll
    for (int n = 0; n < NV; n++)
        for (int o = 16; o > 0; o >>= 1) v[n] += __shfl_down_sync(0xffffffffu, v[n], o);
    if (lane == 0)
#pragma unroll
        for (int n = 0; n < NV; n++) wsum[warp][n] = v[n];
    __syncthreads();
    if (warp == 0) {
        double b[NV];
#pragma unroll
        for (int n = 0; n < NV; n++) {
            b[n] = lane < (int)(blockDim.x >> 5) ? wsum[lane][n] : 0.0;
            for (int o = 16; o > 0; o >>= 1) b[n] += __shfl_down_sync(0xffffffffu, b[n], o);
        }
        if (lane == 0) {
            if (PUBLISH) __threadfence();
#pragma unroll
            for (int n = 0; n < NV; n++) slot_put(buf + ((size_t)rank * NV + n) * 2, b[n], e);
        }
        __syncwarp();
    }
    if (nb <= ALL_POLL_BLOCKS) {
        if (warp == 0) {
#pragma unroll
            for (int n = 0; n < NV; n++) {
                double t = 0.0;
                if (lane < (int)nb && !slot_get<PUBLISH>(buf + ((size_t)lane * NV + n) * 2, e, t, sl.error, sl.code)) good = 0;
                for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
                if (lane == 0) total[n] = t;
            }
        }
    } else if (rank == 0) {
        for (unsigned q = threadIdx.x; q < nb; q += blockDim.x)
#pragma unroll
            for (int n = 0; n < NV; n++)
                if (!slot_get<PUBLISH>(buf + ((size_t)q * NV + n) * 2, e, vals[n][q], sl.error, sl.code)) good = 0;
        __syncthreads();
        if (warp == 0) {
            double t[NV];
#pragma unroll
            for (int n = 0; n < NV; n++) {
                t[n] = 0.0;
                for (unsigned q = lane; q < nb; q += 32) t[n] += vals[n][q];
                for (int o = 16; o > 0; o >>= 1) t[n] += __shfl_xor_sync(0xffffffffu, t[n], o);
            }
            if (lane == 0) {
                if (PUBLISH) __threadfence();
#pragma unroll
                for (int n = 0; n < NV; n++) {
                    slot_put(buf + ((size_t)nb * NV + n) * 2, t[n], e);
                    total[n] = t[n];
                }
            }
        }
    } else if (threadIdx.x == 0) {
#pragma unroll
        for (int n = 0; n < NV; n++)
            if (!slot_get<PUBLISH>(buf + ((size_t)nb * NV + n) * 2, e, total[n], sl.error, sl.code)) good = 0;
    }
    good = __syncthreads_and(good);
#pragma unroll
    for (int n = 0; n < NV; n++) v[n] = total[n];
    return good != 0;
}

}  // namespace pvof

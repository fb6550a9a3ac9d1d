// grid_sums.cuh -- sums over all blocks of a cooperative launch, with which the
// blocks also meet: the barrier of the one-launch iteration loops (tv.cu,
// wavelet.cu).
//
// A block stores its K partial sums and adds itself to a running count; one of
// its threads polls the count until every block of the round is in, and then
// every block takes all partials and adds them up in the same order, so the
// blocks agree on the sums to the last bit and none has to send them out again.
// (A flag per block that every block polls instead of the count saves the
// atomics' turns but floods L2: 512 blocks took 51 us a round against 14.)
// Partials are double buffered by the round's parity: a block can write round
// r + 2 only after every block has read round r.
//
// A wait gives up after two seconds, or as soon as another block's has; the
// caller then leaves its loop and the host reports the failure.
#pragma once

namespace ctprj {

constexpr unsigned long long kMeetNs = 2000000000ull;

struct GridMeet {
    unsigned *count;   // zero before the launch
    int *failed;       // zero before the launch
    double *part;      // 2 * K * blocks doubles, 16-byte aligned
};

template <int K, int THREADS>
struct GridSumsSmem {
    double red[K][THREADS / 32];
    double sum[K];
    int ok;
};

// v: this thread's share of the K sums (K even) of round `round` = 1, 2, ...;
// returns false when the meeting failed, else the sums over all blocks in v.
// Every thread of the block takes part; what the block wrote to global memory
// before is visible to the others after (read it past L1).
template <int K, int THREADS>
__device__ __forceinline__ bool grid_sums(const GridMeet &m, unsigned round, unsigned block, unsigned nblocks,
                                          double (&v)[K], GridSumsSmem<K, THREADS> &S)
{
    const int t = threadIdx.x;
    auto block_sums = [&]() {   // the warps' sums of v in S.red
#pragma unroll
        for (int k = 0; k < K; ++k) {
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) v[k] += __shfl_down_sync(0xffffffffu, v[k], o);
            if ((t & 31) == 0) S.red[k][t >> 5] = v[k];
        }
        __syncthreads();
    };
    block_sums();
    double *part = m.part + (size_t)K * nblocks * (round & 1);
    if (t == 0) {
#pragma unroll
        for (int k = 0; k < K; ++k) {
            double w = 0.0;
#pragma unroll
            for (int q = 0; q < THREADS / 32; ++q) w += S.red[k][q];
            __stcg(part + (size_t)K * block + k, w);
        }
        __threadfence();
        atomicAdd(m.count, 1u);
        const unsigned want = round * nblocks;
        unsigned long long t0 = 0, now;
        int ok = 1;
        for (unsigned n = 0;; ++n) {
            unsigned r;
            asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(r) : "l"(m.count) : "memory");
            if (r >= want) break;
            if ((n & 255) != 255) continue;   // a long wait: look at the clock
            asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(now));
            if (t0 == 0) t0 = now;
            if (*(volatile int *)m.failed || now - t0 > kMeetNs) {
                atomicExch(m.failed, 1);
                ok = 0;
                break;
            }
        }
        S.ok = ok;
    }
    __syncthreads();
    if (!S.ok) return false;
#pragma unroll
    for (int k = 0; k < K; ++k) v[k] = 0.0;
    for (unsigned b = t; b < nblocks; b += THREADS)
#pragma unroll
        for (int k = 0; k < K; k += 2) {
            const double2 u = __ldcg(reinterpret_cast<const double2 *>(part + (size_t)K * b + k));
            v[k] += u.x;
            v[k + 1] += u.y;
        }
    block_sums();
    if (t < K) {
        double w = 0.0;
#pragma unroll
        for (int q = 0; q < THREADS / 32; ++q) w += S.red[t][q];
        S.sum[t] = w;
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < K; ++k) v[k] = S.sum[k];
    return true;
}

}  // namespace ctprj

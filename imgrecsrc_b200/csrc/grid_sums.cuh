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
// A meeting is a chain of latencies (the fence, the count, the partials), about
// 4000 cycles, so it comes in steps between which a loop puts the work that does
// not wait for the sums:
//   sums_fold    the threads' sums to one per warp
//   __syncthreads
//   sums_post    the block's sums stored (warp 0)
//   __syncthreads, when more than the partials is to be visible to the others
//   sums_arrive  the block counted in
//   sums_wait    every block's sums and earlier writes visible (read them past L1)
//   sums_load    this thread's share of all blocks' sums
//   sums_fold, __syncthreads, sums_of_block   the sums over all blocks
// Every warp reads what was folded, so a buffer may be folded into again only
// after a barrier that follows the sums_post or sums_of_block that read it: the
// two folds of a round have a buffer each, and the other one's barriers lie
// between a buffer's uses.
// Rounds are 1, 2, ...  A wait gives up after two seconds, or as soon as another
// block's has; the block then leaves its loop without a result.  In the last round
// one block may give up while the others meet, so the host goes by the failure
// word as well as by the state that block 0 leaves (loop_met), and then takes the
// launch-per-iteration kernels, which wait for nothing.  A cooperative launch
// starts once there is room for all its blocks (beside a kernel that held half the
// GPU for four seconds the loops started when it ended, and met), so a wait runs
// out only where the whole GPU is taken from the program for that long.
#pragma once

namespace ctprj {

constexpr unsigned long long kMeetNs = 2000000000ull;

struct GridMeet {
    unsigned *count;   // zero before the launch
    int *failed;       // zero before the launch
    double *part;      // 2 * K * blocks doubles, 16-byte aligned
};

// Whether `count` arrivals, counted modulo 2^32, are the `want` = round * blocks of
// a round.  No block is more than one round ahead of another, so the two are less
// than 2^31 apart; their product passes 2^32 after some 7 million rounds.
__host__ __device__ inline bool all_in(unsigned count, unsigned want) { return (int)(count - want) >= 0; }

// whether a loop's result stands
inline bool loop_met(int done, int failed) { return done && !failed; }

// Launches a loop's blocks, all of them to be on the GPU at once.  started: false
// where the device has no room for that; the launch-per-iteration kernels need none.
inline int launch_loop(const void *kernel, dim3 grid, int threads, size_t smem, void **args, cudaStream_t s, bool *started)
{
    const cudaError_t e = cudaLaunchCooperativeKernel(kernel, grid, dim3(threads), args, smem, s);
    *started = e == cudaSuccess;
    if (e != cudaErrorCooperativeLaunchTooLarge) return cuda_error(e, "one-launch loop");
    cudaGetLastError();
    return CTPRJ_OK;
}

template <int K, int THREADS>
struct GridSumsSmem {
    double red[K][THREADS / 32];
    int ok;
};

// K = 2 or 4 sums per thread to one per warp: each halving of the lanes also
// halves the sums a lane carries on (6 exchanges for four sums, not 20); sum k in
// lanes k * 32 / K on
template <int K, int THREADS>
__device__ __forceinline__ void sums_fold(const double (&v)[K], GridSumsSmem<K, THREADS> &S)
{
    static_assert(K == 2 || K == 4, "two or four sums");
    const int lane = threadIdx.x & 31;
    const bool hi = lane & 16;
    double w;
    if constexpr (K == 4) {
        const double a = (hi ? v[2] : v[0]) + __shfl_xor_sync(0xffffffffu, hi ? v[0] : v[2], 16);
        const double b = (hi ? v[3] : v[1]) + __shfl_xor_sync(0xffffffffu, hi ? v[1] : v[3], 16);
        const bool h8 = lane & 8;
        w = (h8 ? b : a) + __shfl_xor_sync(0xffffffffu, h8 ? a : b, 8);
    } else {
        w = (hi ? v[1] : v[0]) + __shfl_xor_sync(0xffffffffu, hi ? v[0] : v[1], 16);
        w += __shfl_xor_sync(0xffffffffu, w, 8);
    }
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) w += __shfl_xor_sync(0xffffffffu, w, o);
    if (lane % (32 / K) == 0) S.red[lane / (32 / K)][threadIdx.x >> 5] = w;
}

// the sum over the warps of what they left in S.red: sum k in lanes k * 32 / K on
// (by all lanes of a warp)
template <int K, int THREADS>
__device__ __forceinline__ double sums_of_warps(const GridSumsSmem<K, THREADS> &S)
{
    constexpr int L = 32 / K;   // lanes per sum
    const int lane = threadIdx.x & 31;
    double w = 0.0;
#pragma unroll
    for (int q = 0; q < THREADS / 32; q += L)
        if (q + lane % L < THREADS / 32) w += S.red[lane / L][q + lane % L];
#pragma unroll
    for (int o = L / 2; o > 0; o >>= 1) w += __shfl_xor_sync(0xffffffffu, w, o);
    return w;
}

template <int K, int THREADS>
__device__ __forceinline__ void sums_post(const GridMeet &m, unsigned round, unsigned block, unsigned nblocks,
                                          const GridSumsSmem<K, THREADS> &S)
{
    if (threadIdx.x >= 32) return;
    const double w = sums_of_warps(S);
    if (threadIdx.x % (32 / K) == 0)
        __stcg(m.part + K * ((size_t)nblocks * (round & 1) + block) + threadIdx.x / (32 / K), w);
    __syncwarp();
}

__device__ __forceinline__ void sums_arrive(const GridMeet &m)
{
    if (threadIdx.x == 0)
        asm volatile("fence.acq_rel.gpu;\n\tred.relaxed.gpu.global.add.u32 [%0], 1;" ::"l"(m.count) : "memory");
}

// false when the meeting failed (the same in every thread of the block)
template <int K, int THREADS>
__device__ __forceinline__ bool sums_wait(const GridMeet &m, unsigned round, unsigned nblocks,
                                          GridSumsSmem<K, THREADS> &S)
{
    if (threadIdx.x == 0) {
        const unsigned want = round * nblocks;
        unsigned long long t0 = 0, now;
        int ok = 1;
        for (unsigned n = 0;; ++n) {
            unsigned r;
            asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(r) : "l"(m.count) : "memory");
            if (all_in(r, want)) break;
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
    return S.ok;
}

// this thread's share of every block's sums (one to three turns; unrolled, they
// would take more registers than the loops have left)
template <int K>
__device__ __forceinline__ void sums_load(const GridMeet &m, unsigned round, unsigned nblocks, double (&v)[K])
{
    const double *part = m.part + (size_t)K * nblocks * (round & 1);
#pragma unroll
    for (int k = 0; k < K; ++k) v[k] = 0.0;
#pragma unroll 1
    for (unsigned b = threadIdx.x; b < nblocks; b += blockDim.x)
#pragma unroll
        for (int k = 0; k < K; k += 2) {
            const double2 u = __ldcg(reinterpret_cast<const double2 *>(part + (size_t)K * b + k));
            v[k] += u.x;
            v[k + 1] += u.y;
        }
}

// the sums of the warps' folded ones, after a __syncthreads
template <int K, int THREADS>
__device__ __forceinline__ void sums_of_block(double (&v)[K], const GridSumsSmem<K, THREADS> &S)
{
    const double w = sums_of_warps(S);
#pragma unroll
    for (int k = 0; k < K; ++k) v[k] = __shfl_sync(0xffffffffu, w, k * (32 / K));
}

}  // namespace ctprj

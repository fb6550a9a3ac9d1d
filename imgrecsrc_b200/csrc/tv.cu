// tv.cu -- the total-variation proximal map of the density step on the GPU.
//
// The reference's 'tviso' / 'tvl1' regularisation (bhc/beamhardenSpline.m:
// 199-224) makes the density step's proximal map a bounded TV denoising,
//     min_X ||X - Xobs||^2 + 2 lambda TV(X)   subject to  lb <= X <= ub,
// solved by Beck and Teboulle's fast gradient projection on the dual
// (utils/denoise_bound_mod.m, after A. Beck, M. Teboulle, IEEE TIP 18(11),
// 2009): dual variables P = (P1, P2) on the vertical and horizontal pixel
// differences (utils/Ltrans.m, adjoint utils/Lforward.m), each iteration
//     C = Xobs - lambda L(R),  D = clamp(C),  P = proj(R + L^T(D) / (8 lambda)),
//     R = P + (t_k - 1)/t_{k+1} (P - P_old),
// with the reference's stopping rule (five consecutive relative changes of D
// below epsilon, or max_iter iterations) and its restart (t reset to 1 when the
// dual objective |C|^2 - |C - D|^2 rises).
//
// One fused kernel per iteration does the primal and the dual half on a
// 32 x 32 tile: it forms R = P + c (P - P_prev) on the tile and a one-pixel
// halo in shared memory, C = Xobs - lambda L(R) and D = clamp(C) on the tile
// plus its bottom row and right column, then the new P on the tile, with the
// FP64 partial sums the stopping rule needs.  Per pixel it reads Xobs, D_old,
// P and P_prev (float2 pairs of both components) and writes D and the new P:
// 36 bytes, no R image.  P is triple buffered (the new P cannot overwrite
// P_prev while neighbouring tiles still read its halo), D double buffered,
// both indexed by the device-side iteration counter.  The last block of each
// launch reduces the partials in a fixed order and advances the scalars
// (count, restart, t, the momentum coefficient, done), so every decision
// stays on the device; the host checks the done flag every eight
// iterations, and launches after convergence change nothing.  Images that fit
// the GPU's registers and shared memory take k_tv_loop instead, one launch that the
// host waits for once.
#include <algorithm>
#include <cmath>

#include "ctprj_internal.h"
#include "grid_sums.cuh"
#include "../../include/ctprj_tv.h"

namespace ctprj {

struct TvState {
    double tk;          // t of the coming iteration
    double c;           // momentum coefficient of the R the coming iteration forms
    double fold;        // dual objective of the last iteration
    int count;          // consecutive relative changes below epsilon
    int iter;           // completed iterations
    int done;
    unsigned arrived;   // blocks of the running iteration that have written their partials
};

// ws.buf: D (2 images), then the dual buffers 0, 1, 2, each an image of
// float2 (P1, P2) pairs
__host__ __device__ inline float *tv_d(float *buf, size_t px, int k) { return buf + px * (size_t)k; }
__host__ __device__ inline float2 *tv_p(float *buf, size_t px, int b)
{
    return reinterpret_cast<float2 *>(buf + px * (size_t)(2 + 2 * b));
}

struct TvArgs {
    const float *xobs;
    float *buf;
    size_t px;
    int m, n;          // rows, columns
    float lam, lb, ub;
    int iso;
    int max_iter;
    double eps;
    TvState *st;
    double *part;      // per-block partials, 4 per block
};

constexpr int kTvTile = 32;               // tile of kTvTile x kTvTile pixels
constexpr int kTvThreads = 256;           // 32 x 8 threads
constexpr int kTvValueRows = 8;           // rows per block of k_tv_value

__device__ __forceinline__ void block_sum4(double a[4], double *out)
{
    __shared__ double red[4][kTvThreads / 32];
    const int t = threadIdx.y * blockDim.x + threadIdx.x;
#pragma unroll
    for (int k = 0; k < 4; ++k)
        for (int o = 16; o > 0; o >>= 1) a[k] += __shfl_down_sync(0xffffffffu, a[k], o);
    if ((t & 31) == 0)
#pragma unroll
        for (int k = 0; k < 4; ++k) red[k][t >> 5] = a[k];
    __syncthreads();
    if (t == 0)
        for (int k = 0; k < 4; ++k) {
            double v = 0.0;
            for (int w = 0; w < kTvThreads / 32; ++w) v += red[k][w];
            out[k] = v;
        }
}

// The iteration's scalars from the summed partials: stopping count, restart,
// t, momentum coefficient, done.
// t_{k+1}, and in c the step of R = P + (t_k - 1) / t_{k+1} (P - P_old)
__device__ double tv_next_t(double tk, double &c)
{
    const double tkp1 = 0.5 * (1.0 + sqrt(1.0 + 4.0 * tk * tk));
    c = (tk - 1.0) / tkp1;
    return tkp1;
}

__device__ void tv_advance(TvState *st, const double s[4], int max_iter, double eps, double tkp1)
{
    const double re = sqrt(s[0]) / sqrt(s[1]);   // NaN for D = 0: not a small change
    st->count = re < eps ? st->count + 1 : 0;
    const double fval = s[3] - s[2];
    st->tk = fval > st->fold ? 1.0 : tkp1;     // restart when the dual objective rises
    st->fold = fval;
    st->iter += 1;
    if (st->count >= 5 || st->iter >= max_iter) st->done = 1;
}

// cp.async copies of 8 or 4 bytes into shared memory; src_size 0 (a tile cell
// outside the image) writes zeros and reads nothing
__device__ __forceinline__ void cp_async8(void *smem, const void *gmem, bool valid)
{
    const unsigned sa = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(sa), "l"(gmem), "r"(valid ? 8 : 0));
}
__device__ __forceinline__ void cp_async4(void *smem, const void *gmem, bool valid)
{
    const unsigned sa = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;\n" ::"r"(sa), "l"(gmem), "r"(valid ? 4 : 0));
}
// 16 bytes, the first `bytes` of them read (the rest zero); both addresses 16-byte aligned
__device__ __forceinline__ void cp_async16(void *smem, const void *gmem, int bytes)
{
    const unsigned sa = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(sa), "l"(gmem), "r"(bytes));
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::); }
__device__ __forceinline__ void cp_async_wait1() { asm volatile("cp.async.wait_group 1;\n" ::); }

// Shared-memory stage of one tile: P and P_prev on rows i0-1 .. i0+T and
// columns j0-2 .. j0+T+1 (float2 pairs; the extra column on each side keeps
// the 16-byte copies aligned), Xobs on rows i0 .. i0+T and columns
// j0 .. j0+T+3, D_old on the tile.  Cells outside the image are zero, which is
// what P, the difference operators and the clamped reads need there.
constexpr int kTvPR = kTvTile + 2, kTvPW = kTvTile + 4, kTvXR = kTvTile + 1, kTvXW = kTvTile + 4;
struct TvStage {
    float2 P[kTvPR][kTvPW];
    float2 Q[kTvPR][kTvPW];
    float X[kTvXR][kTvXW];
    float D[kTvTile][kTvTile];
};
struct TvSmem {
    TvStage st[2];
    float R1s[kTvTile + 2][kTvTile + 1];   // rows i0-1 .. i0+T, cols j0 .. j0+T
    float R2s[kTvTile + 1][kTvTile + 2];   // rows i0 .. i0+T, cols j0-1 .. j0+T
    float Ds[kTvTile + 1][kTvTile + 1];    // rows i0 .. i0+T, cols j0 .. j0+T
};

// 16-byte copies (two dual pairs or four floats) when a row starts 16-byte
// aligned (cols % 4 == 0), else 8- / 4-byte copies
template <bool VEC>
__device__ __forceinline__ void tv_stage_load(TvStage &S, const TvArgs &a, const float2 *P, const float2 *Q,
                                              const float *Dold, int i0, int j0, int t)
{
    constexpr int T = kTvTile;
    const int m = a.m, n = a.n;
    if (VEC) {
        for (int e = t; e < kTvPR * (kTvPW / 2); e += kTvThreads) {   // pairs of float2
            const int r = e / (kTvPW / 2), c = 2 * (e % (kTvPW / 2));
            const int i = i0 - 1 + r, j = j0 - 2 + c;
            const int cnt = (i >= 0 && i < m && j >= 0) ? max(0, min(2, n - j)) : 0;
            const int q = cnt ? i * n + j : 0;
            cp_async16(&S.P[r][c], P + q, 8 * cnt);
            cp_async16(&S.Q[r][c], Q + q, 8 * cnt);
        }
        for (int e = t; e < kTvXR * (kTvXW / 4); e += kTvThreads) {   // quads of floats
            const int r = e / (kTvXW / 4), c = 4 * (e % (kTvXW / 4));
            const int i = i0 + r, j = j0 + c;
            const int cnt = i < m ? max(0, min(4, n - j)) : 0;
            cp_async16(&S.X[r][c], a.xobs + (cnt ? i * n + j : 0), 4 * cnt);
        }
        for (int e = t; e < T * (T / 4); e += kTvThreads) {
            const int r = e / (T / 4), c = 4 * (e % (T / 4));
            const int i = i0 + r, j = j0 + c;
            const int cnt = i < m ? max(0, min(4, n - j)) : 0;
            cp_async16(&S.D[r][c], Dold + (cnt ? i * n + j : 0), 4 * cnt);
        }
        return;
    }
    for (int e = t; e < kTvPR * kTvPW; e += kTvThreads) {
        const int r = e / kTvPW, c = e % kTvPW;
        const int i = i0 - 1 + r, j = j0 - 2 + c;
        const bool v = i >= 0 && i < m && j >= 0 && j < n;
        const int q = v ? i * n + j : 0;
        cp_async8(&S.P[r][c], P + q, v);
        cp_async8(&S.Q[r][c], Q + q, v);
    }
    for (int e = t; e < kTvXR * kTvXW; e += kTvThreads) {
        const int r = e / kTvXW, c = e % kTvXW;
        const int i = i0 + r, j = j0 + c;
        const bool v = i < m && j < n;
        cp_async4(&S.X[r][c], a.xobs + (v ? i * n + j : 0), v);
    }
    for (int e = t; e < T * T; e += kTvThreads) {
        const int r = e / T, c = e % T;
        const int i = i0 + r, j = j0 + c;
        const bool v = i < m && j < n;
        cp_async4(&S.D[r][c], Dold + (v ? i * n + j : 0), v);
    }
}

// One FGP iteration.  Persistent blocks step through the kTvTile x kTvTile
// tiles; while a block computes one tile from a shared-memory stage, cp.async
// streams its next tile into the other stage, so the memory system stays
// busy across the compute phases.  Per tile: R = P + c (P - P_prev) on the
// tile and a one-pixel halo, C = Xobs - lambda L(R) and D = clamp(C) on the
// tile plus its bottom row and right column, then the new P on the tile.
// Thread (tx, ty) of the 32 x 8 block owns column tx of rows ty, ty + 8, ...
// The last block to finish sums every block's partials in a fixed order and
// advances the scalars, so an iteration is one launch.
template <bool VEC>
__global__ void __launch_bounds__(kTvThreads) k_tv_iter(const TvArgs a, int tiles_x, int ntiles)
{
    constexpr int T = kTvTile;
    extern __shared__ __align__(16) unsigned char tv_smem[];
    TvSmem &S = *reinterpret_cast<TvSmem *>(tv_smem);
    __shared__ bool last;
    TvState *st = a.st;
    if (st->done) return;
    const int it = st->iter;
    const float c = (float)st->c;
    const int m = a.m, n = a.n;
    const float2 *P = tv_p(a.buf, a.px, it % 3);          // P
    const float2 *Q = tv_p(a.buf, a.px, (it + 2) % 3);    // P_prev
    float2 *N = tv_p(a.buf, a.px, (it + 1) % 3);          // new P
    const float *Dold = tv_d(a.buf, a.px, it & 1);
    float *Dn = tv_d(a.buf, a.px, (it + 1) & 1);
    const int tx = threadIdx.x, ty = threadIdx.y, t = ty * 32 + tx;
    const float lam = a.lam, lb = a.lb, ub = a.ub, inv8l = 1.0f / (8.0f * lam);
    double s[4] = {0.0, 0.0, 0.0, 0.0};
    int tile = blockIdx.x, stage = 0;
    if (tile < ntiles) tv_stage_load<VEC>(S.st[0], a, P, Q, Dold, (tile / tiles_x) * T, (tile % tiles_x) * T, t);
    cp_async_commit();
    for (; tile < ntiles; tile += gridDim.x) {
        const int next = tile + gridDim.x;
        if (next < ntiles)
            tv_stage_load<VEC>(S.st[stage ^ 1], a, P, Q, Dold, (next / tiles_x) * T, (next % tiles_x) * T, t);
        cp_async_commit();
        cp_async_wait1();          // this tile's copies have landed (this thread's)
        __syncthreads();           // ... and every thread's
        const TvStage &G = S.st[stage];
        const int i0 = (tile / tiles_x) * T, j0 = (tile % tiles_x) * T;
        const int j = j0 + tx;
        // R on rows i0-1 .. i0+T (stage row r), columns j0-1 .. j0+T (stage
        // column cc + 1): R1 from column j0 + cc, R2 from column j0 - 1 + cc
        for (int e = t; e < (T + 2) * (T + 2); e += kTvThreads) {
            const int r = e / (T + 2), cc = e % (T + 2);
            const float2 p = G.P[r][cc + 1], q = G.Q[r][cc + 1];
            if (cc >= 1) S.R1s[r][cc - 1] = fmaf(c, p.x - q.x, p.x);
            if (r >= 1) S.R2s[r - 1][cc] = fmaf(c, p.y - q.y, p.y);
        }
        __syncthreads();
        // C = Xobs - lambda L(R), D = clamp(C) on the tile (partials) and its halo
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const int r = ty + 8 * k, i = i0 + r;
            if (i < m && j < n) {
                const float L = (S.R1s[r + 1][tx] - S.R1s[r][tx]) + (S.R2s[r][tx + 1] - S.R2s[r][tx]);
                const float C = fmaf(-lam, L, G.X[r][tx]);
                const float Dv = fminf(fmaxf(C, lb), ub);
                S.Ds[r][tx] = Dv;
                Dn[i * n + j] = Dv;
                const double dd = (double)Dv - (double)G.D[r][tx], cd = (double)C - (double)Dv;
                s[0] = fma(dd, dd, s[0]);
                s[1] = fma((double)Dv, (double)Dv, s[1]);
                s[2] = fma(cd, cd, s[2]);
                s[3] = fma((double)C, (double)C, s[3]);
            }
        }
        if (ty < 2) {   // the bottom row (warp 0) and the right column (warp 1)
            const int r = ty == 0 ? T : tx, cc = ty == 0 ? tx : T;
            if (i0 + r < m && j0 + cc < n) {
                const float L = (S.R1s[r + 1][cc] - S.R1s[r][cc]) + (S.R2s[r][cc + 1] - S.R2s[r][cc]);
                S.Ds[r][cc] = fminf(fmaxf(fmaf(-lam, L, G.X[r][cc]), lb), ub);
            }
        }
        __syncthreads();
        // P_new = proj(R + Ltrans(D) / (8 lambda)) on the tile
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const int r = ty + 8 * k, i = i0 + r;
            if (i < m && j < n) {
                const float d = S.Ds[r][tx];
                float p1 = i < m - 1 ? fmaf(d - S.Ds[r + 1][tx], inv8l, S.R1s[r + 1][tx]) : 0.0f;
                float p2 = j < n - 1 ? fmaf(d - S.Ds[r][tx + 1], inv8l, S.R2s[r][tx + 1]) : 0.0f;
                if (a.iso) {   // P / max(1, |P|): scaled only outside the unit ball
                    const float q2 = fmaf(p1, p1, p2 * p2);
                    if (q2 > 1.0f) {
                        const float rs = rsqrtf(q2);
                        p1 *= rs;
                        p2 *= rs;
                    }
                } else {
                    p1 = fminf(fmaxf(p1, -1.0f), 1.0f);
                    p2 = fminf(fmaxf(p2, -1.0f), 1.0f);
                }
                N[i * n + j] = make_float2(p1, p2);
            }
        }
        __syncthreads();           // the stage and the R / D tiles are free again
        stage ^= 1;
    }
    double out[4];
    block_sum4(s, out);
    const unsigned nblocks = gridDim.x;
    if (t == 0) {
        for (int k = 0; k < 4; ++k) a.part[4 * (size_t)blockIdx.x + k] = out[k];
        __threadfence();
        last = atomicAdd(&st->arrived, 1u) == nblocks - 1;
    }
    __syncthreads();
    if (!last) return;
    // the last block: sum the partials in a fixed order (thread t takes
    // blocks t, t + 256, ...; then a fixed tree), advance the scalars
    __threadfence();
    double v[4] = {0.0, 0.0, 0.0, 0.0};
    for (unsigned b = t; b < nblocks; b += kTvThreads)
#pragma unroll
        for (int k = 0; k < 4; ++k) v[k] += __ldcg(a.part + 4 * (size_t)b + k);
    double(*red)[kTvThreads] = reinterpret_cast<double(*)[kTvThreads]>(tv_smem);   // the stages are free now
#pragma unroll
    for (int k = 0; k < 4; ++k) red[k][t] = v[k];
    __syncthreads();
    for (int h = kTvThreads / 2; h > 0; h >>= 1) {
        if (t < h)
#pragma unroll
            for (int k = 0; k < 4; ++k) red[k][t] += red[k][t + h];
        __syncthreads();
    }
    if (t == 0) {
        const double tot[4] = {red[0][0], red[1][0], red[2][0], red[3][0]};
        const double tkp1 = tv_next_t(st->tk, st->c);
        tv_advance(st, tot, a.max_iter, a.eps, tkp1);
        st->arrived = 0;
    }
}

__global__ void k_tv_start(TvState *st, int done)
{
    st->tk = 1.0;
    st->c = 0.0;
    st->fold = INFINITY;
    st->count = 0;
    st->iter = 0;
    st->done = done;
    st->arrived = 0;
}

// ---- images that fit the GPU's registers and shared memory: one launch ----
// Up to about 1.2 million pixels every tile of the image has a block of its own
// on the GPU, so the whole iteration loop is one cooperative launch: a thread
// keeps the dual P of its eight pixels in registers (P_prev, too, or in shared
// memory), the tile's Xobs and D stay in shared memory, and per iteration a block
// reads only its halo of P and writes the edge of its new P.  The blocks meet once
// per iteration, at the sums of the stopping rule (grid_sums.cuh), after which every
// warp advances its own copy of the scalars: no host check, no second launch.
// What bounds an
// iteration is a chain of latencies, of which the meeting (fence, count, partials
// and halo from L2) is half; so a thread takes eight rows of one column, whose
// neighbours above and below are mostly its own, reads shared memory four pixels
// ahead of their use, posts its sums before the projection, works t out while
// it waits, and begins the next iteration's R before it takes the sums.  Nothing
// lies in local memory: what a thread keeps between iterations is its P, a word of
// bits that say where its pixels lie and a few indices.  (With the predicates and
// addresses kept as well the kernels had stack frames of 32 to 168 bytes.)  Per
// iteration, a launch each / this loop in the sums' order / with those frames / as
// it stands: 512^2 12.7 / 6.1 / 3.8 / 3.5 us, 768^2 - / 7.6 / 4.95 / 4.7, 1024^2
// 21 / 10.3 / 10.4 / 7.3.
constexpr int kTvpW = 64, kTvpPer = 8;                // tile columns, pixels per thread
constexpr int tvp_threads(int H) { return H * kTvpW / kTvpPer; }

template <int H>
struct TvpSmem {
    float R1[H + 2][kTvpW + 1];   // rows i0-1 .. i0+H, columns j0 .. j0+W
    float R2[H + 1][kTvpW + 2];   // rows i0 .. i0+H, columns j0-1 .. j0+W
    float D[H + 1][kTvpW + 1];    // rows i0 .. i0+H, columns j0 .. j0+W
    float X[H + 1][kTvpW + 1];
    GridSumsSmem<4, tvp_threads(H)> sums, taken;
    float2 hp[tvp_threads(H)], hq[tvp_threads(H)];   // each thread's halo cell: P and P of the iteration before
    TvState st[tvp_threads(H) / 32];                 // the scalars, a copy per warp
    double tkp1[tvp_threads(H) / 32];
};

template <bool ISO, int H, int PER_SM>
__global__ void __launch_bounds__(tvp_threads(H), PER_SM)
k_tv_loop(const TvArgs a, const GridMeet meet, float *__restrict__ out, int tiles_x)
{
    extern __shared__ __align__(16) unsigned char tv_smem[];
    TvpSmem<H> &S = *reinterpret_cast<TvpSmem<H> *>(tv_smem);
    constexpr int B = 4;   // pixels whose shared-memory reads are on their way together
    int t = threadIdx.x, tx = t % kTvpW, r0 = t / kTvpW * kTvpPer;   // the thread's pixels: (r0 + k, tx)
    const int i0 = (blockIdx.x / tiles_x) * H, j0 = (blockIdx.x % tiles_x) * kTvpW;
    const int m = a.m, n = a.n, j = j0 + tx;
    // bits of pixel k: k it lies in the image, 8 + k and not in its last row, 16 + k and
    // not in its last column, 24 + k and on the tile's edge, another block's halo
    unsigned at = 0;
    for (int k = 0; k < kTvpPer; ++k) {
        const int r = r0 + k, i = i0 + r;
        const bool in = i < m && j < n, edge = tx == 0 || tx == kTvpW - 1 || r == 0 || r == H - 1;
        at |= (in ? 1u << k : 0) | (in && i < m - 1 ? 0x100u << k : 0) | (in && j < n - 1 ? 0x10000u << k : 0) |
              (in && edge ? 0x1000000u << k : 0);
    }
    const float lam = a.lam, lb = a.lb, ub = a.ub, inv8l = 1.0f / (8.0f * lam);
    for (int e = t; e < (H + 1) * (kTvpW + 1); e += tvp_threads(H)) {
        const int r = e / (kTvpW + 1), c = e % (kTvpW + 1);
        S.X[r][c] = i0 + r < m && j0 + c < n ? a.xobs[(size_t)(i0 + r) * n + j0 + c] : 0.0f;
        S.D[r][c] = 0.0f;
    }
    // P of the thread's pixels, and Q: R until P is renewed, then the P before it.  Where
    // a thread has 64 registers, Q lies in the pixels' own places of R1 and R2, which no
    // other thread reads between the renewal and the next R.
    constexpr bool KEEP = PER_SM * tvp_threads(H) <= 512;
    float2 P[kTvpPer], Q[KEEP ? kTvpPer : 1];
    auto get_q = [&](int k) {
        if constexpr (KEEP) return Q[k];
        else return make_float2(S.R1[r0 + k + 1][tx], S.R2[r0 + k][tx + 1]);
    };
    auto set_q = [&](int k, float2 q) {
        if constexpr (KEEP) {
            Q[k] = q;
        } else {
            S.R1[r0 + k + 1][tx] = q.x;
            S.R2[r0 + k][tx + 1] = q.y;
        }
    };
#pragma unroll
    for (int k = 0; k < kTvpPer; ++k) {
        P[k] = make_float2(0.0f, 0.0f);
        set_q(k, P[k]);
    }
    // this thread's halo cell: the row above with the right corner, the row
    // below, the left column with the bottom corner, the right column
    int hr = 0, hc = 0;
    bool halo = true;
    if (t <= kTvpW) {
        hr = -1;
        hc = t;
    } else if (t <= 2 * kTvpW) {
        hr = H;
        hc = t - kTvpW - 1;
    } else if (t <= 2 * kTvpW + 1 + H) {
        hr = t - 2 * kTvpW - 1;
        hc = -1;
    } else if (t <= 2 * kTvpW + 1 + 2 * H) {
        hr = t - 2 * kTvpW - 2 - H;
        hc = kTvpW;
    } else {
        halo = false;
    }
    // its place in R1 (low half) and R2, 0xffff for none, and the pixel's in the image, -1
    const int hi = i0 + hr, hj = j0 + hc;
    unsigned hs = (halo && hc >= 0 ? (hr + 1) * (kTvpW + 1) + hc : 0xffff) |
                  (halo && hr >= 0 ? hr * (kTvpW + 2) + hc + 1 : 0xffff) << 16;
    int hx = halo && hi >= 0 && hi < m && hj >= 0 && hj < n ? hi * n + hj : -1, x0 = (i0 + r0) * n + j;
    S.hp[t] = S.hq[t] = make_float2(0.0f, 0.0f);
    const TvState &st = S.st[0];   // (every warp's copy says the same)
    if ((t & 31) == 0) {
        S.st[t >> 5] = {1.0, 0.0, INFINITY, 0, 0, a.max_iter <= 0, 0u};
        S.tkp1[t >> 5] = 1.0;
    }
    bool ok = true;
    __syncthreads();
    double s[4];
    for (unsigned round = 1; !st.done; ++round) {
        // what a thread keeps between rounds, not the predicates and addresses that follow
        // from these, which do not fit the registers
        asm volatile("" : "+r"(at), "+r"(hs), "+r"(hx), "+r"(x0), "+r"(t), "+r"(tx), "+r"(r0));
        TvState &own = S.st[t >> 5];
        double &tkp1 = S.tkp1[t >> 5];
        // c, which the sums of the last iteration do not decide (a restart tells
        // one iteration later), starts this one before they are taken
        const float c = (float)own.c;
        if (round > 1) sums_load(meet, round - 1, gridDim.x, s);
#pragma unroll
        for (int k = 0; k < kTvpPer; ++k) {
            float2 q = get_q(k);
            q.x = fmaf(c, P[k].x - q.x, P[k].x);
            q.y = fmaf(c, P[k].y - q.y, P[k].y);
            set_q(k, q);
            S.R2[r0 + k][tx + 1] = q.y;
            if (k == kTvpPer - 1) S.R1[r0 + k + 1][tx] = q.x;
        }
        // R on the halo
        const float2 hp = S.hp[t], hq = S.hq[t];
        if ((hs & 0xffff) != 0xffff) S.R1[0][hs & 0xffff] = fmaf(c, hp.x - hq.x, hp.x);
        if (hs >> 16 != 0xffff) S.R2[0][hs >> 16] = fmaf(c, hp.y - hq.y, hp.y);
        if (round > 1) sums_fold(s, S.taken);
        __syncthreads();
        if (round > 1) {
            sums_of_block(s, S.taken);
            if ((t & 31) == 0) tv_advance(&own, s, a.max_iter, a.eps, tkp1);
            __syncwarp();
            if (own.done) break;
        }
        // C = Xobs - lambda L(R), D = clamp(C) on the tile (partials) and its halo
        s[0] = s[1] = s[2] = s[3] = 0.0;
        float up = S.R1[r0][tx];
#pragma unroll
        for (int k0 = 0; k0 < kTvpPer; k0 += B) {
            float left[B], X[B], D[B];
#pragma unroll
            for (int k = 0; k < B; ++k) {
                left[k] = S.R2[r0 + k0 + k][tx];
                X[k] = S.X[r0 + k0 + k][tx];
                D[k] = S.D[r0 + k0 + k][tx];
            }
#pragma unroll
            for (int k = 0; k < B; ++k) {
                const float2 R = get_q(k0 + k);
                const bool in = at >> (k0 + k) & 1;
                const float C = in ? fmaf(-lam, (R.x - up) + (R.y - left[k]), X[k]) : 0.0f;
                up = R.x;
                const float Dv = in ? fminf(fmaxf(C, lb), ub) : 0.0f;
                S.D[r0 + k0 + k][tx] = Dv;
                const double dv = (double)Dv, dc = (double)C, dd = dv - (double)D[k], cd = dc - dv;
                s[0] = fma(dd, dd, s[0]);
                s[1] = fma(dv, dv, s[1]);
                s[2] = fma(cd, cd, s[2]);
                s[3] = fma(dc, dc, s[3]);
            }
        }
        if (t < kTvpW + H) {   // the bottom row and the right column
            const int r = t < kTvpW ? H : t - kTvpW, cc = t < kTvpW ? t : kTvpW;
            if (i0 + r < m && j0 + cc < n) {
                const float L = (S.R1[r + 1][cc] - S.R1[r][cc]) + (S.R2[r][cc + 1] - S.R2[r][cc]);
                S.D[r][cc] = fminf(fmaxf(fmaf(-lam, L, S.X[r][cc]), lb), ub);
            }
        }
        sums_fold(s, S.sums);
        __syncthreads();
        sums_post(meet, round, blockIdx.x, gridDim.x, S.sums);
        // P_new = proj(R + Ltrans(D) / (8 lambda)) on the tile
        float2 *N = tv_p(a.buf, a.px, round & 1);
        float d = S.D[r0][tx];
#pragma unroll
        for (int k0 = 0; k0 < kTvpPer; k0 += B) {
            float right[B], down[B];
#pragma unroll
            for (int k = 0; k < B; ++k) {
                right[k] = S.D[r0 + k0 + k][tx + 1];
                down[k] = S.D[r0 + k0 + k + 1][tx];
            }
#pragma unroll
            for (int k = 0; k < B; ++k) {
                const float2 R = get_q(k0 + k);
                float p1 = at >> (8 + k0 + k) & 1 ? fmaf(d - down[k], inv8l, R.x) : 0.0f;
                float p2 = at >> (16 + k0 + k) & 1 ? fmaf(d - right[k], inv8l, R.y) : 0.0f;
                d = down[k];
                if (ISO) {   // P / max(1, |P|): scaled only outside the unit ball
                    const float q2 = fmaf(p1, p1, p2 * p2), rs = rsqrtf(fmaxf(q2, 1.0f));
                    p1 = q2 > 1.0f ? p1 * rs : p1;
                    p2 = q2 > 1.0f ? p2 * rs : p2;
                } else {
                    p1 = fminf(fmaxf(p1, -1.0f), 1.0f);
                    p2 = fminf(fmaxf(p2, -1.0f), 1.0f);
                }
                set_q(k0 + k, P[k0 + k]);
                P[k0 + k] = make_float2(p1, p2);
                // only the tile's edge is another block's halo
                if (at >> (24 + k0 + k) & 1) __stcg(N + x0 + (k0 + k) * n, P[k0 + k]);
            }
        }
        __syncthreads();
        sums_arrive(meet);
        if ((t & 31) == 0) tkp1 = tv_next_t(own.tk, own.c);
        if (!(ok = sums_wait(meet, round, gridDim.x, S.sums))) break;
        S.hq[t] = S.hp[t];
        if (hx >= 0) S.hp[t] = __ldcg(N + hx);
    }
    if (!ok) return;
#pragma unroll
    for (int k = 0; k < kTvpPer; ++k)
        if (at >> k & 1) out[x0 + k * n] = S.D[r0 + k][tx];
    if (blockIdx.x == 0 && t == 0) {
        a.st->iter = st.iter;
        a.st->done = 1;
    }
}

// per-block partials of the TV of x (utils/tlv.m): block 32 x 8 over a
// 32-column, kTvValueRows-row strip
__global__ void __launch_bounds__(kTvThreads)
k_tv_value(const float *__restrict__ x, int m, int n, int iso, double *__restrict__ part)
{
    const int i = blockIdx.y * kTvValueRows + threadIdx.y, j = blockIdx.x * 32 + threadIdx.x;
    double s[4] = {0.0, 0.0, 0.0, 0.0};
    if (i < m && j < n) {
        const size_t q = (size_t)i * n + j;
        const double v = x[q];
        const double q1 = i < m - 1 ? v - (double)x[q + n] : 0.0;
        const double q2 = j < n - 1 ? v - (double)x[q + 1] : 0.0;
        s[0] = iso ? sqrt(q1 * q1 + q2 * q2) : fabs(q1) + fabs(q2);
    }
    double out[4];
    block_sum4(s, out);
    if (threadIdx.x == 0 && threadIdx.y == 0) part[(size_t)blockIdx.y * gridDim.x + blockIdx.x] = out[0];
}

__global__ void k_tv_sum(const double *__restrict__ part, int nblocks, double *__restrict__ out)
{
    sum_partials(part, nblocks, 1, 1, out);
}

static int tv_loop_tiles(int m, int n, int H = 32)
{
    return ((n + kTvpW - 1) / kTvpW) * ((m + H - 1) / H);
}

// the state, and the one-launch loop's failure word and count
constexpr size_t kTvStateBytes = sizeof(TvState) + 2 * sizeof(int);

int TvWorkspace::alloc(int m, int n, cudaStream_t s)
{
    if (buf && rows == m && cols == n) return CTPRJ_OK;
    release(s);
    const size_t px = (size_t)m * n;
    const size_t iter_blocks = (size_t)((n + kTvTile - 1) / kTvTile) * ((m + kTvTile - 1) / kTvTile);
    const size_t value_blocks = (size_t)((n + 31) / 32) * ((m + kTvValueRows - 1) / kTvValueRows);
    // the one-launch loop keeps the partials of two iterations
    const size_t loop_blocks = 2 * (size_t)tv_loop_tiles(m, n);
    blocks = (int)std::max(std::max(iter_blocks, value_blocks), loop_blocks);
    int st;
    if ((st = cuda_error(cudaMallocAsync((void **)&buf, sizeof(float) * px * 8, s), "TV buffers")) ||
        (st = cuda_error(cudaMallocAsync((void **)&part, sizeof(double) * 4 * (size_t)blocks, s), "TV partials")) ||
        (st = cuda_error(cudaMallocAsync((void **)&state, kTvStateBytes, s), "TV state"))) {
        release(s);
        return st;
    }
    rows = m;
    cols = n;
    return CTPRJ_OK;
}

void TvWorkspace::release(cudaStream_t s)
{
    if (buf) cudaFreeAsync(buf, s);
    if (part) cudaFreeAsync(part, s);
    if (state) cudaFreeAsync(state, s);
    buf = nullptr;
    part = nullptr;
    state = nullptr;
    rows = cols = 0;
}

// The loop's variant for an image.  Up to two 32-row tiles per SM a thread may
// take 128 registers; beyond, two blocks per SM of twice the rows meet sooner
// than four (1024^2: 7.3 us per iteration against 8.3, 1056^2 7.5 against 8.7),
// and those four are left for the sizes whose 64-row tiles would not all fit.
struct TvLoop {
    const void *kernel;
    int tiles, threads;
    size_t smem;
};

template <int H, int PER_SM>
static TvLoop tv_loop_variant(int m, int n, int iso)
{
    const void *kernel = iso ? (const void *)k_tv_loop<true, H, PER_SM> : (const void *)k_tv_loop<false, H, PER_SM>;
    return {kernel, tv_loop_tiles(m, n, H), tvp_threads(H), sizeof(TvpSmem<H>)};
}

static TvLoop tv_loop_of(int m, int n, int iso, int sms)
{
    if (tv_loop_tiles(m, n, 32) <= 2 * sms) return tv_loop_variant<32, 2>(m, n, iso);
    if (tv_loop_tiles(m, n, 64) <= 2 * sms) return tv_loop_variant<64, 2>(m, n, iso);
    return tv_loop_variant<32, 4>(m, n, iso);
}

int tv_denoise(TvWorkspace &ws, const float *xobs, int m, int n, double lambda, double lb, double ub,
               int iso, int max_iter, double eps, float *out, int *iterations, cudaStream_t s)
{
    int st;
    if ((st = ws.alloc(m, n, s))) return st;
    const size_t px = (size_t)m * n;
    TvArgs a;
    a.xobs = xobs;
    a.buf = ws.buf;
    a.px = px;
    a.m = m;
    a.n = n;
    a.lam = (float)lambda;
    a.lb = (float)lb;
    a.ub = std::isinf(ub) ? INFINITY : (float)ub;
    a.iso = iso;
    a.max_iter = max_iter;
    a.eps = eps;
    a.st = (TvState *)ws.state;
    a.part = ws.part;
    int dev = 0, sms = 148, per_sm = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    // every tile a block of its own on the GPU at once: the loop in one launch
    const TvLoop loop = tv_loop_of(m, n, iso, sms);
    if ((st = cuda_error(cudaFuncSetAttribute(loop.kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)loop.smem),
                         "TV shared memory")) ||
        (st = cuda_error(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, loop.kernel, loop.threads, loop.smem),
                         "TV occupancy")))
        return st;
    if (loop.tiles <= sms * per_sm) {
        struct {
            TvState st;
            int failed;
        } h{};
        // after the state: the failure word and the count of the meetings
        int *failed = (int *)(a.st + 1);
        GridMeet meet = {(unsigned *)(failed + 1), failed, ws.part};
        int tx = (n + kTvpW - 1) / kTvpW;
        void *args[] = {&a, &meet, &out, &tx};
        bool started = false;
        if ((st = cuda_error(cudaMemsetAsync(a.st, 0, kTvStateBytes, s), "TV start")) ||
            (st = launch_loop(loop.kernel, dim3(loop.tiles), loop.threads, loop.smem, args, s, &started)) ||
            (st = cuda_error(cudaMemcpyAsync(&h, a.st, sizeof h, cudaMemcpyDeviceToHost, s), "TV state")) ||
            (st = cuda_error(cudaStreamSynchronize(s), "TV state")))
            return st;
        if (started && loop_met(h.st.done, h.failed)) {
            if (iterations) *iterations = h.st.iter;
            return CTPRJ_OK;
        }
    }
    const int tiles_x = (n + kTvTile - 1) / kTvTile, ntiles = tiles_x * ((m + kTvTile - 1) / kTvTile);
    const dim3 block(32, kTvThreads / 32);
    const size_t smem = sizeof(TvSmem);
    // 16-byte aligned rows for the vector copies
    const bool vec = n % 4 == 0 && ((uintptr_t)xobs & 15) == 0;
    auto kern = vec ? k_tv_iter<true> : k_tv_iter<false>;
    if ((st = cuda_error(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem),
                         "TV shared memory")) ||
        (st = cuda_error(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, kTvThreads, smem),
                         "TV occupancy")))
        return st;
    const int grid = std::min(ntiles, sms * std::max(per_sm, 1));   // persistent blocks
    // D = 0 and P = P_prev = 0 (denoise_bound_mod starts from D = 0, whose
    // projected dual is P = 0, R = P)
    if ((st = cuda_error(cudaMemsetAsync(tv_d(ws.buf, px, 0), 0, sizeof(float) * px, s), "TV start")) ||
        (st = cuda_error(cudaMemsetAsync(tv_p(ws.buf, px, 0), 0, sizeof(float2) * px, s), "TV start")) ||
        (st = cuda_error(cudaMemsetAsync(tv_p(ws.buf, px, 2), 0, sizeof(float2) * px, s), "TV start")))
        return st;
    k_tv_start<<<1, 1, 0, s>>>(a.st, max_iter <= 0 ? 1 : 0);
    TvState h{};
    for (int it = 0; it < max_iter; ++it) {
        kern<<<grid, block, smem, s>>>(a, tiles_x, ntiles);
        if ((st = cuda_error(cudaGetLastError(), "TV iteration"))) return st;
        if ((it & 7) == 7 && it != max_iter - 1) {
            if ((st = cuda_error(cudaMemcpyAsync(&h, a.st, sizeof h, cudaMemcpyDeviceToHost, s), "TV state")) ||
                (st = cuda_error(cudaStreamSynchronize(s), "TV state")))
                return st;
            if (h.done) break;
        }
    }
    if ((st = cuda_error(cudaMemcpyAsync(&h, a.st, sizeof h, cudaMemcpyDeviceToHost, s), "TV state")) ||
        (st = cuda_error(cudaStreamSynchronize(s), "TV state")) ||
        (st = cuda_error(cudaMemcpyAsync(out, tv_d(ws.buf, px, h.iter & 1), sizeof(float) * px,
                                         cudaMemcpyDeviceToDevice, s), "TV result")))
        return st;
    if (iterations) *iterations = h.iter;
    return CTPRJ_OK;
}

int tv_value(TvWorkspace &ws, const float *x, int m, int n, int iso, double *d_out, cudaStream_t s)
{
    int st;
    if ((st = ws.alloc(m, n, s))) return st;
    const dim3 grid((n + 31) / 32, (m + kTvValueRows - 1) / kTvValueRows), block(32, kTvValueRows);
    k_tv_value<<<grid, block, 0, s>>>(x, m, n, iso, ws.part);
    k_tv_sum<<<1, 256, 0, s>>>(ws.part, (int)(grid.x * grid.y), d_out);
    return cuda_error(cudaGetLastError(), "TV value");
}

}  // namespace ctprj

using namespace ctprj;

extern "C" int ctprj_tv_denoise(const float *d_xobs, int rows, int cols, double lambda, double lb, double ub,
                                int tv_type, int max_iter, double epsilon, float *d_out, int *iterations,
                                void *stream)
{
    if (!d_xobs || !d_out) return set_error(CTPRJ_EINVAL, "NULL buffer");
    if (rows < 2 || cols < 2) return set_error(CTPRJ_EINVAL, "image of at least 2 x 2 pixels");
    if ((long long)rows * cols >= (1LL << 31)) return set_error(CTPRJ_EINVAL, "image of 2^31 pixels or more");
    if (!(lambda > 0.0)) return set_error(CTPRJ_EINVAL, "lambda must be positive");
    if (!(lb < ub)) return set_error(CTPRJ_EINVAL, "lower bound must be below the upper bound");
    if (tv_type != CTPRJ_TV_ISO && tv_type != CTPRJ_TV_L1) return set_error(CTPRJ_EINVAL, "unknown TV type");
    cudaStream_t s = (cudaStream_t)stream;
    TvWorkspace ws;
    int st = tv_denoise(ws, d_xobs, rows, cols, lambda, lb, ub, tv_type == CTPRJ_TV_ISO, max_iter, epsilon, d_out,
                        iterations, s);
    ws.release(s);
    return st;
}

extern "C" int ctprj_tv_value(const float *d_x, int rows, int cols, int tv_type, double *d_tv, void *stream)
{
    if (!d_x || !d_tv) return set_error(CTPRJ_EINVAL, "NULL buffer");
    if (rows < 1 || cols < 1) return set_error(CTPRJ_EINVAL, "empty image");
    if ((long long)rows * cols >= (1LL << 31)) return set_error(CTPRJ_EINVAL, "image of 2^31 pixels or more");
    if (tv_type != CTPRJ_TV_ISO && tv_type != CTPRJ_TV_L1) return set_error(CTPRJ_EINVAL, "unknown TV type");
    cudaStream_t s = (cudaStream_t)stream;
    TvWorkspace ws;
    int st = tv_value(ws, d_x, rows, cols, tv_type == CTPRJ_TV_ISO, d_tv, s);
    ws.release(s);
    return st;
}

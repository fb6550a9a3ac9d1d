// projector.cu -- forward projection and backprojection kernels for sm_100a.
//
// Both passes exploit the eight-fold symmetry of the square pixel grid under
// rotations by 90 degrees and reflections, exactly as the reference does
// (prj/cpuPrj.c:46-616): one footprint weight, computed for a base view, serves
// the eight mirrored (view, detector, pixel) triples.  That keeps the effective
// view angles of every output identical to the reference's (they are the
// base view's float-formed angle carried through exact symmetries) and divides
// the arithmetic per ray-pixel update by eight.
//
//  forward   one thread per base ray (view b <= prjFull/8, detector k), marching
//            down the image rows (ray-driven, prj/cpuPrj.c:319-616).  The eight
//            mirrored pixels of a pixel come from the plan's quad image (two
//            float4 per pixel, built at the start of each call), so that every
//            gather is a 16-byte load coalesced along x.
//  backward  one thread per pair of octant pixels 0 <= y <= x (pixel-driven,
//            prj/cpuPrj.c:46-317), looping over the base views and the
//            detectors under the pair's shadow, staged in shared memory; each
//            thread owns its sixteen output pixels, so no atomics are needed.
//
// Precision: the weights are FP32, but x cos R + y sin R - offset, which cancels
// to O(1) from terms of O(n), is formed in FP64 and then rounded: in the forward
// per row of a ray, in the unstaged backprojection per pixel and detector, in the
// staged one per 8 x 8 square and view, from where FP32 steps of a few units lead
// to the square's pixels and detectors.  That keeps the projections within
// 1e-7..1e-6 of the FP64 oracle, where the reference's own FP32 build is 1.5e-5
// off on signed inputs.
// The footprint itself is branch-free (footprint.cuh).
#include <cstdio>
#include <type_traits>

#include <cooperative_groups.h>

#include "ctprj_internal.h"
#include "footprint.cuh"
#include "row_parts.h"
#include "bhc_spline.cuh"

namespace ctprj {

// a forward block is kFwdViews adjacent base views x 32 adjacent rays, one view
// per warp: the warps march over nearly the same image lines at the same time,
// so the rows they gather are shared in L1.  CTPRJ_FWD_VIEWS and
// CTPRJ_FWD_MINBLOCKS (resident blocks asked of the register allocator) are
// build-time launch-shape choices, as is CTPRJ_BWD_MINBLOCKS for the staged
// backprojection.
#ifndef CTPRJ_FWD_VIEWS
#define CTPRJ_FWD_VIEWS 4
#endif
#ifndef CTPRJ_FWD_MINBLOCKS
#define CTPRJ_FWD_MINBLOCKS 5
#endif
#ifndef CTPRJ_BWD_MINBLOCKS
#define CTPRJ_BWD_MINBLOCKS 5
#endif
constexpr int kFwdViews = CTPRJ_FWD_VIEWS;
constexpr int kFwdThreads = 32 * kFwdViews;
constexpr int kBwdTile = 16;   // 16 x 16 octant pixels per block
// detectors of the staged backprojection (below): effectiveRate 1, below, above
enum { kBwdUnit = 0, kBwdNarrow = 1, kBwdRange = 2 };
constexpr int kBwdTablePad = 80;   // zero entries beyond the detectors at each end of a table row

// Each pass is two launches, a table of its input and the pass itself, of which
// the second may start while the first runs (programmatic dependent launch): the
// first lets it at once, the second prepares its geometry and waits for the
// first's end where it needs the table.  The first is an ordinary launch, so
// everything before it in the stream has ended.
__device__ __forceinline__ void let_next_start() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void wait_for_table() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

template <class... P, class... A>
static cudaError_t launch_after_table(void (*kern)(P...), dim3 grid, int threads, int cluster, cudaStream_t s, A... args)
{
    cudaLaunchConfig_t c = {};
    c.gridDim = grid;
    c.blockDim = dim3(threads);
    c.stream = s;
    cudaLaunchAttribute at[2];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    at[1].id = cudaLaunchAttributeClusterDimension;
    at[1].val.clusterDim.x = cluster;
    at[1].val.clusterDim.y = at[1].val.clusterDim.z = 1;
    c.attrs = at;
    c.numAttrs = cluster > 1 ? 2 : 1;
    return cudaLaunchKernelEx(&c, kern, args...);
}

// --------------------------------------------------------------- quad image

// The forward pass reads, for each pixel (x, y) a ray crosses, the eight images
// of (x, y) under the symmetries of the square.  The quad image holds them as
// two float4 per pixel: Q[yy][c] = {I(x, yy), I(x, -yy), I(yy, x), I(-yy, x)}
// for rows yy = 0..half and columns c = x + half, x = -half..half, where
// I(a, b) = img[(b + n/2) n + a + n/2]; (x, y) and (-x, y) give all eight.
// One 32 x 32 tile of Q: the I(yy, x) and I(-yy, x) components are image
// columns, staged through shared memory so that every global read is along a
// row.
__device__ __forceinline__ void quad_tile(const float *__restrict__ img, float4 *__restrict__ Q, int n,
                                          int tile, float (&tz)[32][33], float (&tw)[32][33])
{
    const int half = (n - 1) / 2, h2 = n / 2, QW = 2 * half + 1;
    const int tcols = (QW + 31) / 32;
    const int c0 = (tile % tcols) * 32, y0 = (tile / tcols) * 32;
    __syncthreads();
    // tz[i][j] = I(y0 + j, x_i), tw[i][j] = I(-(y0 + j), x_i) with x_i = c0 + i - half
    for (int i = threadIdx.y; i < 32; i += 8) {
        const int c = c0 + i, yy = y0 + threadIdx.x;
        if (c < QW && yy <= half) {
            const float *row = img + (size_t)(c - half + h2) * n + h2;
            tz[i][threadIdx.x] = row[yy];
            tw[i][threadIdx.x] = row[-yy];
        }
    }
    __syncthreads();
    for (int j = threadIdx.y; j < 32; j += 8) {
        const int c = c0 + threadIdx.x, yy = y0 + j;
        if (c < QW && yy <= half) {
            const int x = c - half;
            const float a = img[(size_t)(yy + h2) * n + x + h2];
            const float b = img[(size_t)(h2 - yy) * n + x + h2];
            Q[(size_t)yy * QW + c] = make_float4(a, b, tz[threadIdx.x][j], tw[threadIdx.x][j]);
        }
    }
}

__global__ void __launch_bounds__(256) k_quad(const float *__restrict__ img, float4 *__restrict__ Q, int n)
{
    __shared__ float tz[32][33], tw[32][33];
    let_next_start();
    quad_tile(img, Q, n, blockIdx.x, tz, tw);
}

int launch_quad(const float *img, float4 *Q, int n, cudaStream_t s)
{
    k_quad<<<quad_tiles(n), dim3(32, 8), 0, s>>>(img, Q, n);
    return cuda_error(cudaGetLastError(), "quad image launch");
}

// ----------------------------------------------------------------- forward

// Polychromatic epilogue of one sinogram entry (bhc/poissLAlpha.m:2-13 and
// bhc/gaussLAlpha.m:2-16 per ray): s = Ts * proj, BL(s) and dBL/ds over the
// spectrum (FP64), and the likelihood term; keeps s, r = df/dBL and
// r dBL/ds when asked.
__device__ __forceinline__ double bhc_entry(const BhcArgs &a, const double *tab,
                                            const double *Ie, float proj, size_t idx)
{
    const double s = a.Ts * (double)proj;
    const SplineEval e = b1_eval(s, tab, Ie, a.J);
    const double m = (double)__ldg(a.imea + idx);
    const RayTerms t = ray_terms(a.noise, e.BL, m);
    if (a.w_out) {
        a.w_out[idx] = (float)(t.r * e.sBL);
        a.s_out[idx] = (float)s;
        a.r_out[idx] = t.r;
    }
    return t.f;
}

__device__ __forceinline__ double block_sum(double v, double *red)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (lane == 0) red[warp] = v;
    __syncthreads();
    double t = 0.0;
    if (threadIdx.x == 0)
        for (int w = 0; w < (int)(blockDim.x >> 5); ++w) t += red[w];
    return t;
}

// Constants of forward ray (base view b, detector k): its direction
// (cos R, sin R) and offset from the isocentre, the pixel range of each row
// as xl(y) = Al - y Sl, xr(y) = Ar - y Sr -- the intersections of the two beam
// edges with the row's band (prj/cpuPrj.c:365-369 parallel, :514-536 fan) --
// the fan's magnified beam width bwc + (x sinT - y cosT) kbw, and the
// footprint with its per-pixel steps in ramp units.
struct FwdRay {
    double cR, sR, off;
    float Al, Sl, Ar, Sr;
    float cT, sT, bwc, kbw;
    FootprintV fp;
    float cRw, dhbw;
};

template <bool FAN>
__device__ __forceinline__ FwdRay fwd_ray(const FwdParams &p, int b, int k)
{
    const Geo &g = p.g;
    const double cT = p.view[b].c, sT = p.view[b].s;
    const DetEntry de = p.det[k];
    const double hbw = 0.5 * g.beamWidth;
    const double tl = de.t - hbw, tr = de.t + hbw;
    // every product-sum is an explicit fma, so that no kernel this is inlined
    // into contracts it differently: the batched and per-plan launches must
    // give the same bits
    double cR, sR, off, Al, Sl, Ar, Sr;
    float bwc = g.beamWidthF, kbw = 0.0f;
    if (FAN) {
        const double d = g.d;
        cR = fma(de.cB, cT, -(de.sB * sT));
        sR = fma(de.sB, cT, de.cB * sT);
        off = de.t * de.cB;   // d t / bq
        const double qxl = fma(tl, cT, d * sT), qyl = fma(-tl, sT, d * cT);
        const double qxr = fma(tr, cT, d * sT), qyr = fma(-tr, sT, d * cT);
        Al = fma(qxl > 0 ? -0.5 : 0.5, qxl, d * tl) / qyl;
        Sl = qxl / qyl;
        Ar = fma(qxr > 0 ? 0.5 : -0.5, qxr, d * tr) / qyr;
        Sr = qxr / qyr;
        const double bwcd = g.beamWidth * de.cB;
        bwc = (float)bwcd;
        kbw = (float)(bwcd / d);
    } else {
        cR = cT;
        sR = sT;
        off = de.t;
        Al = fma(-0.5, sT, tl) / cT;
        Sl = sT / cT;
        Ar = fma(0.5, sT, tr) / cT;
        Sr = Sl;
    }
    FwdRay r;
    r.cR = cR;
    r.sR = sR;
    r.off = off;
    r.Al = (float)Al;
    r.Sl = (float)Sl;
    r.Ar = (float)Ar;
    r.Sr = (float)Sr;
    r.cT = (float)cT;
    r.sT = (float)sT;
    r.bwc = bwc;
    r.kbw = kbw;
    const float dhb = FAN ? 0.5f * r.sT * kbw : 0.0f;   // half beam width step per pixel
    r.fp = make_footprint_v((float)cR, (float)sR);
    r.cRw = (float)cR * r.fp.iw;
    r.dhbw = dhb * r.fp.iw;
    return r;
}

// The rays of one forward block: V adjacent base views (one per warp) x 32
// adjacent detectors; block (bx, by) of the per-plan grid.  `part` of the rows
// (of p.rsplit) is summed by this thread: its warp's, or, with kAllParts, every
// part in turn, for the persistent launches.  The sums of the parts are added
// in their order either way.  Returns this thread's likelihood terms in
// polychromatic mode.
constexpr int kAllParts = -1;

// A quad image's entry.  NC: through the read-only path, which holds for data
// that nothing writes while the kernel runs; a kernel that starts beside the one
// that builds the image takes an ordinary load.
template <bool NC>
__device__ __forceinline__ float4 load_quad(const float4 *q)
{
    if constexpr (NC) return __ldg(q);
    else return *q;
}

// The rows of one part for one ray: S += the eight images' sums.  Row y reads
// the quad row |y|:
//   q[x] = {I(x, |y|), I(x, -|y|), I(|y|, x), I(-|y|, x)},
// so that for y >= 0 the eight sums take, per pixel x,
//   S0 += I(x, y), S6 += I(-x, y), S4 += I(x, -y), S2 += I(-x, -y),
//   S5 += I(y, x), S3 += I(y, -x), S1 += I(-y, x), S7 += I(-y, -x)
// from q[x] and q[-x]; for y < 0 the pairs of components swap.
// wcode: 3 / 4: window of 3 / 4 pixels; 5: bounded range loop (one for the warp).
template <bool FAN, int MODE, bool NC>
__device__ __forceinline__ void march_rows(const Geo &g, const FwdRay &ray, int wcode, int ytop, int ybot,
                                           const float4 *quad, float (&S)[8], unsigned long long &nz)
{
    const double cR = ray.cR, sR = ray.sR, off = ray.off;
    const float Alf = ray.Al, Slf = ray.Sl, Arf = ray.Ar, Srf = ray.Sr;
    const float cTf = ray.cT, sTf = ray.sT, bwc = ray.bwc, kbw = ray.kbw;
    const FootprintV fp = ray.fp;
    const float cRw = ray.cRw, dhbw = ray.dhbw;
    const int half = g.half;
    const int QW = 2 * half + 1;
    auto march_row = [&](const int y, const float4 *q, auto neg) {
        constexpr bool NEG = decltype(neg)::value;
        const float yf = (float)y;
        const float xl = fmaf(-yf, Slf, Alf), xr = fmaf(-yf, Srf, Arf);
        // nearest pixel to each edge; exact half-way ties (where the
        // reference rounds away from zero) only decide pixels whose
        // footprint just touches the beam edge, with weight zero; the
        // conversion saturates, so far-out edges clamp
        const int x0 = max(__float2int_rn(xl), -half);
        const int x1 = min(__float2int_rn(xr), half);
        if (x0 > x1) return;
        // distance of pixel (x0, y) from the ray, in FP64 then rounded;
        // distances and half beam widths in units of the footprint's ramp
        const float r0 = (float)fma((double)x0, cR, fma((double)y, sR, -off)) * fp.iw;
        const float hb0 = (FAN ? 0.5f * fmaf(fmaf((float)x0, sTf, -yf * cTf), kbw, bwc)
                               : 0.5f * g.beamWidthF) * fp.iw;
        auto accumulate = [&](const float w, const float4 pp, const float4 pm) {
            const float ap = NEG ? pp.y : pp.x, am = NEG ? pm.y : pm.x;   // I(+-x, y)
            const float bp = NEG ? pp.x : pp.y, bm = NEG ? pm.x : pm.y;   // I(+-x, -y)
            const float cp = NEG ? pp.w : pp.z, cm = NEG ? pm.w : pm.z;   // I(y, +-x)
            const float dp = NEG ? pp.z : pp.w, dm = NEG ? pm.z : pm.w;   // I(-y, +-x)
            S[0] = fmaf(w, ap, S[0]);
            S[6] = fmaf(w, am, S[6]);
            S[4] = fmaf(w, bp, S[4]);
            S[2] = fmaf(w, bm, S[2]);
            S[5] = fmaf(w, cp, S[5]);
            S[3] = fmaf(w, cm, S[3]);
            S[1] = fmaf(w, dp, S[1]);
            S[7] = fmaf(w, dm, S[7]);
        };
        // Pixel x0 + j sits at D = fma(j, cRw, r0) (j even) or that of
        // j - 1 plus cRw (j odd), and likewise for H.  At unit beam width
        // a ray crosses one to three pixels of a row below 37 degrees of
        // obliquity and two to four above, so one straight-line step takes
        // the first three pixels, their gathers issued together and each
        // predicated on the pixel being in the run (a lane past its run
        // sends no request), and single steps the rest; per sum the order
        // of the terms is x0, x0 + 1, ...
        auto coef = [&](const int j, float &D, float &H) {
            const float je = (float)(j & ~1);
            D = fmaf(je, cRw, r0);
            H = FAN ? fmaf(je, dhbw, hb0) : hb0;
            if (j & 1) {
                D += cRw;
                if (FAN) H += dhbw;
            }
        };
        {
            const bool p1 = x0 < x1, p2 = x0 + 1 < x1;
            float D0, H0, D1, H1, D2, H2;
            coef(0, D0, H0);
            coef(1, D1, H1);
            coef(2, D2, H2);
            if (MODE == kModeCount) {
                nz += (footprint_weight_v(D0, H0, fp) != 0.0f);
                if (p1) nz += (footprint_weight_v(D1, H1, fp) != 0.0f);
                if (p2) nz += (footprint_weight_v(D2, H2, fp) != 0.0f);
            } else {
                const float4 pp0 = load_quad<NC>(q + x0), pm0 = load_quad<NC>(q - x0);
                float4 pp1 = {}, pm1 = {}, pp2 = {}, pm2 = {};
                if (p1) {
                    pp1 = load_quad<NC>(q + x0 + 1);
                    pm1 = load_quad<NC>(q - x0 - 1);
                }
                if (p2) {
                    pp2 = load_quad<NC>(q + x0 + 2);
                    pm2 = load_quad<NC>(q - x0 - 2);
                }
                accumulate(footprint_weight_v(D0, H0, fp), pp0, pm0);
                if (p1) accumulate(footprint_weight_v(D1, H1, fp), pp1, pm1);
                if (p2) accumulate(footprint_weight_v(D2, H2, fp), pp2, pm2);
            }
        }
        for (int x = x0 + 3; x <= x1; ++x) {
            float D, H;
            coef(x - x0, D, H);
            if (MODE == kModeCount) {
                nz += (footprint_weight_v(D, H, fp) != 0.0f);
                continue;
            }
            accumulate(footprint_weight_v(D, H, fp), load_quad<NC>(q + x), load_quad<NC>(q - x));
        }
    };
    // The fixed-window march (plain and polychromatic modes).  Where a
    // ray's run across a row is always narrower than 1.95 (2.95) pixels,
    // the pixels of the run lie within the 3 (4) centred on the ray's
    // crossing xc = (xl + xr) / 2: they are summed straight, without the
    // run's bounds.  A pixel of the window outside the run lies beyond
    // the beam and adds a weight of exactly zero (for fan beams: below
    // 1e-7 within ~1e-4 pixel of a run edge, where the footprint and the
    // beam edges differ).  The window is chosen per warp (the widest any
    // of its rays needs), so the warp stays converged.
    const float Acf = 0.5f * (Alf + Arf), Scf = 0.5f * (Slf + Srf);
    auto march_win = [&](const int y, const float4 *q, auto neg, auto wn) {
        constexpr bool NEG = decltype(neg)::value;
        constexpr int WN = decltype(wn)::value;
        const float yf = (float)y;
        const float xc = fmaf(-yf, Scf, Acf);
        // rows whose run misses the image (the run lies within xc +- 1.5)
        if (xc < -(float)half - 2.0f || xc > (float)half + 2.0f) return;
        int xs = (WN == 3 ? __float2int_rn(xc) : __float2int_rd(xc)) - 1;
        xs = min(max(xs, -half), half - (WN - 1));
        const float r0 = (float)fma((double)xs, cR, fma((double)y, sR, -off)) * fp.iw;
        const float hb0 = (FAN ? 0.5f * fmaf(fmaf((float)xs, sTf, -yf * cTf), kbw, bwc)
                               : 0.5f * g.beamWidthF) * fp.iw;
        float4 pp[WN], pm[WN];
#pragma unroll
        for (int j = 0; j < WN; ++j) {
            pp[j] = load_quad<NC>(q + xs + j);
            pm[j] = load_quad<NC>(q - xs - j);
        }
#pragma unroll
        for (int j = 0; j < WN; ++j) {
            const float D = fmaf((float)j, cRw, r0);
            const float H = FAN ? fmaf((float)j, dhbw, hb0) : hb0;
            const float w = footprint_weight_v(D, H, fp);
            const float ap = NEG ? pp[j].y : pp[j].x, am = NEG ? pm[j].y : pm[j].x;
            const float bp = NEG ? pp[j].x : pp[j].y, bm = NEG ? pm[j].x : pm[j].y;
            const float cp = NEG ? pp[j].w : pp[j].z, cm = NEG ? pm[j].w : pm[j].z;
            const float dp = NEG ? pp[j].z : pp[j].w, dm = NEG ? pm[j].z : pm[j].w;
            S[0] = fmaf(w, ap, S[0]);
            S[6] = fmaf(w, am, S[6]);
            S[4] = fmaf(w, bp, S[4]);
            S[2] = fmaf(w, bm, S[2]);
            S[5] = fmaf(w, cp, S[5]);
            S[3] = fmaf(w, cm, S[3]);
            S[1] = fmaf(w, dp, S[1]);
            S[7] = fmaf(w, dm, S[7]);
        }
    };
    const float4 *q = quad + (size_t)max(ytop, 0) * QW + half;   // row |y|, x = 0
    const int ypos = max(ybot, 0), yneg = min(ytop, -1);
    if (wcode == 3) {
        for (int y = ytop; y >= ypos; --y, q -= QW)
            march_win(y, q, std::false_type{}, std::integral_constant<int, 3>{});
    } else if (wcode == 4) {
        for (int y = ytop; y >= ypos; --y, q -= QW)
            march_win(y, q, std::false_type{}, std::integral_constant<int, 4>{});
    } else {
        for (int y = ytop; y >= ypos; --y, q -= QW) march_row(y, q, std::false_type{});
    }
    q = quad + (size_t)(-yneg) * QW + half;
    if (wcode == 3) {
        for (int y = yneg; y >= ybot; --y, q += QW)
            march_win(y, q, std::true_type{}, std::integral_constant<int, 3>{});
    } else if (wcode == 4) {
        for (int y = yneg; y >= ybot; --y, q += QW)
            march_win(y, q, std::true_type{}, std::integral_constant<int, 4>{});
    } else {
        for (int y = yneg; y >= ybot; --y, q += QW) march_row(y, q, std::true_type{});
    }
}

// The rows that the rays of a warp can meet (row_parts.h).  Every lane of the
// warp takes part, lanes without a ray with no rows.
__device__ __forceinline__ RowRange warp_rows(const FwdRay &ray, bool live, int half)
{
    const RowRange r = live ? ray_rows(0.5f * (ray.Al + ray.Ar), 0.5f * (ray.Sl + ray.Sr), half) : no_rows(half);
    return {__reduce_min_sync(0xffffffffu, r.bottom), __reduce_max_sync(0xffffffffu, r.top)};
}

// Stores image j's sum of ray (view b, detector k), scaled, or takes it through
// the polychromatic epilogue: to its sinogram row and detector, and for
// parallel beam to the point-reflected detector of the view that image j ^ 2
// belongs to (prj/cpuPrj.c:403-460), which is the one kept where the two
// coincide (the central detector).  Returns the likelihood terms.
template <bool FAN, int MODE>
__device__ __forceinline__ double put_image(const FwdParams &p, int b, int k, int j, float sum,
                                            float *__restrict__ sino, const double *tab, const double *Ie)
{
    const Geo &g = p.g;
    const int det = j < 4 ? k : 2 * g.pC - k, det2 = 2 * g.pC - det;
    const int v = p.view[b].out[j], v2 = FAN ? -1 : p.view[b].out[j ^ 2];
    const float val = sum / g.effRate;
    double f = 0.0;
    auto put = [&](size_t idx) {
        if constexpr (MODE == kModeBhc) {
            f += bhc_entry(p.bhc, tab, Ie, val, idx);
            if (p.bhc.proj_out) p.bhc.proj_out[idx] = val;
        } else {
            sino[idx] = val;
        }
    };
    if (v >= 0 && (FAN || det2 != det)) put((size_t)v * g.W + det);
    if (!FAN && v2 >= 0) put((size_t)v2 * g.W + det2);
    return f;
}

template <bool FAN, int MODE, int V, int R>
__device__ __forceinline__ double forward_rays(const FwdParams &p, int bx, int by, const float4 *quad,
                                               float *__restrict__ sino, unsigned long long *__restrict__ counter,
                                               const double *tab, const double *Ie, float *parts)
{
    const Geo &g = p.g;
    const int warp = (int)(threadIdx.x >> 5), lane = (int)(threadIdx.x & 31);
    const int b = bx * V + warp % V, seg = warp / V;
    const int r = by * 32 + lane;
    double fsum = 0.0;            // polychromatic mode: this thread's likelihood terms

    // The window a warp marches with is the widest any of its rays needs: xr -
    // xl is affine in y, so a ray's widest run is at the first or the last row.
    // Every lane of the (full) warp takes part in the maximum, lanes without a
    // ray with 0, so the choice depends on the warp's rays alone and a batched
    // launch makes the same one.
    const bool live = b < p.nb && r < p.nk;
    const int k = p.k0 + r;
    FwdRay ray = {};
    int wcode = 0;   // 3 / 4: window of 3 / 4 pixels; 5: bounded range loop
    if (live) {
        ray = fwd_ray<FAN>(p, b, k);
        wcode = 5;
        if (MODE != kModeCount && g.half >= 3) {
            const float wa = ray.Ar - ray.Al, ws = ray.Sr - ray.Sl, hf = (float)g.half;
            const float wmax = fmaxf(fabsf(fmaf(-hf, ws, wa)), fabsf(fmaf(hf, ws, wa)));
            wcode = wmax < 1.95f ? 3 : (wmax < 2.95f ? 4 : 5);
        }
    }
    wcode = __reduce_max_sync(0xffffffffu, wcode);
    // The quad image.  Until it is there the sinogram is not touched: it may lie
    // on the image that the first kernel reads.
    if (R != kAllParts) wait_for_table();
    // detector 0 of an even-width sinogram: no ray, zero projection
    if (MODE != kModeCount && p.zero_col0 && bx == 0 && by == 0)
        for (int v = threadIdx.x; v < g.np; v += blockDim.x) {
            if constexpr (MODE == kModeBhc) {
                fsum += bhc_entry(p.bhc, tab, Ie, 0.0f, (size_t)v * g.W);
                if (p.bhc.proj_out) p.bhc.proj_out[(size_t)v * g.W] = 0.0f;
            } else {
                sino[(size_t)v * g.W] = 0.0f;
            }
        }
    float S[8];
    unsigned long long nz = 0;
    RowRange all = {-g.half, g.half};
    if (wcode != 5) all = warp_rows(ray, live, g.half);
    auto rows_of = [&](int s) {
        const RowRange r = part_rows(all, s, p.rsplit);
#pragma unroll
        for (int j = 0; j < 8; ++j) S[j] = 0.0f;
        if (live && r.top >= r.bottom) march_rows<FAN, MODE, R == kAllParts>(g, ray, wcode, r.top, r.bottom, quad, S, nz);
    };
    if constexpr (R > 1) {
        // a part of the rows per warp; each warp then takes its share of the images
        rows_of(seg);
        float(*ps)[8][32] = reinterpret_cast<float(*)[8][32]>(parts);
#pragma unroll
        for (int j = 0; j < 8; ++j) ps[warp][j][lane] = S[j];
        __syncthreads();
        if (live) {
#pragma unroll 1
            for (int j = seg; j < 8; j += R) {
                float sum = ps[warp % V][j][lane];
#pragma unroll
                for (int q = 1; q < R; ++q) sum += ps[q * V + warp % V][j][lane];
                fsum += put_image<FAN, MODE>(p, b, k, j, sum, sino, tab, Ie);
            }
        }
        return fsum;
    }
    rows_of(0);
    if constexpr (R == kAllParts) {
        float *tot = parts + threadIdx.x;
        const int step = blockDim.x;
        for (int s = 1; s < p.rsplit; ++s) {
#pragma unroll
            for (int j = 0; j < 8; ++j) tot[j * step] = s == 1 ? S[j] : tot[j * step] + S[j];
            rows_of(s);
        }
#pragma unroll
        for (int j = 0; j < 8; ++j) S[j] = tot[j * step] + S[j];
    }
    if (!live) return fsum;
    if constexpr (MODE == kModeCount) {
        unsigned long long entries = 0;
        for (int j = 0; j < 8; ++j) {
            const int det = j < 4 ? k : 2 * g.pC - k;
            if (p.view[b].out[j] >= 0) entries += (!FAN && 2 * g.pC - det != det) ? 2 : 1;
        }
        if (nz * entries) atomicAdd(counter, nz * entries);
    } else {
#pragma unroll
        for (int j = 0; j < 8; ++j) put_image<FAN, MODE>(p, b, k, j, S[j], sino, tab, Ie);
    }
    return fsum;
}

// floats of shared memory a forward block of `warps` warps needs for its parts
__host__ __device__ constexpr int fwd_part_floats(int warps) { return warps * 8 * 32; }

template <bool FAN, int MODE, int V, int R>
__global__ void __launch_bounds__(32 * V * R, V * R <= 4 ? CTPRJ_FWD_MINBLOCKS : 2)
k_forward(const FwdParams p, const float4 *quad, float *__restrict__ sino,
          unsigned long long *__restrict__ counter)
{
    const double *tab = nullptr, *Ie = nullptr;
    __shared__ float parts[R > 1 ? fwd_part_floats(V * R) : 1];
    if constexpr (MODE == kModeBhc) {
        __shared__ double sm[kMaxJ * (kSplStride + 1)];
        for (int i = threadIdx.x; i < p.bhc.J * kSplStride; i += blockDim.x) sm[i] = p.bhc.tab[i];
        for (int i = threadIdx.x; i < p.bhc.J; i += blockDim.x) sm[kMaxJ * kSplStride + i] = p.bhc.Ie[i];
        __syncthreads();
        tab = sm;
        Ie = sm + kMaxJ * kSplStride;
    }
    const int bx = blockIdx.x, by = blockIdx.y;
    const double fsum = forward_rays<FAN, MODE, V, R>(p, bx, by, quad, sino, counter, tab, Ie, parts);
    if constexpr (MODE == kModeBhc) {
        __shared__ double red[V * R];
        const double t = block_sum(fsum, red);
        if (threadIdx.x == 0) p.bhc.part[(size_t)by * gridDim.x + bx] = t;
    }
}

// Parts a plan's image rows are summed in, one warp each: the rows between the
// first and the last that its rays meet, so that a short chord's parts are as
// even as a long one's (equal parts of the image's rows leave the outer ones
// empty towards the detectors' ends; 512^2 fan 112 us, parallel 101, 1001^2
// 523).  The base rays alone fill only part of the GPU below 1024^2 (276 warps
// at 256^2, where it holds 2960), so up to three and a half waves of warps come
// from a split.  Beyond that it evens out the rays' uneven ways through the image:
// two parts while those are within seven waves, four for the long sums above
// (whose parts are still hundreds of rows).  Measured, 1 / 2 / 4 / 8 parts: 64^2
// fan 28.7 / 18.5 / 12.4 / 10.3 us, 256^2 parallel 84 / 49 / 29 / 21, 512^2 fan
// (1024 detectors) 172 / 142 / 117 / 100, parallel 165 / 107 / 85 / 86, 1001^2
// parallel 582 / 521 / 474 / 494, 1024^2 fan (1536 detectors) 560 / 571 / 542 /
// 546, 1500^2 fan 1587 / 1547 / 1538 / 1632 and with the polychromatic epilogue
// 1752 / 1681 / 1697 / 1835, 2048^2 fan 3505 / 3442 / 3398 / 3521 and 3801 / 3706
// / 3701 / 3900, 2048^2 parallel 3750 / 3525 / 3485 / 3668.
static int forward_split(const ctprj_plan *pl)
{
    int sms = 148;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, pl->device);
    const long long warps = (long long)pl->nb * ((pl->nk + 31) / 32), wave = 4LL * CTPRJ_FWD_MINBLOCKS * sms;
    if (2 * warps >= 7 * wave) return 4;
    int R = 2;
    while (R < 8 && 2 * warps * R < 7 * wave) R *= 2;
    return R;
}

static FwdParams fwd_params(const ctprj_plan *pl)
{
    FwdParams p;
    p.rsplit = forward_split(pl);
    p.g = pl->g;
    p.nb = pl->nb;
    p.k0 = pl->k0;
    p.nk = pl->nk;
    p.zero_col0 = (pl->g.W % 2 == 0);
    p.view = pl->d_fview;
    p.det = pl->d_det;
    p.bhc = BhcArgs{};
    return p;
}

// views per forward block when the rows are summed in R parts: blocks of four
// warps, eight for eight parts
static int fwd_views(int R) { return R >= 4 ? 1 : kFwdViews / R; }

static dim3 fwd_grid(const ctprj_plan *pl, int R)
{
    const int V = fwd_views(R);
    return dim3((pl->nb + V - 1) / V, (pl->nk + 31) / 32);
}

int forward_blocks(const ctprj_plan *pl)
{
    const dim3 g = fwd_grid(pl, forward_split(pl));
    return (int)(g.x * g.y);
}

template <bool FAN, int MODE>
static cudaError_t launch_forward_t(const FwdParams &p, dim3 grid, const float4 *quad, float *sino,
                                    unsigned long long *counter, cudaStream_t s)
{
    switch (p.rsplit) {
    case 2: return launch_after_table(k_forward<FAN, MODE, kFwdViews / 2, 2>, grid, kFwdThreads, 1, s, p, quad, sino, counter);
    case 4: return launch_after_table(k_forward<FAN, MODE, 1, 4>, grid, kFwdThreads, 1, s, p, quad, sino, counter);
    default: return launch_after_table(k_forward<FAN, MODE, 1, 8>, grid, 256, 1, s, p, quad, sino, counter);
    }
}

int launch_forward(const ctprj_plan *pl, const float4 *quad, float *sino,
                   unsigned long long *counter, cudaStream_t s)
{
    FwdParams p = fwd_params(pl);
    const bool fan = pl->g.fan != 0;
    if (counter) {
        p.rsplit = 1;
        const dim3 grid = fwd_grid(pl, 1);
        if (fan) k_forward<true, kModeCount, kFwdViews, 1><<<grid, kFwdThreads, 0, s>>>(p, quad, sino, counter);
        else k_forward<false, kModeCount, kFwdViews, 1><<<grid, kFwdThreads, 0, s>>>(p, quad, sino, counter);
    } else {
        const dim3 grid = fwd_grid(pl, p.rsplit);
        const cudaError_t e = fan ? launch_forward_t<true, kModePlain>(p, grid, quad, sino, counter, s)
                                  : launch_forward_t<false, kModePlain>(p, grid, quad, sino, counter, s);
        if (e != cudaSuccess) return cuda_error(e, "forward launch");
    }
    return cuda_error(cudaGetLastError(), "forward launch");
}

int launch_forward_bhc(const ctprj_plan *pl, const float4 *quad,
                       const BhcArgs &a, int *nparts, cudaStream_t s)
{
    FwdParams p = fwd_params(pl);
    p.bhc = a;
    const dim3 grid = fwd_grid(pl, p.rsplit);
    const cudaError_t e = pl->g.fan ? launch_forward_t<true, kModeBhc>(p, grid, quad, nullptr, nullptr, s)
                                    : launch_forward_t<false, kModeBhc>(p, grid, quad, nullptr, nullptr, s);
    if (nparts) *nparts = (int)(grid.x * grid.y);
    return cuda_error(e, "fused polychromatic forward launch");
}

// ---------------------------------------------------------------- backward

// The eight images of octant pixel (x, y), in the order of the accumulators
// (prj/cpuPrj.c:308-316): (x,y) (-y,x) (-x,-y) (y,-x) (x,-y) (y,x) (-x,y) (-y,-x).
__device__ __forceinline__ void image_of(int j, int x, int y, int &gx, int &gy)
{
    switch (j) {
    case 0: gx = x; gy = y; break;
    case 1: gx = -y; gy = x; break;
    case 2: gx = -x; gy = -y; break;
    case 3: gx = y; gy = -x; break;
    case 4: gx = x; gy = -y; break;
    case 5: gx = y; gy = x; break;
    case 6: gx = -x; gy = y; break;
    default: gx = -y; gy = -x; break;
    }
}

// A sinogram sample.  LIVE: of a launch during which sinograms arrive (the
// streaming backprojection): past L1, whose 32-byte sectors may hold the first
// samples of a slice as they were when its neighbour in memory was read.
template <bool LIVE>
__device__ __forceinline__ float load_sample(const float *p)
{
    if constexpr (LIVE) {
        float v;
        asm volatile("ld.relaxed.gpu.global.f32 %0, [%1];" : "=f"(v) : "l"(p) : "memory");
        return v;
    } else {
        return __ldg(p);
    }
}

// One base view of the pixel-driven backprojection for octant pixel (x, y):
// the detectors under the pixel's shadow, one footprint weight each, serving
// the eight symmetric images (prj/cpuPrj.c:213-300).  Everything is read from
// global memory (L1); used by k_backward and backward_tile_direct, which a plan
// takes as a whole where any view's tile shadow exceeds the staging capacity (the
// staged kernel counts on every span fitting its buffers).
template <bool FAN, bool COUNT, bool FBP, bool LIVE = false>
__device__ __forceinline__ void bwd_view_direct(const BwdParams &p, const float *__restrict__ sino,
                                                int i, int x, int y, int nimg, float (&S)[8],
                                                unsigned long long &nz)
{
    const Geo &g = p.g;
    const int dmax = (g.W - 1) / 2, pC = g.pC;
    const float dSf = (float)g.dSize;
    const double xd = x, yd = y;
    const float xf = (float)x, yf = (float)y;
    const BwdView &bv = p.view[i];
    const double cT = bv.c, sT = bv.s;
    const float cTf = bv.cf, sTf = bv.sf;
    const double u = fma(xd, cT, yd * sT);    // along the detector
    float tlo, thi, qe = 0.0f;
    double v = 0.0;
    if (FAN) {
        // shadow of the pixel's corners on the virtual detector
        // (prj/cpuPrj.c:218-244)
        v = fma(yd, cT, -xd * sT);
        qe = (float)(g.d - v);
        const float ocm = fmaf(xf - 0.5f, cTf, (yf - 0.5f) * sTf);
        const float qem = fmaf(xf - 0.5f, sTf, -(yf - 0.5f) * cTf) + g.dF;
        const float t0 = g.dF * ocm / qem;
        const float t1 = g.dF * (ocm + cTf) / (qem + sTf);
        const float t2 = g.dF * (ocm + cTf + sTf) / (qem + sTf - cTf);
        const float t3 = g.dF * (ocm + sTf) / (qem - cTf);
        tlo = fminf(fminf(t0, t1), fminf(t2, t3));
        thi = fmaxf(fmaxf(t0, t1), fmaxf(t2, t3));
    } else {
        const float hw = 0.5f * (fabsf(cTf) + fabsf(sTf));
        const float uf = (float)u;
        tlo = uf - hw;
        thi = uf + hw;
    }
    int dl = (int)roundf(fmaxf(tlo / dSf, (float)(-dmax - 1)));
    int dr = (int)roundf(fminf(thi / dSf, (float)(dmax + 1)));
    dl = max(dl, -dmax);
    dr = min(dr, dmax);
    Footprint pfp;
    if (!FAN) {
        pfp.h = bv.h; pfp.b1 = bv.b1; pfp.b2 = bv.b2; pfp.w = bv.w; pfp.iw2 = bv.iw2;
    }
    for (int dt = dl; dt <= dr; ++dt) {
        const DetEntry &de = p.det[dt + pC];
        float w;
        if (FAN) {
            // distance from the detector's ray: cos B (u - t) + sin B v
            const float dist = (float)fma(de.cB, u - de.t, de.sB * v);
            const float cR = fmaf(de.cBf, cTf, -de.sBf * sTf);
            const float sR = fmaf(de.sBf, cTf, de.cBf * sTf);
            const Footprint fp = make_footprint(cR, sR);
            w = footprint_weight(dist, qe * g.beamWidthF * de.invbq, fp);
            if (FBP) w = w * g.dF * g.dF / qe / qe;
        } else {
            w = footprint_weight((float)(u - de.t), g.beamWidthF, pfp);
        }
        if (COUNT) {
            if (w != 0.0f) nz += (nimg == 8 ? bv.cnt8 : bv.cnt4);
            continue;
        }
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const int sg = j < 4 ? dt : -dt;
            const int row = bv.row[j];
            if (row >= 0) S[j] = fmaf(w, load_sample<LIVE>(sino + row + pC + sg), S[j]);
            if (!FAN) {
                const int row2 = bv.row2[j];
                if (row2 >= 0) S[j] = fmaf(w, load_sample<LIVE>(sino + row2 + pC - sg), S[j]);
            }
        }
    }
}

__device__ __forceinline__ void decode_tile(int tile, int &tx, int &ty)
{
    tx = (int)((sqrtf(8.0f * (float)tile + 1.0f) - 1.0f) * 0.5f);
    while ((tx + 1) * (tx + 2) / 2 <= tile) ++tx;
    while (tx * (tx + 1) / 2 > tile) --tx;
    ty = tile - tx * (tx + 1) / 2;
}

__device__ __forceinline__ void write_octant(const BwdParams &p, float *__restrict__ img, int x,
                                             int y, int nimg, const float (&S)[8])
{
    const Geo &g = p.g;
    const int h2 = g.h2, N = g.n;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        if (j >= nimg) break;
        int gx, gy;
        image_of(j, x, y, gx, gy);
        const float val = S[j] * p.scale;
        img[(size_t)(gy + h2) * N + (gx + h2)] = val / g.effRate;
    }
}

// one tile of the unstaged backprojection (plain mode), for persistent use
template <bool FAN, bool LIVE>
__device__ __forceinline__ void backward_tile_direct(const BwdParams &p, int tile,
                                                     const float *__restrict__ sino,
                                                     float *__restrict__ img)
{
    const Geo &g = p.g;
    if (p.zero_axes && tile == 0)
        for (int i = threadIdx.x; i < g.n; i += blockDim.x) {
            img[i] = 0.0f;
            img[(size_t)i * g.n] = 0.0f;
        }
    int tx, ty;
    decode_tile(tile, tx, ty);
    for (int e = threadIdx.x; e < kBwdTile * kBwdTile; e += blockDim.x) {
        const int x = tx * kBwdTile + e % kBwdTile, y = ty * kBwdTile + e / kBwdTile;
        if (x > g.half || y > x) continue;
        const int nimg = (y == 0 || y == x) ? 4 : 8;
        float S[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) S[j] = 0.0f;
        unsigned long long nz = 0;
        for (int i = 0; i < p.nv; ++i) bwd_view_direct<FAN, false, false, LIVE>(p, sino, i, x, y, nimg, S, nz);
        write_octant(p, img, x, y, nimg, S);
    }
}

template <bool FAN, bool COUNT, bool FBP>
__global__ void __launch_bounds__(kBwdTile * kBwdTile)
k_backward(const BwdParams p, const float *__restrict__ sino, float *__restrict__ img,
           unsigned long long *__restrict__ counter)
{
    const Geo &g = p.g;
    if (!COUNT && p.zero_axes && blockIdx.x == 0)
        for (int i = threadIdx.x; i < g.n; i += blockDim.x) {
            img[i] = 0.0f;
            img[(size_t)i * g.n] = 0.0f;
        }
    int tx, ty;
    decode_tile(blockIdx.x, tx, ty);
    const int x = tx * kBwdTile + (int)(threadIdx.x % kBwdTile);
    const int y = ty * kBwdTile + (int)(threadIdx.x / kBwdTile);
    if (x > g.half || y > x) return;
    const int nimg = (y == 0 || y == x) ? 4 : 8;
    float S[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) S[j] = 0.0f;
    unsigned long long nz = 0;
    for (int i = 0; i < p.nv; ++i) bwd_view_direct<FAN, COUNT, FBP>(p, sino, i, x, y, nimg, S, nz);
    if (COUNT) {
        if (nz) atomicAdd(counter, nz);
        return;
    }
    write_octant(p, img, x, y, nimg, S);
}

// ------------------------------------------------------ backward, staged tiles
//
// The same backprojection with the per-(view, detector) work hoisted out of the
// per-pixel loop.  Its operands come from two tables.  The sample image holds,
// for base view i < prjFull/4 and detector k, the eight mirrored sinogram
// samples one weight multiplies (two float4 planes, built by k_samples at the
// start of each call; parallel beam: a sample plus its point-reflected partner
// of the opposite view, which takes the same weight).  Base view i + a prjFull/4
// reads the same samples, rotated among the images, so the accumulators are
// rotated instead at each quarter.  The footprint table (fan beam) holds each
// ray's trapezoid; a quarter turn leaves it as it is.
//
// A block owns a 16 x 16 tile of octant pixels.  For a batch of VB base views
// it copies the detectors under the tile's shadow into shared memory by 16-byte
// cp.async, double-buffered: the next batch is in flight while this one is
// summed, at one barrier per batch.  A thread owns two pixels side by side and
// reads each staged detector of the union of their windows once for both.
//
// What bounds it: the shared-memory data path (a warp's 16-byte load takes four
// wavefronts whatever its lanes read) and instruction issue, about equally.
// Samples and footprint of a fan detector are 48 bytes, twelve wavefronts; a
// pixel on its own needs three detectors per view, a pair four (or three), so a
// view costs 26 (20) wavefronts per 32 pixels instead of 38.  Packed
// fma.rn.f32x2 gains nothing here: it takes two turns of the FP32 pipe.
// Against one pixel per thread with samples gathered by each tile: 4.60 -> 3.01
// ms at the 2048^2 fan workload, 149 -> 70 us at 512^2 (1024 detectors, 360
// views), parallel 1001^2 (720 views) 814 -> 386 us and 256^2 78 -> 19 us.  At
// 1024^2 (fan, 720 views): 116 warp instructions per 32 pixels and view, issue
// 77 % active, shared-memory wavefronts 59 %, FP32 pipe 55 % (ncu).
//
// Geometry, in units of (distance from the ray) / cos B: with T = t / d the
// tangent of detector k's fan angle, a pixel at (u, v) along / across the
// detector lies at E_k = u - t_k + T_k v from ray k, the ray spacing there is
// G = (d - v) dSize / d exactly, the half beam width G effectiveRate / 2, and
// the pixel's trapezoid has lo = min(|c - T s|, |s + T c|) and hi = max(.).  So
// E_k = E_r - (k - r) G from any reference detector r, the beam edges of
// neighbouring detectors coincide (effectiveRate = 1), and cos B drops out.
// The reference detector is the one nearest the centre of a warp's 8 x 8
// pixels, with E_r formed in FP64 there: everything a pixel then adds is at
// most a few units in size, so its rounding stays below 3e-7.  Parallel beam:
// T = 0, G = dSize.
//
// Window: the beams that meet a pixel's footprint lie within rho = (shadow
// width + effectiveRate) / 2 detectors of its projected centre.  The two pixels
// project Delta = |c - T s| / G apart; if the right one's window starts o
// detectors after the left one's, n detectors each hold both as soon as
// n >= 2 rho + |Delta - o|.  The smallest n (and its smallest o) is chosen per
// view and warp, so every lane takes the same straight code.  A beam wider than
// the pitch (effectiveRate > 1) also meets pixels whose shadow its detector
// lies outside of, which the reference's range rule (prj/cpuPrj.c:81-105,
// :218-244) leaves out: such plans (RANGE) also test each detector against the
// pixel's own corner shadow.

struct TileSpan {
    int klo, nseg;
};

// Detectors any pixel of tile (tx, ty) can reach in base view bv, as the first
// one (relative to the centre bin) and a count, with one spare on each side;
// `past` entries beyond the first and last detector may belong to it.
// nseg = 1 << 20 flags a tile the source sees from behind or edge-on.
__device__ __forceinline__ float tile_corner(const Geo &g, float cf, float sf, int tx, int ty, int q, int &bad)
{
    const float X0 = tx * kBwdTile - 0.5f, Y0 = ty * kBwdTile - 0.5f;
    const float cx = (q == 1 || q == 2) ? X0 + kBwdTile : X0, cy = q >= 2 ? Y0 + kBwdTile : Y0;
    const float oc = fmaf(cx, cf, cy * sf);
    if (!g.fan) return oc;
    const float qe = fmaf(cx, sf, -cy * cf) + g.dF;
    bad |= !(qe > 1e-3f * g.dF);
    return g.dF * oc / qe;
}

__device__ __forceinline__ TileSpan span_of(const Geo &g, float lo, float hi, int bad, int past)
{
    const int dmax = (g.W - 1) / 2 + past;
    TileSpan sp;
    const float inv = (float)(1.0 / g.dSize), lim = (float)dmax + 2.0f;
    const int klo = max(__float2int_rd(fminf(fmaxf(lo * inv, -lim), lim)) - 1, -dmax);
    const int khi = min(__float2int_ru(fminf(fmaxf(hi * inv, -lim), lim)) + 1, dmax);
    sp.klo = klo;
    sp.nseg = bad ? (1 << 20) : khi - klo + 1;
    return sp;
}

__device__ __forceinline__ TileSpan tile_span(const Geo &g, const BwdView &bv, int tx, int ty)
{
    int bad = 0;
    float lo = 0.0f, hi = 0.0f;
    for (int q = 0; q < 4; ++q) {
        const float tq = tile_corner(g, bv.cf, bv.sf, tx, ty, q, bad);
        lo = q == 0 ? tq : fminf(lo, tq);
        hi = q == 0 ? tq : fmaxf(hi, tq);
    }
    return span_of(g, lo, hi, bad, 0);
}

__global__ void k_tile_span_max(const BwdParams p, int tiles, int *__restrict__ out)
{
    int m = 0;
    const long long total = (long long)tiles * p.nv;
    for (long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x; e < total;
         e += (long long)gridDim.x * blockDim.x) {
        int tx, ty;
        decode_tile((int)(e / p.nv), tx, ty);
        m = max(m, tile_span(p.g, p.view[e % p.nv], tx, ty).nseg);
    }
    atomicMax(out, m);
}

// footprint of the direction (a, b), scaled by any positive factor: 1 / lo,
// (foot half width) / lo, 1 / (2 shoulder half width), lo / (2 hi).  Zero ramp
// or shoulder widths get a tiny floor: the huge ratios saturate and are
// multiplied by the zero width.
__device__ __forceinline__ float4 staged_footprint(float a, float b)
{
    a = fabsf(a);
    b = fabsf(b);
    const float hi = fmaxf(a, b), lo = fminf(a, b);
    const float cw = 1.0f / fmaxf(lo, 1e-30f);
    return make_float4(cw, 0.5f * (hi + lo) * cw, 1.0f / fmaxf(hi - lo, 1e-30f), 0.5f * lo / hi);
}

// The footprint table of a fan plan: row i < prjFull/4, entry k + W/2 + kBwdTablePad.
__global__ void __launch_bounds__(256) k_footprints(const BwdParams p, float4 *__restrict__ foot)
{
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= p.Wp) return;
    const float T = (float)(k - p.g.pC - kBwdTablePad) * p.cG;
    for (int i = blockIdx.y; i < p.g.P / 4; i += gridDim.y) {
        const float c = p.view[i].cf, s = p.view[i].sf;
        foot[(size_t)i * p.Wp + k] = staged_footprint(fmaf(-T, s, c), fmaf(T, c, s));
    }
}

// Row i of the sample image (a block's threads along the detectors); the
// entries beyond the detectors stay zero.
template <bool LIVE>
__device__ __forceinline__ void sample_row(const BwdParams &p, const float *__restrict__ sino, int i,
                                           int k0, int step)
{
    const Geo &g = p.g;
    const int dmax = (g.W - 1) / 2, pC = g.pC, Q = g.P / 4;
    const float *src[8], *src2[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        // rows of the symmetric views (the host's view_of), and of the opposite ones
        const int q = j < 4 ? j : (j - 2) & 3;
        int v = j < 4 ? q * Q + i : q * Q - i;
        v = v < 0 ? v + g.P : v;
        int v2 = v + 2 * Q;
        v2 = v2 >= g.P ? v2 - g.P : v2;
        src[j] = v < g.np ? sino + (size_t)v * g.W + pC : nullptr;
        src2[j] = !g.fan && v2 < g.np ? sino + (size_t)v2 * g.W + pC : nullptr;
    }
    float4 *dst = p.samp + (size_t)i * 2 * p.Wp + pC + kBwdTablePad;
    for (int k = k0 - dmax; k <= dmax; k += step) {
        float v[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) v[j] = src[j] ? load_sample<LIVE>(src[j] + (j < 4 ? k : -k)) : 0.0f;
        if (!g.fan)
#pragma unroll
            for (int j = 0; j < 8; ++j)
                if (src2[j]) v[j] += load_sample<LIVE>(src2[j] - (j < 4 ? k : -k));
        dst[k] = make_float4(v[0], v[1], v[2], v[3]);
        dst[p.Wp + k] = make_float4(v[4], v[5], v[6], v[7]);
    }
}

constexpr int kSampThreads = 128;

__global__ void __launch_bounds__(kSampThreads) k_samples(const BwdParams p, const float *__restrict__ sino)
{
    // Started beside this kernel, a large backprojection's blocks crowd onto the SMs
    // it leaves free and stay there (256^2 20.5 -> 25.6 us, 512^2 fan 68 -> 78); at
    // one block per SM the early start is worth 2 of 12 us (64^2)
    if (p.tiles_side * (p.tiles_side + 1) / 2 * p.split <= 128) let_next_start();
    for (int i = blockIdx.y; i < p.g.P / 4; i += gridDim.y)
        sample_row<false>(p, sino, i, blockIdx.x * kSampThreads + threadIdx.x, gridDim.x * kSampThreads);
}

constexpr int kBwdThreads = kBwdTile * kBwdTile / 2;   // two pixels per thread
constexpr int kBwdWarps = kBwdThreads / 32;            // one 8 x 8 pixel square each
// Staged past the detectors' ends (zeros), so that the union of two windows up
// to two detectors apart can lie anywhere on them; a row of the staging buffer
// holds the plan's widest span and these.
constexpr int kBwdPast = 2;
constexpr int kBwdGroup = 32;  // views whose geometry the block prepares at a time
constexpr float kBwdMagic = 12582912.0f;   // 1.5 * 2^23: x + it rounds |x| < 2^22 to an integer,
constexpr int kBwdMagicBits = 0x4B400000;  // whose value is the sum's bits minus these

// one view as a warp's pixel square sees it
struct BwdSquare {
    float E, T, qec;   // reference detector r: E_r and T_r; d - v of the square's centre (parallel: r)
    int ioff;          // staged index of detector r, minus kBwdMagicBits
    float c, s;        // direction of the view
    float lo, hi;      // range of the union's first detector, relative to r
    float off;         // (n - 1 + o) / 2: from a pair's projection to that detector
    float kh, g;       // half the step of E, and of G, from the pixel at x to the one at x + 1
    int code;          // n, and the offsets in the union of x's window << 8 and x + 1's << 16
};

// shared memory of one staged tile: two buffers of VB views
template <bool FAN, int SEG, int VB>
struct TiledSmem {
    float4 seg[2][VB][FAN ? 3 : 2][SEG + 2 * kBwdPast];     // samples 0-3, samples 4-7, footprints
    BwdSquare sq[2][kBwdGroup][kBwdWarps];
    float4 fp[2][FAN ? 1 : kBwdGroup];       // parallel beam: the view's footprint
};

__device__ __forceinline__ void stage16(float4 *smem, const float4 *gmem)
{
    const unsigned sa = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(sa), "l"(gmem) : "memory");
}

__device__ __forceinline__ float sat_fma(float a, float b, float c) { return __saturatef(fmaf(a, b, c)); }

// Weight of a detector between its beam edges el and er: the trapezoid's area
// between them (footprint_weight_v's form: rising and falling ramps P and R,
// plateau Q).
__device__ __forceinline__ float edge_weight(float el, float er, float4 f)
{
    const float P1 = sat_fma(er, f.x, f.y), R1 = sat_fma(er, -f.x, f.y), Q1 = sat_fma(er, f.z, 0.5f);
    const float P2 = sat_fma(el, f.x, f.y), R2 = sat_fma(el, -f.x, f.y), Q2 = sat_fma(el, f.z, 0.5f);
    const float dQ = Q1 - Q2;
    const float X = fmaf(R2, R2, fmaf(-P2, P2, fmaf(-R1, R1, P1 * P1)));
    return fmaf(f.w, fmaf(-2.0f, dQ, X), dQ);
}

// area of the trapezoid from its centre to the edge e, plus a constant
// (parallel beam: every detector of a view has the same footprint, so
// neighbouring weights share it)
__device__ __forceinline__ float edge_area(float e, float4 f)
{
    const float P = sat_fma(e, f.x, f.y), R = sat_fma(e, -f.x, f.y), Q = sat_fma(e, f.z, 0.5f);
    return fmaf(f.w, fmaf(-2.0f, Q, fmaf(-R, R, P * P)), Q);
}

// the geometry of view i for square w of tile (tx, ty), whose detectors are
// staged from klo; the window (n, o) is returned in q.code, q.lo, q.hi left open
template <bool FAN>
__device__ __forceinline__ BwdSquare square_view(const BwdParams &p, const BwdView &bv, int tx, int ty, int w, int klo,
                                                 int seg)
{
    const Geo &g = p.g;
    const double xw = tx * kBwdTile + (w & 1) * 8 + 3.5, yw = ty * kBwdTile + (w >> 1) * 8 + 3.5;
    const double uc = fma(xw, bv.c, yw * bv.s);
    BwdSquare q;
    q.c = bv.cf;
    q.s = bv.sf;
    // (r is held near the detector: squares that project far off it meet no ray
    // whatever the reference)
    const float rmax = (float)(g.W / 2 + 128);
    float r, G, Gmin, slack = 0.0f;
    if (FAN) {
        const double qd = g.d - fma(yw, bv.c, -xw * bv.s);
        q.qec = (float)qd;
        r = fminf(fmaxf(rintf(__fdividef((float)uc * p.invG, q.qec)), -rmax), rmax);
        const double T = (double)r * g.dSize * p.invd;
        q.T = (float)T;
        q.E = (float)fma(-T, qd, uc);
        // a pixel lies within 5 of the square's centre and every pixel of a
        // staged tile has qe > d / 1000; the rays that meet the square differ
        // from r's tangent by at most (5 (1 + |T|) + G + 3/4) / qe
        const float qm = fmaxf(q.qec - 5.0f, 1e-3f * g.dF);
        G = q.qec * p.cG;
        Gmin = qm * p.cG;
        slack = __fdividef(fmaf(1.5f, G, fmaf(9.0f, fabsf(q.T), 9.0f)), qm);
    } else {
        r = fminf(fmaxf(rintf((float)uc * p.invG), -rmax), rmax);
        q.T = 0.0f;
        q.qec = r;
        q.E = (float)fma(-(double)r, g.dSize, uc);
        G = Gmin = (float)g.dSize;
    }
    const float kx = fmaf(-q.T, q.s, q.c), ky = fmaf(q.T, q.c, q.s);
    q.kh = 0.5f * kx;
    q.g = FAN ? 0.5f * q.s * p.cG : 0.0f;
    // 2 rho, and the range of Delta over the square
    const float inv = __fdividef(1.0f, Gmin);
    const float reach = fmaf(fabsf(kx) + fabsf(ky) + slack, inv, g.effRate + 2e-3f);
    const float dlo = fmaf(-slack, inv, __fdividef(fabsf(kx), G)), dhi = fmaf(slack, inv, fabsf(kx) * inv);
    int n = 1 << 20, o = 0;
#pragma unroll
    for (int t = 0; t < 3; ++t) {
        const float need = reach + fmaxf(fabsf(dlo - (float)t), fabsf(dhi - (float)t));
        const int nt = max(__float2int_ru(fminf(need, 4096.0f)), 2);
        if (nt < n) {
            n = nt;
            o = t;
        }
    }
    n = min(n, seg - o);   // the union never exceeds the staged detectors
    q.off = 0.5f * (float)(n - 1 + o);
    q.code = n | (o << (kx < 0.0f ? 8 : 16));   // the window of the pixel further along starts later
    q.ioff = (int)r - klo - kBwdMagicBits;
    q.lo = (float)klo - r;
    q.hi = q.lo;
    return q;
}

// what a thread's pair of pixels takes from a view before its weights
struct PairView {
    float EA, EB, GA, GB;   // of the pixels at x and x + 1
    float cb;               // first detector of the union, relative to r
    int i0;                 // its staged index
};

template <bool FAN>
__device__ __forceinline__ PairView pair_start(const BwdParams &p, const BwdSquare &q, float dx, float dy)
{
    const float du = fmaf(dx, q.c, dy * q.s), dv = fmaf(dy, q.c, -dx * q.s);
    const float E = FAN ? fmaf(q.T, dv, q.E + du) : q.E + du;
    const float qe = FAN ? q.qec - dv : 1.0f;
    // the pair's projection E / G in detectors from r, less its offset in the union
    const float t = FAN ? fmaf(E * p.invG, __fdividef(1.0f, qe), -q.off) : fmaf(E, p.invG, -q.off);
    // nearest integer by an FP32 add; its bits are the staged index
    const float m = fminf(fmaxf(t, q.lo), q.hi) + kBwdMagic;
    PairView v;
    v.cb = m - kBwdMagic;
    v.i0 = __float_as_int(m) + q.ioff;
    v.EA = E - q.kh;
    v.EB = E + q.kh;
    const float G = FAN ? qe * p.cG : (float)p.g.dSize;
    v.GA = FAN ? G - q.g : G;
    v.GB = FAN ? G + q.g : G;
    return v;
}

// S += w p for the eight images of a pixel
__device__ __forceinline__ void add_samples(float (&S)[8], float w, float4 p0, float4 p1)
{
    S[0] = fmaf(w, p0.x, S[0]);
    S[1] = fmaf(w, p0.y, S[1]);
    S[2] = fmaf(w, p0.z, S[2]);
    S[3] = fmaf(w, p0.w, S[3]);
    S[4] = fmaf(w, p1.x, S[4]);
    S[5] = fmaf(w, p1.y, S[5]);
    S[6] = fmaf(w, p1.z, S[6]);
    S[7] = fmaf(w, p1.w, S[7]);
}

// FBP weight of a pixel, (d / qe)^2 with qe = G / cG
template <bool FAN, bool FBP>
__device__ __forceinline__ float fbp_weight(const BwdParams &p, float G)
{
    if (!FAN || !FBP) return 1.0f;
    const float f = __fdividef((float)p.g.dSize, G);
    return f * f;
}

// One view for a pair of pixels, A and B the sums of x and x + 1: windows of N
// detectors at OA and OB in the union.
template <bool FAN, bool FBP, int SEG, bool UNIT, int N, int OA, int OB>
__device__ __forceinline__ void pair_view(const BwdParams &p, const PairView &v, const float4 *__restrict__ seg,
                                          float4 fpar, float (&A)[8], float (&B)[8])
{
    constexpr int U = N + (OA > OB ? OA : OB);
    const float4 *s0 = seg + v.i0, *s1 = s0 + SEG + 2 * kBwdPast, *fp = s1 + SEG + 2 * kBwdPast;
    const float hb = 0.5f * p.g.effRate;
    const float fA = fbp_weight<FAN, FBP>(p, v.GA), fB = fbp_weight<FAN, FBP>(p, v.GB);
    // left edges of the first detectors (a window's edges are a few pitches from
    // them); parallel beam: the areas up to them
    const float aA = fmaf(v.cb + ((float)OA - hb), v.GA, -v.EA), aB = fmaf(v.cb + ((float)OB - hb), v.GB, -v.EB);
    float eA = aA, eB = aB;
    if (!FAN && UNIT) {
        eA = edge_area(eA, fpar);
        eB = edge_area(eB, fpar);
    }
    // weight of the window's j-th detector: its right edge becomes the next one's left
    auto weight = [&](float &e, int j, float G, float a, float4 f) {
        const float r = fmaf((float)j + (UNIT ? 1.0f : p.g.effRate), G, a), l = e;
        if (!FAN && UNIT) {
            e = edge_area(r, f);
            return e - l;
        }
        e = UNIT ? r : fmaf((float)(j + 1), G, a);
        return edge_weight(l, r, f);
    };
#pragma unroll
    for (int j = 0; j < U; ++j) {
        const float4 f = FAN ? fp[j] : fpar, p0 = s0[j], p1 = s1[j];
        if (j >= OA && j < OA + N) {
            const float w = weight(eA, j - OA, v.GA, aA, f);
            add_samples(A, FBP && FAN ? w * fA : w, p0, p1);
        }
        if (j >= OB && j < OB + N) {
            const float w = weight(eB, j - OB, v.GB, aB, f);
            add_samples(B, FBP && FAN ? w * fB : w, p0, p1);
        }
    }
}

// The same for any window, and with RANGE only the detectors of the pixel's
// corner shadow (prj/cpuPrj.c:218-244), rounded to the nearest detectors.
template <bool FAN, bool FBP, int SEG, bool RANGE>
__device__ __forceinline__ void pair_view_any(const BwdParams &p, const BwdSquare &q, const PairView &v,
                                              const float4 *__restrict__ seg, float4 fpar, float (&A)[8], float (&B)[8],
                                              const BwdView &bv, int x, int y)
{
    const float4 *s0 = seg + v.i0, *s1 = s0 + SEG + 2 * kBwdPast, *fp = s1 + SEG + 2 * kBwdPast;
    const int n = q.code & 255, oa = (q.code >> 8) & 255, ob = q.code >> 16;
    const float hb = 0.5f * p.g.effRate;
    const float fA = fbp_weight<FAN, FBP>(p, v.GA), fB = fbp_weight<FAN, FBP>(p, v.GB);
    float loA = 0.0f, hiA = 0.0f, loB = 0.0f, hiB = 0.0f;
    if (RANGE) {
        const float ca = 0.5f * (q.c + q.s), cb = 0.5f * (q.c - q.s);
        const float r = FAN ? rintf(q.T * p.invG) : q.qec;
        auto range = [&](float E, float G, int px, float &lo, float &hi) {
            float tlo, thi;
            if (FAN) {
                const float qe = G * p.invG, ea = fmaf(q.T, cb, ca), eb = fmaf(-q.T, ca, cb);
                const float t0 = __fdividef(E - ea, qe + cb), t1 = __fdividef(E + eb, qe + ca);
                const float t2 = __fdividef(E + ea, qe - cb), t3 = __fdividef(E - eb, qe - ca);
                tlo = fminf(fminf(t0, t1), fminf(t2, t3)) * p.invG;
                thi = fmaxf(fmaxf(t0, t1), fmaxf(t2, t3)) * p.invG;
            } else {
                // (in FP64: views along an axis put every shadow edge half way
                // between detectors, give or take the rounding of the view's angle)
                const double u = fma((double)px, bv.c, y * bv.s), hw = 0.5 * (fabs(bv.c) + fabs(bv.s));
                lo = (float)(round((u - hw) / p.g.dSize) - (double)r);
                hi = (float)(round((u + hw) / p.g.dSize) - (double)r);
                return;
            }
            // nearest detector, half-way cases away from the centre as the
            // reference's round(): relative to r, by the sign of the place
            auto nearest = [&](float t) { return r + t < 0.0f ? ceilf(t - 0.5f) : floorf(t + 0.5f); };
            lo = nearest(tlo);
            hi = nearest(thi);
        };
        range(v.EA, v.GA, x, loA, hiA);
        range(v.EB, v.GB, x + 1, loB, hiB);
    }
    for (int j = 0; j < n + oa + ob; ++j) {   // one of the offsets is zero
        const float k = v.cb + (float)j;
        const float4 f = FAN ? fp[j] : fpar, p0 = s0[j], p1 = s1[j];
        if (j >= oa && j < oa + n && (!RANGE || (k >= loA && k <= hiA))) {
            const float w = edge_weight(fmaf(k - hb, v.GA, -v.EA), fmaf(k + hb, v.GA, -v.EA), f);
            add_samples(A, FBP && FAN ? w * fA : w, p0, p1);
        }
        if (j >= ob && j < ob + n && (!RANGE || (k >= loB && k <= hiB))) {
            const float w = edge_weight(fmaf(k - hb, v.GB, -v.EB), fmaf(k + hb, v.GB, -v.EB), f);
            add_samples(B, FBP && FAN ? w * fB : w, p0, p1);
        }
    }
}

// the accumulators of one quarter of the views for the next: base view i +
// prjFull/4 finds image j's sample where view i has that of the image a quarter
// turn on
__device__ __forceinline__ void rotate_sums(float (&S)[8])
{
    const float a = S[3], b = S[4];
    S[3] = S[2];
    S[2] = S[1];
    S[1] = S[0];
    S[0] = a;
    S[4] = S[5];
    S[5] = S[6];
    S[6] = S[7];
    S[7] = b;
}

// Adds the base views [v0, v1), all of one quarter that begins at view vq, to
// the sums of one tile: A of a thread's pixel x and B of x + 1 (all threads of
// the block take part).  Every product that meets a sum in here and in what it
// calls is an explicit fma, so that no kernel this is inlined into contracts
// it differently: the batched and per-plan launches must give the same bits.
template <bool FAN, bool FBP, int SEG, int VB, int MODE>
__device__ __forceinline__ void quarter_sums(const BwdParams &p, int tx, int ty, int v0, int v1, int vq, float (&A)[8],
                                             float (&B)[8], TiledSmem<FAN, SEG, VB> &sm)
{
    constexpr int kPer = VB / kBwdWarps;         // views a warp stages per batch
    constexpr int kBatches = kBwdGroup / VB;     // batches per prepared group
    constexpr bool UNIT = MODE == kBwdUnit, RANGE = MODE == kBwdRange;
    const Geo &g = p.g;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    // eight lanes of a warp take a 4 x 4 square of pixels: their window loads
    // fall in at most six consecutive 16-byte entries, which share no bank
    const float dx = (float)(((lane >> 3) & 1) * 4 + (lane & 1) * 2) - 3.0f;   // the pair's middle
    const float dy = (float)((lane >> 4) * 4 + ((lane >> 1) & 3)) - 3.5f;
    // squares above the diagonal of a diagonal tile, or past the image, hold no pixel
    const int xw = tx * kBwdTile + (warp & 1) * 8, yw = ty * kBwdTile + (warp >> 1) * 8;
    const bool live = xw <= g.half && yw <= xw + 7;
    // The geometry of a group of views: lanes 4 l .. 4 l + 3 of warp w take
    // view (l / kPer) VB + w kPer + l % kPer of the group, one corner of the
    // tile and one square each, and keep the view's detector span, so that the
    // warp can stage its views of a batch without waiting for another.
    int klo = 0, cnt = 0;
    auto prepare = [&](int grp) {
        const int l = lane >> 2, gv = (l / kPer) * VB + warp * kPer + l % kPer;
        const BwdView &bv = p.view[min(v0 + grp * kBwdGroup + gv, v1 - 1)];
        int bad = 0;
        float lo = tile_corner(g, bv.cf, bv.sf, tx, ty, lane & 3, bad), hi = lo;
#pragma unroll
        for (int o = 1; o <= 2; o <<= 1) {
            lo = fminf(lo, __shfl_xor_sync(0xffffffffu, lo, o));
            hi = fmaxf(hi, __shfl_xor_sync(0xffffffffu, hi, o));
        }
        const TileSpan sp = span_of(g, lo, hi, 0, kBwdPast);
        klo = sp.klo;
        BwdSquare q = square_view<FAN>(p, bv, tx, ty, lane & 3, klo, SEG);
        const int un = (q.code & 255) + ((q.code >> 8) & 255) + (q.code >> 16);
        cnt = max(sp.nseg, un);
#pragma unroll
        for (int o = 1; o <= 2; o <<= 1) cnt = max(cnt, __shfl_xor_sync(0xffffffffu, cnt, o));
        cnt = min(cnt, SEG + 2 * kBwdPast);   // the plan chose SEG above every span
        q.hi = q.lo + (float)(cnt - un);
        sm.sq[grp & 1][gv][lane & 3] = q;
        if (!FAN && (lane & 3) == 0) sm.fp[grp & 1][FAN ? 0 : gv] = staged_footprint(q.c, q.s);
    };
    auto stage = [&](int b) {
#pragma unroll
        for (int u = 0; u < kPer; ++u) {
            const int l = (b % kBatches) * kPer + u, iv = warp * kPer + u;
            const int k0 = __shfl_sync(0xffffffffu, klo, 4 * l), n = __shfl_sync(0xffffffffu, cnt, 4 * l);
            const int i = v0 + b * VB + iv;
            if (i >= v1) continue;
            const float4 *sp = p.samp + (size_t)(i - vq) * 2 * p.Wp + (k0 + g.pC + kBwdTablePad);
            const float4 *fp = p.foot + (size_t)(i - vq) * p.Wp + (k0 + g.pC + kBwdTablePad);
            for (int kk = lane; kk < n; kk += 32) {
                stage16(&sm.seg[b & 1][iv][0][kk], sp + kk);
                stage16(&sm.seg[b & 1][iv][1][kk], sp + p.Wp + kk);
                if (FAN) stage16(&sm.seg[b & 1][iv][FAN ? 2 : 0][kk], fp + kk);
            }
        }
        asm volatile("cp.async.commit_group;\n" ::: "memory");
    };
    const int nbatch = (v1 - v0 + VB - 1) / VB;
    prepare(0);
    wait_for_table();   // the sample image (nothing to wait for but in the first quarter)
    stage(0);
    for (int b = 0; b < nbatch; ++b) {
        const bool more = b + 1 < nbatch;
        if (more && (b + 1) % kBatches == 0) prepare((b + 1) / kBatches);
        asm volatile("cp.async.wait_group 0;\n" ::: "memory");
        __syncthreads();   // batch b and its geometry have landed; the other buffer is free
        if (more) stage(b + 1);
        if (!live) continue;
        const int nb = min(VB, v1 - (v0 + b * VB)), gv = (b % kBatches) * VB, gb = (b / kBatches) & 1;
        const BwdSquare *sq = &sm.sq[gb][gv][warp];
        const float4 *fp = &sm.fp[gb][FAN ? 0 : gv], *seg = &sm.seg[b & 1][0][0][0];
        for (int iv = 0; iv < nb; ++iv, sq += kBwdWarps, seg += (FAN ? 3 : 2) * (SEG + 2 * kBwdPast), fp += FAN ? 0 : 1) {
            const BwdSquare q = *sq;
            const float4 fpar = FAN ? make_float4(0.0f, 0.0f, 0.0f, 0.0f) : *fp;
            const PairView v = pair_start<FAN>(p, q, dx, dy);
            if (RANGE) {
                pair_view_any<FAN, FBP, SEG, true>(p, q, v, seg, fpar, A, B, p.view[v0 + b * VB + iv],
                                                   xw + (int)(dx + 3.0f), yw + (int)(dy + 3.5f));
                continue;
            }
            switch (q.code) {
            case 3 | (1 << 16): pair_view<FAN, FBP, SEG, UNIT, 3, 0, 1>(p, v, seg, fpar, A, B); break;
            case 3 | (1 << 8): pair_view<FAN, FBP, SEG, UNIT, 3, 1, 0>(p, v, seg, fpar, A, B); break;
            case 3: pair_view<FAN, FBP, SEG, UNIT, 3, 0, 0>(p, v, seg, fpar, A, B); break;
            case 4 | (1 << 16): pair_view<FAN, FBP, SEG, UNIT, 4, 0, 1>(p, v, seg, fpar, A, B); break;
            case 4 | (1 << 8): pair_view<FAN, FBP, SEG, UNIT, 4, 1, 0>(p, v, seg, fpar, A, B); break;
            default: pair_view_any<FAN, FBP, SEG, false>(p, q, v, seg, fpar, A, B, *p.view, 0, 0); break;
            }
        }
    }
    __syncthreads();   // the buffers are free for what follows
}

// The sums of one tile over the base views [v0, v1)
template <bool FAN, bool FBP, int SEG, int VB, int MODE>
__device__ __forceinline__ void tile_sums(const BwdParams &p, int tx, int ty, int v0, int v1, float (&A)[8],
                                          float (&B)[8], TiledSmem<FAN, SEG, VB> &sm)
{
    const int Q = p.g.P / 4;
#pragma unroll
    for (int j = 0; j < 8; ++j) A[j] = B[j] = 0.0f;
    int turn = v0 / Q;
    for (int v = v0; v < v1; ++turn) {
        const int e = min(v1, (turn + 1) * Q);
        quarter_sums<FAN, FBP, SEG, VB, MODE>(p, tx, ty, v, e, turn * Q, A, B, sm);
        v = e;
        rotate_sums(A);
        rotate_sums(B);
    }
    for (; (turn & 3) != 0; ++turn) {   // a full turn: each image's sums are back in its place
        rotate_sums(A);
        rotate_sums(B);
    }
}

// A tile's sums by image and pixel, for the stores: a row of 16 pixels and one
// of padding, so that rows and columns are read without bank conflicts.
constexpr int kBwdRow = kBwdTile + 1;
using TileSums = float[8][kBwdTile * kBwdRow];
constexpr int kBwdValues = 8 * kBwdTile * kBwdTile;

// this thread's slot of pixel x (pixel x + 1 is the next)
__device__ __forceinline__ int own_slot()
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int lx = (warp & 1) * 8 + ((lane >> 3) & 1) * 4 + (lane & 1) * 2;
    const int ly = (warp >> 1) * 8 + (lane >> 4) * 4 + ((lane >> 1) & 3);
    return ly * kBwdRow + lx;
}

// image and pixel of value e: consecutive values are consecutive pixels of an
// image row, which runs along x for even images and along y for odd ones
__device__ __forceinline__ void value_of(int e, int &j, int &lx, int &ly)
{
    j = e / (kBwdTile * kBwdTile);
    const int a = e % kBwdTile, b = e / kBwdTile % kBwdTile;
    lx = (j & 1) ? b : a;
    ly = (j & 1) ? a : b;
}

// image j of octant pixel (x, y), if the pixel is one and the image its own
// (the centre pixel's four images are one pixel, which image 3 is kept for)
__device__ __forceinline__ void write_image(const BwdParams &p, float *__restrict__ img, int x, int y, int j, float sum)
{
    const Geo &g = p.g;
    if (x > g.half || y > x || (j >= 4 && (y == 0 || y == x)) || (x == 0 && j != 3)) return;
    int gx, gy;
    image_of(j, x, y, gx, gy);
    const float val = sum * p.scale;
    img[(size_t)(gy + g.h2) * g.n + (gx + g.h2)] = val / g.effRate;
}

// base views of part s of S
__device__ __forceinline__ int part_begin(int nv, int s, int S) { return (int)((long long)nv * s / S); }

__device__ __forceinline__ void zero_axes(const BwdParams &p, float *__restrict__ img)
{
    for (int i = threadIdx.x; i < p.g.n; i += blockDim.x) {
        img[i] = 0.0f;
        img[(size_t)i * p.g.n] = 0.0f;
    }
}

// Staged backprojection, one tile per cluster of p.split blocks, each block
// the views of its part.  The parts' sums meet in distributed shared memory:
// every block adds up its share of the tile's pixel images over the parts, in
// the parts' order, and writes it, sixteen pixels of an image row at a time
// (the caller's image may be page-locked host memory, where scattered words
// cost a bus transaction each).
template <bool FAN, bool FBP, int SEG, int VB, int MODE>
__global__ void __launch_bounds__(kBwdThreads, CTPRJ_BWD_MINBLOCKS)
k_backward_tiled(const BwdParams p, float *__restrict__ img)
{
    __shared__ union {
        TiledSmem<FAN, SEG, VB> st;
        TileSums sums;
    } sm;
    const int S = p.split, tile = blockIdx.x / S, s = blockIdx.x % S;
    if (p.zero_axes && blockIdx.x == 0) zero_axes(p, img);
    int tx, ty;
    decode_tile(tile, tx, ty);
    float A[8], B[8];
    tile_sums<FAN, FBP, SEG, VB, MODE>(p, tx, ty, part_begin(p.nv, s, S), part_begin(p.nv, s + 1, S), A, B, sm.st);
    const int own = own_slot();
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        sm.sums[j][own] = A[j];
        sm.sums[j][own + 1] = B[j];
    }
    namespace cg = cooperative_groups;
    cg::cluster_group cl = cg::this_cluster();
    if (S > 1) cl.sync();
    else __syncthreads();
    for (int e = s * (kBwdValues / S) + threadIdx.x; e < (s + 1) * (kBwdValues / S); e += kBwdThreads) {
        int j, lx, ly;
        value_of(e, j, lx, ly);
        float *v = &sm.sums[j][ly * kBwdRow + lx];
        float sum = S > 1 ? *cl.map_shared_rank(v, 0) : *v;
        for (int q = 1; q < S; ++q) sum += *cl.map_shared_rank(v, q);
        write_image(p, img, tx * kBwdTile + lx, ty * kBwdTile + ly, j, sum);
    }
    if (S > 1) cl.sync();   // a block's sums stay until every block has read them
}

// One tile by one block, for the persistent launches: the parts one after the
// other, added in the same order.
template <bool FAN, bool FBP, int SEG, int VB, int MODE>
__device__ __forceinline__ void backward_tile(const BwdParams &p, int tile, float *__restrict__ img,
                                              TiledSmem<FAN, SEG, VB> &sm, TileSums &sums)
{
    const int S = p.split;
    if (p.zero_axes && tile == 0) zero_axes(p, img);
    int tx, ty;
    decode_tile(tile, tx, ty);
    const int own = own_slot();
    for (int s = 0; s < S; ++s) {
        float A[8], B[8];
        tile_sums<FAN, FBP, SEG, VB, MODE>(p, tx, ty, part_begin(p.nv, s, S), part_begin(p.nv, s + 1, S), A, B, sm);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            sums[j][own] = s == 0 ? A[j] : sums[j][own] + A[j];
            sums[j][own + 1] = s == 0 ? B[j] : sums[j][own + 1] + B[j];
        }
    }
    __syncthreads();
    for (int e = threadIdx.x; e < kBwdValues; e += kBwdThreads) {
        int j, lx, ly;
        value_of(e, j, lx, ly);
        write_image(p, img, tx * kBwdTile + lx, ty * kBwdTile + ly, j, sums[j][ly * kBwdRow + lx]);
    }
}

static BwdParams bwd_params(const ctprj_plan *pl, int fbp, float scale)
{
    BwdParams p;
    p.g = pl->g;
    p.nv = pl->nv;
    const int T = (pl->g.half + 1 + kBwdTile - 1) / kBwdTile;
    p.tiles_side = T;
    p.zero_axes = (pl->g.n % 2 == 0);
    p.scale = fbp ? (float)((double)(kRefPiF / (float)pl->g.np) / pl->g.dSize / pl->g.dSize)
                  : scale;
    p.view = pl->d_bview;
    p.det = pl->d_det;
    p.invd = pl->g.fan ? 1.0 / pl->g.d : 0.0;
    p.cG = pl->g.fan ? (float)(pl->g.dSize / pl->g.d) : 0.0f;
    p.invG = (float)(pl->g.fan ? pl->g.d / pl->g.dSize : 1.0 / pl->g.dSize);
    p.split = pl->bwd_split > 0 ? pl->bwd_split : 1;
    p.mode = pl->g.effRate == 1.0f ? kBwdUnit : (pl->g.effRate < 1.0f ? kBwdNarrow : kBwdRange);
    p.Wp = pl->g.W + 2 * kBwdTablePad;
    p.samp = pl->d_samp;
    p.foot = pl->d_foot;
    return p;
}

// widest tile shadow of the plan's geometry, in detectors (plan creation)
int backward_max_span(const ctprj_plan *pl, int *max_span)
{
    const BwdParams p = bwd_params(pl, 0, 1.0f);
    const int tiles = p.tiles_side * (p.tiles_side + 1) / 2;
    int *d = (int *)pl->d_count;   // zero since the upload
    int st;
    k_tile_span_max<<<296, 256>>>(p, tiles, d);
    if (!(st = cuda_error(cudaGetLastError(), "span launch")))
        st = cuda_error(cudaMemcpy(max_span, d, sizeof(int), cudaMemcpyDeviceToHost), "span readback");
    return st;
}

// Parts the staged backprojection sums a plan's base views in: a cluster of as
// many blocks per tile.  A small image has fewer tiles than the GPU holds blocks
// (36 at 256^2 against 740), so its views are split to fill it; beyond one
// wave a split evens out the last one.  The cost of a split weighs both: waves
// of blocks (the last one half used on average) per part, and 2.5 % per part
// for the blocks' start and the sums' meeting.  Measured, split 1 / 2 / 4 / 8:
// 256^2 parallel 55 / 35 / 27 / 19 us, 512^2 fan 115 / 84 / 70 / 77,
// 1024^2 fan 453 / 451 / 443 / 443, 2048^2 fan 3114 / 3006 / 3113 / 3171.
int backward_split(const ctprj_plan *pl)
{
    const int T = (pl->g.half + 1 + kBwdTile - 1) / kBwdTile, tiles = T * (T + 1) / 2;
    int sms = 148, best = 1;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, pl->device);
    const double slots = (double)CTPRJ_BWD_MINBLOCKS * sms;
    double cost = 0.0;
    for (int S = 1; S <= 8 && pl->nv >= 4 * S; S *= 2) {
        const double x = tiles * S / slots, c = (x <= 1.0 ? 1.0 : x + 0.5) / S * (1.0 + 0.025 * S);
        if (S == 1 || c < cost) {
            cost = c;
            best = S;
        }
    }
    return best;
}

// The tables of the staged backprojection in `mem`: the sample image (zero
// beyond the detectors) and, for fan beam, the rays' footprints.
size_t backward_table_bytes(const Geo &g)
{
    return sizeof(float4) * (size_t)(g.W + 2 * kBwdTablePad) * (size_t)(g.P / 4) * (g.fan ? 3 : 2);
}

int backward_tables(ctprj_plan *pl, float4 *mem)
{
    const BwdParams p = bwd_params(pl, 0, 1.0f);
    const size_t samples = 2 * (size_t)(pl->g.P / 4) * p.Wp;
    int st;
    pl->d_samp = mem;
    if ((st = cuda_error(cudaMemsetAsync(mem, 0, sizeof(float4) * samples, 0), "sample image"))) return st;
    if (pl->g.fan) {
        pl->d_foot = mem + samples;
        const int Q = pl->g.P / 4;
        k_footprints<<<dim3((p.Wp + 255) / 256, Q < 32768 ? Q : 32768), 256>>>(p, pl->d_foot);
        st = cuda_error(cudaGetLastError(), "footprint table");
    }
    return st;
}

static void launch_samples(const BwdParams &p, const float *sino, cudaStream_t s)
{
    const int Q = p.g.P / 4;
    k_samples<<<dim3((p.g.W + kSampThreads - 1) / kSampThreads, Q < 32768 ? Q : 32768), kSampThreads, 0, s>>>(p, sino);
}

template <bool FAN, bool FBP, int SEG, int VB, int MODE>
static cudaError_t launch_tiled_t(const BwdParams &p, int tiles, float *img, cudaStream_t s)
{
    return launch_after_table(k_backward_tiled<FAN, FBP, SEG, VB, MODE>, dim3(tiles * p.split), kBwdThreads, p.split, s,
                              p, img);
}

template <bool FAN, bool FBP, int SEG, int VB>
static cudaError_t launch_tiled_mode(const BwdParams &p, int tiles, float *img, cudaStream_t s)
{
    if (p.mode == kBwdRange) return launch_tiled_t<FAN, FBP, SEG, VB, kBwdRange>(p, tiles, img, s);
    if (p.mode == kBwdNarrow) return launch_tiled_t<FAN, FBP, SEG, VB, kBwdNarrow>(p, tiles, img, s);
    return launch_tiled_t<FAN, FBP, SEG, VB, kBwdUnit>(p, tiles, img, s);
}

template <int SEG, int VB>
static cudaError_t launch_tiled(const BwdParams &p, int fbp, int tiles, float *img, cudaStream_t s)
{
    // the FBP distance weight is a fan's: parallel beam takes the plain kernel
    if (!p.g.fan) return launch_tiled_mode<false, false, SEG, VB>(p, tiles, img, s);
    return fbp ? launch_tiled_mode<true, true, SEG, VB>(p, tiles, img, s)
               : launch_tiled_mode<true, false, SEG, VB>(p, tiles, img, s);
}

int launch_backward(const ctprj_plan *pl, const float *sino, float *img, int fbp,
                    unsigned long long *counter, cudaStream_t s, float scale)
{
    const BwdParams p = bwd_params(pl, fbp, scale);
    const int T = p.tiles_side;
    dim3 grid(T * (T + 1) / 2), block(kBwdTile * kBwdTile);
    const bool fan = pl->g.fan != 0;
    if (counter) {
        if (fan) k_backward<true, true, false><<<grid, block, 0, s>>>(p, sino, img, counter);
        else k_backward<false, true, false><<<grid, block, 0, s>>>(p, sino, img, counter);
    } else if (pl->bwd_seg == 0) {
        if (fbp) {
            if (fan) k_backward<true, false, true><<<grid, block, 0, s>>>(p, sino, img, counter);
            else k_backward<false, false, true><<<grid, block, 0, s>>>(p, sino, img, counter);
        } else {
            if (fan) k_backward<true, false, false><<<grid, block, 0, s>>>(p, sino, img, counter);
            else k_backward<false, false, false><<<grid, block, 0, s>>>(p, sino, img, counter);
        }
    } else {
        launch_samples(p, sino, s);
        const cudaError_t e = pl->bwd_seg <= 32 ? launch_tiled<32, 8>(p, fbp, (int)grid.x, img, s)
                                                : launch_tiled<64, 4>(p, fbp, (int)grid.x, img, s);
        if (e != cudaSuccess) return cuda_error(e, "backward launch");
    }
    return cuda_error(cudaGetLastError(), "backward launch");
}

// ------------------------------------------------------------ batched launches
//
// One persistent launch serves a batch of slices of different geometries: each
// block repeatedly takes the next work item from a device counter -- a forward
// block (V views x 32 rays) or a backprojection tile of some slice -- finds its
// slice by binary search over the item prefix sums, and runs the same block
// body as the per-slice kernels.  Work is handed out in the slice order the
// host chose (e.g. largest slices first), so the tail of the launch is short.

__device__ __forceinline__ int find_slot(const long long *prefix, int n, long long item)
{
    int lo = 0, hi = n;
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (prefix[mid] <= item) lo = mid;
        else hi = mid;
    }
    return lo;
}

__device__ __forceinline__ long long next_item(unsigned long long *counter, long long *slot)
{
    __syncthreads();
    if (threadIdx.x == 0) *slot = (long long)atomicAdd(counter, 1ULL);
    __syncthreads();
    return *slot;
}

__global__ void __launch_bounds__(256) k_quad_batch(const BatchArgs a)
{
    __shared__ float tz[32][33], tw[32][33];
    for (long long e = blockIdx.x; e < a.ttotal; e += gridDim.x) {
        const int i = find_slot(a.tprefix, a.nslices, e);
        const BatchSlice &sl = a.slices[i];
        quad_tile(sl.img, sl.quad, sl.fp.g.n, (int)(e - a.tprefix[i]), tz, tw);
    }
}

// resident blocks asked of the register allocator: as many warps per SM as the
// per-plan forward
template <int V>
__global__ void __launch_bounds__(32 * V, 4 * CTPRJ_FWD_MINBLOCKS / V) k_forward_batch(const BatchArgs a)
{
    __shared__ long long slot;
    __shared__ float parts[fwd_part_floats(V)];
    for (;;) {
        const long long item = next_item(a.counter, &slot);
        if (item >= a.total) return;
        const int i = find_slot(a.prefix, a.nslices, item);
        const BatchSlice &sl = a.slices[a.order[i]];
        const int local = (int)(item - a.prefix[i]);
        const int gx = (sl.fp.nb + V - 1) / V;
        const int bx = local % gx, by = local / gx;
        if (sl.fp.g.fan)
            forward_rays<true, kModePlain, V, kAllParts>(sl.fp, bx, by, sl.quad, sl.sino, nullptr, nullptr, nullptr, parts);
        else
            forward_rays<false, kModePlain, V, kAllParts>(sl.fp, bx, by, sl.quad, sl.sino, nullptr, nullptr, nullptr, parts);
    }
}

// the sample images of every staged slice: item = a row of a slice
__global__ void __launch_bounds__(kSampThreads) k_samples_batch(const BatchArgs a)
{
    for (long long e = blockIdx.x; e < a.stotal; e += gridDim.x) {
        const int i = find_slot(a.sprefix, a.nslices, e);
        const BatchSlice &sl = a.slices[i];
        sample_row<false>(sl.bp, sl.bsino, (int)(e - a.sprefix[i]), threadIdx.x, kSampThreads);
    }
}

// shared memory of a persistent backprojection block, for either beam
template <int SEG, int VB>
struct BatchSmem {
    union {
        TiledSmem<true, SEG, VB> fan;
        TiledSmem<false, SEG, VB> par;
    } st;
    TileSums sums;
};

// one tile of a batch slice
template <int SEG, int VB, bool LIVE>
__device__ __forceinline__ void batch_tile(const BatchSlice &sl, int tile, BatchSmem<SEG, VB> &sm)
{
    const BwdParams &p = sl.bp;
    if (!sl.tiled) {
        if (p.g.fan) backward_tile_direct<true, LIVE>(p, tile, sl.bsino, sl.bimg);
        else backward_tile_direct<false, LIVE>(p, tile, sl.bsino, sl.bimg);
    } else if (p.g.fan) {
        if (p.mode == kBwdUnit) backward_tile<true, false, SEG, VB, kBwdUnit>(p, tile, sl.bimg, sm.st.fan, sm.sums);
        else if (p.mode == kBwdNarrow) backward_tile<true, false, SEG, VB, kBwdNarrow>(p, tile, sl.bimg, sm.st.fan, sm.sums);
        else backward_tile<true, false, SEG, VB, kBwdRange>(p, tile, sl.bimg, sm.st.fan, sm.sums);
    } else {
        if (p.mode == kBwdUnit) backward_tile<false, false, SEG, VB, kBwdUnit>(p, tile, sl.bimg, sm.st.par, sm.sums);
        else if (p.mode == kBwdNarrow) backward_tile<false, false, SEG, VB, kBwdNarrow>(p, tile, sl.bimg, sm.st.par, sm.sums);
        else backward_tile<false, false, SEG, VB, kBwdRange>(p, tile, sl.bimg, sm.st.par, sm.sums);
    }
}

template <int SEG, int VB>
__global__ void __launch_bounds__(kBwdThreads, CTPRJ_BWD_MINBLOCKS) k_backward_batch(const BatchArgs a)
{
    extern __shared__ __align__(16) unsigned char batch_smem[];
    BatchSmem<SEG, VB> &sm = *reinterpret_cast<BatchSmem<SEG, VB> *>(batch_smem);
    __shared__ long long slot;
    for (;;) {
        const long long item = next_item(a.counter, &slot);
        if (item >= a.total) return;
        const int i = find_slot(a.prefix, a.nslices, item);
        const BatchSlice &sl = a.slices[a.order[i]];
        const int tile = (int)(item - a.prefix[i]);
        batch_tile<SEG, VB, false>(sl, tile, sm);
    }
}

// ------------------------------------------------- streaming backprojection
//
// A persistent backprojection whose inputs arrive while it runs: the host
// publishes slice i by setting ready[i] != 0 in host-mapped memory once its
// sinogram is on the device.  A block that takes a tile of slice i waits for
// that flag -- polling with __nanosleep -- for at most timeout_ns of
// %globaltimer time; past it, the slice is marked timed out (status[i] = 1),
// its remaining tiles are skipped by every block, and the host reports
// CTPRJ_ETIMEOUT.  No wait is unbounded and nothing traps, so the context stays
// usable after a timeout.

__device__ __forceinline__ unsigned long long global_ns()
{
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// Waits until word[0] reaches `want` (one thread), while the slice is not given
// up; past the deadline the slice is.  Returns whether the word got there.
__device__ __forceinline__ int wait_for(const volatile int *word, int want, int *status, unsigned long long timeout_ns)
{
    const unsigned long long t0 = global_ns();
    for (;;) {
        if (*word >= want) return 1;
        if (*(volatile int *)status != 0) return 0;
        if (global_ns() - t0 > timeout_ns) {
            atomicExch(status, 1);
            return 0;
        }
        __nanosleep(1000);
    }
}

// Items of slice i: its sample rows, then its tiles.  Both wait for the host's
// flag, a tile then also for the slice's rows, which blocks that are running have
// taken before it (items are handed out in order).  The host's limit is for the
// publication alone: the rows, which take microseconds once the flag is up, have
// at least kRowsNs.
constexpr unsigned long long kRowsNs = 2000000000ull;

template <int SEG, int VB>
__global__ void __launch_bounds__(kBwdThreads, CTPRJ_BWD_MINBLOCKS)
k_backward_stream(const BatchArgs a, const volatile int *__restrict__ ready, int *__restrict__ rows_done,
                  int *__restrict__ status, unsigned long long timeout_ns)
{
    extern __shared__ __align__(16) unsigned char batch_smem[];
    BatchSmem<SEG, VB> &sm = *reinterpret_cast<BatchSmem<SEG, VB> *>(batch_smem);
    __shared__ long long slot;
    __shared__ int go;
    for (;;) {
        const long long item = next_item(a.counter, &slot);
        if (item >= a.total + a.stotal) return;
        // items before slice position i: its tiles' and its sample rows' prefixes
        int lo = 0, hi = a.nslices;
        while (hi - lo > 1) {
            const int mid = (lo + hi) >> 1;
            if (a.prefix[mid] + a.oprefix[mid] <= item) lo = mid;
            else hi = mid;
        }
        const int i = lo, s = a.order[i];
        const BatchSlice &sl = a.slices[s];
        const int local = (int)(item - a.prefix[i] - a.oprefix[i]), rows = (int)(a.oprefix[i + 1] - a.oprefix[i]);
        const bool sample = local < rows;
        if (threadIdx.x == 0)
            go = ((volatile int *)status)[s] == 0 && wait_for(ready + s, 1, status + s, timeout_ns) &&
                 (sample || wait_for(rows_done + s, rows, status + s, timeout_ns > kRowsNs ? timeout_ns : kRowsNs));
        __syncthreads();
        if (!go) continue;
        __threadfence();   // the sinogram was published before the flag, the rows before their count
        if (sample) {
            sample_row<true>(sl.bp, sl.bsino, local, threadIdx.x, kBwdThreads);
            __threadfence();
            __syncthreads();
            if (threadIdx.x == 0) atomicAdd(&rows_done[s], 1);
        } else {
            batch_tile<SEG, VB, true>(sl, local - rows, sm);
        }
    }
}

template <int SEG, int VB, class K>
static int batch_kernel_smem(K kern)
{
    return cuda_error(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                           (int)sizeof(BatchSmem<SEG, VB>)), "batch shared memory");
}

template <int SEG, int VB>
static int launch_stream_t(const BatchArgs &a, int ctas, const int *ready, int *rows_done, int *status,
                           unsigned long long timeout_ns, cudaStream_t s)
{
    const int st = batch_kernel_smem<SEG, VB>(k_backward_stream<SEG, VB>);
    if (st) return st;
    k_backward_stream<SEG, VB><<<ctas, kBwdThreads, sizeof(BatchSmem<SEG, VB>), s>>>(a, ready, rows_done, status,
                                                                                      timeout_ns);
    return cuda_error(cudaGetLastError(), "streaming backward launch");
}

int launch_backward_stream(const BatchArgs &a, int seg, int vb, int ctas, const int *ready, int *rows_done,
                           int *status, unsigned long long timeout_ns, cudaStream_t s)
{
    if (seg > 32) return launch_stream_t<64, 4>(a, ctas, ready, rows_done, status, timeout_ns, s);
    return vb == 16 ? launch_stream_t<32, 8>(a, ctas, ready, rows_done, status, timeout_ns, s)
                    : launch_stream_t<32, 4>(a, ctas, ready, rows_done, status, timeout_ns, s);
}

int launch_quad_batch(const BatchArgs &a, cudaStream_t s)
{
    const long long blocks = a.ttotal < 65536 ? a.ttotal : 65536;
    k_quad_batch<<<(int)(blocks > 0 ? blocks : 1), dim3(32, 8), 0, s>>>(a);
    return cuda_error(cudaGetLastError(), "batched quad image launch");
}

int launch_forward_batch(const BatchArgs &a, int views, int ctas, cudaStream_t s)
{
    switch (views) {
    case 2: k_forward_batch<2><<<ctas, 64, 0, s>>>(a); break;
    case 8: k_forward_batch<8><<<ctas, 256, 0, s>>>(a); break;
    default: k_forward_batch<4><<<ctas, 128, 0, s>>>(a); break;
    }
    return cuda_error(cudaGetLastError(), "batched forward launch");
}

template <int SEG, int VB>
static int launch_backward_batch_t(const BatchArgs &a, int ctas, cudaStream_t s)
{
    const int st = batch_kernel_smem<SEG, VB>(k_backward_batch<SEG, VB>);
    if (st) return st;
    if (a.stotal > 0) k_samples_batch<<<(int)(a.stotal < 65536 ? a.stotal : 65536), kSampThreads, 0, s>>>(a);
    k_backward_batch<SEG, VB><<<ctas, kBwdThreads, sizeof(BatchSmem<SEG, VB>), s>>>(a);
    return cuda_error(cudaGetLastError(), "batched backward launch");
}

int launch_backward_batch(const BatchArgs &a, int seg, int vb, int ctas, cudaStream_t s)
{
    if (seg > 32) return launch_backward_batch_t<64, 4>(a, ctas, s);
    return vb == 16 ? launch_backward_batch_t<32, 8>(a, ctas, s) : launch_backward_batch_t<32, 4>(a, ctas, s);
}

template <int SEG, int VB>
static cudaError_t batch_occupancy(int *per_sm)
{
    if (batch_kernel_smem<SEG, VB>(k_backward_batch<SEG, VB>)) return cudaGetLastError();
    return cudaOccupancyMaxActiveBlocksPerMultiprocessor(per_sm, k_backward_batch<SEG, VB>, kBwdThreads,
                                                         sizeof(BatchSmem<SEG, VB>));
}

// resident blocks per SM of a batched kernel: kind 0 forward (param = views),
// kind 1 backward (param = seg * 100 + views in its two staging buffers)
int batch_max_ctas(int kind, int param, int *per_sm)
{
    cudaError_t e;
    if (kind == 0) {
        if (param == 2) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(per_sm, k_forward_batch<2>, 64, 0);
        else if (param == 8) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(per_sm, k_forward_batch<8>, 256, 0);
        else e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(per_sm, k_forward_batch<4>, 128, 0);
    } else {
        if (param == 3216) e = batch_occupancy<32, 8>(per_sm);
        else if (param == 3208) e = batch_occupancy<32, 4>(per_sm);
        else e = batch_occupancy<64, 4>(per_sm);
    }
    return cuda_error(e, "occupancy query");
}

FwdParams make_fwd_params(const ctprj_plan *pl) { return fwd_params(pl); }
BwdParams make_bwd_params(const ctprj_plan *pl) { return bwd_params(pl, 0, 1.0f); }

}  // namespace ctprj

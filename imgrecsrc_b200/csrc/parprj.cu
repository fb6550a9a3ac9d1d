// parprj.cu -- the double-precision masked parallel-beam operator (mParPrj)
// on the GPU.
//
// Same operator as prj/parPrj.c: for angle theta (degrees) and a masked pixel
// at column-major index m of an nr x nc image, x = m / nr - nc/2 and
// y = m % nr - nr/2, dist = x cos + y sin, and detector k (unit pitch, centred
// at max(nc, nr)/2) receives the overlap of its beam [k - bw/2, k + bw/2] with
// the pixel's trapezoid footprint.  The reference forms that footprint from the
// angle |trunc(fmod(theta, 90) - 45)| in whole degrees (prj/parPrj.c:111 passes
// a double to the integer abs()) with pi = 3.14159265; the view table below is
// built on the host the same way, and the overlap uses the reference's
// piecewise formula including its value when the beam is wider than the whole
// footprint (prj/parPrj.c:133-168).  Detectors with k + centre outside
// [0, nc) are skipped as in the reference (prj/parPrj.c:170), and also those
// beyond prjWidth, which the reference would write past its row.
//
//  forward   from a dense copy of the masked image, so that the sum does not
//            depend on the order in which the mask lists its pixels.  Lines of
//            the image (rows where the angle's band is closer to the columns,
//            else columns) are taken in turn, the pixels of a line from the
//            copy in which they are contiguous.  With unit beams a lane owns a
//            detector edge (edge_lines below); otherwise a detector whose
//            pixels it weighs one by one.
//            No atomics on sums: results repeat bit for bit.
//  backward  one thread (or eight) per masked pixel, gathering over angles and
//            detectors; no atomics.
#include <climits>
#include <cmath>
#include <cstring>
#include <mutex>
#include <vector>

#include "ctprj_internal.h"
#include "../../include/parprj.h"

namespace ctprj {

struct ParView {
    double c, s, height, b1, b2, areaT, areaR;
    double inv_s, inv_c;   // 1 / s and 1 / c, 0 where zero
    double half, ramp;     // half the footprint's area; height / (2 (b2 - b1))
    int edges;             // 1: the edge form below holds (bw = 1, 1/2 <= b2, b1 < b2)
    int box;               // 1: and the footprint has next to no ramps
};

struct ParArgs {
    double bw;
    int nc, nr, np, W, xC, yC, pC;
    int parts;             // warps (thread groups) that share a detector's (pixel's) sum
    const ParView *view;
};

constexpr double kParPi = 3.14159265;   // prj/parPrj.c:29
constexpr double kParEps = 1e-8;        // prj/parPrj.h:8

static ParView par_view(double theta, double bw)
{
    ParView v;
    int whole = (int)(fmod(theta, 90) - 45);
    if (whole < 0) whole = -whole;
    const double tmp = whole * kParPi / 180;
    v.height = 1 / sin(tmp + kParPi / 4);
    v.b1 = sqrt(2.0) / 2 * sin(tmp);
    v.b2 = sqrt(2.0) / 2 * cos(tmp);
    v.areaT = 0.5 * v.height * (v.b2 - v.b1);
    v.areaR = v.height * v.b1 * 2;
    v.c = cos(theta * kParPi / 180);
    v.s = sin(theta * kParPi / 180);
    v.inv_s = v.s != 0.0 ? 1.0 / v.s : 0.0;
    v.inv_c = v.c != 0.0 ? 1.0 / v.c : 0.0;
    v.half = v.areaT + 0.5 * v.areaR;
    v.ramp = 0.5 * v.height / (v.b2 - v.b1);
    // (negative angles get footprints with b2 < b1 from the truncated angle:
    // those keep the reference's piecewise formula)
    // (the pixels of a line are at least b2 <= sqrt(1/2) apart, as edge_lines counts on)
    v.edges = bw == 1.0 && v.b2 > v.b1 && v.b2 >= 0.5 && fmax(fabs(v.c), fabs(v.s)) >= v.b2 - 1e-12;
    v.box = v.edges && v.b2 - v.b1 < 1e-6;
    return v;
}

__device__ __forceinline__ double sq(double a) { return a * a; }

// distance of pixel (px, py) from the central ray of angle v (prj/parPrj.c:123),
// one rounding order for both directions
__device__ __forceinline__ double par_dist(const ParView &v, int px, int py)
{
    return fma((double)py, v.s, (double)px * v.c);
}

// overlap of the beam of detector k with the footprint centred at dist, by the
// zones of the beam's two edges (prj/parPrj.c:133-168)
__device__ __forceinline__ double par_overlap(const ParView &v, double dist, double k, double bw)
{
    const double hb = bw / 2, w = v.b2 - v.b1, H = v.height;
    const double ul = k - hb - dist, ur = k + hb - dist;
    const double aT = v.areaT, aR = v.areaR;
    if (ul <= -v.b2) {
        if (ur <= -v.b1) return aT * sq((ur + v.b2) / w);
        if (ur <= v.b1) return aT + H * (ur + v.b1);
        return aT * 2 + aR - aT * sq((v.b2 - ur) / w);
    }
    if (ul <= -v.b1) {
        const double rise = aT * (1 - sq((ul + v.b2) / w));
        if (ur <= -v.b1) return H / w * (k - dist + v.b2) * bw;
        if (ur <= v.b1) return rise + H * (ur + v.b1);
        if (ur <= v.b2) return rise + aR + aT * (1 - sq((v.b2 - ur) / w));
        return rise + aR + aT;
    }
    if (ul <= v.b1) {
        if (ur <= v.b1) return H * bw;
        if (ur <= v.b2) return H * (v.b1 - ul) + aT * (1 - sq((v.b2 - ur) / w));
        return H * (v.b1 - ul) + aT;
    }
    if (ur <= v.b2) return H / w * (dist + v.b2 - k) * bw;
    return 0.5 * H / w * sq(dist + v.b2 - k + hb);
}

constexpr int kParThreads = 256;

// the masked pixel values in a dense nr x nc image, column-major (ximg) and
// row-major (ximgT), zero elsewhere.  A pixel listed twice in the mask holds
// the sum of its values; indices outside the image are not projected.
__global__ void k_par_scatter(const double *__restrict__ x, const double *__restrict__ mask,
                              long long npix, int nr, int nc, double *__restrict__ ximg,
                              double *__restrict__ ximgT)
{
    const long long nimg = (long long)nr * nc;
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < npix;
         i += (long long)gridDim.x * blockDim.x) {
        const long long m = (long long)mask[i];
        if (m >= 0 && m < nimg) {
            atomicAdd(&ximg[m], x[i]);
            atomicAdd(&ximgT[(m % nr) * nc + m / nr], x[i]);
        }
    }
}

// The edge form.  With bw = 1 the beams tile the detector and a beam is never
// wider than the footprint (2 b2 >= 1), so the reference's overlap is the
// footprint's area between the beam's two edges, and neighbouring detectors
// share an edge.  par_area(u): that area from the footprint's centre to u, odd
// in u, without branches: with z = |u|, half the area less what lies beyond z,
// which is quadratic on the falling ramp and linear on the plateau.  The
// reference also leaves out a detector whose beam reaches less than 1e-8 into a
// footprint (prj/parPrj.c:124-125).  That sliver weighs below 1e-14 unless the
// footprint is a box (angles that are multiples of 90 degrees); there the edge of
// a beam that is left out counts as outside the footprint.
__device__ __forceinline__ double par_area(const ParView &v, double u)
{
    const double z = fabs(u), q = v.b2 - z;
    const double r = q < 0.0 ? 0.0 : q;
    const double rest = z < v.b1 ? fma(v.height, v.b1 - z, v.areaT) : v.ramp * r * r;
    return copysign(v.half - rest, u);
}

// sum of w * x over the pixels that reach detector kk, added to acc: the
// pixel's own range test (prj/parPrj.c:124-125) and weight (:133-168).  Lines as
// the edge form takes them; the pixels of one that can reach the detector are
// bracketed from |dist - k| <= b2 + bw/2 with a margin.
__device__ __forceinline__ double par_gather(const ParArgs &a, const ParView &v, double k, const double *__restrict__ ximg,
                                             const double *__restrict__ ximgT, double acc)
{
    const bool rows = fabs(v.s) < fabs(v.c);   // the band is closer to the columns
    const double hw = v.b2 + a.bw / 2 + 1e-6;
    const double across = rows ? v.s : v.c, inv = rows ? v.inv_c : v.inv_s;
    const int lines = rows ? a.nr : a.nc, lmid = rows ? a.yC : a.xC;
    const int len = rows ? a.nc : a.nr, mid = rows ? a.xC : a.yC;
    const double *line = (rows ? ximgT : ximg) + mid;
#pragma unroll 1
    for (int l = -lmid; l < lines - lmid; ++l, line += len) {
        const double o = (double)l * across;
        const double r0 = (k - hw - o) * inv, r1 = (k + hw - o) * inv;
        const int q0 = (int)ceil(fmax(fmin(r0, r1), (double)-mid));
        const int q1 = (int)floor(fmin(fmax(r0, r1), (double)(len - 1 - mid)));
#pragma unroll 1
        for (int q = q0; q <= q1; ++q) {
            const double xv = line[q];
            if (xv == 0.0) continue;
            const double dist = rows ? par_dist(v, q, l) : par_dist(v, l, q);
            const double ub = floor(dist + v.b2 + a.bw / 2 - kParEps);
            const double lb = ceil(dist - v.b2 - a.bw / 2 + kParEps);
            if (k < lb || k > ub) continue;
            const double w = par_overlap(v, dist, k, a.bw);
            if (w != 0.0) acc += w * xv;
        }
    }
    return acc;
}

// One warp of the forward: 32 detector edges kk0 - 1/2 + lane of angle v over
// the lines [l0, l1) of the image (rows where the band is closer to the columns,
// else columns), 31 detectors.  Per line, with q the pixel index along it in the
// direction of growing distance, q0 is the first pixel whose footprint's far end
// lies beyond lane e's edge: everything before it lies left of the edge.  Pixels
// are max(|c|, |s|) >= b2 apart (sqrt(1/2) lies between the two), so the edge cuts
// q0 and q0 + 1 at most, the latter left of its centre.  The mass left of the edge
// is that of the pixels before q0 plus S = sum x (area(edge - dist) + half), so
// detector k's share of the line is 2 half X + S(k + 1) - S(k), X the pixels
// between the two edges' q0 (one or two, at hand).  Summed over the lines before
// the lanes meet, so a pixel costs one area instead of two per detector that it
// might reach (3.3 on average).  Rounding may move q0 by one pixel; what that puts
// on the other side of the edge weighs the square of a rounding.
// Bound by the latency of the lines' loads (four lines on their way) and the FP64
// pipe: 512^2, 360 angles: pixel by pixel 1.57 ms, three areas a line 0.51, two
// 0.37; the backward, whose samples come from L2, 1.11 -> 0.31 ms (0.30 -> 0.27
// without local memory).  64^2, 40
// angles: 116 -> 27 and 71 -> 17 us.
// S: of the edge as a beam's left one; Sr: as the right one, which differs at box
// angles only.
template <bool ROWS, bool BOX>
__device__ __forceinline__ void edge_lines(const ParArgs &a, const ParView &v, int k, int l0, int l1,
                                           const double *__restrict__ img, double &S, double &Sr, double &X)
{
    // along a line: step per pixel (> 0 in q), offset per line
    const double along = ROWS ? v.c : v.s, across = ROWS ? v.s : v.c, inv = fabs(ROWS ? v.inv_c : v.inv_s);
    const int sg = along < 0.0 ? -1 : 1, len = ROWS ? a.nc : a.nr, mid = ROWS ? a.xC : a.yC, lmid = ROWS ? a.yC : a.xC;
    const double step = fabs(along), kMagic = 6755399441055744.0;   // 1.5 * 2^52: rounds to an integer
    // first pixel with dist > edge - b2: floor(t) + 1, t = (edge - b2 - offset) / step,
    // by the same arithmetic for an edge in every lane
    const double edge = (double)k - 0.5, full = 2.0 * v.half;
#pragma unroll 4
    for (int l = l0; l < l1; ++l) {
        const double e = fma(-(double)(l - lmid), across, edge);
        // floor(t) + 1, t = (e - b2) / step
        const double m = fma(e - v.b2, inv, -0.5) + kMagic;
        const int q0 = __double2loint(m) + 1, two = __shfl_down_sync(0xffffffffu, q0, 1) - q0;
        const double u0 = fma(-step, m - kMagic, e) - step, z1 = step - u0;   // u1 = -z1
        const double *line = img + (size_t)l * len;
        double x[2];
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            const int i = mid + sg * (q0 + j);
            x[j] = (unsigned)i < (unsigned)len ? __ldg(line + i) : 0.0;
        }
        // (an infinite pixel turns the sums of the edges near it into NaN:
        // the caller takes those detectors pixel by pixel)
        // par_area + half: |u0| <= b2 but for rounding, and u1 <= 0
        const double z0 = fabs(u0), r0 = v.b2 - z0, rest = z0 < v.b1 ? fma(v.height, v.b1 - z0, v.areaT) : v.ramp * r0 * r0;
        const double f0 = __double2hiint(u0) < 0 ? rest : full - rest;
        const double r1 = __double2hiint(v.b2 - z1) < 0 ? 0.0 : v.b2 - z1;
        const double f1 = z1 < v.b1 ? fma(v.height, v.b1 - z1, v.areaT) : v.ramp * r1 * r1;
        S = fma(BOX && u0 > v.b2 - kParEps ? full : f0, x[0], S);
        S = fma(f1, x[1], S);
        if (BOX) {
            Sr = fma(u0 < -v.b2 + kParEps ? 0.0 : f0, x[0], Sr);
            Sr = fma(-z1 < -v.b2 + kParEps ? 0.0 : f1, x[1], Sr);
        }
        X += two > 0 ? x[0] : 0.0;
        X += two > 1 ? x[1] : 0.0;
    }
}

// lines of the image that a detector of the warp can meet: offset + along * q
// = k has |q| <= len / 2 + 4 (every lane takes part)
__device__ __forceinline__ void clip_lines(double k, double along, double across, int half, int lines, int lmid, int &l0,
                                           int &l1)
{
    float lo = 0.0f, hi = (float)(lines - 1);
    if (fabs(across) > 1e-6) {
        const float r = (float)(fabs(along) * (half + 4)), ia = 1.0f / (float)across;
        const float p = ((float)k - r) * ia, q = ((float)k + r) * ia;
        lo = fmaxf(lo, fminf(p, q) + (float)lmid - 2.0f);
        hi = fminf(hi, fmaxf(p, q) + (float)lmid + 2.0f);
    }
    l0 = max(l0, __reduce_min_sync(0xffffffffu, lo <= hi ? __float2int_rd(lo) : INT_MAX));
    l1 = min(l1, __reduce_max_sync(0xffffffffu, lo <= hi ? __float2int_ru(hi) + 1 : INT_MIN));
}

constexpr int kParWarps = 4;

// y[it, kk] = (y[it, kk] + sum of w * x) / bw.  Block: 4 warps that take the
// detectors (a.parts = 1) or the lines (4: their sums meet in shared memory, in
// order) of one angle.
__global__ void __launch_bounds__(32 * kParWarps, 6)
k_par_forward(const ParArgs a, const double *__restrict__ ximg, const double *__restrict__ ximgT,
              double *__restrict__ y)
{
    __shared__ double sums[kParWarps][3][32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, it = blockIdx.y;
    const int parts = a.parts, part = warp % parts, group = blockIdx.x * (kParWarps / parts) + warp / parts;
    const ParView v = a.view[it];
    const int nd = min(a.W, a.nc);   // detectors with k + centre >= nc are skipped (prj/parPrj.c:170)
    const int kk = group * 31 + lane, k = kk - a.pC;
    double *yr = y + (size_t)it * a.W;
    double S = 0.0, Sr = 0.0, X = 0.0;
    if (v.edges) {
        const bool rows = fabs(v.s) < fabs(v.c);
        const int lines = rows ? a.nr : a.nc, lmid = rows ? a.yC : a.xC;
        int l0 = (int)((long long)lines * part / parts), l1 = (int)((long long)lines * (part + 1) / parts);
        clip_lines((double)k, rows ? v.c : v.s, rows ? v.s : v.c, max(a.xC, a.yC) + 1, lines, lmid, l0, l1);
        if (group * 31 < nd) {
            if (v.box) {
                if (rows) edge_lines<true, true>(a, v, k, l0, l1, ximgT, S, Sr, X);
                else edge_lines<false, true>(a, v, k, l0, l1, ximg, S, Sr, X);
            } else {
                if (rows) edge_lines<true, false>(a, v, k, l0, l1, ximgT, S, Sr, X);
                else edge_lines<false, false>(a, v, k, l0, l1, ximg, S, Sr, X);
                Sr = S;
            }
        }
    }
    if (parts > 1) {
        sums[warp][0][lane] = S;
        sums[warp][1][lane] = X;
        sums[warp][2][lane] = Sr;
        __syncthreads();
        if (part != 0) return;
        for (int q = 1; q < parts; ++q) {
            S += sums[warp + q][0][lane];
            X += sums[warp + q][1][lane];
            Sr += sums[warp + q][2][lane];
        }
    }
    const double Sn = __shfl_down_sync(0xffffffffu, Sr, 1);
    if (lane < 31 && kk < nd) {
        double r = yr[kk] + fma(2.0 * v.half, X, Sn - S);
        // no edge form with this beam; or a value that is not finite, which
        // must not reach the neighbours' sums
        if (!v.edges || !isfinite(r)) r = par_gather(a, v, (double)k, ximg, ximgT, yr[kk]);
        yr[kk] = r / a.bw;
    }
    if (group == 0)   // the detectors that are skipped
        for (int e = nd + lane; e < a.W; e += 32) yr[e] /= a.bw;
}

// x = (x + sum of w * y) / bw over angles and detectors.  EDGES: every angle has
// the edge form (the kernel then holds no division, whose calls would keep
// registers in local memory).  In the edge form a footprint is cut by the edges e1 and e2 of at most three detectors k0 .. k0 + 2
// (2 b2 + 1 <= 2.42); the outer edges lie outside it but for 1e-8.
__device__ __forceinline__ double par_back_angle(const ParArgs &a, const ParView &v, const double *__restrict__ row,
                                                 int px, int py, double acc)
{
    const double dist = par_dist(v, px, py);
    const double ub = floor(dist + v.b2 + a.bw / 2 - kParEps);
    const double lb = ceil(dist - v.b2 - a.bw / 2 + kParEps);
    for (int k = (int)lb; k <= ub; ++k) {
        if (k < -a.pC || k + a.pC >= a.nc || k + a.pC >= a.W) continue;
        const double w = par_overlap(v, dist, (double)k, a.bw);
        if (w != 0.0) acc += row[k + a.pC] * w;
    }
    return acc;
}

constexpr int kParViews = 64;

template <bool EDGES>
__global__ void __launch_bounds__(kParThreads, EDGES ? 0 : 3)
k_par_backward(const ParArgs a, const double *__restrict__ y, const double *__restrict__ mask,
               long long npix, double *__restrict__ x)
{
    __shared__ double part[kParThreads];
    __shared__ ParView views[kParViews];
    const int parts = a.parts, per = kParThreads / parts;
    const int p = threadIdx.x / per, t = threadIdx.x % per;
    const long long i = (long long)blockIdx.x * per + t;
    const bool live = i < npix;
    const int m = live ? (int)mask[i] : 0;
    const int px = m / a.nr - a.xC, py = m % a.nr - a.yC;
    const unsigned nd = (unsigned)min(a.W, a.nc);
    double acc = live && p == 0 ? x[i] : 0.0;
    // the views in turns of kParViews through shared memory, of which each part
    // takes a run
    for (int base = 0; base < a.np; base += kParViews) {
        const int n = min(kParViews, a.np - base);
        __syncthreads();
        const double *src = reinterpret_cast<const double *>(a.view + base);
        for (int e = threadIdx.x; e < n * (int)(sizeof(ParView) / sizeof(double)); e += kParThreads)
            reinterpret_cast<double *>(views)[e] = src[e];
        __syncthreads();
        const int q0 = n * p / parts, q1 = n * (p + 1) / parts;
        const double *row = y + (size_t)(base + q0) * a.W;
#pragma unroll 2
        for (int q = q0; q < q1; ++q, row += a.W) {
            const ParView &v = views[q];
            if (!EDGES && !v.edges) {
                if (live) acc = par_back_angle(a, v, row, px, py, acc);
                continue;
            }
            const double dist = par_dist(v, px, py);
            const double k0 = ceil(dist - v.b2 - 0.5 + kParEps);
            const int d0 = (int)k0 + a.pC;
            const double y0 = (unsigned)d0 < nd ? __ldg(row + d0) : 0.0;
            const double y1 = (unsigned)(d0 + 1) < nd ? __ldg(row + d0 + 1) : 0.0;
            const double y2 = (unsigned)(d0 + 2) < nd ? __ldg(row + d0 + 2) : 0.0;
            const double F1 = par_area(v, k0 + 0.5 - dist), F2 = par_area(v, k0 + 1.5 - dist);
            double w0 = F1 + v.half, w1 = F2 - F1, w2 = v.half - F2;
            if (v.box) {   // the outer edges may lie 1e-8 inside, and a sliver is left out
                const double e0 = k0 - 0.5 - dist, ub = floor(dist + v.b2 + 0.5 - kParEps);
                const double F0 = par_area(v, e0), F3 = par_area(v, e0 + 3.0);
                w0 = F1 - F0;
                if (k0 + 1.0 > ub) w1 = 0.0;
                w2 = k0 + 2.0 > ub ? 0.0 : F3 - F2;
                if (k0 > ub) w0 = 0.0;
            }
            if (w0 != 0.0) acc = fma(w0, y0, acc);
            if (w1 != 0.0) acc = fma(w1, y1, acc);
            if (w2 != 0.0) acc = fma(w2, y2, acc);
        }
    }
    if (parts > 1) {
        part[threadIdx.x] = acc;
        __syncthreads();
        if (p != 0) return;
        for (int q = 1; q < parts; ++q) acc += part[q * per + t];
    }
    if (live) x[i] = EDGES ? acc : acc / a.bw;   // (the edge form has bw = 1)
}

static int par_validate(const ctprj_par_conf *c, long long npix)
{
    if (!c) return set_error(CTPRJ_EINVAL, "NULL configuration");
    if (c->nc < 1 || c->nr < 1 || c->np < 0 || c->prjWidth < 1 || npix < 0 || !(c->bw > 0))
        return set_error(CTPRJ_EINVAL, "invalid parPrj configuration");
    if ((long long)c->np * c->prjWidth >= (1LL << 31) || npix >= (1LL << 31) ||
        (long long)c->nc * c->nr >= (1LL << 31))
        return set_error(CTPRJ_ERANGE, "parPrj sizes exceed 2^31");
    return CTPRJ_OK;
}

static ParArgs par_args(const ctprj_par_conf *c, const ParView *view)
{
    ParArgs a;
    a.bw = c->bw;
    a.nc = c->nc;
    a.nr = c->nr;
    a.np = c->np;
    a.W = c->prjWidth;
    a.xC = c->nc / 2;
    a.yC = c->nr / 2;
    a.pC = a.xC > a.yC ? a.xC : a.yC;
    a.view = view;
    return a;
}

// view table in stream-ordered device memory (released after the kernels)
static int par_table(const ctprj_par_conf *c, const double *theta, ParView **d_view, cudaStream_t s,
                     bool *edges = nullptr)
{
    std::vector<ParView> tab((size_t)(c->np > 0 ? c->np : 1));
    for (int it = 0; it < c->np; ++it) tab[it] = par_view(theta[it], c->bw);
    if (edges) {
        *edges = true;
        for (int it = 0; it < c->np; ++it) *edges = *edges && tab[it].edges;
    }
    int st = cuda_error(cudaMallocAsync((void **)d_view, sizeof(ParView) * tab.size(), s),
                        "parPrj view table");
    if (st) return st;
    return cuda_error(cudaMemcpyAsync(*d_view, tab.data(), sizeof(ParView) * tab.size(),
                                      cudaMemcpyHostToDevice, s),
                      "parPrj view upload");
}

static int sm_count()
{
    int dev = 0, sms = 148;
    if (cudaGetDevice(&dev) == cudaSuccess)
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    return sms;
}

}  // namespace ctprj

using namespace ctprj;

extern "C" int ctprj_par_forward(const ctprj_par_conf *conf, const double *theta_host,
                                 const double *d_mask, long long npix, const double *d_x,
                                 double *d_y, void *stream)
{
    int st = par_validate(conf, npix);
    if (st) return st;
    if (conf->np > 0 && (!theta_host || !d_y)) return set_error(CTPRJ_EINVAL, "NULL buffer");
    if (npix > 0 && (!d_mask || !d_x)) return set_error(CTPRJ_EINVAL, "NULL buffer");
    cudaStream_t s = (cudaStream_t)stream;
    if (conf->np == 0) return CTPRJ_OK;
    ParView *d_view = nullptr;
    double *d_img = nullptr;
    if ((st = par_table(conf, theta_host, &d_view, s))) return st;
    ParArgs a = par_args(conf, d_view);
    const size_t img_elems = (size_t)conf->nc * (size_t)conf->nr, img_bytes = 2 * sizeof(double) * img_elems;
    if (!(st = cuda_error(cudaMallocAsync((void **)&d_img, img_bytes, s), "parPrj dense image")) &&
        !(st = cuda_error(cudaMemsetAsync(d_img, 0, img_bytes, s), "parPrj dense image"))) {
        if (npix > 0) {
            const long long blocks = (npix + kParThreads - 1) / kParThreads;
            k_par_scatter<<<(int)(blocks < 8 * sm_count() ? blocks : 8 * sm_count()), kParThreads, 0, s>>>(
                d_x, d_mask, npix, conf->nr, conf->nc, d_img, d_img + img_elems);
            st = cuda_error(cudaGetLastError(), "parPrj scatter");
        }
        if (!st) {
            // a warp per 31 detectors and angle; few of them share each one's
            // lines among four warps (64^2, 64 angles: 192 warps)
            const int nd = conf->prjWidth < conf->nc ? conf->prjWidth : conf->nc, groups = (nd + 30) / 31;
            a.parts = (long long)groups * conf->np < 24LL * sm_count() ? kParWarps : 1;
            const int per = kParWarps / a.parts;
            for (int it0 = 0; it0 < conf->np && !st; it0 += 65535) {
                ParArgs b = a;
                b.view += it0;
                b.np = conf->np - it0 < 65535 ? conf->np - it0 : 65535;
                k_par_forward<<<dim3((groups + per - 1) / per, b.np), 32 * kParWarps, 0, s>>>(
                    b, d_img, d_img + img_elems, d_y + (size_t)it0 * conf->prjWidth);
                st = cuda_error(cudaGetLastError(), "parPrj forward");
            }
        }
    }
    if (d_img) cudaFreeAsync(d_img, s);
    cudaFreeAsync(d_view, s);
    return st;
}

extern "C" int ctprj_par_backward(const ctprj_par_conf *conf, const double *theta_host,
                                  const double *d_mask, long long npix, const double *d_y,
                                  double *d_x, void *stream)
{
    int st = par_validate(conf, npix);
    if (st) return st;
    if (npix == 0) return CTPRJ_OK;
    if (!d_mask || !d_x || (conf->np > 0 && (!theta_host || !d_y)))
        return set_error(CTPRJ_EINVAL, "NULL buffer");
    cudaStream_t s = (cudaStream_t)stream;
    ParView *d_view = nullptr;
    bool edges = false;
    if ((st = par_table(conf, theta_host, &d_view, s, &edges))) return st;
    ParArgs a = par_args(conf, d_view);
    // few pixels share each one's angles among eight threads
    a.parts = npix < 384LL * sm_count() ? 8 : 1;
    const int per = kParThreads / a.parts, blocks = (int)((npix + per - 1) / per);
    if (edges) k_par_backward<true><<<blocks, kParThreads, 0, s>>>(a, d_y, d_mask, npix, d_x);
    else k_par_backward<false><<<blocks, kParThreads, 0, s>>>(a, d_y, d_mask, npix, d_x);
    st = cuda_error(cudaGetLastError(), "parPrj backward");
    cudaFreeAsync(d_view, s);
    return st;
}

// ---------------------------------------------- prj/parPrj.h entry points

static std::mutex g_par_mu;
static double *g_img = nullptr, *g_prj = nullptr, *g_mask = nullptr;
static parConf g_opt;
static size_t g_tot = 0;
static bool g_conf_set = false;

extern "C" int parPrjConf(double *t_img, double *t_prj, double *t_maskIdx, parConf *t_opt,
                          size_t t_totPixels)
{
    std::lock_guard<std::mutex> lk(g_par_mu);
    g_img = t_img;
    g_prj = t_prj;
    g_mask = t_maskIdx;
    if (t_opt) g_opt = *t_opt;
    g_tot = t_totPixels;
    g_conf_set = t_opt != nullptr;
    return 0;
}

extern "C" int parPrjThread(void)
{
    std::lock_guard<std::mutex> lk(g_par_mu);
    if (!g_conf_set) return set_error(CTPRJ_ENOTSETUP, "parPrjConf() has not been called");
    const ctprj_par_conf c = {g_opt.bw, g_opt.nc, g_opt.nr, g_opt.np, g_opt.prjWidth};
    const long long npix = (long long)g_tot;
    int st = par_validate(&c, npix);
    if (st) return st;
    const size_t ny = (size_t)c.np * c.prjWidth;
    if ((npix > 0 && (!g_img || !g_mask)) || (ny > 0 && (!g_prj || !g_opt.theta)))
        return set_error(CTPRJ_EINVAL, "NULL buffer in the parPrj configuration");
    double *d_img = nullptr, *d_prj = nullptr, *d_mask = nullptr;
    cudaStream_t s = 0;
    if ((st = cuda_error(cudaMalloc((void **)&d_img, sizeof(double) * (npix ? npix : 1)), "parPrj buffers")) ||
        (st = cuda_error(cudaMalloc((void **)&d_prj, sizeof(double) * (ny ? ny : 1)), "parPrj buffers")) ||
        (st = cuda_error(cudaMalloc((void **)&d_mask, sizeof(double) * (npix ? npix : 1)), "parPrj buffers")))
        goto done;
    if ((npix && ((st = cuda_error(cudaMemcpy(d_img, g_img, sizeof(double) * npix, cudaMemcpyHostToDevice), "copy")) ||
                  (st = cuda_error(cudaMemcpy(d_mask, g_mask, sizeof(double) * npix, cudaMemcpyHostToDevice), "copy")))) ||
        (ny && (st = cuda_error(cudaMemcpy(d_prj, g_prj, sizeof(double) * ny, cudaMemcpyHostToDevice), "copy"))))
        goto done;
    if (g_opt.fwd) {
        if ((st = ctprj_par_forward(&c, g_opt.theta, d_mask, npix, d_img, d_prj, s))) goto done;
        if (ny) st = cuda_error(cudaMemcpy(g_prj, d_prj, sizeof(double) * ny, cudaMemcpyDeviceToHost), "copy back");
    } else {
        if ((st = ctprj_par_backward(&c, g_opt.theta, d_mask, npix, d_prj, d_img, s))) goto done;
        if (npix) st = cuda_error(cudaMemcpy(g_img, d_img, sizeof(double) * npix, cudaMemcpyDeviceToHost), "copy back");
    }
done:
    cudaFree(d_img);
    cudaFree(d_prj);
    cudaFree(d_mask);
    return st;
}

extern "C" int parPrjRun(void) { return parPrjThread(); }

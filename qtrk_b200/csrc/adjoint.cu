// Differentiable Z-LUT match: the radial-profile-to-LUT cost, its adjoint (gradients with respect to
// the bead position (x, y, z) and to the LUT entries), and the joint Gauss-Newton (x, y, z)
// refinement that runs after the Z fit in the LT_B200_JointRefine mode. No counterpart in the
// reference; the cost is built from the reference's own Z-match pieces:
//   p(x, y)  radial profile (cputrack/utils.cpp:275-320): per bin the mean of the in-bounds bilinear
//            samples (utils.h:40-58 truncation and outside rule) over z_angsteps directions, or the
//            image mean with at most 4 samples in bounds;
//   phat     NormalizeRadialProfile (utils.cpp:230-261) when LT_NormalizeProfile is set;
//   Lz       the bead's LUT, linear between planes iz = clamp(floor z, 0, planes-2) and iz+1;
//   cost     sum_r (w_r (phat_r - Lz_r))^2 with the Z radial weights w (1 when unset), the score
//            LUTProfileCompare (cpu_tracker.cpp:791-868) maximises, negated, between planes.
// dp/dx is the mean of the samples' bilinear x-derivatives ((v10-v00)(1-fy) + (v11-v01)fy), likewise
// dp/dy; through the normalisation dphat = (dp - mean(dp) - phat sum_j(phat_j dp_j)/n) / rms.
// Profiles are recomputed from the ROI (kept in shared memory), never stored as polar samples.
#include <cstdint>

#include "kernels.h"
#include "tile.cuh"

namespace qtrk {

namespace {

constexpr int kAdjThreads = 128;     // adjoint: eight CTAs per SM hide its one-warp section
constexpr int kRefineThreads = 256;  // joint refinement: many profiles of one ROI in turn
constexpr int kGaussNllThreads = 256;
constexpr int kRefineSteps = 5;
constexpr float kPriorScale = 100.0f;  // x, y prior stiffness / z curvature (see joint_refine_kernel)

struct AdjSmem {
    uint32_t *img;        // the tile (tile.cuh)
    double *p, *dx, *dy;  // [nb] profile and its x/y derivatives (normalised in place)
    double *red;          // 32 doubles of reduction scratch
    double *misc;         // 16 doubles: broadcast values, the last two the mbarrier of the ROI's copy and copy_late's word
    __device__ __forceinline__ uint64_t *mbar() const { return reinterpret_cast<uint64_t *>(misc + 14); }
};

__host__ __device__ inline int adj_smem_bytes(const TrackParams &P, int ts)
{
    return tile_region_bytes(P.width, P.height, ts) + 3 * P.z_nbins * 8 + 32 * 8 + 16 * 8;
}

// Padded rows where they fit in shared memory.
inline int adj_pitch(const TrackParams &P)
{
    const int ts = tile_pitch(P.width);
    return adj_smem_bytes(P, ts) <= 227 * 1024 ? ts : P.width;
}

__device__ __forceinline__ AdjSmem adj_view(uint8_t *smem, const TrackParams &P, int ts)
{
    AdjSmem s;
    s.img = reinterpret_cast<uint32_t *>(smem);
    double *d = reinterpret_cast<double *>(smem + tile_region_bytes(P.width, P.height, ts));
    s.p = d;
    s.dx = d + P.z_nbins;
    s.dy = d + 2 * P.z_nbins;
    s.red = d + 3 * P.z_nbins;
    s.misc = s.red + 32;
    return s;
}

// Load the ROI's tile; every thread gets the image mean (FP64 sum; asked only where a bin falls back to it).
template <int F, int T>
__device__ __forceinline__ float adj_load(const AdjSmem &s, const TrackParams &P, int ts, const uint8_t *src, int pitch,
                                          int bead)
{
    const int W = P.width, n = W * P.height;
    uint32_t isum = 0u;
    if (F == kTileF32 && packed_rows(W, ts)) {
        if (threadIdx.x == 0) copy_late(s.mbar()) = 0u;
        load_roi(BlockGroup{s.red}, reinterpret_cast<float *>(s.img), src, pitch, P, bead);
    } else {
        const uint8_t *raw = load_raw<F, T>(s.img, ts, P, src, pitch, s.mbar(), [] {});
        convert_raw<F, T>(s.img, raw, ts, P, bead, isum);
    }
    __syncthreads();
    double v[1] = {(double)isum};  // integer pixels: exact
    if (F == kTileF32) {
        v[0] = 0.0;
        const int units = ((W + 3) >> 2) * P.height;
        UnitWalk w(threadIdx.x, T, W, ts);
        for (int u = threadIdx.x; u < units; u += T, w.step())
            for (int j = 0; j < 4 && w.x + j < W; j++) v[0] += (double)__uint_as_float(s.img[w.off + j]);
    }
    BlockGroup{s.red}.sum<1>(v);
    return (float)(v[0] / n);
}

// Profile (and derivatives) at (cx, cy), ROI in the tile: as radial_profile, eight lanes per bin with the direction
// pairs (j, j + h), j = lane, lane + 8, ..., two samples per step in packed FP32x2; four pairs are summed in FP32
// and folded into FP64. The x-derivative of a sample is d0 (1 - fy) + d1 fy, its y-derivative v1 - v0 (the values
// cells2 returns). Sample coordinates are fma(d, r, c), as before: which cell a sample near a pixel edge falls
// into decides its derivative. Ends with a block barrier.
template <int F, int T>
__device__ __forceinline__ void profile_grad(const uint32_t *img, int ts, const TrackParams &P, float cx, float cy,
                                             float mean, double *p, double *dx, double *dy)
{
    const int nb = P.z_nbins, W = P.width, H = P.height, sub = threadIdx.x & 7, h = P.z_angsteps >> 1;
    const bool odd = (P.z_angsteps & 1) != 0;
    const float rstep = (P.z_maxr - P.z_minr) / (float)nb;
    const float2 *dirs = static_cast<const float2 *>(P.z_dirs);
    const TileAddr ta(img, ts);
    const float2 K = make_float2(kBias, kBias), nK = make_float2(-kBias, -kBias), m1 = make_float2(-1.0f, -1.0f);
    const float2 one = make_float2(1.0f, 1.0f);
    const double inv_all = 1.0 / P.z_angsteps;
#pragma unroll 1
    for (int bin = threadIdx.x >> 3; bin - (int)((threadIdx.x & 31) >> 3) < nb; bin += T / 8) {
        const float r = P.z_minr + rstep * (float)bin;
        double s = 0.0, sx = 0.0, sy = 0.0;
        int c = 0;
        // one path per warp
        const bool inside = __all_sync(0xffffffffu, bin >= nb || circle_inside(cx, cy, fabsf(r), W, H));
        const float2 rr = make_float2(r, r), cxx = make_float2(cx, cx), cyy = make_float2(cy, cy);
        if (inside) {
            float2 a = make_float2(0.0f, 0.0f), ax = a, ay = a;
            auto fold = [&] {
                s += (double)(a.x + a.y);
                sx += (double)(ax.x + ax.y);
                sy += (double)(ay.x + ay.y);
                a = ax = ay = make_float2(0.0f, 0.0f);
            };
            auto pair = [&](float2 d0, float2 d1) {
                const float2 X = __ffma2_rn(make_float2(d0.x, d1.x), rr, cxx);
                const float2 Y = __ffma2_rn(make_float2(d0.y, d1.y), rr, cyy);
                const float2 TX = __fadd2_rz(X, K), TY = __fadd2_rz(Y, K);
                const float2 FX = __ffma2_rn(__fadd2_rn(TX, nK), m1, X), FY = __ffma2_rn(__fadd2_rn(TY, nK), m1, Y);
                const Cells q = cells2<F>(ta.at(ta.row(TY.x), TX.x), ta.at(ta.row(TY.y), TX.y), ta.ts4);
                const float2 v0 = __ffma2_rn(q.d0, FX, q.v00), v1 = __ffma2_rn(q.d1, FX, q.v01);
                const float2 gy = __ffma2_rn(v0, m1, v1);
                a = __fadd2_rn(a, __ffma2_rn(gy, FY, v0));
                ay = __fadd2_rn(ay, gy);
                ax = __fadd2_rn(ax, __ffma2_rn(q.d1, FY, __fmul2_rn(q.d0, __ffma2_rn(FY, m1, one))));
            };
            const int np = bin < nb && sub < h ? (h - sub + 7) >> 3 : 0;
            const float2 *dl = dirs + sub;
            int k = 0;
#pragma unroll 1
            for (; k + 2 <= np; k += 2) {
                pair(__ldg(dl + 8 * k), __ldg(dl + 8 * k + h));
                pair(__ldg(dl + 8 * k + 8), __ldg(dl + 8 * k + 8 + h));
                if (k & 2) fold();
            }
            if (k < np) pair(__ldg(dl + 8 * k), __ldg(dl + 8 * k + h));
            fold();
            if (odd && sub == 0 && bin < nb) {
                const float2 d = __ldg(dirs + P.z_angsteps - 1);
                pair(d, d);
                s += (double)a.x;
                sx += (double)ax.x;
                sy += (double)ay.x;
            }
            c = P.z_angsteps;
        } else {
            const float xhi = (float)(W - 1), yhi = (float)(H - 1);
            const int end = bin < nb ? P.z_angsteps : 0;
            float a = 0.0f, ax = 0.0f, ay = 0.0f;
            int in_part = 0;
#pragma unroll 1
            for (int j = sub; j < end; j += 8) {
                const float2 d = __ldg(dirs + j);
                const float x = fmaf(d.x, r, cx), y = fmaf(d.y, r, cy);
                if (x > -1.0f && x < xhi && y > -1.0f && y < yhi) {
                    const float tx = __fadd_rz(fmaxf(x, 0.0f), kBias), ty = __fadd_rz(fmaxf(y, 0.0f), kBias);
                    const float fx = x - (tx - kBias), fy = y - (ty - kBias);
                    const uint32_t w = ta.at(ta.row(ty), tx);
                    const Cells q = cells2<F>(w, w, ta.ts4);
                    const float v0 = fmaf(q.d0.x, fx, q.v00.x), v1 = fmaf(q.d1.x, fx, q.v01.x);
                    a += fmaf(v1 - v0, fy, v0);
                    ax += fmaf(q.d1.x, fy, q.d0.x * (1.0f - fy));
                    ay += v1 - v0;
                    c++;
                }
                if (++in_part == 5) {  // FP32 partials of five samples
                    s += (double)a;
                    sx += (double)ax;
                    sy += (double)ay;
                    a = ax = ay = 0.0f;
                    in_part = 0;
                }
            }
            s += (double)a;
            sx += (double)ax;
            sy += (double)ay;
#pragma unroll
            for (int o = 4; o > 0; o >>= 1) c += __shfl_xor_sync(0xffffffffu, c, o);
        }
#pragma unroll
        for (int o = 4; o > 0; o >>= 1) {
            s += __shfl_xor_sync(0xffffffffu, s, o);
            sx += __shfl_xor_sync(0xffffffffu, sx, o);
            sy += __shfl_xor_sync(0xffffffffu, sy, o);
        }
        if (sub == 0 && bin < nb) {
            const double inv = inside ? inv_all : 1.0 / c;
            p[bin] = c > 4 ? s * inv : (double)mean;
            dx[bin] = c > 4 ? sx * inv : 0.0;
            dy[bin] = c > 4 ? sy * inv : 0.0;
        }
    }
    __syncthreads();
}

__device__ __forceinline__ double warp_sum(double v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

struct CostTerms {
    double cost, g[3];      // cost and its gradient
    double A[6];            // J^T J: xx, xy, xz, yy, yz, zz (residual Jacobian, weights applied)
    double Jr[3];           // J^T res
};

// Warp 0: normalise p (and its derivatives) in place when asked, then the cost against the bead's
// LUT L [planes][nb] at z and its derivatives. Every lane of warp 0 returns the totals.
__device__ CostTerms cost_terms(const TrackParams &P, double *p, double *dx, double *dy, const float *L, float z)
{
    const int lane = threadIdx.x & 31, nb = P.z_nbins, planes = P.lut_planes;
    __syncwarp();  // the sums below run as one warp
    if (P.mode & kLT_NormalizeProfile) {
        const double inv_nb = 1.0 / nb;
        double m = 0, mx = 0, my = 0;
        for (int i = lane; i < nb; i += 32) {
            m += p[i];
            mx += dx[i];
            my += dy[i];
        }
        m = warp_sum(m) * inv_nb;
        mx = warp_sum(mx) * inv_nb;
        my = warp_sum(my) * inv_nb;
        double ss = 0;
        for (int i = lane; i < nb; i += 32) ss += (p[i] - m) * (p[i] - m);
        const double inv_rms = 1.0 / sqrt(warp_sum(ss) * inv_nb);
        double kx = 0, ky = 0;
        for (int i = lane; i < nb; i += 32) {
            const double ph = (p[i] - m) * inv_rms;
            p[i] = ph;
            kx += ph * dx[i];
            ky += ph * dy[i];
        }
        kx = warp_sum(kx) * inv_nb;
        ky = warp_sum(ky) * inv_nb;
        for (int i = lane; i < nb; i += 32) {
            dx[i] = (dx[i] - mx - p[i] * kx) * inv_rms;
            dy[i] = (dy[i] - my - p[i] * ky) * inv_rms;
        }
    }
    int iz = (int)floorf(z);
    iz = max(0, min(planes - 2, iz));
    const double fz = (double)z - iz;
    CostTerms t = {};
    for (int i = lane; i < nb; i += 32) {
        const double l0 = L[iz * nb + i], l1 = L[(iz + 1) * nb + i];
        const double w = P.z_weights ? (double)P.z_weights[i] : 1.0, w2 = w * w;
        const double e = p[i] - (l0 + (l1 - l0) * fz);
        const double J[3] = {dx[i], dy[i], -(l1 - l0)};
        t.cost += w2 * e * e;
        for (int a = 0; a < 3; a++) t.Jr[a] += w2 * J[a] * e;
        t.A[0] += w2 * J[0] * J[0];
        t.A[1] += w2 * J[0] * J[1];
        t.A[2] += w2 * J[0] * J[2];
        t.A[3] += w2 * J[1] * J[1];
        t.A[4] += w2 * J[1] * J[2];
        t.A[5] += w2 * J[2] * J[2];
    }
    t.cost = warp_sum(t.cost);
    for (int a = 0; a < 3; a++) t.Jr[a] = warp_sum(t.Jr[a]);
    for (int a = 0; a < 6; a++) t.A[a] = warp_sum(t.A[a]);
    for (int a = 0; a < 3; a++) t.g[a] = 2.0 * t.Jr[a];
    return t;
}

// Adjoint: one block per ROI. xyz[3*roi], bead[roi] (or 0), out cost[roi], grad[3*roi], and
// glut[bead][plane][bin] += dcost/dL (atomically: ROIs of a bead share its LUT rows).
// What bounds it: instruction issue. A warp over the directions of one bin at a time, every sample checked and
// scalar, took 25.4 k warp instructions per 80x80 ROI, the packed pairs and pixel formats 12.8 k: 51,200 ROIs of
// 80x80 u16 with the LUT gradient 1.377 -> 0.76 ms.
template <int F>
__global__ void __launch_bounds__(kAdjThreads, 8)
    zcost_grad_kernel(TrackParams P, int ts, const uint8_t *__restrict__ pixels, int pitch, int64_t roi_stride,
                      int count, const float *__restrict__ xyz, const int *__restrict__ beads,
                      float *__restrict__ cost, float *__restrict__ grad, float *__restrict__ glut)
{
    extern __shared__ __align__(16) uint8_t smem[];
    const int roi = blockIdx.x;
    if (roi >= count) return;
    const AdjSmem s = adj_view(smem, P, ts);
    const int bead = beads ? beads[roi] : 0;
    bool ok = bead >= 0 && bead < P.lut_count && P.lut_planes >= 2;
    const float mean = adj_load<F, kAdjThreads>(s, P, ts, pixels + (int64_t)roi * roi_stride, pitch, ok ? bead : 0);
    ok = ok && !copy_late(s.mbar());  // asked here: where the results are written it cost 13 us of 775
    const float x = xyz[3 * roi], y = xyz[3 * roi + 1], z = xyz[3 * roi + 2];
    profile_grad<F, kAdjThreads>(s.img, ts, P, x, y, mean, s.p, s.dx, s.dy);
    if (threadIdx.x >= 32) return;
    if (!ok) {  // nothing to the LUT's gradient either
        if (threadIdx.x == 0) {
            cost[roi] = nanf("");
            grad[3 * roi] = grad[3 * roi + 1] = grad[3 * roi + 2] = nanf("");
        }
        return;
    }
    const int nb = P.z_nbins, planes = P.lut_planes;
    const float *L = P.lut + (size_t)bead * planes * nb;
    const CostTerms t = cost_terms(P, s.p, s.dx, s.dy, L, z);
    if (threadIdx.x == 0) {
        cost[roi] = (float)t.cost;
        grad[3 * roi] = (float)t.g[0];
        grad[3 * roi + 1] = (float)t.g[1];
        grad[3 * roi + 2] = (float)t.g[2];
    }
    if (glut) {
        int iz = (int)floorf(z);
        iz = max(0, min(planes - 2, iz));
        const double fz = (double)z - iz;
        float *G = glut + (size_t)bead * planes * nb;
        for (int i = threadIdx.x; i < nb; i += 32) {
            const double l0 = L[iz * nb + i], l1 = L[(iz + 1) * nb + i];
            const double w = P.z_weights ? (double)P.z_weights[i] : 1.0;
            const double de = 2.0 * w * w * (s.p[i] - (l0 + (l1 - l0) * fz));
            atomicAdd(&G[iz * nb + i], (float)(-de * (1.0 - fz)));
            atomicAdd(&G[(iz + 1) * nb + i], (float)(-de * fz));
        }
    }
}

// 3x3 solve A d = rhs by Cramer's rule (A symmetric, given as xx, xy, xz, yy, yz, zz).
__device__ bool solve3(const double A6[6], const double rhs[3], double d[3])
{
    const double a[3][3] = {{A6[0], A6[1], A6[2]}, {A6[1], A6[3], A6[4]}, {A6[2], A6[4], A6[5]}};
    const double det = a[0][0] * (a[1][1] * a[2][2] - a[1][2] * a[2][1]) - a[0][1] * (a[1][0] * a[2][2] - a[1][2] * a[2][0]) +
                       a[0][2] * (a[1][0] * a[2][1] - a[1][1] * a[2][0]);
    if (det == 0.0) return false;
    for (int c = 0; c < 3; c++) {
        double M[3][3];
        for (int i = 0; i < 3; i++)
            for (int j = 0; j < 3; j++) M[i][j] = (j == c) ? rhs[i] : a[i][j];
        d[c] = (M[0][0] * (M[1][1] * M[2][2] - M[1][2] * M[2][1]) - M[0][1] * (M[1][0] * M[2][2] - M[1][2] * M[2][0]) +
                M[0][2] * (M[1][0] * M[2][1] - M[1][1] * M[2][0])) /
               det;
    }
    return true;
}

// Joint Gauss-Newton refinement of a localized ROI (LT_B200_JointRefine), one block per ROI, in
// place on results[roi].pos. Minimises cost(x, y, z) + k ((x-x0)^2 + (y-y0)^2) from the located
// (x0, y0, z0), with k = 100 x the cost's z-curvature at the starting plane: a radial profile is
// insensitive to first order to its centre (the x-derivative of a radially symmetric image
// averages to zero over a circle), so the prior keeps QI's x, y precision while z follows the
// LUT interpolation. Per step: normal equations with the prior and a Levenberg term of
// 1e-9 x trace, Cramer's rule, and the step halved up to 4 times until the objective drops (the
// refinement stops when none does); z is clamped to [0, planes-1]. The fallback value of sparse
// bins is the ROI's image mean, as in the Z fit.
template <int F>
__global__ void __launch_bounds__(kRefineThreads)
    joint_refine_kernel(TrackParams P, int ts, const uint8_t *__restrict__ pixels, int pitch, int64_t roi_stride,
                        const int64_t *__restrict__ roi_offsets, const LocalizationJob *__restrict__ jobs, int count,
                        LocalizationResult *__restrict__ results)
{
    extern __shared__ __align__(16) uint8_t smem[];
    const int roi = blockIdx.x;
    if (roi >= count) return;
    const AdjSmem s = adj_view(smem, P, ts);
    const int bead = jobs ? jobs[roi].zlutIndex : 0;
    if (bead < 0 || bead >= P.lut_count || P.lut_planes < 2) return;  // no LUT for this ROI: no Z fit to refine
    const int64_t off = roi_offsets ? roi_offsets[roi] : (int64_t)roi * roi_stride;
    adj_load<F, kRefineThreads>(s, P, ts, pixels + off, pitch, bead);
    LocalizationResult *res = results + roi;
    const float mean = res->imageMean;
    const float x0 = res->pos.x, y0 = res->pos.y;
    float x = x0, y = y0, z = res->pos.z;
    const int nb = P.z_nbins, planes = P.lut_planes;
    const float *L = P.lut + (size_t)bead * planes * nb;
    double k = 0.0, cur = 0.0;
    for (int step = 0; step < kRefineSteps; step++) {
        profile_grad<F, kRefineThreads>(s.img, ts, P, x, y, mean, s.p, s.dx, s.dy);
        if (threadIdx.x < 32) {
            const CostTerms t = cost_terms(P, s.p, s.dx, s.dy, L, z);
            if (threadIdx.x == 0) {
                if (step == 0) k = kPriorScale * t.A[5];
                cur = t.cost + k * ((double)(x - x0) * (x - x0) + (double)(y - y0) * (y - y0));
                double A6[6] = {t.A[0] + k, t.A[1], t.A[2], t.A[3] + k, t.A[4], t.A[5]};
                const double tr = A6[0] + A6[3] + A6[5];
                A6[0] += 1e-9 * tr + 1e-30;
                A6[3] += 1e-9 * tr + 1e-30;
                A6[5] += 1e-9 * tr + 1e-30;
                const double rhs[3] = {-(t.Jr[0] + k * (x - x0)), -(t.Jr[1] + k * (y - y0)), -t.Jr[2]};
                double d[3];
                const bool solved = solve3(A6, rhs, d);
                s.misc[0] = solved ? 1.0 : 0.0;
                s.misc[1] = d[0];
                s.misc[2] = d[1];
                s.misc[3] = d[2];
                s.misc[4] = cur;
                s.misc[5] = k;
            }
        }
        __syncthreads();
        if (s.misc[0] == 0.0) break;
        const double d0 = s.misc[1], d1 = s.misc[2], d2 = s.misc[3];
        cur = s.misc[4];
        k = s.misc[5];
        bool taken = false;
        for (int hv = 0; hv < 5 && !taken; hv++) {
            const double tstep = ldexp(1.0, -hv);
            const float nx = (float)(x + tstep * d0), ny = (float)(y + tstep * d1);
            const float nz = fminf(fmaxf((float)(z + tstep * d2), 0.0f), (float)(planes - 1));
            profile_grad<F, kRefineThreads>(s.img, ts, P, nx, ny, mean, s.p, s.dx, s.dy);
            if (threadIdx.x < 32) {
                const CostTerms t = cost_terms(P, s.p, s.dx, s.dy, L, nz);
                if (threadIdx.x == 0)
                    s.misc[6] = t.cost + k * ((double)(nx - x0) * (nx - x0) + (double)(ny - y0) * (ny - y0));
            }
            __syncthreads();
            if (s.misc[6] < cur) {
                x = nx;
                y = ny;
                z = nz;
                cur = s.misc[6];
                taken = true;
            }
            __syncthreads();
        }
        if (!taken) break;
    }
    if (threadIdx.x == 0) {
        if (copy_late(s.mbar())) x = y = z = nanf("");
        res->pos.x = x;
        res->pos.y = y;
        res->pos.z = z;
    }
}

// Gaussian-MLE adjoint: Poisson NLL = sum mu - I ln mu of the 5-parameter integrated-Gaussian
// model (the model gauss5_mle fits, erff per column/row, FP32 per pixel, FP64 sums) and its
// gradient sum (1 - I/mu) dmu/dp for p = (x, y, I0, bg, sigma) = params[5 roi ..]. One block per ROI;
// windows of at most 32x32 pixels take gauss_nll_warp_kernel (gauss.cu).
__global__ void __launch_bounds__(kGaussNllThreads) gauss_nll_grad_kernel(TrackParams P, const uint8_t *__restrict__ pixels,
                                                                     int pitch, int64_t roi_stride, int count,
                                                                     const float *__restrict__ params,
                                                                     float *__restrict__ nll, float *__restrict__ grad)
{
    extern __shared__ __align__(16) uint8_t smem[];
    const int roi = blockIdx.x;
    if (roi >= count) return;
    const int W = P.width, H = P.height;
    float *img = reinterpret_cast<float *>(smem);
    float *col = img + ((W * H + 3) & ~3);
    float *row = col + 3 * W;
    double *red = reinterpret_cast<double *>(smem + (((size_t)((W * H + 3) & ~3) + 3 * (W + H)) * 4 + 15) / 16 * 16);
    BlockGroup g{red};
    load_roi(g, img, pixels + (int64_t)roi * roi_stride, pitch, P, 0);
    float p[5];
#pragma unroll
    for (int k = 0; k < 5; k++) p[k] = params[5 * roi + k];
    const float s = p[4];
    const float k1 = 1.0f / (sqrtf(2.0f) * s);
    const float k2 = 1.0f / (sqrtf(2 * 3.14159265359f) * s);
    for (int c = threadIdx.x; c < W + H; c += blockDim.x) {
        const bool is_col = c < W;
        const int cc = is_col ? c : c - W;
        const float pc = is_col ? p[0] : p[1];
        const float a0 = (cc - pc + .5f) * k1, a1 = (cc - pc - .5f) * k1;
        const float e0 = expf(-a0 * a0), e1 = expf(-a1 * a1);
        float *t = is_col ? col + 3 * cc : row + 3 * cc;
        t[0] = 0.5f * (erff(a0) - erff(a1));
        t[1] = (e1 - e0) * k2;
        t[2] = ((cc - pc - .5f) * e1 - (cc - pc + .5f) * e0) * k2 / s;
    }
    __syncthreads();
    double acc[6] = {0, 0, 0, 0, 0, 0};
    for (int i = threadIdx.x; i < W * H; i += blockDim.x) {
        const int y = i / W, x = i - y * W;
        const float DX = col[3 * x], dX = col[3 * x + 1], sX = col[3 * x + 2];
        const float DY = row[3 * y], dY = row[3 * y + 1], sY = row[3 * y + 2];
        const float mu = p[3] + p[2] * DX * DY;
        const float I = img[i];
        const float f = 1.0f - I / mu;
        acc[0] += (double)(mu - I * logf(mu));
        acc[1] += (double)(f * p[2] * dX * DY);
        acc[2] += (double)(f * p[2] * DX * dY);
        acc[3] += (double)(f * DX * DY);
        acc[4] += (double)f;
        acc[5] += (double)(f * p[2] * (sX * DY + DX * sY));
    }
    g.sum(acc);
    if (threadIdx.x == 0) {
        nll[roi] = (float)acc[0];
#pragma unroll
        for (int k = 0; k < 5; k++) grad[5 * roi + k] = (float)acc[1 + k];
    }
}

}  // namespace

cudaError_t launch_zcost_grad(const TrackParams &P, const uint8_t *pixels, int pitch, int64_t roi_stride, int count,
                              const float *xyz, const int *beads, float *cost, float *grad, float *glut,
                              cudaStream_t stream)
{
    if (count <= 0) return cudaSuccess;
    const int ts = adj_pitch(P), smem = adj_smem_bytes(P, ts), f = tile_format(P, ts);
    const auto kernel = f == kTileF32 ? zcost_grad_kernel<kTileF32>
                                      : (f == kTileU16 ? zcost_grad_kernel<kTileU16> : zcost_grad_kernel<kTileU8>);
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return e;
    kernel<<<count, kAdjThreads, smem, stream>>>(P, ts, pixels, pitch, roi_stride, count, xyz, beads, cost, grad, glut);
    return cudaGetLastError();
}

cudaError_t launch_gauss_nll_grad(const TrackParams &P, const uint8_t *pixels, int pitch, int64_t roi_stride, int count,
                                  const float *params, float *nll, float *grad, cudaStream_t stream)
{
    if (count <= 0) return cudaSuccess;
    if (use_gauss_nll_warp(P)) return launch_gauss_nll_warp(P, pixels, pitch, roi_stride, count, params, nll, grad, stream);
    const int W = P.width, H = P.height;
    const int smem = (int)((((size_t)((W * H + 3) & ~3) + 3 * (W + H)) * 4 + 15) / 16 * 16) + 6 * 32 * 8;
    cudaError_t e = cudaFuncSetAttribute(gauss_nll_grad_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return e;
    gauss_nll_grad_kernel<<<count, kGaussNllThreads, smem, stream>>>(P, pixels, pitch, roi_stride, count, params, nll, grad);
    return cudaGetLastError();
}

cudaError_t launch_joint_refine(const TrackParams &P, const uint8_t *pixels, int pitch, int64_t roi_stride,
                                const int64_t *roi_offsets, const LocalizationJob *jobs, int count,
                                LocalizationResult *results, cudaStream_t stream)
{
    if (count <= 0) return cudaSuccess;
    const int ts = adj_pitch(P), smem = adj_smem_bytes(P, ts), f = tile_format(P, ts);
    const auto kernel = f == kTileF32 ? joint_refine_kernel<kTileF32>
                                      : (f == kTileU16 ? joint_refine_kernel<kTileU16> : joint_refine_kernel<kTileU8>);
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return e;
    kernel<<<count, kRefineThreads, smem, stream>>>(P, ts, pixels, pitch, roi_stride, roi_offsets, jobs, count, results);
    return cudaGetLastError();
}

}  // namespace qtrk

// 2D Gaussian MLE of small spots (ROIs of at most 32x32 pixels), half a warp or one warp per ROI (sm_100a).
//
// gauss_warp_kernel<4>: CPUTracker::Compute2DGaussianMLE (cputrack/cpu_tracker.cpp:514-589), the
//   4-parameter per-parameter Newton of gauss4_mle (device_common.cuh).
// gauss_warp_kernel<5>: the 5-parameter Fisher-scoring form of gauss5_mle.
// gauss_nll_warp_kernel: the likelihood of the 5-parameter model and its gradient (the small-window form
//   of gauss_nll_grad_kernel, adjoint.cu).
//
// The model is separable, mu = bg + I0 DX(x) DY(y), and so is every derivative. A ROI of up to 16 columns
// has 16 lanes, a wider one 32. Lane l takes column x = l mod cw (cw: W rounded up to 8, 16 or 32) of
// rows l / cw, l / cw + lanes / cw, ..., so its column terms factor out of all sums: per pixel only
// products of row terms with f = (I - mu) / mu and with the weight (I / mu^2, or 1 / mu) are
// accumulated, and the column factors are applied once per lane and iteration. f, the weight and one
// reciprocal are all that a pixel computes itself. Two ROIs per warp share the instructions of what
// is left per iteration: the sums across lanes, the divisions and the 5x5 solve.
//
// What bounds it: instruction issue (75 % used at 24-32 warps per SM). Measured on 100,000 16x16 f32
// ROIs, 8 iterations: 4 parameters 1.520 -> 0.404 ms, 5 parameters (20,000 15x15 u16) 0.434 -> 0.136 ms
// against one warp per ROI with every pixel forming all its products in FP32 and adding eight (or twenty)
// sums; one warp per ROI with the column factors taken out reached 0.613 and 0.232 ms.
#include <cstdint>

#include "device_common.cuh"
#include "kernels.h"

namespace qtrk {

namespace {

constexpr int kGaussWarps = 8;  // ROIs (warps) per CTA
constexpr int kGaussRow = 48;   // bytes of row terms per image row

// Per-warp shared memory: the float ROI, the row terms, the column terms and 20 reduction totals.
struct GaussSmem {
    int rows, cols, tot, bytes;
};

__host__ __device__ inline GaussSmem gauss_smem(int W, int H)
{
    GaussSmem s;
    s.rows = (W * H * 4 + 15) & ~15;
    s.cols = s.rows + H * kGaussRow;
    s.tot = s.cols + ((W * 12 + 15) & ~15);
    s.bytes = s.tot + 20 * 8;
    return s;
}

// One halving step of a transposing sum over lanes: the N values of each lane become H = ceil(N/2),
// lanes with bit `o` set keeping the upper part. Repeated over all lane bits it leaves each total in
// one lane, for 21 exchanged doubles at N = 20 and 32 lanes instead of a butterfly's 100.
template <int N>
__device__ __forceinline__ void fold(double *v, int lane, int o, unsigned mask)
{
    constexpr int H = (N + 1) / 2;
    const bool up = (lane & o) != 0;
#pragma unroll
    for (int k = 0; k < H; k++) {
        const double hi = k + H < N ? v[k + H] : 0.0;
        const double send = up ? v[k] : hi, keep = up ? hi : v[k];
        v[k] = keep + __shfl_xor_sync(mask, send, o);
    }
}

// Fold N values over all bits of a kLanes-lane group. The lane's totals are v[0 .. count-1], of the
// values base .. base + count - 1.
template <int N, int kO>
__device__ __forceinline__ void fold_all(double *v, int lane, unsigned mask, int &base, int &count)
{
    constexpr int H = (N + 1) / 2;
    fold<N>(v, lane, kO, mask);
    const bool up = (lane & kO) != 0;
    base += up ? H : 0;
    count = up ? count - H : min(count, H);
    if constexpr (kO > 1) fold_all<H, kO / 2>(v, lane, mask, base, count);
}

// A symmetric definite 5x5 system (upper triangle in A, row by row) by elimination without pivoting,
// one reciprocal per pivot. The Fisher matrix is a Gram matrix with weights of one sign, for which
// elimination in any order is stable. False when a pivot vanishes (or is not a number).
__device__ __forceinline__ bool solve5_definite(double (&A)[5][5], double (&b)[5], double (&d)[5])
{
    double inv[5];
#pragma unroll
    for (int c = 0; c < 5; c++) {
        if (!(fabs(A[c][c]) > 1e-300)) return false;
        inv[c] = 1.0 / A[c][c];
#pragma unroll
        for (int r = c + 1; r < 5; r++) {
            const double f = A[c][r] * inv[c];
#pragma unroll
            for (int j = r; j < 5; j++) A[r][j] -= f * A[c][j];
            b[r] -= f * b[c];
        }
    }
#pragma unroll
    for (int i = 4; i >= 0; i--) {
        double s = b[i];
#pragma unroll
        for (int j = i + 1; j < 5; j++) s -= A[i][j] * d[j];
        d[i] = s * inv[i];
    }
    return true;
}

struct GaussLane {
    int lane, x, y0, rp;  // lane in the ROI's group, column, first row and row step
    unsigned mask;        // the group's lanes
    bool on;              // x < W
};

template <int kLanes>
__device__ __forceinline__ GaussLane gauss_lane(int W)
{
    GaussLane g;
    const int lc = W <= 8 ? 3 : (W <= 16 ? 4 : 5);
    g.lane = threadIdx.x & (kLanes - 1);
    g.mask = LaneGroup<kLanes>().mask();
    g.x = g.lane & ((1 << lc) - 1);
    g.y0 = g.lane >> lc;
    g.rp = kLanes >> lc;
    g.on = g.x < W;
    return g;
}

// Four parameters. Sums are FP64 throughout: a pixel converts f and I / mu^2 and adds their products
// with the row terms (kept as doubles) by FP64 multiply-adds.
template <int kLanes>
__device__ __forceinline__ void gauss4_lanes(const GaussLane &g, const float *img, int W, int H, float mean, float &px,
                                             float &py, int iters, float sigma, double *rows, float *cols)
{
    float I0 = mean * 0.5f * (float)W * (float)H;
    float bg = mean * 0.5f;
    const float k1 = 1.0f / (sqrtf(2.0f) * sigma);
    const double k2 = 1.0 / (2.506628274631000502 * (double)sigma);  // 1 / (sqrt(2 pi) sigma)
    const double k3 = k2 / ((double)sigma * (double)sigma);
    for (int it = 0; it < iters; it++) {
        __syncwarp(g.mask);
        for (int c = g.lane; c < W + H; c += kLanes) {
            const bool is_col = c < W;
            const int cc = is_col ? c : c - W;
            const GaussAxisTerms t = gauss_axis_terms(cc, is_col ? px : py, k1);
            if (is_col) {
                cols[3 * cc] = t.D;
                cols[3 * cc + 1] = t.g;
                cols[3 * cc + 2] = t.h;
            } else {
                double2 *r = reinterpret_cast<double2 *>(rows + 6 * cc);
                const double D = t.D, gy = t.g;
                r[0] = make_double2(D, gy);
                r[1] = make_double2((double)t.h, D * D);
                r[2] = make_double2(gy * gy, __hiloint2double(0, __float_as_int(t.D)));
            }
        }
        __syncwarp(g.mask);
        double v[8] = {0, 0, 0, 0, 0, 0, 0, 0};
        if (g.on) {
            double sDf = 0, sgf = 0, sf = 0, shf = 0, sDDq = 0, sggq = 0, sq = 0;
            const float DX = cols[3 * g.x], i0dx = I0 * DX;
            const double2 *r = reinterpret_cast<const double2 *>(rows + 6 * g.y0);
            const float *px_y = img + g.y0 * W + g.x;
#pragma unroll 4
            for (int y = g.y0; y < H; y += g.rp, r += 3 * g.rp, px_y += g.rp * W) {
                const double2 a = r[0], b = r[1], c = r[2];
                const float mu = fmaf(i0dx, __int_as_float(__double2loint(c.y)), bg);
                const float smp = *px_y;
                const float inv = rcp(mu);
                const double f = (double)((smp - mu) * inv), q = (double)(smp * inv * inv);
                sDf = fma(a.x, f, sDf);
                sgf = fma(a.y, f, sgf);
                sf += f;
                shf = fma(b.x, f, shf);
                sDDq = fma(b.y, q, sDDq);
                sggq = fma(c.x, q, sggq);
                sq += q;
            }
            const double D = DX, gx = cols[3 * g.x + 1], hx = cols[3 * g.x + 2];
            const double i2 = (double)I0 * k2, i3 = (double)I0 * k3;
            const double jx = i2 * gx, jy = i2 * D;
            v[0] = jx * sDf;                              // d/dx
            v[1] = jy * sgf;                              // d/dy
            v[2] = D * sDf;                               // d/dI0
            v[3] = sf;                                    // d/dbg
            v[4] = i3 * hx * sDf - jx * jx * sDDq;        // second derivatives
            v[5] = i3 * D * shf - jy * jy * sggq;
            v[6] = -(D * D * sDDq);
            v[7] = -sq;
        }
        // the lower half of the lanes ends with the first derivative of parameter
        // k = (lane / (lanes / 8)) mod 4, the upper half with its second: one division serves all four
        fold<8>(v, g.lane, kLanes / 2, g.mask);
        fold<4>(v, g.lane, kLanes / 4, g.mask);
        fold<2>(v, g.lane, kLanes / 8, g.mask);
#pragma unroll
        for (int o = kLanes / 16; o > 0; o >>= 1) v[0] += __shfl_xor_sync(g.mask, v[0], o);
        const double second = __shfl_xor_sync(g.mask, v[0], kLanes / 2);
        const int k = (g.lane / (kLanes / 8)) & 3;
        const float p = k == 0 ? px : (k == 1 ? py : (k == 2 ? I0 : bg));
        const float np = (float)((double)p - v[0] / second);
        px = __shfl_sync(g.mask, np, 0, kLanes);
        py = __shfl_sync(g.mask, np, kLanes / 8, kLanes);
        I0 = __shfl_sync(g.mask, np, 2 * (kLanes / 8), kLanes);
        bg = __shfl_sync(g.mask, np, 3 * (kLanes / 8), kLanes);
    }
}

// Five parameters p = (x, y, I0, bg, sigma). As in gauss5_mle a lane's pixel sums are FP32 and the
// sums across lanes and the 5x5 solve FP64. Row terms: D, dD/dp, dD/dsigma and their six products.
template <int kLanes>
__device__ __forceinline__ void gauss5_lanes(const GaussLane &g, const float *img, int W, int H, float (&p)[5],
                                             int iters, float4 *rows, float *cols, double *tot)
{
    for (int it = 0; it < iters; it++) {
        const float s = p[4];
        const float k1 = 1.0f / (sqrtf(2.0f) * s);
        const float k2 = 1.0f / (sqrtf(2 * 3.14159265359f) * s), k2s = k2 / s;
        __syncwarp(g.mask);
        for (int c = g.lane; c < W + H; c += kLanes) {
            const bool is_col = c < W;
            const int cc = is_col ? c : c - W;
            const float pc = is_col ? p[0] : p[1];
            const float a0 = (cc - pc + .5f) * k1, a1 = (cc - pc - .5f) * k1;
            const float e0 = expf(-a0 * a0), e1 = expf(-a1 * a1);
            const float D = 0.5f * (erff(a0) - erff(a1));
            const float d = (e1 - e0) * k2;                                             // dD/dp
            const float t = ((cc - pc - .5f) * e1 - (cc - pc + .5f) * e0) * k2s;         // dD/dsigma
            if (is_col) {
                cols[3 * cc] = D;
                cols[3 * cc + 1] = d;
                cols[3 * cc + 2] = t;
            } else {
                rows[3 * cc] = make_float4(D, d, t, D * D);
                rows[3 * cc + 1] = make_float4(D * d, D * t, d * d, d * t);
                rows[3 * cc + 2].x = t * t;
            }
        }
        __syncwarp(g.mask);
        double v[20];
#pragma unroll
        for (int k = 0; k < 20; k++) v[k] = 0.0;
        if (g.on) {
            float fD = 0, fd = 0, ft = 0, f1 = 0;
            float DD = 0, Dd = 0, Dt = 0, dd = 0, dt = 0, tt = 0, m1 = 0, mD = 0, md = 0, mt = 0;
            const float DX = cols[3 * g.x], dX = cols[3 * g.x + 1], tX = cols[3 * g.x + 2];
            const float I0 = p[2], i0dx = I0 * DX;
            const float4 *r = rows + 3 * g.y0;
            const float *px_y = img + g.y0 * W + g.x;
#pragma unroll 4
            for (int y = g.y0; y < H; y += g.rp, r += 3 * g.rp, px_y += g.rp * W) {
                const float4 a = r[0], b = r[1];
                const float c = r[2].x;
                const float mu = fmaf(i0dx, a.x, p[3]);
                const float inv = rcp(mu);
                // the quotient with one step of iterative refinement: the gradient decides where the fit
                // ends, the Fisher matrix's weights only steer the steps
                const float d = *px_y - mu, f0 = d * inv;
                const float f = fmaf(fmaf(-f0, mu, d), inv, f0);
                fD = fmaf(a.x, f, fD);
                fd = fmaf(a.y, f, fd);
                ft = fmaf(a.z, f, ft);
                f1 += f;
                mD = fmaf(a.x, inv, mD);
                md = fmaf(a.y, inv, md);
                mt = fmaf(a.z, inv, mt);
                m1 += inv;
                DD = fmaf(a.w, inv, DD);
                Dd = fmaf(b.x, inv, Dd);
                Dt = fmaf(b.y, inv, Dt);
                dd = fmaf(b.z, inv, dd);
                dt = fmaf(b.w, inv, dt);
                tt = fmaf(c, inv, tt);
            }
            const float jx = I0 * dX, jy = I0 * DX, js = I0 * tX;
            // dmu/d(x, y, I0, bg, sigma) = (jx D, jy d, DX D, 1, js D + jy t)
            v[0] = jx * fD;
            v[1] = jy * fd;
            v[2] = DX * fD;
            v[3] = f1;
            v[4] = fmaf(js, fD, jy * ft);
            v[5] = jx * jx * DD;
            v[6] = jx * jy * Dd;
            v[7] = jx * DX * DD;
            v[8] = jx * mD;
            v[9] = jx * fmaf(js, DD, jy * Dt);
            v[10] = jy * jy * dd;
            v[11] = jy * DX * Dd;
            v[12] = jy * md;
            v[13] = jy * fmaf(js, Dd, jy * dt);
            v[14] = DX * DX * DD;
            v[15] = DX * mD;
            v[16] = DX * fmaf(js, DD, jy * Dt);
            v[17] = m1;
            v[18] = fmaf(js, mD, jy * mt);
            v[19] = fmaf(js, fmaf(js, DD, 2.0f * (jy * Dt)), jy * jy * tt);
        }
        int base = 0, own = 20;
        fold_all<20, kLanes / 2>(v, g.lane, g.mask, base, own);
        for (int k = 0; k < 2; k++)
            if (k < own) tot[base + k] = v[k];
        __syncwarp(g.mask);
        double A[5][5], b[5], d[5];
        int k = 5;
#pragma unroll
        for (int u = 0; u < 5; u++) {
            b[u] = tot[u];
#pragma unroll
            for (int w = u; w < 5; w++) A[u][w] = tot[k++];
        }
        if (!solve5_definite(A, b, d)) break;  // the whole group: its lanes solve the same system
#pragma unroll
        for (int u = 0; u < 5; u++) p[u] = (float)((double)p[u] + d[u]);
        p[2] = fmaxf(p[2], 1e-3f);
        p[3] = fmaxf(p[3], 1e-3f);
        p[4] = fminf(fmaxf(p[4], 0.3f), 0.5f * (float)W);
    }
}

template <int kParams, int kLanes>
__global__ void __launch_bounds__(32 * kGaussWarps, kParams == 4 ? 4 : 3)
    gauss_warp_kernel(TrackParams P, const uint8_t *__restrict__ pixels, int pitch, int64_t roi_stride,
                      const int64_t *__restrict__ roi_offsets, const LocalizationJob *__restrict__ jobs, int count,
                      LocalizationResult *__restrict__ results)
{
    extern __shared__ __align__(16) uint8_t smem[];
    const int group = threadIdx.x / kLanes;
    const int roi = blockIdx.x * (32 * kGaussWarps / kLanes) + group;
    if (roi >= count) return;  // whole groups exit together; every sync and shuffle is over one group
    const int W = P.width, H = P.height;
    const GaussSmem sm = gauss_smem(W, H);
    uint8_t *base = smem + group * sm.bytes;
    float *img = reinterpret_cast<float *>(base);
    float *cols = reinterpret_cast<float *>(base + sm.cols);
    const int bead = jobs ? (int)reinterpret_cast<const uint32_t *>(jobs)[(size_t)roi * 6 + 2] : 0;
    const int64_t off = roi_offsets ? roi_offsets[roi] : (int64_t)roi * roi_stride;
    const LaneGroup<kLanes> lg;
    const double2 part = load_roi(lg, img, pixels + off, pitch, P, bead);
    const ComResult com = com_from_sums(lg, img, W, H, part, P.com_bgcorrection);
    float comx = com.x, comy = com.y;
    if (isnan(comx) || isnan(comy)) {  // QueuedCPUTracker.cpp:294-295
        comx = (float)(W / 2);
        comy = (float)(H / 2);
    }
    const GaussLane g = gauss_lane<kLanes>(W);
    float x = comx, y = comy, z = 0.0f;
    if (kParams == 5) {
        float p[5] = {x, y, com.mean * 0.5f * (float)(W * H), com.mean * 0.5f, P.g_sigma};
        gauss5_lanes<kLanes>(g, img, W, H, p, P.g_iterations, reinterpret_cast<float4 *>(base + sm.rows), cols,
                             reinterpret_cast<double *>(base + sm.tot));
        x = p[0];
        y = p[1];
        z = p[4];
    } else {
        gauss4_lanes<kLanes>(g, img, W, H, com.mean, x, y, P.g_iterations, P.g_sigma,
                             reinterpret_cast<double *>(base + sm.rows), cols);
    }
    if (g.lane == 0) {
        uint32_t job[6];
        read_job(jobs, roi, job);
        write_result(results, roi, job, x, y, z, comx, comy, 0u, com.mean);
    }
}

// Poisson NLL = sum mu - I ln mu of the 5-parameter model at params[5 roi ..] = (x, y, I0, bg, sigma) and
// its gradient sum (1 - I / mu) dmu/dp: one pass of the lane layout above, sums in FP64. 50,000 16x16 f32
// ROIs: 0.337 -> 0.045 ms against a CTA of 256 threads per ROI, which spent its time in barriers and in
// six block sums for one pixel per thread.
template <int kLanes>
__global__ void __launch_bounds__(32 * kGaussWarps, 4)
    gauss_nll_warp_kernel(TrackParams P, const uint8_t *__restrict__ pixels, int pitch, int64_t roi_stride, int count,
                          const float *__restrict__ params, float *__restrict__ nll, float *__restrict__ grad)
{
    extern __shared__ __align__(16) uint8_t smem[];
    const int group = threadIdx.x / kLanes;
    const int roi = blockIdx.x * (32 * kGaussWarps / kLanes) + group;
    if (roi >= count) return;  // whole groups exit together
    const int W = P.width, H = P.height;
    const GaussSmem sm = gauss_smem(W, H);
    uint8_t *base = smem + group * sm.bytes;
    float *img = reinterpret_cast<float *>(base);
    double *rows = reinterpret_cast<double *>(base + sm.rows);
    float *cols = reinterpret_cast<float *>(base + sm.cols);
    load_roi(LaneGroup<kLanes>(), img, pixels + (int64_t)roi * roi_stride, pitch, P, 0);
    const GaussLane g = gauss_lane<kLanes>(W);
    float p[5];
#pragma unroll
    for (int k = 0; k < 5; k++) p[k] = params[5 * roi + k];
    const float s = p[4];
    const float k1 = 1.0f / (sqrtf(2.0f) * s);
    const float k2 = 1.0f / (sqrtf(2 * 3.14159265359f) * s);
    for (int c = g.lane; c < W + H; c += kLanes) {
        const bool is_col = c < W;
        const int cc = is_col ? c : c - W;
        const float pc = is_col ? p[0] : p[1];
        const float a0 = (cc - pc + .5f) * k1, a1 = (cc - pc - .5f) * k1;
        const float e0 = expf(-a0 * a0), e1 = expf(-a1 * a1);
        const float D = 0.5f * (erff(a0) - erff(a1));
        const float d = (e1 - e0) * k2;
        const float t = ((cc - pc - .5f) * e1 - (cc - pc + .5f) * e0) * k2 / s;
        if (is_col) {
            cols[3 * cc] = D;
            cols[3 * cc + 1] = d;
            cols[3 * cc + 2] = t;
        } else {
            double2 *r = reinterpret_cast<double2 *>(rows + 6 * cc);
            r[0] = make_double2((double)D, (double)d);
            r[1] = make_double2((double)t, __hiloint2double(0, __float_as_int(D)));
        }
    }
    __syncwarp(g.mask);
    double v[6] = {0, 0, 0, 0, 0, 0};
    if (g.on) {
        double sD = 0, sd = 0, st = 0;
        const float DX = cols[3 * g.x];
        const double2 *r = reinterpret_cast<const double2 *>(rows + 6 * g.y0);
        const float *px_y = img + g.y0 * W + g.x;
#pragma unroll 4
        for (int y = g.y0; y < H; y += g.rp, r += 3 * g.rp, px_y += g.rp * W) {
            const double2 a = r[0], b = r[1];
            const float mu = p[3] + p[2] * DX * __int_as_float(__double2loint(b.y));
            const float I = *px_y;
            const double f = (double)(1.0f - I / mu);
            v[0] += (double)(mu - I * logf(mu));
            v[4] += f;
            sD = fma(a.x, f, sD);
            sd = fma(a.y, f, sd);
            st = fma(b.x, f, st);
        }
        const double I0 = p[2], D = DX;
        v[1] = I0 * cols[3 * g.x + 1] * sD;
        v[2] = I0 * D * sd;
        v[3] = D * sD;
        v[5] = I0 * (cols[3 * g.x + 2] * sD + D * st);
    }
    int first = 0, own = 6;
    fold_all<6, kLanes / 2>(v, g.lane, g.mask, first, own);
    if (own > 0) (first == 0 ? nll[roi] : grad[5 * roi + first - 1]) = (float)v[0];
}

using GaussKernel = void (*)(TrackParams, const uint8_t *, int, int64_t, const int64_t *, const LocalizationJob *, int,
                             LocalizationResult *);

// Two ROIs per warp as long as a row fits half a warp (16x16, 4 parameters: 0.404 ms with 16 lanes per ROI; 0.456 with
// 16 and 0.613 with 32 before the reciprocals became one instruction); wider rows would need two passes over the
// columns per step.
int gauss_lanes_per_roi(const TrackParams &P) { return P.width <= 16 ? 16 : 32; }

GaussKernel gauss_kernel_for(const TrackParams &P)
{
    const bool five = (P.mode & kLT_Gaussian5P) != 0;
    if (gauss_lanes_per_roi(P) == 16) return five ? gauss_warp_kernel<5, 16> : gauss_warp_kernel<4, 16>;
    return five ? gauss_warp_kernel<5, 32> : gauss_warp_kernel<4, 32>;
}

}  // namespace

cudaError_t prepare_gauss_kernels()
{
    const int half = 2 * kGaussWarps * gauss_smem(16, 32).bytes, whole = kGaussWarps * gauss_smem(32, 32).bytes;
    const struct {
        GaussKernel fn;
        int bytes;
    } all[] = {{gauss_warp_kernel<4, 16>, half}, {gauss_warp_kernel<5, 16>, half}, {gauss_warp_kernel<4, 32>, whole},
               {gauss_warp_kernel<5, 32>, whole}};
    cudaError_t e = cudaFuncSetAttribute(gauss_nll_warp_kernel<16>, cudaFuncAttributeMaxDynamicSharedMemorySize, half);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(gauss_nll_warp_kernel<32>, cudaFuncAttributeMaxDynamicSharedMemorySize, whole);
    if (e != cudaSuccess) return e;
    for (const auto &k : all) {
        e = cudaFuncSetAttribute(reinterpret_cast<const void *>(k.fn),
                                                   cudaFuncAttributeMaxDynamicSharedMemorySize, k.bytes);
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

bool use_gauss_nll_warp(const TrackParams &P) { return P.width <= 32 && P.height <= 32; }

cudaError_t launch_gauss_nll_warp(const TrackParams &P, const uint8_t *pixels, int pitch, int64_t roi_stride, int count,
                                  const float *params, float *nll, float *grad, cudaStream_t stream)
{
    const int lanes = gauss_lanes_per_roi(P), per_cta = 32 * kGaussWarps / lanes;
    const int grid = (count + per_cta - 1) / per_cta, bytes = per_cta * gauss_smem(P.width, P.height).bytes;
    (lanes == 16 ? gauss_nll_warp_kernel<16> : gauss_nll_warp_kernel<32>)<<<grid, 32 * kGaussWarps, bytes, stream>>>(
        P, pixels, pitch, roi_stride, count, params, nll, grad);
    return cudaGetLastError();
}

bool use_gauss_warp(const TrackParams &P)
{
    return (P.mode & kLT_Gaussian2D) && !(P.mode & (kLT_QI | kLT_LocalizeZ)) && P.width <= 32 && P.height <= 32;
}

void gauss_warp_node(const TrackParams &P, int count, cudaKernelNodeParams &kp)
{
    const int per_cta = 32 * kGaussWarps / gauss_lanes_per_roi(P);
    kp.func = reinterpret_cast<void *>(gauss_kernel_for(P));
    kp.gridDim = dim3((count + per_cta - 1) / per_cta);
    kp.blockDim = dim3(32 * kGaussWarps);
    kp.sharedMemBytes = per_cta * gauss_smem(P.width, P.height).bytes;
}

cudaError_t launch_gauss_warp(const TrackParams &P, const uint8_t *pixels, int pitch, int64_t roi_stride,
                              const int64_t *roi_offsets, const LocalizationJob *jobs, int count,
                              LocalizationResult *results, cudaStream_t stream)
{
    cudaKernelNodeParams kp{};
    gauss_warp_node(P, count, kp);
    gauss_kernel_for(P)<<<kp.gridDim, kp.blockDim, kp.sharedMemBytes, stream>>>(P, pixels, pitch, roi_stride,
                                                                               roi_offsets, jobs, count, results);
    return cudaGetLastError();
}

}  // namespace qtrk

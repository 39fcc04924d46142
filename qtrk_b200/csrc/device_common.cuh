// Device building blocks of the localization kernels (sm_100a).
//
// Each function restates one step of the reference CPU tracker for one ROI held in
// shared memory by one CTA; the reference file:line each follows is given beside it.
// Thread mappings are chosen for the GPU (one (quadrant, radius) bin per thread or
// per aligned lane group, warp-shuffle reductions, one warp for the QI FFTs); the
// discrete decisions (int truncation, the bilinear "outside" rule, sample-count
// thresholds, the argmax window of the quadratic fit) are those of the reference.
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

#include "qtrk_c_api.h"
#include "track_params.h"

namespace qtrk {

// -------------------------------------------------------------------------------------
// small helpers
// -------------------------------------------------------------------------------------
__device__ __forceinline__ float2 cmul(float2 a, float2 b)
{
    return make_float2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}

__device__ __forceinline__ int ilog2_pow2(int v) { return 31 - __clz(v); }

__device__ __forceinline__ unsigned bitrev(unsigned v, int bits) { return __brev(v) >> (32 - bits); }

// Sum N doubles over the whole CTA; every thread receives the totals.
// red: shared scratch of at least N * (blockDim.x / 32) doubles (256 doubles cover N <= 32
// at 256 threads).
template <int N>
__device__ __forceinline__ void block_sum(double (&v)[N], double *red)
{
#pragma unroll
    for (int k = 0; k < N; k++)
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v[k] += __shfl_xor_sync(0xffffffffu, v[k], o);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
    __syncthreads();
    if (lane == 0)
#pragma unroll
        for (int k = 0; k < N; k++) red[k * nw + warp] = v[k];
    __syncthreads();
#pragma unroll
    for (int k = 0; k < N; k++) {
        double s = 0;
        for (int w = 0; w < nw; w++) s += red[k * nw + w];
        v[k] = s;
    }
}

// Thread groups that process one ROI: the whole CTA, or one warp (small-ROI kernels).
struct BlockGroup {
    static constexpr int kFold = 64;  // pixels per FP32 partial sum of the COM
    double *red;  // >= N*32 doubles of shared scratch for sum<N>
    __device__ __forceinline__ int rank() const { return threadIdx.x; }
    __device__ __forceinline__ int size() const { return blockDim.x; }
    __device__ __forceinline__ void sync() const { __syncthreads(); }
    template <int N>
    __device__ __forceinline__ void sum(double (&v)[N]) const { block_sum<N>(v, red); }
};

// kLanes (16 or 32) consecutive lanes of a warp.
template <int kLanes>
struct LaneGroup {
    static constexpr int kFold = 4;  // 12x12 windows: with 8, COM errors 1.10-1.19 times those of 32 lanes a ROI
    __device__ __forceinline__ unsigned mask() const
    {
        return kLanes == 32 ? 0xffffffffu : ((1u << (kLanes & 31)) - 1u) << (threadIdx.x & 31 & ~(kLanes - 1));
    }
    __device__ __forceinline__ int rank() const { return threadIdx.x & (kLanes - 1); }
    __device__ __forceinline__ int size() const { return kLanes; }
    __device__ __forceinline__ void sync() const { __syncwarp(mask()); }
    template <int N>
    __device__ __forceinline__ void sum(double (&v)[N]) const
    {
#pragma unroll
        for (int k = 0; k < N; k++)
#pragma unroll
            for (int o = kLanes / 2; o > 0; o >>= 1) v[k] += __shfl_xor_sync(mask(), v[k], o);
    }
};

// Bilinear sampling follows Interpolate, utils.h:40-58: rx = (int)x (C truncation); the sample is outside when
// rx < 0, ry < 0, rx+1 >= w or ry+1 >= h. No float->int conversions: truncation keeps a sample inside
// exactly when -1 < x < w-1, and for those x, (int)x == floor(max(x, 0)), which a round-toward-zero add
// of 2^23 puts in the low mantissa bits. The fraction x - rx is formed from the same exact float as the
// reference's x - (float)rx, so the interpolated value is unchanged.

// True when every point cx + a*r, cy + b*r with |a|, |b| <= 1 (any sample of a circle of radius
// r around (cx, cy)) lies strictly inside (0, w-1) x (0, h-1), rounding of the sample
// coordinates included (margin 1e-3 px, far above one ulp of the coordinates).
__device__ __forceinline__ bool circle_inside(float cx, float cy, float r, int w, int h)
{
    const float m = 1e-3f;
    return cx - r > m && cy - r > m && cx + r < (float)(w - 1) - m && cy + r < (float)(h - 1) - m;
}

// CPUTracker::CheckBoundaries, cpu_tracker.cpp:182-188
__device__ __forceinline__ bool check_boundaries(float cx, float cy, float radius, int w, int h)
{
    return cx + radius >= w || cx - radius < 0 || cy + radius >= h || cy - radius < 0;
}

// LsqSqQuadFit + ComputeMaxInterp<T,7>::Compute (LsqQuadraticFit.h:8-176) in FP64, with the eight
// weighted sums formed by lanes 0..6 of one warp (all 32 lanes call; every lane returns the result).
// `at(i)` returns element i of the length-`len` array, iMax is the first index of the maximum;
// the weights are indexed from 0 even when the window is clipped at the array start, as in the
// reference. maxPos = iMax - b/(2a) with a = A/d, b = B/d, so the
// determinant d cancels and one division remains; |a| < 1e-9 is tested as |A| < 1e-9 |d|.
// y is element max(iMax - 3, 0) + lane of the array (read by lanes below the window's length). Not inlined:
// a rare path, and the localization kernel's time depends on how much of it stays in the instruction cache.
static __device__ __noinline__ double max_interp7_clipped(double y, int len, int iMax, const float (&wts)[7])
{
    const int lane = threadIdx.x & 31;
    const int startPos = max(iMax - 3, 0);
    const int endPos = min(iMax + 4, len);
    const int np = endPos - startPos;
    if (np < 3) return (double)iMax;
    double t[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    if (lane < np) {
        const double x = (double)(startPos + lane - iMax), wt = (double)wts[lane];
        const double sq = x * x;
        t[0] = x * wt;        // Sx
        t[1] = y * wt;        // Sy
        t[2] = sq * wt;       // Sx2
        t[3] = sq * x * wt;   // Sx3
        t[4] = sq * sq * wt;  // Sx4
        t[5] = x * y * wt;    // Sxy
        t[6] = sq * y * wt;   // Sx2y
        t[7] = wt;            // Sw
    }
#pragma unroll
    for (int k = 0; k < 8; k++)
#pragma unroll
        for (int o = 4; o > 0; o >>= 1) t[k] += __shfl_xor_sync(0xffffffffu, t[k], o);
#pragma unroll
    for (int k = 0; k < 8; k++) t[k] = __shfl_sync(0xffffffffu, t[k], 0);
    const double Sx = t[0], Sy = t[1], Sx2 = t[2], Sx3 = t[3], Sx4 = t[4], Sxy = t[5], Sx2y = t[6], Sw = t[7];
    const double d = Sx4 * (Sx2 * Sw - Sx * Sx) - Sx3 * (Sx3 * Sw - Sx * Sx2) + Sx2 * (Sx3 * Sx - Sx2 * Sx2);
    const double A = Sx2y * (Sx2 * Sw - Sx * Sx) - Sxy * (Sx3 * Sw - Sx * Sx2) + Sy * (Sx3 * Sx - Sx2 * Sx2);
    const double B = Sx4 * (Sxy * Sw - Sy * Sx) - Sx3 * (Sx2y * Sw - Sy * Sx2) + Sx2 * (Sx2y * Sx - Sxy * Sx2);
    if (fabs(A) < 1e-9 * fabs(d)) return (double)iMax;
    return (double)iMax - B / (2 * A);
}

template <typename Get>
__device__ __forceinline__ double max_interp7_warp(Get at, int len, int iMax, const float (&wts)[7])
{
    const int i = max(iMax - 3, 0) + (threadIdx.x & 31);
    return max_interp7_clipped(i < min(iMax + 4, len) ? (double)at(i) : 0.0, len, iMax, wts);
}

// The same fit for the common case, a window iMax-3 .. iMax+3 inside the array with weights
// symmetric about its centre (the reference's QIWeights and ZLUTWeights). Then S_x = S_x3 = 0
// and the cofactor expansion of LsqSqQuadFit::Coeff::abc reduces to
//   maxPos = iMax - (p0 / (2 Sx2)) N / D,  N = sum w x y,  D = sum w (x^2 Sw - Sx2) y,
//   p0 = Sx4 Sw - Sx2^2,  S_x^k = sum w x^k,  Sw = sum w,
// and a = D / p0 (the |a| < 1e-9 test). Both stencils sum to zero, so y is taken relative to
// y[iMax]: the two 7-term sums run in FP32 on small differences, which keeps the offset to ~1e-7
// of itself, with no FP64 and no cross-lane traffic. Clipped windows take max_interp7_warp.
// All 32 lanes of a warp call (with the same arguments); every lane returns the result.
template <typename Get>
__device__ __forceinline__ float max_interp7_sym(Get at, int len, int iMax, const float (&wts)[7])
{
    if (iMax < 3 || iMax + 4 > len) return (float)max_interp7_warp(at, len, iMax, wts);
    float Sw = 0.0f, Sx2 = 0.0f, Sx4 = 0.0f;
#pragma unroll
    for (int i = 0; i < 7; i++) {
        const float x2 = (float)((i - 3) * (i - 3)), w = wts[i];
        Sw += w;
        Sx2 += w * x2;
        Sx4 += w * x2 * x2;
    }
    const auto yc = at(iMax);
    float N = 0.0f, D = 0.0f;
#pragma unroll
    for (int i = 0; i < 7; i++) {
        if (i == 3) continue;  // y - y[iMax] = 0
        const float x = (float)(i - 3), w = wts[i];
        const float d = (float)(at(iMax - 3 + i) - yc);
        N += w * x * d;
        D += w * (x * x * Sw - Sx2) * d;
    }
    const float p0 = Sx4 * Sw - Sx2 * Sx2;
    if (fabsf(D) < 1e-9f * p0) return (float)iMax;
    return (float)iMax - (p0 / (2.0f * Sx2)) * (N / D);
}

// First index of the maximum of at(0..len), reduced over one warp (all 32 lanes call).
// Matches the strict ">" scan of LsqQuadraticFit.h:140-147 (NaN values never win).
template <typename Get>
__device__ __forceinline__ int warp_argmax(Get at, int len)
{
    using T = decltype(at(0));
    const int lane = threadIdx.x & 31;
    T best = 0;
    int bi = -1;
    for (int i = lane; i < len; i += 32) {
        const T v = at(i);
        if (v == v && (bi < 0 || v > best)) {
            best = v;
            bi = i;
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const T ov = __shfl_xor_sync(0xffffffffu, best, o);
        const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
        if (oi >= 0 && (bi < 0 || ov > best || (ov == best && oi < bi))) {
            best = ov;
            bi = oi;
        }
    }
    return bi < 0 ? 0 : bi;
}

// The words of job i (frame i and zeros without a job array) and the 13 words of a result.
__device__ __forceinline__ void read_job(const LocalizationJob *jobs, int i, uint32_t (&w)[6])
{
    if (jobs) {
        const uint32_t *p = reinterpret_cast<const uint32_t *>(jobs) + (size_t)i * 6;
#pragma unroll
        for (int k = 0; k < 6; k++) w[k] = p[k];
    } else {
        w[0] = (uint32_t)i;
#pragma unroll
        for (int k = 1; k < 6; k++) w[k] = 0;
    }
}

__device__ __forceinline__ void write_result(LocalizationResult *results, int i, const uint32_t (&job)[6], float x,
                                             float y, float z, float gx, float gy, uint32_t err, float mean)
{
    uint32_t *o = reinterpret_cast<uint32_t *>(results) + (size_t)i * 13;
#pragma unroll
    for (int k = 0; k < 6; k++) o[k] = job[k];
    o[6] = __float_as_uint(x);
    o[7] = __float_as_uint(y);
    o[8] = __float_as_uint(z);
    o[9] = __float_as_uint(gx);
    o[10] = __float_as_uint(gy);
    o[11] = err;
    o[12] = __float_as_uint(mean);
}

// -------------------------------------------------------------------------------------
// ROI load: u8/u16/f32 -> f32 tile in shared memory, with the clear-first-four-pixels
// option (QueuedCPUTracker.cpp:280-282) and the per-bead offset/gain step
// (cpu_tracker.cpp:98-112) fused into the same pass.
// -------------------------------------------------------------------------------------
// Exact conversion of an unsigned integer below 2^23 to float without the conversion pipe:
// placing it in the mantissa of 2^23 and subtracting 2^23.
__device__ __forceinline__ float u_to_float(uint32_t u) { return __uint_as_float(0x4B000000u | u) - 8388608.0f; }

__device__ __forceinline__ float finish_pixel(float v, int i, int mode, float off_factor, float gain_factor,
                                              const float *off, const float *gain)
{
    if ((mode & kLT_ClearFirstFourPixels) && i < 4) v = 0.0f;
    if (off && !gain) v = v + off[i] * off_factor;
    if (gain && !off) v = v * gain[i] * gain_factor;
    if (gain && off) v = (v + off[i] * off_factor) * gain[i] * gain_factor;
    return v;
}

// Sums of v and v^2 over a thread's pixels. A CTA's threads add their few dozen pixels in FP32; the lanes of a group,
// which have up to twice as many of a small ROI with 16 lanes as with 32, fold theirs into FP64 after every two.
template <class G>
struct PixelSums {
    static constexpr bool kFolds = G::kFold == 4;
    float s = 0.0f, s2 = 0.0f;
    double d = 0.0, d2 = 0.0;
    __device__ __forceinline__ void add(float v)
    {
        s += v;
        s2 = fmaf(v, v, s2);
    }
    __device__ __forceinline__ void fold()  // after every two pixels
    {
        if (!kFolds) return;
        d += (double)s;
        d2 += (double)s2;
        s = s2 = 0.0f;
    }
    __device__ __forceinline__ double2 total() const
    {
        return kFolds ? make_double2(d + (double)s, d2 + (double)s2) : make_double2((double)s, (double)s2);
    }
};

// Returns this thread's partial sums of v and v^2 over the pixels it converted (the first pass
// of CPUTracker::ComputeMeanAndCOM, cpu_tracker.cpp:687-693, so that com_from_sums need not read
// the tile again for them; callers that do not use them pay nothing once the call is inlined).
template <class G>
__device__ inline double2 load_roi(const G &g, float *img, const uint8_t *src, int pitch, const TrackParams &P, int bead)
{
    const int W = P.width, H = P.height, n = W * H;
    const int bpp = P.pdt == 0 ? 1 : (P.pdt == 1 ? 2 : 4);
    const float *off = nullptr, *gain = nullptr;
    if (bead >= 0 && bead < P.calib_count) {
        if (P.calib_offset) off = P.calib_offset + (size_t)bead * n;
        if (P.calib_gain) gain = P.calib_gain + (size_t)bead * n;
    }
    const bool contiguous = pitch == W * bpp && ((reinterpret_cast<uintptr_t>(src) & 15) == 0) &&
                            ((n * bpp) & 15) == 0 && ((reinterpret_cast<uintptr_t>(img) & 15) == 0);
    PixelSums<G> sums;
    if (contiguous) {
        // Rows are back to back: the ROI is a run of n/4 chunks of four pixels (4, 8 or 16 input
        // bytes), and chunk c becomes the float4 at img + 4c, so a warp's stores fill 512
        // contiguous bytes of shared memory without bank conflicts. Each thread issues
        // kBatch streaming loads (8-16 registers' worth) before converting any of them, so the
        // HBM latency is paid about once per batch rather than once per load.
        const int nc = n >> 2;
        const bool plain = !off && !gain && !(P.mode & kLT_ClearFirstFourPixels);
        float4 *dst = reinterpret_cast<float4 *>(img);
        auto finish4 = [&](float4 f, int c) {
            if (!plain) {
                f.x = finish_pixel(f.x, 4 * c, P.mode, P.offset_factor, P.gain_factor, off, gain);
                f.y = finish_pixel(f.y, 4 * c + 1, P.mode, P.offset_factor, P.gain_factor, off, gain);
                f.z = finish_pixel(f.z, 4 * c + 2, P.mode, P.offset_factor, P.gain_factor, off, gain);
                f.w = finish_pixel(f.w, 4 * c + 3, P.mode, P.offset_factor, P.gain_factor, off, gain);
            }
            sums.add(f.x);
            sums.add(f.y);
            sums.fold();
            sums.add(f.z);
            sums.add(f.w);
            sums.fold();
            dst[c] = f;
        };
        if (P.pdt == 0) {
            constexpr int kBatch = 8;
            const uint32_t *s1 = reinterpret_cast<const uint32_t *>(src);
            for (int c0 = g.rank(); c0 < nc; c0 += kBatch * g.size()) {
                uint32_t q[kBatch];
#pragma unroll
                for (int k = 0; k < kBatch; k++) {
                    const int c = c0 + k * g.size();
                    if (c < nc) q[k] = __ldcs(s1 + c);
                }
#pragma unroll
                for (int k = 0; k < kBatch; k++) {
                    const int c = c0 + k * g.size();
                    if (c >= nc) break;
                    finish4(make_float4(u_to_float(q[k] & 0xffu), u_to_float((q[k] >> 8) & 0xffu),
                                        u_to_float((q[k] >> 16) & 0xffu), u_to_float(q[k] >> 24)),
                            c);
                }
            }
        } else if (P.pdt == 1) {
            constexpr int kBatch = 8;
            const uint2 *s2 = reinterpret_cast<const uint2 *>(src);
            for (int c0 = g.rank(); c0 < nc; c0 += kBatch * g.size()) {
                uint2 q[kBatch];
#pragma unroll
                for (int k = 0; k < kBatch; k++) {
                    const int c = c0 + k * g.size();
                    if (c < nc) q[k] = __ldcs(s2 + c);
                }
#pragma unroll
                for (int k = 0; k < kBatch; k++) {
                    const int c = c0 + k * g.size();
                    if (c >= nc) break;
                    finish4(make_float4(u_to_float(q[k].x & 0xffffu), u_to_float(q[k].x >> 16),
                                        u_to_float(q[k].y & 0xffffu), u_to_float(q[k].y >> 16)),
                            c);
                }
            }
        } else {
            constexpr int kBatch = 4;
            const float4 *s4 = reinterpret_cast<const float4 *>(src);
            for (int c0 = g.rank(); c0 < nc; c0 += kBatch * g.size()) {
                float4 q[kBatch];
#pragma unroll
                for (int k = 0; k < kBatch; k++) {
                    const int c = c0 + k * g.size();
                    if (c < nc) q[k] = __ldcs(s4 + c);
                }
#pragma unroll
                for (int k = 0; k < kBatch; k++) {
                    const int c = c0 + k * g.size();
                    if (c >= nc) break;
                    finish4(q[k], c);
                }
            }
        }
    } else {
        // Rows at a pitch (a ROI inside a frame): warps over rows, lanes along a row, so loads
        // are coalesced along the row and the stores are conflict-free. Rows back to back that are
        // not whole aligned 16-byte units (odd ROI sizes) are one flat run, loaded in batches of
        // eight so that the latency is paid per batch and not per row.
        // The partial sums are then taken from the tile, with whole 4-pixel chunks in the chunk
        // order of the contiguous loads, so that a ROI gives bit-identical results whichever way
        // it arrived (FP32 partial sums depend on which pixels each thread adds).
        const bool chunked = !(n & 3) && !(reinterpret_cast<uintptr_t>(img) & 15);
        auto pixel = [&](const uint8_t *row, int x) {
            if (P.pdt == 0) return u_to_float(row[x]);
            if (P.pdt == 1) return u_to_float(reinterpret_cast<const uint16_t *>(row)[x]);
            return reinterpret_cast<const float *>(row)[x];
        };
        if (pitch == W * bpp) {
            constexpr int kBatch = 8;
            for (int i0 = g.rank(); i0 < n; i0 += kBatch * g.size()) {
                float v[kBatch];
#pragma unroll
                for (int k = 0; k < kBatch; k++) {
                    const int i = i0 + k * g.size();
                    if (i < n) v[k] = pixel(src, i);
                }
#pragma unroll
                for (int k = 0; k < kBatch; k++) {
                    const int i = i0 + k * g.size();
                    if (i < n) img[i] = finish_pixel(v[k], i, P.mode, P.offset_factor, P.gain_factor, off, gain);
                }
            }
        } else {
            const int rl = min(g.size(), 32);  // lanes along a row
            const int lane = g.rank() & (rl - 1), wg = g.rank() / rl, nwg = g.size() / rl;
            for (int y = wg; y < H; y += nwg) {
                const uint8_t *row = src + (size_t)y * pitch;
#pragma unroll 4
                for (int x = lane; x < W; x += rl) {
                    const int i = y * W + x;
                    img[i] = finish_pixel(pixel(row, x), i, P.mode, P.offset_factor, P.gain_factor, off, gain);
                }
            }
        }
        g.sync();
        if (!chunked) {
            int k = 0;
            for (int i = g.rank(); i < n; i += g.size()) {
                sums.add(img[i]);
                if (!(++k & 1)) sums.fold();
            }
        }
        if (chunked) {
            const float4 *img4 = reinterpret_cast<const float4 *>(img);
            for (int c = g.rank(); c < (n >> 2); c += g.size()) {
                const float4 f = img4[c];
                sums.add(f.x);
                sums.add(f.y);
                sums.fold();
                sums.add(f.z);
                sums.add(f.w);
                sums.fold();
            }
        }
    }
    g.sync();
    return sums.total();
}

// -------------------------------------------------------------------------------------
// CPUTracker::ComputeMeanAndCOM, cpu_tracker.cpp:681-729 (FP64 accumulation as in the
// reference; mean and stdev rounded to float where the reference stores floats).
// -------------------------------------------------------------------------------------
struct ComResult {
    float x, y, mean, stdev;
};

// From this thread's partial sums of v and v^2 (first pass, part) and the tile: the FP64 sums
// across the group, mean and stdev as the reference rounds them, then the background-corrected
// moments. Each thread walks a fixed set of pixels with its column/row as float counters, keeps
// FP32 partial sums over its few dozen pixels, and the partials are added in FP64 across the
// group (the reference accumulates the whole image in FP64; the partial sums keep its result
// to ~1e-7 relative, far inside the 1e-4 px COM tolerance; for integer pixels the first pass's
// partial sums, and so the mean, are exact).
template <class G>
__device__ ComResult com_from_sums(const G &g, const float *img, int W, int H, double2 part, float bgcorr)
{
    const int n = W * H, stride = g.size();
    const int dx = stride % W, dy = stride / W;
    double s[2] = {part.x, part.y};
    g.sum(s);
    const float invN = 1.0f / (float)n;
    ComResult r;
    r.mean = (float)(s[0] * (double)invN);
    r.stdev = sqrtf((float)(s[1] * (double)invN - (double)(r.mean * r.mean)));
    const float thr = bgcorr * r.stdev;
    double m[3] = {0.0, 0.0, 0.0};
    if (!(W & 3) && !(reinterpret_cast<uintptr_t>(img) & 15)) {
        // rows are whole float4 chunks: chunk c holds pixels 4c .. 4c+3 of one row, at column fx
        // and row fy; per chunk S = sum v', Sj = sum j v', so sum x v' = fx S + Sj
        const int nc = n >> 2, cstride = stride * 4;
        const float fW = (float)W, fdx = (float)(cstride % W), fdy = (float)(cstride / W);
        float fx = (float)((4 * g.rank()) % W), fy = (float)((4 * g.rank()) / W);
        const float4 *img4 = reinterpret_cast<const float4 *>(img);
        for (int c = g.rank(); c < nc;) {
            float q0 = 0.0f, qx = 0.0f, qy = 0.0f;
            for (const int end = min(nc, c + G::kFold / 4 * stride); c < end; c += stride) {
                const float4 q = img4[c];
                float a0, a1, a2, a3;
                if (thr == 0.0f) {  // max(0, |d| - 0) is |d|
                    a0 = fabsf(q.x - r.mean);
                    a1 = fabsf(q.y - r.mean);
                    a2 = fabsf(q.z - r.mean);
                    a3 = fabsf(q.w - r.mean);
                } else {
                    a0 = fmaxf(0.0f, fabsf(q.x - r.mean) - thr);
                    a1 = fmaxf(0.0f, fabsf(q.y - r.mean) - thr);
                    a2 = fmaxf(0.0f, fabsf(q.z - r.mean) - thr);
                    a3 = fmaxf(0.0f, fabsf(q.w - r.mean) - thr);
                }
                const float S = (a0 + a1) + (a2 + a3);
                const float Sj = fmaf(3.0f, a3, fmaf(2.0f, a2, a1));
                q0 += S;
                qx += fmaf(fx, S, Sj);
                qy = fmaf(fy, S, qy);
                fx += fdx;
                fy += fdy;
                if (fx >= fW) {
                    fx -= fW;
                    fy += 1.0f;
                }
            }
            m[0] += (double)q0;
            m[1] += (double)qx;
            m[2] += (double)qy;
        }
    } else {
        int x = g.rank() % W, y = g.rank() / W;
        float fx = (float)x, fy = (float)y;
        for (int i = g.rank(); i < n;) {
            float q0 = 0.0f, qx = 0.0f, qy = 0.0f;
            for (const int end = min(n, i + G::kFold * stride); i < end; i += stride) {
                const float v = fmaxf(0.0f, fabsf(img[i] - r.mean) - thr);
                q0 += v;
                qx += fx * v;
                qy += fy * v;
                x += dx;
                fx += (float)dx;
                fy += (float)dy;
                if (x >= W) {
                    x -= W;
                    fx -= (float)W;
                    fy += 1.0f;
                }
            }
            m[0] += (double)q0;
            m[1] += (double)qx;
            m[2] += (double)qy;
        }
    }
    g.sum(m);
    r.x = (float)(m[1] / m[0]);
    r.y = (float)(m[2] / m[0]);
    return r;
}

// Radix-2 decimation-in-time FFT of length L (power of two, input in bit-reversed order),
// executed by one warp over shared memory. tw[k] = e^{-2 pi i k / L}, k < L/2.
// Stage s pairs (i, i + 2^(s-1)) with twiddle tw[(i mod 2^(s-1)) * (L >> s)]. Two consecutive
// stages are done together in registers on groups of four elements, which halves the
// shared-memory round trips and warp barriers without changing any butterfly.
__device__ __forceinline__ float2 fft_tw(const float2 *tw, int k, bool inverse)
{
    float2 w = tw[k];
    if (inverse) w.y = -w.y;
    return w;
}

__device__ inline void warp_fft(float2 *buf, int L, int log2L, const float2 *tw, bool inverse)
{
    const int lane = threadIdx.x & 31;
    int s = 1;
    if (log2L & 1) {  // a single radix-2 stage first (twiddle 1)
        for (int j = lane; j < (L >> 1); j += 32) {
            const float2 a = buf[2 * j], b = buf[2 * j + 1];
            buf[2 * j] = make_float2(a.x + b.x, a.y + b.y);
            buf[2 * j + 1] = make_float2(a.x - b.x, a.y - b.y);
        }
        __syncwarp();
        s = 2;
    }
    for (; s < log2L; s += 2) {
        const int h = 1 << (s - 1);
        for (int j = lane; j < (L >> 2); j += 32) {
            const int pos = j & (h - 1);
            const int i0 = ((j >> (s - 1)) << (s + 1)) + pos;
            float2 a0 = buf[i0], a1 = buf[i0 + h], a2 = buf[i0 + 2 * h], a3 = buf[i0 + 3 * h];
            const float2 w1 = fft_tw(tw, pos * (L >> s), inverse);
            float2 b = cmul(a1, w1);
            a1 = make_float2(a0.x - b.x, a0.y - b.y);
            a0 = make_float2(a0.x + b.x, a0.y + b.y);
            b = cmul(a3, w1);
            a3 = make_float2(a2.x - b.x, a2.y - b.y);
            a2 = make_float2(a2.x + b.x, a2.y + b.y);
            const float2 w2 = fft_tw(tw, pos * (L >> (s + 1)), inverse);
            const float2 w3 = fft_tw(tw, (pos + h) * (L >> (s + 1)), inverse);
            b = cmul(a2, w2);
            buf[i0] = make_float2(a0.x + b.x, a0.y + b.y);
            buf[i0 + 2 * h] = make_float2(a0.x - b.x, a0.y - b.y);
            b = cmul(a3, w3);
            buf[i0 + h] = make_float2(a1.x + b.x, a1.y + b.y);
            buf[i0 + 3 * h] = make_float2(a1.x - b.x, a1.y - b.y);
        }
        __syncwarp();
    }
}

// The unnormalised correlation of each concatenated profile p with its reverse, as
// produced by CPUTracker::QI_ComputeOffset (cpu_tracker.cpp:375-401):
//   out[n] = L * sum_m p[(n+m) mod L] * p[L-1-m].
// Both axes are packed into one complex signal z = px + i py. Because
// FFT(reverse(p))* = e^{-2 pi i k/L} FFT(p) for real p, the product the reference forms
// from two forward FFTs equals e^{-2 pi i k/L} P[k]^2, so one forward and one inverse
// FFT per iteration give both axes. Result: ac[n] = (out_x[n], out_y[n]). A holds the packed
// profile in bit-reversed order on entry (as qi_profiles writes it). Warp 0 only.
__device__ inline void qi_autoconv_fft_filled(int nr, float2 *A, float2 *ac, const float2 *tw)
{
    const int lane = threadIdx.x & 31;
    const int L = 2 * nr, log2L = ilog2_pow2(L);
    warp_fft(A, L, log2L, tw, false);
    for (int k = lane; k < L; k += 32) {
        const float2 Zk = A[k];
        const float2 Zc = A[(L - k) & (L - 1)];
        // split the packed transform: Px = (Z[k] + conj Z[L-k]) / 2, Py = (Z[k] - conj Z[L-k]) / 2i
        const float2 Px = make_float2(0.5f * (Zk.x + Zc.x), 0.5f * (Zk.y - Zc.y));
        const float2 Py = make_float2(0.5f * (Zk.y + Zc.y), -0.5f * (Zk.x - Zc.x));
        float2 e = tw[k & ((L >> 1) - 1)];
        if (k >= (L >> 1)) e = make_float2(-e.x, -e.y);
        const float2 Ax = cmul(e, cmul(Px, Px));
        const float2 Ay = cmul(e, cmul(Py, Py));
        ac[bitrev(k, log2L)] = make_float2(Ax.x - Ay.y, Ax.y + Ay.x);
    }
    __syncwarp();
    warp_fft(ac, L, log2L, tw, true);
}


// The same correlation for L = 32 E (E = 1, 2, 4, 8 or 16), held in the registers of one warp: lane l has the
// elements l + 32 e. The transform over e runs inside the lane, the 32-point transforms over the lanes by
// shuffles (decimation in frequency forward, in time back, so no reordering pass lies between them:
// lane l, slot e holds frequency bitrev(e) + E bitrev(l)). A holds the packed profile in natural order. The
// passes through shared memory above load four elements and three twiddles per butterfly group and wait at a
// warp barrier after each: with the fit, 3.8 k cycles for one update of 2 nr = 128 points alone on an SM, against
// 1.5 k here (the instructions cached).
__device__ __forceinline__ constexpr int bitrev_c(int v, int bits)
{
    int r = 0;
    for (int i = 0; i < bits; i++) r |= ((v >> i) & 1) << (bits - 1 - i);
    return r;
}

// z * e^{-2 pi i J / N} (or its conjugate) for compile-time J, N with N <= 16.
template <int N, int J>
__device__ __forceinline__ float2 cmul_root(float2 z, bool conj)
{
    constexpr float c16[4] = {1.0f, 0.92387953251128675613f, 0.70710678118654752440f, 0.38268343236508977173f};
    constexpr int j = J * (16 / N);  // sixteenths of a turn, 0 .. 7
    if constexpr (j == 0) return z;
    if constexpr (j == 4) return conj ? make_float2(-z.y, z.x) : make_float2(z.y, -z.x);
    constexpr float wr = j < 4 ? c16[j & 3] : -c16[(8 - j) & 3];
    constexpr float wi = -(j < 4 ? c16[(4 - j) & 3] : c16[(j - 4) & 3]);
    const float s = conj ? -wi : wi;
    return make_float2(z.x * wr - z.y * s, z.x * s + z.y * wr);
}

template <int E, int H, int I = 0>
__device__ __forceinline__ void lane_dif_stage(float2 (&z)[E])
{
    if constexpr (I < E) {
        if constexpr ((I & H) == 0) {
            const float2 a = z[I], b = z[I + H];
            z[I] = make_float2(a.x + b.x, a.y + b.y);
            z[I + H] = cmul_root<2 * H, I & (H - 1)>(make_float2(a.x - b.x, a.y - b.y), false);
        }
        lane_dif_stage<E, H, I + 1>(z);
    }
}

template <int E, int H, int I = 0>
__device__ __forceinline__ void lane_dit_stage(float2 (&z)[E])
{
    if constexpr (I < E) {
        if constexpr ((I & H) == 0) {
            const float2 a = z[I], b = cmul_root<2 * H, I & (H - 1)>(z[I + H], true);
            z[I] = make_float2(a.x + b.x, a.y + b.y);
            z[I + H] = make_float2(a.x - b.x, a.y - b.y);
        }
        lane_dit_stage<E, H, I + 1>(z);
    }
}

template <int E, int H = E / 2>
__device__ __forceinline__ void lane_dif(float2 (&z)[E])
{
    if constexpr (H >= 1) {
        lane_dif_stage<E, H>(z);
        lane_dif<E, H / 2>(z);
    }
}

template <int E, int H = 1>
__device__ __forceinline__ void lane_dit(float2 (&z)[E])
{
    if constexpr (H < E) {
        lane_dit_stage<E, H>(z);
        lane_dit<E, 2 * H>(z);
    }
}

__device__ __forceinline__ float2 shfl2(float2 v, int src)
{
    return make_float2(__shfl_sync(0xffffffffu, v.x, src), __shfl_sync(0xffffffffu, v.y, src));
}

__device__ __forceinline__ float2 shfl2_xor(float2 v, int o)
{
    return make_float2(__shfl_xor_sync(0xffffffffu, v.x, o), __shfl_xor_sync(0xffffffffu, v.y, o));
}

// tw[k] = e^{-2 pi i k / L}, k < L/2. On return z[e] of lane l is (out_x[n], out_y[n]) at n = l + 32 e.
template <int E>
__device__ __forceinline__ void qi_autoconv_regs(const float2 *A, const float2 *tw, float2 (&z)[E])
{
    constexpr int L = 32 * E, lE = E == 1 ? 0 : (E == 2 ? 1 : (E == 4 ? 2 : (E == 8 ? 3 : 4)));
    const int lane = threadIdx.x & 31;
    auto root = [&](int k) {  // e^{-2 pi i k / L}, k < L
        const float2 w = tw[k & (L / 2 - 1)];
        return k & (L / 2) ? make_float2(-w.x, -w.y) : w;
    };
#pragma unroll
    for (int e = 0; e < E; e++) z[e] = A[lane + 32 * e];
    float2 t[4];  // twiddles of the lane distances 16, 8, 4, 2 (1 for the lanes that keep the sum)
#pragma unroll
    for (int s = 0; s < 4; s++) {
        const int d = 16 >> s;
        t[s] = (lane & d) ? tw[((lane & (d - 1)) << s) * E] : make_float2(1.0f, 0.0f);
    }
    lane_dif<E>(z);
#pragma unroll
    for (int e = 1; e < E; e++) z[e] = cmul(z[e], root(lane * bitrev_c(e, lE)));
#pragma unroll
    for (int s = 0; s < 5; s++) {
        const int d = 16 >> s;
        const float sg = (lane & d) ? -1.0f : 1.0f;
#pragma unroll
        for (int e = 0; e < E; e++) {
            const float2 o = shfl2_xor(z[e], d);
            z[e] = make_float2(fmaf(sg, z[e].x, o.x), fmaf(sg, z[e].y, o.y));
            if (s < 4) z[e] = cmul(z[e], t[s]);
        }
    }
    // split the packed transform (see qi_autoconv_fft_filled): the conjugate frequency L - k lies in the
    // mirrored lane's slot E - q, for q = 0 in its own slot of the lane that holds -m mod 32
    const int m = (int)bitrev(lane, 5), opp = (int)bitrev((32 - m) & 31, 5);
    float2 p[E];
#pragma unroll
    for (int e = 0; e < E; e++) {
        const int q = bitrev_c(e, lE);
        const float2 Zk = z[e], Zc = q == 0 ? shfl2(z[0], opp) : shfl2_xor(z[bitrev_c((E - q) & (E - 1), lE)], 31);
        const float2 Px = make_float2(0.5f * (Zk.x + Zc.x), 0.5f * (Zk.y - Zc.y));
        const float2 Py = make_float2(0.5f * (Zk.y + Zc.y), -0.5f * (Zk.x - Zc.x));
        const float2 X = cmul(Px, Px), Y = cmul(Py, Py);
        p[e] = cmul(root(q + E * m), make_float2(X.x - Y.y, X.y + Y.x));
    }
#pragma unroll
    for (int s = 4; s >= 0; s--) {
        const int d = 16 >> s;
        const float sg = (lane & d) ? -1.0f : 1.0f;
#pragma unroll
        for (int e = 0; e < E; e++) {
            const float2 v = s < 4 ? cmul(p[e], make_float2(t[s].x, -t[s].y)) : p[e];
            const float2 o = shfl2_xor(v, d);
            p[e] = make_float2(fmaf(sg, v.x, o.x), fmaf(sg, v.y, o.y));
        }
    }
#pragma unroll
    for (int e = 0; e < E; e++) {
        const float2 w = e > 0 ? root(lane * bitrev_c(e, lE)) : make_float2(1.0f, 0.0f);
        z[e] = e > 0 ? cmul(p[e], make_float2(w.x, -w.y)) : p[e];
    }
    lane_dit<E>(z);
}

// warp_argmax over doubles: the keys' high and low words reduced in turn, then the smallest index.
template <typename Get>
__device__ __forceinline__ int warp_argmax_f64(Get at, int len)
{
    const int lane = threadIdx.x & 31;
    long long best = (long long)0x8000000000000000ull;
    int bi = 0x7fffffff;
    for (int i = lane; i < len; i += 32) {
        const double v = at(i) + 0.0;
        long long k = __double_as_longlong(v);
        k = v == v ? k ^ ((k >> 63) & 0x7fffffffffffffffll) : (long long)0x8000000000000000ull;
        if (k > best) {
            best = k;
            bi = i;
        }
    }
    const int hi = (int)(best >> 32), mhi = __reduce_max_sync(0xffffffffu, hi);
    const unsigned lo = hi == mhi ? (unsigned)best : 0u, mlo = __reduce_max_sync(0xffffffffu, lo);
    bi = __reduce_min_sync(0xffffffffu, hi == mhi && lo == mlo ? bi : 0x7fffffff);
    return bi == 0x7fffffff ? 0 : bi;
}

// A float as a signed integer of the same order; NaN below everything, -0 with +0.
__device__ __forceinline__ int order_key(float v)
{
    const int b = __float_as_int(v + 0.0f);
    return v == v ? b ^ ((b >> 31) & 0x7fffffff) : (int)0x80000000;
}

// The score of CPUTracker::LUTProfileCompare (cpu_tracker.cpp:820-830): -sum_r d^2 with d = (double)(p_r -
// L_kr), the difference taken in FP32 as the reference takes it, then d *= w_r, summed in FP64. The bins are
// cut into zlut_runs(planes) runs whose sums meet pairwise (0+1, 2+3, ...), in this order wherever a score
// is formed, so that it does not depend on which kernel asks (FP64 rounding differs from a single run's
// by about 1e-16 of the sum).
// Runs: 1, 2, 4 or 8 neighbouring threads share four planes as long as 128 threads suffice for all planes.
__device__ __forceinline__ int zlut_log2_runs(int planes)
{
    int lg = 0;
    while (lg < 3 && ((planes + 3) >> 2) << (lg + 1) <= 128) lg++;
    return lg;
}

// One plane's score; lut_k[r] is L_kr.
__device__ __forceinline__ double zlut_score(const float *prof, const float *lut_k, const float *w, int nb, int planes)
{
    const int lg = zlut_log2_runs(planes), len = (nb + (1 << lg) - 1) >> lg;
    double part[3] = {0.0, 0.0, 0.0}, v = 0.0;  // part: pending sums of 1, 2 and 4 runs
    for (int s = 0; s < 1 << lg; s++) {
        v = 0.0;
        const int end = min(nb, (s + 1) * len);
#pragma unroll 8
        for (int r = s * len; r < end; r++) {
            double d = (double)(prof[r] - __ldg(lut_k + r));
            if (w) d *= (double)__ldg(w + r);
            v = fma(d, d, v);
        }
        if (s & 1) v = part[0] + v;
        if ((s & 3) == 3) v = part[1] + v;
        if ((s & 7) == 7) v = part[2] + v;
        if (!(s & 1)) part[0] = v;
        if ((s & 3) == 1) part[1] = v;
        if ((s & 7) == 3) part[2] = v;
    }
    return -v;
}

// The plain Z match over the transposed LUT ([bin][plane], `pitch` planes per bin, a multiple of 32): a thread
// takes four planes (16-byte loads, four independent FP64 chains) over one run of bins. What a thread waits for
// is the LUT (L2): one thread per plane over all bins in turn took 17.2 k of a 100x100 ROI's 146 k cycles (200 planes
// x 64 bins, 128 threads, full load), this 7.1 k.
template <int T, bool kWeights>
__device__ __forceinline__ void zlut_scores_runs(const float *prof, const float4 *lut4, int pitch4, int planes, int nb,
                                                 const float *weights, double *scores)
{
    const int quads = (planes + 3) >> 2, lg = zlut_log2_runs(planes), len = (nb + (1 << lg) - 1) >> lg;
    const int total = quads << lg;
    // loads in flight per thread: more where one ROI has the SM to itself and waits for the LUT
    constexpr int kUnroll = T >= 256 ? 8 : 4;
    for (int base = 0; base < total; base += T) {  // uniform: the sums below shuffle whole warps
        const int t = base + threadIdx.x;
        if ((t & ~31) >= total) break;  // whole warps
        const int q = min(t >> lg, quads - 1), h = t & ((1 << lg) - 1);
        const int r0 = h * len, r1 = min(nb, r0 + len);
        const float4 *l = lut4 + (size_t)r0 * pitch4 + q;
        double v[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll kUnroll
        for (int r = r0; r < r1; r++, l += pitch4) {
            const float4 f = __ldg(l);
            const float p = prof[r];
            double d[4] = {(double)(p - f.x), (double)(p - f.y), (double)(p - f.z), (double)(p - f.w)};
            const double w = kWeights ? (double)__ldg(weights + r) : 1.0;
#pragma unroll
            for (int i = 0; i < 4; i++) {
                if (kWeights) d[i] *= w;
                v[i] = fma(d[i], d[i], v[i]);
            }
        }
        for (int o = 1; o < 1 << lg; o <<= 1)
#pragma unroll
            for (int i = 0; i < 4; i++) v[i] += __shfl_xor_sync(0xffffffffu, v[i], o);
        if (t < total && h == 0)
#pragma unroll
            for (int i = 0; i < 4; i++)
                if (4 * q + i < planes) scores[4 * q + i] = -v[i];
    }
    __syncthreads();
}

template <int T>
__device__ __forceinline__ void zlut_scores_plain(const float *prof, const float *lut_t, int pitch, int planes, int nb,
                                                  const float *weights, double *scores)
{
    const float4 *lut4 = reinterpret_cast<const float4 *>(lut_t);
    if (weights)
        zlut_scores_runs<T, true>(prof, lut4, pitch >> 2, planes, nb, weights, scores);
    else
        zlut_scores_runs<T, false>(prof, lut4, pitch >> 2, planes, nb, weights, scores);
}

// QueuedTracker::ZLUTBiasCorrection, cputrack/QueuedTracker.cpp:115-140: four fixed-point steps
// pos = z - bias(pos), bias read from the bead's row of the table by Interpolate1D
// (cputrack/utils.h:60-67: truncating index, clamped to the first/last entry).
__device__ __forceinline__ float zlut_bias_correct(float z, int planes, const float *table, int tw, int tcount,
                                                   int bead)
{
    if (!table || bead < 0 || bead >= tcount || tw <= 0) return z;
    const float *row = table + (size_t)bead * tw;
    float pos = z;
    for (int k = 0; k < 4; k++) {
        const float tblpos = pos / (float)planes * tw;
        const int fx = (int)tblpos;
        float bias;
        if (fx < 0)
            bias = row[0];
        else if (fx >= tw - 1)
            bias = row[tw - 1];
        else
            bias = (row[fx + 1] - row[fx]) * (tblpos - fx) + row[fx];
        pos = z - bias;
    }
    return pos;
}

// -------------------------------------------------------------------------------------
// 2D Gaussian MLE, CPUTracker::Compute2DGaussianMLE (cpu_tracker.cpp:514-589):
// 4 parameters (x, y, I0, bg), fixed sigma, per-parameter Newton steps. The erf is the
// Abramowitz & Stegun 7.1.26 form the reference binds (utils.h:395-417). Per iteration the
// erf/exp terms depend only on the column (x) or the row (y), so they are evaluated once
// per column and per row and combined per pixel.
// -------------------------------------------------------------------------------------
// 1 / x to 1 ulp, subnormal x as zero (one special-function instruction).
__device__ __forceinline__ float rcp(float x)
{
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

__device__ __forceinline__ float erf_as(float x, float e_mx2)
{
    // e_mx2 = exp(-x*x)
    const float a1 = 0.254829592f, a2 = -0.284496736f, a3 = 1.421413741f, a4 = -1.453152027f,
                a5 = 1.061405429f, p = 0.3275911f;
    const float sign = x < 0 ? -1.0f : 1.0f;
    const float ax = fabsf(x);
    // the reciprocal refined once: within rounding of the quotient, which the fit's error shows (4 parameters, 12 to 24
    // px: as with a division; 1.003-1.024 times that with the unrefined reciprocal). Bounded, as inf * 0 is not a number.
    const float a = 1.0f + p * fminf(ax, 1e30f), r = rcp(a), t = fmaf(fmaf(-a, r, 1.0f), r, r);
    const float y = 1.0f - (((((a5 * t + a4) * t) + a3) * t + a2) * t + a1) * t * e_mx2;
    return sign * y;
}

// Column (or row) terms for coordinate c at position p: D = 0.5 erf(c0) - 0.5 erf(c1),
// g = e^{-c1^2} - e^{-c0^2}, h = (c-p-.5) e^{-c1^2} - (c-p+.5) e^{-c0^2}.
struct GaussAxisTerms {
    float D, g, h;
};

__device__ __forceinline__ GaussAxisTerms gauss_axis_terms(int c, float p, float k1)
{
    const float e0 = (c - p + .5f) * k1;
    const float e1 = (c - p - .5f) * k1;
    const float x0 = expf(-e0 * e0), x1 = expf(-e1 * e1);
    GaussAxisTerms t;
    t.D = 0.5f * erf_as(e0, x0) - 0.5f * erf_as(e1, x1);
    t.g = x1 - x0;
    t.h = (c - p - .5f) * x1 - (c - p + .5f) * x0;
    return t;
}


// CPUTracker::Compute2DGaussianMLE, cpu_tracker.cpp:514-589. col: 3*W floats, row: 3*H floats
// of shared scratch. px/py enter as the start position (the COM) and leave as the estimate.
template <class G>
__device__ inline void gauss4_mle(const G &g, const float *img, int W, int H, float mean, float &px, float &py, int iters,
                           float sigma, float *col, float *row)
{
    float I0 = mean * 0.5f * (float)W * (float)H;
    float bg = mean * 0.5f;
    const float k1 = 1.0f / (sqrtf(2.0f) * sigma);
    const float k2 = 1.0f / (sqrtf(2 * 3.14159265359f) * sigma);
    const float k3 = 1.0f / (sqrtf(2 * 3.14159265359f) * sigma * sigma * sigma);
    for (int it = 0; it < iters; it++) {
        g.sync();
        for (int c = g.rank(); c < W; c += g.size()) {
            const GaussAxisTerms t = gauss_axis_terms(c, px, k1);
            col[3 * c] = t.D;
            col[3 * c + 1] = t.g;
            col[3 * c + 2] = t.h;
        }
        for (int r = g.rank(); r < H; r += g.size()) {
            const GaussAxisTerms t = gauss_axis_terms(r, py, k1);
            row[3 * r] = t.D;
            row[3 * r + 1] = t.g;
            row[3 * r + 2] = t.h;
        }
        g.sync();
        double acc[8] = {0, 0, 0, 0, 0, 0, 0, 0};
        for (int i = g.rank(); i < W * H; i += g.size()) {
            const int y = i / W, x = i - y * W;
            const float DX = col[3 * x], gX = col[3 * x + 1], hX = col[3 * x + 2];
            const float DY = row[3 * y], gY = row[3 * y + 1], hY = row[3 * y + 2];
            const float mu = bg + I0 * DX * DY;
            const float dmu_dx = I0 * k2 * gX * DY;
            const float dmu_dy = I0 * k2 * gY * DX;
            const float dmu_dI0 = DX * DY;
            const float smp = img[i];
            const float f = smp / mu - 1;
            acc[0] += dmu_dx * f;
            acc[1] += dmu_dy * f;
            acc[2] += dmu_dI0 * f;
            acc[3] += f;
            const float d2mu_dx = I0 * k3 * hX * DY;
            const float d2mu_dy = I0 * k3 * hY * DX;
            const float mu2 = mu * mu;
            acc[4] += d2mu_dx * f - dmu_dx * dmu_dx * smp / mu2;
            acc[5] += d2mu_dy * f - dmu_dy * dmu_dy * smp / mu2;
            acc[6] += -dmu_dI0 * dmu_dI0 * smp / mu2;
            acc[7] += -smp / mu2;
        }
        g.sum(acc);
        px = (float)((double)px - acc[0] / acc[4]);
        py = (float)((double)py - acc[1] / acc[5]);
        I0 = (float)((double)I0 - acc[2] / acc[6]);
        bg = (float)((double)bg - acc[3] / acc[7]);
    }
}

// Solve the symmetric 5x5 system A d = b (Gaussian elimination, partial pivoting, FP64).
// Gaussian elimination with partial pivoting. The pivot row is found by swapping, row by row, any
// row whose entry is larger in magnitude into the pivot position: every index is a compile-time
// constant after unrolling, so the matrix stays in registers (a dynamically indexed row swap
// would put it in local memory). The pivot chosen and every operation on a row are those of
// the classic search-then-swap form.
__device__ __forceinline__ bool solve5(double (&A)[5][5], double (&b)[5], double (&d)[5])
{
#pragma unroll
    for (int c = 0; c < 5; c++) {
#pragma unroll
        for (int r = c + 1; r < 5; r++) {
            const bool sw = fabs(A[r][c]) > fabs(A[c][c]);
#pragma unroll
            for (int j = 0; j < 5; j++) {
                const double t = A[c][j];
                A[c][j] = sw ? A[r][j] : t;
                A[r][j] = sw ? t : A[r][j];
            }
            const double t = b[c];
            b[c] = sw ? b[r] : t;
            b[r] = sw ? t : b[r];
        }
        if (!(fabs(A[c][c]) > 1e-300)) return false;
#pragma unroll
        for (int r = c + 1; r < 5; r++) {
            const double f = A[r][c] / A[c][c];
#pragma unroll
            for (int j = c; j < 5; j++) A[r][j] -= f * A[c][j];
            b[r] -= f * b[c];
        }
    }
#pragma unroll
    for (int i = 4; i >= 0; i--) {
        double s = b[i];
#pragma unroll
        for (int j = i + 1; j < 5; j++) s -= A[i][j] * d[j];
        d[i] = s / A[i][i];
    }
    return true;
}

// Extension (no reference counterpart): 5-parameter (x, y, I0, bg, sigma) Poisson MLE of an
// integrated Gaussian spot, full Newton (Fisher-scoring) steps. Likelihood terms and
// gradients in FP32 per pixel, FP64 reduction and an FP64 5x5 solve per step. p[] = {x, y,
// I0, bg, sigma}; col/row: 5*W and 5*H floats of shared scratch.
template <class G>
__device__ inline void gauss5_mle(const G &g, const float *img, int W, int H, float (&p)[5], int iters, float *col,
                           float *row)
{
    for (int it = 0; it < iters; it++) {
        const float s = p[4];
        const float k1 = 1.0f / (sqrtf(2.0f) * s);
        const float k2 = 1.0f / (sqrtf(2 * 3.14159265359f) * s);
        g.sync();
        for (int c = g.rank(); c < W + H; c += g.size()) {
            const bool is_col = c < W;
            const int cc = is_col ? c : c - W;
            const float pc = is_col ? p[0] : p[1];
            const float a0 = (cc - pc + .5f) * k1, a1 = (cc - pc - .5f) * k1;
            const float e0 = expf(-a0 * a0), e1 = expf(-a1 * a1);
            float *t = is_col ? col + 3 * cc : row + 3 * cc;
            t[0] = 0.5f * (erff(a0) - erff(a1));
            t[1] = (e1 - e0) * k2;                                                  // dD/dp
            t[2] = ((cc - pc - .5f) * e1 - (cc - pc + .5f) * e0) * k2 / s;          // dD/dsigma
        }
        g.sync();
        float a[20];
#pragma unroll
        for (int k = 0; k < 20; k++) a[k] = 0.0f;
        for (int i = g.rank(); i < W * H; i += g.size()) {
            const int y = i / W, x = i - y * W;
            const float DX = col[3 * x], dX = col[3 * x + 1], sX = col[3 * x + 2];
            const float DY = row[3 * y], dY = row[3 * y + 1], sY = row[3 * y + 2];
            const float mu = p[3] + p[2] * DX * DY;
            const float J[5] = {p[2] * dX * DY, p[2] * DX * dY, DX * DY, 1.0f, p[2] * (sX * DY + DX * sY)};
            const float f = img[i] / mu - 1.0f;
            const float imu = 1.0f / mu;
            int k = 5;
#pragma unroll
            for (int u = 0; u < 5; u++) {
                a[u] += J[u] * f;
#pragma unroll
                for (int v = u; v < 5; v++) a[k++] += J[u] * J[v] * imu;
            }
        }
        double acc[20];
#pragma unroll
        for (int k = 0; k < 20; k++) acc[k] = a[k];
        g.sum(acc);
        double A[5][5], b[5], d[5];
        int k = 5;
#pragma unroll
        for (int u = 0; u < 5; u++) {
            b[u] = acc[u];
#pragma unroll
            for (int v = u; v < 5; v++) A[u][v] = A[v][u] = acc[k++];
        }
        if (!solve5(A, b, d)) break;
#pragma unroll
        for (int u = 0; u < 5; u++) p[u] = (float)((double)p[u] + d[u]);
        p[2] = fmaxf(p[2], 1e-3f);
        p[3] = fmaxf(p[3], 1e-3f);
        p[4] = fminf(fmaxf(p[4], 0.3f), 0.5f * (float)W);
    }
}

}  // namespace qtrk

// Localization kernels for sm_100a.
//
// localize_qi_kernel: one CTA per ROI runs the whole per-ROI pipeline of
//   QueuedCPUTracker::ProcessJob (cputrack/QueuedCPUTracker.cpp:273-361) on a tile of the ROI in
//   shared memory (tile.cuh): bulk copy (or batched loads) + convert (+ calibration) fused with the
//   pixel sum -> COM -> QI iterations -> radial profile -> Z-LUT match -> result. Pixels are
//   read from HBM exactly once; everything after the load works on-chip.
// localize_gauss_kernel: one CTA per ROI, COM -> 2D Gaussian MLE (-> Z) on a plain tile.
// build_lut_kernel / finalize_lut_kernel: QueuedCPUTracker::BuildLUT / FinalizeLUT
//   (cputrack/QueuedCPUTracker.cpp:580-659) with the accumulation on the device.
// profile_kernel: ComputeRadialProfile (cputrack/utils.cpp:275-320) for one image.
#include <algorithm>
#include <cstdint>
#include <cstdio>
#include <cuda_runtime.h>

#include <cuda_bf16.h>

#include "kernels.h"
#include "tile.cuh"

namespace qtrk {

// QI / Z-LUT least-squares weights, cputrack/QueuedTracker.h:349,359
__device__ const float kQIWeights[7] = {0.14f, 0.5f, 0.85f, 1.0f, 0.85f, 0.5f, 0.14f};
__device__ const float kZLUTWeights[7] = {0.15f, 0.5f, 0.85f, 1.0f, 0.85f, 0.5f, 0.15f};

struct SmemView {
    uint32_t *img;  // the tile (tile.cuh)
    float *misc;
    float4 *qdirs;  // QI quadrant directions as (d.x, d.x, d.y, d.y)
    float2 *tw;
    float4 *zdirs;  // full-circle directions in pairs (j, j + n/2), see load_z_tables
    float *qrw;  // QI radial weights (qi_nr floats after the twiddles)
    uint8_t *work;
    double *red;
    __device__ __forceinline__ uint64_t *mbar() const  // of the ROI's copy; copy_late's word behind it
    {
        return reinterpret_cast<uint64_t *>(reinterpret_cast<uint8_t *>(misc) + 32);
    }
};

__device__ __forceinline__ SmemView smem_view(uint8_t *smem, const TrackParams &P)
{
    SmemView v;
    v.img = reinterpret_cast<uint32_t *>(smem + P.sm_img);
    v.misc = reinterpret_cast<float *>(smem + P.sm_misc);
    v.red = reinterpret_cast<double *>(smem + P.sm_red);
    v.work = smem + P.sm_work;
    float2 *tab = reinterpret_cast<float2 *>(smem + P.sm_tables);
    v.qdirs = reinterpret_cast<float4 *>(tab);
    v.tw = tab + 2 * P.qi_angpq;  // L/2 = qi_nr twiddles
    v.qrw = reinterpret_cast<float *>(v.tw + P.qi_nr);
    v.zdirs = reinterpret_cast<float4 *>(smem + P.sm_zdirs);
    return v;
}

// Copy the QI direction / twiddle tables into shared memory (all threads; a barrier must
// follow before use).
__device__ __forceinline__ void load_qi_tables(const SmemView &s, const TrackParams &P)
{
    const float2 *qd = static_cast<const float2 *>(P.qi_dirs);
    const float2 *tw = static_cast<const float2 *>(P.qi_twiddles);
    if (qd)
        for (int i = threadIdx.x; i < P.qi_angpq; i += blockDim.x) {
            const float2 d = qd[i];
            s.qdirs[i] = make_float4(d.x, d.x, d.y, d.y);
        }
    if (tw)
        for (int i = threadIdx.x; i < P.qi_nr; i += blockDim.x) s.tw[i] = tw[i];
    if (P.qi_rweights)
        for (int i = threadIdx.x; i < P.qi_nr; i += blockDim.x) s.qrw[i] = P.qi_rweights[i];
}

// Copy the full-circle direction table (all threads; a barrier must follow before use). Where shared memory
// is short (sm_zdirs == sm_tables) it goes over the QI tables, and the QI stage must be finished.
__device__ __forceinline__ void load_z_tables(const SmemView &s, const TrackParams &P)
{
    const float2 *zd = static_cast<const float2 *>(P.z_dirs);
    if (zd)
        for (int j = threadIdx.x; j < (P.z_angsteps + 1) >> 1; j += blockDim.x) {
            // entry j = (d_j.x, d_{j+h}.x, d_j.y, d_{j+h}.y), h = n/2 rounded down; with n odd the
            // last entry holds d_{n-1} alone (zeros in the second place, never read)
            const int h = P.z_angsteps >> 1;
            const float2 a = zd[j < h ? j : P.z_angsteps - 1];
            const float2 b = j < h ? zd[j + h] : make_float2(0.0f, 0.0f);
            s.zdirs[j] = make_float4(a.x, b.x, a.y, b.y);
        }
}

// The QI position update from the two autoconvolutions (cpu_tracker.cpp:345-357, 400-410):
// ComputeMaxInterp over autoconv[x] = ac[(x + nr) mod L] for X (.x) and Y (.y), by one warp, given the
// first indices ix, iy of the maxima: the 7-point fits of both axes side by side (even lanes X, odd
// lanes Y). Lanes 0 and 1 write the new x and y to misc[0] and misc[1].
__device__ __noinline__ void qi_fit_at(const float2 *ac, int nr, int ix, int iy, float cx, float cy, float rstep,
                                       float *misc)
{
    __builtin_assume(__isShared(ac));
    __builtin_assume(__isShared(misc));
    const int lane = threadIdx.x & 31, L = 2 * nr;
    const bool yaxis = (lane & 1) != 0;
    float m;
    if (ix >= 3 && ix + 4 <= L && iy >= 3 && iy + 4 <= L) {  // both windows inside: per-lane fits
        auto at = [&](int x) {
            int n = x + nr;
            if (n >= L) n -= L;
            return yaxis ? ac[n].y : ac[n].x;
        };
        m = max_interp7_sym(at, L, yaxis ? iy : ix, kQIWeights);
    } else {  // a clipped window takes the warp-wide fit, one axis after the other
        auto atx = [&](int x) {
            int n = x + nr;
            if (n >= L) n -= L;
            return ac[n].x;
        };
        auto aty = [&](int x) {
            int n = x + nr;
            if (n >= L) n -= L;
            return ac[n].y;
        };
        const float mx = max_interp7_sym(atx, L, ix, kQIWeights);
        const float my = max_interp7_sym(aty, L, iy, kQIWeights);
        m = yaxis ? my : mx;
    }
    if (lane < 2) {
        const float off = (m - (float)nr) * (3.14159265359f / 4);
        misc[lane] = (yaxis ? cy : cx) + off * rstep;
    }
}

// Transform, argmax and fit with the autoconvolutions in registers (L = 32 E): the maximum of each axis by
// one integer warp reduction over order_key, its first index by another (as the strict ">" scan of
// LsqQuadraticFit.h:140-147 finds it; NaN never wins). The result replaces the profile in A, for the fit's
// windows (every lane has read its elements before the first shuffle).
template <int E>
__device__ __noinline__ void qi_update_regs(float2 *A, const float2 *tw, float cx, float cy, float rstep, float *misc)
{
    __builtin_assume(__isShared(A));  // not inlined: its pointers' address space is not seen otherwise
    __builtin_assume(__isShared(tw));
    constexpr int L = 32 * E, nr = L / 2;
    const int lane = threadIdx.x & 31;
    float2 z[E];
    qi_autoconv_regs<E>(A, tw, z);
    int kx = (int)0x80000000, ky = kx;
#pragma unroll
    for (int e = 0; e < E; e++) {
        A[lane + 32 * e] = z[e];
        kx = max(kx, order_key(z[e].x));
        ky = max(ky, order_key(z[e].y));
    }
    kx = __reduce_max_sync(0xffffffffu, kx);
    ky = __reduce_max_sync(0xffffffffu, ky);
    int ix = L, iy = L;
#pragma unroll
    for (int e = 0; e < E; e++) {
        const int x = (lane + 32 * e + nr) & (L - 1);
        if (order_key(z[e].x) == kx) ix = min(ix, x);
        if (order_key(z[e].y) == ky) iy = min(iy, x);
    }
    ix = __reduce_min_sync(0xffffffffu, ix);
    iy = __reduce_min_sync(0xffffffffu, iy);
    __syncwarp();
    qi_fit_at(A, nr, ix, iy, cx, cy, rstep, misc);
}

// The same for the other lengths (2 nr < 32 or > 512), through shared memory; A in bit-reversed order.
__device__ __noinline__ void qi_update_smem(float2 *A, float2 *ac, int nr, const float2 *tw, float cx, float cy,
                                            float rstep, float *misc)
{
    const int L = 2 * nr;
    qi_autoconv_fft_filled(nr, A, ac, tw);
    auto at = [&](int x, bool yaxis) {
        int n = x + nr;
        if (n >= L) n -= L;
        return yaxis ? ac[n].y : ac[n].x;
    };
    const int ix = warp_argmax([&](int x) { return at(x, false); }, L);
    const int iy = warp_argmax([&](int x) { return at(x, true); }, L);
    qi_fit_at(ac, nr, ix, iy, cx, cy, rstep, misc);
}

// CPUTracker::ComputeQI, cpu_tracker.cpp:285-360. All threads call; returns the position and the
// boundary flag of the last iteration.
template <int F, int T>
__device__ __forceinline__ void qi_localize(const SmemView &s, const TrackParams &P, float mean, float &cx, float &cy,
                                            bool &bhit, const float *rweights)
{
    const int W = P.width, H = P.height, nr = P.qi_nr, L = 2 * nr;
    const bool regs = L >= 32 && L <= 512;  // L is a power of two
    // work: [ A (L complex) ] [ ac (L complex), only for the transform through shared memory ]
    float2 *A = reinterpret_cast<float2 *>(s.work);
    const float rstep = (P.qi_maxr - P.qi_minr) / (float)nr;  // also pixelsPerProfLen (cpu_tracker.cpp:311,649)
#pragma unroll 1
    for (int k = 0; k < P.qi_iterations; k++) {
        bhit = check_boundaries(cx, cy, P.qi_maxr, W, H);
        qi_profiles<F, T>(s.img, W, H, P.tile_pitch, cx, cy, mean, nr, P.qi_nang[k], P.qi_inv_nang[k], P.qi_stride[k],
                          P.qi_minr, rstep, s.qdirs, rweights, A, regs ? -1 : ilog2_pow2(L));
        __syncthreads();
        if (threadIdx.x < 32) {  // transform and fits on warp 0, the others wait at the next barrier
            __syncwarp();        // its shuffles run as one warp (a lane that diverged earlier may still be apart)
            switch (L) {
            case 32: qi_update_regs<1>(A, s.tw, cx, cy, rstep, s.misc); break;
            case 64: qi_update_regs<2>(A, s.tw, cx, cy, rstep, s.misc); break;
            case 128: qi_update_regs<4>(A, s.tw, cx, cy, rstep, s.misc); break;
            case 256: qi_update_regs<8>(A, s.tw, cx, cy, rstep, s.misc); break;
            case 512: qi_update_regs<16>(A, s.tw, cx, cy, rstep, s.misc); break;
            default: qi_update_smem(A, A + L, nr, s.tw, cx, cy, rstep, s.misc);
            }
        }
        __syncthreads();
        // misc[0..1] is written again only after the next iteration's first barrier, which every
        // thread reaches after these reads
        cx = s.misc[0];
        cy = s.misc[1];
    }
}

// Radial profile + Z-LUT compare (QueuedCPUTracker.cpp:319-338). Returns z (0 without a LUT). With
// P.zprof_f32 set, the profile is written out for the tensor-core match instead.
template <int F, int T>
__device__ __forceinline__ float z_localize(const SmemView &s, const TrackParams &P, int ts, float mean, float x, float y,
                                            int bead, int roi)
{
    const int nb = P.z_nbins;
    float *prof = reinterpret_cast<float *>(s.work);
    double *scores = reinterpret_cast<double *>(s.work + (((nb * 4) + 15) & ~15));
    const float rstep = (P.z_maxr - P.z_minr) / (float)nb;
    if (P.sm_zdirs == P.sm_tables) {
        load_z_tables(s, P);
        __syncthreads();
    }
    radial_profile<F, T>(s.img, P.width, P.height, ts, x, y, mean, nb, P.z_angsteps, P.z_minr, rstep, s.zdirs, prof,
                         (P.mode & kLT_NormalizeProfile) != 0);
    if (P.zprof_f32) {
        // [hi | lo] BF16 split of the weighted profile: v = hi + lo + O(2^-16 v). Of a ROI whose copy was late, not a
        // number
        const bool late = copy_late(s.mbar()) != 0u;
        __nv_bfloat16 *pb = static_cast<__nv_bfloat16 *>(P.zprof_bf16) + (size_t)roi * 2 * P.zprof_nbp;
        for (int r = threadIdx.x; r < P.zprof_nbp; r += blockDim.x) {
            float v = 0.0f;
            if (r < nb) {
                v = late ? __int_as_float(0x7fc00000) : prof[r];
                P.zprof_f32[(size_t)roi * nb + r] = v;
                if (P.z_weights) v *= P.z_weights[r];
            }
            const __nv_bfloat16 h = __float2bfloat16_rn(v);
            pb[r] = h;
            pb[P.zprof_nbp + r] = __float2bfloat16_rn(v - __bfloat162float(h));
        }
        return 0.0f;
    }
    if (!P.lut || bead < 0 || bead >= P.lut_count) return 0.0f;
    if (!P.lut_t) return __int_as_float(0x7fc00000);  // the host launched without refreshing the transposed LUT
    const float *lut_t = P.lut_t + (size_t)bead * nb * P.lut_t_pitch;
    zlut_scores_plain<T>(prof, lut_t, P.lut_t_pitch, P.lut_planes, nb, P.z_weights, scores);
    if (P.cmp_scores)
        for (int k = threadIdx.x; k < P.lut_planes; k += blockDim.x)
            P.cmp_scores[(size_t)bead * P.lut_planes + k] = (float)scores[k];
    if (threadIdx.x < 32) {
        __syncwarp();
        auto at = [&](int i) { return scores[i]; };
        const int im = warp_argmax_f64(at, P.lut_planes);
        const float z = max_interp7_sym(at, P.lut_planes, im, kZLUTWeights);
        if (threadIdx.x == 0) s.misc[2] = zlut_bias_correct(z, P.lut_planes, P.zbias, P.zbias_w, P.zbias_count, bead);
    }
    __syncthreads();
    return s.misc[2];
}

// CTAs per SM the 128-thread kernels are compiled for (72 registers): ROIs of up to about 80 px fit seven times,
// and a frame of 1,000 then runs in one wave (60x60 f32: 57 us, 70 us with five CTAs of 96 registers; 64x64 u16: 55
// and 64 us); larger ROIs, five to an SM by their tiles, lose 1 % by it.
constexpr int kMinBlocks = 7;

// Bring the ROI at `src` into the tile and measure mean and COM; the tables are fetched under the copy.
template <int F, int T>
__device__ __forceinline__ ComResult load_tile(const SmemView &s, const TrackParams &P, const uint8_t *src, int pitch,
                                               int bead, float bgcorr)
{
    const int W = P.width, H = P.height, ts = P.tile_pitch;
    auto tables = [&] {
        load_qi_tables(s, P);
        if (P.sm_zdirs != P.sm_tables) load_z_tables(s, P);
    };
    if (F == kTileF32 && packed_rows(W, ts)) {  // the largest odd ROIs: a tile without room for padded rows
        if (threadIdx.x == 0) copy_late(s.mbar()) = 0u;
        tables();
        const BlockGroup g{s.red};
        float *img = reinterpret_cast<float *>(s.img);
        return com_from_sums(g, img, W, H, load_roi(g, img, src, pitch, P, bead), bgcorr);
    }
    const uint8_t *raw = load_raw<F, T>(s.img, ts, P, src, pitch, s.mbar(), tables);
    uint32_t isum;
    const double sum = convert_raw<F, T>(s.img, raw, ts, P, bead, isum);
    return tile_com<F, T>(s.img, W, H, ts, sum, isum, bgcorr, s.red);
}

// COM / QI (+ Z): QueuedCPUTracker::ProcessJob (QueuedCPUTracker.cpp:273-361), one CTA of T threads per
// ROI on a tile of format F.
template <int F, int T>
__global__ void __launch_bounds__(T, T == 128 ? kMinBlocks : (T == 256 ? 2 : 1))
    localize_qi_kernel(TrackParams P, const uint8_t *__restrict__ pixels, int pitch, int64_t roi_stride,
                       const int64_t *__restrict__ roi_offsets, const LocalizationJob *__restrict__ jobs, int count,
                       LocalizationResult *__restrict__ results)
{
    extern __shared__ __align__(16) uint8_t smem[];
    const int roi = blockIdx.x;
    if (roi >= count) return;
    const SmemView s = smem_view(smem, P);
    const int W = P.width, H = P.height;
    // the job's words are read again for the result (no registers held through QI and Z)
    const int bead = jobs ? (int)reinterpret_cast<const uint32_t *>(jobs)[(size_t)roi * 6 + 2] : 0;
    const int64_t off = roi_offsets ? roi_offsets[roi] : (int64_t)roi * roi_stride;
    const ComResult com = load_tile<F, T>(s, P, pixels + off, pitch, bead, P.com_bgcorrection);
    float comx = com.x, comy = com.y;
    if (isnan(comx) || isnan(comy)) {  // QueuedCPUTracker.cpp:294-295
        comx = (float)(W / 2);
        comy = (float)(H / 2);
    }
    float x = comx, y = comy, z = 0.0f;
    bool bhit = false;
    if (P.mode & kLT_QI) qi_localize<F, T>(s, P, com.mean, x, y, bhit, P.qi_rweights ? s.qrw : nullptr);
    if (P.mode & kLT_LocalizeZ) {
        bhit = check_boundaries(x, y, P.z_maxr, W, H);
        z = z_localize<F, T>(s, P, P.tile_pitch, com.mean, x, y, bead, roi);
    }
    if (threadIdx.x == 0) {
        uint32_t job[6];
        read_job(jobs, roi, job);
        float mean = com.mean;
        if (copy_late(s.mbar())) {
            x = y = z = comx = comy = mean = __int_as_float(0x7fc00000);
            bhit = true;
        }
        write_result(results, roi, job, x, y, z, comx, comy, bhit ? 1u : 0u, mean);
    }
}

// 2D Gaussian MLE (+ Z) for ROIs above 32x32 or with the Z bit: one CTA per ROI on a plain tile.
// Kept apart from the QI kernel, whose registers are not the MLE's. kBlocks: CTAs per SM it is compiled for, see
// gauss_cta_kernel.
template <int kBlocks>
__global__ void __launch_bounds__(kBlockThreads, kBlocks)
    localize_gauss_kernel(TrackParams P, const uint8_t *__restrict__ pixels, int pitch, int64_t roi_stride,
                          const int64_t *__restrict__ roi_offsets, const LocalizationJob *__restrict__ jobs, int count,
                          LocalizationResult *__restrict__ results)
{
    extern __shared__ __align__(16) uint8_t smem[];
    const int roi = blockIdx.x;
    if (roi >= count) return;
    const SmemView s = smem_view(smem, P);
    uint32_t job[6];
    read_job(jobs, roi, job);
    const int bead = (int)job[2];
    const int64_t off = roi_offsets ? roi_offsets[roi] : (int64_t)roi * roi_stride;
    if (threadIdx.x == 0) copy_late(s.mbar()) = 0u;
    BlockGroup g{s.red};
    const int W = P.width, H = P.height;
    float *img = reinterpret_cast<float *>(s.img);
    const double2 part = load_roi(g, img, pixels + off, pitch, P, bead);
    const ComResult com = com_from_sums(g, img, W, H, part, P.com_bgcorrection);
    float comx = com.x, comy = com.y;
    if (isnan(comx) || isnan(comy)) {  // QueuedCPUTracker.cpp:294-295
        comx = (float)(W / 2);
        comy = (float)(H / 2);
    }
    float x = comx, y = comy, z = 0.0f;
    bool bhit = false;
    float *col = reinterpret_cast<float *>(s.work);
    if (P.mode & kLT_Gaussian5P) {
        float p[5] = {x, y, com.mean * 0.5f * (float)(W * H), com.mean * 0.5f, P.g_sigma};
        gauss5_mle(g, img, W, H, p, P.g_iterations, col, col + 3 * W);
        x = p[0];
        y = p[1];
        z = p[4];
    } else {
        gauss4_mle(g, img, W, H, com.mean, x, y, P.g_iterations, P.g_sigma, col, col + 3 * W);
    }
    __syncthreads();
    if (P.mode & kLT_LocalizeZ) {
        if (P.sm_zdirs != P.sm_tables) {
            load_z_tables(s, P);
            __syncthreads();
        }
        bhit = check_boundaries(x, y, P.z_maxr, W, H);
        z = z_localize<kTileF32, kBlockThreads>(s, P, W, com.mean, x, y, bead, roi);
    }
    if (threadIdx.x == 0) write_result(results, roi, job, x, y, z, comx, comy, bhit ? 1u : 0u, com.mean);
}

// One bead of QueuedCPUTracker::BuildLUT (QueuedCPUTracker.cpp:582-645): ROI i of the stack is
// at data + pitch*H*i. Position from known_pos, else COM (no background correction) + QI
// without radial weights (line 603). The profile's fallback value is the tracker's mean,
// which SetImage resets to 0 when known_pos skips the COM (cpu_tracker.h:135).
template <int F, int T>
__global__ void __launch_bounds__(T, T == 128 ? kMinBlocks : (T == 256 ? 2 : 1))
    build_lut_kernel(TrackParams P, const uint8_t *__restrict__ pixels, int pitch, int nbeads, int plane,
                     const float2 *__restrict__ known_pos, int normalize, float *__restrict__ lut)
{
    extern __shared__ __align__(16) uint8_t smem[];
    const int bead = blockIdx.x;
    if (bead >= nbeads) return;
    const SmemView s = smem_view(smem, P);
    const ComResult com = load_tile<F, T>(s, P, pixels + (size_t)pitch * P.height * bead, pitch, bead, 0.0f);
    float x, y, mean = 0.0f;
    if (known_pos) {
        x = known_pos[bead].x;
        y = known_pos[bead].y;
    } else {
        mean = com.mean;
        x = com.x;
        y = com.y;
        bool bhit;
        qi_localize<F, T>(s, P, mean, x, y, bhit, nullptr);
    }
    const int nb = P.z_nbins;
    float *prof = reinterpret_cast<float *>(s.work);
    const float rstep = (P.z_maxr - P.z_minr) / (float)nb;
    __syncthreads();
    if (P.sm_zdirs == P.sm_tables) {
        load_z_tables(s, P);
        __syncthreads();
    }
    radial_profile<F, T>(s.img, P.width, P.height, P.tile_pitch, x, y, mean, nb, P.z_angsteps, P.z_minr, rstep, s.zdirs,
                         prof, normalize != 0);
    float *dst = lut + ((size_t)bead * P.lut_planes + plane) * nb;
    const bool late = copy_late(s.mbar()) != 0u;  // not a number: a row that no match takes
    for (int r = threadIdx.x; r < nb; r += T) dst[r] = late ? __int_as_float(0x7fc00000) : dst[r] + prof[r];
}

// QueuedCPUTracker::FinalizeLUT (QueuedCPUTracker.cpp:648-659): NormalizeRadialProfile
// (utils.cpp:230-261) on every (bead, plane) row. One warp per row.
__global__ void finalize_lut_kernel(float *__restrict__ lut, int rows, int nb)
{
    const int row = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (row >= rows) return;
    const int lane = threadIdx.x & 31;
    float *p = lut + (size_t)row * nb;
    double s = 0;
    for (int i = lane; i < nb; i += 32) s += p[i];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    const float m = (float)(s / nb);
    double s2 = 0;
    for (int i = lane; i < nb; i += 32) {
        const float v = p[i] - m;
        p[i] = v;
        s2 += (double)(v * v);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s2 += __shfl_xor_sync(0xffffffffu, s2, o);
    const double inv = 1.0 / sqrt(s2 / nb);
    for (int i = lane; i < nb; i += 32) p[i] = (float)((double)p[i] * inv);
}

// ComputeRadialProfile (utils.cpp:275-320) of one float image with a given fallback mean.
__global__ void __launch_bounds__(kBlockThreads) profile_kernel(TrackParams P, const float *__restrict__ img_in,
                                                                float cx, float cy, float mean, int normalize,
                                                                float *__restrict__ out)
{
    extern __shared__ __align__(16) uint8_t smem[];
    const SmemView s = smem_view(smem, P);
    load_z_tables(s, P);
    BlockGroup g{s.red};
    load_roi(g, reinterpret_cast<float *>(s.img), reinterpret_cast<const uint8_t *>(img_in), P.width * 4, P, -1);
    float *prof = reinterpret_cast<float *>(s.work);
    const float rstep = (P.z_maxr - P.z_minr) / (float)P.z_nbins;
    radial_profile<kTileF32, kBlockThreads>(s.img, P.width, P.height, P.width, cx, cy, mean, P.z_nbins, P.z_angsteps,
                                            P.z_minr, rstep, s.zdirs, prof, normalize != 0);
    for (int r = threadIdx.x; r < P.z_nbins; r += blockDim.x) out[r] = prof[r];
}

// ------------------------------------------------------------------------------------------
// host-side launchers
// ------------------------------------------------------------------------------------------
static int align16(int v) { return (v + 15) & ~15; }

constexpr int kMaxSmem = 227 * 1024;

// The layout of a localization CTA's shared memory. Where the padded rows and the separate direction tables do
// not fit, rows are packed and the full-circle table goes over the QI tables.
static void plan_smem_form(TrackParams &P, bool compact)
{
    const int W = P.width, H = P.height;
    const int nr = P.qi_nr > 0 ? P.qi_nr : 1, L = 2 * nr;
    P.sm_img = 0;
    P.tile_pitch = compact ? W : tile_pitch(W);
    // The CTA of the Gaussian modes loads row by row, so its compact form needs no room behind the tile for a raw ROI.
    const bool gauss = (P.mode & kLT_Gaussian2D) && !(P.mode & kLT_QI);
    P.sm_tables = compact && gauss ? align16(W * H * 4) : tile_region_bytes(W, H, P.tile_pitch);
    const int qi_tables = align16(P.qi_angpq * 16 + nr * 8 + nr * 4), z_tables = ((P.z_angsteps + 1) >> 1) * 16;
    P.sm_zdirs = compact ? P.sm_tables : P.sm_tables + qi_tables;
    P.sm_work = compact ? P.sm_tables + std::max(qi_tables, z_tables) : P.sm_zdirs + z_tables;
    // QI: the profile (L complex), and its transform where that runs through shared memory
    const int qi_work = (L >= 32 && L <= 512 ? 1 : 2) * L * 8;
    const int z_work = align16(P.z_nbins * 4) + P.lut_planes * 8;
    const int g_work = gauss ? (3 * W + 3 * H) * 4 : 0;
    P.sm_red = P.sm_work + align16(std::max(qi_work, std::max(z_work, g_work)));
    // block sum scratch, N * warps doubles: N <= 20 with 4 warps (Gaussian), 3 with up to 16
    P.sm_misc = P.sm_red + (gauss ? 80 : 48) * 8;
    P.smem_bytes = P.sm_misc + 64;
}

void plan_smem(TrackParams &P)
{
    plan_smem_form(P, false);
    if (P.smem_bytes > kMaxSmem) plan_smem_form(P, true);
}

// The kernel instantiations by tile format and threads per ROI.
using QiKernel = void (*)(TrackParams, const uint8_t *, int, int64_t, const int64_t *, const LocalizationJob *, int,
                          LocalizationResult *);
using LutKernel = void (*)(TrackParams, const uint8_t *, int, int, int, const float2 *, int, float *);
static const QiKernel kQiKernels[3][3] = {
    {localize_qi_kernel<kTileF32, 128>, localize_qi_kernel<kTileF32, 256>, localize_qi_kernel<kTileF32, 512>},
    {localize_qi_kernel<kTileU16, 128>, localize_qi_kernel<kTileU16, 256>, localize_qi_kernel<kTileU16, 512>},
    {localize_qi_kernel<kTileU8, 128>, localize_qi_kernel<kTileU8, 256>, localize_qi_kernel<kTileU8, 512>}};
static const LutKernel kLutKernels[3][3] = {
    {build_lut_kernel<kTileF32, 128>, build_lut_kernel<kTileF32, 256>, build_lut_kernel<kTileF32, 512>},
    {build_lut_kernel<kTileU16, 128>, build_lut_kernel<kTileU16, 256>, build_lut_kernel<kTileU16, 512>},
    {build_lut_kernel<kTileU8, 128>, build_lut_kernel<kTileU8, 256>, build_lut_kernel<kTileU8, 512>}};

// log2(threads / 128) per ROI: CTAs of 128 threads when several ROIs share an SM anyway, wider ones when the ROIs
// do not fill the GPU and a ROI's latency decides (8 lanes per QI radius at most, so 8 nr threads). 50 ROIs of
// 128x128 u8: 36 us with 512 threads each, 76 us with 128 and the tile as floats. 256 threads for every count cost
// 4-8 % where several ROIs share an SM (1,000 x 64x64, 10,000 x 100x100).
static int wide_cta(const TrackParams &P, int count)
{
    if (packed_rows(P.width, P.tile_pitch)) return 0;  // its COM's order depends on the thread count
    // ROIs that share an SM: by their number, or as many as its shared memory holds
    const int per_sm = std::min((count + 147) / 148, (228 * 1024) / (P.smem_bytes + 1024));
    if (per_sm <= 1 && P.qi_nr >= 64) return 2;
    if (per_sm <= 2 && P.qi_nr >= 32) return 1;
    return 0;
}

// The Gaussian kernel by the CTAs per SM that it is compiled for: seven (72 registers, some spills), except for the 20
// FP32 sums of the 5-parameter form where an SM's shared memory holds no more than five CTAs anyway (96 registers). f32,
// compiled for seven and five: 4 parameters, 4,000 x 40x40 408 and 466 us, 2,000 x 64x64 426 and 472, 100x100 970 and
// 964; 5 parameters, 40x40 426 and 459, 2,000 x 88x88 (six fit) 544 and 551, 92x92 (five fit) 569 and 554, 100x100 721
// and 704, 150x150 1839 and 1768.
static QiKernel gauss_cta_kernel(const TrackParams &P)
{
    const bool five = (P.mode & kLT_Gaussian5P) && (228 * 1024) / (P.smem_bytes + 1024) <= 5;
    return five ? localize_gauss_kernel<5> : localize_gauss_kernel<7>;
}

static bool g_attrs_set[64];

cudaError_t prepare_kernels(int device)
{
    if (device < 0 || device >= 64) return cudaErrorInvalidDevice;
    if (g_attrs_set[device]) return cudaSuccess;
    cudaError_t e;
    for (int f = 0; f < 3; f++)
        for (int t = 0; t < 3; t++) {
            if ((e = cudaFuncSetAttribute(reinterpret_cast<const void *>(kQiKernels[f][t]),
                                          cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxSmem)))
                return e;
            if ((e = cudaFuncSetAttribute(reinterpret_cast<const void *>(kLutKernels[f][t]),
                                          cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxSmem)))
                return e;
        }
    for (QiKernel k : {localize_gauss_kernel<5>, localize_gauss_kernel<7>})
        if ((e = cudaFuncSetAttribute(reinterpret_cast<const void *>(k), cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      kMaxSmem)))
            return e;
    if ((e = cudaFuncSetAttribute(profile_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxSmem))) return e;
    if ((e = prepare_gauss_kernels())) return e;
    g_attrs_set[device] = true;
    return cudaSuccess;
}

cudaError_t launch_localize(const TrackParams &P, const uint8_t *pixels, int pitch, int64_t roi_stride,
                            const int64_t *roi_offsets, const LocalizationJob *jobs, int count,
                            LocalizationResult *results, cudaStream_t stream)
{
    if (count <= 0) return cudaSuccess;
    if (use_com_kernel(P, pixels, pitch, roi_stride, roi_offsets))
        return launch_com(P, pixels, roi_stride, jobs, count, results, stream);
    if (use_gauss_warp(P))
        return launch_gauss_warp(P, pixels, pitch, roi_stride, roi_offsets, jobs, count, results, stream);
    if ((P.mode & kLT_Gaussian2D) && !(P.mode & kLT_QI)) {
        gauss_cta_kernel(P)<<<count, kBlockThreads, P.smem_bytes, stream>>>(P, pixels, pitch, roi_stride, roi_offsets,
                                                                           jobs, count, results);
    } else {
        const int wide = wide_cta(P, count);
        kQiKernels[tile_format(P, P.tile_pitch)][wide]<<<count, kBlockThreads << wide, P.smem_bytes, stream>>>(
            P, pixels, pitch, roi_stride, roi_offsets, jobs, count, results);
    }
    return cudaGetLastError();
}

// Bias-table images (QueuedTracker::ComputeZBiasCorrection, cputrack/QueuedTracker.cpp:143-189):
// image i = bead (i / bias_planes) at the ROI centre (w/2, h/2, int division) and
// z = (i % bias_planes) / bias_planes * planes, rendered as GenerateImageFromLUT
// (cputrack/utils.cpp:325-390) does: the bead's LUT interpolated over planes (uniform cubic
// B-spline over 4 planes, or linear), then ovs x ovs samples per pixel, each a linear
// interpolation of that profile at (|offset| - minradius) * bins / (maxradius - minradius),
// clamped to [0, bins - 2]. One block per image; block b renders image first + b into slot b
// of `images` and `jobs` (job: frame = image index, zlutIndex = bead).
__global__ void __launch_bounds__(256) lut_image_kernel(const float *__restrict__ lut, int nb, int planes, int first,
                                                        int bias_planes, int w, int h, float minr, float maxr,
                                                        int ovs, int spline, float *__restrict__ images,
                                                        LocalizationJob *__restrict__ jobs)
{
    extern __shared__ float zi[];  // [nb]
    const int img = first + blockIdx.x;
    const int bead = img / bias_planes, plane = img - bead * bias_planes;
    const float z = plane / (float)bias_planes * planes;
    const float *L = lut + (size_t)bead * planes * nb;
    for (int r = threadIdx.x; r < nb; r += blockDim.x) {
        float v;
        if (spline) {
            const int iz = max(1, min(planes - 3, (int)z));
            const float t = z - iz, t2 = t * t, t3 = t2 * t;
            const float wt[4] = {(1 - 3 * t + 3 * t2 - t3) / 6, (4 - 6 * t2 + 3 * t3) / 6,
                                 (1 + 3 * t + 3 * t2 - 3 * t3) / 6, t3 / 6};
            v = 0.0f;
            for (int i = 0; i < 4; i++) v += wt[i] * L[(i - 1 + iz) * nb + r];
        } else {
            const int iz = (int)z;
            if (iz >= planes - 1) {
                v = L[(planes - 1) * nb + r];
            } else {
                const float a = L[iz * nb + r], b = L[(iz + 1) * nb + r];
                v = a + (b - a) * (z - iz);
            }
        }
        zi[r] = v;
    }
    if (threadIdx.x == 0) {
        LocalizationJob j{};
        j.frame = (uint32_t)img;
        j.zlutIndex = bead;
        jobs[blockIdx.x] = j;
    }
    __syncthreads();
    const float cx = (float)(w / 2), cy = (float)(h / 2);
    const float radialcov = nb / (maxr - minr), step = 1.0f / ovs;
    for (int p = threadIdx.x; p < w * h; p += blockDim.x) {
        const int y = p / w, x = p - y * w;
        float s = 0.0f;
        for (int ox = 0; ox < ovs; ox++)
            for (int oy = 0; oy < ovs; oy++) {
                const float X = x + (ox + 0.5f) * step - cx - 0.5f;
                const float Y = y + (oy + 0.5f) * step - cy - 0.5f;
                float r = (sqrtf(X * X + Y * Y) - minr) * radialcov;
                if (r > nb - 2) r = (float)(nb - 2);
                if (r < 0) r = 0;
                const int i = (int)r;
                s += zi[i] + (zi[i + 1] - zi[i]) * (r - i);
            }
        images[(size_t)blockIdx.x * w * h + p] = s / (ovs * ovs);
    }
}

cudaError_t launch_lut_images(const float *lut, int nb, int planes, int first_image, int n_images, int bias_planes,
                              int w, int h, float minr, float maxr, int ovs, bool spline, float *images,
                              LocalizationJob *jobs, cudaStream_t stream)
{
    if (n_images <= 0) return cudaSuccess;
    lut_image_kernel<<<n_images, 256, sizeof(float) * nb, stream>>>(lut, nb, planes, first_image, bias_planes, w, h,
                                                                    minr, maxr, ovs, spline ? 1 : 0, images, jobs);
    return cudaGetLastError();
}

void localize_node(const TrackParams &P, int count, cudaKernelNodeParams &kp)
{
    kp = cudaKernelNodeParams{};
    if (use_gauss_warp(P)) {
        gauss_warp_node(P, count, kp);
    } else {
        const bool gauss = (P.mode & kLT_Gaussian2D) && !(P.mode & kLT_QI);
        const int wide = gauss ? 0 : wide_cta(P, count);
        kp.func = gauss ? reinterpret_cast<void *>(gauss_cta_kernel(P))
                        : reinterpret_cast<void *>(kQiKernels[tile_format(P, P.tile_pitch)][wide]);
        kp.gridDim = dim3(count);
        kp.blockDim = dim3(kBlockThreads << wide);
        kp.sharedMemBytes = P.smem_bytes;
    }
}

cudaError_t launch_build_lut(const TrackParams &P, const uint8_t *pixels, int pitch, int nbeads, int plane,
                             const float2 *known_pos, bool normalize, float *lut, cudaStream_t stream)
{
    if (nbeads <= 0) return cudaSuccess;
    TrackParams Q = P;  // the layout of a ROI that arrives raw, whatever the instance's mode
    Q.mode &= ~kLT_Gaussian2D;
    plan_smem(Q);
    const int wide = wide_cta(Q, nbeads);
    kLutKernels[tile_format(Q, Q.tile_pitch)][wide]<<<nbeads, kBlockThreads << wide, Q.smem_bytes, stream>>>(
        Q, pixels, pitch, nbeads, plane, known_pos, normalize ? 1 : 0, lut);
    return cudaGetLastError();
}

cudaError_t launch_finalize_lut(float *lut, int rows, int nb, cudaStream_t stream)
{
    if (rows <= 0) return cudaSuccess;
    finalize_lut_kernel<<<(rows + 7) / 8, 256, 0, stream>>>(lut, rows, nb);
    return cudaGetLastError();
}

// lut [count][planes][nb] -> lut_t [count][nb][pitch], planes pitch..planes-1 of each bin zero.
// Reads are strided, writes coalesced; it runs once per LUT change.
__global__ void transpose_lut_kernel(const float *__restrict__ lut, int count, int planes, int nb, int pitch,
                                     float *__restrict__ lut_t)
{
    const size_t total = (size_t)count * nb * pitch;
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < total; i += (size_t)gridDim.x * blockDim.x) {
        const int k = (int)(i % pitch);
        const size_t br = i / pitch;
        const int r = (int)(br % nb);
        const size_t b = br / nb;
        lut_t[i] = k < planes ? lut[(b * planes + k) * nb + r] : 0.0f;
    }
}

cudaError_t launch_transpose_lut(const float *lut, int count, int planes, int nb, int pitch, float *lut_t,
                                 cudaStream_t stream)
{
    const size_t total = (size_t)count * nb * pitch;
    if (total == 0) return cudaSuccess;
    const int blocks = (int)std::min<size_t>((total + 255) / 256, 148 * 16);
    transpose_lut_kernel<<<blocks, 256, 0, stream>>>(lut, count, planes, nb, pitch, lut_t);
    return cudaGetLastError();
}

cudaError_t launch_profile(const TrackParams &P, const float *img, float cx, float cy, float mean, bool normalize,
                           float *out, cudaStream_t stream)
{
    profile_kernel<<<1, kBlockThreads, P.smem_bytes, stream>>>(P, img, cx, cy, mean, normalize ? 1 : 0, out);
    return cudaGetLastError();
}

}  // namespace qtrk

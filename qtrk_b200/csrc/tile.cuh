// The ROI tile of the localization kernels: one ROI in shared memory, loaded, measured (mean, COM) and
// sampled (QI quadrant profiles, radial profile) by a CTA of T threads (sm_100a).
//
// A tile element is one 32-bit word per pixel, in one of three formats:
//   kTileF32  the pixel as a float (float ROIs, and any ROI with per-bead calibration images);
//   kTileU16  the pixel in the low half, its right neighbour in the high half (u16 ROIs);
//   kTileU8   the pixel, its right, lower and lower right neighbours in the four bytes (u8 ROIs).
// A bilinear sample needs the 2x2 pixels of its cell: four 32-bit shared loads of floats, two of pairs, one
// of quads. As floats, 10,000 ROIs of 100x100 u16 kept the shared-memory pipe at 72 % (21.2 k wavefronts per ROI) and
// issue at 50 %; as pairs they need 12.4 k, and what bounds the kernel is instruction issue (61 % used, 59 k
// warp instructions per ROI, a third of them the byte permutes and adds that turn packed pixels into floats)
// with 20 warps per SM and one-warp sections (QI transform and fit) in between. Measured together with the
// transform in registers, the LUT runs and the wider CTAs for few ROIs: 10,000 x 100x100 u16 1.002 -> 0.832 ms,
// 1,000 x 64x64 u16 with own LUTs 127 -> 55 us, 50 x 128x128 u8 78 -> 35 us.
// All formats give bit-identical results for the same pixels: every later operation sees the same floats.
//
// Results also do not depend on T (the launcher picks T by the number of ROIs): whatever is summed in FP32 is
// cut into pieces that are the same for every T (the eight direction subsets of a circle, the 512 pixel
// chains of the COM), and the pieces meet in the same order or in FP64. FP64 sums across threads are formed in an order
// that follows T. Those of the COM's moments are exact, and so the same, as long as no pixel is negative: their
// terms are then multiples of 2^-25 of the mean, and a sum stays below 2^53 of that unit. Moments with negative
// pixels, and a float ROI's mean, agree to FP64 rounding (1e-16), far below that of the FP32 result.
#pragma once
#include "bulk_copy.cuh"
#include "device_common.cuh"

namespace qtrk {

enum : int { kTileF32 = 0, kTileU16 = 1, kTileU8 = 2 };

// Row pitch of the tile in words, whole 16-byte units. A warp's samples lie on a few neighbouring rows, so two
// rows must not start near the same bank: pitches of 4, 8 or 12 modulo 16 keep a gather at about 1.6 wavefronts,
// while multiples of 32 need 5 (simulated over the QI layout for ROIs of 44 to 128 px; 64 px ROIs took 18.6 k
// wavefronts per ROI as floats at pitch 64, 9.2 k at 68).
__host__ __device__ inline int tile_pitch(int W)
{
    const int p = (W + 3) & ~3;
    return p & 15 ? p : p + 4;
}

// Rows back to back without whole 16-byte units: the layout of ROIs that fit in no other.
__host__ __device__ inline bool packed_rows(int W, int ts) { return ts == W && (W & 3); }

// Bytes of the tile region: the tile, and room for the raw ROI to be brought to its end at the alignment it
// has in global memory (raw_offset), far enough behind the tile words that replace it (convert_raw).
__host__ __device__ inline int tile_region_bytes(int W, int H, int ts) { return ((H * ts * 4 + 15) & ~15) + 32; }
__host__ __device__ inline int raw_offset(int W, int H, int ts, int bpp, int misalign)
{
    return tile_region_bytes(W, H, ts) - ((W * H * bpp + 15) & ~15) - 16 + misalign;
}

// Integer pixels are packed unless calibration images turn them into fractions, or rows are.
__host__ __device__ inline int tile_format(const TrackParams &P, int ts)
{
    if (P.pdt == 2 || P.calib_count > 0 || packed_rows(P.width, ts)) return kTileF32;
    return P.pdt == 1 ? kTileU16 : kTileU8;
}

__host__ __device__ inline int tile_bpp(const TrackParams &P) { return P.pdt == 0 ? 1 : (P.pdt == 1 ? 2 : 4); }

// ---- pixels of a word -----------------------------------------------------------------------------------
// Pixel k of a word (0 itself, 1 right, 2 below, 3 below right) as 2^23 + pixel: the integer placed in the
// mantissa of 2^23. Differences of two such floats are exact, and subtracting 2^23 gives the pixel exactly.
template <int F, int K>
__device__ __forceinline__ float biased(uint32_t w)
{
    if (F == kTileU16) return __uint_as_float(__byte_perm(w, 0x4B000000u, K ? 0x7432u : 0x7410u));
    return __uint_as_float(__byte_perm(w, 0x4B000000u, 0x7540u + K));
}

constexpr float kBias = 8388608.0f;  // 2^23

// A tile word at a 32-bit shared-memory address (+ kOff bytes). Not volatile, so that loads of one sample may be
// scheduled among another's arithmetic: the compiler sees a function of the address alone. What keeps it behind the
// barrier that completes the tile is its address, which only a TileAddr gives.
template <int kOff = 0>
__device__ __forceinline__ uint32_t tile_word(uint32_t a)
{
    uint32_t v;
    asm("ld.shared.b32 %0, [%1+%2];" : "=r"(v) : "r"(a), "n"(kOff));
    return v;
}
template <int kOff = 0>
__device__ __forceinline__ float tile_float(uint32_t a)
{
    return __uint_as_float(tile_word<kOff>(a));
}

// Addresses of cells from biased coordinates (2^23 + the truncated coordinate, as the round-toward-zero add
// leaves them): row() of a y and at() of an x in that row. The biases are folded into one constant.
// Constructed behind the barrier that completes the tile. The base passes through a statement that the compiler keeps
// in order with barriers and memory accesses, so that no address, and no load, exists before it: neither the
// position nor the directions need to come from behind the barrier (the adjoint's come from global memory).
struct TileAddr {
    uint32_t base, ts4;
    __device__ __forceinline__ TileAddr(const uint32_t *tile, int ts) : ts4(4u * ts)
    {
        base = smem_addr(tile) - 0x4B000000u * (ts4 + 4u);
        asm volatile("" : "+r"(base)::"memory");
    }
    __device__ __forceinline__ uint32_t row(float ty) const { return __float_as_uint(ty) * ts4 + base; }
    __device__ __forceinline__ uint32_t at(uint32_t row, float tx) const { return row + (__float_as_uint(tx) << 2); }
};

// The corners of two samples' cells, at the words at p and q: the upper and lower left pixels v00 and v01, and the
// differences d0 = v10 - v00 and d1 = v11 - v01 along x (fma(v00, -1, v10), exact before its one rounding).
struct Cells {
    float2 v00, v01, d0, d1;
};

template <int F>
__device__ __forceinline__ Cells cells2(uint32_t p, uint32_t q, uint32_t ts4)
{
    const float2 m1 = make_float2(-1.0f, -1.0f);
    Cells c;
    if (F == kTileF32) {
        c.v00 = make_float2(tile_float(p), tile_float(q));
        c.d0 = __ffma2_rn(c.v00, m1, make_float2(tile_float<4>(p), tile_float<4>(q)));
        p += ts4;
        q += ts4;
        c.v01 = make_float2(tile_float(p), tile_float(q));
        c.d1 = __ffma2_rn(c.v01, m1, make_float2(tile_float<4>(p), tile_float<4>(q)));
    } else {
        const float2 nK = make_float2(-kBias, -kBias);
        const uint32_t p0 = tile_word(p), q0 = tile_word(q);
        float2 b01, b11;
        const float2 b00 = make_float2(biased<F, 0>(p0), biased<F, 0>(q0));
        const float2 b10 = make_float2(biased<F, 1>(p0), biased<F, 1>(q0));
        if (F == kTileU16) {
            const uint32_t p1 = tile_word(p + ts4), q1 = tile_word(q + ts4);
            b01 = make_float2(biased<F, 0>(p1), biased<F, 0>(q1));
            b11 = make_float2(biased<F, 1>(p1), biased<F, 1>(q1));
        } else {
            b01 = make_float2(biased<F, 2>(p0), biased<F, 2>(q0));
            b11 = make_float2(biased<F, 3>(p0), biased<F, 3>(q0));
        }
        c.d0 = __ffma2_rn(b00, m1, b10);
        c.d1 = __ffma2_rn(b01, m1, b11);
        c.v00 = __fadd2_rn(b00, nK);
        c.v01 = __fadd2_rn(b01, nK);
    }
    return c;
}

// Bilinear values of the two samples with fractions fx = (fx_p, fx_q) and fy: v0 + (v1 - v0) fy with
// v0 = v00 + (v10 - v00) fx and v1 likewise from the row below, in packed FP32x2 (each component rounds as the
// scalar operation does).
template <int F>
__device__ __forceinline__ float2 cell2(uint32_t p, uint32_t q, uint32_t ts4, float2 fx, float2 fy)
{
    const Cells c = cells2<F>(p, q, ts4);
    const float2 v0 = __ffma2_rn(c.d0, fx, c.v00), v1 = __ffma2_rn(c.d1, fx, c.v01);
    return __ffma2_rn(__ffma2_rn(v0, make_float2(-1.0f, -1.0f), v1), fy, v0);
}

// The same for one sample.
template <int F>
__device__ __forceinline__ float cell(uint32_t p, uint32_t ts4, float fx, float fy)
{
    float v00, v10, v01, v11;
    if (F == kTileF32) {
        v00 = tile_float(p), v10 = tile_float<4>(p);
        v01 = tile_float(p + ts4), v11 = tile_float<4>(p + ts4);
    } else {
        const uint32_t a = tile_word(p), b = F == kTileU16 ? tile_word(p + ts4) : a;
        v00 = biased<F, 0>(a) - kBias, v10 = biased<F, 1>(a) - kBias;
        v01 = biased<F, F == kTileU16 ? 0 : 2>(b) - kBias, v11 = biased<F, F == kTileU16 ? 1 : 3>(b) - kBias;
    }
    const float v0 = fmaf(v10 - v00, fx, v00), v1 = fmaf(v11 - v01, fx, v01);
    return fmaf(v1 - v0, fy, v0);
}

// The pixel of a word as a float.
template <int F>
__device__ __forceinline__ float word_pixel(uint32_t w)
{
    return F == kTileF32 ? __uint_as_float(w) : biased<F, 0>(w) - kBias;
}

// ---- load -----------------------------------------------------------------------------------------------
// Bring the ROI's raw bytes (rows of rowb bytes at `pitch`) to `raw`, rows back to back, in the widest unit that
// the addresses allow. All threads; a barrier must follow.
template <int T, typename U>
__device__ __forceinline__ void copy_rows(uint8_t *raw, const uint8_t *src, int pitch, int rowb, int H)
{
    const int per_row = rowb / (int)sizeof(U), total = per_row * H;
    const int dx = T % per_row, dy = T / per_row;
    int x = threadIdx.x % per_row, y = threadIdx.x / per_row;
    U *dst = reinterpret_cast<U *>(raw);
    constexpr int kBatch = 8;
#pragma unroll 1
    for (int i0 = threadIdx.x; i0 < total; i0 += kBatch * T) {
        U v[kBatch];
#pragma unroll
        for (int k = 0; k < kBatch; k++) {
            if (i0 + k * T < total) v[k] = __ldcs(reinterpret_cast<const U *>(src + (size_t)y * pitch) + x);
            x += dx;
            y += dy;
            if (x >= per_row) {
                x -= per_row;
                y++;
            }
        }
#pragma unroll
        for (int k = 0; k < kBatch; k++)
            if (i0 + k * T < total) dst[i0 + k * T] = v[k];
    }
}

template <int T>
__device__ __noinline__ void load_rows(uint8_t *raw, const uint8_t *src, int pitch, int rowb, int H)
{
    const unsigned a = (unsigned)reinterpret_cast<uintptr_t>(src) | (unsigned)pitch | (unsigned)rowb;
    if (!(a & 15))
        copy_rows<T, uint4>(raw, src, pitch, rowb, H);
    else if (!(a & 3))
        copy_rows<T, uint32_t>(raw, src, pitch, rowb, H);
    else if (!(a & 1))
        copy_rows<T, uint16_t>(raw, src, pitch, rowb, H);
    else
        copy_rows<T, uint8_t>(raw, src, pitch, rowb, H);
}

// Bytes from which on a contiguous ROI is brought by a bulk copy (at least one whole 16-byte unit inside it,
// wherever it starts).
constexpr int kMinBulkBytes = 64;

// Start the bulk copy of the ROI's whole 16-byte units (thread 0); raw has src's alignment modulo 16.
__device__ __forceinline__ void bulk_load_inner(uint8_t *raw, const uint8_t *src, int bytes, uint64_t *mbar)
{
    const int head = (int)(-reinterpret_cast<uintptr_t>(src) & 15), inner = (bytes - head) & ~15;
    bulk_load(raw + head, src + head, (uint32_t)inner, mbar);
}

// The up to 15 bytes before and behind them (one per thread, all inside the ROI). A barrier must follow.
__device__ __forceinline__ void load_ends(uint8_t *raw, const uint8_t *src, int bytes)
{
    const int head = (int)(-reinterpret_cast<uintptr_t>(src) & 15), inner = (bytes - head) & ~15;
    const int t = threadIdx.x, i = t < 16 ? t : head + inner + t - 16;
    if (t < 16 ? t < head : (t < 32 && i < bytes)) raw[i] = src[i];
}

// i / d for 0 <= i < 2^20, 1 <= d < 2^10, by the reciprocal: (i + 0.5) / d is at least 0.5 / d away from an integer,
// far more than the rounding errors (2^-22 of a quotient that is below 2^12 where it is used).
struct SmallDiv {
    float inv;
    __device__ __forceinline__ explicit SmallDiv(int d) : inv(1.0f / (float)d) {}
    __device__ __forceinline__ int operator()(int i) const { return (int)(((float)i + 0.5f) * inv); }
};

constexpr uint32_t kStageWaitLimit = 1u << 22;  // mbarrier polls that a late copy gets before its CTA ends

// Whether the ROI's copy was late: the word behind its mbarrier, set by load_raw.
__device__ __forceinline__ uint32_t &copy_late(uint64_t *mbar) { return *reinterpret_cast<uint32_t *>(mbar + 1); }

// Bring the ROI at `src` to the raw area of the tile region and return where it starts. A contiguous ROI arrives by
// one bulk copy (cp.async.bulk, completion on an mbarrier) that thread 0 starts first, while all run `meanwhile`
// (fetching tables); its up to 15 bytes before and behind the whole 16-byte units are loaded directly. Frame
// bands, and small or misaligned ROIs, are loaded row by row. Ends with a barrier.
// A copy that is late (P.copy_polls) is flagged and given a last bounded wait, since it writes into this CTA's shared
// memory; the word behind the mbarrier (copy_late) then says so, and the caller writes NaN results at its end. (Every
// step is in bounds whatever the pixels are. Leaving early costs more than it saves: with a branch around the rest,
// 10,000 100x100 u16 ROIs took 864 us instead of 831.)
template <int F, int T, typename Fn>
__device__ __forceinline__ const uint8_t *load_raw(uint32_t *tile, int ts, const TrackParams &P, const uint8_t *src,
                                                   int pitch, uint64_t *mbar, const Fn &meanwhile)
{
    const int W = P.width, H = P.height, bpp = tile_bpp(P), bytes = W * H * bpp;
    const int misalign = (int)(reinterpret_cast<uintptr_t>(src) & 15);
    const bool bulk = pitch == W * bpp && bytes >= kMinBulkBytes && !(misalign & (bpp - 1));
    uint8_t *raw = reinterpret_cast<uint8_t *>(tile) + raw_offset(W, H, ts, bpp, bulk ? misalign : 0);
    if (bulk && threadIdx.x == 0) {
        mbar_init(mbar);
        bulk_load_inner(raw, src, bytes, mbar);
    }
    meanwhile();
    if (bulk) {
        load_ends(raw, src, bytes);
        // one thread waits for the copy (its acquire, then the barrier, order the copied bytes
        // before every thread's reads); the others wait at the barrier without polling
        if (threadIdx.x == 0) {
            const bool late = !mbar_wait(mbar, 0, P.copy_polls);
            if (late) {
                if (P.err_flag) atomicOr(P.err_flag, 4u);
                mbar_wait(mbar, 0, kStageWaitLimit);
            }
            copy_late(mbar) = late;
        }
    } else {
        if (threadIdx.x == 0) copy_late(mbar) = 0u;
        load_rows<T>(raw, src, pitch, W * bpp, H);
    }
    __syncthreads();
    if (F != kTileF32 && (P.mode & kLT_ClearFirstFourPixels)) {  // QueuedCPUTracker.cpp:280-282
        if (threadIdx.x < 4 * bpp) raw[threadIdx.x] = 0;
        __syncthreads();
    }
    return raw;
}

// Walks the tile's units at a fixed stride. A unit is four pixels of a row from a column that is a multiple of
// four (the last of a row may reach past it): unit u is at row u / upr, column 4 (u mod upr), upr units per row.
struct UnitWalk {
    int x, off, pix;          // column, tile word and pixel index of the unit
    int dx, doff, dpix;       // their change per step
    int row_x, row_off, row_pix;  // their change when the column passes the row's end
    int W;
    __device__ __forceinline__ UnitWalk(int first, int stride, int W_, int ts) : W(W_)
    {
        const int upr = (W + 3) >> 2;
        const SmallDiv div(upr);
        const int r = div(first), rs = div(stride);
        x = 4 * (first - r * upr);
        off = r * ts + x;
        pix = r * W + x;
        dx = 4 * (stride - rs * upr);
        doff = rs * ts + dx;
        dpix = rs * W + dx;
        row_x = 4 * upr;
        row_off = ts - row_x;
        row_pix = W - row_x;
    }
    __device__ __forceinline__ void step()
    {
        x += dx;
        off += doff;
        pix += dpix;
        if (x >= W) {
            x -= row_x;
            off += row_off;
            pix += row_pix;
        }
    }
};

// The pixel steps of a float tile that a plain ROI does not have: clearing the first four pixels and the per-bead
// calibration. Not inlined (a rare path).
static __device__ __noinline__ float finish_pixel_call(float v, int i, int mode, float off_factor, float gain_factor,
                                                       const float *off, const float *gain)
{
    return finish_pixel(v, i, mode, off_factor, gain_factor, off, gain);
}

// Five consecutive pixels of an integer ROI from byte address a (shared memory), at any alignment the pixel type
// allows: the first four in x, y as they lie in memory (u8: x alone), the fifth in nx. Whole 32-bit words are read;
// they reach at most 7 bytes past the pixels, inside the CTA's shared memory.
template <int F>
__device__ __forceinline__ void raw_five(const uint8_t *a, uint32_t &x, uint32_t &y, uint32_t &nx)
{
    const uint32_t s = (uint32_t)reinterpret_cast<uintptr_t>(a) & 3u;
    const uint32_t *w = reinterpret_cast<const uint32_t *>(a - s);
    if (F == kTileU16) {
        const uint32_t w0 = w[0], w1 = w[1], w2 = w[2];
        x = __funnelshift_r(w0, w1, 8 * s);
        y = __funnelshift_r(w1, w2, 8 * s);
        nx = w2 >> (8 * s);
    } else {
        const uint32_t w0 = w[0], w1 = w[1];
        x = __funnelshift_r(w0, w1, 8 * s);
        y = 0u;
        nx = w1 >> (8 * s);
    }
}

// Turn the raw ROI (at `raw`, rows back to back, behind the tile's words) into the tile, in place: every thread
// reads a batch of raw units, a barrier passes, the words are written. The words of unit (row, x) end at byte
// 4 (row ts + x) + 16 at most, and the pixels of later units start at raw + bpp (pixel index): the region holds
// the raw ROI so far back (tile_region_bytes, raw_offset; ts >= W) that the former never exceeds the latter, so
// a batch overwrites no raw pixel of a later one. Returns this thread's pixel sum: exact as an integer
// (isum), or FP32 sums of a unit's pixels added in FP64 (kTileF32). Every thread runs the same number of
// batches.
// kPlain: whole units that lie aligned in the raw ROI (read with one load) and, for kTileF32, are floats that nothing
// changes; the other ROIs take a call.
template <int F, int T, bool kPlain>
__device__ __forceinline__ double convert_units(uint32_t *tile, const uint8_t *raw, int ts, const TrackParams &P,
                                                int bead, uint32_t &isum)
{
    const int W = P.width, H = P.height, n = W * H, upr = (W + 3) >> 2, units = upr * H;
    const int bpp = F == kTileU16 ? 2 : (F == kTileU8 ? 1 : (kPlain ? 4 : tile_bpp(P)));
    constexpr bool aligned = kPlain;
    double sum = 0.0;
    isum = 0u;
    UnitWalk w(threadIdx.x, T, W, ts);
    if constexpr (F != kTileF32) {
        constexpr int kBatch = 4;
#pragma unroll 1
        for (int u0 = threadIdx.x, b0 = 0; b0 < units; b0 += kBatch * T, u0 += kBatch * T) {
            // pixels 0-3 of the unit in (x, y) and pixel 4 in nx; for u8 y holds the row below and nx both rows'
            // fifth pixels
            uint32_t x[kBatch], y[kBatch], nx[kBatch];
            UnitWalk v = w;
#pragma unroll
            for (int k = 0; k < kBatch; k++) {
                x[k] = y[k] = nx[k] = 0u;
                if (u0 + k * T < units) {
                    const uint8_t *a = raw + v.pix * bpp;
                    if (F == kTileU16) {
                        if (aligned) {
                            const uint2 q = *reinterpret_cast<const uint2 *>(a);
                            x[k] = q.x;
                            y[k] = q.y;
                            nx[k] = reinterpret_cast<const uint16_t *>(a)[4];
                        } else {
                            raw_five<F>(a, x[k], y[k], nx[k]);
                        }
                    } else {
                        // the row below the last one is never sampled: its own row again
                        const uint8_t *b = v.pix + W < n ? a + W : a;
                        if (aligned) {
                            x[k] = *reinterpret_cast<const uint32_t *>(a);
                            y[k] = *reinterpret_cast<const uint32_t *>(b);
                            nx[k] = a[4] | (uint32_t)b[4] << 8;
                        } else {
                            uint32_t none, na, nb;
                            raw_five<F>(a, x[k], none, na);
                            raw_five<F>(b, y[k], none, nb);
                            nx[k] = __byte_perm(na, nb, 0x0040u);
                        }
                    }
                }
                v.step();
            }
            __syncthreads();
#pragma unroll
            for (int k = 0; k < kBatch; k++) {
                if (u0 + k * T < units) {
                    uint4 q;
                    if (F == kTileU16) {
                        q = make_uint4(x[k], __byte_perm(x[k], y[k], 0x5432u), y[k], __byte_perm(y[k], nx[k], 0x5432u));
                        uint32_t sx = x[k], sy = y[k];
                        if (W & 3) {  // pixels past the row's end do not count
                            const int r = W - w.x;
                            if (r < 2) sx &= 0xffffu;
                            if (r < 4) sy = r == 3 ? sy & 0xffffu : 0u;
                        }
                        isum = __dp2a_lo(sx, 0x0101u, isum);
                        isum = __dp2a_lo(sy, 0x0101u, isum);
                    } else {
                        q = make_uint4(__byte_perm(x[k], y[k], 0x5410u), __byte_perm(x[k], y[k], 0x6521u),
                                       __byte_perm(x[k], y[k], 0x7632u),
                                       __byte_perm(__byte_perm(x[k], nx[k], 0x4443u), __byte_perm(y[k], nx[k], 0x5553u),
                                                   0x5410u));
                        uint32_t sx = x[k];
                        if ((W & 3) && W - w.x < 4) sx &= (1u << 8 * (W - w.x)) - 1u;
                        isum = __dp4a(sx, 0x01010101u, isum);
                    }
                    *reinterpret_cast<uint4 *>(tile + w.off) = q;
                }
                w.step();
            }
        }
    } else {
        constexpr int kBatch = 4;
        const float *off = nullptr, *gain = nullptr;
        if (!kPlain && bead >= 0 && bead < P.calib_count) {
            if (P.calib_offset) off = P.calib_offset + (size_t)bead * n;
            if (P.calib_gain) gain = P.calib_gain + (size_t)bead * n;
        }
        const bool plain = kPlain || (!off && !gain && !(P.mode & kLT_ClearFirstFourPixels));
#pragma unroll 1
        for (int u0 = threadIdx.x, b0 = 0; b0 < units; b0 += kBatch * T, u0 += kBatch * T) {
            float f[kBatch][4];
            UnitWalk v = w;
#pragma unroll
            for (int k = 0; k < kBatch; k++) {
                const int count = u0 + k * T < units ? min(4, W - v.x) : 0;
                if (aligned) {
                    const float4 q = count ? reinterpret_cast<const float4 *>(raw)[v.pix >> 2] : make_float4(0, 0, 0, 0);
                    f[k][0] = q.x, f[k][1] = q.y, f[k][2] = q.z, f[k][3] = q.w;
                } else {
#pragma unroll
                    for (int j = 0; j < 4; j++) {
                        f[k][j] = 0.0f;
                        if (j < count)
                            f[k][j] = P.pdt == 2 ? reinterpret_cast<const float *>(raw)[v.pix + j]
                                                 : u_to_float(P.pdt == 1 ? reinterpret_cast<const uint16_t *>(raw)[v.pix + j]
                                                                         : raw[v.pix + j]);
                    }
                }
                v.step();
            }
            __syncthreads();
#pragma unroll
            for (int k = 0; k < kBatch; k++) {
                if (u0 + k * T < units) {
                    if (!plain)
#pragma unroll
                        for (int j = 0; j < 4; j++)
                            if (w.x + j < W)
                                f[k][j] = finish_pixel_call(f[k][j], w.pix + j, P.mode, P.offset_factor, P.gain_factor,
                                                            off, gain);
                    *reinterpret_cast<float4 *>(tile + w.off) = make_float4(f[k][0], f[k][1], f[k][2], f[k][3]);
                    sum += (double)((f[k][0] + f[k][1]) + (f[k][2] + f[k][3]));  // zeros past the row's end
                }
                w.step();
            }
        }
    }
    return sum;
}

// What the conversion of a ROI that is not plain needs of TrackParams (a call's arguments).
struct RawForm {
    int W, H, pdt, mode, calib_count;
    float off_factor, gain_factor;
    const float *offset, *gain;
};

template <int F, int T>
__device__ __noinline__ double convert_call(uint32_t *tile, const uint8_t *raw, int ts, RawForm f, int bead,
                                            uint32_t *isum)
{
    TrackParams P;
    P.width = f.W;
    P.height = f.H;
    P.pdt = f.pdt;
    P.mode = f.mode;
    P.calib_count = f.calib_count;
    P.calib_offset = f.offset;
    P.calib_gain = f.gain;
    P.offset_factor = f.off_factor;
    P.gain_factor = f.gain_factor;
    uint32_t s;
    const double sum = convert_units<F, T, false>(tile, raw, ts, P, bead, s);
    *isum = s;
    return sum;
}

template <int F, int T>
__device__ __forceinline__ double convert_raw(uint32_t *tile, const uint8_t *raw, int ts, const TrackParams &P, int bead,
                                              uint32_t &isum)
{
    const int unit = 4 * (F == kTileU16 ? 2 : (F == kTileU8 ? 1 : 4));
    bool plain = !(P.width & 3) && !((uint32_t)reinterpret_cast<uintptr_t>(raw) & (unit - 1));
    if (F == kTileF32) plain = plain && P.pdt == 2 && P.calib_count == 0 && !(P.mode & kLT_ClearFirstFourPixels);
    if (plain) return convert_units<F, T, true>(tile, raw, ts, P, bead, isum);
    const RawForm f = {P.width,         P.height,       P.pdt,          P.mode,      P.calib_count,
                       P.offset_factor, P.gain_factor, P.calib_offset, P.calib_gain};
    uint32_t s;
    const double sum = convert_call<F, T>(tile, raw, ts, f, bead, &s);
    isum = s;
    return sum;
}

// ---- mean and COM -----------------------------------------------------------------------------------------
// This thread's FP64 sum of the pixels' squares (for the background threshold), over the units of convert_raw.
template <int F, int T>
__device__ __noinline__ double square_sum(const uint32_t *tile, int W, int H, int ts)
{
    double s = 0.0;
    const int units = ((W + 3) >> 2) * H;
    UnitWalk w(threadIdx.x, T, W, ts);
    for (int u = threadIdx.x; u < units; u += T, w.step()) {
        float q = 0.0f;
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const float v = w.x + j < W ? word_pixel<F>(tile[w.off + j]) : 0.0f;
            q = fmaf(v, v, q);
        }
        s += (double)q;
    }
    return s;
}

// CPUTracker::ComputeMeanAndCOM, cpu_tracker.cpp:681-729, on a converted tile (no barrier since): the mean from
// the pixel sums, the background threshold's stdev, then the moments of v' = max(0, |v - mean| - thr). The
// moments run over 512 chains of units (unit u in chain u mod 512; FP32 within a chain, a few dozen
// pixels, FP64 across chains; the reference accumulates in FP64).
constexpr int kComChains = 512;

// The moments over this thread's chains (kThr: with a threshold).
template <int F, int T, bool kThr>
__device__ __forceinline__ void com_moments(const uint32_t *tile, int W, int H, int ts, float mean, float thr,
                                            double (&m)[3])
{
    const float2 nK = make_float2(-kBias, -kBias), nm = make_float2(-mean, -mean);
    auto dev = [&](float d) { return kThr ? fmaxf(0.0f, fabsf(d) - thr) : fabsf(d); };
    // column and row as floats; the step to this thread's next chain (c) and the step along a chain (k)
    const int upr = (W + 3) >> 2, units = upr * H;
    const SmallDiv div(upr);
    const int r0 = div(threadIdx.x), rc = div(T), rk = div(kComChains);
    const float fW = (float)W, fend = (float)(4 * upr);
    float cx = (float)(4 * ((int)threadIdx.x - r0 * upr)), cy = (float)r0;
    const float cdx = (float)(4 * (T - rc * upr)), cdy = (float)rc, kdx = (float)(4 * (kComChains - rk * upr)), kdy = (float)rk;
    const int wrap = ts - 4 * upr;
    int coff = r0 * ts + 4 * ((int)threadIdx.x - r0 * upr);
    const int cdo = rc * ts + 4 * (T - rc * upr), kdo = rk * ts + 4 * (kComChains - rk * upr);
    const bool ragged = (W & 3) != 0;
#pragma unroll 1
    for (int chain = threadIdx.x; chain < kComChains && chain < units; chain += T) {
        float q0 = 0.0f, qx = 0.0f, qy = 0.0f, fx = cx, fy = cy;
        int off = coff;
#pragma unroll 1
        for (int u = chain; u < units; u += kComChains) {
            const uint4 w = *reinterpret_cast<const uint4 *>(tile + off);
            float2 a01, a23;
            if (F == kTileF32) {
                a01 = make_float2(__uint_as_float(w.x), __uint_as_float(w.y));
                a23 = make_float2(__uint_as_float(w.z), __uint_as_float(w.w));
            } else {  // a pixel and its right neighbour in words 0 and 2
                a01 = __fadd2_rn(make_float2(biased<F, 0>(w.x), biased<F, 1>(w.x)), nK);
                a23 = __fadd2_rn(make_float2(biased<F, 0>(w.z), biased<F, 1>(w.z)), nK);
            }
            a01 = __fadd2_rn(a01, nm);
            a23 = __fadd2_rn(a23, nm);
            float a0 = dev(a01.x), a1 = dev(a01.y), a2 = dev(a23.x), a3 = dev(a23.y);
            if (ragged) {  // nothing past the row's end
                if (fx + 1.0f >= fW) a1 = 0.0f;
                if (fx + 2.0f >= fW) a2 = 0.0f;
                if (fx + 3.0f >= fW) a3 = 0.0f;
            }
            const float s23 = a2 + a3, S = (a0 + a1) + s23;
            const float Sj = fmaf(2.0f, s23, a1 + a3);  // sum j v' = a1 + 2 a2 + 3 a3, so that sum x v' = fx S + Sj
            q0 += S;
            qx += fmaf(fx, S, Sj);
            qy = fmaf(fy, S, qy);
            fx += kdx;
            fy += kdy;
            off += kdo;
            if (fx >= fW) {
                fx -= fend;
                fy += 1.0f;
                off += wrap;
            }
        }
        m[0] += (double)q0;
        m[1] += (double)qx;
        m[2] += (double)qy;
        cx += cdx;
        cy += cdy;
        coff += cdo;
        if (cx >= fW) {
            cx -= fend;
            cy += 1.0f;
            coff += wrap;
        }
    }
}

// With a threshold, as a call: the kernels are fetched cold by small launches, and what few ROIs need stays out of
// the way (with the conversions above: 10,000 100x100 u16 ROIs 0.846 -> 0.832 ms, the adjoint of 51,200 80x80 u16
// ones 0.795 -> 0.763 ms).
template <int F, int T>
__device__ __noinline__ void com_moments_call(const uint32_t *tile, int W, int H, int ts, float mean, float thr,
                                              double *m)
{
    double v[3] = {0.0, 0.0, 0.0};
    com_moments<F, T, true>(tile, W, H, ts, mean, thr, v);
    for (int k = 0; k < 3; k++) m[k] = v[k];
}

template <int F, int T>
__device__ __forceinline__ ComResult tile_com(const uint32_t *tile, int W, int H, int ts, double sum, uint32_t isum,
                                              float bgcorr, double *red)
{
    constexpr int kWarps = T / 32;
    const BlockGroup g{red};
    const int n = W * H;
    if (F == kTileF32) {
        double v[1] = {sum};
        g.sum(v);
        sum = v[0];
    } else {
        // exact: at most 65535 x 58,000 pixels (shared memory) < 2^32
        uint32_t *ired = reinterpret_cast<uint32_t *>(red);
        isum = __reduce_add_sync(0xffffffffu, isum);
        if ((threadIdx.x & 31) == 0) ired[threadIdx.x >> 5] = isum;
        __syncthreads();
        isum = 0u;
        for (int k = 0; k < kWarps; k++) isum += ired[k];
        sum = (double)isum;
    }
    const float invN = 1.0f / (float)n;
    ComResult r;
    r.mean = (float)(sum * (double)invN);
    r.stdev = 0.0f;
    float thr = 0.0f;
    if (bgcorr != 0.0f) {
        double v[1] = {square_sum<F, T>(tile, W, H, ts)};
        g.sum(v);
        r.stdev = sqrtf((float)(v[0] * (double)invN - (double)(r.mean * r.mean)));
        thr = bgcorr * r.stdev;
    }
    double m[3] = {0.0, 0.0, 0.0};
    if (bgcorr != 0.0f)
        com_moments_call<F, T>(tile, W, H, ts, r.mean, thr, m);
    else
        com_moments<F, T, false>(tile, W, H, ts, r.mean, 0.0f, m);
    g.sum(m);
    if (bgcorr == 0.0f && m[0] < 1e-3 * fabs((double)r.mean) * n) {
        // A nearly flat image: the reference's stdev may be the root of a negative difference, and its
        // threshold 0 * stdev then leaves no pixel, so that the COM is not a number.
        double v[1] = {square_sum<F, T>(tile, W, H, ts)};
        g.sum(v);
        if (v[0] * (double)invN - (double)(r.mean * r.mean) < 0.0) m[0] = m[1] = m[2] = 0.0;
    }
    r.x = (float)(m[1] / m[0]);
    r.y = (float)(m[2] / m[0]);
    return r;
}

// ---- QI quadrant profiles -----------------------------------------------------------------------------------
// CPUTracker::ComputeQuadrantProfile (cpu_tracker.cpp:631-677) for all four quadrants at once, written as the
// FFT input of the QI autoconvolution. The four quadrants sample the same table direction d at radius r with
// mirrored signs (x = cx +- d.x r, y = cy +- d.y r), so one thread takes one radius and a subset of the
// directions and produces all four samples of each: the truncations and fractions of the two x and two y
// coordinates are shared by four samples. The table holds each direction as (d.x, d.x, d.y, d.y) so that
// (x+, x-) = (cx, cx) + (d.x, d.x) * (r, -r) is one packed multiply-add; the diagonal quadrants q0 (+, +) and
// q2 (-, -) then share the packed fractions (fx+, fx-), (fy+, fy-), and q3 (+, -) and q1 (-, +) the same fx
// with fy swapped. On circles that lie inside the image every sample counts and needs no check.
//
// A radius has eight direction subsets (a mod 8). Its threads are eight neighbouring lanes with one subset each, or
// four with two each (in separate sums, added first) when the CTA has fewer than 8 nr threads: the order of
// the sum is the same. A warp covers neighbouring radii and neighbouring directions, so its samples lie
// close together and share words.
//
// Bins with fewer than 4 samples in bounds take the mean. A receives one complex value z = X + iY per position, in
// bit-reversed order (log2L = log2(2 nr)) or in natural order when log2L < 0. A barrier must follow.
template <int F, int T>
__device__ __forceinline__ void qi_profiles(const uint32_t *img, int W, int H, int ts, float cx, float cy, float mean,
                                            int nr, int nang, float inv_nang, int stride, float minr, float rstep,
                                            const float4 *dirs, const float *rweights, float2 *A, int log2L)
{
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const TileAddr ta(img, ts);
    const bool two = 8 * nr > T;  // two subsets per lane
    const int lA = two ? 2 : 3, sub = lane & ((1 << lA) - 1);
#pragma unroll 1
    for (int i0 = warp << (5 - lA); i0 < nr; i0 += (T / 32) << (5 - lA)) {
        const int i = i0 + (lane >> lA);
        const float r = __fadd_rn(minr, __fmul_rn(rstep, (float)i));
        float sm[4];
        int cnt[4];
        // One path per aligned block of eight radii (a warp's, or two warps' of four): when any of its circles
        // may leave the image, all take the checked body. (A warp running both bodies one after the other
        // would hold up the CTA's other warps at the next barrier, and the two round their means
        // differently, so the choice must not depend on T.)
        const float rlo = __fadd_rn(minr, __fmul_rn(rstep, (float)(i & ~7)));
        const float rhi = __fadd_rn(minr, __fmul_rn(rstep, (float)(i | 7)));
        const bool fast = circle_inside(cx, cy, fmaxf(fabsf(rlo), fabsf(rhi)), W, H);
        if (fast) {
            const float2 rr = make_float2(r, -r), cxx = make_float2(cx, cx), cyy = make_float2(cy, cy);
            const float2 K = make_float2(kBias, kBias), nK = make_float2(-kBias, -kBias);
            const float2 m1 = make_float2(-1.0f, -1.0f);
            float2 s02[2] = {}, s31[2] = {};
            auto sample = [&](int a, float2 &c02, float2 &c31) {
                const float4 d = dirs[stride * a];
                const float2 X = __ffma2_rn(make_float2(d.x, d.y), rr, cxx);  // (x+, x-)
                const float2 Y = __ffma2_rn(make_float2(d.z, d.w), rr, cyy);  // (y+, y-)
                const float2 TX = __fadd2_rz(X, K), TY = __fadd2_rz(Y, K);
                const float2 FX = __ffma2_rn(__fadd2_rn(TX, nK), m1, X);  // X - trunc(X)
                const float2 FY = __ffma2_rn(__fadd2_rn(TY, nK), m1, Y);
                const uint32_t rowp = ta.row(TY.x), rowm = ta.row(TY.y);
                c02 = cell2<F>(ta.at(rowp, TX.x), ta.at(rowm, TX.y), ta.ts4, FX, FY);
                c31 = cell2<F>(ta.at(rowm, TX.x), ta.at(rowp, TX.y), ta.ts4, FX, make_float2(FY.y, FY.x));
            };
            const int end = i < nr ? nang : 0;
#pragma unroll 1
            for (int a = sub; a < end; a += 8) {
                float2 c02, c31;
                sample(a, c02, c31);
                s02[0] = __fadd2_rn(s02[0], c02);
                s31[0] = __fadd2_rn(s31[0], c31);
                if (two && a + 4 < end) {
                    sample(a + 4, c02, c31);
                    s02[1] = __fadd2_rn(s02[1], c02);
                    s31[1] = __fadd2_rn(s31[1], c31);
                }
            }
            s02[0] = __fadd2_rn(s02[0], s02[1]);
            s31[0] = __fadd2_rn(s31[0], s31[1]);
            sm[0] = s02[0].x;
            sm[1] = s31[0].y;
            sm[2] = s02[0].y;
            sm[3] = s31[0].x;
        } else {
            // the rule of Interpolate (utils.h:40-58) per coordinate: a sample is inside when -1 < x < W-1 and
            // -1 < y < H-1, and its cell starts at the truncation of max(x, 0)
            const float xhi = (float)(W - 1), yhi = (float)(H - 1);
            float s2[4] = {0.0f, 0.0f, 0.0f, 0.0f};
            sm[0] = sm[1] = sm[2] = sm[3] = 0.0f;
            cnt[0] = cnt[1] = cnt[2] = cnt[3] = 0;
            const int end = i < nr ? nang : 0, inc = two ? 4 : 8;
            bool odd = false;
#pragma unroll 1
            for (int a = sub; a < end; a += inc) {
                const float4 d = dirs[stride * a];
                const float xp = fmaf(d.x, r, cx), xm = fmaf(d.x, -r, cx);
                const float yp = fmaf(d.z, r, cy), ym = fmaf(d.z, -r, cy);
                const bool vxp = xp > -1.0f && xp < xhi, vxm = xm > -1.0f && xm < xhi;
                const bool vyp = yp > -1.0f && yp < yhi, vym = ym > -1.0f && ym < yhi;
                const float txp = __fadd_rz(fmaxf(xp, 0.0f), kBias), txm = __fadd_rz(fmaxf(xm, 0.0f), kBias);
                const float typ = __fadd_rz(fmaxf(yp, 0.0f), kBias), tym = __fadd_rz(fmaxf(ym, 0.0f), kBias);
                const float fxp = xp - (txp - kBias), fxm = xm - (txm - kBias);
                const float fyp = yp - (typ - kBias), fym = ym - (tym - kBias);
                const uint32_t rowp = ta.row(typ), rowm = ta.row(tym);
                const bool in[4] = {vxp && vyp, vxm && vyp, vxm && vym, vxp && vym};
#pragma unroll
                for (int q = 0; q < 4; q++) {
                    if (!in[q]) continue;
                    const bool right = q == 0 || q == 3, up = q < 2;
                    const float v = cell<F>(ta.at(up ? rowp : rowm, right ? txp : txm), ta.ts4, right ? fxp : fxm,
                                            up ? fyp : fym);
                    cnt[q]++;
                    if (two && odd)
                        s2[q] += v;
                    else
                        sm[q] += v;
                }
                odd = !odd;
            }
#pragma unroll
            for (int q = 0; q < 4; q++) sm[q] += s2[q];
        }
        // subsets of one radius: neighbouring lanes (on the fast path every count is nang)
        if (!two)
#pragma unroll
            for (int q = 0; q < 4; q++) sm[q] += __shfl_xor_sync(0xffffffffu, sm[q], 4);
#pragma unroll
        for (int o = 1; o < 4; o <<= 1)
#pragma unroll
            for (int q = 0; q < 4; q++) sm[q] += __shfl_xor_sync(0xffffffffu, sm[q], o);
        if (!fast)
            for (int o = 1; o < 1 << lA; o <<= 1)
#pragma unroll
                for (int q = 0; q < 4; q++) cnt[q] += __shfl_xor_sync(0xffffffffu, cnt[q], o);
        if (sub == 0 && i < nr) {
            const float rw = rweights ? rweights[i] : 1.0f;
            float v[4];
#pragma unroll
            for (int k = 0; k < 4; k++) {  // nang >= 4: on the fast path the mean, as sum * (1 / nang)
                v[k] = fast ? sm[k] * inv_nang : (cnt[k] >= 4 ? sm[k] / (float)cnt[k] : mean);
                if (rweights) v[k] *= rw;
            }
            const int n0 = nr - 1 - i, n1 = nr + i;
            A[log2L >= 0 ? (int)bitrev(n0, log2L) : n0] = make_float2(v[1] + v[2], v[2] + v[3]);
            A[log2L >= 0 ? (int)bitrev(n1, log2L) : n1] = make_float2(v[0] + v[3], v[0] + v[1]);
        }
    }
}

// ---- radial profile -------------------------------------------------------------------------------------
// ComputeRadialProfile, utils.cpp:275-320: for each bin, the mean of the in-bounds bilinear samples on the full
// circle (FP64 sum), or `mean` when no more than 4 samples are in bounds; then NormalizeRadialProfile
// (utils.cpp:230-261) when asked. dirs[j] = (d_j.x, d_{j+h}.x, d_j.y, d_{j+h}.y) for j < h = nang / 2, and d_{nang-1}
// alone in dirs[h] when nang is odd. A bin has eight lanes; lane s takes the pairs j = s, s + 8, ... (two samples
// per step, packed FP32x2) and lane 0 the unpaired direction. Four pairs are summed in FP32 (four
// samples per component) and folded into FP64; the reference adds every sample in FP64.
template <int F, int T>
__device__ __forceinline__ void radial_profile(const uint32_t *img, int W, int H, int ts, float cx, float cy, float mean,
                                               int nb, int nang, float minr, float rstep, const float4 *dirs,
                                               float *prof, bool normalize)
{
    const int sub = threadIdx.x & 7, h = nang >> 1;
    const TileAddr ta(img, ts);
#pragma unroll 1
    for (int b0 = threadIdx.x >> 3; b0 - (int)((threadIdx.x & 31) >> 3) < nb; b0 += T / 8) {
        const int bin = b0;
        double sum = 0.0;
        int cnt = 0;
        const float r = minr + rstep * (float)bin;
        // one path per warp: four bins, whatever T is (see qi_profiles)
        const bool inside = __all_sync(0xffffffffu, bin >= nb || circle_inside(cx, cy, fabsf(r), W, H));
        if (inside) {
            const float2 rr = make_float2(r, r), cxx = make_float2(cx, cx), cyy = make_float2(cy, cy);
            const float2 K = make_float2(kBias, kBias), nK = make_float2(-kBias, -kBias), m1 = make_float2(-1.0f, -1.0f);
            auto pair = [&](const float4 &d) {
                const float2 X = __ffma2_rn(make_float2(d.x, d.y), rr, cxx);
                const float2 Y = __ffma2_rn(make_float2(d.z, d.w), rr, cyy);
                const float2 TX = __fadd2_rz(X, K), TY = __fadd2_rz(Y, K);
                const float2 FX = __ffma2_rn(__fadd2_rn(TX, nK), m1, X), FY = __ffma2_rn(__fadd2_rn(TY, nK), m1, Y);
                return cell2<F>(ta.at(ta.row(TY.x), TX.x), ta.at(ta.row(TY.y), TX.y), ta.ts4, FX, FY);
            };
            const int np = bin < nb && sub < h ? (h - sub + 7) >> 3 : 0;
            const float4 *dl = dirs + sub;
            int k = 0;
#pragma unroll 1
            for (; k + 4 <= np; k += 4) {
                float2 part = make_float2(0.0f, 0.0f);
#pragma unroll 2
                for (int u = 0; u < 4; u++) part = __fadd2_rn(part, pair(dl[(k + u) * 8]));
                sum += (double)(part.x + part.y);
            }
            if (k < np) {
                float2 part = make_float2(0.0f, 0.0f);
#pragma unroll 1
                for (; k < np; k++) part = __fadd2_rn(part, pair(dl[k * 8]));
                sum += (double)(part.x + part.y);
            }
            if ((nang & 1) && sub == 0 && bin < nb) {
                const float4 d = dirs[h];
                sum += (double)pair(make_float4(d.x, d.x, d.z, d.z)).x;
            }
            cnt = nang;
        } else {
            // every sample checked; FP32 partials of up to 8 samples folded into FP64
            const float xhi = (float)(W - 1), yhi = (float)(H - 1);
            float part = 0.0f;
            int in_part = 0;
#pragma unroll 1
            for (int j = sub; j < h && bin < nb; j += 8) {
                const float4 d = dirs[j];
#pragma unroll 1
                for (int u = 0; u < 2; u++) {
                    const float x = fmaf(u ? d.y : d.x, r, cx), y = fmaf(u ? d.w : d.z, r, cy);
                    if (x > -1.0f && x < xhi && y > -1.0f && y < yhi) {
                        const float tx = __fadd_rz(fmaxf(x, 0.0f), kBias), ty = __fadd_rz(fmaxf(y, 0.0f), kBias);
                        part += cell<F>(ta.at(ta.row(ty), tx), ta.ts4, x - (tx - kBias), y - (ty - kBias));
                        cnt++;
                    }
                }
                if (++in_part == 4) {
                    sum += (double)part;
                    part = 0.0f;
                    in_part = 0;
                }
            }
            sum += (double)part;
            if ((nang & 1) && sub == 0 && bin < nb) {
                const float4 d = dirs[h];
                const float x = fmaf(d.x, r, cx), y = fmaf(d.z, r, cy);
                if (x > -1.0f && x < xhi && y > -1.0f && y < yhi) {
                    const float tx = __fadd_rz(fmaxf(x, 0.0f), kBias), ty = __fadd_rz(fmaxf(y, 0.0f), kBias);
                    sum += (double)cell<F>(ta.at(ta.row(ty), tx), ta.ts4, x - (tx - kBias), y - (ty - kBias));
                    cnt++;
                }
            }
#pragma unroll
            for (int o = 4; o > 0; o >>= 1) cnt += __shfl_xor_sync(0xffffffffu, cnt, o);
        }
#pragma unroll
        for (int o = 4; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
        if (bin < nb && sub == 0) prof[bin] = cnt > 4 ? (float)(sum / cnt) : mean;
    }
    __syncthreads();
    if (normalize && threadIdx.x < 32) {
        __syncwarp();
        const int lane = threadIdx.x;
        double s = 0;
        for (int i = lane; i < nb; i += 32) s += prof[i];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        const float m = (float)(s / nb);
        double s2 = 0;
        for (int i = lane; i < nb; i += 32) {
            const float p = prof[i] - m;
            prof[i] = p;
            s2 += (double)(p * p);
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) s2 += __shfl_xor_sync(0xffffffffu, s2, o);
        const double inv = 1.0 / sqrt(s2 / nb);
        for (int i = lane; i < nb; i += 32) prof[i] = (float)((double)prof[i] * inv);
    }
    __syncthreads();
}

}  // namespace qtrk

// Lighting products against 1440-azimuth horizon tiles on sm_100a:
// sun fraction (float32 and byte), body-centre margin, PSR.
//
// Semantics follow src/lunarscout/_numba_horizon/lightmap_cpu.py:25-183 (the
// per-pixel FP64 east/north/up frame, float32 per time step, 16-slice solar
// disk of src/lunarscout/_numba_horizon/lightmap.py:15-29) and
// psr_cuda.py:57-186 (PSR).  Arithmetic is the reference CPU backend's, op by
// op (this file builds with --fmad=false); atan2f is CUDA's.
//
// Design: the per-pixel frame (FP64 trigonometry) is computed once per tile
// into 12 floats per pixel; the time loop is split into chunks so that a
// tile's 16384 pixels x T times fill all SMs; one thread owns one pixel of
// one chunk and writes time-major rows [t, 128*128] (coalesced across the
// warp).  Many tiles may share one launch (blockIdx.z).  Long launches settle
// the clear samples without their exact direction (staged_samples).
#define LS200_LIGHTING_KERNELS
#include <cuda_fp16.h>

#include <algorithm>
#include <cmath>

#include "internal.cuh"
#include "lighting.cuh"

namespace ls200 {

// Whether the disk constants are on a device yet.  Contexts on one device
// each hold only their own lock, so the flag has a lock of its own.
static std::mutex g_constants_lock;
static bool g_constants_ready[64] = {};

void ensure_lighting_constants(ls200_context *ctx) {
    std::lock_guard<std::mutex> hold(g_constants_lock);
    if (g_constants_ready[ctx->device]) return;
    // Half-chords of a 16-column disk of radius float32(0.27) deg
    // (lightmap.py:19-25), rounded once to float32; the normaliser is twice
    // their float32 running sum.
    float hc[16];
    float sum = 0.0f;
    for (int i = 0; i < 16; ++i) {
        const double x = 7.5 - i;
        hc[i] = static_cast<float>(std::sqrt(64.0 - x * x) / 8.0 * static_cast<double>(0.27f));
        sum = sum + hc[i];
    }
    const float max_photons = 2.0f * sum;
    LS_CUDA(cudaMemcpyToSymbol(c_half_circle, hc, sizeof hc));
    LS_CUDA(cudaMemcpyToSymbol(c_max_photons, &max_photons, sizeof max_photons));
    g_constants_ready[ctx->device] = true;
}

// FP64 east/north/up frame of one DEM pixel (lightmap_cpu.py:51-103).
__device__ Frame32 pixel_frame(const TileGeo &g, int column, int row, float height) {
    const double *gt = g.gt, *proj = g.proj;
    const double crs_x = gt[0] + gt[1] * column + gt[2] * row;
    const double crs_y = gt[3] + gt[4] * column + gt[5] * row;
    const double xp = crs_x - proj[4];
    const double yp = crs_y - proj[5];
    const double rho = sqrt(xp * xp + yp * yp);
    double latitude, longitude;
    if (rho <= 1e-12) {
        longitude = proj[2];
        latitude = proj[1];
    } else {
        const double c = 2.0 * atan2(rho, 2.0 * proj[3] * proj[0]);
        double sin_c, cos_c, sin_o, cos_o;
        sincos(c, &sin_c, &cos_c);
        sincos(proj[1], &sin_o, &cos_o);
        latitude = asin(cos_c * sin_o + yp * sin_c * cos_o / rho);
        longitude = proj[2] + atan2(xp * sin_c, rho * cos_o * cos_c - yp * sin_o * sin_c);
    }
    const double radius = proj[0] + static_cast<double>(height);
    double sin_lat, cos_lat, sin_lon, cos_lon;
    sincos(latitude, &sin_lat, &cos_lat);
    sincos(longitude, &sin_lon, &cos_lon);
    const double moon_x = radius * cos_lat * cos_lon;
    const double moon_y = radius * cos_lat * sin_lon;
    const double moon_z = radius * sin_lat;
    const double up_x = cos_lat * cos_lon, up_y = cos_lat * sin_lon, up_z = sin_lat;
    const double east_x = -sin_lon, east_y = cos_lon;
    const double north_x = -sin_lat * cos_lon, north_y = -sin_lat * sin_lon, north_z = cos_lat;
    Frame32 f;
    f.v[0] = static_cast<float>(east_x);   // r00
    f.v[1] = static_cast<float>(north_x);  // r01
    f.v[2] = static_cast<float>(up_x);     // r02
    f.v[3] = static_cast<float>(east_y);   // r10
    f.v[4] = static_cast<float>(north_y);  // r11
    f.v[5] = static_cast<float>(up_y);     // r12
    f.v[6] = 0.0f;                         // r20
    f.v[7] = static_cast<float>(north_z);  // r21
    f.v[8] = static_cast<float>(up_z);     // r22
    f.v[9] = static_cast<float>(-(moon_x * east_x + moon_y * east_y));
    f.v[10] = static_cast<float>(-(moon_x * north_x + moon_y * north_y + moon_z * north_z));
    f.v[11] = static_cast<float>(-(moon_x * up_x + moon_y * up_y + moon_z * up_z));
    return f;
}

__global__ void __launch_bounds__(128) frames_kernel(const __grid_constant__ LightingBatch B) {
    const int tile = blockIdx.y;
    const int index = blockIdx.x * blockDim.x + threadIdx.x;
    if (index >= kPatch * kPatch) return;
    const TileGeo &g = B.tiles[tile];
    const int sample = index % kPatch, line = index / kPatch;
    Frame32 f{};
    if (sample < g.valid_width && line < g.valid_height)
        f = pixel_frame(g, g.tile_x + sample, g.tile_y + line,
                        B.patch_dem[static_cast<size_t>(tile) * kPatch * kPatch + index]);
    float *dst = B.frames + (static_cast<size_t>(tile) * kPatch * kPatch + index) * 12;
#pragma unroll
    for (int k = 0; k < 12; ++k) dst[k] = f.v[k];
}

// The frame of pixel `pixel` (tile * 16384 + index): three 16-byte loads where
// the caller's table allows them.
__device__ __forceinline__ Frame32 load_frame(const float *frames, size_t pixel) {
    if (reinterpret_cast<uintptr_t>(frames) & 15) {
        Frame32 f;
#pragma unroll
        for (int k = 0; k < 12; ++k) f.v[k] = __ldg(frames + pixel * 12 + k);
        return f;
    }
    const float4 *src = reinterpret_cast<const float4 *>(frames + pixel * 12);
    const float4 a = __ldg(src), b = __ldg(src + 1), c = __ldg(src + 2);
    return Frame32{{a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w, c.x, c.y, c.z, c.w}};
}

// Per-thread window of staged horizon bins (stride 33 spreads the threads'
// windows over the 32 shared-memory banks).
constexpr int kWindowBins = 32;
constexpr int kWindowStride = kWindowBins + 1;

template <int kSpan>
__device__ __forceinline__ BinPosition signal_position(float azimuth_deg) {
    return kSpan == 5 ? sun_position(azimuth_deg) : margin_position(azimuth_deg);
}

// The sun fraction (kSpan 5) or the margin (kSpan 2) of a pixel.
template <int kSpan, class Bins>
__device__ __forceinline__ float signal_bins(const Bins &bin, float fraction, float elevation) {
    return kSpan == 5 ? sun_fraction_bins(bin, fraction, elevation)
                      : horizon_margin_bins(bin, fraction, elevation);
}

// Stage the bins that positions [k0, k1) of the launch's order read (kSpan
// bins from each step's first bin: 2 for the margin, 5 for the fraction)
// into `window`; returns the number staged (0: none) and sets `first`, the
// window's first bin.  In longitude order the body's azimuth moves
// monotonically across a chunk, so the bins between those of its first and
// last steps, plus the span and a margin of 2 on each side, cover it; a step
// outside them reads its row directly.
template <int kSpan>
__device__ __forceinline__ int stage_window(const LightingBatch &B, const Frame32 &f,
                                            const float *horizon, int k0, int k1, float *window,
                                            int &first) {
    float azimuth_deg, elevation;
    const float *v = B.vectors + 3 * static_cast<size_t>(__ldg(B.order + k0));
    body_direction(f, __ldg(v), __ldg(v + 1), __ldg(v + 2), azimuth_deg, elevation);
    const int a = signal_position<kSpan>(azimuth_deg).left;
    v = B.vectors + 3 * static_cast<size_t>(__ldg(B.order + k1 - 1));
    body_direction(f, __ldg(v), __ldg(v + 1), __ldg(v + 2), azimuth_deg, elevation);
    const int b = signal_position<kSpan>(azimuth_deg).left;
    int arc = b - a;
    if (arc < 0) arc += kAzimuths;
    int start = arc <= kAzimuths / 2 ? a : b;
    if (arc > kAzimuths / 2) arc = kAzimuths - arc;
    start -= 2;
    if (start < 0) start += kAzimuths;
    const int width = arc + kSpan + 4;
    if (width > kWindowBins) return 0;
    first = start;
    for (int i = 0; i < width; ++i) {
        int bin = first + i;
        if (bin >= kAzimuths) bin -= kAzimuths;
        window[i] = __ldg(horizon + bin);
    }
    return width;
}

// Evaluates positions [k0, k1) of the launch's order for one pixel and calls
// put(time index, signal); `windowed`: with the bins staged (ordered launches).
// The loops are unrolled as measured: a margin's (3 steps without a window, 4
// with one) keep several row reads in flight, 16 patches of 125 and 1460 steps of
// a year 429 and 3055 us against 710 and 4175 with the loops left to the
// compiler; fractions take 2 and 1, bytes 2 and 2 (1 % better than others, and 4
// is 7 % worse).  kWindows: launches without groups have no windows at all, nor
// their shared memory.
template <int kSpan, bool kWindows, int kDirectUnroll, int kWindowUnroll, class Put>
__device__ __forceinline__ void exact_samples(const LightingBatch &B, const Frame32 &f,
                                              const float *horizon, int k0, int k1,
                                              bool windowed, float *window, const Put &put) {
    auto direction = [&](int k, float &azimuth_deg, float &elevation) {
        const int t = B.order ? __ldg(B.order + k) : B.time_start + k;
        const float *v = B.vectors + 3 * static_cast<size_t>(t);
        body_direction(f, __ldg(v), __ldg(v + 1), __ldg(v + 2), azimuth_deg, elevation);
        return t;
    };
    int first = 0, width = 0;
    if (kWindows && windowed && k0 < k1)
        width = stage_window<kSpan>(B, f, horizon, k0, k1, window, first);
    // One loop for the warp, the one that most of its lanes want.
    const unsigned lanes = __activemask();
    if (!kWindows || 2 * __popc(__ballot_sync(lanes, width > 0)) <= __popc(lanes)) {
#pragma unroll kDirectUnroll
        for (int k = k0; k < k1; ++k) {
            float azimuth_deg, elevation;
            const int t = direction(k, azimuth_deg, elevation);
            const BinPosition p = signal_position<kSpan>(azimuth_deg);
            put(t, signal_bins<kSpan>(GlobalBins{horizon, p.left}, p.fraction, elevation));
        }
        return;
    }
#pragma unroll kWindowUnroll
    for (int k = k0; k < k1; ++k) {
        float azimuth_deg, elevation;
        const int t = direction(k, azimuth_deg, elevation);
        const BinPosition p = signal_position<kSpan>(azimuth_deg);
        int offset = p.left - first;
        if (offset < 0) offset += kAzimuths;
        float signal;
        if (offset + kSpan <= width)
            signal = signal_bins<kSpan>(SharedBins{window, offset}, p.fraction, elevation);
        else
            signal = signal_bins<kSpan>(GlobalBins{horizon, p.left}, p.fraction, elevation);
        put(t, signal);
    }
}

// The steps of a block of an exact launch.  Short chunks hide the latency of
// the row reads; a window costs two directions and its bins, and pays from some
// 16 steps on that read the same bins.  So B.group chunks of B.chunk steps form
// a group: where its first and last vectors lie close together in longitude, the
// first of its blocks takes all of it with a window and the others end; where
// not, each takes its own chunk without one.  Close: as many bins as a window
// holds, and no more than the window saves (2 a step for the fraction, which
// reads 5; 0.75 for the margin, which reads 2).  Four patches, 355 steps of a
// year and of a day: fractions 461 and 360 us (a window tried in every chunk of
// 16: 469 and 358; chunks of 10 without windows: 433 and 487), margins 239 and
// 186 us (366 and 200; a window tried in every chunk of 10: 280 and 205).  Launches
// too small for groups take kernels without windows.
struct ExactSteps {
    int first, last;
    bool windowed;
};

template <int kSpan, bool kWindows>
__device__ __forceinline__ ExactSteps exact_steps(const LightingBatch &B) {
    const int y = blockIdx.y;
    if (!kWindows) return ExactSteps{y * B.chunk, min((y + 1) * B.chunk, B.time_count), false};
    // The first parts of all groups come first: they have the most to do.
    const int groups = gridDim.y / B.group, part = y / groups;
    const int g0 = (y - part * groups) * B.group * B.chunk;
    const int g1 = min(g0 + B.group * B.chunk, B.time_count);
    const float *a = B.vectors + 3 * static_cast<size_t>(__ldg(B.order + g0));
    const float *b = B.vectors + 3 * static_cast<size_t>(__ldg(B.order + g1 - 1));
    const float ax = __ldg(a), ay = __ldg(a + 1), bx = __ldg(b), by = __ldg(b + 1);
    const float bins = kSpan == 5 ? fminf(24.0f, 2.0f * (g1 - g0))
                                  : fminf(24.0f, 0.75f * (g1 - g0));
    // (A NaN, or vectors a quarter turn apart, is not close.)  0.25 deg a bin.
    if (fabsf(ax * by - ay * bx) <= 4.36e-3f * bins * (ax * bx + ay * by))
        return ExactSteps{g0, part ? g0 : g1, true};
    return ExactSteps{min(g0 + part * B.chunk, g1), min(g0 + (part + 1) * B.chunk, g1), false};
}

// Chunk length of an ordered launch with windows: a chunk of c steps sweeps
// about c * 1440 / T bins; keep that to 20 so its bins fit the window.
static int ordered_chunk(int chunk, int time_count) {
    return std::min(chunk, std::max(16, (kWindowBins - 12) * time_count / kAzimuths));
}

// Enough (pixel-block x chunk x tile) blocks for ~8 waves of 128-thread
// blocks on every SM, chunks of at least `least` time steps.
static int lighting_chunk(ls200_context *ctx, int tiles, int time_count, int least) {
    const int blocks_per_chunk = (kPatch * kPatch / 128) * tiles;
    const int want = ctx->props.multiProcessorCount * 16 * 8;
    int chunks = std::max(1, want / std::max(1, blocks_per_chunk));
    chunks = std::min(chunks, std::max(1, time_count / least));
    return (time_count + chunks - 1) / chunks;
}

// Sets the chunks of an exact launch and returns how many there are.  At least 4
// steps a chunk: a short table's launch is bound by the latency of its row reads
// (125 steps of one patch took 56 us in chunks of 16, 47 in chunks of 5: 32-byte
// sectors of 2 M rows).  Ordered launches take about 24 blocks per SM where that
// leaves shorter chunks than windows want, and groups of the latter's length;
// but none where the groups' first blocks alone would leave the chip idle (one
// patch, 125 steps of an hour: 76 us without, 79 with).
static int exact_chunks(ls200_context *ctx, LightingBatch &B, int tiles) {
    B.chunk = lighting_chunk(ctx, tiles, B.time_count, 4);
    B.group = 0;
    if (!B.order) return (B.time_count + B.chunk - 1) / B.chunk;
    const int blocks = (kPatch * kPatch / 128) * tiles, sms = ctx->props.multiProcessorCount;
    const int windowed = ordered_chunk(lighting_chunk(ctx, tiles, B.time_count, 16), B.time_count);
    const int chunks = std::max(1, sms * 24 / blocks);
    const int small = std::max(4, (B.time_count + chunks - 1) / chunks);
    if (static_cast<long long>(B.time_count / windowed) * blocks < sms * 8) {
        B.chunk = std::min(small, windowed);
        return (B.time_count + B.chunk - 1) / B.chunk;
    }
    const int parts = std::max(1, (windowed + small - 1) / small);
    B.chunk = (windowed + parts - 1) / parts;
    B.group = parts;
    const int steps = parts * B.chunk;
    return (B.time_count + steps - 1) / steps * parts;
}

// ---------------------------------------------------------------------------
// Ordered launches: settled samples.
//
// In longitude order a chunk of steps sees the body move through a narrow
// window of azimuths, and nearly every sample is clear: the whole disk (or the
// body's centre) stands well above the horizon around it, or well below.  For
// those the exact direction (two atan2f, a root: some 150 instructions) and the
// disk's 16 columns are not needed.  Each thread stages, per horizon bin of its
// pixel's window, the tangents of the elevation above which the signal is
// certainly high and below which it is certainly low; a step then rotates the
// vector into the window's own axes (10 multiply-adds), takes the bin from the
// sine of the angle to the window's middle and the tangent of the elevation
// from one reciprocal root, and compares: 30 instructions.  Samples in between
// (about 3 %) are collected per warp and evaluated by the exact functions, 32
// at a time.
//
// Margins: the approximate direction is within 4e-7 rad (2.3e-5 deg) of the
// exact one in both its own and the reference's rounding, for bodies at least
// 50 planet radii away.  (A table with a nearer one takes the exact kernels:
// four patches, a year of bytes of a body 20,000 km away 3.91 ms, 13.4 as
// undecided samples of the queue.)
// Near the vertical that error, relative to the whole vector, is not small
// against its horizontal part, and the azimuth is lost: a step settles only
// where the horizontal part exceeds a thousandth of the chunk's longest vector
// (below 89.94 deg: 0.1 bin).  A chunk with a vector whose square is beyond a
// float's range settles nothing.
// Taking the angle for its sine is 0.11 bin off at the window's end (8 deg).
// An entry therefore covers one bin more than a sample reads and is chosen half
// a bin low.  The elevations keep 1.2e-3 deg (kClear), of which the exact
// fraction needs 1e-3 to round to 0 or 1 and tan_degrees up to 4e-5.
constexpr int kEntries = 32;        // staged bins per pixel
constexpr int kEntryStride = kEntries + 1;
constexpr int kMaxChunk = 256;      // staged vectors per block
constexpr float kClear = 1.2e-3f;   // deg
constexpr float kBinsPerRadian = 229.1831180523293f;  // 1440 / 2 pi

// tan of an elevation in degrees from the fast sine and cosine (each within
// 5e-7): within 4e-5 deg of the angle.  Beyond 85 deg (a bin may hold any
// value) the tangent of 85, which entry_limits turns into no limit.
__device__ __forceinline__ float tan_degrees(float degrees) {
    const float x = fminf(fmaxf(degrees, -85.0f), 85.0f) * 0.017453292519943295f;
    return __fdividef(__sinf(x), __cosf(x));
}

// The limits of one entry: the highest tangent raised and the lowest lowered by
// a small angle, as halves rounded outwards (11 bits: 2^-10 covers them).
// `margin` is 1.02 times the angle (up to 0.28 deg): tan(x + m) - tan x =
// tan m (1 + tan^2 x) / (1 - tan x tan m), and up to tan x = 4 the factor is
// within 2 % of 1.
__device__ __forceinline__ __half2 entry_limits(float top, float bottom, float margin) {
    float high = __fmaf_rn(margin, __fmaf_rn(top, top, 1.0f), top);
    float low = __fmaf_rn(-margin, __fmaf_rn(bottom, bottom, 1.0f), bottom);
    high = fabsf(top) < 4.0f ? __fmaf_rn(fabsf(high), 0x1p-10f, high) : INFINITY;
    low = fabsf(bottom) < 4.0f ? __fmaf_rn(fabsf(low), -0x1p-10f, low) : -INFINITY;
    return __floats2half2_rn(high, low);
}

__device__ __forceinline__ float4 horizon_quad(const float *horizon, int bin) {
    if (bin < 0) bin += kAzimuths;
    else if (bin >= kAzimuths) bin -= kAzimuths;
    return __ldg(reinterpret_cast<const float4 *>(horizon + bin));
}

// One pixel's frame turned so that its first axis is across the window's
// middle azimuth and its second along it.
struct WindowAxes {
    float2 x, y, z, t;     // (across, along) per vector component, translation
    float ux, uy, uz, ut;  // up
    float position;        // of the middle, in entries
    float least;           // horizontal length that a settled step needs
};

// A step's vector as the packed arithmetic wants it: (x, x, y, y) and
// (z, z, the operation's two words).
struct StagedVector {
    float4 xy, zw;
    __device__ __forceinline__ uint2 words() const {
        return make_uint2(__float_as_uint(zw.z), __float_as_uint(zw.w));
    }
    __device__ __forceinline__ float3 vector() const { return make_float3(xy.x, xy.z, zw.x); }
};

// Sine of the angle from the window's middle and tangent of the elevation;
// returns whether the body is on the middle's side and far enough from the
// vertical.
__device__ __forceinline__ bool approximate_direction(const WindowAxes &w, const StagedVector &v,
                                                      float &sine, float &tangent) {
    float2 h = __ffma2_rn(make_float2(v.xy.x, v.xy.y), w.x, w.t);
    h = __ffma2_rn(make_float2(v.xy.z, v.xy.w), w.y, h);
    h = __ffma2_rn(make_float2(v.zw.x, v.zw.y), w.z, h);
    const float up = __fmaf_rn(v.zw.x, w.uz,
                               __fmaf_rn(v.xy.z, w.uy, __fmaf_rn(v.xy.x, w.ux, w.ut)));
    const float inverse = rsqrtf(__fmaf_rn(h.x, h.x, h.y * h.y));
    sine = h.x * inverse;
    tangent = up * inverse;
    return h.y > w.least;
}

// Shared memory of a staged launch's block.
struct StagedBlock {
    __half2 entries[128 * kEntryStride];   // (high above, low below)
    float4 vectors[2 * kMaxChunk];
    uint16_t queue[4][64];                 // undecided samples: step << 5 | lane
    unsigned longest;                      // bits of the largest squared length
    __device__ __forceinline__ StagedVector vector(int k) const {
        return StagedVector{vectors[2 * k], vectors[2 * k + 1]};
    }
};

// Stage the thread's entries for the block's `steps` vectors; returns their
// number.  A sample reads kSpan bins from bin
// azimuth * 4 - kSpan's offset on (5: the disk's columns, 2: the body's centre).
// The limits lie `clearance` (deg, small: see entry_limits) above the highest
// and below the lowest of them, all raised by `shift` (deg, any).
template <int kSpan>
__device__ __forceinline__ int stage_entries(StagedBlock &S, const Frame32 &f,
                                             const float *horizon, int steps, float shift,
                                             float clearance, WindowAxes &w) {
    const float3 middle = S.vector(steps >> 1).vector();
    float azimuth_deg, elevation;
    body_direction(f, middle.x, middle.y, middle.z, azimuth_deg, elevation);
    float sin_a = __fmaf_rn(middle.z, f.v[6], __fmaf_rn(middle.y, f.v[3],
                                                        __fmaf_rn(middle.x, f.v[0], f.v[9])));
    float cos_a = __fmaf_rn(middle.z, f.v[7], __fmaf_rn(middle.y, f.v[4],
                                                        __fmaf_rn(middle.x, f.v[1], f.v[10])));
    const float inverse = rsqrtf(__fmaf_rn(sin_a, sin_a, cos_a * cos_a));
    sin_a *= inverse;
    cos_a *= inverse;
    w.x = make_float2(f.v[0] * cos_a - f.v[1] * sin_a, f.v[0] * sin_a + f.v[1] * cos_a);
    w.y = make_float2(f.v[3] * cos_a - f.v[4] * sin_a, f.v[3] * sin_a + f.v[4] * cos_a);
    w.z = make_float2(f.v[6] * cos_a - f.v[7] * sin_a, f.v[6] * sin_a + f.v[7] * cos_a);
    w.t = make_float2(f.v[9] * cos_a - f.v[10] * sin_a, f.v[9] * sin_a + f.v[10] * cos_a);
    w.least = 1e-3f * sqrtf(__uint_as_float(S.longest));
    w.ux = f.v[2], w.uy = f.v[5], w.uz = f.v[8], w.ut = f.v[11];
    w.position = azimuth_deg * 4.0f - (kSpan == 5 ? 1.58f : 0.0f);
    float low = w.position, high = w.position;
#pragma unroll
    for (int end = 0; end < 2; ++end) {
        float sine, tangent;
        if (approximate_direction(w, S.vector(end ? steps - 1 : 0), sine, tangent) &&
            fabsf(sine) < 0.14f) {
            low = fminf(low, __fmaf_rn(sine, kBinsPerRadian, w.position));
            high = fmaxf(high, __fmaf_rn(sine, kBinsPerRadian, w.position));
        }
    }
    // Whole quads of bins from two below the lowest position; steps that fall
    // outside the entries are evaluated exactly.
    const int first = (static_cast<int>(floorf(low)) - 2) & ~3;
    const int count = min(kEntries, static_cast<int>(floorf(high)) + 3 - first);
    w.position -= static_cast<float>(first) + 0.5f;
    const float margin = 1.02f * 0.017453292519943295f * clearance;
    __half2 *entries = S.entries + threadIdx.x * kEntryStride;
    float bins[9];  // tangents of the horizon from entry e's bin on
    float sum = 0.0f;
    auto take = [&](int at, float4 h) {
        sum = (h.x + h.y) + (h.z + h.w);
        bins[at] = tan_degrees(h.x + shift);
        bins[at + 1] = tan_degrees(h.y + shift);
        bins[at + 2] = tan_degrees(h.z + shift);
        bins[at + 3] = tan_degrees(h.w + shift);
    };
    take(0, horizon_quad(horizon, first));
    float sum0 = sum;
    take(4, horizon_quad(horizon, first + 4));
    float sum1 = sum;
    float4 next = horizon_quad(horizon, first + 8);
    int bin0 = first < 0 ? first + kAzimuths : first;
    for (int e = 0; e < count; e += 4) {
        const float4 c = next;
        next = horizon_quad(horizon, first + e + 12);
        bins[8] = tan_degrees(c.x + shift);
        const float sum2 = (c.x + c.y) + (c.z + c.w);
        const bool finite = fabsf(sum0 + sum1 + sum2) < 1e6f;
        // The disk's first bin below azimuth 0.395 deg is special (its columns
        // extrapolate): bins 1437 to 1439 settle nothing.
        const bool seam = kSpan == 5 && bin0 == kAzimuths - 4;
        float most[8], least[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            most[k] = fmaxf(bins[k], bins[k + 1]);
            least[k] = fminf(bins[k], bins[k + 1]);
        }
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            float top, bottom;
            if (kSpan == 5) {  // bins k .. k + 5
                top = fmaxf(fmaxf(most[k], most[k + 2]), most[k + 4]);
                bottom = fminf(fminf(least[k], least[k + 2]), least[k + 4]);
            } else {           // bins k .. k + 2
                top = fmaxf(most[k], most[k + 1]);
                bottom = fminf(least[k], least[k + 1]);
            }
            __half2 limits = entry_limits(top, bottom, margin);
            if (!finite || (seam && k > 0)) limits = __floats2half2_rn(INFINITY, -INFINITY);
            entries[e + k] = limits;
        }
        sum0 = sum1;
        sum1 = sum2;
#pragma unroll
        for (int k = 0; k < 4; ++k) bins[k] = bins[k + 4];
        bins[4] = bins[8];
        bins[5] = tan_degrees(c.y + shift);
        bins[6] = tan_degrees(c.z + shift);
        bins[7] = tan_degrees(c.w + shift);
        bin0 = bin0 + 4 >= kAzimuths ? bin0 + 4 - kAzimuths : bin0 + 4;
    }
    return count;
}

// The block's vectors for positions [k0, k0 + steps) of the launch's order,
// with the operation's words for each time index.
template <class Op>
__device__ __forceinline__ void stage_vectors(StagedBlock &S, const LightingBatch &B, int k0,
                                              int steps, const Op &op) {
    if (threadIdx.x == 0) S.longest = 0u;
    __syncthreads();
    unsigned longest = 0u;  // positive floats order as their bits; NaN is above +inf
    for (int k = threadIdx.x; k < steps; k += blockDim.x) {
        const int t = __ldg(B.order + k0 + k);
        const float *v = B.vectors + 3 * static_cast<size_t>(t);
        const float x = __ldg(v), y = __ldg(v + 1), z = __ldg(v + 2);
        const uint2 words = op.words(t);
        S.vectors[2 * k] = make_float4(x, x, y, y);
        S.vectors[2 * k + 1] =
            make_float4(z, z, __uint_as_float(words.x), __uint_as_float(words.y));
        const float squared = x * x + y * y + z * z;
        longest = max(longest, __float_as_uint(squared < 1e38f ? squared : INFINITY));
    }
    longest = __reduce_max_sync(0xffffffffu, longest);
    if ((threadIdx.x & 31) == 0) atomicMax(&S.longest, longest);
    __syncthreads();
}

// Visits every sample of the block: op.settled(words, high) where the entries
// decide the thread's own pixel, op.outside(words) where that lies outside the
// valid rectangle (!valid), and op.put(pixel offset, signal, words) otherwise,
// for a pixel of the thread's warp.
template <int kSpan, class Op>
__device__ __forceinline__ void staged_samples(StagedBlock &S, const LightingBatch &B, bool valid,
                                               float shift, float clearance, Op &op) {
    const int lane = threadIdx.x & 31;
    const size_t pixel = static_cast<size_t>(blockIdx.z) * kPatch * kPatch +
                         blockIdx.x * 128 + threadIdx.x;
    uint16_t *queue = S.queue[threadIdx.x >> 5];
    const int k0 = blockIdx.y * B.chunk;
    const int steps = min(B.chunk, B.time_count - k0);
    stage_vectors(S, B, k0, steps, op);
    WindowAxes w{};
    int count = 0;
    if (valid)
        count = stage_entries<kSpan>(S, load_frame(B.frames, pixel),
                                     B.horizons + pixel * kAzimuths, steps, shift, clearance, w);
    const __half2 *entries = S.entries + threadIdx.x * kEntryStride;
    int pending = 0;  // queued samples of the warp
    for (int first = 0; first < steps; first += 32) {
        const int group = min(32, steps - first);
        uint32_t undecided = 0;  // of the group's steps
        if (valid) {
#pragma unroll 4
            for (int j = 0; j < group; ++j) {
                const StagedVector v = S.vector(first + j);
                float sine, tangent;
                const bool ahead = approximate_direction(w, v, sine, tangent);
                const int e = __float2int_rd(__fmaf_rn(sine, kBinsPerRadian, w.position));
                const bool staged =
                    static_cast<unsigned>(e) < static_cast<unsigned>(count) && ahead;
                float2 limits = make_float2(0.0f, 0.0f);
                if (staged) limits = __half22float2(entries[e]);
                const bool high = staged && tangent > limits.x;
                const bool low = staged && tangent < limits.y;
                if (high || low) op.settled(v.words(), high);
                else undecided |= 1u << j;
            }
        } else {
            for (int j = 0; j < group; ++j) op.outside(S.vector(first + j).words());
        }
        // Queue the undecided, one of each lane a round, and evaluate them
        // whenever a warp's worth (or, at the end, the rest) is there.
        const bool last = first + 32 >= steps;
        for (;;) {
            const unsigned from = __ballot_sync(0xffffffffu, undecided != 0);
            if (undecided) {
                const int j = __ffs(undecided) - 1;
                undecided &= undecided - 1;
                queue[pending + __popc(from & ((1u << lane) - 1u))] =
                    static_cast<uint16_t>((first + j) << 5 | lane);
            }
            pending += __popc(from);
            if (pending < 32 && (from || !last || !pending)) {
                if (!from) break;
                continue;
            }
            const int n = min(pending, 32);
            __syncwarp();
            if (lane < n) {
                const int entry = queue[lane];
                const int offset = (entry & 31) - lane;
                const StagedVector v = S.vector(entry >> 5);
                const float3 body = v.vector();
                float azimuth_deg, elevation;
                body_direction(load_frame(B.frames, pixel + offset), body.x, body.y, body.z,
                               azimuth_deg, elevation);
                const BinPosition p = signal_position<kSpan>(azimuth_deg);
                op.put(offset,
                       signal_bins<kSpan>(
                           GlobalBins{B.horizons + (pixel + offset) * kAzimuths, p.left},
                           p.fraction, elevation),
                       v.words());
            }
            __syncwarp();
            if (lane + n < pending) queue[lane] = queue[lane + n];
            pending -= n;
            __syncwarp();
        }
    }
}

// Sets the chunks of a staged launch, about 20 bins of azimuth, so that their
// entries fit, and returns how many there are.  Launches below kStagedSteps steps spend more on staging than
// they save: one patch takes 212 us against 342 at 720 steps, 236 either way
// at 360.
static int staged_chunks(LightingBatch &B) {
    B.chunk = std::max(4, std::min(kMaxChunk, static_cast<int>(20ll * B.time_count / kAzimuths)));
    return (B.time_count + B.chunk - 1) / B.chunk;
}
constexpr int kStagedSteps = 720;
// (Rows are staged in 16-byte quads, and a word plane's 32-bit offset bounds
// the bits' time axis to 2^22 steps.)
static bool staged_launch(const LightingBatch &B, int tiles) {
    double radius = 0.0;
    for (int t = 0; t < tiles; ++t) radius = std::max(radius, std::fabs(B.tiles[t].proj[0]));
    return B.order && B.time_count >= kStagedSteps && B.time_count < (1 << 22) &&
           (reinterpret_cast<uintptr_t>(B.horizons) & 15) == 0 &&
           B.shortest >= 50.0 * radius + 1.0;
}

// Fractions (float32 or bytes) into the launch's time-major output; the words
// of a step are its plane's 64-bit offset.  step() is the same by time index
// for the exact kernels.
template <class T>
struct StoreSample {
    T *out;  // the thread's pixel in the first plane
    int time_start;
    __device__ __forceinline__ uint2 words(int t) const {
        const unsigned long long offset =
            static_cast<unsigned long long>(t - time_start) * (kPatch * kPatch);
        return make_uint2(static_cast<unsigned>(offset), static_cast<unsigned>(offset >> 32));
    }
    __device__ __forceinline__ T *place(uint2 w) const {
        return out + (static_cast<unsigned long long>(w.y) << 32 | w.x);
    }
    static __device__ __forceinline__ T value(float visible) {
        return sizeof(T) == 1 ? static_cast<T>(static_cast<int>(__fmul_rn(255.0f, visible)))
                              : static_cast<T>(visible);
    }
    __device__ __forceinline__ void settled(uint2 w, bool high) const {
        *place(w) = high ? static_cast<T>(sizeof(T) == 1 ? 255 : 1) : static_cast<T>(0);
    }
    __device__ __forceinline__ void outside(uint2 w) const { *place(w) = static_cast<T>(0); }
    __device__ __forceinline__ void put(int offset, float signal, uint2 w) const {
        place(w)[offset] = value(signal);
    }
    __device__ __forceinline__ void step(int t, float signal) const {
        out[static_cast<size_t>(t - time_start) * (kPatch * kPatch)] = value(signal);
    }
};

// Blocks per SM of the staged kernels: 7 (72 registers) took 2.08 ms for four
// patches of a year's hourly bytes, 8 (64, a few spills) 2.13.
constexpr int kStagedBlocks = 7;

// Sun fractions of an ordered launch.  Four patches, 8761 steps, bytes (B200,
// whole call): 5.66 ms with the exact functions for every sample, 1.89 ms.  A
// warp's step takes 48 instructions with its share of exact samples (about 14),
// a chunk's staging 2300; 78 % of the issue slots are busy.
template <class T>
__global__ void __launch_bounds__(128, kStagedBlocks)
    staged_fraction_kernel(const __grid_constant__ LightingBatch B) {
    __shared__ StagedBlock S;
    const TileGeo &g = B.tiles[blockIdx.z];
    const int index = blockIdx.x * 128 + threadIdx.x;
    const bool valid = index % kPatch < g.valid_width && index / kPatch < g.valid_height;
    StoreSample<T> op{static_cast<T *>(B.out) +
                          static_cast<size_t>(blockIdx.z) * B.time_count * (kPatch * kPatch) +
                          index,
                      B.time_start};
    staged_samples<5>(S, B, valid, 0.0f, c_half_circle[7] + kClear, op);
}

// Margins, and fractions of launches that are not staged: every sample exactly.
template <int kSpan, class T, bool kWindows>
__global__ void __launch_bounds__(128) lighting_kernel(const __grid_constant__ LightingBatch B) {
    __shared__ float windows[kWindows ? 128 * kWindowStride : 1];
    const int tile = blockIdx.z;
    const int index = blockIdx.x * 128 + threadIdx.x;
    const TileGeo &g = B.tiles[tile];
    const ExactSteps steps = exact_steps<kSpan, kWindows>(B);
    const StoreSample<T> op{static_cast<T *>(B.out) +
                                static_cast<size_t>(tile) * B.time_count * (kPatch * kPatch) +
                                index,
                            B.time_start};
    if (index % kPatch >= g.valid_width || index / kPatch >= g.valid_height) {
        for (int k = steps.first; k < steps.last; ++k)
            op.step(B.order ? __ldg(B.order + k) : B.time_start + k, 0.0f);
        return;
    }
    const size_t pixel = static_cast<size_t>(tile) * kPatch * kPatch + index;
    exact_samples<kSpan, kWindows, kSpan == 2 ? 3 : 2, kSpan == 2 ? 4 : sizeof(T) == 1 ? 2 : 1>(
        B, load_frame(B.frames, pixel), B.horizons + pixel * kAzimuths, steps.first, steps.last,
        steps.windowed, windows + (kWindows ? threadIdx.x * kWindowStride : 0),
        [&](int t, float signal) { op.step(t, signal); });
}

// PSR (psr_cuda.py:57-186): 255 unless a reduced vector's centre rises above
// the interpolated horizon minus 0.545/2 deg.
__device__ __forceinline__ bool psr_lit(const Frame32 &f, const float *horizon, const float *v) {
    float azimuth_deg, elevation;
    body_direction(f, __ldg(v), __ldg(v + 1), __ldg(v + 2), azimuth_deg, elevation);
    float position = __fmul_rn(azimuth_deg, 4.0f);
    if (position >= static_cast<float>(kAzimuths)) position = 0.0f;
    const int lower = static_cast<int>(position);
    const float fraction = __fsub_rn(position, static_cast<float>(lower));
    const int upper = lower + 1 >= kAzimuths ? 0 : lower + 1;
    const float h1 = __ldg(horizon + lower), h2 = __ldg(horizon + upper);
    const float h = __fadd_rn(h1, __fmul_rn(fraction, __fsub_rn(h2, h1)));
    return __fsub_rn(elevation, h) > -0.2725f;
}

__device__ __forceinline__ bool psr_valid(const LightingBatch &B, int index) {
    const TileGeo &g = B.tiles[blockIdx.z];
    return index % kPatch < g.valid_width && index / kPatch < g.valid_height;
}

// One warp per pixel, a vector per lane, until any lane is lit.  The lanes'
// vectors lie a 32nd of the table apart, so each round looks in 32 directions and
// a lit pixel usually ends in the first rounds; a shadowed one takes count / 32
// rounds of the warp instead of `count` of one thread, which held its whole
// launch (four patches, 2100 vectors: 1388 us with a thread per pixel).
// kLooked: psr_look_kernel has run, and only the pixels it left dark are open.
constexpr int kPsrWarps = 8;

template <bool kLooked>
__global__ void __launch_bounds__(kPsrWarps * 32)
    psr_kernel(const __grid_constant__ LightingBatch B) {
    const int lane = threadIdx.x & 31;
    const int index = blockIdx.x * kPsrWarps + (threadIdx.x >> 5);
    const size_t pixel = static_cast<size_t>(blockIdx.z) * kPatch * kPatch + index;
    uint8_t *out = static_cast<uint8_t *>(B.out) + pixel;
    if (kLooked ? *out == 0 : !psr_valid(B, index)) {
        if (!kLooked && lane == 0) *out = 0;
        return;
    }
    const Frame32 f = load_frame(B.frames, pixel);
    const float *horizon = B.horizons + pixel * kAzimuths;
    const int rounds = (B.time_count + 31) / 32;
    for (int r = 0; r < rounds; ++r) {
        const int t = lane * rounds + r;
        const bool lit = t < B.time_count &&
                         psr_lit(f, horizon, B.vectors + 3 * static_cast<size_t>(t));
        if (__any_sync(0xffffffffu, lit)) {
            if (lane == 0) *out = 0;
            return;
        }
    }
    if (!kLooked && lane == 0) *out = 255;
}

// A look by one thread per pixel, at `looks` vectors spread over the table: all
// of a short table, or a first one, which decides most lit pixels of a launch
// whose warps would fill the chip several times.  Whole calls of four patches
// (with a thread per pixel throughout; with warps only): 100 vectors, lit
// 116 us (114; 129), dark 185 (228; 174); 8 vectors 129 (130; 140).
constexpr int kPsrLookTiles = 3;   // patches of a launch from which on it looks first
constexpr int kPsrShort = 16;      // table that it then looks at wholly
constexpr int kPsrLooks = 2;

__global__ void __launch_bounds__(128) psr_look_kernel(const __grid_constant__ LightingBatch B,
                                                       int looks) {
    const int index = blockIdx.x * 128 + threadIdx.x;
    const size_t pixel = static_cast<size_t>(blockIdx.z) * kPatch * kPatch + index;
    bool lit = !psr_valid(B, index);  // 0 outside the valid rectangle too
    if (!lit) {
        const Frame32 f = load_frame(B.frames, pixel);
        for (int i = 0; i < looks && !lit; ++i) {
            const int t = static_cast<int>(static_cast<long long>(B.time_count) * i / looks);
            lit = psr_lit(f, B.horizons + pixel * kAzimuths,
                          B.vectors + 3 * static_cast<size_t>(t));
        }
    }
    static_cast<uint8_t *>(B.out)[pixel] = lit ? 0 : 255;
}

static void psr_launch(ls200_context *ctx, const LightingBatch &B, int tiles) {
    const dim3 grid(kPatch * kPatch / kPsrWarps, 1, tiles);
    if (tiles < kPsrLookTiles) {
        psr_kernel<false><<<grid, kPsrWarps * 32, 0, ctx->stream>>>(B);
        return;
    }
    const int looks = B.time_count <= kPsrShort ? B.time_count : kPsrLooks;
    psr_look_kernel<<<dim3(kPatch * kPatch / 128, 1, tiles), 128, 0, ctx->stream>>>(B, looks);
    if (looks == B.time_count) return;
    LS_CUDA(cudaGetLastError());
    psr_kernel<true><<<grid, kPsrWarps * 32, 0, ctx->stream>>>(B);
}

// Diagnostic: sun fraction for given (azimuth, elevation) per horizon row
// (the reference's _sun_fraction_reference, lightmap.py:32-73).
__global__ void sun_fraction_kernel(const float *horizons, const float *azimuth_deg,
                                    const float *elevation_deg, int n, float *out) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    out[i] = sun_fraction(horizons + static_cast<size_t>(i) * kAzimuths, azimuth_deg[i],
                          elevation_deg[i]);
}

// The time indices of a table in longitude order, to a bin of 0.044 degrees (a
// sixth of a horizon bin: what the staged windows gain is the neighbourhood,
// and outputs do not depend on the order).  A counting sort in one block, the
// bins of the steps kept in `scratch` [count]; non-finite longitudes count as
// 0.  Creating and closing a table took a sort by atan2 on the host: 31 us for
// 125 vectors, 231 for 8,761, 677 for 26,281; now 28, 46 and 76.
constexpr int kOrderThreads = 1024;
constexpr int kOrderBins = 8192;

__global__ void __launch_bounds__(kOrderThreads) longitude_order_kernel(
    const float *__restrict__ vectors, int count, int *__restrict__ scratch,
    int *__restrict__ order) {
    constexpr int kPer = kOrderBins / kOrderThreads;
    __shared__ int bins[kOrderBins];
    __shared__ int warp_sums[32];
    for (int b = threadIdx.x; b < kOrderBins; b += kOrderThreads) bins[b] = 0;
    __syncthreads();
    for (int t = threadIdx.x; t < count; t += kOrderThreads) {
        const float *v = vectors + 3 * static_cast<size_t>(t);
        const float longitude = atan2f(v[1], v[0]);
        const float scaled =
            (isfinite(longitude) ? longitude : 0.0f) * (kOrderBins / 6.2831855f) + kOrderBins / 2;
        const int bin = min(max(static_cast<int>(scaled), 0), kOrderBins - 1);
        scratch[t] = bin;
        atomicAdd(&bins[bin], 1);
    }
    __syncthreads();
    // Exclusive sums: the thread's own bins, its warp, the block.
    const int lane = threadIdx.x & 31;
    int mine = 0;
#pragma unroll
    for (int j = 0; j < kPer; ++j) mine += bins[threadIdx.x * kPer + j];
    int sum = mine;
#pragma unroll
    for (int offset = 1; offset < 32; offset <<= 1) {
        const int add = __shfl_up_sync(0xffffffffu, sum, offset);
        if (lane >= offset) sum += add;
    }
    if (lane == 31) warp_sums[threadIdx.x >> 5] = sum;
    __syncthreads();
    int position = sum - mine;
    for (int w = 0; w < static_cast<int>(threadIdx.x >> 5); ++w) position += warp_sums[w];
#pragma unroll
    for (int j = 0; j < kPer; ++j) {
        const int n = bins[threadIdx.x * kPer + j];
        bins[threadIdx.x * kPer + j] = position;
        position += n;
    }
    __syncthreads();
    for (int t = threadIdx.x; t < count; t += kOrderThreads)
        order[atomicAdd(&bins[scratch[t]], 1)] = t;
}

cudaError_t longitude_order_launch(ls200_vectors *table) {
    longitude_order_kernel<<<1, kOrderThreads, 0, table->ctx->stream>>>(
        table->data, table->count, table->window, table->order);
    return cudaGetLastError();
}

// window = the entries of `order` inside [t0, t0 + n), in order: one block,
// each thread counting and then copying a contiguous run of `order` at the
// offset given by a block scan of the counts.

__global__ void __launch_bounds__(kOrderThreads) order_window_kernel(
    const int *__restrict__ order, int count, int t0, int n, int *__restrict__ window) {
    __shared__ int sums[kOrderThreads];
    const int per = (count + kOrderThreads - 1) / kOrderThreads;
    const int begin = min(count, static_cast<int>(threadIdx.x) * per);
    const int end = min(count, begin + per);
    int mine = 0;
    for (int k = begin; k < end; ++k) {
        const int t = order[k];
        mine += (t >= t0 && t < t0 + n) ? 1 : 0;
    }
    sums[threadIdx.x] = mine;
    __syncthreads();
    for (int offset = 1; offset < kOrderThreads; offset <<= 1) {
        const int add = threadIdx.x >= static_cast<unsigned>(offset) ? sums[threadIdx.x - offset]
                                                                     : 0;
        __syncthreads();
        sums[threadIdx.x] += add;
        __syncthreads();
    }
    int position = sums[threadIdx.x] - mine;
    for (int k = begin; k < end; ++k) {
        const int t = order[k];
        if (t >= t0 && t < t0 + n) window[position++] = t;
    }
}

void lighting_launch(ls200_context *ctx, LightingBatch &B, int tiles, int signal,
                     const ls200_vectors *table) {
    ensure_lighting_constants(ctx);
    B.order = nullptr;
    if (table && table->order && signal != kSignalPsr) {
        B.shortest = table->shortest;
        if (B.time_start == 0 && B.time_count == table->count) {
            B.order = table->order;
        } else {
            order_window_kernel<<<1, kOrderThreads, 0, ctx->stream>>>(
                table->order, table->count, B.time_start, B.time_count, table->window);
            LS_CUDA(cudaGetLastError());
            B.order = table->window;
        }
    }
    dim3 grid_frames(kPatch * kPatch / 128, tiles);
    frames_kernel<<<grid_frames, 128, 0, ctx->stream>>>(B);
    LS_CUDA(cudaGetLastError());
    if (signal == kSignalPsr) {
        psr_launch(ctx, B, tiles);
    } else if (signal != kSignalMargin && staged_launch(B, tiles)) {
        dim3 grid(kPatch * kPatch / 128, staged_chunks(B), tiles);
        if (signal == kSignalBytes)
            staged_fraction_kernel<uint8_t><<<grid, 128, 0, ctx->stream>>>(B);
        else
            staged_fraction_kernel<float><<<grid, 128, 0, ctx->stream>>>(B);
    } else {
        dim3 grid(kPatch * kPatch / 128, exact_chunks(ctx, B, tiles), tiles);
        const auto kernel = signal == kSignalFraction
                                ? (B.group ? lighting_kernel<5, float, true>
                                           : lighting_kernel<5, float, false>)
                            : signal == kSignalBytes
                                ? (B.group ? lighting_kernel<5, uint8_t, true>
                                           : lighting_kernel<5, uint8_t, false>)
                                : (B.group ? lighting_kernel<2, float, true>
                                           : lighting_kernel<2, float, false>);
        kernel<<<grid, 128, 0, ctx->stream>>>(B);
    }
    LS_CUDA(cudaGetLastError());
}

__global__ void __launch_bounds__(128) directions_kernel(const __grid_constant__ LightingBatch B,
                                                         float2 *__restrict__ out) {
    const int tile = blockIdx.z;
    const int index = blockIdx.x * blockDim.x + threadIdx.x;
    if (index >= kPatch * kPatch) return;
    const TileGeo &g = B.tiles[tile];
    const int sample = index % kPatch, line = index / kPatch;
    const int t0 = B.time_start + blockIdx.y * B.chunk;
    const int t1 = min(t0 + B.chunk, B.time_start + B.time_count);
    const size_t plane = static_cast<size_t>(kPatch) * kPatch;
    const size_t tile_out = static_cast<size_t>(tile) * B.time_count * plane;
    const bool valid = sample < g.valid_width && line < g.valid_height;
    Frame32 f;
    const float *src = B.frames + (static_cast<size_t>(tile) * plane + index) * 12;
#pragma unroll
    for (int k = 0; k < 12; ++k) f.v[k] = src[k];
    for (int t = t0; t < t1; ++t) {
        float2 direction = make_float2(0.0f, 0.0f);
        if (valid) {
            const float *v = B.vectors + 3 * static_cast<size_t>(t);
            body_direction(f, __ldg(v), __ldg(v + 1), __ldg(v + 2), direction.x, direction.y);
        }
        out[tile_out + static_cast<size_t>(t - B.time_start) * plane + index] = direction;
    }
}

void directions_launch(ls200_context *ctx, LightingBatch &B, int tiles, float2 *out) {
    LS_REQUIRE(tiles >= 1 && tiles <= kMaxBatchTiles, "1 to 32 tiles per launch");
    dim3 grid_frames(kPatch * kPatch / 128, tiles);
    frames_kernel<<<grid_frames, 128, 0, ctx->stream>>>(B);
    LS_CUDA(cudaGetLastError());
    B.chunk = lighting_chunk(ctx, tiles, B.time_count, 4);
    dim3 grid(kPatch * kPatch / 128, (B.time_count + B.chunk - 1) / B.chunk, tiles);
    directions_kernel<<<grid, 128, 0, ctx->stream>>>(B, out);
    LS_CUDA(cudaGetLastError());
}

// Threshold bits of one signal of one body, word-major [tiles, words, 16384]
// (zeroed before the launch): bit t is set where signal >= threshold
// (kAtLeast) or signal < threshold.  kSpan 5 is the sun fraction, 2 the
// margin.  Each thread visits a chunk of the body's table in its longitude
// order and sets the bits of its steps with atomicOr (other chunks own the
// word's other steps).  Each signal runs in its own body's order.
template <bool kAtLeast>
__device__ __forceinline__ bool passes(float value, float threshold) {
    return kAtLeast ? value >= threshold : value < threshold;
}

// The words of a step: the offset of its word's plane, and its bit.
template <int kSpan, bool kAtLeast>
struct SetBit {
    uint32_t *bits;  // the thread's pixel in the first word plane
    float threshold;
    bool high, low;  // the bit of a settled high or low signal
    __device__ __forceinline__ uint2 words(int t) const {
        return make_uint2(static_cast<unsigned>(t >> 5) * (kPatch * kPatch), 1u << (t & 31));
    }
    __device__ __forceinline__ void settled(uint2 w, bool is_high) const {
        if (is_high ? high : low) atomicOr(bits + w.x, w.y);
    }
    __device__ __forceinline__ void outside(uint2) const {}
    __device__ __forceinline__ void put(int offset, float signal, uint2 w) const {
        if (passes<kAtLeast>(signal, threshold)) atomicOr(bits + offset + w.x, w.y);
    }
    __device__ __forceinline__ void step(int t, float signal) const {
        if (passes<kAtLeast>(signal, threshold))
            atomicOr(bits + static_cast<size_t>(t >> 5) * (kPatch * kPatch), 1u << (t & 31));
    }
};

template <int kSpan, bool kAtLeast>
__global__ void __launch_bounds__(128, kStagedBlocks)
    staged_bits_kernel(const __grid_constant__ LightingBatch B, float threshold, int words,
                       uint32_t *__restrict__ bits) {
    __shared__ StagedBlock S;
    const TileGeo &g = B.tiles[blockIdx.z];
    const int index = blockIdx.x * 128 + threadIdx.x;
    const bool valid = index % kPatch < g.valid_width && index / kPatch < g.valid_height;
    // A settled margin is above or below the threshold itself.
    SetBit<kSpan, kAtLeast> op{
        bits + static_cast<size_t>(blockIdx.z) * words * (kPatch * kPatch) + index, threshold,
        kSpan == 5 ? passes<kAtLeast>(1.0f, threshold) : kAtLeast,
        kSpan == 5 ? passes<kAtLeast>(0.0f, threshold) : !kAtLeast};
    staged_samples<kSpan>(S, B, valid, kSpan == 5 ? 0.0f : threshold,
                          kSpan == 5 ? c_half_circle[7] + kClear : kClear, op);
}

// The same without an order, or for a short table: every sample exactly.
template <int kSpan, bool kAtLeast, bool kWindows>
__global__ void __launch_bounds__(128) signal_bits_kernel(const __grid_constant__ LightingBatch B,
                                                          float threshold, int words,
                                                          uint32_t *__restrict__ bits) {
    __shared__ float windows[kWindows ? 128 * kWindowStride : 1];
    const int index = blockIdx.x * 128 + threadIdx.x;
    const TileGeo &g = B.tiles[blockIdx.z];
    if (index % kPatch >= g.valid_width || index / kPatch >= g.valid_height) return;
    const size_t pixel = static_cast<size_t>(blockIdx.z) * kPatch * kPatch + index;
    const SetBit<kSpan, kAtLeast> op{
        bits + static_cast<size_t>(blockIdx.z) * words * (kPatch * kPatch) + index, threshold,
        false, false};
    const ExactSteps steps = exact_steps<kSpan, kWindows>(B);
    exact_samples<kSpan, kWindows, kSpan == 2 ? 3 : 1, kSpan == 2 ? 4 : 1>(
        B, load_frame(B.frames, pixel), B.horizons + pixel * kAzimuths, steps.first, steps.last,
        steps.windowed, windows + (kWindows ? threadIdx.x * kWindowStride : 0),
        [&](int t, float signal) { op.step(t, signal); });
}

// Zero `bits` ([tiles, words, 16384] words) and set the threshold bits of
// one signal of `body`, whose table replaces the batch's vectors; the frames are
// already in place.
template <int kSpan, bool kAtLeast>
static void signal_bits_launch(ls200_context *ctx, LightingBatch B, int tiles,
                               const ls200_vectors *body, float threshold, int words,
                               uint32_t *bits) {
    LS_CUDA(cudaMemsetAsync(bits, 0,
                            sizeof(uint32_t) * static_cast<size_t>(tiles) * words * kPatch * kPatch,
                            ctx->stream));
    B.vectors = body->data;
    B.order = body->order;
    B.shortest = body->shortest;
    const bool staged = staged_launch(B, tiles);
    dim3 grid(kPatch * kPatch / 128,
              staged ? staged_chunks(B) : exact_chunks(ctx, B, tiles), tiles);
    if (staged)
        staged_bits_kernel<kSpan, kAtLeast>
            <<<grid, 128, 0, ctx->stream>>>(B, threshold, words, bits);
    else if (B.group)
        signal_bits_kernel<kSpan, kAtLeast, true>
            <<<grid, 128, 0, ctx->stream>>>(B, threshold, words, bits);
    else
        signal_bits_kernel<kSpan, kAtLeast, false>
            <<<grid, 128, 0, ctx->stream>>>(B, threshold, words, bits);
    LS_CUDA(cudaGetLastError());
}

// Longest right-censored candidate run per start interval
// (nh/mission_duration.py:212-256), one thread per pixel over the bits.  For
// a run of true samples [rs, re] and a start window [ws, we) the candidate
// starts at max(rs, ws) when that lies in the window and accrues every
// sample's duration through re; the answer per interval is the maximum over
// runs.  Durations are summed in sample order in FP64 as the reference does
// (or read from exact prefix sums when every sample duration is an integer).
// The bits are read a word at a time, eight words in flight, and only run
// starts and ends are visited (a bit per step: 1981 us for two patches, one
// year hourly, 12 windows).
constexpr int kMaxDurationIntervals = 64;

struct DurationParams {
    const uint32_t *bits;        // [tiles, words, 16384] sun fraction >= threshold
    const uint32_t *earth_bits;  // the same for Earth margin >= threshold, or NULL
    const double *hours;   // [T] sample durations
    const double *prefix;  // [T + 1] exact prefix sums, or NULL
    const int2 *windows;   // [I] (first, end) sample indices of each start window
    float *out;            // [tiles, I, 16384]
    int words, time_count, interval_count, tiles, days;
    int2 valid[kMaxBatchTiles];
};

__device__ __forceinline__ double run_hours(const DurationParams &P, int first, int last) {
    if (P.prefix) return P.prefix[last + 1] - P.prefix[first];
    double sum = 0.0;
    for (int t = first; t <= last; ++t) sum += P.hours[t];
    return sum;
}

// Start windows of one thread: their maxima stay in registers, and a product
// with more windows has more threads per pixel.
constexpr int kThreadIntervals = 4;

__global__ void __launch_bounds__(128) duration_kernel(const __grid_constant__ DurationParams P) {
    const int tile = blockIdx.y;
    const int index = blockIdx.x * blockDim.x + threadIdx.x;
    if (index >= kPatch * kPatch) return;
    const size_t plane = static_cast<size_t>(kPatch) * kPatch;
    const int interval0 = blockIdx.z * kThreadIntervals;
    double longest[kThreadIntervals] = {};
    int2 window[kThreadIntervals];
#pragma unroll
    for (int i = 0; i < kThreadIntervals; ++i)  // an empty window for none
        window[i] = interval0 + i < P.interval_count ? P.windows[interval0 + i] : make_int2(0, 0);
    const bool valid =
        index % kPatch < P.valid[tile].x && index / kPatch < P.valid[tile].y;
    if (valid) {
        // Word-major bits: word w of this pixel at row[w * plane].  The
        // condition is the Sun bit, and with Earth vectors also the Earth bit.
        const size_t offset = static_cast<size_t>(tile) * P.words * plane + index;
        const uint32_t *row = P.bits + offset;
        const uint32_t *earth_row = P.earth_bits ? P.earth_bits + offset : nullptr;
        int run_start = -1;
        auto end_run = [&](int run_end) {
#pragma unroll
            for (int i = 0; i < kThreadIntervals; ++i) {
                const int first = max(run_start, window[i].x);
                if (first >= window[i].y || first > run_end) continue;
                const double d = run_hours(P, first, run_end);
                if (d > longest[i]) longest[i] = d;
            }
            run_start = -1;
        };
        // Whole words: only the bits where a run starts or ends are visited
        // (bits at and beyond time_count are zero and end the last run).
        constexpr int kAhead = 8;  // words loaded together
        for (int w0 = 0; w0 < P.words; w0 += kAhead) {
            uint32_t words[kAhead];
#pragma unroll
            for (int j = 0; j < kAhead; ++j) {
                const size_t at = static_cast<size_t>(w0 + j) * plane;
                words[j] = w0 + j < P.words ? __ldg(row + at) : 0u;
                if (earth_row && w0 + j < P.words) words[j] &= __ldg(earth_row + at);
            }
#pragma unroll
            for (int j = 0; j < kAhead; ++j) {
                if (w0 + j >= P.words) break;
                const int t0 = (w0 + j) * 32;
                // Bits that differ from the one before them.
                uint32_t edges = words[j] ^ ((words[j] << 1) | (run_start >= 0 ? 1u : 0u));
                while (edges) {
                    const int bit = __ffs(edges) - 1;
                    edges &= edges - 1;
                    if (run_start < 0) run_start = t0 + bit;
                    else end_run(t0 + bit - 1);
                }
            }
        }
        if (run_start >= 0) end_run(P.time_count - 1);
    }
#pragma unroll
    for (int i = 0; i < kThreadIntervals; ++i) {
        if (interval0 + i >= P.interval_count) break;
        const double v = P.days ? longest[i] / 24.0 : longest[i];
        P.out[(static_cast<size_t>(tile) * P.interval_count + interval0 + i) * plane + index] =
            static_cast<float>(v);
    }
}

void mission_duration_launch(ls200_context *ctx, LightingBatch &B, int tiles,
                             const ls200_vectors *sun, const ls200_vectors *earth,
                             float sun_threshold, float earth_threshold, uint32_t *bits,
                             const double *hours, const double *prefix, const int2 *windows,
                             int interval_count, bool days, float *out) {
    LS_REQUIRE(tiles >= 1 && tiles <= kMaxBatchTiles, "1 to 32 tiles per launch");
    LS_REQUIRE(interval_count >= 1 && interval_count <= kMaxDurationIntervals,
               "1 to 64 start intervals");
    ensure_lighting_constants(ctx);
    dim3 grid_frames(kPatch * kPatch / 128, tiles);
    frames_kernel<<<grid_frames, 128, 0, ctx->stream>>>(B);
    LS_CUDA(cudaGetLastError());
    const int words = (B.time_count + 31) / 32;
    const size_t stream_words = static_cast<size_t>(tiles) * words * kPatch * kPatch;
    signal_bits_launch<5, true>(ctx, B, tiles, sun, sun_threshold, words, bits);
    if (earth)
        signal_bits_launch<2, true>(ctx, B, tiles, earth, earth_threshold, words,
                                    bits + stream_words);
    DurationParams P{};
    P.bits = bits;
    P.earth_bits = earth ? bits + stream_words : nullptr;
    P.hours = hours;
    P.prefix = prefix;
    P.windows = windows;
    P.out = out;
    P.words = words;
    P.time_count = B.time_count;
    P.interval_count = interval_count;
    P.tiles = tiles;
    P.days = days ? 1 : 0;
    for (int t = 0; t < tiles; ++t)
        P.valid[t] = make_int2(B.tiles[t].valid_width, B.tiles[t].valid_height);
    const int groups = (interval_count + kThreadIntervals - 1) / kThreadIntervals;
    duration_kernel<<<dim3(kPatch * kPatch / 128, tiles, groups), 128, 0, ctx->stream>>>(P);
    LS_CUDA(cudaGetLastError());
}

// Per-pixel safe-haven reducer (safe_haven.py:75-243), one thread per pixel
// over the condition bits in time order.  The reference credits a low-Sun run
// to every month band in which one of its samples saw an Earth outage, with
// the run's length at each of its samples; run lengths only grow, so the
// credit equals the run's final (or right-censored) length, applied once
// when the run ends.  Per band the scratch holds the longest credited run and
// flags 1 (an outage sample), 2 (a sample without outage), 4 (the current run
// touched this band); the flags of the band in use are gathered in a
// register and stored when the band changes or a run ends.  Output: band
// hours = float32(longest) * float32(time_step_hours), NaN where the band saw
// no outage or nothing else (safe_haven.py:231-240) and outside the valid
// rectangle.
//
// The bits are taken a word at a time: the warp splits a word where the month
// changes (the months are the same for every pixel), and within a part only
// the ends of low-Sun runs are visited.  One step at a time was a chain of 25
// instructions for each sample of a pixel; the scratch, a chain of memory
// latencies at each run's end, is touched only where a run or the bits cross
// into another month (kernel, two tiles, 17,545 hours: 420 us,
// 485 with every run's end in memory).
struct HavenParams {
    const uint32_t *low, *outage;  // [tiles, words, 16384]
    const int *month;              // [T] band of each time step, -1 for none
    int *longest;                  // [tiles, bands, 16384] scratch
    uint8_t *flags;                // [tiles, bands, 16384] scratch
    float *out;                    // [tiles, bands, 16384]
    float hours;
    int words, time_count, bands;
    int2 valid[kMaxBatchTiles];
};

__global__ void __launch_bounds__(128) haven_kernel(const __grid_constant__ HavenParams P) {
    const int tile = blockIdx.y;
    const int index = blockIdx.x * blockDim.x + threadIdx.x;
    if (index >= kPatch * kPatch) return;
    const size_t plane = static_cast<size_t>(kPatch) * kPatch;
    const size_t band0 = static_cast<size_t>(tile) * P.bands * plane + index;
    int *longest = P.longest + band0;
    uint8_t *flags = P.flags + band0;
    float *out = P.out + band0;
    const bool valid = index % kPatch < P.valid[tile].x && index / kPatch < P.valid[tile].y;
    if (!valid) {
        for (int b = 0; b < P.bands; ++b) out[b * plane] = __int_as_float(0x7fffffff);
    }
    // The other lanes of the warp stay for the votes on the months.
    if (!__any_sync(0xffffffffu, valid)) return;
    if (valid) {
        for (int b = 0; b < P.bands; ++b) {
            longest[b * plane] = 0;
            flags[b * plane] = 0;
        }
    }
    int run = 0;
    int lo = P.bands, hi = -1;       // bands the current run touched lie in [lo, hi]
    int cached = -1;                 // band whose flags sit in `bits`
    unsigned bits = 0u;
    int top = 0;                     // longest credit of that band not yet in `longest`
    bool spread = false;             // a stored band's flag 4 is set
    auto store = [&]() {
        if (cached >= 0) {
            if (bits) flags[cached * plane] |= static_cast<uint8_t>(bits);
            if (top) longest[cached * plane] = max(longest[cached * plane], top);
            spread = spread || (bits & 4u);
        }
        bits = 0u;
        top = 0;
    };
    auto credit = [&]() {
        if (!spread) {  // a run inside one month: all of it in registers
            top = max(top, run);
            bits &= ~4u;
        } else {
            store();
            for (int b = lo; b <= hi; ++b) {
                const unsigned f = flags[b * plane];
                if (f & 4u) {
                    longest[b * plane] = max(longest[b * plane], run);
                    flags[b * plane] = static_cast<uint8_t>(f & ~4u);
                }
            }
            spread = false;
        }
        lo = P.bands;
        hi = -1;
    };
    // Samples [first, last) of a word, all of month m.
    auto part = [&](uint32_t low_word, uint32_t outage_word, int first, int last, int m) {
        const uint32_t mask = (0xffffffffu >> (32 - last)) & (0xffffffffu << first);
        const uint32_t high = ~low_word & mask;
        uint32_t touches = 0u;  // samples that credit their run to the band
        if (m >= 0) {
            if (m != cached) {
                store();
                cached = m;
            }
            bits |= ((outage_word & mask) ? 1u : 0u) | ((~outage_word & mask) ? 2u : 0u);
            touches = low_word & outage_word & mask;
        }
        auto touch = [&](uint32_t run_mask) {
            if (touches & run_mask) {
                bits |= 4u;
                lo = min(lo, m);
                hi = max(hi, m);
            }
        };
        int from = first;  // every sample of the part below it is done
        uint32_t left = high;
        while (left) {
            const int end = __ffs(left) - 1;  // the run, if any, is [.., end)
            run += end - from;
            touch((1u << end) - (1u << from));
            if (hi >= 0) credit();
            run = 0;
            const uint32_t lows = low_word & mask & (0xffffffffu << end);
            if (!lows) return;
            from = __ffs(lows) - 1;
            left = high & (0xffffffffu << from);
        }
        run += last - from;
        touch(mask & (0xffffffffu << from));
    };
    const int lane = threadIdx.x & 31;
    const size_t word0 = static_cast<size_t>(tile) * P.words * plane + index;
    constexpr int kAhead = 4;  // words loaded together
    for (int w0 = 0; w0 < P.words; w0 += kAhead) {
        uint32_t low_words[kAhead], outage_words[kAhead];
        int months[kAhead];
#pragma unroll
        for (int j = 0; j < kAhead; ++j) {
            const int w = min(w0 + j, P.words - 1);
            low_words[j] = __ldg(P.low + word0 + w * plane);
            outage_words[j] = __ldg(P.outage + word0 + w * plane);
            months[j] = __ldg(P.month + min(w * 32 + lane, P.time_count - 1));
        }
#pragma unroll
        for (int j = 0; j < kAhead; ++j) {
            if (w0 + j >= P.words) break;
            const int steps = min(32, P.time_count - (w0 + j) * 32);
            for (int first = 0; first < steps;) {
                const int m = __shfl_sync(0xffffffffu, months[j], first);
                const uint32_t others =
                    __ballot_sync(0xffffffffu, months[j] != m) & (0xffffffffu << first);
                const int last = others ? min(__ffs(others) - 1, steps) : steps;
                if (valid) part(low_words[j], outage_words[j], first, last, m);
                first = last;
            }
        }
    }
    if (!valid) return;
    if (hi >= 0) credit();  // the run still open at the end is right-censored
    store();
    for (int b = 0; b < P.bands; ++b) {
        const unsigned f = flags[b * plane];
        out[b * plane] = (f & 3u) == 3u
                             ? __fmul_rn(__int2float_rn(longest[b * plane]), P.hours)
                             : __int_as_float(0x7fffffff);
    }
}

void safe_haven_launch(ls200_context *ctx, LightingBatch &B, int tiles,
                       const ls200_vectors *sun, const ls200_vectors *earth,
                       float sunlight_threshold, float earth_threshold, uint32_t *bits,
                       const int *month, int bands, float hours, int *longest, uint8_t *flags,
                       float *out) {
    LS_REQUIRE(tiles >= 1 && tiles <= kMaxBatchTiles, "1 to 32 tiles per launch");
    ensure_lighting_constants(ctx);
    dim3 grid_frames(kPatch * kPatch / 128, tiles);
    frames_kernel<<<grid_frames, 128, 0, ctx->stream>>>(B);
    LS_CUDA(cudaGetLastError());
    const int words = (B.time_count + 31) / 32;
    const size_t stream_words = static_cast<size_t>(tiles) * words * kPatch * kPatch;
    // Low Sun (fraction < threshold) in the Sun's order, Earth outage
    // (margin < threshold) in the Earth's (safe_haven.py:156-160).
    signal_bits_launch<5, false>(ctx, B, tiles, sun, sunlight_threshold, words, bits);
    signal_bits_launch<2, false>(ctx, B, tiles, earth, earth_threshold, words,
                                 bits + stream_words);
    HavenParams P{};
    P.low = bits;
    P.outage = bits + stream_words;
    P.month = month;
    P.longest = longest;
    P.flags = flags;
    P.out = out;
    P.hours = hours;
    P.words = words;
    P.time_count = B.time_count;
    P.bands = bands;
    for (int t = 0; t < tiles; ++t)
        P.valid[t] = make_int2(B.tiles[t].valid_width, B.tiles[t].valid_height);
    haven_kernel<<<dim3(kPatch * kPatch / 128, tiles), 128, 0, ctx->stream>>>(P);
    LS_CUDA(cudaGetLastError());
}

// Earth-visibility fraction: per pixel, the share of time steps whose Earth
// margin (the a13 signal of lighting_kernel, lightmap_cpu.py:121-141) is >=
// threshold.  Each thread counts its pixel over one time chunk and adds the
// count to the pixel's counter; visibility_finalize divides by T (FP64, then
// rounded to float32).
struct CountVisible {
    unsigned *counts;  // the thread's pixel
    float threshold;
    unsigned count;
    __device__ __forceinline__ uint2 words(int) const { return make_uint2(0u, 0u); }
    __device__ __forceinline__ void settled(uint2, bool high) { count += high ? 1u : 0u; }
    __device__ __forceinline__ void outside(uint2) const {}
    __device__ __forceinline__ void put(int offset, float signal, uint2) const {
        if (signal >= threshold) atomicAdd(counts + offset, 1u);
    }
    __device__ __forceinline__ void step(int, float signal) {
        count += signal >= threshold ? 1u : 0u;
    }
};

__global__ void __launch_bounds__(128, kStagedBlocks)
    staged_visibility_kernel(const __grid_constant__ LightingBatch B, float threshold,
                             unsigned *__restrict__ counts) {
    __shared__ StagedBlock S;
    const TileGeo &g = B.tiles[blockIdx.z];
    const int index = blockIdx.x * 128 + threadIdx.x;
    const bool valid = index % kPatch < g.valid_width && index / kPatch < g.valid_height;
    CountVisible op{counts + static_cast<size_t>(blockIdx.z) * (kPatch * kPatch) + index,
                    threshold, 0u};
    staged_samples<2>(S, B, valid, threshold, kClear, op);
    if (op.count) atomicAdd(op.counts, op.count);
}

// The same without an order, or for a short table: every sample exactly.
template <bool kWindows>
__global__ void __launch_bounds__(128) visibility_kernel(const __grid_constant__ LightingBatch B,
                                                         float threshold,
                                                         unsigned *__restrict__ counts) {
    __shared__ float windows[kWindows ? 128 * kWindowStride : 1];
    const int index = blockIdx.x * 128 + threadIdx.x;
    const TileGeo &g = B.tiles[blockIdx.z];
    if (index % kPatch >= g.valid_width || index / kPatch >= g.valid_height) return;
    const size_t pixel = static_cast<size_t>(blockIdx.z) * kPatch * kPatch + index;
    CountVisible op{counts + pixel, threshold, 0u};
    const ExactSteps steps = exact_steps<2, kWindows>(B);
    exact_samples<2, kWindows, 3, 4>(
        B, load_frame(B.frames, pixel), B.horizons + pixel * kAzimuths, steps.first, steps.last,
        steps.windowed, windows + (kWindows ? threadIdx.x * kWindowStride : 0),
        [&](int t, float signal) { op.step(t, signal); });
    if (op.count) atomicAdd(op.counts, op.count);
}

__global__ void visibility_finalize(const unsigned *__restrict__ counts, int n, int time_count,
                                    const int2 *__restrict__ valid, float *__restrict__ out) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int tile = i / (kPatch * kPatch), index = i % (kPatch * kPatch);
    const bool inside = index % kPatch < valid[tile].x && index / kPatch < valid[tile].y;
    out[i] = inside ? static_cast<float>(static_cast<double>(counts[i]) / time_count)
                    : __int_as_float(0x7fffffff);
}

void visibility_launch(ls200_context *ctx, LightingBatch &B, int tiles,
                       const ls200_vectors *earth, float threshold, unsigned *counts,
                       int2 *valid, float *out) {
    LS_REQUIRE(tiles >= 1 && tiles <= kMaxBatchTiles, "1 to 32 tiles per launch");
    ensure_lighting_constants(ctx);
    B.order = earth->order;
    B.shortest = earth->shortest;
    const int n = tiles * kPatch * kPatch;
    LS_CUDA(cudaMemsetAsync(counts, 0, sizeof(unsigned) * n, ctx->stream));
    dim3 grid_frames(kPatch * kPatch / 128, tiles);
    frames_kernel<<<grid_frames, 128, 0, ctx->stream>>>(B);
    LS_CUDA(cudaGetLastError());
    const bool staged = staged_launch(B, tiles);
    dim3 grid(kPatch * kPatch / 128,
              staged ? staged_chunks(B) : exact_chunks(ctx, B, tiles), tiles);
    if (staged)
        staged_visibility_kernel<<<grid, 128, 0, ctx->stream>>>(B, threshold, counts);
    else if (B.group)
        visibility_kernel<true><<<grid, 128, 0, ctx->stream>>>(B, threshold, counts);
    else
        visibility_kernel<false><<<grid, 128, 0, ctx->stream>>>(B, threshold, counts);
    LS_CUDA(cudaGetLastError());
    visibility_finalize<<<(n + 255) / 256, 256, 0, ctx->stream>>>(counts, n, B.time_count, valid,
                                                                  out);
    LS_CUDA(cudaGetLastError());
}

void sun_fraction_launch(ls200_context *ctx, const float *horizons, const float *azimuth_deg,
                         const float *elevation_deg, int n, float *out) {
    ensure_lighting_constants(ctx);
    sun_fraction_kernel<<<(n + 127) / 128, 128, 0, ctx->stream>>>(horizons, azimuth_deg,
                                                                  elevation_deg, n, out);
    LS_CUDA(cudaGetLastError());
}

}  // namespace ls200

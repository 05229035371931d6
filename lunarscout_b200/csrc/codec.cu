// Horizon tile codec (.cbin) on the device.
//
// Format (src/lunarscout/_numba_horizon/file_format.py:39-73, 135-182): for
// each of the 16384 pixels of a tile, a little-endian u16 block length, then
// the block: the first sample quantised to a big-endian i16, then one delta
// per sample — 7 bits (one byte) when -64 <= d < 63, else 15 bits in two
// bytes with the top bit set.  Samples are degrees clamped to [-50, 50] and
// quantised as round-half-away(float32(value) * float32(32767)/float32(50));
// -inf (pixels outside the DEM) encodes as -50.
//
// Encoding: one warp per pixel.  Its 1440 samples are read in 45 coalesced
// groups of 32; a sample's delta needs only its left neighbour's quantised
// value, and its byte offset is a ballot count of the two-byte deltas before
// it, so the row needs no serial walk.  (Only a jump of more than 15 bits is
// clamped and carries into the samples after it: a group takes its jumps one
// after another.  Whole call, a tile of noise 346 us and one with a gap in every
// row 94; 919 and 898 when such a row was walked by one lane.)  The block is
// built in shared memory and leaves as 16-byte words into a fixed slot; a scan
// turns lengths into offsets and a copy kernel packs [length][block] records,
// again one warp per pixel in whole words.
// Decoding: the host walks the 16384 length prefixes (validating structure);
// one warp per pixel expands its block 32 bytes at a time, see decode_kernel.
// One thread per pixel left the chip idle: 438 us to encode, 546 us to decode
// a tile on a B200.  Now encode, scan and pack take 41 + 8 + 12 us (the encode
// kernel 2.3 TB/s of reads, bound by its instructions: 45 groups x ~35 per
// warp) and decode 99 us.
#include "staging.cuh"

#include <vector>

namespace ls200 {

constexpr int kCodecPixels = 128 * 128;
constexpr int kCodecSamples = 1440;
constexpr int kMaxBlock = 2 * kCodecSamples;

constexpr int kCodecWarps = 8;   // pixels per block
constexpr int kSlot = 2880 + 32;  // slot bytes: 16-byte aligned, room for whole words

__device__ __forceinline__ int quantize(float degrees, float short_scale) {
    // NaN never reaches the encoder.
    float v = degrees < 50.0f ? degrees : 50.0f;
    v = v > -50.0f ? v : -50.0f;
    // Round half away from zero: below 2^23 the fraction is exact.
    const float scaled = __fmul_rn(v, short_scale);
    const float whole = truncf(scaled);
    int q = static_cast<int>(whole);
    if (fabsf(scaled - whole) >= 0.5f) q += scaled >= 0.0f ? 1 : -1;
    return q > 32767 ? 32767 : (q < -32767 ? -32767 : q);
}

// The two bytes a delta is stored as; one byte when -64 <= delta < 63.
__device__ __forceinline__ bool wide_delta(int delta) { return delta < -64 || delta >= 63; }

__global__ void __launch_bounds__(kCodecWarps * 32)
    encode_kernel(const float *__restrict__ degrees, float short_scale,
                  uint8_t *__restrict__ slots, int *__restrict__ lengths) {
    __shared__ __align__(16) uint8_t blocks[kCodecWarps][kSlot];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int pixel = blockIdx.x * kCodecWarps + warp;
    const float *row = degrees + static_cast<size_t>(pixel) * kCodecSamples;
    uint8_t *out = blocks[warp];
    const unsigned below = (1u << lane) - 1u;
    int n = 1;         // bytes so far (the same in every lane)
    int previous = 0;  // last stored value of the group before
    constexpr int kGroups = kCodecSamples / 32, kBatch = 9;
    static_assert(kGroups % kBatch == 0, "whole batches of groups");
    for (int first = 0; first < kGroups; first += kBatch) {
        float values[kBatch];
#pragma unroll
        for (int j = 0; j < kBatch; ++j) values[j] = __ldg(row + (first + j) * 32 + lane);
#pragma unroll
        for (int j = 0; j < kBatch; ++j) {
            int value = quantize(values[j], short_scale);
            int left = __shfl_up_sync(0xffffffffu, value, 1);
            if (lane == 0) left = previous;
            int delta = value - left;
            // The first sample itself (byte 0 and 1) goes in as a one-byte
            // delta at byte 1, overwritten below.
            if (j == 0 && first == 0 && lane == 0) delta = 0;
            // Jumps of more than 15 bits, in order: what is stored falls short
            // of the sample, and the next one's delta starts from there.
            for (;;) {
                const unsigned jumps =
                    __ballot_sync(0xffffffffu, delta < -16384 || delta > 16383);
                if (!jumps) break;
                const int at = __ffs(jumps) - 1;
                if (lane == at) {
                    delta = delta < 0 ? -16384 : 16383;
                    value = left + delta;
                }
                left = __shfl_sync(0xffffffffu, value, at);
                if (lane == at + 1) delta = value - left;
                else left = value - delta;
            }
            previous = __shfl_sync(0xffffffffu, value, 31);
            const bool wide = wide_delta(delta);
            const unsigned wides = __ballot_sync(0xffffffffu, wide);
            const int at = n + lane + __popc(wides & below);
            out[at] = static_cast<uint8_t>(wide ? (delta >> 8) | 0x80 : delta & 0x7F);
            if (wide) out[at + 1] = static_cast<uint8_t>(delta);
            n += 32 + __popc(wides);
        }
    }
    if (lane == 0) {
        const int q = quantize(__ldg(row), short_scale);
        out[0] = static_cast<uint8_t>(q >> 8);
        out[1] = static_cast<uint8_t>(q);
    }
    __syncwarp();
    uint4 *slot = reinterpret_cast<uint4 *>(slots + static_cast<size_t>(pixel) * kSlot);
    for (int i = lane; i * 16 < n; i += 32) slot[i] = reinterpret_cast<const uint4 *>(out)[i];
    if (lane == 0) lengths[pixel] = n;
}

// Exclusive scan of (2 + length) over the 16384 pixels in one block of 1024
// threads: thread t takes pixels 16t .. 16t + 15 (four 16-byte loads), warp
// sums by shuffles, then the 32 warp totals; plus the total.
__global__ void __launch_bounds__(1024) scan_kernel(const int *__restrict__ lengths,
                                                    long long *__restrict__ offsets,
                                                    long long *__restrict__ total) {
    __shared__ int warp_sums[32];
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    int local[16];  // 16384 records of at most 2882 bytes fit an int
    int sum = 0;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int4 v = reinterpret_cast<const int4 *>(lengths)[t * 4 + i];
        local[4 * i] = sum, sum += 2 + v.x;
        local[4 * i + 1] = sum, sum += 2 + v.y;
        local[4 * i + 2] = sum, sum += 2 + v.z;
        local[4 * i + 3] = sum, sum += 2 + v.w;
    }
    int inclusive = sum;
#pragma unroll
    for (int offset = 1; offset < 32; offset <<= 1) {
        const int add = __shfl_up_sync(0xffffffffu, inclusive, offset);
        if (lane >= offset) inclusive += add;
    }
    if (lane == 31) warp_sums[warp] = inclusive;
    __syncthreads();
    int before = inclusive - sum;
    for (int w = 0; w < warp; ++w) before += warp_sums[w];
    longlong2 *out = reinterpret_cast<longlong2 *>(offsets + t * 16);
#pragma unroll
    for (int i = 0; i < 8; ++i)
        out[i] = make_longlong2(before + local[2 * i], before + local[2 * i + 1]);
    if (t == 1023) *total = before + sum;
}

// One warp copies a record [length][block] to its byte offset in the payload:
// whole 4-byte words of the destination (each from two words of the slot,
// shifted into place), the bytes of a word shared with a neighbour one by one.
__global__ void __launch_bounds__(kCodecWarps * 32)
    pack_kernel(const uint8_t *__restrict__ slots, const int *__restrict__ lengths,
                const long long *__restrict__ offsets, uint8_t *__restrict__ payload) {
    const int lane = threadIdx.x & 31;
    const int pixel = blockIdx.x * kCodecWarps + (threadIdx.x >> 5);
    const int n = lengths[pixel];
    const uint8_t *src = slots + static_cast<size_t>(pixel) * kSlot;
    uint8_t *dst = payload + offsets[pixel];
    if (lane < 2) dst[lane] = static_cast<uint8_t>(n >> (8 * lane));
    dst += 2;
    // Bytes before the first aligned word of dst.
    const int head = min(n, static_cast<int>(-reinterpret_cast<uintptr_t>(dst) & 3));
    if (lane < head) dst[lane] = src[lane];
    const int words = (n - head) >> 2;
    const uint32_t *from = reinterpret_cast<const uint32_t *>(src);
    uint32_t *to = reinterpret_cast<uint32_t *>(dst + head);
    for (int w = lane; w < words; w += 32)
        to[w] = __funnelshift_r(from[w], from[w + 1], 8 * head);
    const int done = head + 4 * words;
    if (lane < n - done) dst[done + lane] = src[done + lane];
}

// One warp per pixel, 32 bytes of the block at a time.  Which bytes start a
// delta: after a byte without its top bit the next one does; in a run of bytes
// with the top bit set, starts and second bytes alternate.  So a byte is a
// second byte when the run of top-bit bytes just before it is odd, which one
// ballot tells.  Starts are numbered by a ballot count and the deltas summed
// by a warp scan (modulo 2^16, as the format wraps).
__global__ void __launch_bounds__(kCodecWarps * 32)
    decode_kernel(const uint8_t *__restrict__ payload, const long long *__restrict__ block_start,
                  const int *__restrict__ lengths, float elevation_scale,
                  float *__restrict__ degrees, int *__restrict__ error) {
    const int lane = threadIdx.x & 31;
    const int pixel = blockIdx.x * kCodecWarps + (threadIdx.x >> 5);
    const uint8_t *p = payload + block_start[pixel];
    const int n = lengths[pixel];
    float *row = degrees + static_cast<size_t>(pixel) * kCodecSamples;
    int value = static_cast<int16_t>((static_cast<int>(p[0]) << 8) | p[1]);
    if (lane == 0) row[0] = __fmul_rn(static_cast<float>(value), elevation_scale);
    int k = 1;            // samples written
    unsigned odd = 0;     // 1: the group before ended in a start with a second byte to come
    bool complete = true;
    int next = 2 + lane < n ? p[2 + lane] : 0;
    for (int offset = 2; offset < n; offset += 32) {
        const bool inside = offset + lane < n;
        const int byte = next;
        next = offset + 32 + lane < n ? p[offset + 32 + lane] : 0;
        int after = __shfl_down_sync(0xffffffffu, byte, 1);
        const int follow = __shfl_sync(0xffffffffu, next, 0);
        if (lane == 31) after = follow;
        const unsigned top = __ballot_sync(0xffffffffu, inside && (byte & 0x80));
        // Top-bit bytes in the run just below this lane; a run that reaches the
        // group's start continues the one before it.
        const unsigned below = (1u << lane) - 1u;
        const int run = __clz(~((top << 1) << (31 - lane)));
        const bool second = (run + (run == lane ? odd : 0u)) & 1u;
        const bool start = inside && !second;
        const bool wide = start && (byte & 0x80);
        int delta = 0;
        if (wide) {
            const int high = ((byte << 1) & 0x80) | (byte & 0x7F);
            delta = static_cast<int16_t>((high << 8) | after);
            if (offset + lane + 1 >= n) complete = false;
        } else if (start) {
            delta = byte & 0x7F;
            if (delta & 0x40) delta -= 0x80;
        }
        int sum = delta;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const int add = __shfl_up_sync(0xffffffffu, sum, d);
            if (lane >= d) sum += add;
        }
        const unsigned starts = __ballot_sync(0xffffffffu, start);
        const int index = k + __popc(starts & below);
        if (start && index < kCodecSamples)
            row[index] = __fmul_rn(static_cast<float>(static_cast<int16_t>(value + sum)),
                                   elevation_scale);
        value += __shfl_sync(0xffffffffu, sum, 31);
        k += __popc(starts);
        odd = __shfl_sync(0xffffffffu, wide ? 1u : 0u, 31);
    }
    const bool whole = __all_sync(0xffffffffu, complete);
    if (lane == 0 && (k != kCodecSamples || !whole)) atomicExch(error, pixel + 1);
}

static float short_scale() { return 32767.0f / 50.0f; }
static float elevation_scale() { return 50.0f / 32767.0f; }

struct CodecBuffers {
    DeviceBuffer slots, lengths, offsets, total, payload, degrees, error;
    StagedCopies staged;
};

static CodecBuffers &codec_buffers(ls200_context *ctx) {
    if (!ctx->codec) ctx->codec = new CodecBuffers();
    return *ctx->codec;
}

void release_codec(ls200_context *ctx) {
    delete ctx->codec;
    ctx->codec = nullptr;
}

// Encode device degrees [16384, 1440] into device `payload` (capacity at
// least 16384 * 2882); returns the payload size (synchronises).
int64_t cbin_encode(ls200_context *ctx, const float *degrees, uint8_t *payload) {
    CodecBuffers &b = codec_buffers(ctx);
    b.slots.reserve(size_t(kCodecPixels) * kSlot);
    b.lengths.reserve(sizeof(int) * kCodecPixels);
    b.offsets.reserve(sizeof(long long) * kCodecPixels);
    b.total.reserve(sizeof(long long));
    encode_kernel<<<kCodecPixels / kCodecWarps, kCodecWarps * 32, 0, ctx->stream>>>(
        degrees, short_scale(), b.slots.as<uint8_t>(), b.lengths.as<int>());
    LS_CUDA(cudaGetLastError());
    scan_kernel<<<1, 1024, 0, ctx->stream>>>(b.lengths.as<int>(), b.offsets.as<long long>(),
                                             b.total.as<long long>());
    LS_CUDA(cudaGetLastError());
    pack_kernel<<<kCodecPixels / kCodecWarps, kCodecWarps * 32, 0, ctx->stream>>>(
        b.slots.as<uint8_t>(), b.lengths.as<int>(), b.offsets.as<long long>(), payload);
    LS_CUDA(cudaGetLastError());
    long long total = 0;
    LS_CUDA(cudaMemcpyAsync(&total, b.total.ptr, sizeof total, cudaMemcpyDeviceToHost,
                            ctx->stream));
    LS_CUDA(cudaStreamSynchronize(ctx->stream));
    return total;
}

}  // namespace ls200

using namespace ls200;

extern "C" {

ls200_status ls200_cbin_encode_device(ls200_context *ctx, const float *device_degrees,
                                      uint8_t *device_payload, int64_t *size) {
    return guard([&] {
        LS_REQUIRE(ctx && device_degrees && device_payload && size, "NULL argument");
        std::lock_guard<std::mutex> hold(ctx->lock);
        activate(ctx);
        *size = cbin_encode(ctx, device_degrees, device_payload);
    });
}

ls200_status ls200_cbin_encode(ls200_context *ctx, const float *degrees, uint8_t *payload,
                               int64_t capacity, int64_t *size) {
    return guard([&] {
        LS_REQUIRE(ctx && degrees && payload && size, "NULL argument");
        LS_REQUIRE(capacity >= int64_t(kCodecPixels) * (kMaxBlock + 2),
                   "payload capacity must be at least 16384 * 2882 bytes");
        std::lock_guard<std::mutex> hold(ctx->lock);
        activate(ctx);
        CodecBuffers &b = codec_buffers(ctx);
        const size_t n = sizeof(float) * size_t(kCodecPixels) * kCodecSamples;
        b.degrees.reserve(n);
        b.payload.reserve(size_t(kCodecPixels) * (kMaxBlock + 2));
        LS_CUDA(cudaMemcpyAsync(b.degrees.ptr, degrees, n, cudaMemcpyHostToDevice, ctx->stream));
        const int64_t total = cbin_encode(ctx, b.degrees.as<float>(), b.payload.as<uint8_t>());
        LS_CUDA(cudaMemcpyAsync(payload, b.payload.ptr, size_t(total), cudaMemcpyDeviceToHost,
                                ctx->stream));
        LS_CUDA(cudaStreamSynchronize(ctx->stream));
        *size = total;
    });
}

ls200_status ls200_cbin_decode(ls200_context *ctx, const uint8_t *payload, int64_t size,
                               float *degrees) {
    return guard([&] {
        LS_REQUIRE(ctx && payload && degrees && size >= 0, "invalid arguments");
        // Structure (file_format.py:135-182): 16384 records, each a u16 LE
        // length in [2, 2880] followed by that many bytes, and no trailing
        // bytes.
        std::vector<long long> starts(kCodecPixels);
        std::vector<int> lengths(kCodecPixels);
        long long offset = 0;
        for (int p = 0; p < kCodecPixels; ++p) {
            LS_REQUIRE(offset + 2 <= size, "compressed horizon ended while reading a block length");
            const int length = payload[offset] | (payload[offset + 1] << 8);
            offset += 2;
            LS_REQUIRE(length >= 2 && length <= kMaxBlock, "compressed horizon block length is invalid");
            LS_REQUIRE(offset + length <= size, "compressed horizon ended inside a block");
            starts[p] = offset;
            lengths[p] = length;
            offset += length;
        }
        LS_REQUIRE(offset == size, "compressed horizon contains trailing bytes");
        std::lock_guard<std::mutex> hold(ctx->lock);
        activate(ctx);
        CodecBuffers &b = codec_buffers(ctx);
        const size_t n = sizeof(float) * size_t(kCodecPixels) * kCodecSamples;
        b.payload.reserve(size_t(size) > 0 ? size_t(size) : 1);
        b.offsets.reserve(sizeof(long long) * kCodecPixels);
        b.lengths.reserve(sizeof(int) * kCodecPixels);
        b.degrees.reserve(n);
        b.error.reserve(sizeof(int));
        b.staged.to_device(ctx->device, b.payload.ptr, payload, size_t(size), ctx->stream);
        LS_CUDA(cudaMemcpyAsync(b.offsets.ptr, starts.data(), sizeof(long long) * kCodecPixels,
                                cudaMemcpyHostToDevice, ctx->stream));
        LS_CUDA(cudaMemcpyAsync(b.lengths.ptr, lengths.data(), sizeof(int) * kCodecPixels,
                                cudaMemcpyHostToDevice, ctx->stream));
        LS_CUDA(cudaMemsetAsync(b.error.ptr, 0, sizeof(int), ctx->stream));
        decode_kernel<<<kCodecPixels / kCodecWarps, kCodecWarps * 32, 0, ctx->stream>>>(
            b.payload.as<uint8_t>(), b.offsets.as<long long>(), b.lengths.as<int>(),
            elevation_scale(), b.degrees.as<float>(), b.error.as<int>());
        LS_CUDA(cudaGetLastError());
        int error = 0;
        LS_CUDA(cudaMemcpyAsync(&error, b.error.ptr, sizeof error, cudaMemcpyDeviceToHost,
                                ctx->stream));
        b.staged.to_host(ctx->device, degrees, b.degrees.ptr, n, ctx->stream);
        LS_CUDA(cudaStreamSynchronize(ctx->stream));
        LS_REQUIRE(error == 0, "compressed horizon block did not decode to 1440 samples");
    });
}

}  // extern "C"

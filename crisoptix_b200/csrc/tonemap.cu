// tonemap.cu -- ToneMapping (src/kernel/tonemap.cu:23-39, called once per
// frame from src/main.cpp:127): linear float RGB to sRGB bytes.
//
// The byte of one channel is srgb8(c) (rt_common.cuh): the reference's curve
// in the reference's own arithmetic.  It is 0 for NaN, for negative c and for
// c above c_max (where 12.92 c overflows and the blend turns NaN), and on
// [0, c_max] a non-decreasing step function of c with 255 steps: every float
// operation in it rounds monotonically, and the power is the correctly
// rounded one except within 1e-14 of a rounding midpoint, far below the 5e-8
// relative gap between the powers of neighbouring floats.  So the kernel does
// not evaluate the curve, which costs about ninety double-precision
// operations per channel and would make this copy-shaped kernel FP64-bound.
// The host finds, once, the smallest float T[k] with srgb8(T[k]) >= k for
// k = 1..255 by bisection over float bit patterns, checks both sides of every
// step, and files the steps into 1665 buckets of float bit patterns (one
// exponent and 7 leading mantissa bits each) so that no bucket holds more
// than one step.  A bucket stores the byte at its start and the bit pattern of
// its step's offset; the kernel copies the buckets to shared memory and finds a
// channel's byte with one bucket load and one integer compare
// (srgb8_lookup).  The bytes are the formula's by construction.
//
// Memory: 12 bytes read and 3 written per pixel.  Each thread takes four
// pixels (three 16-byte loads, three 4-byte stores) when both pointers are
// aligned for that, and the ragged tail pixel by pixel.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <mutex>
#include <stdexcept>
#include <utility>
#include <vector>

#include "context.h"
#include "device_memory.h"
#include "passes.cuh"

namespace crisb {
namespace {

constexpr int kToneBlock = 512;

// Buckets of float bit patterns: bucket i (1 <= i < kBuckets) holds the
// patterns [kBucketBase + (i << kBucketShift), kBucketBase + ((i + 1) <<
// kBucketShift)), i.e. one exponent and 7 leading mantissa bits between
// 2^-12 and 2; bucket 0 also holds everything below, bucket kBuckets
// everything from 2 up to c_max.
constexpr uint32_t kBucketShift = 16;                  // 23 - 7 mantissa bits
constexpr uint32_t kBucketBase = (127u - 12u) << 23;   // 2^-12
constexpr uint32_t kBuckets = 13u << (23 - kBucketShift);  // 2^-12 .. 2

struct SrgbTable {
    float t[256];  // t[0] = 0; t[k] smallest float c >= 0 with srgb8(c) >= k
    float c_max;   // largest float c with 12.92f * c finite
    // per bucket: the byte at its first pattern and the bit pattern of the
    // next step above it (0xffffffff for byte 255)
    uint2 bucket[kBuckets + 1];
};

float bits_to_float(uint32_t b) {
    float f;
    memcpy(&f, &b, sizeof f);
    return f;
}
uint32_t float_bits(float f) {
    uint32_t b;
    memcpy(&b, &f, sizeof b);
    return b;
}

SrgbTable build_srgb_table() {
    SrgbTable tab{};
    // c_max: largest float with a finite 12.92f * c (positive floats order as
    // their bit patterns)
    uint32_t lo = 0, hi = 0x7f7fffffu;  // 12.92 * 0 finite; FLT_MAX * 12.92 not
    while (hi - lo > 1) {
        const uint32_t mid = lo + (hi - lo) / 2;
        if (std::isinf(12.92f * bits_to_float(mid)))
            hi = mid;
        else
            lo = mid;
    }
    tab.c_max = bits_to_float(lo);
    const uint32_t max_bits = lo;
    if (srgb8(tab.c_max) != 255) throw std::runtime_error("sRGB table: byte below c_max is not 255");
    if (srgb8(0.0f) != 0) throw std::runtime_error("sRGB table: byte of 0 is not 0");
    tab.t[0] = 0.0f;
    uint32_t tb[257];
    tb[0] = 0;
    for (uint32_t k = 1; k < 256; ++k) {
        uint32_t a = 0, b = max_bits;  // srgb8(a) < k <= srgb8(b)
        while (b - a > 1) {
            const uint32_t mid = a + (b - a) / 2;
            if (srgb8(bits_to_float(mid)) >= k)
                b = mid;
            else
                a = mid;
        }
        tab.t[k] = bits_to_float(b);
        tb[k] = b;
        if (srgb8(tab.t[k]) < k || srgb8(bits_to_float(b - 1)) >= k || tab.t[k] < tab.t[k - 1])
            throw std::runtime_error("sRGB table: step check failed");
    }
    tb[256] = 0xffffffffu;
    // byte of pattern x (0 <= x <= max_bits): steps at or below x
    auto count = [&](uint32_t x) {
        uint32_t k = 0;
        while (k < 255 && tb[k + 1] <= x) ++k;
        return k;
    };
    if (tb[1] < kBucketBase + (1u << kBucketShift) || tb[255] >= kBucketBase + (kBuckets << kBucketShift))
        throw std::runtime_error("sRGB table: steps outside the bucketed range");
    for (uint32_t i = 0; i <= kBuckets; ++i) {
        const uint32_t first = i == 0 ? 0u : kBucketBase + (i << kBucketShift);
        const uint32_t last = i == kBuckets ? max_bits : kBucketBase + ((i + 1) << kBucketShift) - 1;
        const uint32_t b0 = count(first);
        if (count(last) > b0 + 1) throw std::runtime_error("sRGB table: two steps in one bucket");
        tab.bucket[i] = make_uint2(b0, tb[b0 + 1]);
    }
    return tab;
}

const SrgbTable& srgb_table() {
    static const SrgbTable tab = build_srgb_table();
    return tab;
}

// A bucket as the kernel reads it, 4 bytes: bits 24-31 the byte at the bucket's
// start, bits 0-16 its step's offset in the bucket (0x10000: no step)
constexpr uint32_t kNoStep = 0x10000u;

// Byte of a channel from its bit pattern: 0 for negative (sign bit set), NaN
// and values above c_max (patterns above c_max's); otherwise the byte at the
// start of the bucket, plus one if the bucket's single step is at or below it.
// (Bucket 0, which also takes every value below the first, has no step, nor has
// the last one, which takes every value from 2 up.)
RT_D uint32_t srgb8_lookup(const uint32_t* bucket, float c, uint32_t max_bits) {
    const uint32_t x = __float_as_uint(c);
    const uint32_t y = max(x, kBucketBase) - kBucketBase;
    const uint32_t e = bucket[min(y >> kBucketShift, kBuckets)];
    const uint32_t v = (e >> 24) + ((y & 0xffffu) >= (e & 0x1ffffu) ? 1u : 0u);
    return x > max_bits ? 0u : v;
}

RT_D uint32_t srgb8_word(const uint32_t* bucket, float4 v, uint32_t max_bits) {
    return srgb8_lookup(bucket, v.x, max_bits) | srgb8_lookup(bucket, v.y, max_bits) << 8 |
           srgb8_lookup(bucket, v.z, max_bits) << 16 | srgb8_lookup(bucket, v.w, max_bits) << 24;
}

// streaming load that stays behind the wait for the work before the kernel
RT_D float4 ld_image(const float4* p) {
    float4 v;
    asm volatile("ld.global.cs.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p));
    return v;
}

// kVec: pixels [0, 4 * quads) four per thread with vector accesses (rgb 16-byte and
// out 4-byte aligned), a thread's next pixels loaded before its present ones are
// stored, and the last few one per thread.  Else pixels one by one, kTurns of a
// thread's loaded before they are stored, in a kernel of its own: the registers of the
// vector loop would leave it 3 instead of 4 blocks of 512 threads per SM, and with
// that and a pixel at a time 33.2 million unaligned pixels took 151 us, now 95.  What
// bounds it: launch and
// table load for small images, memory for large ones (3840x3840: 221 MB in 36 us,
// 6.1 TB/s).  Launched beside the end of the work before it (launch_tonemap_srgb8), a
// block copies the table, which never changes, before it waits for that work; the
// wait comes before the first access to the caller's memory.  4-byte instead of
// 8-byte buckets halve the table and the bank conflicts of its random reads.  Work
// that still runs at the kernel's start may write the image, so no load of it goes
// through the read-only path (no __restrict__) or may move above the wait.
// Back to back, before and after: 1920x1080 12.4 -> 9.4 us (the host's launch rate;
// 12.1 without the early launch), 3840x2160 28.7 -> 22.1, 3840x3840 45.1 -> 36.2.
template <bool kVec>
__global__ void __launch_bounds__(kToneBlock) k_tonemap_srgb8(const float* rgb, uint8_t* out, uint32_t n,
                                                             uint32_t quads, const uint32_t* table,
                                                             uint32_t max_bits) {
    __shared__ uint32_t t[kBuckets + 1];
    const uint32_t stride = gridDim.x * blockDim.x;
    const uint32_t tid = blockIdx.x * blockDim.x + threadIdx.x;
    asm volatile("griddepcontrol.launch_dependents;");
    for (uint32_t i = threadIdx.x; i <= kBuckets; i += blockDim.x) t[i] = __ldg(table + i);
    asm volatile("griddepcontrol.wait;" ::: "memory");
    if (kVec) {
        const float4* in4 = reinterpret_cast<const float4*>(rgb);
        uint32_t* out4 = reinterpret_cast<uint32_t*>(out);
        uint64_t q = tid;
        float4 a, b, c;
        if (q < quads) {
            a = ld_image(in4 + 3 * q);
            b = ld_image(in4 + 3 * q + 1);
            c = ld_image(in4 + 3 * q + 2);
        }
        __syncthreads();
        while (q < quads) {
            const uint64_t next = q + stride;
            float4 na, nb, nc;
            if (next < quads) {
                na = ld_image(in4 + 3 * next);
                nb = ld_image(in4 + 3 * next + 1);
                nc = ld_image(in4 + 3 * next + 2);
            }
            __stcs(out4 + 3 * q, srgb8_word(t, a, max_bits));
            __stcs(out4 + 3 * q + 1, srgb8_word(t, b, max_bits));
            __stcs(out4 + 3 * q + 2, srgb8_word(t, c, max_bits));
            a = na;
            b = nb;
            c = nc;
            q = next;
        }
        const uint64_t i = 4 * static_cast<uint64_t>(quads) + tid;
        if (i < n)
            for (int ch = 0; ch < 3; ++ch)
                out[3 * i + ch] = static_cast<uint8_t>(srgb8_lookup(t, rgb[3 * i + ch], max_bits));
    } else {
        constexpr uint64_t kTurns = 4;
        __syncthreads();
        for (uint64_t i = tid; i < n; i += kTurns * stride) {
            float v[kTurns][3];
#pragma unroll
            for (uint64_t k = 0; k < kTurns; ++k) {
                const uint64_t p = i + k * stride;
                if (p < n)
                    for (int ch = 0; ch < 3; ++ch) v[k][ch] = rgb[3 * p + ch];
            }
#pragma unroll
            for (uint64_t k = 0; k < kTurns; ++k) {
                const uint64_t p = i + k * stride;
                if (p < n)
                    for (int ch = 0; ch < 3; ++ch)
                        out[3 * p + ch] = static_cast<uint8_t>(srgb8_lookup(t, v[k][ch], max_bits));
            }
        }
    }
}

// the buckets as the kernel reads them
std::vector<uint32_t> bucket_words(const SrgbTable& tab) {
    std::vector<uint32_t> w(kBuckets + 1);
    for (uint32_t i = 0; i <= kBuckets; ++i) {
        const uint32_t lo = kBucketBase + (i << kBucketShift);
        uint32_t step = kNoStep;
        if (tab.bucket[i].y >= lo && tab.bucket[i].y - lo < kNoStep) step = tab.bucket[i].y - lo;
        if (tab.bucket[i].x > 255u || (step != kNoStep && (i == 0 || i == kBuckets)))
            throw std::runtime_error("sRGB table: a step outside the buckets");
        w[i] = (tab.bucket[i].x << 24) | step;
    }
    return w;
}

// the bucket table in device memory, uploaded once per CUDA context (7 KB)
// and kept for the life of that context: no handle owns it, and a table freed
// while a caller's stream still runs a tone-mapping kernel would be read after
// free.  Keyed by context id (context.h), so a context created after a
// cudaDeviceReset, or a caller's own context, gets a table of its own.
const uint32_t* device_table() {
    static std::mutex mu;
    static std::vector<std::pair<unsigned long long, const uint32_t*>> tables;
    unsigned long long ctx = 0;
    if (current_context_id(&ctx) != cudaSuccess) throw std::runtime_error("no current CUDA context");
    std::lock_guard<std::mutex> lock(mu);
    for (const auto& t : tables)
        if (t.first == ctx) return t.second;
    void* p = nullptr;
    const std::vector<uint32_t> words = bucket_words(srgb_table());
    const size_t bytes = words.size() * sizeof(uint32_t);
    if (device_malloc(&p, bytes) != cudaSuccess) throw std::runtime_error("sRGB table allocation");
    if (cudaMemcpy(p, words.data(), bytes, cudaMemcpyHostToDevice) != cudaSuccess) {
        cudaFree(p);
        throw std::runtime_error("sRGB table upload");
    }
    tables.emplace_back(ctx, static_cast<const uint32_t*>(p));
    return tables.back().second;
}

// blocks of the kernel resident on the whole device at once
template <bool kVec>
unsigned tone_grid_cap() {
    int dev = 0, sms = 0, per_sm = 0;
    if (cudaGetDevice(&dev) == cudaSuccess &&
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) == cudaSuccess &&
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_tonemap_srgb8<kVec>, kToneBlock, 0) == cudaSuccess &&
        sms > 0 && per_sm > 0)
        return static_cast<unsigned>(sms * per_sm);
    return 148u * 8u;
}

}  // namespace

void srgb8_thresholds(float* t256, float* c_max) {
    const SrgbTable& tab = srgb_table();
    memcpy(t256, tab.t, sizeof tab.t);
    *c_max = tab.c_max;
}

cudaError_t launch_tonemap_srgb8(const float* rgb, uint8_t* out, uint32_t n, cudaStream_t st, bool beside) {
    if (n == 0) return cudaSuccess;
    const bool vec = (reinterpret_cast<uintptr_t>(rgb) % 16 == 0) && (reinterpret_cast<uintptr_t>(out) % 4 == 0);
    const uint32_t quads = vec ? n / 4 : 0;
    const uint32_t work = quads + (n - 4 * quads);
    static const unsigned caps[2] = {tone_grid_cap<false>(), tone_grid_cap<true>()};
    const unsigned cap = caps[vec ? 1 : 0];
    // as many blocks as give every thread the same number of turns
    const uint64_t turns = (static_cast<uint64_t>(work) + static_cast<uint64_t>(cap) * kToneBlock - 1) /
                           (static_cast<uint64_t>(cap) * kToneBlock);
    const unsigned grid = static_cast<unsigned>((work + turns * kToneBlock - 1) / (turns * kToneBlock));
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = kToneBlock;
    cfg.stream = st;
    cudaLaunchAttribute early{};
    early.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    early.val.programmaticStreamSerializationAllowed = 1;
    if (beside) {
        // a captured launch stays a plain node
        cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
        if (cudaStreamIsCapturing(st, &capture) != cudaSuccess) cudaGetLastError();
        else if (capture == cudaStreamCaptureStatusNone) {
            cfg.attrs = &early;
            cfg.numAttrs = 1;
        }
    }
    const cudaError_t e = cudaLaunchKernelEx(&cfg, vec ? k_tonemap_srgb8<true> : k_tonemap_srgb8<false>, rgb, out, n, quads, device_table(),
                                             float_bits(srgb_table().c_max));
    if (e != cudaSuccess) return e;
    return cudaGetLastError();
}

}  // namespace crisb

// Film outputs on the device: FrameBuffer's writers and tone mappers (film.cpp) for an
// image in the layout mcrt_render writes ([height][width][3] floats, row 0 the bottom).
//
//   k_film_hdr    FrameBuffer::dumpHDR (film.cpp:35-108): every pixel's RGBE bytes go
//                 straight to their place in the file (rows top to bottom, per row the
//                 scanline marker and four channel blocks of literal runs of <= 127 bytes),
//                 so the file is one pass over the image
//   k_film_ppm    FrameBuffer::dumpPPM (film.cpp:9-33)
//   k_film_gamma  FrameBuffer::tonemapGamma (film.cpp:196-203), in place
//   Reinhard      FrameBuffer::tonemapReinhard (film.cpp:110-194): its contrast is fixed at
//                 0.77 and its light adaptation at 0, so each pixel maps x -> x / (x + K_c)
//                 with K_c = (0.5 mean_c + 0.5 mean_lum)^0.77 per channel; the means are
//                 float sums in pixel order with the reference's rounding (see "ordered
//                 float sums"), K_c is evaluated on the host with the C library's powf as the
//                 reference does
//
// Byte- and bit-exact against the reference except tonemapGamma, whose per-pixel powf is
// CUDA's (within its documented ulp bound of the C library's).
#include <cuda_runtime.h>

#include <cmath>
#include <cstdint>
#include <string>
#include <vector>

#include "../../include/mcrt_gb300.h"
#include "wavefront.h"

namespace mcrt {
namespace {

std::string hdr_header(int w, int h)
{
    return "#?RADIANCE\n# Made with custom writer\nFORMAT=32-bit_rle_rgbe\nEXPOSURE=1.0\n\n-Y " + std::to_string(h) +
           " +X " + std::to_string(w) + "\n";
}

std::string ppm_header(int w, int h) { return "P6\n" + std::to_string(w) + " " + std::to_string(h) + "\n255\n"; }

int64_t hdr_runs(int w) { return (w + 126) / 127; }
int64_t hdr_line_bytes(int w) { return 4 + 4 * (w + hdr_runs(w)); }

__global__ void k_film_hdr(const float* __restrict__ rgb, int w, int h, uint8_t* __restrict__ out, int64_t head)
{
    const int64_t n = static_cast<int64_t>(w) * h;
    const int64_t runs = (w + 126) / 127;
    const int64_t line = 4 + 4 * (w + runs);
    for (int64_t p = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; p < n;
         p += static_cast<int64_t>(gridDim.x) * blockDim.x)
    {
        const int j = static_cast<int>(p / w), i = static_cast<int>(p - static_cast<int64_t>(j) * w);
        const float* c = rgb + 3 * p;
        // toRGBE (film.cpp:49-64): d = m 2^e; m * 256 / d = 2^(8 - e) exactly
        float   d = c[0] > c[1] ? c[0] : c[1];
        d = d > c[2] ? d : c[2];
        uint8_t q[4] = {0, 0, 0, 0};
        if (!(static_cast<double>(d) <= 1e-32))
        {
            int         e;
            const float m = frexpf(d, &e);
            const float s = __fdiv_rn(__fmul_rn(m, 256.0f), d);
            q[0] = static_cast<uint8_t>(__fmul_rn(c[0], s));
            q[1] = static_cast<uint8_t>(__fmul_rn(c[1], s));
            q[2] = static_cast<uint8_t>(__fmul_rn(c[2], s));
            q[3] = static_cast<uint8_t>(e + 128);
        }
        uint8_t* row = out + head + static_cast<int64_t>(h - 1 - j) * line;
        if (i == 0)
        {
            row[0] = 2;
            row[1] = 2;
            row[2] = static_cast<uint8_t>((w >> 8) & 0xFF);
            row[3] = static_cast<uint8_t>(w & 0xFF);
        }
        const int64_t run = i / 127, in_run = i - run * 127;
        for (int k = 0; k < 4; ++k)
        {
            uint8_t* chan = row + 4 + k * (w + runs);
            if (in_run == 0) chan[run * 128] = static_cast<uint8_t>(min(127, w - i));
            chan[run * 128 + 1 + in_run] = q[k];
        }
    }
}

__global__ void k_film_ppm(const float* __restrict__ rgb, int w, int h, uint8_t* __restrict__ out, int64_t head)
{
    const int64_t n = 3 * static_cast<int64_t>(w) * h;
    for (int64_t q = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; q < n;
         q += static_cast<int64_t>(gridDim.x) * blockDim.x)
    {
        const int64_t p = q / 3;
        const int     k = static_cast<int>(q - 3 * p);
        const int     j = static_cast<int>(p / w), i = static_cast<int>(p - static_cast<int64_t>(j) * w);
        const float   v = rgb[q];
        const float   c = 1.0f < v ? 1.0f : v;  // f_min(1, v)
        out[head + (static_cast<int64_t>(h - 1 - j) * w + i) * 3 + k] = static_cast<uint8_t>(__fmul_rn(c, 255.0f));
    }
}

__global__ void k_film_gamma(float* rgb, int64_t n, float inv_gamma)
{
    for (int64_t q = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; q < n;
         q += static_cast<int64_t>(gridDim.x) * blockDim.x)
    {
        float x = rgb[q];
        x = x < 0.0f ? 0.0f : x > 1.0f ? 1.0f : x;  // clampf
        rgb[q] = powf(x, inv_gamma);
    }
}

// ---------------------------------------------------------------------------
// ordered float sums: s = fl(... fl(fl(0 + x_0) + x_1) ... + x_{n-1}), bit for bit, in parallel
//
// While s stays in one binade [2^e, 2^(e+1)) it is an integer m times u = 2^(e-23), and adding
// x >= 0 adds a fixed integer to m: x / u rounded to nearest, a tie going up or down with the
// parity of m + floor(x / u).  So a run of additions is m -> m + a[m & 1], two integers, and
// runs compose.  Only where m reaches 2^24 must the addition itself be done, once per binade.
//   k_film_chunk_sums   approximate sums per chunk, and whether a channel has an addend the
//                       scheme does not cover (negative, infinite, NaN)
//   k_film_chunk_incs   per chunk and channel: the binade s is expected to be in (from the
//                       sums before it) and the chunk's two increments for that binade
//   k_film_means        a block per channel joins the chunks, 256 at a time; one whose binade or
//                       end does not fit (about log2 n of them) is redone from s as it is, by the whole
//                       block, up to each addition that leaves the binade.  The addends of a
//                       channel that is not covered, and of an image of one chunk, are added by
//                       one thread.
// One thread summing the four channels, a dependent addition and load after another, made the
// tone mapping of 1023x767 pixels 34.3 ms and of 3840x2160 471 ms; they take 0.23 and 1.4 ms.
// What is left is latency: about ten passes of one block over the first chunk (a binade each)
// and as many redone chunks after it.
// ---------------------------------------------------------------------------
constexpr int kChunkThreads = 256, kChunkEach = 8, kChunk = kChunkThreads * kChunkEach;
constexpr int kFull = 1 << 24;   // m at the end of a binade
constexpr int kMany = 1 << 28;   // increments are cut off here (far past the binade's end)

struct Inc
{
    int a[2];  // what is added to an even / odd m
};

__host__ __device__ __forceinline__ Inc inc_then(Inc f, Inc g)
{
    Inc r;
    r.a[0] = f.a[0] + g.a[f.a[0] & 1];
    r.a[1] = f.a[1] + g.a[(f.a[1] + 1) & 1];
    r.a[0] = r.a[0] < kMany ? r.a[0] : kMany;
    r.a[1] = r.a[1] < kMany ? r.a[1] : kMany;
    return r;
}

// biased exponent of a non-negative float's binade; subnormals (and 0) share the one above them
__host__ __device__ __forceinline__ int binade(unsigned bits) { return bits >> 23 ? static_cast<int>(bits >> 23) : 1; }
// the float as a multiple of its binade's u
__host__ __device__ __forceinline__ int multiple(unsigned bits)
{
    return static_cast<int>(bits >> 23 ? (bits & 0x7fffffu) | 0x800000u : bits);
}
__host__ __device__ __forceinline__ unsigned float_from(int m, int e)
{
    return m & 0x800000 ? (static_cast<unsigned>(e) << 23) | (static_cast<unsigned>(m) & 0x7fffffu)
                        : static_cast<unsigned>(m);  // subnormal (e is 1)
}

// what adding x (bits, finite and >= 0) does to m in binade e.  -0.0 is among them and adds nothing;
// its sign bit read as part of the exponent would put it far above every sum, and chunk_add would
// spend a pass of the block on each (a 64x64 image of them 8.0 ms instead of 0.13).
__host__ __device__ __forceinline__ Inc inc_of(unsigned bits, int e)
{
    bits &= 0x7fffffffu;
    const int shift = e - binade(bits), mant = multiple(bits);
    Inc       r;
    if (shift < 0)
    {
        r.a[0] = r.a[1] = mant ? kMany : 0;
        return r;
    }
    if (shift > 24)
    {
        r.a[0] = r.a[1] = 0;
        return r;
    }
    const int q = mant >> shift, rest = mant & ((1 << shift) - 1), half = shift ? 1 << (shift - 1) : 1;
    const int up = rest > half ? 1 : 0;
    r.a[0] = q + up;
    r.a[1] = q + up;
    if (shift && rest == half)  // a tie: to even
    {
        r.a[0] = q + (q & 1);
        r.a[1] = q + ((q + 1) & 1);
    }
    return r;
}

// luminance (numeric.cpp:62-66): in double, then clamped at 1e-7 (film.cpp:118-120)
__device__ __forceinline__ float film_lum(float r, float g, float b)
{
    const double l = __dadd_rn(__dadd_rn(__dmul_rn(0.299, r), __dmul_rn(0.587, g)), __dmul_rn(0.114, b));
    const float  f = static_cast<float>(l);
    return f < 1e-7f ? 1e-7f : f;
}
// addend of channel c (0 luminance, 1-3 r, g, b) at pixel p
__device__ __forceinline__ float film_addend(const float* __restrict__ rgb, int64_t p, int c)
{
    const float* x = rgb + 3 * p;
    return c == 0 ? film_lum(x[0], x[1], x[2]) : x[c - 1];
}

// the sums are only a guess at s: any order and precision will do
__global__ void __launch_bounds__(kChunkThreads) k_film_chunk_sums(const float* __restrict__ rgb, int64_t n,
                                                                   float* __restrict__ sums, int* __restrict__ bad)
{
    __shared__ float part[4][kChunkThreads / 32];
    const int64_t    first = static_cast<int64_t>(blockIdx.x) * kChunk;
    float            s[4] = {0.f, 0.f, 0.f, 0.f};
    int              odd = 0;
    for (int k = 0; k < kChunkEach; ++k)
    {
        const int64_t p = first + k * kChunkThreads + threadIdx.x;
        if (p >= n) break;
        const float r = rgb[3 * p], g = rgb[3 * p + 1], b = rgb[3 * p + 2];
        const float x[4] = {film_lum(r, g, b), r, g, b};
        for (int c = 0; c < 4; ++c)
        {
            s[c] += x[c];
            if (!(x[c] >= 0.f && x[c] <= 3.4028234663852886e38f)) odd |= 1 << c;
        }
    }
    if (odd) atomicOr(bad, odd);
    for (int c = 0; c < 4; ++c)
    {
        for (int off = 16; off > 0; off >>= 1) s[c] += __shfl_down_sync(0xffffffffu, s[c], off);
        if ((threadIdx.x & 31) == 0) part[c][threadIdx.x >> 5] = s[c];
    }
    __syncthreads();
    if (threadIdx.x < 4)
    {
        float t = 0.f;
        for (int w = 0; w < kChunkThreads / 32; ++w) t += part[threadIdx.x][w];
        sums[4 * static_cast<int64_t>(blockIdx.x) + threadIdx.x] = t;
    }
}

// ordered composition of the block's increments: `mine` per thread in, the composition of all
// lower threads' out (the identity for thread 0); `total` of the block for every thread
__device__ __forceinline__ Inc block_scan_inc(Inc mine, Inc* warp_inc, Inc& total)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    Inc       incl = mine;
    for (int off = 1; off < 32; off <<= 1)
    {
        Inc lo;
        lo.a[0] = __shfl_up_sync(0xffffffffu, incl.a[0], off);
        lo.a[1] = __shfl_up_sync(0xffffffffu, incl.a[1], off);
        if (lane >= off) incl = inc_then(lo, incl);
    }
    __syncthreads();  // warp_inc may still be read from the call before
    if (lane == 31) warp_inc[warp] = incl;
    __syncthreads();
    Inc base = {{0, 0}}, all = {{0, 0}};
    for (int w = 0; w < kChunkThreads / 32; ++w)
    {
        if (w == warp) base = all;
        all = inc_then(all, warp_inc[w]);
    }
    total = all;
    Inc excl;
    excl.a[0] = __shfl_up_sync(0xffffffffu, incl.a[0], 1);
    excl.a[1] = __shfl_up_sync(0xffffffffu, incl.a[1], 1);
    return lane == 0 ? base : inc_then(base, excl);
}

struct ChunkInc
{
    int e;
    Inc inc;
    int pad;
};

__global__ void __launch_bounds__(kChunkThreads) k_film_chunk_incs(const float* __restrict__ rgb, int64_t n,
                                                                   const float* __restrict__ sums,
                                                                   ChunkInc* __restrict__ out, int chunks)
{
    __shared__ float before[4];
    __shared__ Inc   warp_inc[kChunkThreads / 32];
    const int        chunk = blockIdx.x;
    if (threadIdx.x < 4) before[threadIdx.x] = 0.f;
    __syncthreads();
    float s[4] = {0.f, 0.f, 0.f, 0.f};
    for (int j = threadIdx.x; j < chunk; j += kChunkThreads)
        for (int c = 0; c < 4; ++c) s[c] += sums[4 * static_cast<int64_t>(j) + c];
    for (int c = 0; c < 4; ++c)
    {
        for (int off = 16; off > 0; off >>= 1) s[c] += __shfl_down_sync(0xffffffffu, s[c], off);
        if ((threadIdx.x & 31) == 0 && s[c] != 0.f) atomicAdd(&before[c], s[c]);
    }
    __syncthreads();
    const int64_t first = static_cast<int64_t>(chunk) * kChunk + static_cast<int64_t>(threadIdx.x) * kChunkEach;
    for (int c = 0; c < 4; ++c)
    {
        const int e = binade(__float_as_uint(fabsf(before[c])));
        Inc       mine = {{0, 0}};
        for (int k = 0; k < kChunkEach; ++k)
            if (first + k < n) mine = inc_then(mine, inc_of(__float_as_uint(film_addend(rgb, first + k, c)), e));
        Inc total;
        block_scan_inc(mine, warp_inc, total);
        if (threadIdx.x == 0)
        {
            ChunkInc r;
            r.e = e;
            r.inc = total;
            r.pad = 0;
            out[static_cast<int64_t>(c) * chunks + chunk] = r;
        }
    }
}

// a chunk's addends of channel c into shared memory (addend k at padded(k): a thread's
// kChunkEach consecutive addends then lie in different banks from its neighbours'); the
// luminance is in double, a few per clock, so it is worth making once
constexpr int kPadded = kChunk + kChunk / kChunkEach;
__device__ __forceinline__ int padded(int k) { return k + k / kChunkEach; }
__device__ int chunk_load(const float* __restrict__ rgb, int64_t n, int c, int64_t chunk, float* x)
{
    const int64_t base = chunk * kChunk;
    const int     count = static_cast<int>(n - base < kChunk ? n - base : kChunk);
    __syncthreads();
    for (int k = threadIdx.x; k < count; k += kChunkThreads) x[padded(k)] = film_addend(rgb, base + k, c);
    __syncthreads();
    return count;
}

// adds the chunk in x to s, by the whole block; returns the new s in every thread
__device__ float chunk_add(const float* x, int count, float s, Inc* warp_inc, int* at, float* next)
{
    const int     k0 = threadIdx.x * kChunkEach;
    int           from = 0;  // addends of the chunk already in s
    for (int pass = 0; pass < kChunk && from < count; ++pass)
    {
        const unsigned bits = __float_as_uint(s);
        const int      e = binade(bits), m = multiple(bits);
        Inc            mine = {{0, 0}};
        for (int k = k0; k < k0 + kChunkEach; ++k)
            if (k >= from && k < count) mine = inc_then(mine, inc_of(__float_as_uint(x[padded(k)]), e));
        Inc       total;
        const Inc excl = block_scan_inc(mine, warp_inc, total);
        if (m + total.a[m & 1] < kFull)
        {
            s = __uint_as_float(float_from(m + total.a[m & 1], e));
            break;
        }
        // one thread's addends take m over the binade's end
        const int m0 = m + excl.a[m & 1];
        if (m0 < kFull && m0 + mine.a[m0 & 1] >= kFull)
        {
            float t = __uint_as_float(float_from(m0, e));
            int   k = k0 < from ? from : k0;
            bool  over = false;
            while (!over && k < count)
            {
                const float xk = x[padded(k)];
                const int   mt = multiple(__float_as_uint(t));
                over = mt + inc_of(__float_as_uint(xk), e).a[mt & 1] >= kFull;
                t = __fadd_rn(t, xk);
                ++k;
            }
            *at = k;
            *next = t;
        }
        __syncthreads();
        from = *at;
        s = *next;
        __syncthreads();
        if (__float_as_uint(s) >= 0x7f800000u) break;  // the sum overflowed: infinite from here on
    }
    return s;
}

__global__ void __launch_bounds__(kChunkThreads) k_film_means(const float* __restrict__ rgb, int64_t n,
                                                              const ChunkInc* __restrict__ incs, int chunks,
                                                              const int* __restrict__ bad, float* __restrict__ means)
{
    __shared__ Inc      warp_inc[kChunkThreads / 32];
    __shared__ int      at, redo;
    __shared__ float    next, sum, x[kPadded];
    const int           c = blockIdx.x;
    float               s = 0.f;
    if (*bad & (1 << c))
    {
        // the block makes a chunk's addends, one thread adds them in order
        for (int j = 0; j < chunks; ++j)
        {
            const int m = chunk_load(rgb, n, c, j, x);
            if (threadIdx.x == 0)
                for (int k = 0; k < m; ++k) s = __fadd_rn(s, x[padded(k)]);
        }
    }
    else
    {
        for (int j0 = 0; j0 < chunks;)
        {
            // chunks j0 ... as far as they fit, a thread each
            const unsigned bits = __float_as_uint(s);
            const int      e = binade(bits), m = multiple(bits);
            const int      count = min(kChunkThreads, chunks - j0);
            ChunkInc       mine = {-1, {{kMany, kMany}}, 0};
            if (threadIdx.x < count) mine = incs[static_cast<int64_t>(c) * chunks + j0 + threadIdx.x];
            if (mine.e != e) mine.inc.a[0] = mine.inc.a[1] = kMany;  // made for another binade
            if (threadIdx.x == 0) redo = count;
            Inc       total;
            const Inc excl = block_scan_inc(mine.inc, warp_inc, total);
            const int m0 = m + excl.a[m & 1];
            const int m1 = m0 < kFull ? m0 + mine.inc.a[m0 & 1] : kFull;
            if (threadIdx.x < count && m0 < kFull)
            {
                if (m1 >= kFull)
                {
                    redo = threadIdx.x;  // the first that does not fit: its m0 does
                    sum = __uint_as_float(float_from(m0, e));
                }
                else if (threadIdx.x == count - 1)
                    sum = __uint_as_float(float_from(m1, e));
            }
            __syncthreads();
            s = sum;
            const int fit = redo;
            j0 += fit;
            if (fit < count)
            {
                const int k = chunk_load(rgb, n, c, j0, x);
                s = chunk_add(x, k, s, warp_inc, &at, &next);
                ++j0;
                if (__float_as_uint(s) >= 0x7f800000u) break;  // infinite from here on
            }
            __syncthreads();
        }
    }
    if (threadIdx.x == 0) means[c] = __fdiv_rn(s, static_cast<float>(n));
}

__global__ void k_film_reinhard(float* rgb, int64_t n, float kr, float kg, float kb)
{
    for (int64_t p = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; p < n;
         p += static_cast<int64_t>(gridDim.x) * blockDim.x)
    {
        float* x = rgb + 3 * p;
        x[0] = __fdiv_rn(x[0], __fadd_rn(x[0], kr));
        x[1] = __fdiv_rn(x[1], __fadd_rn(x[1], kg));
        x[2] = __fdiv_rn(x[2], __fadd_rn(x[2], kb));
    }
}

int grid_for(int64_t n) { return static_cast<int>(std::min<int64_t>((n + 255) / 256, 152 * 16)); }

#define FCK(x)                                                                                             \
    do                                                                                                     \
    {                                                                                                      \
        cudaError_t e_ = (x);                                                                              \
        if (e_ != cudaSuccess)                                                                             \
        {                                                                                                  \
            release();                                                                                     \
            return set_error(e_ == cudaErrorMemoryAllocation ? MCRT_ERR_OUT_OF_MEMORY : MCRT_ERR_CUDA,     \
                             std::string(#x) + ": " + cudaGetErrorString(e_));                             \
        }                                                                                                  \
    } while (0)

}  // namespace
}  // namespace mcrt

using namespace mcrt;

extern "C" int mcrt_film_encode(const float* rgb, int32_t width, int32_t height, int32_t format, uint8_t* out,
                                int64_t capacity, int64_t* size, int32_t ptr_mode, void* stream)
{
    try
    {
        if (!rgb || !size || width <= 0 || height <= 0)
            return set_error(MCRT_ERR_INVALID_ARGUMENT, "mcrt_film_encode: null image or size, or empty image");
        if (format != MCRT_FILM_HDR && format != MCRT_FILM_PPM)
            return set_error(MCRT_ERR_INVALID_ARGUMENT, "mcrt_film_encode: unknown format");
        const std::string head = format == MCRT_FILM_HDR ? hdr_header(width, height) : ppm_header(width, height);
        const int64_t     body = format == MCRT_FILM_HDR ? hdr_line_bytes(width) * height
                                                         : 3 * static_cast<int64_t>(width) * height;
        *size = static_cast<int64_t>(head.size()) + body;
        if (!out) return MCRT_OK;  // size query
        if (capacity < *size) return set_error(MCRT_ERR_INVALID_ARGUMENT, "mcrt_film_encode: output buffer too small");
        cudaStream_t st = static_cast<cudaStream_t>(stream);
        const float* d_rgb = rgb;
        uint8_t*     d_out = out;
        void*        tmp_in = nullptr;
        void*        tmp_out = nullptr;
        auto         release = [&]() {
            cudaFree(tmp_in);
            cudaFree(tmp_out);
        };
        const size_t img_bytes = sizeof(float) * 3 * static_cast<size_t>(width) * height;
        if (ptr_mode != MCRT_PTR_DEVICE)
        {
            FCK(cudaMalloc(&tmp_in, img_bytes));
            FCK(cudaMalloc(&tmp_out, static_cast<size_t>(*size)));
            FCK(cudaMemcpyAsync(tmp_in, rgb, img_bytes, cudaMemcpyHostToDevice, st));
            d_rgb = static_cast<const float*>(tmp_in);
            d_out = static_cast<uint8_t*>(tmp_out);
        }
        FCK(cudaMemcpyAsync(d_out, head.data(), head.size(), cudaMemcpyHostToDevice, st));
        const int64_t n = static_cast<int64_t>(width) * height;
        if (format == MCRT_FILM_HDR)
            k_film_hdr<<<grid_for(n), 256, 0, st>>>(d_rgb, width, height, d_out, static_cast<int64_t>(head.size()));
        else
            k_film_ppm<<<grid_for(3 * n), 256, 0, st>>>(d_rgb, width, height, d_out,
                                                         static_cast<int64_t>(head.size()));
        FCK(cudaGetLastError());
        if (ptr_mode != MCRT_PTR_DEVICE)
            FCK(cudaMemcpyAsync(out, d_out, static_cast<size_t>(*size), cudaMemcpyDeviceToHost, st));
        FCK(cudaStreamSynchronize(st));
        release();
        return MCRT_OK;
    }
    catch (...)
    {
        return set_error(MCRT_ERR_INTERNAL, "unexpected exception in mcrt_film_encode");
    }
}

extern "C" int mcrt_film_tonemap(float* rgb, int32_t width, int32_t height, int32_t op, float gamma, int32_t ptr_mode,
                                 void* stream)
{
    try
    {
        if (!rgb || width <= 0 || height <= 0)
            return set_error(MCRT_ERR_INVALID_ARGUMENT, "mcrt_film_tonemap: null or empty image");
        if (op != MCRT_TONEMAP_GAMMA && op != MCRT_TONEMAP_REINHARD)
            return set_error(MCRT_ERR_INVALID_ARGUMENT, "mcrt_film_tonemap: unknown operator");
        cudaStream_t  st = static_cast<cudaStream_t>(stream);
        const int64_t n = static_cast<int64_t>(width) * height;
        const size_t  img_bytes = sizeof(float) * 3 * static_cast<size_t>(n);
        float*        d_rgb = rgb;
        void*         tmp = nullptr;
        void*         work = nullptr;
        auto          release = [&]() {
            cudaFree(tmp);
            cudaFree(work);
        };
        if (ptr_mode != MCRT_PTR_DEVICE)
        {
            FCK(cudaMalloc(&tmp, img_bytes));
            FCK(cudaMemcpyAsync(tmp, rgb, img_bytes, cudaMemcpyHostToDevice, st));
            d_rgb = static_cast<float*>(tmp);
        }
        if (op == MCRT_TONEMAP_GAMMA)
        {
            k_film_gamma<<<grid_for(3 * n), 256, 0, st>>>(d_rgb, 3 * n, 1.0f / gamma);
        }
        else
        {
            const int64_t chunks = (n + kChunk - 1) / kChunk;
            // means, the channels not covered, chunk increments and sums
            const size_t  bytes = 32 + (sizeof(ChunkInc) * 4 + sizeof(float) * 4) * static_cast<size_t>(chunks);
            int           device = -1;
            bool          failed = false;
            FCK(cudaGetDevice(&device));
            void* scratch = thread_scratch(device, bytes, failed);
            if (!scratch)
            {
                FCK(cudaMalloc(&work, bytes));
                scratch = work;
            }
            float*    d_means = static_cast<float*>(scratch);
            int*      d_bad = reinterpret_cast<int*>(d_means + 4);
            ChunkInc* d_incs = reinterpret_cast<ChunkInc*>(d_means + 8);
            float*    d_sums = reinterpret_cast<float*>(d_incs + 4 * chunks);
            const int grid = static_cast<int>(chunks);
            // An image of one chunk: no other chunk's sum to compose it with, and the block's passes over
            // the chunk (one per binade) take longer than one thread's additions from shared memory.  All
            // channels go as ones that are not covered (k_film_means), without the two kernels before:
            // 1 / 527 / 2,048 pixels 63 / 94 / 109 -> 49 / 58 / 64 us a call (2,049 pixels, two chunks: 112).
            const bool plain = chunks == 1;
            FCK(cudaMemsetAsync(d_bad, plain ? 0xff : 0, sizeof(int), st));
            if (!plain)
            {
                k_film_chunk_sums<<<grid, kChunkThreads, 0, st>>>(d_rgb, n, d_sums, d_bad);
                k_film_chunk_incs<<<grid, kChunkThreads, 0, st>>>(d_rgb, n, d_sums, d_incs, grid);
            }
            k_film_means<<<4, kChunkThreads, 0, st>>>(d_rgb, n, d_incs, grid, d_bad, d_means);
            float means[4];
            FCK(cudaMemcpyAsync(means, d_means, sizeof(means), cudaMemcpyDeviceToHost, st));
            FCK(cudaStreamSynchronize(st));
            // film.cpp:149-186 with c = 0.5, a = 0, f = exp(-0) = 1, m = 0.77
            const float c = 0.5f, m = 0.77f, f = std::exp(-0.0f);
            const float kr = std::pow(f * (c * means[1] + (1.0f - c) * means[0]), m);
            const float kg = std::pow(f * (c * means[2] + (1.0f - c) * means[0]), m);
            const float kb = std::pow(f * (c * means[3] + (1.0f - c) * means[0]), m);
            k_film_reinhard<<<grid_for(n), 256, 0, st>>>(d_rgb, n, kr, kg, kb);
        }
        FCK(cudaGetLastError());
        if (ptr_mode != MCRT_PTR_DEVICE) FCK(cudaMemcpyAsync(rgb, d_rgb, img_bytes, cudaMemcpyDeviceToHost, st));
        FCK(cudaStreamSynchronize(st));
        release();
        return MCRT_OK;
    }
    catch (...)
    {
        return set_error(MCRT_ERR_INTERNAL, "unexpected exception in mcrt_film_tonemap");
    }
}

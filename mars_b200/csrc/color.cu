// Colour input of the codec and the error metric, on the device.
//
//   ycbcr / rgb_from_ycbcr (crates/mars-core/src/metrics.rs:377-460): BT.601 full range in
//     f64, the reference's operations in its order, rounded half away from zero (CUDA's
//     round() is f64::round), clamped to 0..255 and truncated;
//   downsample_box / upsample_nearest (crates/mars-codec/src/color.rs:60-101): 2x2 box mean
//     (sum + 2) / 4 with the last row/column replicated at odd sides, and its nearest-
//     neighbour inverse;
//   mse (metrics.rs:29-48): the exact integer sum of squared differences (u64), divided by
//     the pixel count on the host.
// All are elementwise or small-stencil byte work, so each should be bound by HBM: a thread takes
// 16 bytes of a plane (8 where two rows make one) whatever the alignment allows, and the
// conversions stay off the f64 pipe.  A 3840 x 2160 frame through all of them (convert, halve and
// restore two planes, convert back, error) took 148 us on one B200 with a byte or an f64 value
// at a time, and takes 95 us, the host's wait for the error included.
#include <cuda_runtime.h>

#include <algorithm>

#include "kernels.cuh"

namespace mars {
namespace {

__device__ __forceinline__ uint32_t round_u8(double x) {
    double r = round(x);
    if (r < 0.0) r = 0.0;
    if (r > 255.0) r = 255.0;
    return (uint32_t)r;
}

__device__ __forceinline__ void ycc_pixel(uint32_t r8, uint32_t g8, uint32_t b8, uint32_t* y,
                                          uint32_t* cb, uint32_t* cr) {
    const double r = (double)r8, g = (double)g8, b = (double)b8;
    *y = round_u8(__dadd_rn(__dadd_rn(__dmul_rn(0.299, r), __dmul_rn(0.587, g)),
                            __dmul_rn(0.114, b)));
    *cb = round_u8(__dadd_rn(__dsub_rn(__dsub_rn(128.0, __dmul_rn(0.168736, r)),
                                       __dmul_rn(0.331264, g)),
                             __dmul_rn(0.5, b)));
    *cr = round_u8(__dsub_rn(__dsub_rn(__dadd_rn(128.0, __dmul_rn(0.5, r)),
                                       __dmul_rn(0.418688, g)),
                             __dmul_rn(0.081312, b)));
}

__device__ __forceinline__ void rgb_pixel(uint32_t y8, uint32_t cb8, uint32_t cr8, uint32_t* r,
                                          uint32_t* g, uint32_t* b) {
    const double y = (double)y8, cb = (double)cb8 - 128.0, cr = (double)cr8 - 128.0;
    *r = round_u8(__dadd_rn(y, __dmul_rn(1.402, cr)));
    *g = round_u8(__dsub_rn(__dsub_rn(y, __dmul_rn(0.344136, cb)), __dmul_rn(0.714136, cr)));
    *b = round_u8(__dadd_rn(y, __dmul_rn(1.772, cb)));
}

// The conversions of four pixels in f32, and in f64 only where f32 cannot decide the rounding.
// The f32 value is off by less than 2^-13 (three roundings below 512 and the coefficients'), so
// a value further than 2^-12 from a half rounds as the f64 one does; the others, the exact
// halves among them (299 r + 587 g + 114 b = 500 mod 1000, one colour in a thousand), take the
// f64 form.  Adding 1.5 * 2^23 rounds to an integer in the low mantissa bits, so no conversion
// instruction (a quarter-rate pipe or slower) is left.  The f64 form of every pixel took
// 25.6 us (ycbcr) and 24.3 us (back) for 3840 x 2160, 2.0 TB/s of the planes' bytes.
constexpr float kRoundMagic = 12582912.0f;
constexpr float kNearHalf = 0.5f - 1.0f / 4096.0f;

__device__ __forceinline__ float byte_f32(uint32_t word, int k) {
    return __uint_as_float(__byte_perm(word, 0x4B000000u, 0x7440 | k)) - 8388608.0f;
}

// v rounded, in the low bits of the returned word; off: the largest distance rounded so far.
__device__ __forceinline__ uint32_t round_bits(float v, float& off) {
    v = fminf(fmaxf(v, 0.0f), 255.0f);
    const float t = v + kRoundMagic;
    off = fmaxf(off, fabsf(v - (t - kRoundMagic)));
    return __float_as_uint(t);
}

template <bool inverse>
__device__ __forceinline__ void convert4(uint32_t a, uint32_t b, uint32_t c, uint32_t& o0,
                                         uint32_t& o1, uint32_t& o2) {
    uint32_t x[4], y[4], z[4], redo = 0u;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const float p = byte_f32(a, k);
        float q = byte_f32(b, k), r = byte_f32(c, k), off = 0.0f;
        if (inverse) {
            q -= 128.0f;
            r -= 128.0f;
            x[k] = round_bits(fmaf(1.402f, r, p), off);
            y[k] = round_bits(fmaf(-0.714136f, r, fmaf(-0.344136f, q, p)), off);
            z[k] = round_bits(fmaf(1.772f, q, p), off);
        } else {
            x[k] = round_bits(fmaf(0.114f, r, fmaf(0.587f, q, 0.299f * p)), off);
            y[k] = round_bits(fmaf(0.5f, r, fmaf(-0.331264f, q, fmaf(-0.168736f, p, 128.0f))), off);
            z[k] = round_bits(fmaf(-0.081312f, r, fmaf(-0.418688f, q, fmaf(0.5f, p, 128.0f))), off);
        }
        redo |= off > kNearHalf ? 1u << k : 0u;
    }
    auto pack = [](const uint32_t (&v)[4]) {
        return __byte_perm(__byte_perm(v[0], v[1], 0x0040), __byte_perm(v[2], v[3], 0x0040), 0x5410);
    };
    o0 = pack(x);
    o1 = pack(y);
    o2 = pack(z);
    while (redo) {
        const uint32_t s = 8u * (uint32_t)(__ffs(redo) - 1);
        redo &= redo - 1u;
        uint32_t u, v, w;
        if (inverse) rgb_pixel((a >> s) & 255u, (b >> s) & 255u, (c >> s) & 255u, &u, &v, &w);
        else ycc_pixel((a >> s) & 255u, (b >> s) & 255u, (c >> s) & 255u, &u, &v, &w);
        const uint32_t keep = ~(255u << s);
        o0 = (o0 & keep) | u << s;
        o1 = (o1 & keep) | v << s;
        o2 = (o2 & keep) | w << s;
    }
}

// Three input planes -> three output planes; `inverse` picks the direction.  T: uint4 where all
// six planes start on 16 bytes and are large, uint32_t where they start on 4, uint8_t otherwise; a
// thread takes P pixels, the last ones byte by byte.
template <bool inverse, class T>
__global__ void __launch_bounds__(256)
    convert_kernel(const uint8_t* __restrict__ p0, const uint8_t* __restrict__ p1,
                   const uint8_t* __restrict__ p2, size_t n, uint8_t* __restrict__ q0,
                   uint8_t* __restrict__ q1, uint8_t* __restrict__ q2) {
    constexpr int P = sizeof(T) < 4 ? 4 : (int)sizeof(T);
    const size_t i = ((size_t)blockIdx.x * blockDim.x + threadIdx.x) * P;
    if (i >= n) return;
    if (sizeof(T) >= 4 && i + P <= n) {
        constexpr int W = P / 4;
        union Words {
            T all;
            uint32_t w[W];
        } a, b, c, x, y, z;
        a.all = *reinterpret_cast<const T*>(p0 + i);
        b.all = *reinterpret_cast<const T*>(p1 + i);
        c.all = *reinterpret_cast<const T*>(p2 + i);
#pragma unroll
        for (int k = 0; k < W; ++k)
            convert4<inverse>(a.w[k], b.w[k], c.w[k], x.w[k], y.w[k], z.w[k]);
        *reinterpret_cast<T*>(q0 + i) = x.all;
        *reinterpret_cast<T*>(q1 + i) = y.all;
        *reinterpret_cast<T*>(q2 + i) = z.all;
        return;
    }
    // Byte by byte, four to a conversion (with one to each, planes at odd addresses took 57 us of
    // 3840 x 2160, and take 22; aligned ones 18).
    for (size_t k = i; k < n && k < i + P; k += 4) {
        uint32_t a = 0u, b = 0u, c = 0u, x, y, z;
#pragma unroll
        for (int j = 0; j < 4; ++j)
            if (k + j < n) {
                a |= (uint32_t)p0[k + j] << (8 * j);
                b |= (uint32_t)p1[k + j] << (8 * j);
                c |= (uint32_t)p2[k + j] << (8 * j);
            }
        convert4<inverse>(a, b, c, x, y, z);
#pragma unroll
        for (int j = 0; j < 4; ++j)
            if (k + j < n) {
                q0[k + j] = (uint8_t)(x >> (8 * j));
                q1[k + j] = (uint8_t)(y >> (8 * j));
                q2[k + j] = (uint8_t)(z >> (8 * j));
            }
    }
}

// Eight bytes from address p, not necessarily aligned, of which the caller's plane holds
// `inside` (at least 8) from p on: two aligned loads where they stay in the plane.
__device__ __forceinline__ uint64_t unaligned8(const uint8_t* p, size_t inside) {
    const unsigned s = (unsigned)(reinterpret_cast<uintptr_t>(p) & 7);
    const uint64_t* q = reinterpret_cast<const uint64_t*>(p - s);
    if (s == 0) return __ldg(q);
    if (inside >= 16) {
        // The first word's leading bytes lie before p, in the same 8-byte word as p's.
        return (__ldg(q) >> (8 * s)) | (__ldg(q + 1) << (64 - 8 * s));
    }
    uint64_t v = 0;
#pragma unroll
    for (int k = 0; k < 8; ++k) v |= (uint64_t)__ldg(p + k) << (8 * k);
    return v;
}

// Both resamplings walk the output as one run of bytes in aligned chunks of K, so that a chunk
// is one store at any width; a chunk inside one row and away from the replicated border comes
// from word loads, any other byte by byte.
struct Chunk {
    uint32_t x, y;
    size_t begin, end;  // of the output's bytes
};

template <int K>
__device__ __forceinline__ bool output_chunk(const uint8_t* dst, size_t n, uint32_t w, Chunk* c) {
    const size_t lead = reinterpret_cast<uintptr_t>(dst) & (K - 1);
    const size_t at = ((size_t)blockIdx.x * blockDim.x + threadIdx.x) * K;
    if (at >= n + lead) return false;
    c->begin = at < lead ? 0 : at - lead;
    c->end = min(at + K - lead, n);
    c->y = (uint32_t)c->begin / w;  // sides are at most 65535: 32 bits hold any position
    c->x = (uint32_t)c->begin - c->y * w;
    return true;
}

// Bytes taken one by one: all loaded before the first is stored, so that a chunk across a row's
// end costs one round trip (as a loop of loads and stores these chunks, one a row at odd widths,
// made a small frame slower than a byte a thread was).
template <int K>
__device__ __forceinline__ void store_chunk(uint8_t* dst, const Chunk& c, const uint32_t (&v)[K]) {
    if (c.end - c.begin == K) {
        uint32_t w[K / 4];
#pragma unroll
        for (int k = 0; k < K / 4; ++k)
            w[k] = v[4 * k] | v[4 * k + 1] << 8 | v[4 * k + 2] << 16 | v[4 * k + 3] << 24;
        if (K == 16)
            *reinterpret_cast<uint4*>(dst + c.begin) = make_uint4(w[0], w[1], w[K / 4 - 2], w[K / 4 - 1]);
        else
            *reinterpret_cast<uint2*>(dst + c.begin) = make_uint2(w[0], w[1]);
        return;
    }
#pragma unroll
    for (int k = 0; k < K; ++k)
        if (c.begin + k < c.end) dst[c.begin + k] = (uint8_t)v[k];
}

// A byte a thread, for small planes whose rows are no whole chunks: a chunk across a row's end is
// eight or sixteen bytes one by one in one thread, which such a plane waits for.  (The parameters
// are a multiple of eight bytes: with four fewer a launch took the host 0.3 us more.)
__global__ void __launch_bounds__(256)
    downsample_box_bytes_kernel(const uint8_t* __restrict__ src, int w, int h,
                                uint8_t* __restrict__ dst, int ow, int oh) {
    const int x = blockIdx.x * blockDim.x + threadIdx.x, y = blockIdx.y;
    if (x >= ow || y >= oh) return;
    const int x1 = min(2 * x + 1, w - 1), y1 = min(2 * y + 1, h - 1);
    const uint8_t *top = src + (size_t)(2 * y) * w, *low = src + (size_t)y1 * w;
    const uint32_t sum = (uint32_t)top[2 * x] + top[x1] + low[2 * x] + low[x1];
    dst[(size_t)y * ow + x] = (uint8_t)((sum + 2) / 4);
}

__global__ void __launch_bounds__(256)
    upsample_nearest_bytes_kernel(const uint8_t* __restrict__ src, int sw, int sh,
                                  uint8_t* __restrict__ dst, int w, int h) {
    const int x = blockIdx.x * blockDim.x + threadIdx.x, y = blockIdx.y;
    if (x < w && y < h)
        dst[(size_t)y * w + x] = src[(size_t)min(y / 2, sh - 1) * sw + min(x / 2, sw - 1)];
}

// 9.2 us a 3840 x 2160 plane with a byte a thread.
__global__ void __launch_bounds__(256)
    downsample_box_kernel(const uint8_t* __restrict__ src, int w, int h, uint8_t* __restrict__ dst,
                          int ow, int oh) {
    Chunk c;
    if (!output_chunk<8>(dst, (size_t)ow * oh, (uint32_t)ow, &c)) return;
    const size_t total = (size_t)w * h;
    if (c.end - c.begin == 8 && c.x + 8 <= (uint32_t)(w / 2)) {
        const size_t top = (size_t)(2 * c.y) * w + 2 * c.x;
        const size_t low = (int)(2 * c.y + 1) < h ? top + w : top;
        uint32_t out[2];
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            const uint64_t a = unaligned8(src + top + 8 * k, total - top - 8 * k);
            const uint64_t b = unaligned8(src + low + 8 * k, total - low - 8 * k);
            // Byte pairs' sums in 16-bit lanes, two rows, rounded.
            constexpr uint64_t kEven = 0x00FF00FF00FF00FFull;
            const uint64_t s = (a & kEven) + (a >> 8 & kEven) + (b & kEven) + (b >> 8 & kEven) +
                               0x0002000200020002ull;
            const uint64_t m = s >> 2;
            out[k] = __byte_perm((uint32_t)m, (uint32_t)(m >> 32), 0x6420);
        }
        *reinterpret_cast<uint2*>(dst + c.begin) = make_uint2(out[0], out[1]);
        return;
    }
    uint32_t v[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        // Past the chunk's end the last byte again.
        const int x0 = 2 * (int)c.x, y0 = 2 * (int)c.y;
        const int x1 = min(x0 + 1, w - 1), y1 = min(y0 + 1, h - 1);
        const uint32_t sum = (uint32_t)src[(size_t)y0 * w + x0] + src[(size_t)y0 * w + x1] +
                             src[(size_t)y1 * w + x0] + src[(size_t)y1 * w + x1];
        v[k] = (sum + 2) / 4;
        if (c.begin + k + 1 < c.end && ++c.x == (uint32_t)ow) {
            c.x = 0;
            ++c.y;
        }
    }
    store_chunk<8>(dst, c, v);
}

// 22.3 us for a 3840 x 2160 output with a byte a thread.
__global__ void __launch_bounds__(256)
    upsample_nearest_kernel(const uint8_t* __restrict__ src, int sw, int sh,
                            uint8_t* __restrict__ dst, int w, int h) {
    Chunk c;
    if (!output_chunk<16>(dst, (size_t)w * h, (uint32_t)w, &c)) return;
    const size_t total = (size_t)sw * sh;
    const uint32_t sx = c.x / 2;
    if (c.end - c.begin == 16 && c.x + 16 <= (uint32_t)w && sx + 8 + (c.x & 1u) <= (uint32_t)sw) {
        const size_t at = (size_t)min((int)(c.y / 2), sh - 1) * sw + sx;
        const uint64_t v = unaligned8(src + at, total - at);
        const uint32_t lo = (uint32_t)v, hi = (uint32_t)(v >> 32);
        uint32_t o[4] = {__byte_perm(lo, 0, 0x1100), __byte_perm(lo, 0, 0x3322),
                         __byte_perm(hi, 0, 0x1100), __byte_perm(hi, 0, 0x3322)};
        if (c.x & 1u) {  // starts with the second copy of its first sample
            const uint32_t last = __ldg(src + at + 8);
            o[0] = __funnelshift_r(o[0], o[1], 8);
            o[1] = __funnelshift_r(o[1], o[2], 8);
            o[2] = __funnelshift_r(o[2], o[3], 8);
            o[3] = __funnelshift_r(o[3], last, 8);
        }
        *reinterpret_cast<uint4*>(dst + c.begin) = make_uint4(o[0], o[1], o[2], o[3]);
        return;
    }
    uint32_t v[16];
#pragma unroll
    for (int k = 0; k < 16; ++k) {
        v[k] = src[(size_t)min((int)(c.y / 2), sh - 1) * sw + min((int)(c.x / 2), sw - 1)];
        if (c.begin + k + 1 < c.end && ++c.x == (uint32_t)w) {
            c.x = 0;
            ++c.y;
        }
    }
    store_chunk<16>(dst, c, v);
}

// Sum of squared differences: per-thread partial sums over 16-byte chunks, a warp and block
// reduction, one 64-bit atomic per block (exact: integers throughout).
__global__ void sse_kernel(const uint8_t* __restrict__ a, const uint8_t* __restrict__ b,
                           size_t n, bool vec, unsigned long long* __restrict__ out) {
    __shared__ unsigned long long part[32];
    unsigned long long acc = 0;
    const size_t stride = (size_t)gridDim.x * blockDim.x;
    const size_t tid = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (vec) {
        const size_t nv = n / 16;
        for (size_t v = tid; v < nv; v += stride) {
            const uint4 x = reinterpret_cast<const uint4*>(a)[v];
            const uint4 y = reinterpret_cast<const uint4*>(b)[v];
            const uint32_t xs[4] = {x.x, x.y, x.z, x.w}, ys[4] = {y.x, y.y, y.z, y.w};
            uint32_t s = 0;  // 16 squares of at most 65025: fits 32 bits
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const uint32_t d = __vabsdiffu4(xs[k], ys[k]);
                s = __dp4a(d, d, s);
            }
            acc += s;
        }
        for (size_t i = nv * 16 + tid; i < n; i += stride) {
            const int d = (int)a[i] - (int)b[i];
            acc += (unsigned long long)(d * d);
        }
    } else {
        for (size_t i = tid; i < n; i += stride) {
            const int d = (int)a[i] - (int)b[i];
            acc += (unsigned long long)(d * d);
        }
    }
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (lane == 0) part[warp] = acc;
    __syncthreads();
    if (warp == 0) {
        acc = lane < (int)(blockDim.x >> 5) ? part[lane] : 0ull;
        for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
        if (lane == 0) atomicAdd(out, acc);
    }
}

}  // namespace

// Blocks of 256 threads for the chunks of n output bytes (output_chunk).
static unsigned chunk_blocks(const uint8_t* dst, size_t n, size_t k) {
    const size_t chunks = (n + (reinterpret_cast<uintptr_t>(dst) & (k - 1)) + k - 1) / k;
    return (unsigned)((chunks + 255) / 256);
}

// Whether an output of w x h bytes goes byte by byte: less than `most`, rows no whole chunks of k.
static bool ragged_bytes(const uint8_t* dst, int w, int h, size_t k, size_t most) {
    return (size_t)w * h < most &&
           (w % k != 0 || (reinterpret_cast<uintptr_t>(dst) & (k - 1)) != 0);
}

cudaError_t launch_ycbcr(const uint8_t* r, const uint8_t* g, const uint8_t* b, size_t n,
                         uint8_t* y, uint8_t* cb, uint8_t* cr, bool inverse, cudaStream_t st) {
    if (n == 0) return cudaSuccess;
    const uintptr_t at = reinterpret_cast<uintptr_t>(r) | reinterpret_cast<uintptr_t>(g) |
                         reinterpret_cast<uintptr_t>(b) | reinterpret_cast<uintptr_t>(y) |
                         reinterpret_cast<uintptr_t>(cb) | reinterpret_cast<uintptr_t>(cr);
    auto launch = [&](auto kernel, size_t per_thread) {
        const size_t threads = (n + per_thread - 1) / per_thread;
        kernel<<<(unsigned)((threads + 255) / 256), 256, 0, st>>>(r, g, b, n, y, cb, cr);
    };
    // Sixteen pixels a thread are a longer chain: worth it once they still fill the device.
    if (at % 16 == 0 && n >= (1u << 21)) {
        if (inverse) launch(convert_kernel<true, uint4>, 16);
        else launch(convert_kernel<false, uint4>, 16);
    } else if (at % 4 == 0) {
        if (inverse) launch(convert_kernel<true, uint32_t>, 4);
        else launch(convert_kernel<false, uint32_t>, 4);
    } else {
        if (inverse) launch(convert_kernel<true, uint8_t>, 4);
        else launch(convert_kernel<false, uint8_t>, 4);
    }
    return cudaGetLastError();
}

cudaError_t launch_downsample_box(const uint8_t* src, int w, int h, uint8_t* dst,
                                  cudaStream_t st) {
    const int ow = (w + 1) / 2, oh = (h + 1) / 2;
    if (ow == 0 || oh == 0) return cudaSuccess;
    // us in chunks and in bytes, launch after launch: halving 340 x 260 4.1 and 3.2, 1000 x 750 4.1
    // and 3.2, 1601 x 1201 4.1 and 4.2; whole chunks a row, 512 x 512, 3.1 and 3.1.
    if (ragged_bytes(dst, ow, oh, 8, 1u << 19))
        downsample_box_bytes_kernel<<<dim3((ow + 255) / 256, oh), 256, 0, st>>>(src, w, h, dst, ow,
                                                                                oh);
    else
        downsample_box_kernel<<<chunk_blocks(dst, (size_t)ow * oh, 8), 256, 0, st>>>(src, w, h, dst,
                                                                                     ow, oh);
    return cudaGetLastError();
}

cudaError_t launch_upsample_nearest(const uint8_t* src, int sw, int sh, uint8_t* dst, int w,
                                    int h, cudaStream_t st) {
    if (w == 0 || h == 0) return cudaSuccess;
    // To 340 x 260 4.1 and 3.2, to 486 x 324 4.1 and 3.2, to 604 x 506 4.1 and 4.1.
    if (ragged_bytes(dst, w, h, 16, 1u << 18))
        upsample_nearest_bytes_kernel<<<dim3((w + 255) / 256, h), 256, 0, st>>>(src, sw, sh, dst, w,
                                                                                h);
    else
        upsample_nearest_kernel<<<chunk_blocks(dst, (size_t)w * h, 16), 256, 0, st>>>(src, sw, sh,
                                                                                      dst, w, h);
    return cudaGetLastError();
}

cudaError_t launch_sse(const uint8_t* a, const uint8_t* b, size_t n, int num_sms,
                       unsigned long long* out, cudaStream_t st) {
    cudaError_t e = cudaMemsetAsync(out, 0, sizeof(unsigned long long), st);
    if (e != cudaSuccess || n == 0) return e;
    const bool vec = ((reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(b)) & 15) == 0;
    const size_t want = (n / 16 + 255) / 256;
    const unsigned blocks = (unsigned)std::max<size_t>(1, std::min<size_t>(want, (size_t)num_sms * 8));
    sse_kernel<<<blocks, 256, 0, st>>>(a, b, n, vec, out);
    return cudaGetLastError();
}

}  // namespace mars

// Fixed-point decode iteration as a gather.
//
// decode_step / decode_leaf (crates/mars-codec/src/ifs.rs:299-309, 406-484) scatter each
// leaf's (u, v) domain samples to range positions (i, j) = map(iso, u, v).  Every output
// pixel belongs to exactly one leaf, so the same map is computed here as a gather: the
// owner map (one leaf index per 2^lg x 2^lg cell, lg the largest power of two dividing
// every leaf's row, column and size) names the leaf of each pixel, and the inverse
// isometry names its domain sample.  Values use the reference's f64 association,
// (0.5 + d*alfa) + beta (+ the mode-3 residual); pixels no leaf covers are written 0, as
// the reference's zero-filled `next` buffer is.
//
// The 16-byte packed leaves are expanded once per leaf list (decode_expand_kernel): alfa
// and beta are dequantised with the reference's operations in its order, so the doubles
// are the ones decode_leaf computes.
//
// decode_cell_kernel (lg >= 2, width % 4 == 0): one thread per 4x4 output cell.  A cell lies
// in one leaf, and the inverse isometry maps it onto a 4x4 set of domain samples, i.e. one
// 8x8 byte window of the previous iterate: the thread takes its eight rows from aligned 16-byte
// loads (and 8 bytes more where a row reaches past them) that are in flight together, forms
// the sixteen 2x2 sums with byte-pair SIMD adds in 16-bit lanes, evaluates the sixteen
// values in sample order (in integers where the leaf allows it, else in f64), moves them to
// output order with byte permutes (row reversal, byte reversal, 4x4 transpose) and stores four
// 4-byte rows.  decode_pixel_kernel covers any other geometry; decode_resident_kernel runs every
// step of a small plane in one launch, the sorted_* kernels a step of a large one.
#include "grid_meet.cuh"
#include "kernels.cuh"

namespace mars {
namespace {

struct Unpacked {
    double alfa, beta, gx, gy;  // mode 1: alfa holds b0
    int row, col, size, mode, iso, dom_row, dom_col;
    bool domain;                // qalfa != 0 and mode != 1: the leaf reads a domain block
};

// ifs.rs:416-439.
__device__ __forceinline__ Unpacked unpack(const DecodeLeaf p, const DecodeConsts& c) {
    Unpacked L;
    L.row = (int)(p.x & 0xFFFFu);
    L.col = (int)(p.x >> 16);
    L.size = (int)(p.y & 0xFFFu);
    L.mode = (int)((p.y >> 12) & 3u);
    const double qbeta = (double)(p.y >> 16);
    L.gx = L.gy = 0.0;
    L.iso = 0;
    L.dom_row = L.dom_col = 0;
    L.domain = false;
    if (L.mode == 1) {
        L.alfa = __dmul_rn(__ddiv_rn(qbeta, c.beta_den), 255.0);
        L.beta = 0.0;
        L.gx = __ddiv_rn((double)(int32_t)p.z, 64.0);
        L.gy = __ddiv_rn((double)(int32_t)p.w, 64.0);
    } else {
        const uint32_t qalfa = p.w & 0x1FFFFu;
        L.iso = (int)(p.w >> 24);
        L.dom_row = (int)(p.z & 0xFFFFu);
        L.dom_col = (int)(p.z >> 16);
        L.domain = qalfa != 0;
        L.alfa = __dmul_rn(__ddiv_rn((double)qalfa, c.alfa_den), c.max_alfa);
        L.beta = __dmul_rn(__ddiv_rn(qbeta, c.beta_den),
                           __dmul_rn(__dadd_rn(1.0, fabs(L.alfa)), 255.0));
        if (L.alfa > 0.0) L.beta = __dsub_rn(L.beta, __dmul_rn(L.alfa, 255.0));
    }
    return L;
}

__device__ __forceinline__ uint32_t clamp_u8(double value) {
    if (!(value >= 0.0)) value = 0.0;
    if (value > 255.0) value = 255.0;
    return (uint32_t)value;
}

// clamp(0, 255) then truncation: truncating first and clamping the integer gives the same
// byte (a NaN converts to 0 either way).
__device__ __forceinline__ uint32_t to_u8(double value) {
    return (uint32_t)min(max(__double2int_rz(value), 0), 255);
}

// (u, v) = (cu + ai*i + aj*j, cv + bi*i + bj*j): the inverse of isometry::map
// (isometry.rs:7-19) as an affine map of the range position (i, j), with S1 = size - 1.
// Three bits describe it: tr (u follows j and v follows i: isometries 1, 2, 6, 7), uneg (u
// counts down from S1: 2, 3, 5, 7) and vneg (v counts down: 1, 3, 4, 7).
struct IsoInv {
    int cu, ai, aj, cv, bi, bj;
};
__device__ __forceinline__ IsoInv iso_inverse(int k, int S1) {
    const bool tr = (0xC6u >> k) & 1u, uneg = (0xACu >> k) & 1u, vneg = (0x9Au >> k) & 1u;
    const int su = uneg ? -1 : 1, sv = vneg ? -1 : 1;
    return {uneg ? S1 : 0, tr ? 0 : su, tr ? su : 0, vneg ? S1 : 0, tr ? sv : 0, tr ? 0 : sv};
}

// A 4x4 byte tile in four row words (byte q of word p = element (p, q)): transposed.
__device__ __forceinline__ void transpose4x4(uint32_t& r0, uint32_t& r1, uint32_t& r2,
                                             uint32_t& r3) {
    // 2x2 blocks of bytes first, then bytes within each block.
    const uint32_t a0 = __byte_perm(r0, r2, 0x5410), a1 = __byte_perm(r1, r3, 0x5410);
    const uint32_t a2 = __byte_perm(r0, r2, 0x7632), a3 = __byte_perm(r1, r3, 0x7632);
    r0 = __byte_perm(a0, a1, 0x6240);
    r1 = __byte_perm(a0, a1, 0x7351);
    r2 = __byte_perm(a2, a3, 0x6240);
    r3 = __byte_perm(a2, a3, 0x7351);
}

__global__ void decode_expand_kernel(const DecodeLeaf* __restrict__ leaves,
                                     const int32_t* __restrict__ resid_off, int n,
                                     DecodeConsts c, DecodeMap* __restrict__ maps) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    const Unpacked L = unpack(leaves[k], c);
    DecodeMap m;
    // Domain kinds keep alfa / 4: (sum / 4) * alfa == sum * (alfa / 4) exactly, both
    // scalings by 1/4 being exact.
    m.a = L.mode == 1 ? L.alfa : __dmul_rn(L.alfa, 0.25);
    m.b = L.beta;
    m.gx = L.gx;
    m.gy = L.gy;
    m.rc = (uint32_t)L.row | ((uint32_t)L.col << 16);
    m.dom = (uint32_t)L.dom_row | ((uint32_t)L.dom_col << 16);
    m.roff = -1;
    uint32_t kind, cbyte = 0, flags = 0;
    if (L.mode == 1) {
        kind = kLeafAffine;
    } else if (L.mode == 3 && resid_off && resid_off[k] >= 0) {
        // A zero-alpha residual leaf still adds its residual (ifs.rs:459-479).
        kind = kLeafResidual;
        m.roff = resid_off[k];
        if (!L.domain) flags = kLeafNoDomain;
    } else if (!L.domain) {
        // d = 0: (0.5 + 0*alfa) + beta, the same for every pixel of the leaf.
        kind = kLeafConst;
        cbyte = clamp_u8(__dadd_rn(__dadd_rn(0.5, __dmul_rn(0.0, L.alfa)), L.beta));
    } else {
        kind = kLeafDomain;
    }
    // The integer form.  Where alfa / 4 is A / 64 (A up to 32: contrasts in sixteenths up to 2,
    // as streams have them), 0.5 + sum * A / 64 is exact and the pixel is the f64 sum of that and
    // beta, truncated: floor((32 + sum * A + floor(64 beta)) / 64) in integers, unless the f64
    // sum rounds up to the next integer, for which the fraction of 64 beta must be nearly 1
    // (sums stay below 2^11, so within 2^-36; the limit of 2^-20 is generous).  An affine pixel's
    // gradients are sixty-fourths, its half rounds up (below zero everything clamps), and its two
    // roundings are below 2^-23 sixty-fourths for |64 value| < 2^29.
    m.n0 = m.n1 = m.n2 = m.unused = 0;
    const double b64 = 64.0 * (kind == kLeafAffine ? m.a : m.b), low = floor(b64);
    const bool whole = b64 - low < 1.0 - 0x1p-20;
    if (kind == kLeafDomain) {
        const double times = 64.0 * m.a, base = low + 32.0;
        if (whole && times == floor(times) && times >= 0.0 && times <= 32.0 && base >= -32768.0 &&
            base + 1020.0 * times <= 32767.0) {
            m.n0 = (int)(((uint32_t)(int)base & 0xFFFFu) * 0x10001u);
            m.n1 = (int)times;
            flags |= kLeafInteger;
        }
    } else if (kind == kLeafAffine) {
        const double reach = (fabs(m.gx) + fabs(m.gy)) * 64.0 * L.size + fabs(b64);
        if (whole && reach < 0x1p29) {
            m.n0 = (int)low + 32;
            m.n1 = (int)leaves[k].z;
            m.n2 = (int)leaves[k].w;
            flags |= kLeafInteger;
        }
    }
    m.info = (uint32_t)L.size | (kind << 12) | ((uint32_t)L.iso << 14) | flags | (cbyte << 24);
    maps[k] = m;
}

// The values a residual leaf adds (residual.hpp values(), ifs.rs:441-456): dead-zone
// dequantisation, then the inverse DCT, columns before rows.  Every output is one thread's
// left-to-right f64 sum from -0.0, no product fused into it, over the host's basis: the host's
// doubles.  A block a leaf.  Bound by the f64 sums' latency.  A one-shot decode until stable of
// 1000 x 752 with a quarter of its domain leaves residual took 2.3 ms and more with the values made
// on the host and sent, and 0.6 ms with this (0.44 ms without residuals).
__global__ void __launch_bounds__(128) residual_values_kernel(
    const DecodeLeaf* __restrict__ leaves, const int32_t* __restrict__ resid_off,
    const int32_t* __restrict__ levels, const ResidualBases bases, double step,
    double* __restrict__ values) {
    extern __shared__ double coef[];
    const int32_t at = resid_off[blockIdx.x];
    if (at < 0) return;
    const int n = (int)(leaves[blockIdx.x].y & 0xFFFu), nn = n * n;
    const double* __restrict__ b = bases.basis + bases.at[n];
    double* half = coef + nn;
    const double threshold = __dmul_rn(0.5, step);  // the dead zone is half a step
    for (int k = threadIdx.x; k < nn; k += blockDim.x) {
        const int32_t level = levels[at + k];
        double v = 0.0;
        if (level != 0) {
            const uint32_t size = level < 0 ? 0u - (uint32_t)level : (uint32_t)level;
            const double mag = __dadd_rn(
                threshold, __dmul_rn(__dadd_rn(__dsub_rn((double)size, 1.0), 0.5), step));
            v = level < 0 ? -mag : mag;
        }
        coef[k] = v;
    }
    __syncthreads();
    for (int t = threadIdx.x; t < nn; t += blockDim.x) {
        const int i = t / n, c = t - i * n;
        double s = -0.0;
#pragma unroll 4
        for (int k = 0; k < n; ++k) s = __dadd_rn(s, __dmul_rn(coef[k * n + c], __ldg(b + k * n + i)));
        half[t] = s;
    }
    __syncthreads();
    for (int t = threadIdx.x; t < nn; t += blockDim.x) {
        const int r = t / n, i = t - r * n;
        double s = -0.0;
#pragma unroll 4
        for (int k = 0; k < n; ++k) s = __dadd_rn(s, __dmul_rn(half[r * n + k], __ldg(b + k * n + i)));
        values[at + t] = s;
    }
}

__device__ __forceinline__ double domain_value(int sum, const DecodeMap& m) {
    // The four samples are small integers, so their f64 sum in the reference's order is
    // the integer sum exactly, and d * alfa = (sum / 4) * alfa = sum * (alfa / 4).
    return __dadd_rn(__dadd_rn(0.5, __dmul_rn((double)sum, m.a)), m.b);
}

__device__ __forceinline__ uint32_t sixty_fourths(int n) {
    return (uint32_t)min(max(n >> 6, 0), 255);
}

// Mode 1: round(b0 + gx*u + gy*v) with (u, v) = (i, j) (ifs.rs:416-431); f64::round and
// CUDA's round() both round half away from zero.
__device__ __forceinline__ uint32_t affine_pixel(const DecodeMap& m, int i, int j) {
    if (m.info & kLeafInteger) return sixty_fourths(m.n0 + m.n1 * i + m.n2 * j);
    return clamp_u8(round(__dadd_rn(__dadd_rn(m.a, __dmul_rn(m.gx, (double)i)),
                                    __dmul_rn(m.gy, (double)j))));
}

// Max-delta bookkeeping of the convergence-tested decode (decode_until_stable,
// ifs.rs:321-353): a step that starts after convergence writes nothing, and every step
// folds max |next - prev| of its pixels into its slot.
struct StableState {
    const int* done;  // set once an earlier step's delta met the threshold
    int* delta;       // this step's max |next - prev|
};

__device__ __forceinline__ void fold_delta(uint32_t d, int* slot) {
    for (int o = 16; o > 0; o >>= 1) d = max(d, __shfl_xor_sync(0xffffffffu, d, o));
    if ((threadIdx.x & 31) == 0 && d) atomicMax(slot, (int)d);
}

// One pixel per thread (any owner-map granularity or width).
template <bool kStable>
__global__ void decode_pixel_kernel(const uint8_t* __restrict__ src, uint8_t* __restrict__ dst,
                                    int w, int h, int lg, int mw,
                                    const int32_t* __restrict__ owner,
                                    const DecodeMap* __restrict__ maps,
                                    const double* __restrict__ resid, StableState ss) {
    if (kStable && *ss.done) return;
    const int x = blockIdx.x * blockDim.x + threadIdx.x;
    const int y = blockIdx.y;
    if (kStable && (x >= w || y >= h)) {
        fold_delta(0u, ss.delta);
        return;
    }
    if (x >= w || y >= h) return;
    const int32_t li = owner[(size_t)(y >> lg) * mw + (x >> lg)];
    uint32_t out = 0;
    if (li >= 0) {
        // The f64 form throughout: a pixel has little arithmetic, and a map's integer form is 16
        // bytes more to load (ten steps of 6002 x 6000: 2,258 us with it, 2,223 without).
        DecodeMap m;
        const uint4 head = *reinterpret_cast<const uint4*>(&maps[li].rc);
        const double2 ab = *reinterpret_cast<const double2*>(&maps[li].a);
        m.rc = head.x;
        m.info = head.y & ~kLeafInteger;
        m.dom = head.z;
        m.roff = (int32_t)head.w;
        m.a = ab.x;
        m.b = ab.y;
        const uint32_t kind = (m.info >> 12) & 3u;
        const int i = y - (int)(m.rc & 0xFFFFu), j = x - (int)(m.rc >> 16);
        if (kind == kLeafConst) {
            out = m.info >> 24;
        } else if (kind == kLeafAffine) {
            m.gx = maps[li].gx;
            m.gy = maps[li].gy;
            out = affine_pixel(m, i, j);
        } else {
            const int S = (int)(m.info & 0xFFFu);
            const IsoInv t = iso_inverse((int)((m.info >> 14) & 7u), S - 1);
            const int u = t.cu + t.ai * i + t.aj * j, v = t.cv + t.bi * i + t.bj * j;
            int sum = 0;
            if (!(m.info & kLeafNoDomain)) {
                const size_t p = ((size_t)(m.dom & 0xFFFFu) + 2 * u) * w + (m.dom >> 16) + 2 * v;
                sum = (int)src[p] + (int)src[p + w] + (int)src[p + 1] + (int)src[p + w + 1];
            }
            double value = domain_value(sum, m);
            if (kind == kLeafResidual) value = __dadd_rn(value, resid[m.roff + u * S + v]);
            out = to_u8(value);
        }
    }
    dst[(size_t)y * w + x] = (uint8_t)out;
    if (kStable) {
        const uint32_t prev = src[(size_t)y * w + x];
        fold_delta(out > prev ? out - prev : prev - out, ss.delta);
    }
}

// Loads of a plane, made where they stand.  FRESH: other SMs write the plane during the launch,
// so L1 is passed by (and no load may move across a barrier).
template <bool FRESH>
__device__ __forceinline__ uint4 plane16(const uint8_t* p) {
    if (!FRESH) return __ldg(reinterpret_cast<const uint4*>(p));
    uint4 v;
    asm volatile("ld.global.cg.v4.u32 {%0, %1, %2, %3}, [%4];"
                 : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
                 : "l"(p)
                 : "memory");
    return v;
}
// Eight bytes where `take`, else 0, without a branch.
template <bool FRESH>
__device__ __forceinline__ uint64_t plane8_if(const uint8_t* p, bool take) {
    uint64_t v;
    if (FRESH)
        asm volatile("{.reg .pred q; setp.ne.u32 q, %2, 0; mov.u64 %0, 0;"
                     " @q ld.global.cg.u64 %0, [%1];}"
                     : "=l"(v)
                     : "l"(p), "r"((uint32_t)take)
                     : "memory");
    else
        asm volatile("{.reg .pred q; setp.ne.u32 q, %2, 0; mov.u64 %0, 0;"
                     " @q ld.global.nc.u64 %0, [%1];}"
                     : "=l"(v)
                     : "l"(p), "r"((uint32_t)take));
    return v;
}
template <bool FRESH>
__device__ __forceinline__ uint32_t plane1(const uint8_t* p) {
    if (!FRESH) return __ldg(p);
    uint32_t v;
    asm volatile("ld.global.cg.u8 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

// Byte-pair sums of a 4-byte word in two 16-bit lanes: [b0 + b1, b2 + b3].
__device__ __forceinline__ uint32_t pair_sums(uint32_t x) {
    return (x & 0x00FF00FFu) + ((x >> 8) & 0x00FF00FFu);
}

// The 2x2 sums of the 8x8 byte window at `off` of the plane src[0 .. total), in 16-bit lanes.
// A row's 8 bytes come from the aligned 16 around their start, and the next 8 where they reach
// past those (3 in 8, columns being even).  All rows' loads are in flight together: there is one
// branch, for the windows so close to an end of the plane that an aligned load might leave it.
// (With a branch and two 8-byte loads a row the rows waited for one another: with the f64 values
// as well, ten steps of 512 x 512 took 85 us, 47 now, of 4096 x 4096 417, 314 now.)
// Those windows' bytes are in flight together too: small planes have them in most warps.  (One after
// the other, a hundred steps of 64 x 64 took 821 us, and take 412.)
template <bool FRESH>
__device__ __forceinline__ void window_sums(const uint8_t* src, size_t off, int w, size_t total,
                                            uint32_t (&sums)[4][2]) {
    if (off >= 15 && off + 7 * (size_t)w + 24 <= total) {
        const uint8_t* p = src + off;
        uint4 x[8];
        uint64_t t[8];
#pragma unroll
        for (int r = 0; r < 8; ++r) {
            const uint8_t* q = p + (size_t)r * w;
            const unsigned s = (unsigned)(reinterpret_cast<uintptr_t>(q) & 15);
            x[r] = plane16<FRESH>(q - s);
            t[r] = plane8_if<FRESH>(q - s + 16, s > 8);
        }
#pragma unroll
        for (int r = 0; r < 8; ++r) {
            const unsigned s = (unsigned)(reinterpret_cast<uintptr_t>(p + (size_t)r * w) & 15);
            // The 24 bytes x | t from byte s on, in 32-bit funnel shifts.
            const bool up = s & 8, mid = s & 4;
            const uint32_t w0 = up ? x[r].z : x[r].x, w1 = up ? x[r].w : x[r].y;
            const uint32_t w2 = up ? (uint32_t)t[r] : x[r].z;
            const uint32_t w3 = up ? (uint32_t)(t[r] >> 32) : x[r].w;
            const uint32_t a = mid ? w1 : w0, b = mid ? w2 : w1, c = mid ? w3 : w2;
            const unsigned at = 8 * (s & 3);
            const uint32_t lo = pair_sums(__funnelshift_r(a, b, at));
            const uint32_t hi = pair_sums(__funnelshift_r(b, c, at));
            uint32_t(&to)[2] = sums[r / 2];
            to[0] = r & 1 ? to[0] + lo : lo;
            to[1] = r & 1 ? to[1] + hi : hi;
        }
        return;
    }
#pragma unroll
    for (int r = 0; r < 8; ++r) {
        uint64_t row = 0;
#pragma unroll
        for (int k = 0; k < 8; ++k)
            row |= (uint64_t)plane1<FRESH>(src + off + (size_t)r * w + k) << (8 * k);
        uint32_t(&to)[2] = sums[r / 2];
        to[0] = (r & 1 ? to[0] : 0u) + pair_sums((uint32_t)row);
        to[1] = (r & 1 ? to[1] : 0u) + pair_sums((uint32_t)(row >> 32));
    }
}

// Four values of the integer form, two to a word: the lanes' products stay below 2^15.
__device__ __forceinline__ uint32_t integer_values(const uint32_t (&sums)[2], uint32_t times,
                                                   uint32_t base) {
    const uint32_t a = __viaddmin_s16x2_relu(sums[0] * times, base, 0x3FFF3FFFu) >> 6;
    const uint32_t b = __viaddmin_s16x2_relu(sums[1] * times, base, 0x3FFF3FFFu) >> 6;
    return __byte_perm(a, b, 0x6420);
}

// Values in sample order (byte q of word p is sample (umin + p, vmin + q)) to output order:
// sample (p, q) is output pixel (a, b) with a = p (or 3 - p when u counts down) and b = q (or
// 3 - q when v counts down), transposed for isometries 1, 2, 6, 7.
__device__ __forceinline__ void to_output_order(int k, uint32_t (&rw)[4]) {
    const bool tr = (0xC6u >> k) & 1u, uneg = (0xACu >> k) & 1u, vneg = (0x9Au >> k) & 1u;
    if (vneg) {
#pragma unroll
        for (int p = 0; p < 4; ++p) rw[p] = __byte_perm(rw[p], 0, 0x0123);
    }
    if (uneg) {
        const uint32_t t0 = rw[0], t1 = rw[1];
        rw[0] = rw[3];
        rw[1] = rw[2];
        rw[2] = t1;
        rw[3] = t0;
    }
    if (tr) transpose4x4(rw[0], rw[1], rw[2], rw[3]);
}

// The first sample (umin, vmin) of a domain cell's 4x4, (x0, y0) the cell.
__device__ __forceinline__ void cell_sample(const DecodeMap& m, int x0, int y0, int* umin,
                                            int* vmin) {
    const IsoInv t = iso_inverse((int)((m.info >> 14) & 7u), (int)(m.info & 0xFFFu) - 1);
    const int i0 = y0 - (int)(m.rc & 0xFFFFu), j0 = x0 - (int)(m.rc >> 16);
    *umin = t.cu + t.ai * i0 + t.aj * j0 - 3 * ((t.ai < 0) | (t.aj < 0));
    *vmin = t.cv + t.bi * i0 + t.bj * j0 - 3 * ((t.bi < 0) | (t.bj < 0));
}

// The four output rows of a cell whose leaf reads no domain, from a loaded map.
__device__ __forceinline__ void still_rows(const DecodeMap& m, int x0, int y0, uint32_t (&rw)[4]) {
    if (((m.info >> 12) & 3u) == kLeafConst) {
        rw[0] = rw[1] = rw[2] = rw[3] = 0x01010101u * (m.info >> 24);
        return;
    }
    const int i0 = y0 - (int)(m.rc & 0xFFFFu), j0 = x0 - (int)(m.rc >> 16);
#pragma unroll
    for (int a = 0; a < 4; ++a) {
        rw[a] = 0u;
#pragma unroll
        for (int b = 0; b < 4; ++b) rw[a] |= affine_pixel(m, i0 + a, j0 + b) << (8 * b);
    }
}

// The four output rows of a domain or residual cell from its window's sums.
__device__ __forceinline__ void domain_rows(const DecodeMap& m, const uint32_t (&sums)[4][2],
                                            const double* __restrict__ resid, int umin, int vmin,
                                            uint32_t (&rw)[4]) {
    if (m.info & kLeafInteger) {
#pragma unroll
        for (int p = 0; p < 4; ++p) rw[p] = integer_values(sums[p], (uint32_t)m.n1, (uint32_t)m.n0);
    } else {
        const bool residual = ((m.info >> 12) & 3u) == kLeafResidual;
        const int S = (int)(m.info & 0xFFFu);
#pragma unroll
        for (int p = 0; p < 4; ++p) {
            rw[p] = 0u;
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const int sum = (int)((sums[p][q >> 1] >> (16 * (q & 1))) & 0xFFFFu);
                double value = domain_value(sum, m);
                if (residual)
                    value = __dadd_rn(value, __ldg(resid + m.roff + (umin + p) * S + vmin + q));
                rw[p] |= to_u8(value) << (8 * q);
            }
        }
    }
    to_output_order((int)((m.info >> 14) & 7u), rw);
}

__device__ __forceinline__ void store_rows(uint8_t* out, int w, int rows, const uint32_t (&rw)[4]) {
#pragma unroll
    for (int a = 0; a < 4; ++a)
        if (a < rows) *reinterpret_cast<uint32_t*>(out + (size_t)a * w) = rw[a];
}

// Largest byte of |a - b| over the cell's rows in the plane, b(row) the previous words.
template <class F>
__device__ __forceinline__ uint32_t rows_delta(const uint32_t (&rw)[4], int rows, F b) {
    uint32_t m = 0;
#pragma unroll
    for (int a = 0; a < 4; ++a)
        if (a < rows) m = __vmaxu4(m, __vabsdiffu4(rw[a], b(a)));
    return max(max(m & 255u, (m >> 8) & 255u), max((m >> 16) & 255u, m >> 24));
}

template <bool kStable>
__global__ void __launch_bounds__(128) decode_cell_kernel(
    const uint8_t* __restrict__ src, uint8_t* __restrict__ dst, int w, int h, int lg, int mw,
    const int32_t* __restrict__ owner, const DecodeMap* __restrict__ maps,
    const double* __restrict__ resid, StableState ss) {
    if (kStable && *ss.done) return;
    const int x0 = 4 * (blockIdx.x * blockDim.x + threadIdx.x);
    const int y0 = 4 * blockIdx.y;
    if (kStable && (x0 >= w || y0 >= h)) {
        fold_delta(0u, ss.delta);
        return;
    }
    if (x0 >= w || y0 >= h) return;
    const int32_t li = owner[(size_t)(y0 >> lg) * mw + (x0 >> lg)];
    uint32_t rw[4] = {0, 0, 0, 0};  // output rows, byte b of word a = pixel (y0 + a, x0 + b)
    if (li >= 0) {
        const DecodeMap m = maps[li];
        if (((m.info >> 12) & 3u) < kLeafDomain) {
            still_rows(m, x0, y0, rw);
        } else {
            int umin, vmin;
            cell_sample(m, x0, y0, &umin, &vmin);
            uint32_t sums[4][2] = {{0, 0}, {0, 0}, {0, 0}, {0, 0}};  // zero without a domain
            if (!(m.info & kLeafNoDomain))
                window_sums<false>(
                    src, ((size_t)(m.dom & 0xFFFFu) + 2 * umin) * w + (m.dom >> 16) + 2 * vmin, w,
                    (size_t)w * h, sums);
            domain_rows(m, sums, resid, umin, vmin, rw);
        }
    }
    const size_t at = (size_t)y0 * w + x0;
    store_rows(dst + at, w, h - y0, rw);
    if (kStable)
        fold_delta(rows_delta(rw, h - y0, [&](int a) {
            return *reinterpret_cast<const uint32_t*>(src + at + (size_t)a * w);
        }), ss.delta);
}

// ---- every step of a small plane's decode in one launch ----
//
// A step of a 512 x 512 plane is 16,384 cells: three dependent loads and a few dozen
// instructions a cell, less than the launch around them.  Here one cooperative launch runs all
// steps: a thread keeps its cell's leaf in registers, cells that read no domain are written to
// both buffers once, and the blocks meet at a counter between steps.  What is read was written by
// other SMs during the launch, so reads pass L1 by.  Bound: the counter's and the windows' round
// trips to L2.  One B200, ten steps of 512 x 512: 39 us, 46 us as launches; of 1024 x 1024: 48
// and 66.  Cooperative launches of several streams run one after the other, where the steps as
// launches overlap (three streams: 39 us a decode against 33), so a plan's run, which does not
// wait, keeps those; the calls that wait for the result take this one.  (One cluster of 16 blocks
// of 1,024 threads and its hardware barrier: 51 us, bound by the windows' bytes through 16 SMs.)

constexpr int kResidentThreads = 128;
struct ResidentArgs {
    uint8_t *buf0, *buf1;
    int w, h, lg, mw;
    const int32_t* owner;
    const DecodeMap* maps;
    const double* resid;
    uint32_t iters;
    uint32_t* sync;  // arrivals, blocks through
    int* delta;      // kStable: per step
    int threshold;
    int* state;
    int* err;
};

template <bool kStable>
__global__ void __launch_bounds__(kResidentThreads) decode_resident_kernel(const ResidentArgs g) {
    __shared__ int largest;
    const uint32_t cw = (uint32_t)g.w / 4, cells = cw * (((uint32_t)g.h + 3) / 4);
    const uint32_t c = blockIdx.x * blockDim.x + threadIdx.x;
    const int x0 = 4 * (int)(c % cw), y0 = 4 * (int)(c / cw);
    const bool in = c < cells;
    const int rows = in ? g.h - y0 : 0;
    const size_t at = (size_t)y0 * g.w + x0, total = (size_t)g.w * g.h;
    const int32_t li = in ? g.owner[(size_t)(y0 >> g.lg) * g.mw + (x0 >> g.lg)] : -1;
    DecodeMap m{};
    uint32_t rw[4] = {0, 0, 0, 0};
    bool moving = false;
    int umin = 0, vmin = 0;
    size_t off = 0;
    if (li >= 0) {
        m = g.maps[li];
        moving = ((m.info >> 12) & 3u) >= kLeafDomain;
        if (moving) {
            cell_sample(m, x0, y0, &umin, &vmin);
            off = ((size_t)(m.dom & 0xFFFFu) + 2 * umin) * g.w + (m.dom >> 16) + 2 * vmin;
        } else {
            still_rows(m, x0, y0, rw);
        }
    }
    // Step 0 reads 128 everywhere.
    uint32_t before[4] = {0x80808080u, 0x80808080u, 0x80808080u, 0x80808080u};
    uint32_t target = 0;
    uint32_t used = 0;
    for (uint32_t it = 0; it < g.iters; ++it) {
        if (moving) {
            uint32_t sums[4][2];
#pragma unroll
            for (int p = 0; p < 4; ++p)
                sums[p][0] = sums[p][1] = m.info & kLeafNoDomain ? 0u : 0x02000200u;
            if (it > 0 && !(m.info & kLeafNoDomain))
                window_sums<true>(it & 1 ? g.buf1 : g.buf0, off, g.w, total, sums);
            domain_rows(m, sums, g.resid, umin, vmin, rw);
        }
        if (moving || it < 2) store_rows((it & 1 ? g.buf0 : g.buf1) + at, g.w, rows, rw);
        if (kStable) {
            fold_delta(rows_delta(rw, rows, [&](int a) { return before[a]; }), g.delta + it);
#pragma unroll
            for (int a = 0; a < 4; ++a) before[a] = rw[a];
        }
        if (!kStable && it + 1 == g.iters) break;
        target += gridDim.x;
        grid_meet(g.sync, target, g.err);
        if (kStable) {
            if (threadIdx.x == 0) largest = *(volatile int*)(g.delta + it);
            __syncthreads();
            if (largest <= g.threshold) {
                used = it + 1;
                break;
            }
            __syncthreads();  // everybody has read it
        }
    }
    if (kStable && blockIdx.x == 0 && threadIdx.x == 0 && used) {
        g.state[0] = 1;
        g.state[1] = (int)used;
    }
    grid_leave(g.sync);
}

// After step `iter`: the first step whose delta met the threshold ends the decode.
__global__ void decode_converged_kernel(const int* __restrict__ delta, int threshold, int iter,
                                    int* __restrict__ done, int* __restrict__ used) {
    if (!*done && *delta <= threshold) {
        *done = 1;
        *used = iter + 1;
    }
}

// ---- source-ordered decode of planes larger than L2 (decode_sorted_*) ----
//
// Gathering cell by cell in output order reads each cell's 8x8 domain window from a random
// place of the previous iterate; once the plane no longer fits in L2, every 8-byte row read
// costs whole DRAM sectors.  The source-ordered form splits a step in two:
//   gather : the domain cells in the order of their windows' source rows (a list built once
//            per leaf list), each computing its 16 output bytes into a cell buffer; the
//            windows of cells running together lie in a narrow band of source rows, which
//            L2 keeps, so the plane is read about once;
//   place  : every output cell in output order, copying its 16 bytes from the cell buffer
//            (domain cells) or computing them (constant and affine cells), four coalesced
//            4-byte row stores.
// The values are the cell kernel's, operation for operation.  Maps with mode-3 residuals keep
// the cell kernel.

__device__ __forceinline__ bool is_domain_cell(const DecodeMap& m) {
    return ((m.info >> 12) & 3u) == kLeafDomain;
}

// Pass 1 of the list build: the domain cells of each source row.
__global__ void sorted_count_kernel(int w, int h, int lg, int mw, const int32_t* __restrict__ owner,
                                    const DecodeMap* __restrict__ maps,
                                    uint32_t* __restrict__ row_count, uint32_t* __restrict__ wide) {
    const int cw = w / 4, chh = (h + 3) / 4;
    const long long c = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= (long long)cw * chh) return;
    const int x0 = 4 * (int)(c % cw), y0 = 4 * (int)(c / cw);
    const int32_t li = owner[(size_t)(y0 >> lg) * mw + (x0 >> lg)];
    if (li < 0) return;
    const DecodeMap m = maps[li];
    if (!is_domain_cell(m)) return;
    int umin, vmin;
    cell_sample(m, x0, y0, &umin, &vmin);
    atomicAdd(&row_count[(m.dom & 0xFFFFu) + 2 * umin], 1u);
    if (!(m.info & kLeafInteger)) *wide = 1u;
}

// Exclusive scan of the row counts (one block): the first list slot of each source row, and
// in cursor[h] the total.
__global__ void sorted_scan_kernel(const uint32_t* __restrict__ row_count, int h,
                                   uint32_t* __restrict__ cursor) {
    __shared__ uint32_t carry;
    __shared__ uint32_t warp_tot[32];
    if (threadIdx.x == 0) carry = 0;
    __syncthreads();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    for (int base = 0; base < h; base += blockDim.x) {
        const int i = base + threadIdx.x;
        const uint32_t v = i < h ? row_count[i] : 0u;
        uint32_t x = v;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= o) x += y;
        }
        if (lane == 31) warp_tot[warp] = x;
        __syncthreads();
        uint32_t before = carry;
        for (int k = 0; k < warp; ++k) before += warp_tot[k];
        if (i < h) cursor[i] = before + x - v;
        __syncthreads();
        if (threadIdx.x == 0) {
            uint32_t all = 0;
            for (int k = 0; k < nw; ++k) all += warp_tot[k];
            carry += all;
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) cursor[h] = carry;  // the number of domain cells
}

// Pass 2: the jobs, eight threads a leaf.  A thread takes a row of the leaf's windows and gives
// its cells (those the leaf still owns) neighbouring slots, in the order of their windows: lanes
// that run together then read one line of the plane where the leaf is wider than a cell, and the
// place pass finds the leaf's cells side by side.  (With a slot for each cell as
// it came, ten steps of 8192 x 8192 took 1,152 us, so 1,110.)
// A job is 8 bytes when every leaf has the integer form (window offset; A | isometry << 8 |
// base << 16), else 16 (window offset; qalfa | isometry << 24; beta).
__global__ void sorted_scatter_kernel(int w, int lg, int mw, const int32_t* __restrict__ owner,
                                      const DecodeMap* __restrict__ maps,
                                      const DecodeLeaf* __restrict__ leaves, int nleaves,
                                      uint32_t* __restrict__ cursor,
                                      const uint32_t* __restrict__ wide,
                                      uint4* __restrict__ jobs, uint32_t* __restrict__ inv) {
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const int li = (int)(t / 8);
    if (li >= nleaves) return;
    const DecodeMap m = maps[li];
    if (!is_domain_cell(m)) return;
    const int S = (int)(m.info & 0xFFFu), k = (int)((m.info >> 14) & 7u);
    const int row = (int)(m.rc & 0xFFFFu), col = (int)(m.rc >> 16);
    const bool tr = (0xC6u >> k) & 1u, uneg = (0xACu >> k) & 1u, vneg = (0x9Au >> k) & 1u;
    const bool big = *wide;
    for (int u = 4 * (int)(t % 8); u < S; u += 32) {
        const int du = uneg ? S - 4 - u : u;
        // The 4x4 of samples (u, v) is the output cell at this position in the leaf.
        auto cell = [&](int v, int* x0, int* y0) {
            const int dv = vneg ? S - 4 - v : v;
            *y0 = row + (tr ? dv : du);
            *x0 = col + (tr ? du : dv);
        };
        uint32_t held = 0;
        for (int v = 0; v < S; v += 4) {
            int x0, y0;
            cell(v, &x0, &y0);
            held += owner[(size_t)(y0 >> lg) * mw + (x0 >> lg)] == li;
        }
        if (!held) continue;
        const uint32_t from = (m.dom & 0xFFFFu) + 2 * u;
        uint32_t pos = atomicAdd(&cursor[from], held);
        for (int v = 0; v < S; v += 4) {
            int x0, y0;
            cell(v, &x0, &y0);
            if (owner[(size_t)(y0 >> lg) * mw + (x0 >> lg)] != li) continue;
            const uint32_t off = (uint32_t)((size_t)from * w + (m.dom >> 16) + 2 * v);
            if (big)
                jobs[pos] = make_uint4(off, (leaves[li].w & 0x1FFFFu) | (uint32_t)k << 24,
                                       (uint32_t)__double2loint(m.b), (uint32_t)__double2hiint(m.b));
            else
                reinterpret_cast<uint2*>(jobs)[pos] =
                    make_uint2(off, (uint32_t)m.n1 | (uint32_t)k << 8 | (uint32_t)m.n0 << 16);
            inv[(size_t)(y0 / 4) * (w / 4) + x0 / 4] = pos++;
        }
    }
}

// Gather pass: job -> the cell's 16 output bytes (row-major 4x4) in the cell buffer.  Bound by
// L1: every row of a window is a line of its own.  8192 x 8192 on one B200: 74 us, with two
// 8-byte loads a row, f64 values and 16-byte jobs 84 us.
template <bool kWide>
__global__ void __launch_bounds__(128) sorted_gather_kernel(
    const uint8_t* __restrict__ src, size_t total, int w, const uint4* __restrict__ jobs,
    uint32_t n, DecodeConsts cst, uint4* __restrict__ cellbuf) {
    const uint32_t pos = blockIdx.x * blockDim.x + threadIdx.x;
    if (pos >= n) return;
    uint32_t sums[4][2], rw[4];
    int k;
    if (kWide) {
        const uint4 jb = jobs[pos];
        k = (int)(jb.y >> 24);
        DecodeMap m{};
        m.info = kLeafDomain << 12 | (uint32_t)k << 14;
        // decode_expand's a = alfa / 4, alfa = (qalfa / 2^bits_alfa) * max_alfa (ifs.rs:434-439).
        m.a = __dmul_rn(__dmul_rn(__ddiv_rn((double)(jb.y & 0x1FFFFu), cst.alfa_den), cst.max_alfa), 0.25);
        m.b = __hiloint2double((int)jb.w, (int)jb.z);
        window_sums<false>(src, jb.x, w, total, sums);
        domain_rows(m, sums, nullptr, 0, 0, rw);
    } else {
        const uint2 jb = reinterpret_cast<const uint2*>(jobs)[pos];
        k = (int)(jb.y >> 8 & 7u);
        window_sums<false>(src, jb.x, w, total, sums);
#pragma unroll
        for (int p = 0; p < 4; ++p)
            rw[p] = integer_values(sums[p], jb.y & 63u, __byte_perm(jb.y, 0, 0x3232));
        to_output_order(k, rw);
    }
    cellbuf[pos] = make_uint4(rw[0], rw[1], rw[2], rw[3]);
}

// Place pass: every 4x4 output cell in output order.
__global__ void __launch_bounds__(128) sorted_place_kernel(
    uint8_t* __restrict__ dst, int w, int h, int lg, int mw, const int32_t* __restrict__ owner,
    const DecodeMap* __restrict__ maps, const uint32_t* __restrict__ inv,
    const uint4* __restrict__ cellbuf) {
    const int x0 = 4 * (blockIdx.x * blockDim.x + threadIdx.x);
    const int y0 = 4 * blockIdx.y;
    if (x0 >= w || y0 >= h) return;
    const int32_t li = owner[(size_t)(y0 >> lg) * mw + (x0 >> lg)];
    uint32_t rw[4] = {0, 0, 0, 0};
    if (li >= 0) {
        const DecodeMap m = maps[li];
        const uint32_t kind = (m.info >> 12) & 3u;
        if (kind == kLeafDomain) {
            const uint4 v = cellbuf[inv[(size_t)(y0 / 4) * (w / 4) + x0 / 4]];
            rw[0] = v.x;
            rw[1] = v.y;
            rw[2] = v.z;
            rw[3] = v.w;
        } else {
            still_rows(m, x0, y0, rw);
        }
    }
    store_rows(dst + (size_t)y0 * w + x0, w, h - y0, rw);
}

}  // namespace

size_t decode_sorted_cells(int w, int h) { return (size_t)(w / 4) * ((h + 3) / 4); }

cudaError_t launch_decode_expand(const DecodeLeaf* leaves, const int32_t* resid_off, int n,
                                 DecodeConsts c, DecodeMap* maps, cudaStream_t st) {
    if (n <= 0) return cudaSuccess;
    decode_expand_kernel<<<(n + 255) / 256, 256, 0, st>>>(leaves, resid_off, n, c, maps);
    return cudaGetLastError();
}

cudaError_t launch_residual_values(const DecodeLeaf* leaves, const int32_t* resid_off, int n,
                                   const int32_t* levels, const ResidualBases& bases, uint32_t most,
                                   double step, double* values, cudaStream_t st) {
    if (n <= 0) return cudaSuccess;
    if (most > kResidualMost) return cudaErrorInvalidValue;
    const size_t smem = 2 * (size_t)most * most * sizeof(double);
    cudaError_t e = cudaFuncSetAttribute(residual_values_kernel,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)(2 * kResidualMost * kResidualMost * sizeof(double)));
    if (e != cudaSuccess) return e;
    residual_values_kernel<<<n, 128, smem, st>>>(leaves, resid_off, levels, bases, step, values);
    return cudaGetLastError();
}

cudaError_t launch_decode_step(const uint8_t* src, uint8_t* dst, int w, int h, int lg,
                               const int32_t* owner, const DecodeMap* maps, const double* resid,
                               cudaStream_t st) {
    const int mw = (w + (1 << lg) - 1) >> lg;
    const bool aligned =
        ((reinterpret_cast<uintptr_t>(src) | reinterpret_cast<uintptr_t>(dst)) & 7) == 0;
    const StableState none{nullptr, nullptr};
    if (lg >= 2 && (w % 4) == 0 && aligned) {
        dim3 grid((w / 4 + 127) / 128, (h + 3) / 4);
        decode_cell_kernel<false><<<grid, 128, 0, st>>>(src, dst, w, h, lg, mw, owner, maps, resid,
                                                        none);
    } else {
        dim3 grid((w + 255) / 256, h);
        decode_pixel_kernel<false><<<grid, 256, 0, st>>>(src, dst, w, h, lg, mw, owner, maps,
                                                         resid, none);
    }
    return cudaGetLastError();
}

bool decode_output_aligned(const uint8_t* out) { return (reinterpret_cast<uintptr_t>(out) & 7) == 0; }

cudaError_t decode_set_output(cudaGraphExec_t exec, cudaGraphNode_t last, bool sorted, uint8_t* out) {
    cudaKernelNodeParams k;
    cudaError_t e = cudaGraphKernelNodeGetParams(last, &k);
    if (e != cudaSuccess) return e;
    // sorted_place_kernel's nine parameters begin with the output; the step kernels' ten have it
    // second.
    void* params[10];
    const int n = sorted ? 9 : 10;
    for (int i = 0; i < n; ++i) params[i] = k.kernelParams[i];
    params[sorted ? 0 : 1] = &out;
    k.kernelParams = params;
    return cudaGraphExecKernelNodeSetParams(exec, last, &k);
}

static size_t resident_blocks(int w, int h) {
    return (decode_sorted_cells(w, h) + kResidentThreads - 1) / kResidentThreads;
}

// Every block must be resident at once, and the counter must not reach its top bit.  Up to four
// blocks an SM (1.2 Mpixel): ten steps of 1024 x 1024 take 48 us here and 66 as launches, but of
// 1280 x 1280, 800 blocks polling one counter, 150 against 99.
bool decode_resident_fits(const uint8_t* buf0, const uint8_t* buf1, int w, int h, int lg,
                          uint32_t iters, int num_sms) {
    const bool aligned =
        ((reinterpret_cast<uintptr_t>(buf0) | reinterpret_cast<uintptr_t>(buf1)) & 7) == 0;
    const size_t blocks = resident_blocks(w, h);
    return lg >= 2 && w % 4 == 0 && aligned && iters > 0 && blocks <= (size_t)num_sms * 4 &&
           (uint64_t)blocks * iters < (1ull << 31);
}

cudaError_t launch_decode_resident(uint8_t* buf0, uint8_t* buf1, int w, int h, int lg,
                                   const int32_t* owner, const DecodeMap* maps,
                                   const double* resid, uint32_t iters, uint32_t* sync, int* delta,
                                   int threshold, int* state, int* err, int num_sms,
                                   cudaStream_t st, bool* taken) {
    *taken = false;
    if (!decode_resident_fits(buf0, buf1, w, h, lg, iters, num_sms)) return cudaSuccess;
    const size_t blocks = resident_blocks(w, h);
    ResidentArgs g{buf0, buf1, w, h, lg, (w + (1 << lg) - 1) >> lg, owner, maps, resid, iters,
                   sync, delta, threshold, state, err};
    const void* kernel = delta ? (const void*)decode_resident_kernel<true>
                               : (const void*)decode_resident_kernel<false>;
    int per_sm = 0;
    cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, kResidentThreads, 0);
    if (e != cudaSuccess) return e;
    if (blocks > (size_t)num_sms * per_sm) return cudaSuccess;
    void* args[] = {&g};
    e = cudaLaunchCooperativeKernel(kernel, dim3((unsigned)blocks), dim3(kResidentThreads), args, 0,
                                    st);
    if (e == cudaErrorCooperativeLaunchTooLarge) {  // fewer SMs than the device has
        cudaGetLastError();
        return cudaSuccess;
    }
    *taken = e == cudaSuccess;
    return e;
}

cudaError_t launch_decode_step_stable(const uint8_t* src, uint8_t* dst, int w, int h, int lg,
                                      const int32_t* owner, const DecodeMap* maps,
                                      const double* resid, const int* done, int* delta,
                                      int threshold, int iter, int* done_w, int* used,
                                      cudaStream_t st) {
    const int mw = (w + (1 << lg) - 1) >> lg;
    const bool aligned =
        ((reinterpret_cast<uintptr_t>(src) | reinterpret_cast<uintptr_t>(dst)) & 7) == 0;
    const StableState ss{done, delta};
    if (lg >= 2 && (w % 4) == 0 && aligned) {
        dim3 grid((w / 4 + 127) / 128, (h + 3) / 4);
        decode_cell_kernel<true><<<grid, 128, 0, st>>>(src, dst, w, h, lg, mw, owner, maps, resid,
                                                       ss);
    } else {
        dim3 grid((w + 255) / 256, h);
        decode_pixel_kernel<true><<<grid, 256, 0, st>>>(src, dst, w, h, lg, mw, owner, maps,
                                                        resid, ss);
    }
    decode_converged_kernel<<<1, 1, 0, st>>>(delta, threshold, iter, done_w, used);
    return cudaGetLastError();
}


bool decode_sorted_eligible(int w, int h, int lg, bool residuals) {
    return lg >= 2 && (w % 4) == 0 && !residuals && w > 0 && h > 0;
}

cudaError_t launch_decode_sorted_build(int w, int h, int lg, const int32_t* owner,
                                       const DecodeMap* maps, const DecodeLeaf* leaves, int nleaves,
                                       uint32_t* row_count, uint32_t* cursor, uint4* jobs,
                                       uint32_t* inv, cudaStream_t st) {
    const int mw = (w + (1 << lg) - 1) >> lg;
    const size_t cells = decode_sorted_cells(w, h);
    uint32_t* wide = cursor + h + 1;
    cudaError_t e = cudaMemsetAsync(row_count, 0, (size_t)h * 4, st);
    if (e == cudaSuccess) e = cudaMemsetAsync(wide, 0, 4, st);
    if (e != cudaSuccess) return e;
    sorted_count_kernel<<<(unsigned)((cells + 255) / 256), 256, 0, st>>>(w, h, lg, mw, owner, maps,
                                                                         row_count, wide);
    sorted_scan_kernel<<<1, 1024, 0, st>>>(row_count, h, cursor);
    sorted_scatter_kernel<<<(unsigned)(((size_t)nleaves * 8 + 255) / 256), 256, 0, st>>>(
        w, lg, mw, owner, maps, leaves, nleaves, cursor, wide, jobs, inv);
    return cudaGetLastError();
}

bool decode_sorted_aligned(const uint8_t* dst) {
    return (reinterpret_cast<uintptr_t>(dst) & 3) == 0;
}

cudaError_t launch_decode_sorted_step(const uint8_t* src, uint8_t* dst, int w, int h, int lg,
                                      const int32_t* owner, const DecodeMap* maps,
                                      const uint4* jobs, uint32_t njobs, bool wide_jobs,
                                      const uint32_t* inv, DecodeConsts c, uint4* cellbuf,
                                      cudaStream_t st) {
    if (!decode_sorted_aligned(dst)) return cudaErrorInvalidValue;
    const int mw = (w + (1 << lg) - 1) >> lg;
    if (njobs) {
        const auto gather = wide_jobs ? sorted_gather_kernel<true> : sorted_gather_kernel<false>;
        gather<<<(njobs + 127) / 128, 128, 0, st>>>(src, (size_t)w * h, w, jobs, njobs, c, cellbuf);
    }
    dim3 grid((w / 4 + 127) / 128, (h + 3) / 4);
    sorted_place_kernel<<<grid, 128, 0, st>>>(dst, w, h, lg, mw, owner, maps, inv, cellbuf);
    return cudaGetLastError();
}

}  // namespace mars

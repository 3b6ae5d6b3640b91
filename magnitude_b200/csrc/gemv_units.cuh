// Device building blocks of the streaming projection kernel: the fixed-point activation image, the
// conversion into it, and the per-type work on one 256-weight record of sixteen weight rows.
#pragma once

#include "common.cuh"

namespace b200q {

// where an activation matrix lives (row m at x + m * ldx elements)
struct XSrc {
    const void *x;
    long long ldx;
    int x_is_bf16;
    int x_vec_ok;       // rows are 16-byte aligned: vector loads allowed
    int K, Kpad;
    const float *gamma; // RMSNorm weight [K] applied on the load (with `rs`), or null
    float rs;           // 1 / sqrt(mean(x^2) + eps) of the row being converted
};

// ---------------------------------------------------------------------------------------------
// The activation image
//
// An activation row is converted once per job into 16-bit fixed point: per block of 32 elements one fp32
// scale sx and per element two signed bytes, x ~= sx * (256 * hi + lo) with lo in [-128, 127] (relative step
// 2^-15 of the block's largest).  The image of a row is one record per 256 elements:
//
//   bytes 0..511   eight blocks of [hi: 32][lo: 32], elements in order
//   then           the blocks' scales sx and, per weight sub-block, isum: the int32 sum of its 16-bit integers
//                  types with 32-weight sub-blocks (64 bytes)  [c = 0..3][(sx, isum) of sub-block c, of sub-block c + 4]
//                  Q6_K, 16-weight sub-blocks (96 bytes)       [sx: 8], then [c = 0..3][isum of sub-block 8 (c / 2) + 2 q + (c & 1), q = 0..3]
//
// so that lane group c of a warp (see WRec) finds the scales of the sub-blocks it finishes side by side.
// ---------------------------------------------------------------------------------------------
constexpr int kXBytes = 512;
__host__ __device__ constexpr int ximg_rec_bytes(int qt) { return qt == QT_Q6_K ? kXBytes + 96 : kXBytes + 64; }

// ---------------------------------------------------------------------------------------------
// Weights: one record of sixteen rows per warp and step, multiplied with integer tensor-core instructions
//
// mma.m16n8k32 takes sixteen weight rows as A (levels as bytes) and eight columns as B.  One activation row
// needs only its two byte planes, so the columns also tell four sub-blocks apart: column 2 s + part holds plane
// `part` of sub-block s of the current set of four and zeros elsewhere in K.  After the record's eight MMAs the
// accumulators are the integer sums of every (row, sub-block, plane): no scale enters before that, nothing has to
// be multiplied per weight, and lane group c (= lane & 3) holds (hi, lo) of sub-block c of every set.  What a
// weight costs is its unpacking (two logic operations per eight weights of Q4_K); dp4a, at half rate and four
// weights per instruction and plane, used to cost four more.  (Sums from such accumulators through a biased fp32
// number instead of an int-to-float conversion were a little slower.)
//
// Shared memory order of K is free: A takes whatever 16 bytes lane group c loads, B the activation bytes of the
// same positions.  B load l (of four, two MMAs each) of lane (n = lane >> 2, kc = lane & 3) reads 16 bytes of
// the image or, where lane group kc's weights do not belong to the column's sub-block, of a zero area.
// ---------------------------------------------------------------------------------------------

// what a lane knows about the activation image: addresses of its B loads
struct XLane {
    uint32_t base[2];     // even / odd loads
    int step[2];          // bytes per record (0 in the zero area)
    uint32_t xs;          // scales and sums of lane group c: (sx, isum) pairs, Q6_K the four sx (the sums follow, see XScales)
};

template <int QT> constexpr bool kNibbleHalves = QT == QT_Q4_K || QT == QT_Q5_K || QT == QT_Q4_0;
template <int QT> constexpr int kSets = QT == QT_Q6_K ? 4 : 2;      // sets of four sub-blocks in a record

// byte offset of B load l from the lane's base address
template <int QT> __device__ __forceinline__ constexpr int bload_off(int l) {
    return QT == QT_Q6_K ? 64 * l : kNibbleHalves<QT> ? 256 * (l >> 1) : 256 * (l >> 1) + 16 * (l & 1);
}

// (run-time type: once per job; parity: the lowest bit of the record numbers the warp works on)
__device__ __forceinline__ XLane xlane(int qt, uint32_t img, uint32_t zero, int lane, int parity) {
    const int n = lane >> 2, kc = lane & 3, part = n & 1;
    XLane x;
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        bool mine;
        uint32_t off;
        if (qt == QT_Q6_K) {                    // lane group kc: half kc / 2, positions 16 (kc & 1).. of every quadrant
            mine = (n >> 1) == kc;
            off = 256 * (kc >> 1) + 32 * part + 16 * (kc & 1);
        } else if (qt == QT_Q8_0 || qt == QT_MXFP4) {      // blocks kc and kc + 4
            mine = (n >> 1) == kc;
            off = 64 * kc + 32 * part;
        } else {                                // 16-byte pieces kc and kc + 4 of the nibbles: half of a sub-block pair
            mine = (n >> 2) == (kc >> 1) && ((n >> 1) & 1) == i;
            off = 64 * (2 * (kc >> 1) + i) + 32 * part + 16 * (kc & 1);
        }
        // (the zero 16 bytes lie in the banks that the other lanes of the load do not touch: records alternate by 64 bytes)
        x.base[i] = mine ? img + off : zero + 64 * ((1 - i) ^ parity);
        x.step[i] = mine ? ximg_rec_bytes(qt) : 0;
    }
    x.xs = img + kXBytes + 16 * (qt == QT_Q6_K ? kc >> 1 : kc);
    return x;
}

// d = a . b (first of a set) and d += a . b, a unsigned or (Q8_0) signed bytes
template <bool SIGNED> __device__ __forceinline__ void imma(int (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1, bool first) {
    const int c0 = first ? 0 : d[0], c1 = first ? 0 : d[1], c2 = first ? 0 : d[2], c3 = first ? 0 : d[3];
    if (SIGNED)
        asm("mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%10, %11, %12, %13};"
            : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3])
            : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "r"(c0), "r"(c1), "r"(c2), "r"(c3));
    else
        asm("mma.sync.aligned.m16n8k32.row.col.s32.u8.s8.s32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%10, %11, %12, %13};"
            : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3])
            : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "r"(c0), "r"(c1), "r"(c2), "r"(c3));
}

// One record of one weight row as lane group c sees it, as loaded.  load(): `rec` = shared address of the record, `doff` =
// of its d (Q6_K).  words(): the A words of the two MMAs of B load l (two each).  s.finish(): the row's share from the
// integer sums v of the lane's sub-block of every set.
template <int QT> struct WRec;

// half c (0..3) / c + 4 of the eight fp16 in `dd`
__device__ __forceinline__ float half_lo(const uint4 &dd, int c) { return half_bits_to_float(((c & 2) ? dd.y : dd.x) >> (16 * (c & 1))); }
__device__ __forceinline__ float half_hi(const uint4 &dd, int c) { return half_bits_to_float(((c & 2) ? dd.w : dd.z) >> (16 * (c & 1))); }

// Q4_K header: scales and mins of sub-blocks c and c + 4 are in byte c of the three scale words
struct KHeader {
    uint4 hdr;
    __device__ __forceinline__ float finish_k(int v0, int v1, int c, const uint4 &xs) const {
        const int s = 8 * c;
        const uint32_t y = hdr.y >> s, z = hdr.z >> s, w = hdr.w >> s;
        const int sc0 = y & 63, mn0 = z & 63;
        const int sc1 = (w & 15) | ((y >> 2) & 0x30), mn1 = ((w >> 4) & 15) | ((z >> 2) & 0x30);
        const float d = half_bits_to_float(hdr.x), dmin = half_bits_to_float(hdr.x >> 16);
        const float f0 = (float)(v0 * sc0), f1 = (float)(v1 * sc1);
        const float u0 = (float)(mn0 * (int)xs.y), u1 = (float)(mn1 * (int)xs.w);
        return __uint_as_float(xs.x) * (d * f0 - dmin * u0) + __uint_as_float(xs.z) * (d * f1 - dmin * u1);
    }
};

template <> struct WRec<QT_Q4_K> {
    struct Scales : KHeader {
        __device__ __forceinline__ float finish(const int (&v)[2], int c, const uint4 *xs) const {
            const int sh = 4 * (c & 1);        // odd sub-blocks are the high nibbles: 16 x leaves the sum here
            return finish_k(v[0] >> sh, v[1] >> sh, c, xs[0]);
        }
    } s;
    uint4 q[2];
    __device__ __forceinline__ void load(uint32_t rec, uint32_t, int c) {
        q[0] = lds128(rec + 16 + 16 * c);
        q[1] = lds128(rec + 80 + 16 * c);
        s.hdr = lds128(rec);
    }
    __device__ __forceinline__ void words(int l, int, uint32_t (&w)[4]) const {
#pragma unroll
        for (int i = 0; i < 4; ++i) w[i] = word_of(q[l >> 1], i) & ((l & 1) ? 0xF0F0F0F0u : 0x0F0F0F0Fu);      // high: 16 x level
    }
};

// Q5_K record on the device: the Q4_K fields, then the 32 bytes of fifth bits (bit s of byte l belongs
// to weight l of sub-block s)
template <> struct WRec<QT_Q5_K> {
    struct Scales : KHeader {
        __device__ __forceinline__ float finish(const int (&v)[2], int c, const uint4 *xs) const { return finish_k(v[0], v[1], c, xs[0]); }
    } s;
    uint4 q[2], h;
    __device__ __forceinline__ void load(uint32_t rec, uint32_t, int c) {
        q[0] = lds128(rec + 16 + 16 * c);
        q[1] = lds128(rec + 80 + 16 * c);
        h = lds128(rec + 144 + 16 * (c & 1));
        s.hdr = lds128(rec);
    }
    __device__ __forceinline__ void words(int l, int c, uint32_t (&w)[4]) const {
        const int sub = 4 * (l >> 1) + (c & 2) + (l & 1);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const uint32_t n = (l & 1) ? word_of(q[l >> 1], i) >> 4 : word_of(q[l >> 1], i);
            w[i] = (n & 0x0F0F0F0Fu) | (((word_of(h, i) >> sub) << 4) & 0x10101010u);
        }
    }
};

// Q4_0 record on the device: the eight fp16 d of its native blocks, then the nibbles in the Q4_K
// arrangement; w = d (q - 8), so a block's dot is d (sum q x - 8 sum x) with both sums integers.
template <> struct WRec<QT_Q4_0> {
    struct Scales {
        uint4 dd;
        __device__ __forceinline__ float finish(const int (&v)[2], int c, const uint4 *xs) const {
            const int sh = 4 * (c & 1);
            const float f0 = (float)((v[0] >> sh) - 8 * (int)xs[0].y), f1 = (float)((v[1] >> sh) - 8 * (int)xs[0].w);
            return __uint_as_float(xs[0].x) * (half_lo(dd, c) * f0) + __uint_as_float(xs[0].z) * (half_hi(dd, c) * f1);
        }
    } s;
    uint4 q[2];
    __device__ __forceinline__ void load(uint32_t rec, uint32_t, int c) {
        q[0] = lds128(rec + 16 + 16 * c);
        q[1] = lds128(rec + 80 + 16 * c);
        s.dd = lds128(rec);
    }
    __device__ __forceinline__ void words(int l, int, uint32_t (&w)[4]) const {
#pragma unroll
        for (int i = 0; i < 4; ++i) w[i] = word_of(q[l >> 1], i) & ((l & 1) ? 0xF0F0F0F0u : 0x0F0F0F0Fu);
    }
};

// MXFP4 record on the device: the eight scale bytes of its native blocks (16 bytes with padding), then per
// block four words of eight e2m1 codes in weight order.  A look-up turns four codes into the bytes
// 64 + value, so a block's dot is 2^(e - 128) (sum b x - 64 sum x) with both sums integers.
template <> struct WRec<QT_MXFP4> {
    struct Scales {
        uint2 ee;
        __device__ __forceinline__ float finish(const int (&v)[2], int c, const uint4 *xs) const {
            const float d0 = __uint_as_float(e8m0_half_bits((ee.x >> (8 * c)) & 0xFF)), d1 = __uint_as_float(e8m0_half_bits((ee.y >> (8 * c)) & 0xFF));
            const float f0 = (float)(v[0] - 64 * (int)xs[0].y), f1 = (float)(v[1] - 64 * (int)xs[0].w);
            return __uint_as_float(xs[0].x) * (d0 * f0) + __uint_as_float(xs[0].z) * (d1 * f1);
        }
    } s;
    uint4 q[2];
    __device__ __forceinline__ void load(uint32_t rec, uint32_t, int c) {
        q[0] = lds128(rec + 16 + 16 * c);
        q[1] = lds128(rec + 80 + 16 * c);
        s.ee = lds64(rec);
    }
    __device__ __forceinline__ void words(int l, int, uint32_t (&w)[4]) const {
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const uint32_t codes = word_of(q[l >> 1], 2 * (l & 1) + i);
            w[2 * i] = mxfp4_bytes(codes);
            w[2 * i + 1] = mxfp4_bytes(codes >> 16);
        }
    }
};

template <> struct WRec<QT_Q8_0> {
    struct Scales {
        uint4 dd;
        __device__ __forceinline__ float finish(const int (&v)[2], int c, const uint4 *xs) const {
            return (half_lo(dd, c) * __uint_as_float(xs[0].x)) * (float)v[0] + (half_hi(dd, c) * __uint_as_float(xs[0].z)) * (float)v[1];
        }
    } s;
    uint4 q[4];
    __device__ __forceinline__ void load(uint32_t rec, uint32_t, int c) {
#pragma unroll
        for (int l = 0; l < 4; ++l) q[l] = lds128(rec + 32 * c + 128 * (l >> 1) + 16 * (l & 1));
        s.dd = lds128(rec + 256);          // the eight d
    }
    __device__ __forceinline__ void words(int l, int, uint32_t (&w)[4]) const {
#pragma unroll
        for (int i = 0; i < 4; ++i) w[i] = word_of(q[l], i);
    }
};

// lane group c: half c / 2 of the record, positions 16 (c & 1).. of each of the half's four 32-weight quadrants
template <> struct WRec<QT_Q6_K> {
    struct Scales {
        uint2 s8;            // the half's eight int8 scales
        uint32_t d16;
        __device__ __forceinline__ float finish(const int (&v)[4], int c, const uint4 *xs) const {
            const int ph = 8 * (c & 1);
            const uint32_t s0 = s8.x >> ph, s1 = s8.y >> ph;       // scales of sub-blocks 8 half + 2 q + (c & 1)
            const float d = half_bits_to_float(d16);
            float r = (d * (float)(int)(int8_t)s0 * __uint_as_float(xs[0].x)) * (float)(v[0] - 32 * (int)xs[1].x);
            r += (d * (float)(int)(int8_t)(s0 >> 16) * __uint_as_float(xs[0].y)) * (float)(v[1] - 32 * (int)xs[1].y);
            r += (d * (float)(int)(int8_t)s1 * __uint_as_float(xs[0].z)) * (float)(v[2] - 32 * (int)xs[1].z);
            r += (d * (float)(int)(int8_t)(s1 >> 16) * __uint_as_float(xs[0].w)) * (float)(v[3] - 32 * (int)xs[1].w);
            return r;
        }
    } s;
    uint4 a, b, h;           // low nibbles of quadrants 0 | 2 and 1 | 3, two high bits of all four
    __device__ __forceinline__ void load(uint32_t rec, uint32_t doff, int c) {
        const uint32_t at = rec + 64 * (c >> 1) + 16 * (c & 1);
        a = lds128(at);
        b = lds128(at + 32);
        h = lds128(rec + 128 + 32 * (c >> 1) + 16 * (c & 1));
        s.s8 = lds64(rec + 192 + 8 * (c >> 1));
        s.d16 = lds16(doff);
    }
    __device__ __forceinline__ void words(int l, int, uint32_t (&w)[4]) const {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const uint32_t n = (l & 1) ? word_of(b, i) : word_of(a, i), t = word_of(h, i);
            const uint32_t hi = l == 0 ? t << 4 : l == 1 ? t << 2 : l == 2 ? t : t >> 2;
            w[i] = ((l & 2 ? n >> 4 : n) & 0x0F0F0F0Fu) | (hi & 0x30303030u);
        }
    }
};

// the scales and sums of lane group c's sub-blocks in one record of one activation row
template <int QT> struct XScales {
    uint4 v[kSets<QT> / 2];
    __device__ __forceinline__ void load(const XLane &xl, int rec, uint32_t row_off, int c) {
        const uint32_t a = xl.xs + rec * ximg_rec_bytes(QT) + row_off;
        v[0] = lds128(a);
        if (QT == QT_Q6_K) v[kSets<QT> / 2 - 1] = lds128(a + 32 + 16 * c - 16 * (c >> 1));
    }
};

// The integer sums of one record of sixteen weight rows (r0, r1: the lane's two) against one activation row.
template <int QT> struct RecSums {
    int d[kSets<QT>][4];
    template <bool HALF>          // there is no r1
    __device__ __forceinline__ void run(const WRec<QT> &r0, const WRec<QT> &r1, const XLane &xl, int rec, uint32_t row_off, int c) {
        // (the zero area is shared by all rows: only real addresses move)
        const uint32_t b0 = xl.base[0] + (xl.step[0] ? rec * xl.step[0] + row_off : 0u);
        const uint32_t b1 = xl.base[1] + (xl.step[1] ? rec * xl.step[1] + row_off : 0u);
#pragma unroll
        for (int l = 0; l < 4; ++l) {
            const uint4 b = lds128(((l & 1) ? b1 : b0) + bload_off<QT>(l));
            const int s = kSets<QT> == 4 ? l : l >> 1;
            const bool first = kSets<QT> == 4 || (l & 1) == 0;
            uint32_t w0[4], w1[4] = {0, 0, 0, 0};
            r0.words(l, c, w0);
            if (!HALF) r1.words(l, c, w1);
            imma<QT == QT_Q8_0>(d[s], w0[0], w1[0], w0[1], w1[1], b.x, b.y, first);
            imma<QT == QT_Q8_0>(d[s], w0[2], w1[2], w0[3], w1[3], b.z, b.w, false);
        }
    }
    // the share of the lane's row h of the two
    __device__ __forceinline__ float finish(int h, const typename WRec<QT>::Scales &sc, const XScales<QT> &xs, int c) const {
        int v[kSets<QT>];
#pragma unroll
        for (int s = 0; s < kSets<QT>; ++s) v[s] = d[s][2 * h] * 256 + d[s][2 * h + 1];
        return sc.finish(v, c, xs.v);
    }
};

// ---------------------------------------------------------------------------------------------
// conversion: activation row -> image
// ---------------------------------------------------------------------------------------------

constexpr float kXMax = 32512.f;   // 127 * 256: hi = (q + 128) >> 8 stays within a signed byte

// Eight elements of one row starting at k0 (K is a multiple of 32) as loaded.
struct XRaw {
    uint4 v[2];           // bf16: the first
    __device__ __forceinline__ void load(const XSrc &p, int m, int k0) {
        if (k0 >= p.K) {
            v[0] = v[1] = make_uint4(0, 0, 0, 0);
        } else if (p.x_vec_ok) {
            const uint4 *src = reinterpret_cast<const uint4 *>(reinterpret_cast<const uint8_t *>(p.x) + (m * p.ldx + k0) * (p.x_is_bf16 ? 2 : 4));
            v[0] = src[0];
            if (!p.x_is_bf16) v[1] = src[1];
        } else if (p.x_is_bf16) {
            const unsigned short *src = reinterpret_cast<const unsigned short *>(p.x) + m * p.ldx + k0;
            uint32_t w[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) w[i] = (uint32_t)src[2 * i] | (uint32_t)src[2 * i + 1] << 16;
            v[0] = make_uint4(w[0], w[1], w[2], w[3]);
        } else {
            const uint32_t *src = reinterpret_cast<const uint32_t *>(p.x) + m * p.ldx + k0;
#pragma unroll
            for (int i = 0; i < 2; ++i) v[i] = make_uint4(src[4 * i], src[4 * i + 1], src[4 * i + 2], src[4 * i + 3]);
        }
    }
    __device__ __forceinline__ void floats(bool bf16, float (&f)[8]) const {
        if (bf16) {
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                f[2 * i] = __uint_as_float(word_of(v[0], i) << 16);
                f[2 * i + 1] = __uint_as_float(word_of(v[0], i) & 0xFFFF0000u);
            }
        } else {
#pragma unroll
            for (int i = 0; i < 8; ++i) f[i] = __uint_as_float(word_of(v[i >> 2], i & 3));
        }
    }
};
// x * rs * gamma
__device__ __forceinline__ void norm_x8(const XSrc &p, int k0, float (&v)[8]) {
    if (k0 >= p.K) return;
    const bool vec = (reinterpret_cast<uintptr_t>(p.gamma) & 15) == 0;
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        const float *src = p.gamma + k0 + 4 * i;
        const float4 g = vec ? *reinterpret_cast<const float4 *>(src) : make_float4(src[0], src[1], src[2], src[3]);
        v[4 * i] *= p.rs * g.x;
        v[4 * i + 1] *= p.rs * g.y;
        v[4 * i + 2] *= p.rs * g.z;
        v[4 * i + 3] *= p.rs * g.w;
    }
}
// sum of squares of this thread's share of activation row m (threads tid of T take 8 elements in turn)
__device__ __forceinline__ float row_square_share(const XSrc &p, int m, int tid, int T) {
    float ss = 0.f;
    XRaw raw;
    raw.load(p, m, tid * 8);
#pragma unroll 1
    for (int k0 = tid * 8; k0 < p.K; k0 += T * 8) {
        float v[8];
        raw.floats(p.x_is_bf16, v);
        raw.load(p, m, k0 + T * 8);
#pragma unroll
        for (int i = 0; i < 8; ++i) ss = fmaf(v[i], v[i], ss);
    }
    return ss;
}

// Eight elements starting at k0 into the image (whole warps; four neighbouring lanes cover one 32-element block).  The
// integers come out of the low mantissa bits of v * inv + 1.5 * 2^23 (+ 128, which turns the balanced high digit into byte 1
// and the low digit, its top bit flipped, into byte 0), so a value costs one fused multiply-add and a byte permute per plane.
__device__ __forceinline__ void prep_store8(bool q6, const float (&v)[8], int k0, uint8_t *img) {
    uint32_t top = 0;                   // largest magnitude as bits: orders infinities and NaN above every number
#pragma unroll
    for (int i = 0; i < 8; ++i) top = max(top, __float_as_uint(v[i]) & 0x7FFFFFFFu);
    top = max(top, __shfl_xor_sync(0xFFFFFFFFu, top, 1));
    top = max(top, __shfl_xor_sync(0xFFFFFFFFu, top, 2));
    const bool bad = top > __float_as_uint(3.0e38f);
    const float amax = __uint_as_float(top);
    // Below kTiny the quotient would overflow: a fixed step instead, so there a block has the fewer bits the smaller it is.
    // (A true division: __fdividef gives 0 for divisors above 2^126.)
    constexpr float kTiny = 9.6e-35f;
    const float inv = amax >= kTiny ? kXMax / amax : kXMax / kTiny;
    uint32_t h[2], l[2];
    int hs = 0, ls = 0;
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        uint32_t e[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) e[j] = __float_as_uint(fmaf(v[4 * i + j], inv, 12583040.f));
        const uint32_t t0 = __byte_perm(e[0], e[1], 0x5140), t1 = __byte_perm(e[2], e[3], 0x5140);
        l[i] = bad ? 0u : __byte_perm(t0, t1, 0x5410) ^ 0x80808080u;
        h[i] = bad ? 0u : __byte_perm(t0, t1, 0x7632);
        hs = dp4a_ss(h[i], 0x01010101u, hs);
        ls = dp4a_ss(l[i], 0x01010101u, ls);
    }
    uint8_t *rec = img + (k0 >> 8) * ximg_rec_bytes(q6 ? QT_Q6_K : QT_Q4_K);
    uint8_t *dst = rec + ((k0 >> 5) & 7) * 64 + (k0 & 31);
    *reinterpret_cast<uint2 *>(dst) = make_uint2(h[0], h[1]);
    *reinterpret_cast<uint2 *>(dst + 32) = make_uint2(l[0], l[1]);
    const float sx = bad ? __int_as_float(0x7FC00000) : fmaxf(amax, amax > 0.f ? kTiny : 0.f) * (1.0f / kXMax);
    int sum = 256 * hs + ls;
    sum += __shfl_xor_sync(0xFFFFFFFFu, sum, 1);
    if (q6) {
        const int s = (k0 >> 4) & 15;       // sub-block 8 half + 2 quadrant + position half
        if ((k0 & 31) == 0) *reinterpret_cast<float *>(rec + kXBytes + 2 * s) = sx;
        if ((k0 & 15) == 0) *reinterpret_cast<int *>(rec + kXBytes + 32 + 16 * (2 * (s >> 3) + (s & 1)) + 4 * ((s >> 1) & 3)) = sum;
    } else {
        sum += __shfl_xor_sync(0xFFFFFFFFu, sum, 2);
        const int s = (k0 >> 5) & 7;
        if ((k0 & 31) == 0)
            *reinterpret_cast<uint2 *>(rec + kXBytes + 16 * (s & 3) + 8 * (s >> 2)) = make_uint2(__float_as_uint(sx), (uint32_t)sum);
    }
}

// Threads tid = 0 .. T-1 (whole warps) convert activation row m, eight elements a thread and round.  The next round's
// elements are on their way while this one's are converted, so a long row costs one trip to L2 and not one per round.
template <bool NORM>
__device__ __forceinline__ void prep_row(const XSrc &p, bool q6, int m, int tid, int T, uint8_t *img) {
    XRaw raw;
    raw.load(p, m, tid * 8);
#pragma unroll 1
    for (int k0 = tid * 8; k0 < p.Kpad; k0 += T * 8) {      // (a warp's 256 elements are all inside or all outside)
        float v[8];
        raw.floats(p.x_is_bf16, v);
        raw.load(p, m, k0 + T * 8);
        if (NORM && p.gamma) norm_x8(p, k0, v);
        prep_store8(q6, v, k0, img);
    }
}

}  // namespace b200q

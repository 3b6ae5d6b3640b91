// Small batches (2..48 activation rows; speculative-decode verify, sequences decoding together):
// Y[m][n] = sum_k X[m][k] * W[n][k] with the packed weights read from HBM once.
//
// Two launches, or one where every block has few slots and makes what it needs of the first itself.
// skinny_prep_kernel (skinny.cu) turns the activations into the fp16 operand fragments the MMAs read,
// one image per 256 values of K: per token and record they are scaled by a power of two so that the largest is
// below 2^9; a bf16 value then is exact in fp16 unless it is 2^-26 times smaller than the record's largest (its lost
// bits are below 2^-34 of it); fp32 rows enter as two halves, high and low (22 bits).  With more than 16 tokens fp32
// rows are rounded to fp16 (the activation format of all larger batches).  (Made by warps of the second kernel
// instead, for every slot anew, the fragments set the pace from 16 tokens on: 7.5 us per 6144 x 4096 product of a
// plan with the products left out.)
//
// skinny_kernel multiplies.  Work unit ("slot") = one 256-weight record of a tile of 256 or 192 weight rows.  The slots of
// a launch, record by record, tile by tile, product by product, are dealt to the SMs as equal contiguous runs, so any
// product fills the chip.  A tile whose records fall to several
// SMs: every warp adds its rows into double sums in L2, and the one that finds itself the tile's last stores them.
// (A separate launch for the sums cost 4 to 9 us a call; partial tiles in memory, read back by the last warp, 3.6 to
// 5.3 us; this 2.3 to 3.)
//   * one lane of the producer warp fetches a slot's packed records with one tiled bulk copy (the streaming layout seen as a 4-D
//     tensor) and the record's fragments with another;
//   * the consumer warps each own 16 rows: they turn packed weights into fp16 operand fragments in registers and
//     multiply with mma.sync.m16n8k16, accumulating in fp32.  The order of K inside a record is free, so a fragment
//     is whatever weights a lane's 16-byte load brings, and the activations are laid out to match.
// Weights enter as exact integers.  Q4_K, and Q5_K above 16 tokens: sub-block scale x level is an integer below 2^11, exact
// in fp16, so d and dmin are applied once per record instead of a scale per 32 weights, and the minimum term is one more
// MMA with the sub-block sums of the activations (high and low fp16 halves).  Q5_K and Q6_K up to 16 tokens: the levels
// alone, and the sums of a sub-block are scaled in fp32 (Q6_K's offset is such a term with the sums as well); Q6_K above 16
// tokens: scale x (level - 32), which may take 13 bits, rounded to fp16.  The types with a scale per 32 weights accumulate
// per block and scale in fp32.
//
// What bounds it: up to 16 tokens the instructions that make fragments, 1.1 per weight and lane for Q4_K (a nibble under a
// high byte 0x64 or 0x54 reads as 1024 + v or 64 + v: one logic operation, on the half-rate pipe, and one fused
// multiply-add per two weights) and 1.7 times that for Q6_K; above, mma.sync (0.5 of a 16x8x16 per clock and SM).  Measured,
// us, against a kernel with one scale per 32 weights and the K range of a tile cut by 2048: sixteen Q4_K 6144 x 4096
// products as a plan, 4 rows 91 -> 65, 16 rows 141 -> 88; Q4_K 28672 x 4096 alone, 16 rows 50 -> 32; 4096 x 4096 8 rows
// 10.4 -> 8.3, 16 rows 12.9 -> 11.3; Q6_K 4096 x 14336 in a plan, 8 rows 15.2 -> 14.2, 16 rows 24.8 -> 17.5.
// Every mbarrier wait is bounded; a wait that runs out raises the status word and a flag that every role polls,
// copies in flight are awaited (again bounded) and the kernel returns.
#pragma once

#include <cuda.h>
#include <cuda_fp16.h>

#include <algorithm>
#include <atomic>
#include <type_traits>

#include "common.cuh"
#include "kernels.h"
#include "skinny_image.cuh"

namespace b200q {
namespace {

template <int QT, int NT, int P> struct SkShape {
    static constexpr int kWarps = sk_warps(NT), kThreads = (kWarps + 1) * 32;
    static constexpr int kRows = sk_tile_rows(NT);
    static constexpr int kW = sk_w_bytes(QT, NT), kD = sk_d_bytes(QT, NT);
    static constexpr int kB = P * NT * 4096;                       // image: activation fragments of 256 weights,
    static constexpr int kX = NT * sk_sum_bytes(QT, NT);           // Q4_K / Q5_K / Q6_K: sub-block sums, as fragments,
    static constexpr int kImg = sk_image_bytes(NT, P, sk_sum_bytes(QT, NT));      // and per token 1 / scale
    static_assert(kSumBytes<sk_map(QT, NT)> == sk_sum_bytes(QT, NT), "sums");
    static constexpr int kStage = sk_stage_bytes(QT, NT, P), kHead = kSkHeadBytes, kDepth = sk_depth(QT, NT, P);
    static_assert(kDepth >= 2, "stages");
};

struct SkHead {
    uint64_t full[kSkMaxDepth];      // the producer's arrival and its copies' bytes
    uint64_t empty[kSkMaxDepth];     // the consumer warps
    int fail;                        // some wait ran out: every role leaves its loop
};
static_assert(sizeof(SkHead) <= kSkHeadBytes, "head");

// Records are added up in double up to 16 tokens: where a tile's K range is cut depends on the launch, and in what order
// its blocks arrive on the run, but the sum of fp32 record sums in double on neither (it is exact unless they differ by
// more than 2^22), so a product has the same bits in a plan, in a call of its own and in every run.  Above 16 tokens a
// block's own records are added up in fp32.
template <int NT> using SkAcc = typename std::conditional<sk_double(NT), double, float>::type;
__device__ __forceinline__ void sk_pin(float v) { asm volatile("" ::"f"(v) : "memory"); }
__device__ __forceinline__ void sk_pin(double v) { asm volatile("" ::"d"(v) : "memory"); }

__device__ __forceinline__ uint32_t ldsn32(uint32_t a) {
    uint32_t v;
    asm("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(a));
    return v;
}
__device__ __forceinline__ uint2 ldsn64(uint32_t a) {
    uint2 v;
    asm("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(a));
    return v;
}
__device__ __forceinline__ uint4 ldsn128(uint32_t a) {
    uint4 v;
    asm("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(a));
    return v;
}
// The consumers' shared-memory reads are plain (non-volatile) asm so that the compiler may interleave them with
// the tensor-core instructions; addresses are laundered after the wait that makes the data valid, and the results
// are pinned before the arrival that gives the memory away.
__device__ __forceinline__ uint32_t hold_after_wait(uint32_t a) {
    asm volatile("" : "+r"(a)::"memory");
    return a;
}

__device__ __forceinline__ __half2 h2(uint32_t v) { return *reinterpret_cast<__half2 *>(&v); }
__device__ __forceinline__ uint32_t u32(__half2 v) { return *reinterpret_cast<uint32_t *>(&v); }
__device__ __forceinline__ uint32_t hfma(uint32_t v, __half2 s, __half2 c) { return u32(__hfma2(h2(v), s, c)); }
__device__ __forceinline__ uint32_t hadd(uint32_t v, uint32_t c) { return u32(__hadd2(h2(v), h2(c))); }

// (v & mask) | base and (v & mask) ^ base as one instruction each: left to itself the compiler takes two (one immediate
// operand per instruction), which made the logic pipe the busiest of the SM.  `v` may already be an or of two fields.
__device__ __forceinline__ uint32_t and_or(uint32_t v, uint32_t mask, uint32_t base) {
    uint32_t r;
    asm("lop3.b32 %0, %1, %2, %3, 0xEA;" : "=r"(r) : "r"(v), "r"(mask), "r"(base));
    return r;
}
__device__ __forceinline__ uint32_t and_xor(uint32_t v, uint32_t mask, uint32_t base) {
    uint32_t r;
    asm("lop3.b32 %0, %1, %2, %3, 0x6A;" : "=r"(r) : "r"(v), "r"(mask), "r"(base));
    return r;
}

// C (+)= A(16x16 fp16, row) * B(16x8 fp16, col)
__device__ __forceinline__ void mma(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void mma0(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%10, %10, %10, %10};"
        : "=f"(c[0]), "=f"(c[1]), "=f"(c[2]), "=f"(c[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "f"(0.f));
}

// ---- one record of a warp's rows ----------------------------------------------------------------------
// row[i]: shared address of the record of the warp's row 8 i + rev3(g); dsm: Q6_K, of the
// rows' d; bs: fragments, + lane * 16; xs: block-sum fragments, + lane * 8; inv: 1 / scale of tokens 2 t, 2 t + 1 of
// tile nt at inv + 32 nt.  acc += the record's contribution.

template <int NT>
__device__ __forceinline__ void sk_mma_unit(float (&c)[NT][4], const uint32_t (&a0)[4], const uint32_t (&a1)[4], uint32_t bs, int u, bool first) {
#pragma unroll
    for (int nt = 0; nt < NT; ++nt) {
        const uint4 b = ldsn128(bs + (nt * 8 + u) * 512);
        if (first) mma0(c[nt], a0, b.x, b.y);
        else mma(c[nt], a0, b.x, b.y);
        mma(c[nt], a1, b.z, b.w);
    }
}
// the same with both activation planes (fp32 rows: high and low halves)
template <int NT, int P>
__device__ __forceinline__ void sk_mma_planes(float (&c)[NT][4], const uint32_t (&a0)[4], const uint32_t (&a1)[4], uint32_t bs, int u, bool first) {
    sk_mma_unit<NT>(c, a0, a1, bs, u, first);
    if (P == 2) sk_mma_unit<NT>(c, a0, a1, bs + NT * 4096, u, false);
}

// four weights of a lane's row as (a0, a2) of its fragment; half = 1: (a1, a3), the row 8 further down
__device__ __forceinline__ void put(uint32_t (&a)[4], int half, uint32_t even, uint32_t odd) {
    a[half] = even;
    a[2 + half] = odd;
}

template <int QT, int NT, int P> struct SkRecord;

template <int QT, int NT, int P> struct SkRecordK {      // Q4_K, Q5_K
    static __device__ __forceinline__ void run(const uint32_t (&row)[2], uint32_t, uint32_t bs, uint32_t xs, uint32_t inv, int t,
                                               SkAcc<NT> (&acc)[NT][4]) {
        const int h = t >> 1;
        __half2 s[2][4], k[2][4];            // [2 jj + high]: sub-block 4 jj + 2 h + high: scale, -base * scale
        uint32_t am[4];                           // the minima as a fragment: k slots 2 t, 2 t + 1 (and again + 8)
        float d[2], dmin[2];
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const uint4 hd = ldsn128(row[i]);
            d[i] = half_bits_to_float(hd.x);
            dmin[i] = half_bits_to_float(hd.x >> 16);
            const uint32_t sl = (hd.y & 0x3F3F3F3Fu) >> (16 * h);
            const uint32_t su = ((hd.w & 0x0F0F0F0Fu) | ((hd.y >> 2) & 0x30303030u)) >> (16 * h);
            const uint32_t m = (t < 2 ? (hd.z & 0x3F3F3F3Fu) : (((hd.w >> 4) & 0x0F0F0F0Fu) | ((hd.z >> 2) & 0x30303030u))) >> (16 * (t & 1));
            s[i][0] = h2(hadd(__byte_perm(sl, 0x64646464u, 0x4040), 0xE400E400u));
            s[i][1] = h2(hadd(__byte_perm(sl, 0x64646464u, 0x4141), 0xE400E400u));
            s[i][2] = h2(hadd(__byte_perm(su, 0x64646464u, 0x4040), 0xE400E400u));
            s[i][3] = h2(hadd(__byte_perm(su, 0x64646464u, 0x4141), 0xE400E400u));
#pragma unroll
            for (int e = 0; e < 4; ++e)               // Q5_K levels always come under 0x64
                k[i][e] = __hmul2(s[i][e], h2((e & 1) && QT == QT_Q4_K ? 0xD400D400u : 0xE400E400u));
            const uint32_t mh = hadd(__byte_perm(m, 0x64646464u, 0x4140), 0xE400E400u);
            put(am, i, mh, mh);
        }
        float c[NT][4];
        uint4 f[QT == QT_Q5_K ? 2 : 1];
        if (QT == QT_Q5_K) {
#pragma unroll
            for (int i = 0; i < 2; ++i) f[i] = ldsn128(row[i] + 144 + 16 * (t & 1));
        }
#pragma unroll
        for (int jj = 0; jj < 2; ++jj) {
            uint4 w[2];
#pragma unroll
            for (int i = 0; i < 2; ++i) w[i] = ldsn128(row[i] + 16 + 64 * jj + 16 * t);
#pragma unroll
            for (int qq = 0; qq < 2; ++qq) {
                uint32_t lo[2][4], hi[2][4];
#pragma unroll
                for (int e = 0; e < 2; ++e) {
#pragma unroll
                    for (int i = 0; i < 2; ++i) {
                        const uint32_t v = word_of(w[i], 2 * qq + e), v8 = v >> 8;
                        const __half2 sl = s[i][2 * jj], sh = s[i][2 * jj + 1], kl = k[i][2 * jj], kh = k[i][2 * jj + 1];
                        if (QT == QT_Q4_K) {
                            put(lo[e], i, hfma(and_or(v, 0x000F000Fu, 0x64006400u), sl, kl), hfma(and_or(v8, 0x000F000Fu, 0x64006400u), sl, kl));
                            put(hi[e], i, hfma(and_or(v, 0x00F000F0u, 0x54005400u), sh, kh), hfma(and_or(v8, 0x00F000F0u, 0x54005400u), sh, kh));
                        } else {
                            // fifth bit of sub-block sb: bit sb of the byte; here at bits 0 (low) and 1 (high)
                            const uint32_t fb = word_of(f[i], 2 * qq + e) >> (4 * jj + 2 * h), f8 = fb >> 8;
                            const uint32_t l0 = and_or(fb << 4, 0x00100010u, and_or(v, 0x000F000Fu, 0x64006400u)), l1 = and_or(f8 << 4, 0x00100010u, and_or(v8, 0x000F000Fu, 0x64006400u));
                            const uint32_t h0 = and_or(fb << 3, 0x00100010u, and_or(v >> 4, 0x000F000Fu, 0x64006400u)), h1 = and_or(f8 << 3, 0x00100010u, and_or(v8 >> 4, 0x000F000Fu, 0x64006400u));
                            put(lo[e], i, hfma(l0, sl, kl), hfma(l1, sl, kl));
                            put(hi[e], i, hfma(h0, sh, kh), hfma(h1, sh, kh));
                        }
                    }
                }
                sk_mma_planes<NT, P>(c, lo[0], lo[1], bs, 4 * jj + qq, jj == 0 && qq == 0);
                sk_mma_planes<NT, P>(c, hi[0], hi[1], bs, 4 * jj + 2 + qq, false);
            }
        }
#pragma unroll
        for (int nt = 0; nt < NT; ++nt) {
            const uint2 bx = ldsn64(xs + nt * 256);
            const uint2 iv = ldsn64(inv + nt * 32);
            const float i0 = __uint_as_float(iv.x), i1 = __uint_as_float(iv.y);
            float x[4];
            mma0(x, am, bx.x, bx.y);
            SkAcc<NT>(&a)[4] = acc[nt];
            a[0] += fmaf(d[0], c[nt][0], -dmin[0] * x[0]) * i0;
            a[1] += fmaf(d[0], c[nt][1], -dmin[0] * x[1]) * i1;
            a[2] += fmaf(d[1], c[nt][2], -dmin[1] * x[2]) * i0;
            a[3] += fmaf(d[1], c[nt][3], -dmin[1] * x[3]) * i1;
        }
    }
};

// ---- Q5_K and Q6_K up to 16 tokens: sums per sub-block -----------------------------------------------------
// With one or two token tiles it is cheaper to scale sums than weights: every MMA stays inside one sub-block, and its sum is
// multiplied by the sub-block's scale, one fused multiply-add per accumulator where a scale per pair of weights took a
// half-rate one each, and for Q6_K a second term and its products (no fp16 pair holds scale x level exactly).  Levels then
// enter as they are, as fp16 subnormals: bits without an exponent, exact, two or three logic operations per pair.  They are
// shifted to the top of the ten mantissa bits (32 x a 5-bit level, 16 x a 6-bit one; the factor goes into d): the tensor
// core aligns its sums to the exponent and not to the leading bit, and levels at the bottom lost six bits (error against 64
// bits 2.6e-6; shifted 2e-7, scaled weights 4e-7 to 7e-7).
// Measured (us per call, inputs larger than L2), scaled weights -> scaled sums, bf16 plan of one type's calls:
//   Q6_K 4096 x 14336: 8 tokens 16.0 -> 14.2, 16 tokens 20.3 -> 17.5; fp32 4 tokens 19.6 -> 16.4
//   Q5_K 4096 x 14336: 8 tokens 13.3 -> 12.5, 16 tokens 15.7 -> 15.3; fp32 4 tokens 15.0 -> 14.0
//   Q4_K 6144 x  4096: 8 tokens 4.78 -> 4.90, 16 tokens 5.98 -> 6.28: 392 instructions per 16-row record instead of 347 (a
//   4-bit level needs one logic operation and one multiply-add as it is), so Q4_K keeps the scaled weights.
// Bound by instruction issue: Q6_K 4096 x 14336, 8 tokens: 92.7 -> 80.2 us for 6 calls under counters, 60 -> 68 % of issue
// slots, tensor pipe 22.7 -> 14.7 %.

// byte k of w minus off as fp32
__device__ __forceinline__ float sk_byte(uint32_t w, int k, float off) {
    return __uint_as_float(__byte_perm(w, 0x4B000000u, 0x7650 | k)) - (8388608.f + off);      // 2^23 + byte
}
template <int NT, int P>
__device__ __forceinline__ void sk_mma_16(float (&c)[NT][4], const uint32_t (&a)[4], uint32_t bs, int u, int half, bool first) {
#pragma unroll
    for (int nt = 0; nt < NT; ++nt)
#pragma unroll
        for (int pl = 0; pl < P; ++pl) {
            const uint2 b = ldsn64(bs + pl * NT * 4096 + (nt * 8 + u) * 512 + 8 * half);
            if (first && pl == 0) mma0(c[nt], a, b.x, b.y);
            else mma(c[nt], a, b.x, b.y);
        }
}
template <int NT>
__device__ __forceinline__ void sk_add_scaled(float (&e)[NT][4], const float (&c)[NT][4], float s0, float s1) {
#pragma unroll
    for (int nt = 0; nt < NT; ++nt) {
        e[nt][0] = fmaf(s0, c[nt][0], e[nt][0]);
        e[nt][1] = fmaf(s0, c[nt][1], e[nt][1]);
        e[nt][2] = fmaf(s1, c[nt][2], e[nt][2]);
        e[nt][3] = fmaf(s1, c[nt][3], e[nt][3]);
    }
}

template <int NT, int P> struct SkRecordSub32 {              // Q5_K
    static __device__ __forceinline__ void run(const uint32_t (&row)[2], uint32_t, uint32_t bs, uint32_t xs, uint32_t inv, int t,
                                               SkAcc<NT> (&acc)[NT][4]) {
        uint32_t sc[2][2], am[4];                // scales of sub-blocks 0..3, 4..7; the minima as a fragment: k slots 2 t, 2 t + 1 (and + 8)
        float d[2], dmin[2];
        uint2 f[2];
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const uint4 hd = ldsn128(row[i]);
            d[i] = half_bits_to_float(hd.x) * 524288.f;       // 2^24 / 32
            dmin[i] = half_bits_to_float(hd.x >> 16);
            sc[i][0] = hd.y & 0x3F3F3F3Fu;
            sc[i][1] = (hd.w & 0x0F0F0F0Fu) | ((hd.y >> 2) & 0x30303030u);
            const uint32_t m = (t < 2 ? (hd.z & 0x3F3F3F3Fu) : (((hd.w >> 4) & 0x0F0F0F0Fu) | ((hd.z >> 2) & 0x30303030u))) >> (16 * (t & 1));
            const uint32_t mh = hadd(__byte_perm(m, 0x64646464u, 0x4140), 0xE400E400u);
            put(am, i, mh, mh);
            f[i] = ldsn64(row[i] + 144 + 8 * t);
        }
        float e[NT][4];
#pragma unroll
        for (int nt = 0; nt < NT; ++nt)
#pragma unroll
            for (int x = 0; x < 4; ++x) e[nt][x] = 0.f;
#pragma unroll
        for (int j = 0; j < 4; ++j) {            // sub-blocks 2 j (low nibbles) and 2 j + 1
            uint2 w[2];
#pragma unroll
            for (int i = 0; i < 2; ++i) w[i] = ldsn64(row[i] + 16 + 32 * j + 8 * t);
            uint32_t lo[2][4], hi[2][4];
#pragma unroll
            for (int x = 0; x < 2; ++x) {
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    const uint32_t v = x ? w[i].y : w[i].x;
                    const uint32_t b = (x ? f[i].y : f[i].x) >> (2 * j);       // fifth bit of sub-block s: bit s of the byte
                    put(lo[x], i, and_or(b << 9, 0x02000200u, (v << 5) & 0x01E001E0u), and_or(b << 1, 0x02000200u, (v >> 3) & 0x01E001E0u));
                    put(hi[x], i, and_or(b << 8, 0x02000200u, (v << 1) & 0x01E001E0u), and_or(b, 0x02000200u, (v >> 7) & 0x01E001E0u));
                }
            }
            float c[NT][4];
            sk_mma_planes<NT, P>(c, lo[0], lo[1], bs, 2 * j, true);
            sk_add_scaled<NT>(e, c, sk_byte(sc[0][j >> 1], 2 * (j & 1), 0.f), sk_byte(sc[1][j >> 1], 2 * (j & 1), 0.f));
            sk_mma_planes<NT, P>(c, hi[0], hi[1], bs, 2 * j + 1, true);
            sk_add_scaled<NT>(e, c, sk_byte(sc[0][j >> 1], 2 * (j & 1) + 1, 0.f), sk_byte(sc[1][j >> 1], 2 * (j & 1) + 1, 0.f));
        }
#pragma unroll
        for (int nt = 0; nt < NT; ++nt) {
            const uint2 bx = ldsn64(xs + nt * 256);
            const uint2 iv = ldsn64(inv + nt * 32);
            const float i0 = __uint_as_float(iv.x), i1 = __uint_as_float(iv.y);
            float x[4];
            mma0(x, am, bx.x, bx.y);
            SkAcc<NT>(&a)[4] = acc[nt];
            a[0] += fmaf(d[0], e[nt][0], -dmin[0] * x[0]) * i0;
            a[1] += fmaf(d[0], e[nt][1], -dmin[0] * x[1]) * i1;
            a[2] += fmaf(d[1], e[nt][2], -dmin[1] * x[2]) * i0;
            a[3] += fmaf(d[1], e[nt][3], -dmin[1] * x[3]) * i1;
        }
    }
};

template <int NT, int P> struct SkRecordSub16 {              // Q6_K: levels 0..63, the offset 32 by the sub-block sums
    static __device__ __forceinline__ void run(const uint32_t (&row)[2], uint32_t dsm, uint32_t bs, uint32_t xs, uint32_t inv, int t,
                                               SkAcc<NT> (&acc)[NT][4]) {
        uint4 sc[2];                             // int8 scales + 128
        uint32_t am[4];                          // scales as a fragment: k slot = sub-block
        float d[2];
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            sc[i] = ldsn128(row[i] + 192);
            sc[i].x ^= 0x80808080u, sc[i].y ^= 0x80808080u, sc[i].z ^= 0x80808080u, sc[i].w ^= 0x80808080u;
            uint16_t dv;
            asm("ld.shared.u16 %0, [%1];" : "=h"(dv) : "r"(dsm + 8 * i * 16));
            d[i] = half_bits_to_float(dv);
            const uint32_t s0 = (t < 2 ? sc[i].x : sc[i].y) >> (16 * (t & 1)), s1 = (t < 2 ? sc[i].z : sc[i].w) >> (16 * (t & 1));
            // byte under 0x64 reads 1024 + 128 + scale
            put(am, i, hadd(__byte_perm(s0, 0x64646464u, 0x4140), 0xE480E480u), hadd(__byte_perm(s1, 0x64646464u, 0x4140), 0xE480E480u));
        }
        float e[NT][4];
#pragma unroll
        for (int nt = 0; nt < NT; ++nt)
#pragma unroll
            for (int x = 0; x < 4; ++x) e[nt][x] = 0.f;
#pragma unroll
        for (int hh = 0; hh < 2; ++hh) {
#pragma unroll
            for (int ph = 0; ph < 2; ++ph) {     // positions 16 ph .. of the half's four 32-weight quadrants
                uint32_t a[4][4];
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    const uint32_t l0 = ldsn32(row[i] + 64 * hh + 16 * ph + 4 * t), l1 = ldsn32(row[i] + 64 * hh + 32 + 16 * ph + 4 * t);
                    const uint32_t q = ldsn32(row[i] + 128 + 32 * hh + 16 * ph + 4 * t);
                    constexpr uint32_t n = 0x00F000F0u, u = 0x03000300u;       // 16 x level: nibble, upper two bits
                    put(a[0], i, and_or(q << 8, u, (l0 << 4) & n), and_or(q, u, (l0 >> 4) & n));
                    put(a[1], i, and_or(q << 6, u, (l1 << 4) & n), and_or(q >> 2, u, (l1 >> 4) & n));
                    put(a[2], i, and_or(q << 4, u, l0 & n), and_or(q >> 4, u, (l0 >> 8) & n));
                    put(a[3], i, and_or(q << 2, u, l1 & n), and_or(q >> 6, u, (l1 >> 8) & n));
                }
#pragma unroll
                for (int qd = 0; qd < 4; ++qd) {
                    float c[NT][4];
                    sk_mma_16<NT, P>(c, a[qd], bs, 4 * hh + qd, ph, true);
                    const int s = 8 * hh + 2 * qd + ph;
                    sk_add_scaled<NT>(e, c, sk_byte(word_of(sc[0], s >> 2), s & 3, 128.f), sk_byte(word_of(sc[1], s >> 2), s & 3, 128.f));
                }
            }
        }
#pragma unroll
        for (int nt = 0; nt < NT; ++nt) {
            const uint2 bh = ldsn64(xs + nt * 512), bl = ldsn64(xs + nt * 512 + 256);
            const uint2 iv = ldsn64(inv + nt * 32);
            const float i0 = __uint_as_float(iv.x), i1 = __uint_as_float(iv.y);
            float x[4];
            mma0(x, am, bh.x, bh.y);
            mma(x, am, bl.x, bl.y);
            SkAcc<NT>(&a)[4] = acc[nt];
            // 2^24 / 16 = 2^20 with the sums and 1 / scale last: in another order a factor may leave fp32's range where the product
            // does not
            a[0] += d[0] * fmaf(1048576.f, e[nt][0], -32.f * x[0]) * i0;
            a[1] += d[0] * fmaf(1048576.f, e[nt][1], -32.f * x[1]) * i1;
            a[2] += d[1] * fmaf(1048576.f, e[nt][2], -32.f * x[2]) * i0;
            a[3] += d[1] * fmaf(1048576.f, e[nt][3], -32.f * x[3]) * i1;
        }
    }
};

template <int NT, int P> struct SkRecord<QT_Q4_K, NT, P> : SkRecordK<QT_Q4_K, NT, P> {};
template <int NT, int P> struct SkRecord<QT_Q5_K, NT, P> : std::conditional<(NT <= 2), SkRecordSub32<NT, P>, SkRecordK<QT_Q5_K, NT, P>>::type {};

// acc += d * inv * c, d of the lane's rows
template <int NT>
__device__ __forceinline__ void sk_scale(SkAcc<NT> (&acc)[NT][4], const float (&c)[NT][4], const float (&d)[2], uint32_t inv) {
#pragma unroll
    for (int nt = 0; nt < NT; ++nt) {
        const uint2 iv = ldsn64(inv + nt * 32);
        const float i0 = __uint_as_float(iv.x), i1 = __uint_as_float(iv.y);
        SkAcc<NT>(&a)[4] = acc[nt];
        a[0] += d[0] * i0 * c[nt][0];
        a[1] += d[0] * i1 * c[nt][1];
        a[2] += d[1] * i0 * c[nt][2];
        a[3] += d[1] * i1 * c[nt][3];
    }
}

template <int NT, int P> struct SkRecordQ6 {                 // more than 16 tokens: scale x (level - 32) rounded to fp16
    static __device__ __forceinline__ void run(const uint32_t (&row)[2], uint32_t dsm, uint32_t bs, uint32_t, uint32_t inv, int t,
                                               SkAcc<NT> (&acc)[NT][4]) {
        const int h = t >> 1;
        const uint32_t sel = 0x4040u + 0x0101u * t;
        uint4 sc[2];
        float d[2];
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            sc[i] = ldsn128(row[i] + 192);           // int8 scales: word 2 hh + high, byte t
            uint16_t dv;
            asm("ld.shared.u16 %0, [%1];" : "=h"(dv) : "r"(dsm + 8 * i * 16));
            d[i] = half_bits_to_float(dv);
        }
        float c[NT][4];
#pragma unroll
        for (int hh = 0; hh < 2; ++hh) {
            uint4 l[2], q[2];
            __half2 s[2][2];
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                l[i] = ldsn128(row[i] + 64 * hh + 16 * t);
                q[i] = ldsn128(row[i] + 128 + 32 * hh + 16 * (t & 1));
#pragma unroll
                for (int e = 0; e < 2; ++e)          // byte ^ 0x80 under 0x64 reads 1024 + 128 + scale
                    s[i][e] = h2(hadd(__byte_perm(word_of(sc[i], 2 * hh + e) ^ 0x80808080u, 0x64646464u, sel), 0xE480E480u));
            }
#pragma unroll
            for (int qq = 0; qq < 2; ++qq) {
                uint32_t lo[2][4], hi[2][4];
#pragma unroll
                for (int e = 0; e < 2; ++e) {
#pragma unroll
                    for (int i = 0; i < 2; ++i) {
                        const uint32_t v = word_of(l[i], 2 * qq + e), x = word_of(q[i], 2 * qq + e);
                        // upper bits: field 2 h (low nibbles' weights) and 4 + 2 h (high nibbles')
                        const uint32_t v8 = v >> 8, xs = x >> (2 * h), xs8 = xs >> 8;          // low weights' field at bits 0-1, high at 4-5
                        const uint32_t l0 = and_or(xs << 4, 0x00300030u, and_or(v, 0x000F000Fu, 0x64006400u)), l1 = and_or(xs8 << 4, 0x00300030u, and_or(v8, 0x000F000Fu, 0x64006400u));
                        const uint32_t h0 = and_or(xs, 0x00300030u, and_or(v >> 4, 0x000F000Fu, 0x64006400u)), h1 = and_or(xs8, 0x00300030u, and_or(v8 >> 4, 0x000F000Fu, 0x64006400u));
                        auto q6 = [](uint32_t a, __half2 sv) { return u32(__hmul2(h2(hadd(a, 0xE420E420u)), sv)); };      // (1024 + q - 1056) s
                        put(lo[e], i, q6(l0, s[i][0]), q6(l1, s[i][0]));
                        put(hi[e], i, q6(h0, s[i][1]), q6(h1, s[i][1]));
                    }
                }
                sk_mma_planes<NT, P>(c, lo[0], lo[1], bs, 4 * hh + qq, hh == 0 && qq == 0);
                sk_mma_planes<NT, P>(c, hi[0], hi[1], bs, 4 * hh + 2 + qq, false);
            }
        }
        sk_scale<NT>(acc, c, d, inv);
    }
};
template <int NT, int P> struct SkRecord<QT_Q6_K, NT, P> : std::conditional<(NT <= 2), SkRecordSub16<NT, P>, SkRecordQ6<NT, P>>::type {};

// Types with one scale per 32 weights: units are blocks; e += d_block * c, then acc += inv * e
template <int QT, int NT, int P> struct SkRecordBlock {
    static __device__ __forceinline__ void run(const uint32_t (&row)[2], uint32_t, uint32_t bs, uint32_t, uint32_t inv, int t,
                                               SkAcc<NT> (&acc)[NT][4]) {
        uint4 hd[2];                              // eight fp16 d (MXFP4: eight scale bytes)
#pragma unroll
        for (int i = 0; i < 2; ++i) hd[i] = ldsn128(row[i] + (QT == QT_Q8_0 ? 256 : 0));
        float e[NT][4];
#pragma unroll
        for (int nt = 0; nt < NT; ++nt)
#pragma unroll
            for (int x = 0; x < 4; ++x) e[nt][x] = 0.f;
        uint2 w[2];
#pragma unroll
        for (int b = 0; b < 8; ++b) {
            uint32_t a0[4], a1[4];
            float d[2];
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                uint32_t x0, x1, y0, y1;
                if (QT == QT_Q8_0) {
                    w[i] = ldsn64(row[i] + 32 * b + 8 * t);
                    x0 = and_xor(w[i].x, 0x00FF00FFu, 0x64806480u), x1 = and_xor(w[i].x >> 8, 0x00FF00FFu, 0x64806480u);
                    y0 = and_xor(w[i].y, 0x00FF00FFu, 0x64806480u), y1 = and_xor(w[i].y >> 8, 0x00FF00FFu, 0x64806480u);
                } else if (QT == QT_Q4_0) {
                    if (b % 2 == 0) {
                        w[i] = ldsn64(row[i] + 16 + 16 * b + 8 * t);
                        x0 = and_or(w[i].x, 0x000F000Fu, 0x64006400u), x1 = and_or(w[i].x >> 8, 0x000F000Fu, 0x64006400u);
                        y0 = and_or(w[i].y, 0x000F000Fu, 0x64006400u), y1 = and_or(w[i].y >> 8, 0x000F000Fu, 0x64006400u);
                    } else {
                        x0 = and_or(w[i].x, 0x00F000F0u, 0x54005400u), x1 = and_or(w[i].x >> 8, 0x00F000F0u, 0x54005400u);
                        y0 = and_or(w[i].y, 0x00F000F0u, 0x54005400u), y1 = and_or(w[i].y >> 8, 0x00F000F0u, 0x54005400u);
                    }
                } else {
                    const uint32_t v = ldsn32(row[i] + 16 + 16 * b + 4 * t);
                    const uint32_t p = mxfp4_bytes(v), r = mxfp4_bytes(v >> 16);
                    x0 = and_or(p, 0x00FF00FFu, 0x64006400u), x1 = and_or(p >> 8, 0x00FF00FFu, 0x64006400u);
                    y0 = and_or(r, 0x00FF00FFu, 0x64006400u), y1 = and_or(r >> 8, 0x00FF00FFu, 0x64006400u);
                }
                // -(1024 + 128); -(1024 + 8) and -(64 + 8); -(1024 + 64)
                const uint32_t off = QT == QT_Q8_0 ? 0xE480E480u : QT == QT_MXFP4 ? 0xE440E440u : b % 2 == 0 ? 0xE408E408u : 0xD480D480u;
                put(a0, i, hadd(x0, off), hadd(x1, off));
                put(a1, i, hadd(y0, off), hadd(y1, off));
                if (QT == QT_MXFP4) d[i] = __uint_as_float(e8m0_half_bits(((b < 4 ? hd[i].x : hd[i].y) >> (8 * (b & 3))) & 0xFF));
                else d[i] = half_bits_to_float(word_of(hd[i], b >> 1) >> (16 * (b & 1)));
            }
            float c[NT][4];
            sk_mma_planes<NT, P>(c, a0, a1, bs, b, true);
#pragma unroll
            for (int nt = 0; nt < NT; ++nt)
#pragma unroll
                for (int x = 0; x < 4; ++x) e[nt][x] = fmaf(d[x >> 1], c[nt][x], e[nt][x]);
        }
        float one[2];
#pragma unroll
        for (int i = 0; i < 2; ++i) one[i] = 1.f;
        sk_scale<NT>(acc, e, one, inv);
    }
};
template <int NT, int P> struct SkRecord<QT_Q8_0, NT, P> : SkRecordBlock<QT_Q8_0, NT, P> {};
template <int NT, int P> struct SkRecord<QT_Q4_0, NT, P> : SkRecordBlock<QT_Q4_0, NT, P> {};
template <int NT, int P> struct SkRecord<QT_MXFP4, NT, P> : SkRecordBlock<QT_MXFP4, NT, P> {};

// ---- the kernel ---------------------------------------------------------------------------------------

// one bounded wait of a role; on expiry (or when another role already gave up) the role leaves
__device__ __forceinline__ bool sk_wait(uint32_t bar, uint32_t parity, volatile int *fail_flag, int *status) {
    if (mbar_try_wait_hint(bar, parity, 32)) return true;
    if (*fail_flag) return false;
    if (mbar_wait_bounded_fast(bar, parity)) return true;
    atomicMax(status, DEV_ERR_PIPE_TIMEOUT);
    *fail_flag = 1;
    return false;
}

// (product, tile, record) of a slot, stepped without dividing and without reading the table
struct SkCursor {
    int ji, tile, rec, nsb, tiles;
    __device__ __forceinline__ void start(const SkJob *jobs, int njobs, int slot) {
        ji = 0;
        while (ji + 1 < njobs && slot >= jobs[ji + 1].slot0) ++ji;
        nsb = jobs[ji].nsb, tiles = jobs[ji].tiles;
        const int local = slot - jobs[ji].slot0;
        tile = local / nsb;
        rec = local - tile * nsb;
    }
    __device__ __forceinline__ void next(const SkJob *jobs, int njobs) {
        if (++rec < nsb) return;
        rec = 0;
        if (++tile < tiles) return;
        tile = 0;
        if (++ji < njobs) nsb = jobs[ji].nsb, tiles = jobs[ji].tiles;
    }
};

__device__ __forceinline__ void sk_tma_4d(uint32_t dst, const CUtensorMap *map, int c0, int c2, int c3, uint32_t bar) {
    asm volatile(
        "cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6}], [%2];"
        ::"r"(dst), "l"(map), "r"(bar), "r"(c0), "r"(0), "r"(c2), "r"(c3)
        : "memory");
}

__device__ __forceinline__ void sk_store_y(const SkJob &J, int n, int m, float v) {
    if (n >= J.N || m >= J.M) return;
    const long long at = (long long)m * J.ldy + n;
    if (J.y_is_bf16) reinterpret_cast<__nv_bfloat16 *>(J.y)[at] = __float2bfloat16_rn(v);
    else reinterpret_cast<float *>(J.y)[at] = v;
}
// N: products the parameters have room for
template <int QT, int NT, int P, int N>
__global__ void __launch_bounds__(SkShape<QT, NT, P>::kThreads, 1) skinny_kernel(const __grid_constant__ SkParamsOf<N> p) {
    using S = SkShape<QT, NT, P>;
    constexpr int kSkConsumers = S::kWarps, D = S::kDepth, REC = rec_bytes(QT);
    extern __shared__ __align__(128) uint8_t smem[];
    SkHead &head = *reinterpret_cast<SkHead *>(smem);
    const uint32_t full0 = smem_u32(head.full), empty0 = smem_u32(head.empty), ring0 = smem_u32(smem + S::kHead);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const SkJob *jobs = p.jobs;
    const int begin = sk_slot_begin(p.slots, gridDim.x, blockIdx.x), end = sk_slot_begin(p.slots, gridDim.x, blockIdx.x + 1);
    volatile int *fail = &head.fail;

    if (threadIdx.x == 0) {
        for (int i = 0; i < D; ++i) {
            mbar_init(full0 + 8 * i, 1);
            mbar_init(empty0 + 8 * i, kSkConsumers);
        }
        head.fail = 0;
        mbar_fence_init();
        fence_proxy_async();
    }
    pdl_launch_dependents();
    __syncthreads();

    SkCursor cur;
    cur.start(jobs, p.njobs, begin);
    int stage = 0;
    uint32_t phase = 0;

    if (warp == kSkConsumers) {
        // ===== producer ======================================================================================
        if (lane == 0) {
            auto fetch_w = [&](const SkCursor &at, int stg) {
                const SkJob &J = jobs[at.ji];
                const int nfull = at.nsb / kChunkRecs;
                const int c = at.rec / kChunkRecs, in = at.rec - c * kChunkRecs;
                const bool tail = c >= nfull;
                const uint32_t bar = full0 + 8 * stg, w = ring0 + stg * S::kStage;
                const int group0 = at.tile * (S::kRows / kRowGroup);
                mbar_expect_tx(bar, S::kW + S::kD + (p.direct ? 0 : S::kImg));
                sk_tma_4d(w, tail ? &J.wtail : &J.w, in * (REC / 4), tail ? 0 : c, group0, bar);
                if (QT == QT_Q6_K) {
                    const int nrec = tail ? at.nsb - c * kChunkRecs : kChunkRecs;
                    sk_tma_4d(w + S::kW, tail ? &J.dtail : &J.d, nrec * (REC / 4), tail ? 0 : c, group0, bar);
                }
            };
            auto fetch_x = [&](const SkCursor &at, int stg) {
                bulk_g2s(ring0 + stg * S::kStage + S::kW + S::kD, jobs[at.ji].img + (size_t)at.rec * S::kImg, S::kImg, full0 + 8 * stg);
            };
            const int first = min(end, begin + D);
            SkCursor at = cur;
            for (int s = begin; s < first; ++s, at.next(jobs, p.njobs)) fetch_w(at, s - begin);      // weights depend on no earlier launch
            if (!p.direct) {
                pdl_wait();                                                                 // the images do
                for (int s = begin; s < first; ++s, cur.next(jobs, p.njobs)) fetch_x(cur, s - begin);
            }
            for (int s = first; s < end; ++s, cur.next(jobs, p.njobs)) {
                if (!sk_wait(empty0 + 8 * stage, phase, fail, p.status)) break;
                fence_proxy_async();         // the consumers' reads of this stage precede the copy engine's writes
                fetch_w(cur, stage);
                fetch_x(cur, stage);
                if (++stage == D) stage = 0, phase ^= 1;
            }
        }
    } else {
        // ===== products ======================================================================================
        const int g = lane >> 2, t = lane & 3;
        // the lane's row: neighbouring g read rows whose loads meet no bank twice (16 bytes: rows 4 apart; 8 bytes of 176:
        // rows 2 apart; 4 bytes of 208: any)
        constexpr int kMap = sk_map(QT, NT);
        const int rev = kMap == SK_SUB32 ? ((g & 3) << 1) | (g >> 2) : kMap == SK_SUB16 ? g : ((g & 1) << 2) | (g & 2) | (g >> 2);
        const int row0 = warp * 16 + rev;
        if (p.direct) {                      // all the block's slots have a stage of their own: their images go straight there
            pdl_wait();
            SkCursor at = cur;
            int from = 0;                    // task = (slot, token), warp after warp
            for (int s = begin; s < end; ++s, at.next(jobs, p.njobs)) {
                const SkJob &J = jobs[at.ji];
                uint8_t *img = smem + S::kHead + (s - begin) * S::kStage + S::kW + S::kD;
                for (int tok = (warp + kSkConsumers - from) % kSkConsumers; tok < J.M; tok += kSkConsumers)
                    sk_make_image<sk_map(QT, NT)>(J, at.rec, tok, lane, img, NT, P);
                from = (from + J.M) % kSkConsumers;
            }
            asm volatile("bar.sync 1, %0;" ::"n"(S::kWarps * 32) : "memory");
        }
        SkAcc<NT> acc[NT][4];
        int seg = begin;                     // first slot of the tile's part in hand
        bool waited = p.direct != 0, ok = true;
        for (int s = begin; s < end; ++s, cur.next(jobs, p.njobs)) {
            if (s == seg) {
#pragma unroll
                for (int nt = 0; nt < NT; ++nt)
#pragma unroll
                    for (int i = 0; i < 4; ++i) acc[nt][i] = 0;
            }
            // after a failure the products are left out, but shared tiles are still counted (below)
            ok = ok && __all_sync(0xFFFFFFFFu, sk_wait(full0 + 8 * stage, phase, fail, p.status));
            if (ok) {
                const uint32_t w = hold_after_wait(ring0 + stage * S::kStage);
                uint32_t row[2];
#pragma unroll
                for (int i = 0; i < 2; ++i) row[i] = w + (row0 + 8 * i) * REC;
                const uint32_t b = w + S::kW + S::kD;
                SkRecord<QT, NT, P>::run(row, w + S::kW + row0 * 16 + 2 * (cur.rec % kChunkRecs), b + lane * 16, b + S::kB + lane * 8,
                                            b + S::kB + S::kX + 8 * t, t, acc);
#pragma unroll
                for (int nt = 0; nt < NT; ++nt)
#pragma unroll
                    for (int i = 0; i < 4; ++i) sk_pin(acc[nt][i]);
                __syncwarp();
                if (lane == 0) mbar_arrive(empty0 + 8 * stage);
                if (++stage == D) stage = 0, phase ^= 1;
            }

            const bool last = cur.rec == cur.nsb - 1;
            if (!last && s + 1 < end) continue;
            const SkJob &J = jobs[cur.ji];
            // the tile ends here, or this block's part of it
            if (!waited) {                   // outputs and partial sums belong to earlier launches until they have finished
                pdl_wait();
                waited = true;
            }
            const int tile0 = s - cur.rec;   // the tile's first slot
            const bool from0 = seg == tile0;
            seg = s + 1;
            if (!(last && from0)) {
                // The tile is shared.  Its blocks add their rows into double sums, one run of 32 lanes per accumulator; the
                // warp whose count is the tile's last takes its rows' sums, leaving zeros, and the count is zero again
                // (also after a failure).  Counting at once rather than at the end of the run: a tile's last block
                // then seldom waits for a block that has other slots to do.
                const int b0 = sk_slot_owner(p.slots, gridDim.x, tile0), b1 = sk_slot_owner(p.slots, gridDim.x, tile0 + cur.nsb - 1);
                double *sum = p.sums + ((size_t)b0 * kSkConsumers + warp) * (NT * 4 * 32) + lane;
                if (ok) {
#pragma unroll
                    for (int nt = 0; nt < NT; ++nt)
#pragma unroll
                        for (int i = 0; i < 4; ++i) atomicAdd(sum + (nt * 4 + i) * 32, (double)acc[nt][i]);
                }
                __syncwarp();
                unsigned old = 0;
                if (lane == 0)       // releases the warp's additions, acquires the other blocks'
                    asm volatile("atom.acq_rel.gpu.global.inc.u32 %0, [%1], %2;"
                                 : "=r"(old)
                                 : "l"(p.count + b0 * kSkConsumers + warp), "r"((unsigned)(b1 - b0))
                                 : "memory");
                if (__shfl_sync(0xFFFFFFFFu, old, 0) != (unsigned)(b1 - b0)) continue;
                __syncwarp();        // what lane 0 acquired is ordered before the other lanes' reads, too (a shuffle orders no memory)
#pragma unroll
                for (int nt = 0; nt < NT; ++nt)
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        acc[nt][i] = (SkAcc<NT>)__ldcg(sum + (nt * 4 + i) * 32);
                        __stcg(sum + (nt * 4 + i) * 32, 0.0);
                    }
            }
            if (!ok) continue;
#pragma unroll
            for (int nt = 0; nt < NT; ++nt)
#pragma unroll
                for (int i = 0; i < 4; ++i)
                    sk_store_y(J, cur.tile * S::kRows + row0 + 8 * (i >> 1), nt * 8 + 2 * t + (i & 1), (float)acc[nt][i]);
        }
    }

    // After a failure copies may still be on their way: they get time to land (far above a copy's latency)
    // before the block's shared memory is released.
    __syncthreads();
    if (*fail) {
        const uint64_t t0 = globaltimer_ns();
        while (globaltimer_ns() - t0 < 100000) {
        }
    }
}

template <int QT, int NT, int P, int N = kSkInline> cudaError_t sk_launch_t(const SkParams &p, int grid, cudaStream_t st) {
    using S = SkShape<QT, NT, P>;
    auto kern = skinny_kernel<QT, NT, P, N>;
    constexpr size_t smem = S::kHead + size_t(S::kDepth) * S::kStage;
    static_assert(smem <= 232448, "shared-memory plan exceeds the 227 KB a block may use");
    static std::atomic<int> configured_dev{-1};     // contexts on several threads may launch at once
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev != configured_dev) {
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return e;
        configured_dev = dev;
    }
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)grid);
    cfg.blockDim = dim3(S::kThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    void *args[] = {const_cast<SkParams *>(&p)};     // its first N jobs
    return cudaLaunchKernelExC(&cfg, reinterpret_cast<const void *>(kern), args);
}

template <int QT> cudaError_t sk_launch_type(const SkParams &p, int NT, int P, int grid, cudaStream_t st) {
    if (p.njobs > kSkInline) {               // plans, of up to 16 rows
        switch (NT * 4 + P) {
        case 1 * 4 + 1: return sk_launch_t<QT, 1, 1, kSkMaxJobs>(p, grid, st);
        case 1 * 4 + 2: return sk_launch_t<QT, 1, 2, kSkMaxJobs>(p, grid, st);
        case 2 * 4 + 1: return sk_launch_t<QT, 2, 1, kSkMaxJobs>(p, grid, st);
        case 2 * 4 + 2: return sk_launch_t<QT, 2, 2, kSkMaxJobs>(p, grid, st);
        default: return cudaErrorInvalidValue;
        }
    }
    switch (NT * 4 + P) {
    case 1 * 4 + 1: return sk_launch_t<QT, 1, 1>(p, grid, st);
    case 1 * 4 + 2: return sk_launch_t<QT, 1, 2>(p, grid, st);
    case 2 * 4 + 1: return sk_launch_t<QT, 2, 1>(p, grid, st);
    case 2 * 4 + 2: return sk_launch_t<QT, 2, 2>(p, grid, st);
    case 4 * 4 + 1: return sk_launch_t<QT, 4, 1>(p, grid, st);
    case 6 * 4 + 1: return sk_launch_t<QT, 6, 1>(p, grid, st);
    default: return cudaErrorInvalidValue;
    }
}

}  // namespace
}  // namespace b200q

// one source file per weight type (they compile side by side)
#define SK_INSTANTIATE(NAME, QT)                                                                          \
    namespace b200q {                                                                                     \
    cudaError_t skinny_launch_##NAME(const SkParams &p, int NT, int P, int grid, cudaStream_t st) {       \
        return sk_launch_type<QT>(p, NT, P, grid, st);                                                    \
    }                                                                                                     \
    cudaError_t skinny_wait_limit_##NAME(unsigned long long ns) {                                         \
        return cudaMemcpyToSymbol(s_wait_limit_ns, &ns, sizeof(ns));                                      \
    }                                                                                                     \
    }

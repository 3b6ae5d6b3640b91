// Pieces shared by the tensor-core kernels: tcgen05 / TMA wrappers, shared-memory descriptors, the
// conversion of packed weights and of activations to fp16, the tensor-map encoder.
#pragma once

#include <cuda.h>
#include <cuda_fp16.h>

#include "common.cuh"

namespace b200q {
namespace {

// ---- tcgen05 wrappers -----------------------------------------------------------------------

__device__ __forceinline__ void tmem_alloc(uint32_t smem_dst, uint32_t ncols) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_dst), "r"(ncols) : "memory");
}
__device__ __forceinline__ void tmem_relinquish() {
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// true in one lane of a converged warp, the same one every time
__device__ __forceinline__ bool elect_one() {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "elect.sync _|p, 0xFFFFFFFF;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok));
    return ok != 0;
}

__device__ __forceinline__ void umma_f16(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
}
// arrives on the mbarrier once every tcgen05.mma issued so far by this thread has completed
__device__ __forceinline__ void umma_commit(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t (&r)[32]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
        "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
          "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
          "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr)
        : "memory");
}
__device__ __forceinline__ void tmem_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

// 2-D tiled TMA load (no multicast): box lands at dst, bytes are counted on the mbarrier
__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap *map, int x, int y, uint32_t bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
        ::"r"(dst), "l"(map), "r"(bar), "r"(x), "r"(y)
        : "memory");
}

// 4-D tiled TMA load (packed weight records: [bytes/4][row in group][chunk][row group])
__device__ __forceinline__ void tma_load_4d(uint32_t dst, const CUtensorMap *map, int c0, int c1, int c2, int c3, uint32_t bar) {
    asm volatile(
        "cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6}], [%2];"
        ::"r"(dst), "l"(map), "r"(bar), "r"(c0), "r"(c1), "r"(c2), "r"(c3)
        : "memory");
}

// shared-memory matrix descriptor: K-major, 128-byte swizzle, rows of 128 bytes, 8-row groups
// 1024 bytes apart (see the tcgen05 matrix-descriptor format: start >> 4 in bits 0..13, leading
// offset in 16..29, stride offset in 32..45, version 1 in 46..47, layout type 2 in 61..63)
__device__ __forceinline__ uint64_t make_desc_sw128(uint32_t saddr) {
    uint64_t d = 0;
    d |= (uint64_t)((saddr & 0x3FFFF) >> 4);
    d |= (uint64_t)1 << 16;                  // leading byte offset (unused for swizzled K-major)
    d |= (uint64_t)(1024 >> 4) << 32;        // stride byte offset
    d |= (uint64_t)1 << 46;                  // descriptor version
    d |= (uint64_t)2 << 61;                  // SWIZZLE_128B
    return d;
}

// ---- dequantization to the swizzled A tile ---------------------------------------------------
//
// A dequant thread owns one weight row of the tile and one 64-weight unit (one K-step) of every
// 256-weight record.  Small integers become fp16 without a conversion instruction: a byte v put
// under the high byte 0x64 reads as the half 1024 + v (under 0x54, a byte with only its high
// nibble set reads as 64 + v / 16).  One exact half2 subtraction removes the offset and one half2
// fused multiply-add applies the block's scale and minimum, two weights per instruction.  Eight fp16 values
// form one 16-byte chunk; chunk cc of row r is stored at chunk position cc ^ (r & 7) of the row
// (128-byte swizzle).

__device__ __forceinline__ void st_chunk(uint32_t row_saddr, int r7, int cc, uint32_t p0, uint32_t p1, uint32_t p2, uint32_t p3) {
    const uint32_t a = row_saddr + ((cc ^ r7) << 4);
    asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(a), "r"(p0), "r"(p1), "r"(p2), "r"(p3) : "memory");
}

__device__ __forceinline__ __half2 as_h2(uint32_t v) { return *reinterpret_cast<__half2 *>(&v); }
__device__ __forceinline__ uint32_t as_u32(__half2 h) { return *reinterpret_cast<uint32_t *>(&h); }

// bytes 0..3 of v -> ((b0, b1) - off) * s + c and ((b2, b3) - off) * s + c, MG the high byte given to each
template <uint32_t MG>
__device__ __forceinline__ void word_affine(uint32_t v, __half2 off, __half2 s, __half2 c, uint32_t &p0, uint32_t &p1) {
    p0 = as_u32(__hfma2(__hsub2(as_h2(__byte_perm(v, MG, 0x4140)), off), s, c));
    p1 = as_u32(__hfma2(__hsub2(as_h2(__byte_perm(v, MG, 0x4342)), off), s, c));
}
template <uint32_t MG>
__device__ __forceinline__ void word_scale(uint32_t v, __half2 off, __half2 s, uint32_t &p0, uint32_t &p1) {
    p0 = as_u32(__hmul2(__hsub2(as_h2(__byte_perm(v, MG, 0x4140)), off), s));
    p1 = as_u32(__hmul2(__hsub2(as_h2(__byte_perm(v, MG, 0x4342)), off), s));
}

// Scale s and minimum m of a Q4_K sub-block (weight = s q - m) as half2 constants around the
// integer q0 nearest m / s:  weight = s (q - q0) - (m - s q0).  Both terms are then of the weight's
// own size, so rounding s and the small remainder to fp16 costs about one extra rounding of the
// weight instead of a rounding of m, which is several times larger than the weights.
// `base` is the offset the byte trick adds (1024 or 64); base + q0 stays an exact fp16 integer.
__device__ __forceinline__ void centered(float s, float m, __half2 base, __half2 &off, __half2 &sh, __half2 &ch) {
    float q0 = rintf(__fdividef(m, s));
    q0 = (q0 >= 0.f && q0 <= 1023.f) ? q0 : (q0 > 1023.f ? 1023.f : 0.f);   // NaN (s == 0) -> 0
    off = __hadd2(base, __float2half2_rn(q0));
    sh = __float2half2_rn(s);
    ch = __float2half2_rn(fmaf(s, q0, -m));
}

template <int QT> struct Unit;

// the 64 converted weights of a thread (eight 16-byte chunks in K order) -> its row of the stage
__device__ __forceinline__ void store_row(const uint32_t (&o)[32], uint32_t row_saddr, int r7) {
#pragma unroll
    for (int c = 0; c < 8; ++c) st_chunk(row_saddr, r7, c, o[4 * c], o[4 * c + 1], o[4 * c + 2], o[4 * c + 3]);
}

template <> struct Unit<QT_Q4_K> {
    uint4 hdr, q0, q1;
    // rec: shared address of the row's 144-byte record; unit j = bytes 32j..32j+31 of the nibbles:
    // low nibbles are weights 0..31 of the K-step (sub-block 2j), high nibbles weights 32..63 (2j+1)
    __device__ __forceinline__ void load(uint32_t rec, uint32_t, int j) {
        hdr = lds128(rec);
        q0 = lds128(rec + 16 + 32 * j);
        q1 = lds128(rec + 32 + 32 * j);
    }
    __device__ __forceinline__ void convert(int j, uint32_t (&o)[32]) const {
        int sa, ma, sb, mb;
        q4k_scale_min(hdr.y, hdr.z, hdr.w, 2 * j, sa, ma);
        q4k_scale_min(hdr.y, hdr.z, hdr.w, 2 * j + 1, sb, mb);
        const float d = half_bits_to_float(hdr.x), dmin = half_bits_to_float(hdr.x >> 16);
        __half2 o_lo, s_lo, c_lo, o_hi, s_hi, c_hi;
        centered(d * (float)sa, dmin * (float)ma, as_h2(0x64006400u), o_lo, s_lo, c_lo);
        centered(d * (float)sb, dmin * (float)mb, as_h2(0x54005400u), o_hi, s_hi, c_hi);
        const uint32_t w[8] = {q0.x, q0.y, q0.z, q0.w, q1.x, q1.y, q1.z, q1.w};
#pragma unroll
        for (int n = 0; n < 4; ++n) {     // chunk n = low nibbles of words 2n, 2n+1; chunk 4 + n = their high nibbles
            word_affine<0x64>(w[2 * n] & 0x0F0F0F0Fu, o_lo, s_lo, c_lo, o[4 * n], o[4 * n + 1]);
            word_affine<0x64>(w[2 * n + 1] & 0x0F0F0F0Fu, o_lo, s_lo, c_lo, o[4 * n + 2], o[4 * n + 3]);
            word_affine<0x54>(w[2 * n] & 0xF0F0F0F0u, o_hi, s_hi, c_hi, o[16 + 4 * n], o[16 + 4 * n + 1]);
            word_affine<0x54>(w[2 * n + 1] & 0xF0F0F0F0u, o_hi, s_hi, c_hi, o[16 + 4 * n + 2], o[16 + 4 * n + 3]);
        }
    }
};

// Q5_K: the device record is the Q4_K record followed by the 32 bytes of fifth bits (bit s of byte l =
// weight l of sub-block s); a level 0..31 still fits the byte trick, so both halves of the unit go
// through the 0x64 form.
template <> struct Unit<QT_Q5_K> {
    uint4 hdr, q0, q1, h0, h1;
    __device__ __forceinline__ void load(uint32_t rec, uint32_t, int j) {
        hdr = lds128(rec);
        q0 = lds128(rec + 16 + 32 * j);
        q1 = lds128(rec + 32 + 32 * j);
        h0 = lds128(rec + 144);
        h1 = lds128(rec + 160);
    }
    __device__ __forceinline__ void convert(int j, uint32_t (&o)[32]) const {
        int sa, ma, sb, mb;
        q4k_scale_min(hdr.y, hdr.z, hdr.w, 2 * j, sa, ma);
        q4k_scale_min(hdr.y, hdr.z, hdr.w, 2 * j + 1, sb, mb);
        const float d = half_bits_to_float(hdr.x), dmin = half_bits_to_float(hdr.x >> 16);
        __half2 o_lo, s_lo, c_lo, o_hi, s_hi, c_hi;
        centered(d * (float)sa, dmin * (float)ma, as_h2(0x64006400u), o_lo, s_lo, c_lo);
        centered(d * (float)sb, dmin * (float)mb, as_h2(0x64006400u), o_hi, s_hi, c_hi);
        const uint32_t w[8] = {q0.x, q0.y, q0.z, q0.w, q1.x, q1.y, q1.z, q1.w};
        const uint32_t f[8] = {h0.x, h0.y, h0.z, h0.w, h1.x, h1.y, h1.z, h1.w};
#pragma unroll
        for (int n = 0; n < 4; ++n) {     // chunk n = weights 8n..8n+7 of sub-block 2j; chunk 4 + n = those of sub-block 2j + 1
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                const uint32_t fb = f[2 * n + i] >> (2 * j);
                const uint32_t lo = (w[2 * n + i] & 0x0F0F0F0Fu) | ((fb & 0x01010101u) << 4);
                const uint32_t hi = ((w[2 * n + i] >> 4) & 0x0F0F0F0Fu) | ((fb & 0x02020202u) << 3);
                word_affine<0x64>(lo, o_lo, s_lo, c_lo, o[4 * n + 2 * i], o[4 * n + 2 * i + 1]);
                word_affine<0x64>(hi, o_hi, s_hi, c_hi, o[16 + 4 * n + 2 * i], o[16 + 4 * n + 2 * i + 1]);
            }
        }
    }
};

// Q4_0: [8 x fp16 d][nibbles in the Q4_K arrangement]; weight = d q - 8 d, centred at q0 = 8 exactly
template <> struct Unit<QT_Q4_0> {
    uint4 hdr, q0, q1;
    __device__ __forceinline__ void load(uint32_t rec, uint32_t, int j) {
        hdr = lds128(rec);
        q0 = lds128(rec + 16 + 32 * j);
        q1 = lds128(rec + 32 + 32 * j);
    }
    __device__ __forceinline__ void convert(int j, uint32_t (&o)[32]) const {
        const uint32_t dw[4] = {hdr.x, hdr.y, hdr.z, hdr.w};
        uint32_t dd = dw[0];
#pragma unroll
        for (int i = 1; i < 4; ++i)
            if (i == j) dd = dw[i];
        const float da = half_bits_to_float(dd), db = half_bits_to_float(dd >> 16);
        __half2 o_lo, s_lo, c_lo, o_hi, s_hi, c_hi;
        centered(da, 8.f * da, as_h2(0x64006400u), o_lo, s_lo, c_lo);
        centered(db, 8.f * db, as_h2(0x54005400u), o_hi, s_hi, c_hi);
        const uint32_t w[8] = {q0.x, q0.y, q0.z, q0.w, q1.x, q1.y, q1.z, q1.w};
#pragma unroll
        for (int n = 0; n < 4; ++n) {
            word_affine<0x64>(w[2 * n] & 0x0F0F0F0Fu, o_lo, s_lo, c_lo, o[4 * n], o[4 * n + 1]);
            word_affine<0x64>(w[2 * n + 1] & 0x0F0F0F0Fu, o_lo, s_lo, c_lo, o[4 * n + 2], o[4 * n + 3]);
            word_affine<0x54>(w[2 * n] & 0xF0F0F0F0u, o_hi, s_hi, c_hi, o[16 + 4 * n], o[16 + 4 * n + 1]);
            word_affine<0x54>(w[2 * n + 1] & 0xF0F0F0F0u, o_hi, s_hi, c_hi, o[16 + 4 * n + 2], o[16 + 4 * n + 3]);
        }
    }
};

// MXFP4: [8 scale bytes, 8 of padding][per block four words of eight e2m1 codes in weight order]; a look-up
// gives the bytes 64 + value, read as the halves 1024 + 64 + value; the scale 2^(e - 128) multiplies exactly
// as long as it is an fp16 number (2^-24 .. 2^15; products beyond fp16's range saturate to inf like any fp16 product)
template <> struct Unit<QT_MXFP4> {
    uint4 hdr, q0, q1;
    __device__ __forceinline__ void load(uint32_t rec, uint32_t, int j) {
        hdr = lds128(rec);
        q0 = lds128(rec + 16 + 32 * j);
        q1 = lds128(rec + 32 + 32 * j);
    }
    __device__ __forceinline__ void convert(int j, uint32_t (&o)[32]) const {
        const uint32_t ew = (j >> 1) ? hdr.y : hdr.x;
        const uint32_t ee = ew >> (16 * (j & 1));
        const __half2 da = __float2half2_rn(__uint_as_float(e8m0_half_bits(ee & 0xFF)));
        const __half2 db = __float2half2_rn(__uint_as_float(e8m0_half_bits((ee >> 8) & 0xFF)));
        const __half2 o1088 = as_h2(0x64406440u);      // 1024 + 64
        const uint32_t wa[4] = {q0.x, q0.y, q0.z, q0.w}, wb[4] = {q1.x, q1.y, q1.z, q1.w};
#pragma unroll
        for (int n = 0; n < 4; ++n) {     // chunk n = weights 8n .. 8n + 7 of block 2j; chunk 4 + n = those of block 2j + 1
            word_scale<0x64>(mxfp4_bytes(wa[n]), o1088, da, o[4 * n], o[4 * n + 1]);
            word_scale<0x64>(mxfp4_bytes(wa[n] >> 16), o1088, da, o[4 * n + 2], o[4 * n + 3]);
            word_scale<0x64>(mxfp4_bytes(wb[n]), o1088, db, o[16 + 4 * n], o[16 + 4 * n + 1]);
            word_scale<0x64>(mxfp4_bytes(wb[n] >> 16), o1088, db, o[16 + 4 * n + 2], o[16 + 4 * n + 3]);
        }
    }
};

template <> struct Unit<QT_Q8_0> {
    uint4 q[4];
    uint32_t dd;
    // rec: shared address of the 272-byte record [8 x 32 int8][8 x fp16 d]; unit j = native blocks 2j, 2j+1
    __device__ __forceinline__ void load(uint32_t rec, uint32_t, int j) {
#pragma unroll
        for (int i = 0; i < 4; ++i) q[i] = lds128(rec + 64 * j + 16 * i);
        dd = lds32(rec + 256 + 4 * j);
    }
    __device__ __forceinline__ void convert(int, uint32_t (&o)[32]) const {
        const __half2 d_lo = as_h2(__byte_perm(dd, 0, 0x1010)), d_hi = as_h2(__byte_perm(dd, 0, 0x3232));
        const __half2 o1152 = as_h2(0x64806480u);      // bytes are taken as unsigned after ^ 0x80: 1024 + 128 + q
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const __half2 d = i < 2 ? d_lo : d_hi;
            const uint32_t w[4] = {q[i].x, q[i].y, q[i].z, q[i].w};
#pragma unroll
            for (int c = 0; c < 2; ++c) {     // chunk 2i + c
                word_scale<0x64>(w[2 * c] ^ 0x80808080u, o1152, d, o[8 * i + 4 * c], o[8 * i + 4 * c + 1]);
                word_scale<0x64>(w[2 * c + 1] ^ 0x80808080u, o1152, d, o[8 * i + 4 * c + 2], o[8 * i + 4 * c + 3]);
            }
        }
    }
};

template <> struct Unit<QT_Q6_K> {
    uint4 l[4], hq[2];
    uint32_t sc4, d16;
    // rec: shared address of the 208-byte record [ql 128][qh 64][sc 16], dptr: of its fp16 d.  Unit u is
    // quadrants 2(u&1), 2(u&1)+1 of half u>>1: 64 bytes of ql (low nibbles for even u, high for odd),
    // 32 bytes of qh (bit pair 2(u&1) + quarter/2), four int8 scales (one per 16 weights).
    __device__ __forceinline__ void load(uint32_t rec, uint32_t dptr, int u) {
        const int hh = u >> 1;
#pragma unroll
        for (int i = 0; i < 4; ++i) l[i] = lds128(rec + 64 * hh + 16 * i);
        hq[0] = lds128(rec + 128 + 32 * hh);
        hq[1] = lds128(rec + 144 + 32 * hh);
        sc4 = lds32(rec + 192 + 8 * hh + 4 * (u & 1));
        d16 = lds16(dptr);
    }
    __device__ __forceinline__ void convert(int u, uint32_t (&o)[32]) const {
        const float d = half_bits_to_float(d16);
        const int lsh = 4 * (u & 1);
        const __half2 o1056 = as_h2(0x64206420u);      // 1024 + 32
#pragma unroll
        for (int qd = 0; qd < 4; ++qd) {
            const __half2 s = __float2half2_rn(d * (float)(int)(int8_t)(sc4 >> (8 * qd)));
            const int hsh = lsh + 2 * (qd >> 1);
            const uint32_t lw[4] = {l[qd].x, l[qd].y, l[qd].z, l[qd].w};
            const uint32_t hw[4] = {hq[qd & 1].x, hq[qd & 1].y, hq[qd & 1].z, hq[qd & 1].w};
#pragma unroll
            for (int cc = 0; cc < 2; ++cc) {     // chunk 2 qd + cc
                uint32_t v[2];
#pragma unroll
                for (int i = 0; i < 2; ++i)
                    v[i] = ((lw[2 * cc + i] >> lsh) & 0x0F0F0F0Fu) | (((hw[2 * cc + i] >> hsh) & 0x03030303u) << 4);
                word_scale<0x64>(v[0], o1056, s, o[8 * qd + 4 * cc], o[8 * qd + 4 * cc + 1]);
                word_scale<0x64>(v[1], o1056, s, o[8 * qd + 4 * cc + 2], o[8 * qd + 4 * cc + 3]);
            }
        }
    }
};

// ---- CTA pairs ------------------------------------------------------------------------------------

__device__ __forceinline__ uint32_t cluster_ctarank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
// shared::cluster address of the same shared-memory location in CTA `rank` of the cluster
__device__ __forceinline__ uint32_t mapa_rank(uint32_t saddr, uint32_t rank) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(saddr), "r"(rank));
    return r;
}
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t cluster_addr) {
    asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}
__device__ __forceinline__ void cluster_sync_all() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// 2-D tiled TMA load into this CTA's shared memory whose bytes are counted on a barrier given by
// its shared::cluster address (here: the leader's); no multicast
__device__ __forceinline__ void tma_load_2d_pair(uint32_t dst, const CUtensorMap *map, int x, int y, uint32_t bar_cluster) {
    asm volatile(
        "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
        ::"r"(dst), "l"(map), "r"(bar_cluster), "r"(x), "r"(y)
        : "memory");
}
__device__ __forceinline__ void umma_f16_pair(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
}
// arrives on the barrier at this offset in both CTAs once the MMAs issued so far have completed
__device__ __forceinline__ void umma_commit_pair(uint32_t bar) {
    const uint16_t mask = 3;
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(bar), "h"(mask)
                 : "memory");
}

// the same MMA with the A operand in tensor memory (this CTA's 128 rows in its own lanes, the peer's in its)
__device__ __forceinline__ void umma_f16_pair_ts(uint32_t tmem_d, uint32_t tmem_a, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
        ::"r"(tmem_d), "r"(tmem_a), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
}
// 32 registers of one thread -> 32 consecutive columns of the thread's tensor-memory lane
__device__ __forceinline__ void tmem_st32(uint32_t taddr, const uint32_t (&r)[32]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
        "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, "
        "%17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};"
        ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]),
          "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]), "r"(r[17]), "r"(r[18]), "r"(r[19]),
          "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]), "r"(r[29]),
          "r"(r[30]), "r"(r[31])
        : "memory");
}
__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// tensor-memory management of the pair: one warp of each CTA executes these (every tcgen05
// instruction of a kernel names the same CTA group)
__device__ __forceinline__ void tmem_alloc_pair(uint32_t smem_dst, uint32_t ncols) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_dst), "r"(ncols) : "memory");
}
__device__ __forceinline__ void tmem_relinquish_pair() {
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc_pair(uint32_t taddr, uint32_t ncols) {
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}

// ---- activations ----------------------------------------------------------------------------------

// Activations -> fp16, the format the weights are dequantized to (both tensor-core operands must
// share one format), rounding to nearest even.  fp16 has three more mantissa bits than bf16 but a
// narrower exponent: bf16 values between 2^-14 and 65504 in magnitude convert exactly, larger ones
// (infinities too) saturate to +-65504, smaller ones lose bits as fp16 subnormals or flush to zero (below 2^-25).
// NaN stays NaN (fminf and fmaxf would return the bound).
__device__ __forceinline__ uint32_t to_h2_sat(float lo, float hi) {
    uint32_t r;
    asm("{\n\t.reg .f32 a, b;\n\t"
        "max.NaN.f32 a, %1, %3;\n\tmin.NaN.f32 a, a, %4;\n\t"
        "max.NaN.f32 b, %2, %3;\n\tmin.NaN.f32 b, b, %4;\n\t"
        "cvt.rn.f16x2.f32 %0, a, b;\n\t}"
        : "=r"(r)
        : "f"(hi), "f"(lo), "f"(-65504.f), "f"(65504.f));
    return r;
}

// eight elements from src + off -> 16 bytes of fp16 at dst (both 16-byte aligned)
template <bool SRC_BF16>
__device__ __forceinline__ void convert_vec8(const void *__restrict__ src, long long off, uint16_t *__restrict__ dst) {
    float f[8];
    if (SRC_BF16) {
        const uint4 v = *reinterpret_cast<const uint4 *>(reinterpret_cast<const uint16_t *>(src) + off);
        const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            f[2 * e] = __uint_as_float(w[e] << 16);
            f[2 * e + 1] = __uint_as_float(w[e] & 0xFFFF0000u);
        }
    } else {
        const float4 a = *reinterpret_cast<const float4 *>(reinterpret_cast<const float *>(src) + off);
        const float4 b = *reinterpret_cast<const float4 *>(reinterpret_cast<const float *>(src) + off + 4);
        f[0] = a.x, f[1] = a.y, f[2] = a.z, f[3] = a.w, f[4] = b.x, f[5] = b.y, f[6] = b.z, f[7] = b.w;
    }
    uint4 o;
    o.x = to_h2_sat(f[0], f[1]);
    o.y = to_h2_sat(f[2], f[3]);
    o.z = to_h2_sat(f[4], f[5]);
    o.w = to_h2_sat(f[6], f[7]);
    *reinterpret_cast<uint4 *>(dst) = o;
}

// ---- tensor maps ----------------------------------------------------------------------------------

typedef CUresult (*EncodeTiledFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
                                  const cuuint64_t *, const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn lookup_encode_fn() {
    void *ptr = nullptr;
    cudaDriverEntryPointQueryResult qres;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &ptr, cudaEnableDefault, &qres) == cudaSuccess &&
        qres == cudaDriverEntryPointSuccess)
        return reinterpret_cast<EncodeTiledFn>(ptr);
    return nullptr;
}
EncodeTiledFn encode_fn() {
    static const EncodeTiledFn fn = lookup_encode_fn();     // initialised once, also under concurrent first calls
    return fn;
}

}  // namespace
}  // namespace b200q

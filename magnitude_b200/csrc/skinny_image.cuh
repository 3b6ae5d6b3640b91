// Activations of the small-batch route -> the fp16 operand fragments its MMAs read.
#pragma once

#include <cuda_fp16.h>

#include "skinny_types.h"

namespace b200q {
namespace {

__device__ __forceinline__ uint32_t sk_u32(__half2 v) { return *reinterpret_cast<uint32_t *>(&v); }

// ---- activations -> fragments ---------------------------------------------------------------------------
// Lane L of a warp holds elements 8 L .. 8 L + 7 of a record; they are the 16 bytes that MMA lane t of a token's quad
// reads for unit u (SUB16: 8 bytes each of lanes t and t + 1).  Which weights a lane meets there is set by the packed
// layout and by the kernel's loads:
//   K (Q4_K; Q5_K at more than 16 tokens): a 16-byte load at 64 jj + 16 t of the nibbles brings weights
//                    128 jj + 64 (t >> 1) + 16 (t & 1) + i (low) and + 32 (high); unit = 4 jj + 2 high + (i >> 3)
//   Q6 (Q6_K at more than 16 tokens): a 16-byte load at 64 hh + 16 t brings 128 hh + 16 t + i (low) and + 64 (high);
//                    unit = 4 hh + 2 high + (i >> 3)
//   BLOCK:           unit = 32-weight block, lane t its weights 8 t .. 8 t + 7: an MMA stays inside one sub-block
//   SUB32 (Q5_K up to 16 tokens): as BLOCK
//   SUB16 (Q6_K up to 16 tokens): unit = 32-weight quadrant, its 16-weight sub-blocks one after the other, lane t weights
//                    4 t .. 4 t + 3 of each
// K, SUB32: sums over the 32-weight sub-blocks as one more fragment; SUB16: over the 16-weight ones as two (high, low).
enum { SK_K = 0, SK_Q6 = 1, SK_BLOCK = 2, SK_SUB32 = 3, SK_SUB16 = 4 };
__host__ __device__ constexpr int sk_map(int qt, int nt) {
    return qt == QT_Q4_K || (qt == QT_Q5_K && nt > 2) ? SK_K
           : qt == QT_Q5_K                            ? SK_SUB32
           : qt == QT_Q6_K                            ? (nt <= 2 ? SK_SUB16 : SK_Q6)
                                                      : SK_BLOCK;
}
template <int MAP> constexpr int kSumBytes = MAP == SK_SUB16 ? 512 : 256;      // of a token tile (sk_sum_bytes)
template <int MAP> __device__ __forceinline__ void sk_unit(int L, int &u, int &t) {
    if (MAP == SK_K) {
        t = 2 * ((L >> 3) & 1) + ((L >> 1) & 1);
        u = (L >> 4) * 4 + ((L >> 2) & 1) * 2 + (L & 1);
    } else if (MAP == SK_Q6) {
        t = (L & 7) >> 1;
        u = (L >> 4) * 4 + ((L >> 3) & 1) * 2 + (L & 1);
    } else {
        u = L >> 2;
        t = MAP == SK_SUB16 ? 2 * (L & 1) : L & 3;
    }
}

__device__ __forceinline__ void sk_load_x(const SkJob &J, long long at, int k, float (&v)[8]) {
    if (J.x_vec_ok && k + 8 <= J.K) {
        if (J.x_is_bf16) {
            const uint4 w = __ldcg(reinterpret_cast<const uint4 *>(reinterpret_cast<const uint16_t *>(J.x) + at));
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                v[2 * i] = __uint_as_float(word_of(w, i) << 16);
                v[2 * i + 1] = __uint_as_float(word_of(w, i) & 0xFFFF0000u);
            }
        } else {
            const float4 a = __ldcg(reinterpret_cast<const float4 *>(reinterpret_cast<const float *>(J.x) + at));
            const float4 b = __ldcg(reinterpret_cast<const float4 *>(reinterpret_cast<const float *>(J.x) + at + 4));
            v[0] = a.x, v[1] = a.y, v[2] = a.z, v[3] = a.w, v[4] = b.x, v[5] = b.y, v[6] = b.z, v[7] = b.w;
        }
        return;
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        v[i] = 0.f;
        if (k + i >= J.K) continue;
        if (J.x_is_bf16) v[i] = __uint_as_float((uint32_t)__ldcg(reinterpret_cast<const unsigned short *>(J.x) + at + i) << 16);
        else v[i] = __ldcg(reinterpret_cast<const float *>(J.x) + at + i);
    }
}

// One warp: token `tok`, elements v of its lanes, into a record's image (in shared or global memory).  Token slots past M
// are left as they are: nothing reads their results.
template <int MAP> __device__ __forceinline__ void sk_put_image(const float (&v)[8], int tok, int lane, uint8_t *img, int NT, int P) {
    uint32_t top = 0;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const uint32_t a = __float_as_uint(v[i]) & 0x7FFFFFFFu;
        top = max(top, a < 0x7F800000u ? a : 0u);          // infinities and NaN keep their own way through fp16
    }
    top = __reduce_max_sync(0xFFFFFFFFu, top);
    const int e = top ? min(135 - (int)(top >> 23), 126) : 0;        // largest value -> [2^8, 2^9)
    const float scale = __uint_as_float((uint32_t)(e + 127) << 23);
    uint32_t hi[4], lo[4];
    float sum = 0.f;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const float a = v[2 * i] * scale, b = v[2 * i + 1] * scale;
        const __half2 h = __floats2half2_rn(a, b);
        const float2 f = __half22float2(h);
        hi[i] = sk_u32(h);
        sum += f.x + f.y;
        if (P == 2) {
            const __half2 l = __floats2half2_rn(a - f.x, b - f.y);
            const float2 r = __half22float2(l);
            lo[i] = sk_u32(l);
            sum += r.x + r.y;
        }
    }
    int u, t;
    sk_unit<MAP>(lane, u, t);
    const int nt = tok >> 3, g = tok & 7;
    // k order of a lane's weights: (0, 2) (1, 3) | (4, 6) (5, 7)
    auto order = [](const uint32_t (&h)[4]) {
        return make_uint4(__byte_perm(h[0], h[1], 0x5410), __byte_perm(h[0], h[1], 0x7632), __byte_perm(h[2], h[3], 0x5410),
                          __byte_perm(h[2], h[3], 0x7632));
    };
    uint8_t *at = img + (nt * 8 + u) * 512 + (g * 4 + t) * 16;
    auto put = [&](uint8_t *to, const uint4 &f) {
        if (MAP == SK_SUB16) {
            to += 8 * ((lane >> 1) & 1);
            *reinterpret_cast<uint2 *>(to) = make_uint2(f.x, f.y);
            *reinterpret_cast<uint2 *>(to + 16) = make_uint2(f.z, f.w);
        } else {
            *reinterpret_cast<uint4 *>(to) = f;
        }
    };
    put(at, order(hi));
    if (P == 2) put(at + NT * 4096, order(lo));
    uint8_t *xs = img + P * NT * 4096;
    if (MAP == SK_K || MAP == SK_SUB32) {
        // sum over the 32-weight sub-block = four lanes, as two fp16 halves: k slots 0..7 (high), 8..15 (low) by sub-block
        sum += __shfl_xor_sync(0xFFFFFFFFu, sum, 1);
        sum += __shfl_xor_sync(0xFFFFFFFFu, sum, 2);
        if ((lane & 3) == 0) {
            const int b = lane >> 2;
            const __half xh = __float2half_rn(sum), xl = __float2half_rn(sum - __half2float(xh));
            __half *q = reinterpret_cast<__half *>(xs + (nt * 32 + g * 4 + (b >> 1)) * 8 + (b & 1) * 2);
            q[0] = xh;
            q[2] = xl;
        }
    }
    if (MAP == SK_SUB16) {
        // sum over the 16-weight sub-block = two lanes: k slot = sub-block (in weight order, as the scales), high halves
        // in the first fragment, low ones in the second
        sum += __shfl_xor_sync(0xFFFFFFFFu, sum, 1);
        if ((lane & 1) == 0) {
            const int b = lane >> 1;
            const __half xh = __float2half_rn(sum), xl = __float2half_rn(sum - __half2float(xh));
            __half *q = reinterpret_cast<__half *>(xs + (nt * 64 + g * 4 + ((b & 7) >> 1)) * 8 + (b >> 3) * 4 + (b & 1) * 2);
            q[0] = xh;
            q[128] = xl;
        }
    }
    if (lane == 0) *reinterpret_cast<uint32_t *>(xs + NT * kSumBytes<MAP> + tok * 4) = (uint32_t)(127 - e) << 23;
}

template <int MAP> __device__ __forceinline__ void sk_make_image(const SkJob &J, int rec, int tok, int lane, uint8_t *img, int NT, int P) {
    float v[8];
    const int k = rec * SB + 8 * lane;
    sk_load_x(J, (long long)tok * J.ldx + k, k, v);
    sk_put_image<MAP>(v, tok, lane, img, NT, P);
}

}  // namespace
}  // namespace b200q

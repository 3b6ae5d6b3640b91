// What the host side of the small-batch route (skinny.cu) and its kernels (skinny_kernel.cuh) share.
#pragma once

#include <cstddef>

#include <cuda.h>

#include "common.cuh"

namespace b200q {

// Consumer warps, 16 weight rows each: as many as the registers of a warp (accumulators grow with the tokens) allow
__host__ __device__ constexpr int sk_warps(int nt) { return nt <= 2 ? 16 : 12; }
__host__ __device__ constexpr int sk_tile_rows(int nt) { return 16 * sk_warps(nt); }
// running sums in double (up to 16 tokens) or float
__host__ __device__ constexpr bool sk_double(int nt) { return nt <= 2; }
// slots [begin(b), begin(b + 1)) belong to block b
__host__ __device__ inline int sk_slot_begin(int slots, int grid, int b) { return (int)((long long)slots * b / grid); }
// the block that a slot belongs to
__host__ __device__ inline int sk_slot_owner(int slots, int grid, int s) { return (int)((((long long)s + 1) * grid - 1) / slots); }
// activation image of one record: fragments [plane][token tile][unit 8][lane 32] x 16 bytes, block-sum fragments
// [token tile][one, Q6_K up to 16 tokens two][lane 32] x 8 bytes, 1 / scale [token] x 4 bytes
__host__ __device__ constexpr int sk_sum_bytes(int qt, int nt) { return qt == QT_Q6_K && nt <= 2 ? 512 : 256; }
__host__ __device__ constexpr int sk_image_bytes(int nt, int planes, int sum_bytes) { return nt * (planes * 4096 + sum_bytes + 32); }

// shared memory: a stage holds a slot's packed records (Q6_K: and its rows' 16-byte groups of fp16 d) and the record's image
constexpr int kSkHeadBytes = 256, kSkMaxDepth = 8;
__host__ __device__ constexpr int sk_w_bytes(int qt, int nt) { return sk_tile_rows(nt) * rec_bytes(qt); }
__host__ __device__ constexpr int sk_d_bytes(int qt, int nt) { return qt == QT_Q6_K ? sk_tile_rows(nt) * 16 : 0; }
__host__ __device__ constexpr int sk_stage_bytes(int qt, int nt, int planes) {
    return (sk_w_bytes(qt, nt) + sk_d_bytes(qt, nt) + sk_image_bytes(nt, planes, sk_sum_bytes(qt, nt)) + 127) / 128 * 128;
}
__host__ __device__ constexpr int sk_depth(int qt, int nt, int planes) {
    return (232448 - kSkHeadBytes) / sk_stage_bytes(qt, nt, planes) < kSkMaxDepth ? (232448 - kSkHeadBytes) / sk_stage_bytes(qt, nt, planes) : kSkMaxDepth;
}

struct SkJob {
    CUtensorMap w, wtail, d, dtail;    // packed records: whole chunks / the shorter last chunk; Q6_K: their d groups
    uint8_t *img;                      // activation images [record]
    const void *x;                     // activations [M][K], bf16 or fp32
    void *y;
    long long ldx, ldy;
    int N, M, K, nsb, nfull, tiles;    // nfull: whole chunks of 8 records
    int x_is_bf16, x_vec_ok, y_is_bf16;
    int slot0;                         // first slot of this job in the launch's order
    int xwarp0;                        // first warp of the preparation that works on this job (none if the image is another job's)
};
constexpr int kSkMaxJobs = 32;
constexpr int kSkInline = 4;           // products of a call
constexpr int kSkMaxGrid = 160;

// Kernel parameters.  The products' descriptions travel in them, a plan's too (20 KB of the 32 that a launch may have): tensor maps
// in global memory need a proxy fence before every use, which cost more (us, fence / parameters: sixteen Q4_K 6144 x 4096 products
// as a plan, 4 rows 66.6 / 64.9; six Q6_K 4096 x 14336 calls, 8 rows 135.7 / 132.0), and an upload to wait for.
template <int N> struct SkParamsOf {
    double *sums;                      // [grid][consumer warps][accumulators][32] sums of the tile that begins in a block and goes on
    unsigned *count;                   // [grid][consumer warps] parts of it seen so far; both zero between launches
    int *status;
    int njobs, slots;
    int direct;                        // 1: every block makes the images of its slots (at most sk_depth of them) itself
    int NT, P, xwarps;                 // token tiles, activation planes, warps of the preparation
    SkJob jobs[N];
};
using SkParams = SkParamsOf<kSkMaxJobs>;
using SkFew = SkParamsOf<kSkInline>;   // the same but for the jobs that are not there
static_assert(sizeof(SkParams) <= 32764 && offsetof(SkFew, jobs) == offsetof(SkParams, jobs), "kernel parameters");

}  // namespace b200q

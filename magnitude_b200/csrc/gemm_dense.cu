// Prefill in two launches: the packed weights become a dense fp16 matrix once, then a dense GEMM runs on it.
//
// The kernels of gemm_tc.cu dequantize a weight tile again for every token tile and pay the hand-over
// from the dequantizing warps to the tensor cores on every K-step (about 970 cycles for a K-step whose
// MMAs take 512, whatever the tile's width).  Here
//   * dense_prep_kernel turns the rows of all the weights of a call (which share x, type and K) into
//     fp16 rows of a workspace, and the activations into fp16 rows of another, in one launch;
//   * dense_gemm_kernel multiplies the two: CTA pairs (tcgen05.mma.cta_group::2, 256 weight rows x up to
//     256 tokens), both operands by tiled TMA, so that one warp feeds and one thread issues, and the tile
//     width is chosen so that the pairs share the tiles evenly.
// The weights' values, the order in which K is added up and so the results are those of the one-launch
// kernels, bit for bit.  The workspace has a fixed size (kDenseScratchBytes); larger weights go through it
// in panels of rows.
#include <algorithm>
#include <atomic>

#include "kernels.h"
#include "tc_common.cuh"

namespace b200q {
namespace {

constexpr int kBK = 64;                       // K-step: one 128-byte swizzle row of fp16
constexpr int kRows = 128;                    // weight rows per CTA
constexpr int kStripe = 2 * kRows;            // weight rows per pair and tile
constexpr int kMaxStages = 12;
constexpr int kABytes = kRows * kBK * 2;      // 16 KB
constexpr int kDataBytes = 224 * 1024;        // operand stages; how many fit depends on the tile's width
constexpr int kEpiWarps = 4;
constexpr int kThreads = (2 + kEpiWarps) * 32;
constexpr int kTmemCols = 512;                // two accumulators of 256 columns
constexpr int kMaxSeg = kDenseMaxWeights;

// ---- preparation ------------------------------------------------------------------------------------

struct PrepSeg {
    const uint8_t *w;        // streaming-layout rows
    int tile_begin;          // first prep tile (4 rows x one chunk of 2048 weights) of this segment
    int group0;              // first 4-row group of the panel
    long long row0;          // row of the workspace that receives the panel's first row
};
struct PrepParams {
    PrepSeg seg[kMaxSeg];
    int nseg, tiles, nchunks, nsb;
    __half *dst;             // [rows][ldd]
    long long ldd;
    int x_blocks;            // blocks that convert activations (the first ones of the grid)
    const void *x;
    long long ldx;
    uint16_t *xdst;
    long long xldd;
    int M, K8;
};

constexpr int kPrepThreads = 128;

// Block = one tile of the streaming layout (4 rows x up to 8 records, contiguous): warp = row, lane = 64-weight
// unit.  The packed bytes come in with 16-byte loads; a lane's 64 halves leave through shared memory so that
// every store of the warp writes 512 consecutive bytes of its row.  Bound by memory: 0.56 bytes read and
// 2 written per Q4_K weight.
template <int QT, bool SRC_BF16>
__global__ void __launch_bounds__(kPrepThreads) dense_prep_kernel(const PrepParams p) {
    __shared__ __align__(16) uint8_t in[kRowGroup * kChunkRecs * rec_bytes(QT) + kRowGroup * 16];
    __shared__ __align__(16) uint8_t out[kRowGroup * 4096];
    pdl_launch_dependents();
    if ((int)blockIdx.x < p.x_blocks) {
        pdl_wait();              // X may come from the launch before, which may also still read the copies
        const unsigned total = (unsigned)p.M * (unsigned)p.K8;
        for (unsigned i = blockIdx.x * kPrepThreads + threadIdx.x; i < total; i += (unsigned)p.x_blocks * kPrepThreads) {
            const unsigned m = i / (unsigned)p.K8, c = i - m * (unsigned)p.K8;
            convert_vec8<SRC_BF16>(p.x, (long long)m * p.ldx + 8 * c, p.xdst + (long long)m * p.xldd + 8 * c);
        }
        return;
    }
    const int tile = blockIdx.x - p.x_blocks;
    int s = 0;
    while (s + 1 < p.nseg && tile >= p.seg[s + 1].tile_begin) ++s;
    const PrepSeg &sg = p.seg[s];
    const int q = tile - sg.tile_begin, g = q / p.nchunks, c = q - g * p.nchunks;
    const int row_b = (int)chunk_row_bytes(QT, c, p.nsb);
    const uint8_t *src = sg.w + tile_off(QT, sg.group0 + g, c, 0, p.nsb);
    for (int i = threadIdx.x; i < kRowGroup * row_b / 16; i += kPrepThreads)
        reinterpret_cast<uint4 *>(in)[i] = __ldg(reinterpret_cast<const uint4 *>(src) + i);
    __syncthreads();
    pdl_wait();                  // the weights depend on no launch, the workspace on the GEMM that last read it
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, rec = lane >> 2;
    const int nrec = min(kChunkRecs, p.nsb - c * kChunkRecs);
    const uint32_t row_s = smem_u32(in) + warp * row_b, out_s = smem_u32(out) + warp * 4096;
    if (rec < nrec) {
        Unit<QT> u;
        u.load(row_s + rec * rec_bytes(QT), row_s + nrec * rec_bytes(QT) + 2 * rec, lane & 3);
        uint32_t o[32];
        u.convert(lane & 3, o);
        store_row(o, out_s + lane * 128, lane & 7);
    }
    __syncwarp();
    uint8_t *d = reinterpret_cast<uint8_t *>(p.dst + (sg.row0 + (long long)g * kRowGroup + warp) * p.ldd) + c * 4096 + lane * 16;
    for (int i = 0; i < nrec; ++i) {
        const int l = 4 * i + (lane >> 3);          // the lane that converted these eight weights
        *reinterpret_cast<uint4 *>(d + i * 512) = lds128(out_s + l * 128 + (((lane & 7) ^ (l & 7)) << 4));
    }
}

// ---- the GEMM ---------------------------------------------------------------------------------------

struct DenseSeg {
    void *y;                 // row m at y + m * ldy elements
    long long ldy;
    int n;                   // rows of the panel
    int stripe_begin;        // first 256-row stripe of the workspace
};
struct DenseParams {
    DenseSeg seg[kMaxSeg];
    int nseg, y_is_bf16;
    int M, ksteps;
    int bn;                  // tokens per tile, a multiple of 32 up to 256
    int stages, stage_bytes; // operand ring: 128 weight rows and bn / 2 tokens per stage and CTA
    int m_tiles, tiles;
    // The last round would leave pairs idle: the tiles from `whole` on (of bn tokens) are cut into `split`
    // tiles of `bn2` tokens each, the last of them what is left of bn.
    int whole, split, bn2;
    int *status;
};

struct DenseTile {
    int stripe, t0, width;   // 256-row stripe, first token, tokens
    int box;                 // tokens that the two activation loads bring: width or more
};
__device__ __forceinline__ DenseTile dense_tile(const DenseParams &p, int tile) {
    int sub = 0, w = p.bn;
    if (tile >= p.whole) {
        const int u = tile - p.whole, q = u / p.split;
        sub = u - q * p.split;
        tile = p.whole + q;
        w = p.bn2;
    }
    DenseTile t;
    t.stripe = tile / p.m_tiles;
    t.t0 = (tile - t.stripe * p.m_tiles) * p.bn + sub * w;
    t.width = min(w, p.bn - sub * w);
    t.box = w;
    return t;
}

struct DenseSmem {
    uint64_t full[kMaxStages];      // leader's copy is used: its own arrival + both CTAs' bytes
    uint64_t empty[kMaxStages];
    uint64_t tmem_full[2];
    uint64_t tmem_empty[2];      // leader's copy is used: 4 local + 4 remote warp arrivals
    uint32_t tmem_base;
    int abort;
};

__device__ __forceinline__ bool dense_wait(uint32_t bar, uint32_t parity, DenseSmem *sm, int *status) {
#pragma unroll 1
    for (int i = 0; i < (1 << 12); ++i)
        if (mbar_try_wait_hint(bar, parity, 40)) return true;
    volatile int *ab = &sm->abort;
    const uint64_t t0 = globaltimer_ns();
#pragma unroll 1
    while (true) {
#pragma unroll 1
        for (int i = 0; i < 64; ++i)
            if (mbar_try_wait(bar, parity)) return true;
        if (*ab) return false;
        if (globaltimer_ns() - t0 > kWaitLimitNs) {
            *ab = 1;
            atomicMax(status, DEV_ERR_PIPE_TIMEOUT);
            return false;
        }
    }
}

// One cluster of two CTAs per tile at a time; see gemm_tc.cu for the pair protocol (which barriers live in
// the leader, what crosses the pair).  Warp 0 feeds, warp 1 issues (leader only), warps 2..5 store.
__global__ void __launch_bounds__(kThreads, 1) dense_gemm_kernel(const DenseParams p, const __grid_constant__ CUtensorMap amap,
                                                                 const __grid_constant__ CUtensorMap bmap, const __grid_constant__ CUtensorMap bmap2) {
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    uint8_t *smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    const uint32_t stage_s = smem_u32(smem);
    DenseSmem *sm = reinterpret_cast<DenseSmem *>(smem + kDataBytes);
    const uint32_t full_s = smem_u32(sm->full), empty_s = smem_u32(sm->empty);
    const uint32_t tfull_s = smem_u32(sm->tmem_full), tempty_s = smem_u32(sm->tmem_empty);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t rank = cluster_ctarank();
    const int pair = blockIdx.x >> 1, n_pairs = gridDim.x >> 1;

    if (threadIdx.x == 0) {
        for (int i = 0; i < p.stages; ++i) {
            mbar_init(full_s + 8 * i, 1);
            mbar_init(empty_s + 8 * i, 1);
        }
        for (int i = 0; i < 2; ++i) {
            mbar_init(tfull_s + 8 * i, 1);
            mbar_init(tempty_s + 8 * i, 2 * kEpiWarps);
        }
        sm->abort = 0;
        mbar_fence_init();
        fence_proxy_async();
    }
    if (warp == 0) {
        tmem_alloc_pair(smem_u32(&sm->tmem_base), kTmemCols);
        tmem_relinquish_pair();
    }
    tc_fence_before();
    __syncthreads();
    cluster_sync_all();
    tc_fence_after();
    const uint32_t tmem_base = *reinterpret_cast<volatile uint32_t *>(&sm->tmem_base);
    pdl_launch_dependents();

    if (warp == 0) {
        if (lane == 0) {
            pdl_wait();                  // the preparation launch wrote both operands
            const uint32_t full_leader = mapa_rank(full_s, 0);
            int stage = 0, phase = 1;    // a fresh barrier's "previous" phase counts as complete
            bool ok = true;
            for (int tile = pair; tile < p.tiles && ok; tile += n_pairs) {
                const DenseTile t = dense_tile(p, tile);
                const int arow = t.stripe * kStripe + (int)rank * kRows, brow = t.t0 + (int)rank * (t.width >> 1);
                const uint32_t bytes_pair = 2u * (kABytes + (uint32_t)(t.box >> 1) * kBK * 2);
                const CUtensorMap *bm = tile < p.whole ? &bmap : &bmap2;
                for (int ks = 0; ks < p.ksteps; ++ks) {
                    ok = dense_wait(empty_s + 8 * stage, phase, sm, p.status);
                    if (!ok) break;
                    if (rank == 0) mbar_expect_tx(full_s + 8 * stage, bytes_pair);
                    const uint32_t a = stage_s + stage * p.stage_bytes;
                    tma_load_2d_pair(a, &amap, ks * kBK, arow, full_leader + 8 * stage);
                    tma_load_2d_pair(a + kABytes, bm, ks * kBK, brow, full_leader + 8 * stage);
                    if (++stage == p.stages) stage = 0, phase ^= 1;
                }
            }
        }
    } else if (warp == 1) {
        // The whole warp walks the loop and an elected lane issues: under `if (lane == 0)` the compiler cannot
        // see that one lane at most is active, and an MMA then cost 160 cycles whatever its width
        // (4096 x 14336 weights, 512 tokens, 128-token tiles: 110 us a call; this way 84).
        if (rank == 0) {
            const uint64_t adesc0 = make_desc_sw128(stage_s), bdesc0 = make_desc_sw128(stage_s + kABytes);
            const uint32_t step = (uint32_t)p.stage_bytes >> 4, stages = (uint32_t)p.stages;
            uint32_t stage = 0, phase = 0;
            int tcount = 0;
            bool seen = false;           // this K-step's operands were found ready by the previous probe
            for (int tile = pair; tile < p.tiles; tile += n_pairs, ++tcount) {
                const int buf = tcount & 1;
                const uint32_t idesc = (1u << 4) | ((uint32_t)(dense_tile(p, tile).width >> 3) << 17) | ((uint32_t)(kStripe >> 4) << 24);
                bool ok = __all_sync(0xFFFFFFFFu, dense_wait(tempty_s + 8 * buf, ((tcount >> 1) & 1) ^ 1, sm, p.status));
                if (!ok) break;
                const uint32_t d_tmem = tmem_base + buf * 256;
                for (int ks = 0; ks < p.ksteps; ++ks) {
                    if (!seen) {
                        ok = __all_sync(0xFFFFFFFFu, dense_wait(full_s + 8 * stage, phase, sm, p.status));
                        if (!ok) break;
                    }
                    tc_fence_after();
                    uint32_t nstage = stage + 1, nphase = phase;
                    if (nstage == stages) nstage = 0, nphase ^= 1;
                    seen = __all_sync(0xFFFFFFFFu, mbar_test_wait(full_s + 8 * nstage, nphase));
                    const uint64_t adesc = adesc0 + stage * step, bdesc = bdesc0 + stage * step;
                    if (elect_one()) {
#pragma unroll
                        for (int kk = 0; kk < kBK / 16; ++kk) umma_f16_pair(d_tmem, adesc + 2 * kk, bdesc + 2 * kk, idesc, (ks | kk) != 0);
                        umma_commit_pair(empty_s + 8 * stage);
                    }
                    __syncwarp();
                    stage = nstage, phase = nphase;
                }
                if (!ok) break;
                if (elect_one()) umma_commit_pair(tfull_s + 8 * buf);
                __syncwarp();
            }
        }
    } else {
        const int q = warp & 3;          // TMEM lane quadrant this warp may read
        const uint32_t tempty_leader = mapa_rank(tempty_s, 0);
        int tcount = 0;
        for (int tile = pair; tile < p.tiles; tile += n_pairs, ++tcount) {
            const DenseTile t = dense_tile(p, tile);
            const int stripe = t.stripe;
            const int buf = tcount & 1;
            bool ok = dense_wait(tfull_s + 8 * buf, (tcount >> 1) & 1, sm, p.status);
            ok = __all_sync(0xFFFFFFFFu, ok);
            if (!ok) break;
            tc_fence_after();
            int s = 0;
            while (s + 1 < p.nseg && stripe >= p.seg[s + 1].stripe_begin) ++s;
            const int n = (stripe - p.seg[s].stripe_begin) * kStripe + (int)rank * kRows + q * 32 + lane;
            const bool row_ok = n < p.seg[s].n;
            const long long ldy = p.seg[s].ldy;
            const int m0 = t.t0, mlim = min(t.width, p.M - m0);
            for (int c0 = 0; c0 < mlim; c0 += 32) {
                uint32_t v[32];
                tmem_ld32(tmem_base + buf * 256 + ((uint32_t)(q * 32) << 16) + c0, v);
                tmem_ld_wait();
                if (row_ok) {
                    const bool whole = c0 + 32 <= mlim;
                    if (p.y_is_bf16) {
                        __nv_bfloat16 *yp = reinterpret_cast<__nv_bfloat16 *>(p.seg[s].y) + (long long)(m0 + c0) * ldy + n;
#pragma unroll
                        for (int i = 0; i < 32; ++i, yp += ldy)
                            if (whole || c0 + i < mlim) *yp = __float2bfloat16_rn(__uint_as_float(v[i]));
                    } else {
                        float *yp = reinterpret_cast<float *>(p.seg[s].y) + (long long)(m0 + c0) * ldy + n;
#pragma unroll
                        for (int i = 0; i < 32; ++i, yp += ldy)
                            if (whole || c0 + i < mlim) *yp = __uint_as_float(v[i]);
                    }
                }
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive_cluster(tempty_leader + 8 * buf);
        }
    }

    // both CTAs meet (also after an abort, with their loads and MMAs given time to land) before either
    // releases shared or tensor memory
    tc_fence_before();
    __syncthreads();
    if (*reinterpret_cast<volatile int *>(&sm->abort)) {
        const uint64_t t0 = globaltimer_ns();
        while (globaltimer_ns() - t0 < 100000) {
        }
        __syncthreads();
    }
    cluster_sync_all();
    if (warp == 0) {
        __syncwarp();
        tc_fence_after();
        tmem_dealloc_pair(tmem_base, kTmemCols);
    }
}

// Tiles of a panel.  A pair's K-step takes the longer of its MMAs (2 cycles per token, 2.7 at the clock that a
// busy chip keeps) and a fixed 300 cycles or so (operand loads of narrow tiles, the issuing warp's loop), and the
// pairs finish together only if the tiles fill whole rounds: the width is the one whose rounds cost least, with
// the last, partial round cut into as many narrower tiles as there are idle pairs.  Ties go to the wider tile.
double pick_tiles(DenseParams &p, int stripes, int pairs, int bn_override) {
    auto step = [](int bn) { return std::max(2.7 * bn, 300 + 0.75 * bn); };
    double best = -1;
    for (int bn = 256; bn >= 32; bn -= 32) {
        if (bn_override >= 32 && bn_override <= 256 && bn_override % 32 == 0 && bn != bn_override) continue;
        const int m_tiles = (p.M + bn - 1) / bn;
        const long long tiles = (long long)m_tiles * stripes;
        const int left = (int)(tiles % pairs);
        int split = 1, bn2 = bn;
        if (left > 0) {
            bn2 = ((bn + pairs / left - 1) / (pairs / left) + 31) / 32 * 32;
            split = (bn + bn2 - 1) / bn2;
        }
        // the last tile's stores (about 10 cycles per token) are not hidden
        const double cost = (double)(tiles / pairs) * p.ksteps * step(bn) + (left ? p.ksteps * step(bn2) + 10.0 * bn2 : 10.0 * bn);
        if (best >= 0 && cost >= best) continue;
        best = cost;
        p.bn = bn;
        p.bn2 = bn2;
        p.split = split;
        p.m_tiles = m_tiles;
        p.whole = (int)(tiles - left);
        p.tiles = p.whole + left * split;
    }
    return best;             // cycles
}

bool encode_2d(CUtensorMap *map, const void *base, long long cols, long long rows, long long ld, int box_rows) {
    EncodeTiledFn enc = encode_fn();
    if (!enc) return false;
    const cuuint64_t gdim[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
    const cuuint64_t gstride[1] = {(cuuint64_t)ld * 2};
    const cuuint32_t box[2] = {(cuuint32_t)kBK, (cuuint32_t)box_rows};
    const cuuint32_t estride[2] = {1, 1};
    return enc(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, const_cast<void *>(base), gdim, gstride, box, estride, CU_TENSOR_MAP_INTERLEAVE_NONE,
               CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <int QT>
cudaError_t launch_prep(const PrepParams &p, bool bf16, cudaStream_t st) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)(p.x_blocks + p.tiles));
    cfg.blockDim = dim3(kPrepThreads);
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return bf16 ? cudaLaunchKernelEx(&cfg, dense_prep_kernel<QT, true>, p) : cudaLaunchKernelEx(&cfg, dense_prep_kernel<QT, false>, p);
}

}  // namespace

// From 128 rows on both ways are open.  The one-launch kernels dequantize a weight tile per token tile at 0.60 us
// a K-step and round of 256-token tiles, whatever the tiles' width; this one pays for the fp16 copy (written
// and read past L2: about 6 TB/s) and a second launch, then runs at the tensor cores' pace.  Measured (us, one
// launch / two): Q4_K 4096 x 4096, 128 rows 45 / 25, 2048 rows 85 / 62; 14336 x 4096, 256 rows 50 / 58, 384 rows
// 84 / 70, 2048 rows 245 / 201; 28672 x 4096, 256 rows 84 / 109, 512 rows 147 / 143; Q6_K 4096 x 14336, 128 rows
// 136 / 78, 2048 rows 292 / 222; the estimates are within 10 % of these.
bool dense_pays(const DenseLaunch &a) {
    const int pairs = a.sm_count / 2, ksteps = a.Kpad / kBK;
    double fused = 0, rows = 0;
    int stripes = 0;
    for (int i = 0; i < a.nw; ++i) {
        const int s = (a.n[i] + kStripe - 1) / kStripe;
        const long long tiles = (long long)s * ((a.M + 255) / 256);
        fused += 7 + 0.60 * ksteps * (double)((tiles + pairs - 1) / pairs);
        stripes += s;
        rows += a.n[i];
    }
    DenseParams p{};
    p.M = a.M;
    p.ksteps = ksteps;
    const double copy = rows * (row_bytes_for(a.qt, a.Kpad / SB) + 2.0 * a.Kpad) / 6.0e6;
    return 12 + copy + pick_tiles(p, stripes, pairs, 0) / 1900 < fused;
}

cudaError_t dense_gemm_run(const DenseLaunch &a, cudaStream_t st, int *launches) {
    const int nsb = a.Kpad / SB;
    const long long x_ldd = (a.K + 7) & ~7;
    const int pairs = a.sm_count / 2;
    if (a.nw < 1 || a.nw > kMaxSeg || a.M < 1 || pairs < 1) return cudaErrorInvalidValue;
    const long long max_stripes = (long long)(a.scratch_bytes / ((size_t)a.Kpad * 2 * kStripe));
    if (max_stripes < 1) return cudaErrorInvalidValue;

    static std::atomic<int> configured_dev{-1};     // contexts on several threads may launch at once
    constexpr size_t smem = kDataBytes + sizeof(DenseSmem) + 1024;
    static_assert(smem <= 232448, "shared-memory plan exceeds the 227 KB a block may use");
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev != configured_dev) {
        cudaError_t e = cudaFuncSetAttribute(dense_gemm_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return e;
        configured_dev = dev;
    }

    // stripes of the weights one after the other, cut into panels of nearly equal height that fit the workspace
    long long stripes_all = 0;
    for (int i = 0; i < a.nw; ++i) stripes_all += (a.n[i] + kStripe - 1) / kStripe;
    const long long panels = (stripes_all + max_stripes - 1) / max_stripes;
    int w_i = 0;                 // weight and stripe of it that the next panel begins with
    long long w_s = 0, left = stripes_all;
    for (long long pn = 0; pn < panels; ++pn) {
        long long take = (left + (panels - pn) - 1) / (panels - pn);
        left -= take;
        PrepParams pp{};
        DenseParams dp{};
        long long stripes = 0;
        pp.nchunks = (nsb + kChunkRecs - 1) / kChunkRecs;
        pp.nsb = nsb;
        pp.dst = reinterpret_cast<__half *>(a.scratch);
        pp.ldd = a.Kpad;
        while (take > 0) {
            const long long have = (a.n[w_i] + kStripe - 1) / kStripe;
            const long long t = std::min(take, have - w_s);
            if (t > 0) {
                const long long r0 = w_s * kStripe, rows = std::min<long long>(a.n[w_i] - r0, t * kStripe);
                PrepSeg &ps = pp.seg[pp.nseg++];
                ps.w = a.w[w_i];
                ps.tile_begin = pp.tiles;
                ps.group0 = (int)(r0 / kRowGroup);
                ps.row0 = stripes * kStripe;
                pp.tiles += (int)((rows + kRowGroup - 1) / kRowGroup) * pp.nchunks;
                DenseSeg &ds = dp.seg[dp.nseg++];
                ds.y = reinterpret_cast<char *>(a.y[w_i]) + r0 * (a.y_is_bf16 ? 2 : 4);
                ds.ldy = a.ldy[w_i];
                ds.n = (int)rows;
                ds.stripe_begin = (int)stripes;
                stripes += t;
                take -= t;
                w_s += t;
            }
            if (w_s == have) ++w_i, w_s = 0;
        }
        if (pn == 0) {
            const int esz = a.x_is_bf16 ? 2 : 4;
            const bool vec = a.K % 8 == 0 && !(reinterpret_cast<uintptr_t>(a.x) & 15) && (a.ldx * esz) % 16 == 0 &&
                             (long long)a.M * (a.K / 8) < (1ll << 31);
            if (vec) {
                pp.x = a.x;
                pp.ldx = a.ldx;
                pp.xdst = reinterpret_cast<uint16_t *>(a.x16);
                pp.xldd = x_ldd;
                pp.M = a.M;
                pp.K8 = a.K / 8;
                pp.x_blocks = (int)std::min<long long>(((long long)a.M * pp.K8 + 2 * kPrepThreads - 1) / (2 * kPrepThreads), 148 * 16);
            } else {
                cudaError_t e = gemm_convert_x(a.x, a.x_is_bf16, a.ldx, a.x16, a.M, a.K, st);
                if (e != cudaSuccess) return e;
                ++*launches;
            }
        }
        cudaError_t e;
        switch (a.qt) {
        case QT_Q4_K: e = launch_prep<QT_Q4_K>(pp, a.x_is_bf16, st); break;
        case QT_Q5_K: e = launch_prep<QT_Q5_K>(pp, a.x_is_bf16, st); break;
        case QT_Q4_0: e = launch_prep<QT_Q4_0>(pp, a.x_is_bf16, st); break;
        case QT_MXFP4: e = launch_prep<QT_MXFP4>(pp, a.x_is_bf16, st); break;
        case QT_Q6_K: e = launch_prep<QT_Q6_K>(pp, a.x_is_bf16, st); break;
        case QT_Q8_0: e = launch_prep<QT_Q8_0>(pp, a.x_is_bf16, st); break;
        default: return cudaErrorInvalidValue;
        }
        if (e != cudaSuccess) return e;
        ++*launches;

        dp.y_is_bf16 = a.y_is_bf16;
        dp.M = a.M;
        dp.ksteps = nsb * (SB / kBK);
        pick_tiles(dp, (int)stripes, pairs, a.bn_override);
        dp.stage_bytes = kABytes + dp.bn / 2 * kBK * 2;      // a multiple of 2 KB: stages keep the swizzle's 1 KB alignment
        dp.stages = std::min(kMaxStages, kDataBytes / dp.stage_bytes);
        dp.status = a.status;
        CUtensorMap amap, bmap, bmap2;
        if (!encode_2d(&amap, a.scratch, a.Kpad, stripes * kStripe, a.Kpad, kRows) || !encode_2d(&bmap, a.x16, a.K, a.M, x_ldd, dp.bn / 2) ||
            !encode_2d(&bmap2, a.x16, a.K, a.M, x_ldd, dp.bn2 / 2))
            return cudaErrorInvalidValue;
        cudaLaunchConfig_t cfg{};
        cfg.gridDim = dim3((unsigned)(2 * std::min(dp.tiles, pairs)));
        cfg.blockDim = dim3(kThreads);
        cfg.dynamicSmemBytes = smem;
        cfg.stream = st;
        cudaLaunchAttribute attr[2];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = 2;
        attr[0].val.clusterDim.y = 1;
        attr[0].val.clusterDim.z = 1;
        attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[1].val.programmaticStreamSerializationAllowed = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 2;
        e = cudaLaunchKernelEx(&cfg, dense_gemm_kernel, dp, amap, bmap, bmap2);
        if (e != cudaSuccess) return e;
        ++*launches;
    }
    return cudaSuccess;
}

cudaError_t dense_set_wait_limit_ns(unsigned long long ns) { return cudaMemcpyToSymbol(s_wait_limit_ns, &ns, sizeof(ns)); }

}  // namespace b200q

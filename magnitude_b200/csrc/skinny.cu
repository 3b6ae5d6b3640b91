// Host side of the small-batch route (kernel: skinny_kernel.cuh) and its first launch, which turns the activations into
// operand fragments.
#include <algorithm>
#include <new>

#include "kernels.h"
#include "skinny_image.cuh"
#include "tc_common.cuh"

namespace b200q {

#define SK_TYPES(X) X(q4_k, QT_Q4_K) X(q5_k, QT_Q5_K) X(q6_k, QT_Q6_K) X(q8_0, QT_Q8_0) X(q4_0, QT_Q4_0) X(mxfp4, QT_MXFP4)
#define SK_DECLARE(NAME, QT)                                                                      \
    cudaError_t skinny_launch_##NAME(const SkParams &p, int NT, int P, int grid, cudaStream_t st); \
    cudaError_t skinny_wait_limit_##NAME(unsigned long long ns);
SK_TYPES(SK_DECLARE)

namespace {

// One warp per (product, record, token).
template <int MAP, int N> __global__ void __launch_bounds__(128) skinny_prep_kernel(const __grid_constant__ SkParamsOf<N> p) {
    pdl_launch_dependents();
    const int wid = blockIdx.x * 4 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (wid >= p.xwarps) return;
    const SkJob *jobs = p.jobs;
    int ji = p.njobs - 1;
    while (jobs[ji].xwarp0 > wid || jobs[ji].xwarp0 < 0) --ji;
    const SkJob &J = jobs[ji];
    const int rec = (wid - J.xwarp0) / J.M, tok = (wid - J.xwarp0) - rec * J.M;
    pdl_wait();                          // X may come from the launch before, which may also still read the images
    sk_make_image<MAP>(J, rec, tok, lane, J.img + (size_t)rec * sk_image_bytes(p.NT, p.P, kSumBytes<MAP>), p.NT, p.P);
}

// box0 words of every row of `rows` weight rows, over the chunks [c0, c0 + nc)
bool sk_encode(EncodeTiledFn enc, CUtensorMap *map, const uint8_t *w, int qt, int nsb, int64_t groups, int c0, int nc, int box0, int rows) {
    const int64_t rb = row_bytes_for(qt, nsb), cb = chunk_row_bytes(qt, c0, nsb);
    const cuuint64_t gdim[4] = {(cuuint64_t)(cb / 4), (cuuint64_t)kRowGroup, (cuuint64_t)nc, (cuuint64_t)groups};
    const cuuint64_t gstride[3] = {(cuuint64_t)cb, (cuuint64_t)(kRowGroup * cb), (cuuint64_t)(kRowGroup * rb)};
    const cuuint32_t box[4] = {(cuuint32_t)box0, (cuuint32_t)kRowGroup, 1, (cuuint32_t)(rows / kRowGroup)};
    const cuuint32_t estride[4] = {1, 1, 1, 1};
    void *base = const_cast<uint8_t *>(w) + kRowGroup * rec_off(qt, (int64_t)c0 * kChunkRecs);
    return enc(map, CU_TENSOR_MAP_DATA_TYPE_UINT32, 4, base, gdim, gstride, box, estride, CU_TENSOR_MAP_INTERLEAVE_NONE,
               CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

int token_tiles(int M) {
    return M <= 8 ? 1 : M <= 16 ? 2 : M <= 32 ? 4 : 6;
}

}  // namespace

int skinny_max_m() { return 16; }
int skinny_max_mid_m() { return 48; }

// Counts of the shared tiles, then their sums: one tile per block, as wide as M asks for (2.4 MB per eight tokens)
static constexpr size_t kSkCountBytes = size_t(kSkMaxGrid) * sk_warps(1) * sizeof(unsigned);
size_t skinny_ws_bytes(int M, int sm_count) {
    const int nt = token_tiles(M);
    return kSkCountBytes + (size_t)std::min(sm_count, kSkMaxGrid) * sk_tile_rows(nt) * 8 * nt * sizeof(double);
}
// Zeroes before it returns, on the legacy stream or on one of its own, which waits for no other.
cudaError_t skinny_ws_init(uint8_t *ws, size_t bytes, bool own_stream) {
    cudaStream_t st = nullptr;
    cudaError_t e = own_stream ? cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking) : cudaSuccess;
    if (e != cudaSuccess) return e;
    e = cudaMemsetAsync(ws, 0, bytes, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (own_stream) cudaStreamDestroy(st);
    return e;
}

static int planes(const SkinnyProduct &a) { return !a.x_is_bf16 && a.M <= skinny_max_m() ? 2 : 1; }
size_t skinny_image_bytes(const SkinnyProduct &a) { return (size_t)(a.Kpad / SB) * sk_image_bytes(token_tiles(a.M), planes(a), sk_sum_bytes(a.qt, token_tiles(a.M))); }

// A prepared call: the kernel parameters of `n` products of one block type and one M.  Built once (per call, or
// per plan) on the host; launching it touches no host memory the caller could have freed.
struct SkinnySet {
    SkParams p;
    int qt = 0, grid = 0;
};

static cudaError_t set_fill(SkinnySet *set, const SkinnyProduct *prods, int n, const SkinnyBuffers &buf) {
    if (n < 1 || n > kSkMaxJobs || !prods) return cudaErrorInvalidValue;
    const int M = prods[0].M, qt = prods[0].qt;
    const bool f32 = !prods[0].x_is_bf16;
    if (M < 1 || M > skinny_max_mid_m() || buf.ws_bytes < skinny_ws_bytes(M, buf.sm_count)) return cudaErrorInvalidValue;
    EncodeTiledFn enc = encode_fn();
    if (!enc) return cudaErrorNotSupported;
    set->qt = qt;
    SkParams &p = set->p;
    p.NT = token_tiles(M);
    p.P = planes(prods[0]);
    p.xwarps = 0;
    const int rows = sk_tile_rows(p.NT), rec4 = rec_bytes(qt) / 4;
    size_t img_off = 0;
    SkJob *jobs = p.jobs;
    int slots = 0;
    for (int i = 0; i < n; ++i) {
        const SkinnyProduct &a = prods[i];
        if (a.qt != qt || a.M != M || (!a.x_is_bf16) != f32 || a.N < 1 || a.K < 1) return cudaErrorInvalidValue;
        SkJob &J = jobs[i];
        J.x = a.x;
        J.ldx = a.ldx;
        J.x_is_bf16 = a.x_is_bf16;
        J.x_vec_ok = !(reinterpret_cast<uintptr_t>(a.x) & 15) && (a.ldx * (a.x_is_bf16 ? 2 : 4)) % 16 == 0;
        J.img = nullptr;
        J.xwarp0 = -1;
        for (int o = 0; o < i && !J.img; ++o)        // products of one activation share its image
            if (prods[o].x == a.x && prods[o].ldx == a.ldx && prods[o].K == a.K) J.img = jobs[o].img;
        if (!J.img) {
            if (img_off + skinny_image_bytes(a) > buf.img_bytes) return cudaErrorInvalidValue;
            J.img = buf.img + img_off;
            img_off += skinny_image_bytes(a);
            J.xwarp0 = p.xwarps;
            p.xwarps += M * (a.Kpad / SB);
        }
        J.y = a.y;
        J.ldy = a.ldy;
        J.y_is_bf16 = a.y_is_bf16;
        J.N = a.N;
        J.M = M;
        J.K = a.K;
        J.nsb = a.Kpad / SB;
        J.nfull = J.nsb / kChunkRecs;
        J.tiles = (a.N + rows - 1) / rows;
        J.slot0 = slots;
        if ((long long)slots + (long long)J.tiles * J.nsb > (1 << 30)) return cudaErrorInvalidValue;
        slots += J.tiles * J.nsb;
        const int64_t groups = padded_rows(a.N) / kRowGroup;
        const bool whole = J.nfull > 0, tail = J.nsb % kChunkRecs != 0;
        bool ok = true;
        if (whole) ok = sk_encode(enc, &J.w, a.w, qt, J.nsb, groups, 0, J.nfull, rec4, rows);
        if (ok && tail) ok = sk_encode(enc, &J.wtail, a.w, qt, J.nsb, groups, J.nfull, 1, rec4, rows);
        if (ok && qt == QT_Q6_K && whole) ok = sk_encode(enc, &J.d, a.w, qt, J.nsb, groups, 0, J.nfull, 4, rows);
        if (ok && qt == QT_Q6_K && tail) ok = sk_encode(enc, &J.dtail, a.w, qt, J.nsb, groups, J.nfull, 1, 4, rows);
        if (!ok) return cudaErrorInvalidValue;
    }
    p.count = reinterpret_cast<unsigned *>(buf.ws);
    p.sums = reinterpret_cast<double *>(buf.ws + kSkCountBytes);
    p.status = buf.status;
    p.njobs = n;
    p.slots = slots;
    int grid = std::min(std::min(buf.sm_count, kSkMaxGrid), slots);
    // A whole number of blocks per tile where that leaves no block with more slots: then no block has two tiles to share.  As
    // few of them as the longest run allows (us a call, 4096 x 14336 Q6_K, 8 rows: 9 blocks of 6 or 7 slots a tile 23.1, 8 of 7 22.5)
    int tiles = 0, nsb = jobs[0].nsb;
    for (int i = 0; i < n; ++i) {
        tiles += jobs[i].tiles;
        if (jobs[i].nsb != nsb) nsb = 0;
    }
    const int each = std::min(grid / tiles, nsb);
    if (each > 0 && (nsb + each - 1) / each <= (slots + grid - 1) / grid) {
        const int most = (nsb + each - 1) / each;
        grid = tiles * ((nsb + most - 1) / most);
    }
    set->grid = grid;
    // Few slots per block: each block makes the images of its own slots, in place, and the first launch falls away
    // (us a call, one launch / two: Q4_K 1024 x 4096, 8 rows 7.3 / 8.4, 16 rows 8.9 / 9.8).  With more slots, warps that
    // make images beside the products set the pace (6144 x 4096 in a plan, 4 rows: 5.0 us against 4.0).
    p.direct = (slots + grid - 1) / grid <= sk_depth(qt, p.NT, p.P) ? 1 : 0;
    return cudaSuccess;
}

cudaError_t skinny_set_create(const SkinnyProduct *prods, int n, const SkinnyBuffers &buf, SkinnySet **out) {
    if (!out) return cudaErrorInvalidValue;
    *out = nullptr;
    SkinnySet *set = new (std::nothrow) SkinnySet();
    if (!set) return cudaErrorMemoryAllocation;
    cudaError_t e = set_fill(set, prods, n, buf);
    if (e != cudaSuccess) {
        delete set;
        return e;
    }
    *out = set;
    return cudaSuccess;
}

void skinny_set_destroy(SkinnySet *set) { delete set; }

template <int MAP, int N> static cudaError_t launch_prep_t(const SkinnySet *set, cudaStream_t st) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)((set->p.xwarps + 3) / 4));
    cfg.blockDim = dim3(128);
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    void *args[] = {const_cast<SkParams *>(&set->p)};            // its first N jobs
    return cudaLaunchKernelExC(&cfg, reinterpret_cast<const void *>(&skinny_prep_kernel<MAP, N>), args);
}

template <int N> static cudaError_t launch_prep(const SkinnySet *set, cudaStream_t st) {
    switch (sk_map(set->qt, set->p.NT)) {
    case SK_K: return launch_prep_t<SK_K, N>(set, st);
    case SK_Q6: return launch_prep_t<SK_Q6, N>(set, st);
    case SK_SUB32: return launch_prep_t<SK_SUB32, N>(set, st);
    case SK_SUB16: return launch_prep_t<SK_SUB16, N>(set, st);
    default: return launch_prep_t<SK_BLOCK, N>(set, st);
    }
}

// The images (unless the blocks make their own), then the products; both with programmatic stream serialization.
cudaError_t skinny_set_launch(const SkinnySet *set, cudaStream_t st) {
    if (!set) return cudaErrorInvalidValue;
    cudaError_t e = set->p.direct ? cudaSuccess : set->p.njobs > kSkInline ? launch_prep<kSkMaxJobs>(set, st) : launch_prep<kSkInline>(set, st);
    if (e != cudaSuccess) return e;
    switch (set->qt) {
#define SK_LAUNCH(NAME, QT) \
    case QT: return skinny_launch_##NAME(set->p, set->p.NT, set->p.P, set->grid, st);
        SK_TYPES(SK_LAUNCH)
    default: return cudaErrorInvalidValue;
    }
}

int skinny_set_launches(const SkinnySet *set) { return set ? (set->p.direct ? 1 : 2) : 0; }

cudaError_t skinny_run(const SkinnyProduct *prods, int n, const SkinnyBuffers &buf, cudaStream_t st, int *launches) {
    if (n > kSkInline) return cudaErrorInvalidValue;     // larger sets go through a plan
    SkinnySet set;
    cudaError_t e = set_fill(&set, prods, n, buf);
    if (e != cudaSuccess) return e;
    e = skinny_set_launch(&set, st);
    if (launches) *launches += skinny_set_launches(&set);
    return e;
}

int skinny_max_products() { return kSkMaxJobs; }

cudaError_t skinny_set_wait_limit_ns(unsigned long long ns) {
    cudaError_t e;
#define SK_LIMIT(NAME, QT) \
    if ((e = skinny_wait_limit_##NAME(ns)) != cudaSuccess) return e;
    SK_TYPES(SK_LIMIT)
    return cudaSuccess;
}

}  // namespace b200q

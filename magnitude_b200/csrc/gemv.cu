// Decode GEMV (M = 1, 2; plans with fused epilogues up to M = 4): the HBM-bound streaming kernel.
//
// Y[m][n] = sum_k X[m][k] * dequant(W)[n][k]   for the streaming layout of common.cuh.
//
// One launch runs a list of projection jobs (one job for b200q_matmul, a whole decode step for a
// plan) on persistent CTAs, one per SM, no CPU fallback, no cluster multicast:
//   * sixteen consumer warps and four producer warps.  The producers keep a ring of slots in shared
//     memory filled with 1-D bulk copies (cp.async.bulk, completion counted on a "full" mbarrier per
//     slot).  A slot holds a quad: up to four tiles of the streaming layout, 16 rows x 8 superblock
//     records (18 KB of Q4_K).  The slots run on across job boundaries: the weights of the next job
//     stream in while the consumers still sum and store the current one or wait for other CTAs at a
//     dependency.  HBM reads never wait for a launch, a conversion or a grid-wide meeting, up to the
//     ring's size (about 150 KB, 3.5 us of one SM's share of the bandwidth).
//   * up to four teams of four consumer warps take the slots in turn; in a slot each warp owns two
//     records of all sixteen rows and multiplies each with eight integer mma.m16n8k32
//     (gemv_units.cuh).  What bounds the kernel is instructions: 240 per 2304 bytes of Q4_K with all
//     bookkeeping, 58 % of the schedulers' slots at 5.2 TB/s; dp4a, at half rate, took 250 slots for the
//     products alone.  A record per warp and two teams (331 instructions) reached 4.6 TB/s, the dp4a
//     kernel before 4.2 (ten independent 25600 x 5120 Q4_K products in a plan; 6.2 of Q8_0, 4.6 of Q6_K).
//   * per job each CTA owns a contiguous range of 4-row groups; a row's partial sums go to shared
//     memory cells by (chunk, record mod 4) and are added in fixed order: results do not depend on
//     the partition or the ring and are bit-reproducible.
//   * the activation is converted once per CTA and job into a 16-bit fixed-point image in shared
//     memory; plans of several independent jobs have a small launch convert all their activations and
//     the CTA fetches each image with one bulk copy, one job ahead where two images fit, else during
//     the final pass of the job before.
//   * a job may declare that it reads what earlier jobs of the same launch wrote; the CTAs then
//     meet at a counter in global memory before converting that job's activation.
//   * every wait (mbarrier, counter) is bounded; on expiry the waiter raises the status word and
//     the kernel drains and returns.
#include <stdlib.h>

#include <algorithm>
#include <atomic>
#include <vector>

#include "gemv_units.cuh"
#include "kernels.h"

namespace b200q {

namespace {

constexpr int kTeams = 4, kTeamWarps = 4;       // a warp has two records of a chunk: fewer barriers per record, two chains to overlap
constexpr int kWarps = kTeams * kTeamWarps;     // consumer warps
constexpr int kConsumers = kWarps * 32;
constexpr int kSlots = 16;                      // ring slots at most
constexpr int KC = kChunkRecs;
constexpr int R = kRowGroup;                    // rows per tile
constexpr int QG = 4;                           // row groups per quad: the 16 rows of an MMA
constexpr int kProducers = kTeams;              // producer warps
constexpr int kThreads = kConsumers + kProducers * 32;
// Five warps per scheduler leave 96 registers a thread; the producers give up most of theirs
constexpr int kLaunchRegs = 96, kConsumerRegs = 112, kProducerRegs = 32;
static_assert(kConsumers * kConsumerRegs + kProducers * 32 * kProducerRegs <= kThreads * kLaunchRegs, "register split");
// What the partial sums of a section (the quads between two final passes) may take; they are there twice, unless that leaves no
// room for a slot (one short row of 84992 Q4_K weights needs all 227 KB: the warps then meet after each final pass).  A pass takes
// about 2000 cycles with its meeting (25600 x 5120 Q4_K, eleven quads: 5570 GB/s in sections of five, 5890 in one), but the
// ring comes first: a launch takes the largest of these sizes that leaves six slots (5120 x 25600 Q6_K beside a 61 KB
// image: 4380 GB/s with five slots, 4660 with six).
constexpr int kSectionBytes[] = {10240, 6144, 3840, 1};
constexpr int quad_bytes(int mt, int nchunks) { return 16 * 16 * mt * nchunks; }
constexpr int kZeroBytes = 384;                 // what the B loads of foreign columns read

struct StreamParams {
    const StreamJob *jobs;   // device table, or nullptr when the single job is `inl`
    StreamJob inl;
    int njobs;
    int M;
    int jobs_bytes;          // shared-memory bytes of the job table
    int x_bytes;             // ... of one activation image area
    int x_bufs;              // 1 or 2 areas
    int partial_floats;      // from one copy of a section's partial sums to the other; 0: there is one
    int ring;                // the ring's place in shared memory
    int slots, slot_bytes;   // ring slots; bytes of one (the largest of the launch's jobs)
    int turn;                // producers and consumer teams at work
    int has_dep;             // some job waits for earlier jobs: CTAs count completions
    int *status;
    unsigned *counter;       // grid-wide completion counter (zero between launches)
    uint8_t *peer_base[kPeerMaxWorld];   // exchange buffers of the tensor-parallel ranks (peer memory)
    int peer_rank, peer_world;           // peer_world <= 1: jobs flagged SUM_RANKS store their own sums
};

// shared-memory header: barriers and failure bookkeeping (the zero area and the job table follow it)
struct SmemHead {
    uint64_t full[kSlots];
    uint64_t empty[kSlots];
    uint64_t xfull[2];           // per image area: the prepared image has landed
    float squares[kWarps];       // RMSNorm: the warps' sums of squares
    int fetched[2];              // images sent for, per area
    int fail;                    // raised by any warp that gave up a wait; everybody then drains and leaves
    int decide[2];               // first thread's sample of `fail`, taken before a barrier so all warps agree
    unsigned xepoch;             // exchanges posted so far (loaded from the exchange buffer)
    int xfail;                   // a wait for a peer's partial sums ran out
};
constexpr size_t kHeadBytes = (sizeof(SmemHead) + 127) & ~size_t(127);

// (value, exchange number) pairs of the in-launch rank sums: one 8-byte store / load each
__device__ __forceinline__ void st_pair(unsigned long long *p, float v, unsigned e) {
    const unsigned long long w = ((unsigned long long)e << 32) | __float_as_uint(v);
    asm volatile("st.volatile.global.u64 [%0], %1;" ::"l"(p), "l"(w) : "memory");
}
__device__ __forceinline__ unsigned long long ld_pair(const unsigned long long *p) {
    unsigned long long w;
    asm volatile("ld.volatile.global.u64 %0, [%1];" : "=l"(w) : "l"(p) : "memory");
    return w;
}

// (segment, row group inside it) of virtual group vg; segments are concatenated in launch order.
// A SWIGLU job interleaves its two segments instead (even groups gate, odd groups up), so that a
// CTA's contiguous range holds the gate rows and the up rows of the same outputs.
// (`glu`: the job's SWIGLU flag, read once per job by the caller: this runs once per work item.)
__device__ __forceinline__ void locate_group(const StreamJob &J, int vg, int &s, int &g, bool glu) {
    if (glu) {
        s = vg & 1;
        g = vg >> 1;
        return;
    }
    s = 0;
#pragma unroll
    for (int i = 1; i < kStreamMaxSeg; ++i)
        if (i < J.nseg && vg >= J.seg[i].group_begin) s = i;
    g = vg - J.seg[s].group_begin;
}

// virtual groups [gb, ge) of job J that CTA b works on: the shares of the job's CTAs differ by one group (one gate/up pair
// for SWIGLU), the others have none
template <bool FUSED = true>
__device__ __forceinline__ void cta_groups(const StreamJob &J, int b, int &gb, int &ge) {
    const int unit = FUSED && (J.flags & STREAM_JOB_SWIGLU) ? 2 : 1;
    b -= J.cta0;
    gb = unit * (b * J.share + min(b, J.share_rest));
    ge = gb + unit * (J.share + (b < J.share_rest ? 1 : 0));
    if ((unsigned)b >= (unsigned)J.ctas) gb = ge = 0;
}

// barrier of the consumer warps (hardware barrier 1; barrier 0 is __syncthreads)
__device__ __forceinline__ void consumers_sync() { asm volatile("bar.sync 1, %0;" ::"n"(kConsumers) : "memory"); }

// What a consumer warp needs to walk the slots of a section ...
struct Walk {
    int q0, q1, nchunks, nsb, wr, lane;
    int bytes_full, bytes_tail, tile_stride, slots, slot_bytes;
    int turn, turn_q, turn_c;      // from one of the team's slots to its next: slots, and as quads and chunks
    uint32_t full0, empty0, ring, img_bytes, partial;
    volatile int *fail;
};
// ... and where it is: the team's next slot (ring index and parity of its full barrier), quad and chunk in it
struct Place {
    int slot, parity, q, c;
};

// A consumer warp's part of a section: records wr and wr + 4 of the team's slots of quads q0..q1-1, the row sums into
// the partial sums.  False if a wait ran out.  HALF: no quad has more than two tiles, so no lane's second row exists.
template <int QT, int MT, bool HALF>
__device__ __forceinline__ bool section_dot(const Walk &t, Place &at, const XLane &xl) {
    // The lane's two rows of a quad: row g / 2 of tiles (g & 1) and (g & 1) + 2, g = lane / 4.  Neighbouring lane
    // groups read different tiles, whose places in the slot are offset so that their 16-byte loads meet no bank twice.
    const int c4 = t.lane & 3, row_tile = (t.lane >> 2) & 1, row_in_tile = t.lane >> 3;
    const uint32_t lane_full = t.ring + row_tile * t.tile_stride + t.wr * rec_bytes(QT) + row_in_tile * t.bytes_full;
    const uint32_t tail_less = row_in_tile * (t.bytes_full - t.bytes_tail);
    const uint32_t step = 2 * t.tile_stride;
    // where the lane leaves its row sums, [quad][m][row][chunk][wr]: lane group h stores row h's
    const int h = c4 & 1;
    const uint32_t row_cells = 16 * t.nchunks, quad_cells = MT * 16 * row_cells;
    const uint32_t cell0 = t.partial + ((row_tile + 2 * h) * R + row_in_tile) * row_cells + 4 * t.wr;
#pragma unroll 1
    while (at.q < t.q1) {
        const uint32_t bar = t.full0 + 8 * at.slot;
        // (Lanes may see the phase end at different moments: the warp votes on the probe before it branches, here and in the
        // producers, so that no lane goes on while another waits for it in a vote.)
        if (!__all_sync(0xFFFFFFFFu, mbar_try_wait(bar, at.parity))) {
            const bool ok = mbar_wait_bounded(bar, at.parity) && !*t.fail;
            if (!__all_sync(0xFFFFFFFFu, ok)) return false;
        }
        const int rec = at.c * KC + t.wr, q = at.q, c = at.c;
        float acc[2][MT];
#pragma unroll
        for (int m = 0; m < MT; ++m) acc[0][m] = acc[1][m] = 0.f;
        uint32_t a = lane_full + at.slot * t.slot_bytes;
        if (c == t.nchunks - 1) a -= tail_less;
        uint32_t d = 0;
        if (QT == QT_Q6_K) d = a + min(KC, t.nsb - c * KC) * 208 - t.wr * 206;     // fp16 d behind the octet
        auto give_back = [&]() {       // one of the team's warps has what it needs of the slot
            __syncwarp();
            if (t.lane == 0) mbar_arrive(t.empty0 + 8 * at.slot);
        };
        if (rec >= t.nsb) give_back();
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            if (rec + 4 * k < t.nsb) {
                WRec<QT> r0, r1;
                r0.load(a + 4 * k * rec_bytes(QT), d + 8 * k, c4);
                if (!HALF) r1.load(a + 4 * k * rec_bytes(QT) + step, d + 8 * k + step, c4);
                if (k == 1 || rec + 4 >= t.nsb) give_back();       // everything is in registers
#pragma unroll
                for (int m = 0; m < MT; ++m) {
                    RecSums<QT> sums;
                    XScales<QT> xs;
                    sums.template run<HALF>(r0, r1, xl, rec + 4 * k, m * t.img_bytes, c4);
                    xs.load(xl, rec + 4 * k, m * t.img_bytes, c4);
                    acc[0][m] += sums.finish(0, r0.s, xs, c4);
                    if (!HALF) acc[1][m] += sums.finish(1, r1.s, xs, c4);
                }
            }
        }
        // the teams take the slots in turn
        at.slot += t.turn;
        const bool wrap = at.slot >= t.slots;
        at.slot -= wrap ? t.slots : 0;
        at.parity ^= wrap;
        at.q += t.turn_q;
        at.c += t.turn_c;
        const bool over = at.c >= t.nchunks;
        at.c -= over ? t.nchunks : 0;
        at.q += over;
        // One cell per (row, chunk, record mod 4), for the final sum in a fixed order: results depend neither on the team
        // nor on the partition.  The four lane groups' shares are added up.
        const uint32_t cell = cell0 + (q - t.q0) * quad_cells + 16 * c;
#pragma unroll
        for (int m = 0; m < MT; ++m) {
            const float mine = h && !HALF ? acc[1][m] : acc[0][m], other = h || HALF ? acc[0][m] : acc[1][m];
            float v = mine + __shfl_xor_sync(0xFFFFFFFFu, other, 1);
            v += __shfl_xor_sync(0xFFFFFFFFu, v, 2);
            if (c4 < (HALF ? 1 : 2)) sts32f(cell + m * 16 * row_cells, v);
        }
    }
    return true;
}

// VAR: which optional code the instantiation carries.  Bit 0: the fused epilogues (SWIGLU, ACCUM, norm on
// the load) for launches that hold such jobs; bit 1: the rank-sum exchange, for launches of attached
// tensor-parallel ranks; bit 2: launches that give no CTA more than two row groups (8 rows) of a job, where half of each MMA's
// rows are not there: their unpacking and scaling is left out (see stream_launch_one).
template <int MT, int VAR>
__global__ void __launch_bounds__(kThreads, 1) stream_kernel(const __grid_constant__ StreamParams p) {
    constexpr bool FUSED = (VAR & 1) != 0, PEER = (VAR & 2) != 0, HALF = (VAR & 4) != 0;
    extern __shared__ __align__(128) uint8_t smem[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

    // shared-memory carve-up: header, zero area, job table, activation images, partial sums, ring
    SmemHead &head = *reinterpret_cast<SmemHead *>(smem);
    const uint32_t full0 = smem_u32(head.full), empty0 = smem_u32(head.empty);
    uint8_t *zero_area = smem + kHeadBytes;
    StreamJob *jobs_s = reinterpret_cast<StreamJob *>(zero_area + kZeroBytes);
    uint8_t *ximg0 = zero_area + kZeroBytes + p.jobs_bytes;
    float *partial0 = reinterpret_cast<float *>(ximg0 + p.x_bufs * p.x_bytes);      // two copies: [quad][m][row][chunk][wr]
    const int partial_floats = p.partial_floats;
    const uint32_t ring = smem_u32(smem) + p.ring;
    volatile int *fail_flag = &head.fail;

    if (threadIdx.x < kSlots) {
        mbar_init(full0 + 8 * threadIdx.x, QG);
        mbar_init(empty0 + 8 * threadIdx.x, kTeamWarps);
        if (threadIdx.x < 2) mbar_init(smem_u32(&head.xfull[threadIdx.x]), 1);
        mbar_fence_init();
        fence_proxy_async();
    }
    if (threadIdx.x == 0) head.fail = head.xfail = head.fetched[0] = head.fetched[1] = 0;
    if (threadIdx.x < kZeroBytes / 4) reinterpret_cast<int *>(zero_area)[threadIdx.x] = 0;
    // the job table (written by the host when the plan was made) moves to shared memory once
    if (p.jobs) {
        const int words = p.njobs * (int)(sizeof(StreamJob) / 4);
        const int *src = reinterpret_cast<const int *>(p.jobs);
        int *dst = reinterpret_cast<int *>(jobs_s);
        for (int i = threadIdx.x; i < words; i += blockDim.x) dst[i] = src[i];
    } else if (threadIdx.x < sizeof(StreamJob) / 4) {
        reinterpret_cast<int *>(jobs_s)[threadIdx.x] = reinterpret_cast<const int *>(&p.inl)[threadIdx.x];
    }
    // let the next kernel in the stream start early (it waits in pdl_wait before touching data)
    pdl_launch_dependents();
    __syncthreads();

    // Producer warps and consumer teams take the slots in turn, from the first job's first to the last job's last.  A
    // warp may only wait for a use of a ring slot when it has seen the use before (two uses ahead have the same parity),
    // so the ring has a multiple of `turn` slots, two for each of the `turn` producers and teams at work.
    const int turn = p.turn;

    // =========================================================================================
    // Producer warps: warp i of the `turn` at work copies slots i, i + turn, ... of all jobs, lane j of it tile j.  (A slot's
    // wait, address arithmetic and copies are a chain of 700 to 1300 cycles, as long as HBM takes for one slot, so up to four
    // warps share them.)
    // =========================================================================================
    if (warp >= kWarps) {
        setmaxnreg_dec<kProducerRegs>();
        const int me = warp - kWarps;
        if (lane >= QG || me >= turn) return;
        const unsigned mask = (1u << QG) - 1;
        int slot = me, uses = 0;       // the warp's next slot: ring index, earlier uses of it
        int c = me;                    // slots from the job's first to it
        int n = 0;                     // slots copied
        bool ok = true;
#pragma unroll 1
        for (int jb = 0; jb < p.njobs && ok; ++jb) {
            const StreamJob &J = jobs_s[jb];
            const bool glu = FUSED && (J.flags & STREAM_JOB_SWIGLU) != 0;
            int gb, ge;
            cta_groups<FUSED>(J, blockIdx.x, gb, ge);
            const int nchunks = J.nchunks;
            const uint32_t bytes_full = R * J.bytes_full, bytes_tail = R * J.bytes_tail;      // a whole tile, padding rows included
            const uint32_t dst0 = ring + lane * J.tile_stride;
            const long long group_stride = J.tile_group_stride;
            const int chunk_stride = J.tile_chunk_stride;
            int g = gb;
#pragma unroll 1
            while (true) {
                while (c >= nchunks && g < ge) {
                    c -= nchunks;
                    g += QG;
                }
                if (g >= ge) break;                    // (c slots into the next job)
                const uint32_t fbar = full0 + 8 * slot;
                if (uses > 0) {
                    const uint32_t ebar = empty0 + 8 * slot;
                    if (!__all_sync(mask, mbar_try_wait(ebar, (uses - 1) & 1))) {
                        uint64_t t0 = 0;
#pragma unroll 1
                        for (int spin = 1; !mbar_try_wait(ebar, (uses - 1) & 1); ++spin) {
                            if (*fail_flag) ok = false;
                            if ((spin & 63) == 0) {
                                if (t0 == 0) pdl_wait();       // (the consumers stand there until the launch before has ended)
                                const uint64_t now = globaltimer_ns();
                                if (t0 == 0) t0 = now;
                                else if (now - t0 > kWaitLimitNs) {
                                    atomicMax(p.status, DEV_ERR_PIPE_TIMEOUT);
                                    *fail_flag = 1;
                                    ok = false;
                                }
                            }
                            if (!ok) break;
                        }
                        ok = __all_sync(mask, ok);
                        if (!ok) break;
                    }
                }
                if (g + lane < ge) {                   // (the CTA's last quad may have fewer tiles)
                    int sg = 0, lg = g + lane;
                    if (FUSED || J.nseg > 1) locate_group(J, g + lane, sg, lg, glu);
                    const uint32_t bytes = c == nchunks - 1 ? bytes_tail : bytes_full;
                    fence_proxy_async();               // the consumers' reads of these bytes precede the engine's writes
                    mbar_expect_tx(fbar, bytes);
                    bulk_g2s(dst0 + slot * p.slot_bytes, J.seg[sg].w + lg * group_stride + (long long)c * chunk_stride, bytes, fbar);
                } else {
                    mbar_arrive(fbar);
                }
                ++n;
                c += turn;
                slot += turn;
                if (slot >= p.slots) {
                    slot -= p.slots;
                    ++uses;
                }
            }
        }
        // shared memory may only be released when the copies have landed
        for (int i = min(n, p.slots / turn); i > 0; --i) {
            slot -= turn;
            if (slot < 0) {
                slot += p.slots;
                --uses;
            }
            if (!mbar_wait_bounded(full0 + 8 * slot, uses & 1)) break;
        }
        return;
    }

    // =========================================================================================
    // consumer warps
    // =========================================================================================
    setmaxnreg_inc<kConsumerRegs>();
    const int tid = threadIdx.x;
    const int team = warp / kTeamWarps, wr = warp & (kTeamWarps - 1);      // wr: the warp's first record in a chunk
    int first_slot = 0;                // number of the job's first slot, modulo turn
    Place at;
    at.slot = team;
    at.parity = 0;
    int section_no = 0;
    uint32_t images = 0;               // images waited for: area 0 in the low half, area 1 in the high one

    // image of job jn (if it has one) into its area, by one thread
    auto fetch_image = [&](int jn, int area) {
        if (jn >= p.njobs || !jobs_s[jn].xq) return;
        const StreamJob &Jn = jobs_s[jn];
        const uint32_t bytes = (uint32_t)MT * Jn.nsb * ximg_rec_bytes(Jn.qt);
        const uint32_t bar = smem_u32(&head.xfull[area]);
        fence_proxy_async();           // reads of the area's last image precede the engine's writes
        *reinterpret_cast<volatile int *>(&head.fetched[area]) += 1;
        mbar_expect_tx(bar, bytes);
        bulk_g2s(smem_u32(ximg0 + area * p.x_bytes), Jn.xq, bytes, bar);
    };
    // the next job from jb on that has something for this CTA (jobs of few rows run on a part of the grid); launches whose
    // jobs wait, and rank sums, are walked through by every CTA
    auto next_job = [&](int jb) {
        for (; jb < p.njobs; ++jb) {
            int gb, ge;
            cta_groups<FUSED>(jobs_s[jb], blockIdx.x, gb, ge);
            if (ge > gb || p.has_dep || (PEER && (jobs_s[jb].flags & STREAM_JOB_SUM_RANKS))) break;
        }
        return jb;
    };
    int own = 0;                       // jobs of this CTA so far

    // n more jobs of this CTA are done, the last of them number jb (first thread; their stores come before).  The launch's
    // last arrival of all puts the counter back: nobody waits any more.
    auto publish = [&](unsigned n, int jb) {
        if (jb + 1 < p.njobs) {
            asm volatile("red.release.gpu.global.add.u32 [%0], %1;" ::"l"(p.counter), "r"(n) : "memory");
        } else {
            __threadfence();
            const unsigned total = gridDim.x * (unsigned)p.njobs;
            if (atomicAdd(p.counter, n) + n == total) *reinterpret_cast<volatile unsigned *>(p.counter) = 0;
        }
    };

    // ---- sums over tensor-parallel ranks, inside the launch -----------------------------------
    // A job flagged SUM_RANKS does not store its row sums: every CTA writes them, as (value,
    // exchange number) pairs, into its slot of every rank's exchange buffer (peer stores over
    // NVLink) and later adds up, in rank order, what the same CTA of every rank delivered, into y;
    // a pair that carries the current exchange number is complete, so there is no flag and no
    // fence.  "Later" is just before the CTA posts its next exchange (or at the end of the launch),
    // so the transfer hides behind the jobs in between; launches whose jobs wait for one another
    // complete it at once.  Two slot sets alternate; a CTA posts exchange e + 1 only after it has
    // read exchange e, and can only read e + 1 after the peers posted it, i.e. after they read e:
    // no pair is overwritten before it has been read.  All ranks run the same plan on the same grid.
    const bool xenabled = PEER && p.peer_world > 1;
    unsigned xe = 0;
    bool xe_loaded = false;
    int xpending = -1;
    auto exchange_complete = [&](int job, unsigned e) {
        const StreamJob &Jc = jobs_s[job];
        const unsigned long long *slots = reinterpret_cast<const unsigned long long *>(p.peer_base[p.peer_rank] + kPeerFusedSlotOff) +
                                          (size_t)(e & 1) * kPeerMaxWorld * kPeerSlotFloats;
        int gbc, gec;
        cta_groups<FUSED>(Jc, blockIdx.x, gbc, gec);
        const int n = Jc.seg[0].n;
        const bool accum = FUSED && (Jc.flags & STREAM_JOB_ACCUM) != 0;
        const int cells = (gec - gbc) * R * MT;
        // Eight lanes share one output: lane r of the group fetches rank r's pair (and waits for it, with the
        // usual limit), so all ranks' pairs travel at the same time; lane 0 then adds them in rank order.
        const bool dead = *reinterpret_cast<volatile int *>(&head.xfail) != 0;
        for (int base = 0; base < cells; base += kConsumers / kPeerMaxWorld) {
            const int t = base + (tid >> 3), r = lane & 7;
            const int rl = t / MT, m = t - rl * MT;
            const int row = gbc * R + rl;
            const bool valid = t < cells && row < n && m < p.M;
            const int si = m * n + row;
            unsigned long long w = 0;
            bool ok = !dead;
            if (valid && r < p.peer_world && ok) {
                const unsigned long long *q = slots + (size_t)r * kPeerSlotFloats + si;
                w = ld_pair(q);
                if ((unsigned)(w >> 32) != e) {
                    const uint64_t t0 = globaltimer_ns();
                    int spins = 0;
                    while ((unsigned)((w = ld_pair(q)) >> 32) != e) {
                        if ((++spins & 63) == 0 && globaltimer_ns() - t0 > kWaitLimitNs) {
                            ok = false;
                            head.xfail = 1;
                            atomicMax(p.status, DEV_ERR_PIPE_TIMEOUT);
                            break;
                        }
                    }
                }
            }
            const float v = __uint_as_float((unsigned)w);
            const int lane0 = lane & ~7;
            float acc = __shfl_sync(0xFFFFFFFFu, v, lane0);
#pragma unroll
            for (int rr = 1; rr < kPeerMaxWorld; ++rr) {
                const float o = __shfl_sync(0xFFFFFFFFu, v, lane0 + rr);
                if (rr < p.peer_world) acc += o;
            }
            const unsigned okmask = __ballot_sync(0xFFFFFFFFu, ok);
            if (valid && r == 0 && ((okmask >> lane0) & 0xFFu) == 0xFFu) {
                float *yp = reinterpret_cast<float *>(Jc.seg[0].y) + (long long)m * Jc.seg[0].ldy + row;
                *yp = accum ? *yp + acc : acc;
            }
        }
    };

    // what the conversions need of HBM may start its way now: RMSNorm weights are nobody's output
    if (FUSED)
        for (int jb = 0; jb < p.njobs; ++jb)
            if (jobs_s[jb].gamma && !jobs_s[jb].xq && tid * 32 < jobs_s[jb].K) asm volatile("prefetch.global.L2 [%0];" ::"l"(jobs_s[jb].gamma + tid * 32));
    pdl_wait();   // the previous kernel's writes (activations, images) are visible from here
    if (tid == 0) fetch_image(next_job(0), 0);
#pragma unroll 1
    for (int jb = next_job(0); jb < p.njobs; jb = next_job(jb + 1), ++own) {
        const StreamJob &J = jobs_s[jb];

        // ---- dependencies --------------------------------------------------------------------
        if (J.flags & STREAM_JOB_WAITS) {
            // every CTA has stored all earlier jobs' outputs once the counter reaches grid * jb
            if (tid == 0) {
                const unsigned target = gridDim.x * (unsigned)jb;
                const uint64_t t0 = globaltimer_ns();
                unsigned seen;
                int spins = 0;
                while (true) {
                    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(seen) : "l"(p.counter) : "memory");
                    if (seen >= target || *fail_flag) break;
                    if ((++spins & 255) == 0 && globaltimer_ns() - t0 > kWaitLimitNs) {
                        atomicMax(p.status, DEV_ERR_PIPE_TIMEOUT);
                        *fail_flag = 1;
                        break;
                    }
                }
            }
            consumers_sync();
        }

        // ---- this job's geometry -------------------------------------------------------------
        int gb, ge;
        cta_groups<FUSED>(J, blockIdx.x, gb, ge);
        const int nquads = (ge - gb + QG - 1) / QG;
        const int nchunks = J.nchunks, nsb = J.nsb, qt = J.qt;
        const bool glu = FUSED && (J.flags & STREAM_JOB_SWIGLU) != 0;
        const uint32_t img_bytes = (uint32_t)nsb * ximg_rec_bytes(qt);

        // ---- activation image ----------------------------------------------------------------
        // All warps have left the job before this one (its last barrier), so with two areas the other one is free: the next
        // job's image can travel while this job runs, sent for by the team whose turn is last.  With one area it is sent for
        // before this job's last final pass.
        const int area = p.x_bufs == 2 ? own & 1 : 0;
        uint8_t *ximg = ximg0 + area * p.x_bytes;
        if (p.x_bufs == 2) {
            if (tid == kTeamWarps * 32 * (first_slot == 0 ? turn - 1 : first_slot - 1)) fetch_image(next_job(jb + 1), area ^ 1);
        }
        if (J.xq) {
            // every thread waits for the image itself, no barrier
            if (!mbar_wait_bounded(smem_u32(&head.xfull[area]), (images >> (16 * area)) & 1u)) {
                atomicMax(p.status, DEV_ERR_PIPE_TIMEOUT);
                *fail_flag = 1;
            } else {
                images += 1u << (16 * area);
            }
            __syncwarp();
        } else {
            XSrc xs;
            xs.x = J.x; xs.ldx = J.ldx; xs.x_is_bf16 = J.x_is_bf16; xs.x_vec_ok = J.x_vec_ok;
            xs.K = J.K; xs.Kpad = J.Kpad;
            xs.gamma = FUSED ? J.gamma : nullptr;
            xs.rs = 1.f;
#pragma unroll 1
            for (int m = 0; m < MT; ++m) {
                if (FUSED && xs.gamma) {
                    // RMSNorm on the load: the CTA adds up the row's squares first
                    float ss = row_square_share(xs, m, tid, kConsumers);
#pragma unroll
                    for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xFFFFFFFFu, ss, o);
                    if (m > 0) consumers_sync();       // the row before has been read
                    if (lane == 0) head.squares[warp] = ss;
                    consumers_sync();
                    float tot = 0.f;
#pragma unroll
                    for (int w = 0; w < kWarps; ++w) tot += head.squares[w];
                    xs.rs = rsqrtf(tot / (float)xs.K + J.norm_eps);
                }
                prep_row<FUSED>(xs, qt == QT_Q6_K, m, tid, kConsumers, ximg + m * img_bytes);
            }
            consumers_sync();
        }
        const XLane xl = xlane(qt, smem_u32(ximg), smem_u32(zero_area), lane, wr & 1);

        const bool xsum = xenabled && (J.flags & STREAM_JOB_SUM_RANKS);
        const bool accum = FUSED && (J.flags & STREAM_JOB_ACCUM) != 0;
        auto store_out = [&](const StreamSeg &S, long long idx, float v) {
            if (J.y_is_bf16) {
                __nv_bfloat16 *yp = reinterpret_cast<__nv_bfloat16 *>(S.y) + idx;
                *yp = __float2bfloat16_rn(accum ? __bfloat162float(*yp) + v : v);
            } else {
                float *yp = reinterpret_cast<float *>(S.y) + idx;
                *yp = accum ? *yp + v : v;
            }
        };

        // ---- sections: a few quads, then their final pass ----------------------------------------
        // (quotients of small numbers: a division takes longer)
        int job_team;
        const int turn_q = (turn >= nchunks) + (turn >= 2 * nchunks) + (turn >= 3 * nchunks) + (turn >= 4 * nchunks);
        const int turn_c = turn - turn_q * nchunks;
        {
            int ahead = team - first_slot;
            if (ahead < 0) ahead += turn;
            at.q = (ahead >= nchunks) + (ahead >= 2 * nchunks) + (ahead >= 3 * nchunks);
            at.c = ahead - at.q * nchunks;
            if (team >= turn) at.q = nquads;
            job_team = first_slot;
            first_slot += nquads * nchunks;
            first_slot = turn == 3 ? first_slot % 3 : first_slot & (turn - 1);
        }
        int q0 = 0;
#pragma unroll 1
        do {

            const int q1 = min(nquads, q0 + J.section);
            // partial sums alternate between two copies: the section before is still being added up by
            // slower threads while this one's first quads are written
            float *partial = partial0 + (section_no & 1) * partial_floats;
            Walk t;
            t.q0 = q0; t.q1 = q1; t.nchunks = nchunks; t.nsb = nsb; t.wr = wr; t.lane = lane;
            t.bytes_full = (int)J.bytes_full; t.bytes_tail = (int)J.bytes_tail; t.tile_stride = J.tile_stride;
            t.slots = p.slots; t.slot_bytes = p.slot_bytes; t.turn = turn; t.turn_q = turn_q; t.turn_c = turn_c;
            t.full0 = full0; t.empty0 = empty0; t.ring = ring; t.img_bytes = img_bytes;
            t.partial = smem_u32(partial);
            t.fail = fail_flag;
            bool ok;
            if (qt == QT_Q4_K) ok = section_dot<QT_Q4_K, MT, HALF>(t, at, xl);
            else if (qt == QT_Q6_K) ok = section_dot<QT_Q6_K, MT, HALF>(t, at, xl);
            else if (qt == QT_Q8_0) ok = section_dot<QT_Q8_0, MT, HALF>(t, at, xl);
            else if (qt == QT_Q5_K) ok = section_dot<QT_Q5_K, MT, HALF>(t, at, xl);
            else if (qt == QT_Q4_0) ok = section_dot<QT_Q4_0, MT, HALF>(t, at, xl);
            else ok = section_dot<QT_MXFP4, MT, HALF>(t, at, xl);
            if (!ok && lane == 0) {
                atomicMax(p.status, DEV_ERR_PIPE_TIMEOUT);
                *fail_flag = 1;
            }
            if (tid == 0) head.decide[section_no & 1] = *fail_flag;
            consumers_sync();
            if (head.decide[section_no & 1]) {
                // Some wait ran out.  The producer waits for its own copies; this CTA's share of the completion count is
                // made up so that the counter returns to zero.
                if (tid == 0) {
                    for (int a = 0; a < p.x_bufs; ++a) {
                        const int seen = (images >> (16 * a)) & 0xFFFF;
                        if (*reinterpret_cast<volatile int *>(&head.fetched[a]) > seen) (void)mbar_wait_bounded(smem_u32(&head.xfull[a]), seen & 1);
                    }
                    if (p.has_dep) publish((unsigned)(p.njobs - jb), p.njobs - 1);
                }
                return;
            }
            ++section_no;
            // with one area: nobody reads this job's image any more, so the next one's travels during the final pass (plans of
            // Q8_0 6144 x 4096, whose 35 KB slots leave room for one: 6.1 us a product when it was sent for at the job's start, 5.3 now)
            if (p.x_bufs == 1 && q1 == nquads && tid == kConsumers - 32) fetch_image(next_job(jb + 1), 0);

            // ---- final pass: every row's partial sums in order, epilogue, store ------------------------
            if (xsum && q0 == 0) {
                if (!xe_loaded) {   // exchanges posted by earlier launches (after pdl_wait: their last write is visible)
                    if (tid == 0)
                        head.xepoch = *(reinterpret_cast<const unsigned *>(p.peer_base[p.peer_rank] + kPeerFusedEpochOff) + blockIdx.x);
                    consumers_sync();
                    xe = head.xepoch;
                    xe_loaded = true;
                }
                if (xpending >= 0) {
                    exchange_complete(xpending, xe);
                    xpending = -1;
                }
                ++xe;
            }
            // Row r of quad q: four neighbouring threads take every fourth chunk, all get the sum.  (Where there is work for a
            // few warps only, it falls to the team that had the job's first slot, as late as possible in turn again.)
            const int ftid = (tid - kTeamWarps * 32 * job_team) & (kConsumers - 1), fsub = ftid & 3, fidx = ftid >> 2;
            auto row_sum = [&](int q, int m, int r) {
                const uint32_t a = smem_u32(partial) + 16 * ((q * MT + m) * 16 + r) * nchunks;
                float v = 0.f;
#pragma unroll 1
                for (int c = fsub; c < nchunks; c += 4) {
                    const float4 w = lds128f(a + 16 * c);
                    v += (w.x + w.y) + (w.z + w.w);
                }
                v += __shfl_xor_sync(0xFFFFFFFFu, v, 1);
                v += __shfl_xor_sync(0xFFFFFFFFu, v, 2);
                return v;
            };
            const int gs = gb + q0 * QG, groups = min(ge - gs, (q1 - q0) * QG);      // the section's row groups
            if (glu) {
                // groups alternate gate, up: output row = silu(gate row) * up row, to the first segment's y
                const int outs = (groups >> 1) * R;
                for (int t0 = 0; t0 < outs * MT; t0 += kConsumers / 4) {
                    const int t = min(t0 + fidx, outs * MT - 1);       // (whole warps stay for the shuffles)
                    const int m = MT == 1 ? 0 : t / outs, o = t - m * outs;      // o = pair * 4 + row in group
                    const int pair = o / R, r = o & (R - 1);
                    const int row = ((gs >> 1) + pair) * R + r;
                    const float gv = row_sum(pair >> 1, m, (pair & 1) * 8 + r), uv = row_sum(pair >> 1, m, (pair & 1) * 8 + 4 + r);
                    if (fsub == 0 && t0 + fidx < outs * MT && row < J.seg[0].n)
                        store_out(J.seg[0], (long long)m * J.seg[0].ldy + row, gv / (1.f + __expf(-gv)) * uv);
                }
            } else {
                const int rows = groups * R;
                for (int t0 = 0; t0 < rows * MT; t0 += kConsumers / 4) {
                    const int t = min(t0 + fidx, rows * MT - 1);
                    const int m = MT == 1 ? 0 : t / rows, o = t - m * rows;      // o = group * 4 + row in group
                    const float v = row_sum(o >> 4, m, o & 15);
                    if (fsub != 0 || t0 + fidx >= rows * MT) continue;
                    int sg, lg;
                    locate_group(J, gs + o / R, sg, lg, false);
                    const int row = lg * R + (o & (R - 1));
                    if (row < J.seg[sg].n) {
                        if (xsum) {     // one segment, fp32 output (checked when the plan was made)
                            const size_t si = (size_t)((xe & 1) * kPeerMaxWorld + p.peer_rank) * kPeerSlotFloats + m * J.seg[0].n + row;
                            for (int r = 0; r < p.peer_world; ++r)
                                st_pair(reinterpret_cast<unsigned long long *>(p.peer_base[r] + kPeerFusedSlotOff) + si, v, xe);
                            continue;
                        }
                        store_out(J.seg[sg], (long long)m * J.seg[sg].ldy + row, v);
                    }
                }
            }
            if (partial_floats == 0) consumers_sync();
            q0 = q1;
        } while (q0 < nquads);
        if (xsum) {
            if (p.has_dep) exchange_complete(jb, xe);   // a later job may read y: finish now
            else xpending = jb;
        }
        if (p.has_dep) {
            // publish: this CTA's outputs of job jb are stored
            consumers_sync();
            if (tid == 0) publish(1, jb);
        }
    }
    if (xpending >= 0) exchange_complete(xpending, xe);
    if (xe_loaded && tid == 0)
        *(reinterpret_cast<unsigned *>(p.peer_base[p.peer_rank] + kPeerFusedEpochOff) + blockIdx.x) = xe;
}

}  // namespace

// ---------------------------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------------------------

int gemv_max_m() { return 4; }

namespace {

// Converts the activation of every job that has an image buffer (StreamJob::xq) to the fixed-point
// image the streaming kernel works on, once per job instead of once per CTA and job: block (job, part)
// handles every `parts`-th run of 8 elements.
__global__ void __launch_bounds__(256) xprep_kernel(const StreamJob *jobs, int M) {
    pdl_launch_dependents();       // the streaming launch may start (it waits before reading the images)
    const StreamJob &J = jobs[blockIdx.x];
    if (!J.xq) return;
    XSrc xs;
    xs.x = J.x; xs.ldx = J.ldx; xs.x_is_bf16 = J.x_is_bf16; xs.x_vec_ok = J.x_vec_ok;
    xs.K = J.K; xs.Kpad = J.Kpad;
    xs.gamma = J.gamma;
    xs.rs = 1.f;
    __shared__ float warp_ss[8];
    const int tid = blockIdx.y * blockDim.x + threadIdx.x, T = gridDim.y * blockDim.x;
    for (int m = 0; m < M; ++m) {
        if (xs.gamma) {
            // RMSNorm on the load: every block of the job adds up the whole row's squares itself
            float ss = row_square_share(xs, m, threadIdx.x, blockDim.x);
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xFFFFFFFFu, ss, o);
            __syncthreads();
            if ((threadIdx.x & 31) == 0) warp_ss[threadIdx.x >> 5] = ss;
            __syncthreads();
            float tot = 0.f;
            for (int w = 0; w < (int)(blockDim.x >> 5); ++w) tot += warp_ss[w];
            xs.rs = rsqrtf(tot / (float)xs.K + J.norm_eps);
        }
        prep_row<true>(xs, J.qt == QT_Q6_K, m, tid, T, const_cast<uint8_t *>(J.xq) + (size_t)m * J.nsb * ximg_rec_bytes(J.qt));
    }
}

}  // namespace

size_t stream_xq_bytes(const StreamJob &J, int M) { return ((size_t)M * J.nsb * ximg_rec_bytes(J.qt) + 255) & ~size_t(255); }

cudaError_t stream_xprep_launch(const StreamJob *jobs_dev, int njobs, int M, cudaStream_t st) {
    if (njobs < 1) return cudaSuccess;
    xprep_kernel<<<dim3((unsigned)njobs, 4), 256, 0, st>>>(jobs_dev, M);
    return cudaGetLastError();
}

namespace {

constexpr int kMaxJobsPerLaunch = 64;   // the job table lives in shared memory

// quads of the CTA with most of them
int job_quads(const StreamJob &J) {
    const int groups = ((J.flags & STREAM_JOB_SWIGLU) ? 2 : 1) * (J.share + (J.share_rest > 0));
    return std::max(1, (groups + QG - 1) / QG);
}
// (no shorter than eight slots, two for every team)
int section_quads(const StreamJob &J, int M, int bytes) {
    return std::min(job_quads(J), std::max((8 + J.nchunks - 1) / J.nchunks, bytes / quad_bytes(M, J.nchunks)));
}
size_t section_bytes(const StreamJob &J, int M, int quads) { return ((size_t)quads * quad_bytes(M, J.nchunks) + 127) & ~size_t(127); }

// shared memory of a launch: the largest activation image and ring slot over its jobs
struct Fit {
    size_t x_bytes = 0, slot = 0, jobs_bytes, partial, limit;
    int copies = 2;          // of the partial sums
    Fit(const StreamJob *jobs, int n, int M, size_t smem_limit, size_t partial_bytes) : partial(partial_bytes), limit(smem_limit) {
        for (int i = 0; i < n; ++i) {
            x_bytes = std::max(x_bytes, ((size_t)M * jobs[i].nsb * ximg_rec_bytes(jobs[i].qt) + 127) & ~size_t(127));
            slot = std::max(slot, (size_t)jobs[i].slot_bytes);
        }
        jobs_bytes = ((size_t)n * sizeof(StreamJob) + 127) & ~size_t(127);
        if (slots(1) < 1) copies = 1;
    }
    size_t fixed(int bufs) const { return kHeadBytes + kZeroBytes + jobs_bytes + bufs * x_bytes + copies * partial; }
    int slots(int bufs) const { return fixed(bufs) > limit ? 0 : (int)std::min<size_t>(kSlots, (limit - fixed(bufs)) / slot); }
};

template <int MT, int VAR>
cudaError_t launch_t(const StreamLaunch &a, StreamParams &p, int grid, cudaStream_t st) {
    // what the partial sums, images and tables leave of the shared memory is the ring
    size_t partial = 0;
    bool images = false;
    for (int i = 0; i < a.njobs; ++i) {
        partial = std::max(partial, section_bytes(a.jobs_host[i], MT, a.jobs_host[i].section));
        images = images || a.jobs_host[i].xq;
    }
    const Fit fit(a.jobs_host, a.njobs, MT, a.smem_limit, partial);
    p.x_bytes = (int)fit.x_bytes;
    p.jobs_bytes = (int)fit.jobs_bytes;
    p.partial_floats = fit.copies == 2 ? (int)(partial / 4) : 0;
    p.slot_bytes = (int)fit.slot;
    // Two slots for each team at work, so that one is filled while the other is read: four teams of eight slots and more,
    // three of six, two of less (27 KB slots of Q6_K: four slots 4.4 TB/s with two teams, 4.2 with four)
    auto turn_of = [](int slots) { return slots >= 8 ? 4 : slots >= 6 ? 3 : slots >= 2 ? 2 : 1; };
    auto usable = [&](int bufs) { return fit.slots(bufs) - fit.slots(bufs) % turn_of(fit.slots(bufs)); };
    // Two image areas let prepared images travel one job ahead; they pay while the ring keeps six slots or loses none.
    p.x_bufs = (images && a.njobs > 1 && usable(2) >= std::min(6, std::max(1, usable(1)))) ? 2 : 1;
    p.slots = usable(p.x_bufs);
    p.turn = turn_of(p.slots);
    if (p.slots < 1) return cudaErrorInvalidValue;
    p.ring = (int)fit.fixed(p.x_bufs);
    const size_t smem = p.ring + p.slots * fit.slot;

    auto kern = stream_kernel<MT, VAR>;
    static std::atomic<size_t> configured{0};   // per instantiation; a context on another device re-sets it
    static std::atomic<int> configured_dev{-1};  // (contexts on several threads may launch at once)
    int dev = 0;
    cudaGetDevice(&dev);
    if (smem > configured.load() || dev != configured_dev.load()) {
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return e;
        configured = smem;
        configured_dev = dev;
    }
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)grid);
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    // A launch whose jobs wait for one another holds its SMs until all its blocks run.  Started early it could share them with
    // such a launch of another stream, each holding what the other lacks, so it starts when the launch before has ended.
    cfg.numAttrs = (a.pdl && !p.has_dep) ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, kern, p);
}

template <int VAR>
cudaError_t launch_m(const StreamLaunch &a, StreamParams &p, int grid, cudaStream_t st) {
    switch (a.M) {
    case 1: return launch_t<1, VAR>(a, p, grid, st);
    case 2: return launch_t<2, VAR>(a, p, grid, st);
    case 3: return launch_t<3, VAR>(a, p, grid, st);
    default: return launch_t<4, VAR>(a, p, grid, st);
    }
}

cudaError_t stream_launch_one(const StreamLaunch &a, cudaStream_t st) {
    if (a.njobs < 1 || a.M < 1 || a.M > 4 || !a.jobs_host) return cudaErrorInvalidValue;
    StreamParams p{};
    p.jobs = a.jobs_dev;
    if (!a.jobs_dev) {
        if (a.njobs != 1) return cudaErrorInvalidValue;
        p.inl = a.jobs_host[0];
    }
    p.njobs = a.njobs;
    p.M = a.M;
    p.status = a.status;
    p.counter = a.counter;
    p.peer_rank = a.peer_rank;
    p.peer_world = a.peer_world;
    for (int r = 0; r < kPeerMaxWorld; ++r) p.peer_base[r] = a.peer_base[r];
    // Up to two row groups a CTA (1184 rows on 148 SMs): the form without second rows.  A kernel of its own: beside the other path in
    // one kernel it cost large launches registers (dependent layers 376 -> 386 us).  Calls of one row, us: full quads / halves (the
    // dp4a kernel, which worked by rows of one tile): Q4_K 512 x 14336 7.0 / 6.2 (6.6), Q5_K 512 x 28672 13.4 / 10.8 (10.6), Q6_K
    // 512 x 14336 8.5 / 7.3 (7.5), 1024 x 4096 4.7 / 4.2 (5.7); of two rows, Q6_K 512 x 14336 12.1 / 10.6 (11.7).  Only for plain
    // launches of the route's own sizes: fused and rank-sum ones are whole layers.
    bool fused = false, sums = false, half = true;
    for (int i = 0; i < a.njobs; ++i) {
        const StreamJob &J = a.jobs_host[i];
        switch (J.qt) {
        case QT_Q4_K: case QT_Q6_K: case QT_Q8_0: case QT_Q5_K: case QT_Q4_0: case QT_MXFP4: break;
        default: return cudaErrorInvalidValue;
        }
        if (J.flags & STREAM_JOB_WAITS) p.has_dep = 1;
        fused = fused || (J.flags & (STREAM_JOB_SWIGLU | STREAM_JOB_ACCUM)) != 0 || J.gamma != nullptr;
        sums = sums || (J.flags & STREAM_JOB_SUM_RANKS) != 0;
        half = half && J.share + (J.share_rest > 0) <= QG / 2;
    }
    const int grid = a.grid;
    if (p.has_dep && grid > a.sm_count) return cudaErrorInvalidValue;   // the counter wait needs every CTA resident
    if (p.peer_world > 1) {
        for (int i = 0; i < a.njobs; ++i) {
            const StreamJob &J = a.jobs_host[i];
            if (!(J.flags & STREAM_JOB_SUM_RANKS)) continue;
            // in-launch sums: per-CTA flags, one segment, fp32 outputs that fit one slot
            if (grid > kPeerCtas || J.nseg != 1 || J.y_is_bf16 || (long long)a.M * J.seg[0].n > kPeerSlotFloats)
                return cudaErrorInvalidValue;
        }
    }
    const bool peer = sums && p.peer_world > 1;
    if (peer) return fused ? launch_m<3>(a, p, grid, st) : launch_m<2>(a, p, grid, st);
    if (fused) return launch_m<1>(a, p, grid, st);
    if (half && a.M <= 2) return a.M == 1 ? launch_t<1, 4>(a, p, grid, st) : launch_t<2, 4>(a, p, grid, st);
    return launch_m<0>(a, p, grid, st);
}

}  // namespace

void stream_job_finish(StreamJob &J, int grid) {
    int groups = 0;
    for (int i = 0; i < J.nseg; ++i) {
        J.seg[i].group_begin = groups;
        groups += (J.seg[i].n + R - 1) / R;
    }
    J.total_groups = groups;
    J.nsb = J.Kpad / SB;
    J.nchunks = (J.nsb + KC - 1) / KC;
    J.bytes_full = (unsigned)chunk_row_bytes(J.qt, 0, J.nsb);
    J.bytes_tail = (unsigned)chunk_row_bytes(J.qt, J.nchunks - 1, J.nsb);
    J.tile_group_stride = tile_off(J.qt, 1, 0, 0, J.nsb);              // both offsets are linear in their index
    J.tile_chunk_stride = (int)tile_off(J.qt, 0, 1, 0, J.nsb);
    // Tiles of a slot: eight lanes read 64 bytes of a row of one tile and 64 of the next tile's (Q8_0: every other 16
    // bytes of 128, Q6_K: two pieces of 32).  Rows of a full chunk are a multiple of 128 bytes (Q6_K: 16 more), so the
    // padding behind a tile is what keeps the two apart in the banks.
    J.tile_stride = R * (int)J.bytes_full + (J.qt == QT_Q8_0 ? 16 : J.qt == QT_Q6_K ? 32 : 64);
    J.slot_bytes = QG * J.tile_stride;
    const int units = (J.flags & STREAM_JOB_SWIGLU) ? groups / 2 : groups;      // SWIGLU: gate and up groups in pairs
    J.cta0 = 0;
    J.ctas = grid;
    J.share = units / grid;
    J.share_rest = units % grid;
}

// A job of a plan costs every CTA that takes part in it about 2 us whatever its share: measured 2.3 us for 16 KB of a CTA
// (1024 x 4096 Q4_K), 2.9 for 64 KB (4096 x 4096), 5.1 for 170 KB.  So independent jobs with small shares are dealt to halves
// or quarters of the grid, each to the one with the least to do so far, if by this estimate the plan gets shorter
// (twenty 1024 x 4096 products 2.3 -> 1.2 us each).
static void deal_small_jobs(StreamJob *jobs, int n, int grid) {
    for (int i = 0; i < n; ++i)
        if (jobs[i].flags & (STREAM_JOB_WAITS | STREAM_JOB_SUM_RANKS)) return;
    if (n < 2 || grid < 8) return;
    constexpr double kBytesPerUs = 42500, kMostUs = 4;     // one SM's share of the HBM bandwidth; the largest share to make
    auto us = [&](const StreamJob &J, int parts) { return (double)J.total_groups * J.tile_group_stride * parts / (grid * kBytesPerUs); };
    auto cost = [](double stream_us) { return std::max(2.0 + 0.6 * stream_us, 1.25 * stream_us); };
    std::vector<int> part(n), parts(n), best_part(n), best_parts(n, 1);
    double best = 0;
    for (int i = 0; i < n; ++i) best += cost(us(jobs[i], 1));
    best *= 0.97;
    for (int most : {2, 4}) {
        double load[4] = {0, 0, 0, 0};
        for (int i = 0; i < n; ++i) {
            int np = (jobs[i].flags & STREAM_JOB_SWIGLU) ? 1 : most;
            while (np > 1 && us(jobs[i], np) > kMostUs) np >>= 1;
            int at = 0;
            double least = 1e30;
            for (int k = 0; k < np; ++k) {
                double l = 0;
                for (int r = k * 4 / np; r < (k + 1) * 4 / np; ++r) l = std::max(l, load[r]);
                if (l < least) {
                    least = l;
                    at = k;
                }
            }
            const double c = cost(us(jobs[i], np));
            for (int r = at * 4 / np; r < (at + 1) * 4 / np; ++r) load[r] = least + c;
            part[i] = at;
            parts[i] = np;
        }
        const double t = *std::max_element(load, load + 4);
        if (t < best) {
            best = t;
            best_part = part;
            best_parts = parts;
        }
    }
    for (int i = 0; i < n; ++i) {
        if (best_parts[i] == 1) continue;
        StreamJob &J = jobs[i];
        J.cta0 = grid * best_part[i] / best_parts[i];
        J.ctas = grid * (best_part[i] + 1) / best_parts[i] - J.cta0;
        J.share = J.total_groups / J.ctas;
        J.share_rest = J.total_groups % J.ctas;
    }
}

void stream_fit_jobs(StreamJob *jobs, int n, int M, int grid, size_t smem_limit) {
    for (int j0 = 0; j0 < n; j0 += kMaxJobsPerLaunch) deal_small_jobs(jobs + j0, std::min(kMaxJobsPerLaunch, n - j0), grid);
    for (int j0 = 0; j0 < n; j0 += kMaxJobsPerLaunch) {
        const int nj = std::min(kMaxJobsPerLaunch, n - j0);
        int best = 1, best_rank = 0;
        for (int b : kSectionBytes) {
            size_t partial = 0;
            for (int i = 0; i < nj; ++i) partial = std::max(partial, section_bytes(jobs[j0 + i], M, section_quads(jobs[j0 + i], M, b)));
            const Fit fit(jobs + j0, nj, M, smem_limit, partial);
            const int s = fit.copies == 2 ? fit.slots(1) : 0;
            const int rank = s >= 6 ? 6 : s >= 2 ? 2 : s;
            if (rank > best_rank) {
                best = b;
                best_rank = rank;
            }
        }
        for (int i = 0; i < nj; ++i) {       // even sections
            StreamJob &J = jobs[j0 + i];
            const int most = section_quads(J, M, best), all = job_quads(J), sections = (all + most - 1) / most;
            J.section = (all + sections - 1) / sections;
        }
    }
}

// Returns cudaSuccess, or cudaErrorInvalidValue when the shapes cannot be staged in shared memory.
cudaError_t stream_launch(const StreamLaunch &a, cudaStream_t st) {
    if (a.njobs <= kMaxJobsPerLaunch) return stream_launch_one(a, st);
    if (!a.jobs_dev || !a.jobs_host) return cudaErrorInvalidValue;
    for (int j0 = 0; j0 < a.njobs; j0 += kMaxJobsPerLaunch) {   // long plans: several launches in a row
        StreamLaunch part = a;
        part.jobs_host = a.jobs_host + j0;
        part.jobs_dev = a.jobs_dev + j0;
        part.njobs = std::min(kMaxJobsPerLaunch, a.njobs - j0);
        cudaError_t e = stream_launch_one(part, st);
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

cudaError_t gemv_set_wait_limit_ns(unsigned long long ns) { return cudaMemcpyToSymbol(s_wait_limit_ns, &ns, sizeof(ns)); }

}  // namespace b200q

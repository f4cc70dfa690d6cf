// Lag kernel with the whole lag history of an element block resident in shared memory: the
// same sums as lag_pipe_kernel (lag.cuh), bit for bit, for launches whose distinct frames fit.
//
// Work decomposition. A CTA owns a block of EB consecutive elements (16 or 32) of the flattened
// frame vector. All distinct frames of the launch (register frames and partners, "rows") of that
// block sit in shared memory at once, 128 bytes per row and 16 elements. The CTA's CW consumer
// warps split the tau entries among themselves: with EB = 16 every half-warp walks a list of its
// own (both halves take units of the same kind in step), with EB = 32 every warp. A thread loads
// the J frames of a sub-batch of its element into registers, then walks its list. A launch pairs
// up to kHistMaxSub sub-batches of J frames one after another against the same resident rows,
// which shift by J rows per sub-batch: 64 frames against 64 taus up to 500 read 563 rows instead
// of twice 497.
//
// Why this split. The ring kernel gives each thread one element and every tau, so a window of
// partners must travel through a small ring: per entry it pays barrier waits, ring wrap-around
// masks and releases, which cost it more issue slots than the pairs do. Here the rows have fixed
// addresses for the whole block: an entry is one table read, J shared loads at constant offsets,
// the arithmetic and the Kahan step. The host deals the entries to the lists, balanced by cost.
//
// Data movement. A producer warp copies the block's pieces of the ring's slabs (layout.cuh), up
// to 4 KB each, with cp.async.bulk, stage by stage (kHistFirstStages stages of a block's rows): a
// stage is refilled for the next block once every consumer warp has released it (empty[], when no
// unit left in its list reads the stage; the units run from the oldest rows to the newest), all
// its pieces at once, one per lane, their addresses held in registers. (One lane working through
// the pieces took 250 - 350 ns per copy, longer than the pairs of a block; lanes polling for their
// own pieces took the consumers' issue slots.) A unit waits only for the stages its rows belong
// to, so a block's pairing starts while its newest rows are on their way; its register frames come
// through a buffer of their own, a block ahead. Where two or more blocks fit in shared memory, whole
// blocks alternate between row buffers instead (one stage per sub-batch, the register frames read
// from the rows: fewer barriers per block). The accumulators of a block (one contiguous piece) are
// prefetched into L2 by the producer and read at the start of an entry, used at its end.
//
// What bounds it, measured (32 frames, 1024^2 with four scales, launch alone; ring kernel beside it):
// 64 taus up to 500 1.66 ms = 6.3 TB/s, 0.96 of the copy bandwidth (2.03 ms), with two batches per
// launch 1.40 ms per 32 frames, bound by issue and latency of the pairs (issue slots 48 %, shared-memory
// pipe 45 %); 64 taus up to 200 1.40 ms (1.56), 48 up to 100 0.89 ms (1.14), 20 up to 30 0.41 ms (0.45),
// bound by the pairs. Slower and not used, in an earlier form of the kernel: runs of eight taus and a loop
// per kind of unit (1.85 -> 2.30 ms beside the FFT, instruction fetch), the next unit's table entry loaded
// ahead (+1 to +5 %).
//
// Sub-batches whose lists differ (the first frames of a stream, where partners are missing) are
// separated by a barrier of the consumer warps, since another thread may then own an entry's
// accumulator. Every wait is bounded as in lag.cuh, with one outcome for the whole warp, and reports
// through *status.
#pragma once

#include "lag.cuh"
#include "layout.cuh"

namespace ddm {

constexpr int kHistMaxSub = 4;  // sub-batches per launch that tables and barriers have room for (engines use one or two)
constexpr int kHistJs[] = {4, 8, 16, 20, 24, 30, 32};
constexpr int kHistMaxJ = 32;
constexpr int kHistRowBytes = 128;  // 16 elements
constexpr int kHistSmemMax = 232448;  // dynamic shared memory of a CTA at most
constexpr int kHistFirstStages = 8;                              // stages of sub-batch 0's rows at most
constexpr int kHistStages = kHistFirstStages + kHistMaxSub - 1;  // and one for each further sub-batch
constexpr int kHistMaxBuffers = 4;                               // row buffers at most

// CTA shapes: consumer warps (plus one producer) and CTAs per SM.
__host__ __device__ constexpr int hist_threads(int CW) { return (CW + 1) * 32; }
__host__ __device__ constexpr int hist_ctas_per_sm(int CW) { return CW == 4 ? 3 : CW == 6 ? 2 : 1; }
// dynamic shared memory each of that many CTAs can have (228 KB per SM, 1 KB of it per CTA)
__host__ __device__ constexpr int hist_smem_limit(int CW) { return CW == 4 ? 76800 : CW == 6 ? 115712 : 232448; }
__host__ __device__ constexpr int hist_halves(int EB) { return 32 / EB; }  // lists per warp

// A unit of a list: the offsets in bytes of its first row (sub-batch 0) and of its accumulator row
// (of a 16-element block), and the mask of register frames whose pair exists (a run: the step in
// bytes between its accumulator rows). With EB = 16 a step holds one unit per half-warp, of the
// same kind. info: the kind, the active bit (a half without a unit repeats the other's without
// storing), the number of stages the step's rows need (bits 4..7), and the number of stages that
// neither this nor a later unit of the warp reads (from bit 8). A warp releases those only once it
// has waited for the stages the step needs, which hold them: a release must not run ahead of the copy.
struct HistStep {
    int row, acc, mask, info;
};
constexpr int kHistKindMask = 3, kHistMasked = 0, kHistFull = 1, kHistRun = 2, kHistActive = 4, kHistNeedShift = 4,
              kHistNeedMask = 15, kHistRelShift = 8;

// Table (ints): header, pieces (rows ascending, then the register frames'), warp -> step offsets,
// then the steps (16-byte aligned). A piece: ring slot in bits 0..19 and rows - 1 in 20..24; then its
// first row in bits 0..15 and its stage in 16.. (register frames: row of their buffer). A stage's
// bytes are those of one 16-element block.
constexpr int kHtNreg = 0, kHtNsub = 1, kHtNrows = 2, kHtNpiece = 3, kHtNx = 4, kHtRegRow = 5, kHtVariants = 6,
              kHtBuffers = 7, kHtSteps = 8, kHtInts = 9,
              kHtXBytes = 10, kHtArrive = 11,           // kHtArrive: arrivals a stage's barrier expects (1)
              kHtSubStages = 12;                        // + b: stages sub-batches 0..b need
constexpr int kHtBytes = kHtSubStages + kHistMaxSub;    // + stage: its bytes
constexpr int kHtHeader = kHtBytes + kHistStages;

// What a launch of an engine reads and writes: the ring in slabs, the accumulators in blocks.
struct HistTarget {
    const float2 *ring;
    float2 *acc;
    RingLayout lay;  // slabs
    int T;           // accumulator rows (of a 16-element block)
    int *status;
    long long wait_cycles;
};

// Shared memory: row buffers (EB / 16 regions), two register-frame buffers (none without pieces for
// them), barriers (full and empty: kHistStages per buffer; register frames full and empty: two each;
// sub-batch), abort word and last stage begun, table.
__host__ __device__ constexpr size_t hist_x_offset(int EB, int buffers, int nrows) {
    return static_cast<size_t>(EB / 16) * buffers * nrows * kHistRowBytes;
}
__host__ __device__ constexpr size_t hist_bar_offset(int EB, int buffers, int nrows, int nx) {
    return hist_x_offset(EB, buffers, nrows) + (nx ? static_cast<size_t>(EB / 16) * 2 * kHistMaxJ * kHistRowBytes : 0);
}
__host__ __device__ constexpr size_t hist_table_offset(int EB, int buffers, int nrows, int nx) {
    return (hist_bar_offset(EB, buffers, nrows, nx) + 8 * (2 * buffers * kHistStages + 5) + 8 + 15) / 16 * 16;
}

// |y - x|^2 added to a pair of sums: the difference as y + x * (-1), which rounds once as a
// subtraction does, and the squares, as packed FP32x2 instructions (the bits of f2_diff_sq_acc).
__device__ __forceinline__ float2 hist_diff_sq_acc(float2 y, float2 x, float2 acc) {
    const float2 d = __ffma2_rn(x, make_float2(-1.f, -1.f), y);
    return __ffma2_rn(d, d, acc);
}

// mbar_wait_bounded by a whole warp, with one outcome: lanes that gave up alone would leave the others
// in the warp's next vote or __syncwarp. Every lane observes the phase itself (it reads what landed).
__device__ __forceinline__ bool hist_warp_wait(uint64_t *bar, uint32_t parity, long long limit) {
    bool done = mbar_try_wait(bar, parity);
    if (__all_sync(0xffffffffu, done)) return true;
    const long long t0 = clock64();
    for (;;) {
        if (!done) done = mbar_try_wait(bar, parity);
        if (__all_sync(0xffffffffu, done)) return true;
        if (__any_sync(0xffffffffu, clock64() - t0 > limit)) return false;
    }
}

template <int J, int EB, int CW>
__device__ __forceinline__ void lag_hist_body(const HistTarget &tgt, const int *__restrict__ table, int block_begin,
                                              int block_end, int block_step) {
    constexpr int kThreads = hist_threads(CW);
    constexpr int kRegions = EB / 16;
    constexpr int kHalves = hist_halves(EB);
    extern __shared__ __align__(1024) unsigned char smem[];
    if (smem_addr(smem) & 1023u) {
        if (threadIdx.x == 0) atomicExch(tgt.status, kLagStatusMisaligned);
        return;
    }
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int nrows = table[kHtNrows], npiece = table[kHtNpiece], nx = table[kHtNx], buffers = table[kHtBuffers];
    const long long wait_cycles = tgt.wait_cycles;
    unsigned char *xbuf = smem + hist_x_offset(EB, buffers, nrows);
    uint64_t *full = reinterpret_cast<uint64_t *>(smem + hist_bar_offset(EB, buffers, nrows, nx));
    uint64_t *empty = full + buffers * kHistStages;
    uint64_t *xfull = empty + buffers * kHistStages, *xempty = xfull + 2;
    uint64_t *sub_done = xempty + 2;
    volatile int *abort_flag = reinterpret_cast<volatile int *>(sub_done + 1);
    volatile int *last_begun = abort_flag + 1;  // running stage number, written by the producer when it ends
    int *tab = reinterpret_cast<int *>(smem + hist_table_offset(EB, buffers, nrows, nx));
    const int ntab = table[kHtInts];
    for (int i = tid; i < ntab; i += kThreads) tab[i] = table[i];
    if (tid == 0) {
        for (int i = 0; i < buffers * kHistStages; i++) {
            mbar_init(&full[i], table[kHtArrive]);
            mbar_init(&empty[i], CW);
        }
        for (int i = 0; i < 2; i++) {
            mbar_init(&xfull[i], 1);
            mbar_init(&xempty[i], CW);
        }
        mbar_init(sub_done, CW);
        *abort_flag = 0;
        fence_mbar_init();
    }
    __syncthreads();
    const int nsub = tab[kHtNsub], nreg = tab[kHtNreg];
    const uint32_t buffer_bytes = static_cast<uint32_t>(nrows) * kHistRowBytes;
    const uint32_t region_bytes = buffer_bytes * buffers;
    constexpr uint32_t kXBytes = kHistMaxJ * kHistRowBytes;  // of one buffer and region
    const int *pieces = tab + kHtHeader;
    const int *lptr = pieces + 2 * (npiece + nx);
    const HistStep *steps = reinterpret_cast<const HistStep *>(tab + tab[kHtSteps]);
    const int nb16 = static_cast<int>(tgt.lay.E >> 4);  // 16-element blocks of a frame

    if (warp == CW) {
        // ---------------- producer: block after block, the next block's register frames and then the
        // block's stages, each as soon as it is released
        constexpr int kHeld = 2;  // row pieces per lane in registers; further ones are read from the table
        struct Copy {
            const float2 *src;  // of element block 0
            uint32_t dst, bytes;
            int stride, stage;
        };
        auto copy_of = [&](int p) {
            const int slot = pieces[2 * p] & 0xFFFFF, row = pieces[2 * p + 1] & 0xFFFF;
            return Copy{tgt.ring + tgt.lay.base(slot), static_cast<uint32_t>(row) * kHistRowBytes,
                        (((pieces[2 * p] >> 20) & 31) + 1u) * kHistRowBytes, tgt.lay.stride(slot), pieces[2 * p + 1] >> 16};
        };
        auto issue = [&](const Copy &c, unsigned char *dst, uint32_t region, int b16, int regions, uint64_t *bar) {
            const float2 *src = c.src + static_cast<long long>(b16) * c.stride;
            for (int i = 0; i < regions; i++) bulk_load(dst + c.dst + i * region, src + i * c.stride, c.bytes, bar);
        };
        Copy held[kHeld], xheld;
#pragma unroll
        for (int h = 0; h < kHeld; h++) {
            held[h].stage = -1;
            if (lane + 32 * h < npiece) held[h] = copy_of(lane + 32 * h);
        }
        if (lane < nx) xheld = copy_of(npiece + lane);  // at most 32 register frames, so at most 32 pieces
        const int nstages = tab[kHtSubStages + nsub - 1];
        const int nblocks = block_begin < block_end ? (block_end - 1 - block_begin) / block_step + 1 : 0;
        bool ok = true;
        auto issue_x = [&](int n) {
            if (nx == 0 || n >= nblocks) return;
            if (n > 1 && !hist_warp_wait(&xempty[n & 1], ((n >> 1) - 1) & 1, wait_cycles)) ok = false;
            if (!ok) return;
            const int b16 = (block_begin + n * block_step) * kRegions;
            const int regions = nb16 - b16 < kRegions ? nb16 - b16 : kRegions;
            if (lane == 0) mbar_expect_tx(&xfull[n & 1], tab[kHtXBytes] * regions);
            __syncwarp();
            if (lane < nx) issue(xheld, xbuf + (n & 1) * kRegions * kXBytes, kXBytes, b16, regions, &xfull[n & 1]);
        };
        int begun = -1, buf = 0, use = 0;  // of block n: its row buffer, and how often that has been filled before
        issue_x(0);
        for (int n = 0; ok && n < nblocks && !__any_sync(0xffffffffu, *abort_flag); n++) {
            const int b16 = (block_begin + n * block_step) * kRegions;
            const int regions = nb16 - b16 < kRegions ? nb16 - b16 : kRegions;
            if (lane < regions)  // the block's accumulators into L2, ahead of their use
                asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(
                                 tgt.acc + static_cast<long long>(b16 + lane) * tgt.T * 16),
                             "r"(static_cast<uint32_t>(tgt.T) * kHistRowBytes)
                             : "memory");
            issue_x(n + 1);
            unsigned char *dst = smem + buf * buffer_bytes;
            for (int st = 0; st < nstages && ok; st++) {
                if (use > 0 && !hist_warp_wait(&empty[buf * kHistStages + st], (use - 1) & 1, wait_cycles)) ok = false;
                if (!ok) break;
                uint64_t *bar = &full[buf * kHistStages + st];
                if (lane == 0) mbar_expect_tx(bar, tab[kHtBytes + st] * regions);
                __syncwarp();
#pragma unroll
                for (int h = 0; h < kHeld; h++)
                    if (held[h].stage == st) issue(held[h], dst, region_bytes, b16, regions, bar);
                for (int p = 32 * kHeld + lane; p < npiece; p += 32) {
                    const Copy more = copy_of(p);
                    if (more.stage == st) issue(more, dst, region_bytes, b16, regions, bar);
                }
                begun = n * kHistStages + st;
            }
            if (++buf == buffers) buf = 0, use++;
        }
        if (!ok) *abort_flag = 1;
        if (lane == 0) *last_begun = begun;
    } else {
        // ---------------- consumers
        const int region = kRegions == 2 ? lane >> 4 : 0;
        const int half = kHalves == 2 ? lane >> 4 : 0;
        const int m = lane & 15;  // element within the 16-element block
        const int variants = tab[kHtVariants];
        unsigned char *acc_base = reinterpret_cast<unsigned char *>(tgt.acc + m);
        // A lane whose wait runs out goes on with its warp to the end of the block: one that left alone would
        // be missing from the warp's next vote or __syncwarp. Lane 0 makes no arrivals after such a wait (a
        // release must not run ahead of its copy), so the producer's waits run out too, and at most a block's
        // waits (one per stage, two of the register frames and the sub-batches) pass their limits.
        bool late = false, arrives = lane == 0;
        auto wait_for = [&](uint64_t *bar, uint32_t phase) {
            if (!mbar_wait_bounded(bar, phase, wait_cycles)) late = true, arrives = false;
        };
        int buf = 0;
        uint32_t parity = 0;  // of the row buffer's barriers
        for (int n = 0, block = block_begin; block < block_end; block += block_step, n++) {
            const int b16 = block * kRegions + region;
            const bool valid = b16 < nb16;
            unsigned char *acc_k = acc_base + static_cast<long long>(b16) * tgt.T * kHistRowBytes;
            const unsigned char *rows = smem + region * region_bytes + buf * buffer_bytes + m * 8;
            uint64_t *stage = &full[buf * kHistStages];
            int have = 0, released = 0;
            auto wait_stages = [&](int need) {
                for (; have < need; have++) wait_for(&stage[have], parity);
            };
            auto release = [&](int rel) {
                if (rel > released) {
                    __syncwarp();
                    if (arrives)
                        for (int st = released; st < rel; st++) mbar_arrive(&empty[buf * kHistStages + st]);
                    released = rel;
                }
            };
            if (nx > 0) wait_for(&xfull[n & 1], (n >> 1) & 1);
            for (int b = 0; b < nsub; b++) {
                if (b > 0 || nx == 0) wait_stages(tab[kHtSubStages + b]);
                const unsigned char *sub_rows = rows + b * nreg * kHistRowBytes;
                float2 x[J];  // the sub-batch's register frames
                {
                    const unsigned char *xr = b == 0 && nx > 0 ? xbuf + ((n & 1) * kRegions + region) * kXBytes + m * 8
                                                     : sub_rows + tab[kHtRegRow] * kHistRowBytes;
                    if (nreg == J) {
#pragma unroll
                        for (int j = 0; j < J; j++) x[j] = *reinterpret_cast<const float2 *>(xr + j * kHistRowBytes);
                    } else {
#pragma unroll
                        for (int j = 0; j < J; j++)
                            x[j] = j < nreg ? *reinterpret_cast<const float2 *>(xr + j * kHistRowBytes) : make_float2(0.f, 0.f);
                    }
                    if (b == 0 && nx > 0) {
                        __syncwarp();
                        if (arrives) mbar_arrive(&xempty[n & 1]);
                    }
                }
                const int *lp = lptr + (variants > 1 ? b * CW : 0) + warp;
                const int s1 = lp[1];
                const bool last = b == nsub - 1;
                for (int s = lp[0]; s < s1; s++) {
                    const int4 st = *reinterpret_cast<const int4 *>(steps + s * kHalves + half);
                    wait_stages((st.w >> kHistNeedShift) & kHistNeedMask);
                    if (last) release(st.w >> kHistRelShift);
                    const unsigned char *w = sub_rows + st.x;
                    unsigned char *ap = acc_k + st.y;
                    const bool mine = valid && (st.w & kHistActive);
                    const int kind = st.w & kHistKindMask;
                    if (kind == kHistRun) {
                        // kLagFuse entries whose windows start one row apart (their accumulators at st.y,
                        // st.y + st.z, ...): position q of their span pairs with register frame q - r of
                        // entry r
                        float2 a[kLagFuse], c[kLagFuse];
#pragma unroll
                        for (int r = 0; r < kLagFuse; r++) {
                            a[r] = c[r] = make_float2(0.f, 0.f);
                            if (mine) a[r] = __ldcg(reinterpret_cast<const float2 *>(ap + r * st.z));
                        }
#pragma unroll
                        for (int q = 0; q < J + kLagFuse - 1; q++) {
                            const float2 y = *reinterpret_cast<const float2 *>(w + q * kHistRowBytes);
#pragma unroll
                            for (int r = 0; r < kLagFuse; r++)
                                if (q - r >= 0 && q - r < J) c[r] = hist_diff_sq_acc(y, x[q - r], c[r]);
                        }
#pragma unroll
                        for (int r = 0; r < kLagFuse; r++) {
                            const float y = (c[r].x + c[r].y) - a[r].y;
                            const float t = a[r].x + y;
                            if (mine) __stcg(reinterpret_cast<float2 *>(ap + r * st.z), make_float2(t, (t - a[r].x) - y));
                        }
                    } else {
                        float2 a = make_float2(0.f, 0.f);
                        if (mine) a = __ldcg(reinterpret_cast<const float2 *>(ap));
                        float2 c[4];
#pragma unroll
                        for (int i = 0; i < 4; i++) c[i] = make_float2(0.f, 0.f);
                        if (kind == kHistFull) {
#pragma unroll
                            for (int j = 0; j < J; j++)
                                c[j & 3] = hist_diff_sq_acc(*reinterpret_cast<const float2 *>(w + j * kHistRowBytes), x[j], c[j & 3]);
                        } else {
                            // by eights: a whole one (in both halves) needs no test per pair
#pragma unroll
                            for (int j0 = 0; j0 < J; j0 += 8) {
                                constexpr unsigned kEight = 255;
                                const unsigned all = j0 + 8 <= J ? kEight : kEight >> (j0 + 8 - J);
                                const unsigned part = (static_cast<unsigned>(st.z) >> j0) & all;
                                if (__all_sync(0xffffffffu, part == all)) {
#pragma unroll
                                    for (int j = j0; j < j0 + 8 && j < J; j++)
                                        c[j & 3] = hist_diff_sq_acc(*reinterpret_cast<const float2 *>(w + j * kHistRowBytes), x[j], c[j & 3]);
                                } else if (part) {
#pragma unroll
                                    for (int j = j0; j < j0 + 8 && j < J; j++)
                                        if (part & (1u << (j - j0)))
                                            c[j & 3] = hist_diff_sq_acc(*reinterpret_cast<const float2 *>(w + j * kHistRowBytes), x[j], c[j & 3]);
                                }
                            }
                        }
                        const float sum = ((c[0].x + c[0].y) + (c[1].x + c[1].y)) + ((c[2].x + c[2].y) + (c[3].x + c[3].y));
                        const float y = sum - a.y;
                        const float t = a.x + y;
                        if (mine) __stcg(reinterpret_cast<float2 *>(ap), make_float2(t, (t - a.x) - y));
                    }
                }
                if (variants > 1 && !last) {
                    __syncwarp();
                    if (arrives) mbar_arrive(sub_done);
                    wait_for(sub_done, (n * (nsub - 1) + b) & 1);
                }
            }
            wait_stages(tab[kHtSubStages + nsub - 1]);
            if (__any_sync(0xffffffffu, late)) {
                *abort_flag = 1;
                break;
            }
            release(tab[kHtSubStages + nsub - 1]);
            if (++buf == buffers) buf = 0, parity ^= 1;
        }
    }
    __syncthreads();
    if (*abort_flag) {
        // drain: wait (bounded) for the copies in flight: the stages begun of the last blocks, and the
        // register frames of the block after
        if (tid == 0) atomicExch(tgt.status, kLagStatusWait);
        const int begun = *last_begun, last = begun < 0 ? -1 : begun / kHistStages;
        for (int n = last >= buffers ? last - buffers + 1 : 0; n <= last; n++)
            if (tid < tab[kHtSubStages + nsub - 1] && n * kHistStages + tid <= begun)
                mbar_wait_bounded(&full[n % buffers * kHistStages + tid], (n / buffers) & 1);
        if (tid < 2 && nx > 0) {  // the phase that is armed, if any, is the one not yet complete
            mbar_wait_bounded(&xfull[tid], 0);
            mbar_wait_bounded(&xfull[tid], 1);
        }
        __syncthreads();
    }
}

// A table small enough travels with the launch (2 KB of kernel parameters): no upload, and none of
// the event records and waits that order one (four to five calls, 6 - 8 us of a small launch).
constexpr int kHistInlineInts = 480;
struct HistInline {
    int v[kHistInlineInts];
};

// One engine's launch: CTA b handles element blocks b, b + gridDim.x, ... below nblocks. The table
// is in device memory, or, with table null, the first ints of inl.
template <int J, int EB, int CW>
__global__ void __launch_bounds__(hist_threads(CW), hist_ctas_per_sm(CW))
    lag_hist_kernel(const __grid_constant__ HistTarget tgt, const int *__restrict__ table, int nblocks,
                    const __grid_constant__ HistInline inl) {
    lag_hist_body<J, EB, CW>(tgt, table ? table : inl.v, static_cast<int>(blockIdx.x), nblocks, static_cast<int>(gridDim.x));
}

// The lag work of several engines (served streams) in one launch: item i owns CTAs [cta_begin,
// cta_begin + ctas), each of which walks every ctas-th of the item's element blocks.
struct HistBatchItem {
    HistTarget target;
    const int *table;
    int cta_begin, ctas, blocks;
};

template <int J, int EB, int CW>
__global__ void __launch_bounds__(hist_threads(CW), hist_ctas_per_sm(CW))
    lag_hist_batch_kernel(const HistBatchItem *__restrict__ items, int n) {
    int lo = 0, hi = n - 1;  // the last item whose first CTA is at or before this one
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (items[mid].cta_begin <= static_cast<int>(blockIdx.x)) lo = mid;
        else hi = mid - 1;
    }
    const HistBatchItem &it = items[lo];
    lag_hist_body<J, EB, CW>(it.target, it.table, static_cast<int>(blockIdx.x) - it.cta_begin, it.blocks, it.ctas);
}

// The instances both kernels are compiled for: X(J, EB, CW), and a key of each.
#define HIST_INSTANCES_J(X, JJ) X(JJ, 32, 4) X(JJ, 16, 4) X(JJ, 16, 6) X(JJ, 16, 12)
#define HIST_INSTANCES(X)                                                                                     \
    HIST_INSTANCES_J(X, 4) HIST_INSTANCES_J(X, 8) HIST_INSTANCES_J(X, 16) HIST_INSTANCES_J(X, 20)            \
    HIST_INSTANCES_J(X, 24) HIST_INSTANCES_J(X, 30) HIST_INSTANCES_J(X, 32)
constexpr int hist_key(int J, int EB, int CW) { return (J * 128 + EB) * 16 + CW; }

}  // namespace ddm

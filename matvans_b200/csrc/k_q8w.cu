// Decode + int8 product over a list of Q8-stripe matrices ("jobs": one matrix
// with its x and y each) in one launch, for sm_100a: a persistent,
// warp-specialised kernel, one CTA per SM.
//
//   unit   one segment of one stripe (32 rows x seg_quads quads): what a decode
//          warp takes at a time
//   item   one stripe, or one of `parts` ranges of its segments: the units
//          that share a decode table and are summed together
//
// Roles within a CTA (warps run on their own; nothing is synchronised CTA-wide
// between the start and the end of a launch):
//   * producer (1 warp): takes items (work queue, or every G-th one), publishes
//     their records in a ring, and keeps a ring of stream slots filled with the
//     units' blocks, in unit order, by 1-D bulk copies (cp.async.bulk, no
//     multicast) that complete on the slot's mbarrier;
//   * stager (1 warp): copies an item's symbol tables to shared memory, one item
//     ahead of its decode;
//   * table warps (4): expand them into one of two decode tables while the decode
//     warps work from the other, and write an item's outputs once its units are
//     decoded (with MMA consumers from tensor memory, one warp per lane quarter);
//   * decode warps (W): each takes the CTA's next unit, waits for its slot and
//     its item's table, decodes, and counts the unit as done.
// One CTA-wide barrier per item, a table build and a cross-warp sum between the
// items of the form this replaced left the SM idle for a third of a launch: the
// seven matrices of a 7B layer took 139 us there with one vector and take 74 us,
// with 16 vectors 136 and 107 us; 64 vectors of 11008x4096, 198 and 46 us.
//
// Decode table: entry (q, lane) = f | sym << 16 | r << 24 (frequency of the
// symbol that owns quantile q, the symbol, r = q - cum), 4 bytes at byte
// q*256 + lane*4 of a 64 KB region; the second table sits in the other half of
// each 256-byte row.  One byte permute of the state forms a lookup address:
// the quantile byte lands in bits 8..15, the lane's byte and the table's half
// in bits 0..7.  A warp's lookup is one conflict-free wavefront.  (8-byte
// entries save two permutes a step but take two wavefronts a lookup, and the
// second table would not fit.)
//
// Decode step (per lane, per quad of 4 symbols):
//   refill:   if (hi == 0) { hi = lo; lo = next word; load the word after it },
//             predicated; the stream position moves one 128-byte word-row on and
//             is clamped every 4 steps to the row after the block
//   update:   r0 + f0 r1 = dp4a of e0 with (r1, 0, 0, 1), one byte permute of e1;
//             f0 f1 by dp2a of the entries; (hi:lo) = hi*P + t0, one 32x32->64
//             multiply-add
//
// What bounds it: issue and the ALU pipe.  A step takes 29 instructions (9 byte
// permutes at half rate; 35 with all that a launch does around it) and 5
// shared-memory wavefronts; a loop of steps alone
// runs at 9.2 SM cycles a step with 16 warps (a single warp's step takes 80), and
// the kernel at 11 on a 7B layer (one vector).
#include <algorithm>

#include <cuda_bf16.h>

#include "mv_device.cuh"
#include "q8w.cuh"
#include "umma.cuh"

namespace mv {

constexpr int kRing = 8;       // items in flight (records, partial sums, counters)
constexpr int kTableWarps = 4; // warps 0..3: one per TMEM lane quarter
constexpr int kProducer = 4;   // the producer warp
constexpr int kStager = 5;     // the warp that stages table data
constexpr int kFirstDecode = 6;
constexpr uint32_t kTdone = 1u << 16;  // arrivals of an item's `tdone`: its units, and the producer for the rest
constexpr int kStages = 2;     // staging areas for table data
constexpr uint32_t kLutBytes = 65536;
constexpr uint32_t kStageOffs = 40;  // u32: 33 relative offsets, [37] where the first entry landed
constexpr uint32_t kStagePad = 16;   // entries: copies start and end on 8-entry boundaries

// One unit as the producer publishes it with its slot.
struct alignas(16) UnitDesc {
    int32_t item;  // running index of its item in this CTA, or -1: no more units
    uint32_t unit;  // its running number
    int32_t seg;
    uint32_t rows;  // word-rows of its block (0: rejected, nothing to decode)
};

// MMA consumers: the warps that hold a part of an item's sums in their first and second accumulator.
struct alignas(8) ItemState {
    uint32_t acc[2];
};

// An item as the producer records it, with what the other warps need of its job (the job table is in global memory:
// a read of it takes longer than an item's epilogue).
struct alignas(16) ItemRec {
    int32_t it, job, stripe, tab;  // it < 0: no more items; tab: decode table
    int32_t gen;        // number of its table's build in this CTA
    int32_t build;      // not 0: the table is built for this item; the items before build - 1 are the last to use the
                        // table that this overwrites
    int32_t area_item;  // the item whose build must be over before this one's data is staged (-1: none)
    int32_t sb;         // first segment
    uint32_t n, u0;     // number of units, and the first one's running number
    int32_t rows, cols, seg_quads, atomic, local;
    float chain_scale;
    const int8_t *x;
    int32_t *y;
    const float *scales;
    float *ys;
    int8_t *chain_out;  // a chain's int8 output, or nullptr
};

namespace {

__device__ __forceinline__ const Q8Job &job_at(const Q8WLaunch &L, int j) { return L.jobs ? L.jobs[j] : L.job0; }

// mbarriers, in the order they are laid out
struct Bars {
    uint32_t base;  // shared-memory address
    int S, W;
    static constexpr int kFixed = 4 * kRing + kStages;
    __device__ __forceinline__ uint32_t at(int i) const { return base + 8u * (uint32_t)i; }
    __device__ __forceinline__ uint32_t rfull(int k) const { return at(k); }              // item record written
    __device__ __forceinline__ uint32_t tfull(int k) const { return at(kRing + k); }      // decode table ready
    __device__ __forceinline__ uint32_t tdone(int k) const { return at(2 * kRing + k); }  // item decoded
    __device__ __forceinline__ uint32_t idone(int k) const { return at(3 * kRing + k); }  // item's outputs written, record read
    __device__ __forceinline__ uint32_t staged(int g) const { return at(4 * kRing + g); } // table data in shared memory
    __device__ __forceinline__ uint32_t sfull(int s) const { return at(kFixed + s); }
    __device__ __forceinline__ uint32_t sempty(int s) const { return at(kFixed + S + s); }
    __device__ __forceinline__ uint32_t mma(int w) const { return at(kFixed + 2 * S + w); }
    __device__ __forceinline__ uint32_t dempty(int w, int b) const { return at(kFixed + 2 * S + W + 2 * w + b); }
    __device__ __forceinline__ uint32_t xfull(int w, int b) const { return at(kFixed + 2 * S + 3 * W + 2 * w + b); }  // XTiles
    static __host__ __device__ constexpr int count(int S, int W, bool mma) { return kFixed + 2 * S + (mma ? 5 * W : 0); }
    // arrivals that complete barrier i's phase
    __device__ __forceinline__ int arrivals(int i) const {
        if (i >= 2 * kRing && i < 3 * kRing) return (int)kTdone;
        if (i >= 3 * kRing && i < 4 * kRing) return 2;  // the table warps, and the stager, which reads every record too
        if (i >= 4 * kRing && i < kFixed) return 33;  // the stager's lanes, and once for the offsets
        return i >= kFixed + 2 * S + W && i < kFixed + 2 * S + 3 * W ? kTableWarps : 1;  // dempty: every table warp has read the sums
    }
};

// Bounded wait.  A wait that runs out raises MV_DEV_WAIT_TIMEOUT and the CTA's failure flag; every later wait of
// the CTA then gives up within a few polls, and every role leaves its loop.
__device__ __noinline__ bool wait_slow(uint32_t bar, uint32_t parity, uint32_t *status, uint32_t limit,
                                       volatile uint32_t *failed) {
    for (uint32_t it = 0; it < limit; it++) {
        __nanosleep(40);  // a polling warp takes issue slots from the decoding ones
        if (mbar_try_wait(bar, parity)) return true;
        if (*failed) return false;
    }
    atomicOr(status, MV_DEV_WAIT_TIMEOUT);
    *failed = 1u;
    return false;
}
__device__ __forceinline__ bool wait_bar(uint32_t bar, uint32_t parity, const Q8WLaunch &L, volatile uint32_t *failed) {
    if (mbar_try_wait(bar, parity)) return true;
    return wait_slow(bar, parity, L.status, L.spin_limit, failed);
}

// One poll without suspension.
__device__ __forceinline__ bool test_bar(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    return ok != 0;
}

__device__ __forceinline__ void arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void arrive_n(uint32_t bar, uint32_t n) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(n) : "memory");
}
__device__ __forceinline__ void arrive_tx(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ void bulk_in(uint32_t dst, const void *src, uint32_t bytes, uint32_t bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
                 "l"(src), "r"(bytes), "r"(bar)
                 : "memory");
}
// Barrier of the four table warps; true if every one of them passes true.
__device__ __forceinline__ bool table_vote(bool ok) {
    uint32_t r;
    asm volatile(
        "{\n\t.reg .pred p, q;\n\t"
        "setp.ne.u32 p, %1, 0;\n\t"
        "barrier.cta.red.and.pred q, 1, 128, p;\n\t"
        "selp.u32 %0, 1, 0, q;\n\t}"
        : "=r"(r)
        : "r"((uint32_t)ok)
        : "memory");
    return r != 0;
}

// CUDA-core consumers: whether the slots hold their segments' x (segments of up to kXQuads quads, not in a chain)
__device__ __forceinline__ bool x_in_slot(const Q8WLaunch &L, int seg_quads) {
    return L.x_off != 0 && !L.ragged && seg_quads <= kXQuads;
}

// ---------------------------------------------------------------- work items

__device__ __forceinline__ void item_segs(const mv_q8_view &m, int ngroups, int group, int &sb, int &se) {
    const int spp = (m.nseg + ngroups - 1) / ngroups;
    sb = group * spp;
    se = min(m.nseg, sb + spp);
}

// Item number -> job, stripe and segment range.  Each CTA takes its items in increasing order, so the job search
// runs forward from the previous item's job: one comparison in the common case, a binary search otherwise.
__device__ __forceinline__ void locate(const Q8WLaunch &L, uint32_t it, int &job, int &stripe, int &sb, int &se) {
    uint32_t rel = it;
    int ng = L.job0.ngroups;
    if (L.jobs) {
        if (job + 1 < L.njobs && ldp(&L.jobs[job + 1].item0) <= it) {
            int lo = job + 1, hi = L.njobs - 1;
            while (lo < hi) {  // last job with item0 <= it
                const int mid = (lo + hi + 1) >> 1;
                if (ldp(&L.jobs[mid].item0) <= it) lo = mid;
                else hi = mid - 1;
            }
            job = lo;
        }
        rel = it - ldp(&L.jobs[job].item0);
        ng = ldp(&L.jobs[job].ngroups);
    }
    stripe = (int)(rel / (uint32_t)ng);
    item_segs(job_at(L, job).m, ng, (int)(rel % (uint32_t)ng), sb, se);
}

// Item `next` (even shares: the units from `next` to the stripe's end or `limit`): what its record says of the matrix, the
// stripe and the buffers.
__device__ __forceinline__ void fill_item(const Q8WLaunch &L, uint32_t next, uint32_t limit, int &job, ItemRec &r) {
    int se = 0;
    if (L.span) {
        const uint32_t nseg = (uint32_t)L.job0.m.nseg;
        r.stripe = (int)(next / nseg);
        r.sb = (int)(next - (uint32_t)r.stripe * nseg);
        se = (int)min(nseg, (uint32_t)r.sb + (limit - next));
    } else {
        locate(L, next, job, r.stripe, r.sb, se);
    }
    r.job = job;
    r.n = (uint32_t)max(0, se - r.sb);
    const Q8Job &J = job_at(L, job);
    r.rows = J.m.rows;
    r.cols = J.m.cols;
    r.seg_quads = J.m.seg_quads;
    r.local = J.m.local;
    r.atomic = L.span ? (int)r.n < J.m.nseg : J.atomic;
    r.x = J.x;
    r.y = J.y;
    r.scales = J.scales;
    r.ys = J.ys;
    if (L.chain_scales) {
        r.chain_scale = ldp(L.chain_scales + job);
        r.chain_out = job + 1 < L.njobs ? const_cast<int8_t *>(L.jobs[job + 1].x) : L.chain_out8;
    }
}

// The chained pipeline's int8 output: the reference's fp32 requantisation (ans-warp-rows-kernel.cu:212-220).
__device__ __forceinline__ int8_t chain_q(const ItemRec &I, int sum) {
    return (int8_t)max(-128, min(127, __float2int_rn((float)sum * I.chain_scale)));
}

// The scale of a row's outputs (loaded ahead of the stores, which a plain load would not pass).
__device__ __forceinline__ float row_scale(const ItemRec &I, int row) {
    return I.ys && row < I.rows ? ldp(I.scales + row) : 0.f;
}

// One output: y (exact int32), its scaled form, and the chain's int8.
__device__ __forceinline__ void emit(const ItemRec &I, int v, int row, int sum, float scale) {
    const size_t i = (size_t)v * I.rows + row;
    if (I.atomic) {
        atomicAdd(I.y + i, sum);
        return;
    }
    I.y[i] = sum;
    if (I.ys) I.ys[i] = (float)sum * scale;
    if (I.chain_out) I.chain_out[i] = chain_q(I, sum);
}

// ------------------------------------------------------------------- producer

// Table data of item r into staging area r.gen % kStages: offsets relative to the first entry by plain loads, the
// entries by 16-byte asynchronous copies (zero-filled past the readable end), both counted on the area's barrier.
__device__ __forceinline__ void stage_table(const Q8WLaunch &L, const ItemRec &r, unsigned char *sm, const Bars &B, int lane) {
    const mv_q8_view &m = job_at(L, r.job).m;
    const int area = r.gen % kStages;
    uint32_t *so = reinterpret_cast<uint32_t *>(sm + L.lay.stage_o) + area * kStageOffs;
    const uint32_t r0 = m.local ? (uint32_t)r.stripe * 32u : 0u;
    const uint32_t nt = m.local ? 32u : 1u;
    const uint32_t *toff = m.tbl_off + r0;  // (the job's fields once, ahead of the stores: a plain load passes none)
    const uint16_t *tbl = m.tbl;
    const uint32_t tbl_len = m.tbl_len;
    const uint32_t o = ldp(toff + min((uint32_t)lane, nt));
    const uint32_t te = ldp(toff + nt);
    const uint32_t tb = __shfl_sync(0xffffffffu, o, 0);
    const bool ok = te >= tb && te <= tbl_len && te - tb <= (uint32_t)L.tbl_stage;
    if ((uint32_t)lane <= nt) so[lane] = (ok && o >= tb && o <= te) ? o - tb : 0u;
    if (lane == 0) {
        if (nt == 32u) so[32] = ok ? te - tb : 0u;
        so[37] = tb & 7u;
        if (!ok) atomicOr(L.status, MV_DEV_BAD_TABLE);
    }
    if (ok) {
        const uint32_t a = tb & ~7u, n = te - a;
        unsigned char *se = sm + L.lay.stage_e + (uint32_t)area * ((uint32_t)L.tbl_stage + kStagePad) * 2u;
        if (((uintptr_t)tbl & 15) == 0) {
            const uint32_t dst = smem_u32(se);
            for (uint32_t c = lane; 8 * c < n; c += 32) {
                const uint32_t avail = min(8u, tbl_len - (a + 8 * c));
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst + 16u * c), "l"(tbl + a + 8 * c),
                             "r"(2u * avail)
                             : "memory");
            }
        } else {
            uint16_t *d = reinterpret_cast<uint16_t *>(se);
            for (uint32_t e = lane; e < n; e += 32) d[e] = ldp(tbl + a + e);
        }
    }
    cp_async_mbar_arrive_noinc(B.staged(area));
    __syncwarp();
    if (lane == 0) arrive(B.staged(area));
}

// The stager warp: the table data of every item that needs a build, as soon as its record is written.
__device__ __forceinline__ void stage_tables(const Q8WLaunch &L, unsigned char *sm, const Bars &B, volatile uint32_t *failed) {
    const int lane = threadIdx.x & 31;
    const ItemRec *ring = reinterpret_cast<const ItemRec *>(sm + L.lay.ring);
    for (int k = 0;; k++) {
        if (!__all_sync(0xffffffffu, wait_bar(B.rfull(k % kRing), (uint32_t)(k / kRing) & 1u, L, failed))) break;
        const ItemRec &r = ring[k % kRing];
        if (r.it < 0) break;
        if (r.build) {
            if (r.area_item >= 0 && r.area_item > k - kRing) {  // (earlier items are done)
                const bool built = wait_bar(B.tfull(r.area_item % kRing), (uint32_t)(r.area_item / kRing) & 1u, L, failed);
                if (!__all_sync(0xffffffffu, built)) break;
            }
            stage_table(L, r, sm, B, lane);
            if (k == 0) grid_dependency_wait();  // (see produce)
        }
        __syncwarp();
        if (lane == 0) arrive(B.idone(k % kRing));  // the record may be overwritten
    }
    cp_async_wait_all();
}

__device__ __forceinline__ void produce(const Q8WLaunch &L, unsigned char *sm, const Bars &B, volatile uint32_t *failed) {
    const int lane = threadIdx.x & 31;
    ItemRec *ring = reinterpret_cast<ItemRec *>(sm + L.lay.ring);
    UnitDesc *desc = reinterpret_cast<UnitDesc *>(sm + L.lay.desc);
    const uint32_t slots = smem_u32(sm) + L.lay.slots;
    const uint32_t S = (uint32_t)L.S, W = (uint32_t)L.W;
    uint32_t u = 0, recorded = 0;  // units published, units of the items recorded
    // the CTA's latest item number (even shares: its first unit); its first one is static
    uint32_t next = L.span ? (uint32_t)((uint64_t)blockIdx.x * L.span / gridDim.x) : blockIdx.x;
    const uint32_t limit = L.span ? (uint32_t)((uint64_t)(blockIdx.x + 1) * L.span / gridDim.x) : L.nitems;
    uint32_t grabbed = 0;        // lane 0: the queue's answer for the item after it
    int job = 0, tjob = -1, tstripe = -1, gen = -1;
    int fb1 = -1, fb2 = -1;  // first items of the two latest table builds (fb1 the latest)
    bool ok = true;

    // Writes item k's record (its number is in `next`) and takes the number after it, so that the queue's latency
    // passes while units go out.
    auto record = [&](int k) {
        if (k >= kRing && ok) ok = wait_bar(B.idone(k % kRing), (uint32_t)(k / kRing - 1) & 1u, L, failed);
        ItemRec r{};
        const bool end = next >= limit;
        r.it = end ? -1 : (int32_t)next;
        r.n = W;  // one end mark per decode warp
        r.u0 = recorded;
        r.area_item = -1;
        if (!end) {
            fill_item(L, next, limit, job, r);
            if (L.queue && k > 0 && lane == 0) grabbed = atomicAdd(L.queue, 1u);
            r.build = job != tjob || (r.local && r.stripe != tstripe);
            if (r.build) {
                // two tables and two staging areas: build g overwrites those of build g - 2
                gen++;
                r.area_item = gen >= 2 ? fb2 : -1;
                r.build = 1 + max(fb1, 0);
                fb2 = fb1;
                fb1 = k;
                tjob = job;
                tstripe = r.stripe;
            }
            r.gen = gen;
            r.tab = gen & 1;
        }
        recorded += r.n;
        if (ok && lane == 0) {
            ring[k % kRing] = r;
            if (!end) arrive_n(B.tdone(k % kRing), kTdone - r.n);  // the units' arrivals are left
            arrive(B.rfull(k % kRing));
        }
        __syncwarp();
        return r;
    };
    ItemRec r = record(0);
    // Up to here, and in the first table's staging and build, only the matrix was read (L.early: see q8w_kernel).  Inputs,
    // outputs and the queue come after the launch before this one.
    grid_dependency_wait();
    grid_launch_dependents();
    if (L.queue && r.it >= 0 && lane == 0) grabbed = atomicAdd(L.queue, 1u);
    for (int k = 0; ok; k++) {
        const bool end = r.it < 0;
        const mv_q8_view &m = job_at(L, r.job).m;
        // The next item's record goes ahead of this item's last units, so that its table is built while this item
        // decodes.
        ItemRec rn{};
        bool ahead = end;
        auto look_ahead = [&]() {
            next = L.queue ? __shfl_sync(0xffffffffu, grabbed, 0) + gridDim.x : next + (L.span ? r.n : gridDim.x);
            // the counter is reset by whoever makes the launch's last grab
            if (L.queue && lane == 0 && next == L.nitems + gridDim.x - 1) atomicExch(L.queue, 0u);
            rn = record(k + 1);
            ahead = true;
        };
        for (uint32_t base = 0; base < r.n && ok; base += 32) {
            const uint32_t i = base + (uint32_t)lane;
            uint32_t o0 = 0, rows = 0;
            if (!end && i < r.n) {
                const int b = r.stripe * m.nseg + r.sb + (int)i;
                o0 = ldp(m.blk_off + b);
                const uint32_t o1 = ldp(m.blk_off + b + 1);
                rows = o1 - o0;
                if (o1 < o0 || o1 > m.blocks_rows || rows < 2 || rows >= L.block_bytes / 128u) {
                    atomicOr(L.status, MV_DEV_STREAM_OVERRUN);
                    rows = 0;
                }
            }
            const uint32_t cnt = min(32u, r.n - base);
            const uint32_t ui = u + (uint32_t)lane, slot = ui % S, turn = ui / S;
            // the slots become free in unit order: publish the leading run of free ones, then wait for the next
            for (uint32_t pos = 0, it = 0; pos < cnt;) {
                const bool mine = (uint32_t)lane >= pos && (uint32_t)lane < cnt;
                const bool free_ = mine && (turn == 0 || test_bar(B.sempty((int)slot), (turn - 1) & 1u));
                const uint32_t ball = __ballot_sync(0xffffffffu, free_) >> pos;
                const uint32_t run = ~ball ? (uint32_t)__ffs((int)~ball) - 1u : 32u;
                if (run) {
                    if (mine && (uint32_t)lane < pos + run) {
                        UnitDesc d;
                        d.item = end ? -1 : k;
                        d.unit = ui;
                        d.seg = r.sb + (int)i;
                        d.rows = rows;
                        desc[slot] = d;
                        const uint32_t dst = slots + slot * L.slot_bytes, bar = B.sfull((int)slot);
                        // the block, and behind it (CUDA-core consumers) the segment's x of every vector
                        const int q = (r.sb + (int)i) * m.seg_quads;
                        const uint32_t xb = x_in_slot(L, m.seg_quads) && rows
                                                ? L.x_quad * (uint32_t)max(0, min(m.seg_quads, (m.cols >> 2) - q))
                                                : 0u;
                        arrive_tx(bar, rows * 128u + xb * (uint32_t)L.batch);
                        if (rows && !L.drop_copy) {
                            bulk_in(dst, m.blocks + (size_t)o0 * 32, rows * 128u, bar);
                            const int8_t *x = r.x + (size_t)L.x_quad * q;
                            if (xb)
                                for (int v = 0; v < L.batch; v++)
                                    bulk_in(dst + L.x_off + L.x_quad * (uint32_t)(v * m.seg_quads), x + (size_t)v * (m.cols >> 2) * L.x_quad, xb, bar);
                        }
                    }
                    __syncwarp();
                    pos += run;
                    it = 0;
                    continue;
                }
                if (!ahead) {
                    look_ahead();
                    if (!ok) break;
                    continue;
                }
                const uint32_t us = u + pos;
                if (mbar_try_wait(B.sempty((int)(us % S)), (us / S - 1) & 1u)) continue;
                __nanosleep(40);
                if (++it >= L.spin_limit || *failed) {
                    if (it >= L.spin_limit && lane == 0) atomicOr(L.status, MV_DEV_WAIT_TIMEOUT);
                    *failed = 1u;
                    ok = false;
                    break;
                }
            }
            u += cnt;
        }
        if (end) break;
        if (ok && !ahead) look_ahead();
        r = rn;
    }
    if (!ok) {
        // a failed launch still leaves the queue at zero: take (and drop) items until one grab fails
        if (L.queue && lane == 0 && next < L.nitems) {
            next = grabbed + gridDim.x;
            for (;;) {
                if (next == L.nitems + gridDim.x - 1) atomicExch(L.queue, 0u);
                if (next >= L.nitems) break;
                next = atomicAdd(L.queue, 1u) + gridDim.x;
            }
        }
        // no copy may be left writing the shared memory of a CTA that has exited: wait (bounded) for each slot's
        // latest one
        const uint32_t live = min(u, S);
        for (uint32_t i = lane; i < live; i += 32) {
            const uint32_t ui = u - 1 - i;
            for (uint32_t it = 0; it < L.spin_limit; it++)
                if (mbar_try_wait(B.sfull((int)(ui % S)), (ui / S) & 1u)) break;
        }
        __syncwarp();
    }
}

// --------------------------------------------------------------- table warps

// Table entries: of the integer consumers f | sym << 16 | r << 24, of the float ones f | r << 8 | bf16(sym) << 16.
template <bool kFloat>
__device__ __forceinline__ uint32_t table_entry(uint32_t ent) {  // r = 0; ent: symbol | f << 8
    if constexpr (kFloat)
        return (ent >> 8) |
               (uint32_t)__bfloat16_as_ushort(__float2bfloat16_rn((float)(int8_t)(uint8_t)(ent & 0xFFu))) << 16;
    else
        return (ent >> 8) | (ent & 0xFFu) << 16;
}

// Decode table from the staged data: warp s fills quantiles [64 s, 64 s + 64), lane l its row's column, with no
// divergence: the column is cleared, each symbol's entry (r = 0) goes to its first quantile, and one pass then
// carries the entries forward, r growing by one per quantile.  (A walk that stores quantile by quantile and moves
// to the next symbol by a branch took 3.2 us a table with the decode warps at work.)
template <bool kFloat>
__device__ __forceinline__ void build_table(const Q8WLaunch &L, int local, unsigned char *lut,
                                            const uint32_t *so, const uint16_t *tsm) {
    const int s = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int t = local ? lane : 0;
    const uint32_t o1 = max(so[t + 1], so[t]);
    const uint32_t qlo = 64u * (uint32_t)s, qhi = qlo + 64u;
    uint32_t k = so[t], cum = 0;
    unsigned char *rows = lut + 256u * qlo;
    {  // clear: lane l the 16 bytes 16 (l % 8) of rows l / 8, l / 8 + 4, ...
        unsigned char *z = rows + 256u * (uint32_t)(lane >> 3) + 16u * (uint32_t)(lane & 7);
#pragma unroll
        for (int i = 0; i < 16; i++) *reinterpret_cast<uint4 *>(z + 1024 * i) = make_uint4(0, 0, 0, 0);
    }
    // symbols that end at or before qlo, four at a time (independent loads)
    while (k + 4 <= o1) {
        const uint32_t c4 = cum + ((uint32_t)tsm[k] >> 8) + ((uint32_t)tsm[k + 1] >> 8) +
                            ((uint32_t)tsm[k + 2] >> 8) + ((uint32_t)tsm[k + 3] >> 8);
        if (c4 > qlo) break;
        cum = c4;
        k += 4;
    }
    uint32_t ent = k < o1 ? (uint32_t)tsm[k] : 0u;
    while (k < o1 && cum + (ent >> 8) <= qlo) {
        cum += ent >> 8;
        k++;
        ent = k < o1 ? (uint32_t)tsm[k] : 0u;
    }
    // the symbol that holds qlo starts the pass; e is one step (r) behind
    bool bad = k >= o1;
    constexpr uint32_t kR = kFloat ? 1u << 8 : 1u << 24;  // one step of r
    uint32_t e = table_entry<kFloat>(ent) + (qlo - cum - 1u) * kR;
    cum += ent >> 8;
    __syncwarp();
    unsigned char *col = rows + 4u * (uint32_t)lane;
    while (cum < qhi) {
        k++;
        if (k >= o1) {  // the table ends early
            bad = true;
            break;
        }
        ent = tsm[k];
        if ((ent >> 8) == 0) bad = true;
        *reinterpret_cast<uint32_t *>(col + 256u * (cum - qlo)) = table_entry<kFloat>(ent);
        cum += ent >> 8;
    }
    __syncwarp();
    if (__any_sync(0xffffffffu, bad)) {
        // not a valid table: entries of one quantile each keep the decode in bounds
        atomicOr(L.status, MV_DEV_BAD_TABLE);
        for (int q = 0; q < 64; q++) *reinterpret_cast<uint32_t *>(col + 256 * q) = 1u;
        return;
    }
#pragma unroll 16
    for (int q = 0; q < 64; q++) {
        const uint32_t v = *reinterpret_cast<const uint32_t *>(col + 256 * q);
        e = v ? v : e + kR;
        *reinterpret_cast<uint32_t *>(col + 256 * q) = e;
    }
}

// Chained pipeline: wait (thread 0, bounded) until every work item of job j is counted.  Items are numbered in job
// order, each CTA takes its items in increasing order and the launch is cooperative, so the items waited for are
// always making progress.
__device__ __forceinline__ void chain_wait(const Q8WLaunch &L, int j, volatile uint32_t *failed) {
    const uint32_t need = (j + 1 < L.njobs ? L.jobs[j + 1].item0 : L.nitems) - L.jobs[j].item0;
    const uint32_t *cnt = &L.jobs[j].pad;
    for (uint32_t it = 0;; it++) {
        uint32_t done;
        asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(done) : "l"(cnt) : "memory");
        if (done >= need) break;
        if (it >= L.spin_limit) {
            atomicOr(L.status, MV_DEV_WAIT_TIMEOUT);
            *failed = 1u;
            break;
        }
        __nanosleep(32);
    }
}

// --------------------------------------------------------------------- decode

// One stream: the lane's 64-bit state, its next refill word (already loaded), the offset of the one after that and
// the bound on that offset (the row after the block).
struct Stream {
    uint32_t lo, hi, nw, koff, kend, P;
    __device__ __forceinline__ Stream(const unsigned char *sm, uint32_t soff, uint32_t rows, int lane) {
        const uint32_t a = smem_u32(sm) + soff + (uint32_t)lane * 4u;
        asm volatile("ld.shared.u32 %0, [%1];" : "=r"(lo) : "r"(a) : "memory");
        asm volatile("ld.shared.u32 %0, [%1+128];" : "=r"(hi) : "r"(a) : "memory");
        asm volatile("ld.shared.u32 %0, [%1+256];" : "=r"(nw) : "r"(a) : "memory");
        koff = a + 384u;
        kend = a + rows * 128u;
        P = 0;
    }
    // the encoder starts every segment from the last quad's frequency product, so the decoder ends there
    __device__ __forceinline__ bool ok() const { return hi == 0 && lo == P; }
    // A corrupt stream stays within 4 word-rows of its block: called every 4 steps.
    __device__ __forceinline__ void clamp() { koff = min(koff, kend); }
    // Refill (predicated: a branch-free `select` form of it takes 4 instructions more) and the four table entries.
    __device__ __forceinline__ void step(const unsigned char *sm, uint32_t lw, uint32_t (&e)[4]) {
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "setp.eq.u32 p, %1, 0;\n\t"
            "@p mov.u32 %1, %0;\n\t"
            "@p mov.u32 %0, %2;\n\t"
            "@p ld.shared.u32 %2, [%3];\n\t"
            "@p add.u32 %3, %3, 128;\n\t}"
            : "+r"(lo), "+r"(hi), "+r"(nw), "+r"(koff)::"memory");
        e[0] = *reinterpret_cast<const uint32_t *>(sm + __byte_perm(lo, lw, 0x7604));
        e[1] = *reinterpret_cast<const uint32_t *>(sm + __byte_perm(lo, lw, 0x7614));
        e[2] = *reinterpret_cast<const uint32_t *>(sm + __byte_perm(lo, lw, 0x7624));
        e[3] = *reinterpret_cast<const uint32_t *>(sm + __byte_perm(lo, lw, 0x7634));
    }
    // (hi:lo) = hi * p01 p23 + u01 + p01 u23 (written as the two halves of one wide multiply-add: the 64-bit C form
    // costs register moves)
    __device__ __forceinline__ void update(uint32_t u01, uint32_t p01, uint32_t u23, uint32_t p23) {
        P = p01 * p23;
        const uint32_t t = u01 + p01 * u23;
        uint32_t h;
        asm("{\n\tmad.lo.cc.u32 %0, %2, %3, %4;\n\tmadc.hi.u32 %1, %2, %3, 0;\n\t}"
            : "=&r"(lo), "=r"(h)
            : "r"(hi), "r"(P), "r"(t));
        hi = h;
    }
    // one step; returns the four packed int8 symbols
    __device__ __forceinline__ uint32_t step_i8(const unsigned char *sm, uint32_t lw) {
        uint32_t e[4];
        step(sm, lw, e);
        // entry bytes (f, 0, sym, r): r0 + f0 r1 = e0 . (r1, 0, 0, 1); f0 f1 = dp2a of e1's low half with e0's f
        const uint32_t u01 = __dp4a(e[0], __byte_perm(e[1], 1u, 0x4553), 0u);
        const uint32_t u23 = __dp4a(e[2], __byte_perm(e[3], 1u, 0x4553), 0u);
        const uint32_t p01 = __dp2a_lo(e[1], e[0], 0u), p23 = __dp2a_lo(e[3], e[2], 0u);
        update(u01, p01, u23, p23);
        return __byte_perm(__byte_perm(e[0], e[1], 0x0062), __byte_perm(e[2], e[3], 0x0062), 0x5410);
    }
    // one step over the float consumers' table: the four entries, whose upper halves are the bf16 symbols
    __device__ __forceinline__ void step_f(const unsigned char *sm, uint32_t lw, uint32_t (&e)[4]) {
        step(sm, lw, e);
        // entry bytes (f, r, bf16): r0 + f0 r1 = e0 . (r1, 1, 0, 0), f0 f1 = e0 . (f1, 0, 0, 0)
        const uint32_t u01 = __dp4a(e[0], __byte_perm(e[1], 1u, 0x5541), 0u);
        const uint32_t u23 = __dp4a(e[2], __byte_perm(e[3], 1u, 0x5541), 0u);
        const uint32_t p01 = __dp4a(e[0], e[1] & 0xFFu, 0u), p23 = __dp4a(e[2], e[3] & 0xFFu, 0u);
        update(u01, p01, u23, p23);
    }
    // the four symbols as two bf16 pairs
    __device__ __forceinline__ void step_bf16(const unsigned char *sm, uint32_t lw, uint32_t &w01, uint32_t &w23) {
        uint32_t e[4];
        step_f(sm, lw, e);
        w01 = __byte_perm(e[0], e[1], 0x7632);
        w23 = __byte_perm(e[2], e[3], 0x7632);
    }
};

// x is read with plain (coherent) loads: in a chain it was written earlier in the same launch.
__device__ __forceinline__ uint4 ldx_u4(const void *p) { return *reinterpret_cast<const uint4 *>(p); }

// Ragged x: the four bytes at p, of which `valid` belong to the row (the others are zero), from two aligned words; by
// single bytes where those would leave the launch's x.
__device__ __forceinline__ uint32_t x_quad_at(const Q8WLaunch &L, const int8_t *p, int valid) {
    if (valid <= 0) return 0u;
    const int8_t *x0 = L.job0.x, *xe = x0 + (size_t)L.batch * L.job0.m.cols;
    const uint32_t *a = reinterpret_cast<const uint32_t *>((uintptr_t)p & ~(uintptr_t)3);
    uint32_t v = 0;
    if ((uintptr_t)a >= (uintptr_t)x0 && (uintptr_t)(a + 2) <= (uintptr_t)xe) {
        v = __funnelshift_r(ldp(a), ldp(a + 1), 8u * (uint32_t)((uintptr_t)p & 3));
        if (valid < 4) v &= (1u << (8 * valid)) - 1u;
    } else {
        for (int j = 0; j < min(valid, 4); j++) v |= (uint32_t)(uint8_t)ldp(p + j) << (8 * j);
    }
    return v;
}

// CUDA-core consumer: NV int8 vectors, dp4a.  The lane's partial sums go to the item's area in shared memory
// (exact integer atomics); the table warps write the outputs.  kRagged: the warp lays out x itself, 64 quads at a time, in
// the slot's place for it, and the last group of a segment may be of fewer than 4 quads.
template <int NV, bool kRagged = false>
struct DotCons {
    static constexpr bool kMma = false, kFloat = false, kStatic = false, kPrepare = false;
    static constexpr int kRed = NV * 32;  // ints of an item's partial sums
    static constexpr int kAreas = kRing;  // of them, in turn
    static constexpr int kLag = NV <= 2 ? 1 : 4;
    static constexpr int kMaxDecode = NV <= 2 ? 16 : NV <= 4 ? 14 : NV <= 8 ? 10 : 6;
    static constexpr uint32_t tile_bytes(int) { return 0; }
    const int8_t *x;
    int cols, seg_quads, qtot;
    bool in_slot;
    static constexpr int kUnroll = NV <= 2 ? 4 : 1;
    int acc[NV];
    __device__ __forceinline__ void init(const Q8WLaunch &, unsigned char *, const Bars &, uint32_t, int) {
#pragma unroll
        for (int v = 0; v < NV; v++) acc[v] = 0;
    }
    __device__ __forceinline__ void begin_item(const Q8WLaunch &L, const ItemRec &I, int) {
        in_slot = x_in_slot(L, I.seg_quads);
        x = I.x;
        cols = I.cols;
        seg_quads = I.seg_quads;
        qtot = (cols + 3) >> 2;
    }
    __device__ __forceinline__ void group(Stream &s, const unsigned char *sm, uint32_t lw, const uint4 (&xv)[NV]) {
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const uint32_t w = s.step_i8(sm, lw);
#pragma unroll
            for (int v = 0; v < NV; v++) {
                const uint32_t xw = j == 0 ? xv[v].x : j == 1 ? xv[v].y : j == 2 ? xv[v].z : xv[v].w;
                acc[v] = __dp4a((int)w, (int)xw, acc[v]);
            }
        }
        s.clamp();
    }
    // 16 bytes of every vector at p (NV is the batch rounded up, so that one or two vectors are all there)
    __device__ __forceinline__ void load_x(const int8_t *p, int batch, uint4 (&xv)[NV]) const {
#pragma unroll
        for (int v = 0; v < NV; v++) {
            xv[v] = ldx_u4(p);
            if (NV <= 2 || v + 1 < batch) p += cols;
        }
    }
    __device__ __forceinline__ void unit(const Q8WLaunch &L, const UnitDesc &d, const unsigned char *sm, uint32_t soff,
                                         uint32_t lw, int lane, volatile uint32_t *) {
        const int q0 = d.seg * seg_quads;
        const int nq = min(seg_quads, qtot - q0);
        Stream s(sm, soff, d.rows, lane);
        if constexpr (kRagged) {
            uint32_t *xs = const_cast<uint32_t *>(reinterpret_cast<const uint32_t *>(sm + soff + L.x_off));
            for (int q = 0; q < nq; q += kXQuads) {
                const int n = min(kXQuads, nq - q);
                for (int v = 0; v < L.batch; v++)
                    for (int i = lane; i < n; i += 32) {
                        const int col = 4 * (q0 + q + i);
                        xs[kXQuads * v + i] = x_quad_at(L, x + (size_t)v * cols + col, cols - col);
                    }
                __syncwarp();
                const uint32_t *xq = xs;
                int i = 0;
#pragma unroll 1
                for (; i + 4 <= n; i += 4, xq += 4) {
                    uint4 xv[NV];
#pragma unroll
                    for (int v = 0; v < NV; v++) xv[v] = *reinterpret_cast<const uint4 *>(xq + kXQuads * v);
                    group(s, sm, lw, xv);
                }
#pragma unroll 1
                for (; i < n; i++, xq++) {
                    const uint32_t w = s.step_i8(sm, lw);
#pragma unroll
                    for (int v = 0; v < NV; v++) acc[v] = __dp4a((int)w, (int)xq[kXQuads * v], acc[v]);
                }
                s.clamp();
                __syncwarp();
            }
        } else if (in_slot) {  // x came with the block and lies behind it
            const unsigned char *xs = sm + soff + L.x_off;
            // unrolled: the loop's back edge costs register moves (4 instructions a step without)
#pragma unroll kUnroll
            for (int i = 0; i < nq; i += 4, xs += 16) {  // segments are whole groups of 4 quads (cols % 16 == 0)
                uint4 xv[NV];
#pragma unroll
                for (int v = 0; v < NV; v++) xv[v] = *reinterpret_cast<const uint4 *>(xs + 4 * v * seg_quads);
                group(s, sm, lw, xv);
            }
        } else {  // x from global memory, one group ahead: long segments, and chains, whose x is not there any earlier
            // (the vectors past the batch, whose sums nobody reads, read its last row: x ends there)
            const int8_t *xp = x + 4 * q0;
            uint4 xn[NV];
            load_x(xp, L.batch, xn);
            for (int i = 0; i < nq; i += 4) {
                uint4 xv[NV];
                xp += i + 4 < nq ? 16 : 0;
#pragma unroll
                for (int v = 0; v < NV; v++) xv[v] = xn[v];
                load_x(xp, L.batch, xn);
                group(s, sm, lw, xv);
            }
        }
        if (!s.ok()) atomicOr(L.status, MV_DEV_FINAL_STATE);
    }
    __device__ __forceinline__ void end_unit(const Q8WLaunch &L, int k, bool, unsigned char *sm, const Bars &B, int lane,
                                             volatile uint32_t *) {
        int *red = reinterpret_cast<int *>(sm + L.lay.red) + (size_t)(k % kRing) * NV * 32 + lane;
#pragma unroll
        for (int v = 0; v < NV; v++) {
            atomicAdd(red + v * 32, acc[v]);
            acc[v] = 0;
        }
        __syncwarp();
        if (lane == 0) arrive(B.tdone(k % kRing));
    }
    // Table warps: the item's sums, one vector per warp at a time, lane = stripe row.
    static __device__ __forceinline__ void epilogue(const Q8WLaunch &L, const ItemRec &I, int k, unsigned char *sm,
                                                    const Bars &, uint32_t) {
        const int q = threadIdx.x >> 5, lane = threadIdx.x & 31;
        volatile int *red = reinterpret_cast<volatile int *>(sm + L.lay.red) + (size_t)(k % kRing) * NV * 32 + lane;
        const int row = I.stripe * 32 + lane;
        const float scale = row_scale(I, row);
        for (int v = q; v < NV; v += kTableWarps) {
            const int sum = red[v * 32];
            red[v * 32] = 0;
            if (row < I.rows && v < L.batch) emit(I, v, row, sum, scale);
        }
    }
    __device__ __forceinline__ void drain(const Q8WLaunch &) {}
};

// x tiles of a decode warp, for consumers of a single matrix with up to 64 vectors: 64 bytes of every vector (a tile row,
// swizzled), brought in by one tensor copy of lane 0.  (As 16-byte asynchronous copies by all lanes: MmaCons, 64 vectors,
// 1400 cycles to issue a tile's copies, a quarter of the decode's time.)  With more than 16 vectors two buffers, the next
// tile's copy a whole tile's decode ahead of its MMAs; a smaller tile comes in while its own weights decode, which leaves
// the memory to the stream slots and so to more decode warps.  Measured on a B200, 64 vectors, before and after:
// 11008x4096, int8 58 -> 46 us, bf16 84 -> 58; 4096x11008, 50 -> 40 and 81 -> 51.
struct XTiles {
    static __host__ __device__ constexpr uint32_t second(int xrows) { return xrows > 16 ? 1u : 0u; }  // a second buffer?
    static constexpr uint32_t bytes(int xrows) { return (1u + second(xrows)) * 64u * (uint32_t)xrows; }
    uint32_t at, bar, n;  // n: copies issued (lane 0)
    uint64_t a_desc;
    __device__ __forceinline__ void init(const Bars &B, int w, uint32_t address) {
        at = address;
        bar = B.xfull(w, 0);
        n = 0;
        a_desc = umma_smem_desc_sw64(address);
    }
    // tile i: columns from col on (its buffer's previous MMAs are done).  Once the CTA has failed nothing is copied any
    // more: the waits for earlier tiles may have given up.
    __device__ __forceinline__ void load(const Q8WLaunch &L, uint32_t i, int col, int lane, volatile uint32_t *failed) {
        if (lane != 0 || *failed) return;
        const uint32_t b = i & second(L.xrows), size = 64u * (uint32_t)L.xrows;
        arrive_tx(bar + 8u * b, size);
        asm volatile(
            "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(
                at + b * size),
            "l"(&L.xmap), "r"(col), "r"(0), "r"(bar + 8u * b)
            : "memory");
        n = i + 1;
    }
    // at a unit's start, and once the MMAs before tile i are done (the unit's tile at col, `next`: with one after it):
    // `pitch` columns a tile
    __device__ __forceinline__ void begin(const Q8WLaunch &L, uint32_t i, int col, int lane, volatile uint32_t *failed) {
        if (second(L.xrows)) load(L, i, col, lane, failed);
    }
    __device__ __forceinline__ void refill(const Q8WLaunch &L, uint32_t i, int col, int pitch, bool next, int lane,
                                           volatile uint32_t *failed) {
        if (!second(L.xrows)) load(L, i, col, lane, failed);
        else if (next) load(L, i + 1, col + pitch, lane, failed);
    }
    // the issuing lane: tile i is there; its descriptor
    __device__ __forceinline__ uint64_t wait(const Q8WLaunch &L, uint32_t i, volatile uint32_t *failed) const {
        const uint32_t two = second(L.xrows);
        wait_bar(bar + 8u * (i & two), (i >> two) & 1u, L, failed);
        return a_desc + (uint64_t)((i & two) * 4u * (uint32_t)L.xrows);
    }
    // no copy may be left writing when the CTA exits
    __device__ __forceinline__ void drain(const Q8WLaunch &L, int lane) const {
        if (lane != 0) return;
        const uint32_t two = second(L.xrows);
        for (uint32_t i = n <= two ? 0u : n - 1u - two; i < n; i++)
            for (uint32_t it = 0; it < L.spin_limit; it++)
                if (mbar_try_wait(bar + 8u * (i & two), (i >> two) & 1u)) break;
    }
};

// Tensor-core consumer, up to 64 int8 vectors: D[vector][row] += x tile . W tile^T, kind::i8, exact int32.
//   A = x: M = 64 vectors (rows past xrows read whatever follows and only reach lanes that are never read), 64 columns
//       at a time, K-major: by tensor copies (XTiles), or, kOwn, whose x may be one of many (stacks), as core matrices
//       (8 vectors x 16 bytes) by the warp's own cp.async;
//   B = W: the 32 rows of the stripe, each lane storing its row's 16-byte pieces (K-major, conflict-free);
//   D: 32 TMEM columns per decode warp, vector v in lane 32 (v / 16) + v % 16.
// Per 16 quads: two MMAs (K = 32) and one commit.  The previous pair's MMAs are waited for after the first 4 quads
// of the next one are decoded, when the W tile is rewritten (kOwn: and the x tile, whose copies land during the other 12).
//
// kOwn (up to 16 vectors): the A operand starts 16 rows per lane quarter early, so that the vectors land in the warp's
// own quarter; the warp reads its sums itself after each unit and adds them to the item's in shared memory.  With more
// vectors the sums stay in TMEM for the item, the table warps read every warp's (one lane quarter each), and items
// alternate between two accumulators, the second in the 16 lanes of each quarter that M = 64 leaves free.
//
// kRagged: the warp gathers its x tiles by plain loads, and a segment may end within a piece.
template <bool kOwn, bool kRagged = false>
struct MmaCons {
    static constexpr bool kMma = true, kFloat = false, kStatic = false, kPrepare = false;
    static constexpr bool kTma = !kOwn && !kRagged;  // x by XTiles
    static constexpr int kPitch = 33;  // words per vector of the item's sums: lanes (vectors) hit distinct banks
    static constexpr int kRed = kOwn ? 16 * kPitch : 0;
    static constexpr int kAreas = kRing;
    static constexpr int kLag = kOwn ? 4 : 2;  // accumulators
    static constexpr int kMaxDecode = 16;
    static constexpr uint32_t kWTile = 2048;  // 32 rows x 64 columns
    static constexpr uint32_t tile_bytes(int xrows) { return kWTile + (kTma ? XTiles::bytes(xrows) : 64u * (uint32_t)xrows); }
    const int8_t *x;
    int cols, seg_quads, qtot;
    XTiles xs;  // kTma
    uint32_t wt, xt, d_tmem, lbo, nmma, ndp;  // nmma: commits so far, ndp: earlier items this warp has had a part in
    uint32_t mbar, dempty;                    // dempty: of the first accumulator; the second's follows
    uint64_t a_desc, b_desc;
    int warp;
    bool any;
    __device__ __forceinline__ void init(const Q8WLaunch &L, unsigned char *sm, const Bars &B, uint32_t tmem, int w) {
        warp = w;
        wt = smem_u32(sm) + L.lay.tiles + (uint32_t)w * tile_bytes(L.xrows);
        xt = wt + kWTile;
        lbo = 16u * (uint32_t)L.xrows;
        const uint32_t quarter = (uint32_t)(w + kFirstDecode) & 3u;  // of TMEM lanes, by the warp's number in the CTA
        d_tmem = tmem + 32u * (uint32_t)w;
        a_desc = umma_smem_desc(kOwn ? xt - 256u * quarter : xt, lbo, 128u);
        if (kTma) xs.init(B, w, xt);
        b_desc = umma_smem_desc(wt, 512u, 128u);
        mbar = B.mma(w);
        dempty = B.dempty(w, 0);
        nmma = ndp = 0;
        any = false;
    }
    __device__ __forceinline__ void begin_item(const Q8WLaunch &, const ItemRec &I, int) {
        if (!kOwn) {
            if (any) ndp++;  // the sums of the item before stay where they are until a table warp has read them
            any = false;
        }
        x = I.x;
        cols = I.cols;
        seg_quads = I.seg_quads;
        qtot = (cols + 3) >> 2;
    }
    // the accumulator of the current item (they alternate) is free: its sums of two items ago are read
    __device__ __forceinline__ void wait_acc(const Q8WLaunch &L, volatile uint32_t *failed) const {
        if (!kOwn && ndp >= 2) wait_bar(dempty + 8u * (ndp & 1u), (ndp / 2u - 1u) & 1u, L, failed);
    }
    // kOwn: 64 columns from col on of every vector: lane (r, c) copies chunk c (16 bytes) of vectors r, r + 8.  What
    // is not there (vectors past the batch, columns past the row) is left as it is: it meets zero weights, or ends
    // up in accumulator lanes that are never read.
    __device__ __forceinline__ void copy_x(const Q8WLaunch &L, int col, int lane) const {
        const int r = lane & 7, c = col + 16 * (lane >> 3);
        const int8_t *src = x + (size_t)r * cols + c;
        uint32_t dst = xt + (uint32_t)(lane >> 3) * lbo + (uint32_t)r * 16u;
        const int n = c < cols ? L.batch - r : 0;
        if (n > 0) cp_async_16(dst, src);
        if (n > 8) cp_async_16(dst + 128u, src + 8 * (size_t)cols);
    }
    __device__ __forceinline__ void gather_x(const Q8WLaunch &L, int col, int lane) const {
        const int r = lane & 7, c = col + 16 * (lane >> 3);
        uint32_t dst = xt + (uint32_t)(lane >> 3) * lbo + (uint32_t)r * 16u;
        for (int v = r; v < L.batch; v += 8, dst += 128u) {
            const int8_t *src = x + (size_t)v * cols + c;
            uint32_t w[4];
#pragma unroll
            for (int j = 0; j < 4; j++) w[j] = x_quad_at(L, src + 4 * j, cols - c - 4 * j);
            asm volatile("st.shared.v4.u32 [%0], {%1,%2,%3,%4};" ::"r"(dst), "r"(w[0]), "r"(w[1]), "r"(w[2]), "r"(w[3]) : "memory");
        }
    }
    // four quads (16 columns) of the lane's row: piece c of the 64-column tile
    __device__ __forceinline__ void store_w(uint32_t c, uint32_t w0, uint32_t w1, uint32_t w2, uint32_t w3, int lane) const {
        asm volatile("st.shared.v4.u32 [%0], {%1,%2,%3,%4};" ::"r"(wt + c * 512u + (uint32_t)lane * 16u), "r"(w0), "r"(w1),
                     "r"(w2), "r"(w3)
                     : "memory");
    }
    // the previous MMAs are done with the tiles; the x copies have the rest of the decode to land in
    __device__ __forceinline__ void refill_tiles(const Q8WLaunch &L, int col, bool next, int lane, volatile uint32_t *failed) {
        if (nmma) wait_bar(mbar, (nmma - 1) & 1u, L, failed);
        if (kRagged) gather_x(L, col, lane);
        else if (!kTma) copy_x(L, col, lane);
        else xs.refill(L, nmma, col, 64, next, lane, failed);
    }
    // the MMAs of a tile: two K steps of 32 columns, or one
    __device__ __forceinline__ void issue(const Q8WLaunch &L, bool two, int lane, volatile uint32_t *failed) {
        if (!any) wait_acc(L, failed);
        if (!kTma && !kRagged) cp_async_wait_all();
        fence_proxy_async_smem();  // both tiles are read by the tensor core (async proxy)
        tcgen05_fence_before();
        __syncwarp();
        if (elect_one()) {  // (one lane by `lane == 0`: 2 to 6 % slower, MmaCons<false>, FwdCons, BwdCons)
            tcgen05_fence_after();
            const uint32_t idesc = umma_idesc_i8(64, 32);
            const uint32_t d = kOwn ? d_tmem : d_tmem + ((ndp & 1u) << 20);  // the second accumulator: 16 lanes further
            const uint64_t a = kTma ? xs.wait(L, nmma, failed) : a_desc;
            umma_i8(d, a, b_desc, idesc, any ? 1u : 0u);
            if (two) umma_i8(d, a + (kTma ? 2u : lbo >> 3), b_desc + 64u, idesc, 1u);
            umma_commit(mbar);
        }
        __syncwarp();
        any = true;
        nmma++;
    }
    __device__ __forceinline__ void unit(const Q8WLaunch &L, const UnitDesc &d, const unsigned char *sm, uint32_t soff,
                                         uint32_t lw, int lane, volatile uint32_t *failed) {
        const int q0 = d.seg * seg_quads;
        const int nq = min(seg_quads, qtot - q0);
        if (kTma) xs.begin(L, nmma, 4 * q0, lane, failed);
        Stream s(sm, soff, d.rows, lane);
        int q = 0;
        for (; q + 16 <= nq; q += 16) {
#pragma unroll
            for (int c = 0; c < 4; c++) {
                const uint32_t w0 = s.step_i8(sm, lw), w1 = s.step_i8(sm, lw), w2 = s.step_i8(sm, lw), w3 = s.step_i8(sm, lw);
                s.clamp();
                if (c == 0) refill_tiles(L, 4 * (q0 + q), q + 16 < nq, lane, failed);
                store_w((uint32_t)c, w0, w1, w2, w3, lane);
            }
            issue(L, true, lane, failed);
        }
        if (q < nq) {  // the segment's last 4, 8 or 12 quads (segments are whole groups of 4: cols % 16 == 0, or ragged)
            const int n = (nq - q + 3) >> 2;
#pragma unroll 1
            for (int c = 0; c < n; c++) {
                const int left = kRagged ? nq - q - 4 * c : 4;
                const uint32_t w0 = s.step_i8(sm, lw), w1 = left > 1 ? s.step_i8(sm, lw) : 0u,
                               w2 = left > 2 ? s.step_i8(sm, lw) : 0u, w3 = left > 3 ? s.step_i8(sm, lw) : 0u;
                s.clamp();
                if (c == 0) refill_tiles(L, 4 * (q0 + q), false, lane, failed);
                store_w((uint32_t)c, w0, w1, w2, w3, lane);
            }
            if (n & 1) store_w((uint32_t)n, 0u, 0u, 0u, 0u, lane);  // a K step is two pieces
            issue(L, n > 2, lane, failed);
        }
        if (!s.ok()) atomicOr(L.status, MV_DEV_FINAL_STATE);
    }
    // Counts the unit once its MMAs are complete, so that whoever sees the item's last unit counted may read the sums.
    __device__ __forceinline__ void end_unit(const Q8WLaunch &L, int k, bool, unsigned char *sm, const Bars &B, int lane,
                                             volatile uint32_t *failed) {
        if (nmma) wait_bar(mbar, (nmma - 1) & 1u, L, failed);
        if (kOwn && any) {
            tcgen05_fence_after();
            uint32_t r[32];
            tmem_ld_32x32b_x32(d_tmem + (((uint32_t)(warp + kFirstDecode) & 3u) << 21), r);  // lane = vector, r[j] = row j
            if (lane < L.batch) {
                int *red = reinterpret_cast<int *>(sm + L.lay.red) + (size_t)(k % kRing) * kRed + lane * kPitch;
#pragma unroll
                for (int j = 0; j < 32; j++) atomicAdd(red + j, (int)r[j]);
            }
            any = false;
        }
        tcgen05_fence_before();
        __syncwarp();
        if (lane == 0) {
            if (!kOwn && any) {
                ItemState *st = reinterpret_cast<ItemState *>(sm + L.lay.cnt) + k % kRing;
                atomicOr(&st->acc[ndp & 1u], 1u << warp);
            }
            arrive(B.tdone(k % kRing));
        }
        __syncwarp();
    }
    __device__ __forceinline__ void drain(const Q8WLaunch &L) {
        if (!kTma) cp_async_wait_all();
        else xs.drain(L, threadIdx.x & 31);
        if (nmma)
            for (uint32_t it = 0; it < L.spin_limit; it++)
                if (mbar_try_wait(mbar, (nmma - 1) & 1u)) break;
    }
    // Table warps: the sums of item I.  kOwn: from shared memory, one vector per warp at a time, lane = stripe row.
    // Otherwise from the accumulators of the warps that took its units: warp q reads lane quarter q (vectors 16 q ..
    // 16 q + 15, in the lower or upper 16 lanes by accumulator), 32 stripe rows per lane.
    static __device__ __forceinline__ void epilogue(const Q8WLaunch &L, const ItemRec &I, int k, unsigned char *sm,
                                                    const Bars &B, uint32_t tmem) {
        const int q = threadIdx.x >> 5, lane = threadIdx.x & 31;
        if constexpr (kOwn) {
            volatile int *red = reinterpret_cast<volatile int *>(sm + L.lay.red) + (size_t)(k % kRing) * kRed + lane;
            const int row = I.stripe * 32 + lane;
            const float scale = row_scale(I, row);
            for (int v = q; v < L.batch; v += kTableWarps) {
                const int sum = red[v * kPitch];
                red[v * kPitch] = 0;
                if (row < I.rows) emit(I, v, row, sum, scale);
            }
        } else {
            tcgen05_fence_after();
            ItemState *st = reinterpret_cast<ItemState *>(sm + L.lay.cnt) + k % kRing;
            const uint32_t m0 = *reinterpret_cast<volatile uint32_t *>(&st->acc[0]);
            const uint32_t m1 = *reinterpret_cast<volatile uint32_t *>(&st->acc[1]);
            const bool active = 16 * q < L.batch;
            if (active) {
#pragma unroll 1
                for (int h = 0; h < 32; h += 16) {  // 16 stripe rows at a time (registers)
                    int sum[16];
#pragma unroll
                    for (int j = 0; j < 16; j++) sum[j] = 0;
                    for (uint32_t left = m0 | m1; left; left &= left - 1u) {
                        const int w = __ffs((int)left) - 1;
                        uint32_t r[16];
                        tmem_ld_32x32b_x16(tmem + 32u * (uint32_t)w + (uint32_t)h + (((uint32_t)q * 32u) << 16), r);
                        const bool mine = (lane < 16 ? m0 : m1) >> w & 1u;  // the accumulator's half of the quarter's lanes
#pragma unroll
                        for (int j = 0; j < 16; j++) sum[j] += mine ? (int)r[j] : 0;
                    }
                    uint32_t base = 0;
                    if (!m0) base = 16;  // every warp was at its second accumulator
                    else if (m1)         // some at the first, some at the second: lane l + 16 to lane l
#pragma unroll
                        for (int j = 0; j < 16; j++) sum[j] += __shfl_down_sync(0xffffffffu, sum[j], 16);
                    const int v = 16 * q + lane - (int)base, row0 = I.stripe * 32 + h;
                    if ((uint32_t)lane >= base && (uint32_t)lane < base + 16u && v < L.batch) {
                        float sc[16];
#pragma unroll
                        for (int j = 0; j < 16; j++) sc[j] = row_scale(I, row0 + j);
                        if (!I.atomic && row0 + 16 <= I.rows && (I.rows & 3) == 0 && (((uintptr_t)I.y | (uintptr_t)I.ys) & 15) == 0) {
                            int4 *dst = reinterpret_cast<int4 *>(I.y + (size_t)v * I.rows + row0);
#pragma unroll
                            for (int j = 0; j < 4; j++)
                                dst[j] = make_int4(sum[4 * j], sum[4 * j + 1], sum[4 * j + 2], sum[4 * j + 3]);
                            if (I.ys) {
                                float4 *ds = reinterpret_cast<float4 *>(I.ys + (size_t)v * I.rows + row0);
#pragma unroll
                                for (int j = 0; j < 4; j++)
                                    ds[j] = make_float4((float)sum[4 * j] * sc[4 * j], (float)sum[4 * j + 1] * sc[4 * j + 1],
                                                        (float)sum[4 * j + 2] * sc[4 * j + 2], (float)sum[4 * j + 3] * sc[4 * j + 3]);
                            }
                        } else {
#pragma unroll
                            for (int j = 0; j < 16; j++)
                                if (row0 + j < I.rows) emit(I, v, row0 + j, sum[j], sc[j]);
                        }
                    }
                }
                tcgen05_fence_before();
            }
            __syncwarp();
            if (lane == 0)
                for (uint32_t left = m0 | m1; left; left &= left - 1u) {
                    const int w = __ffs((int)left) - 1;
                    arrive(B.dempty(w, (int)(m1 >> w & 1u)));
                }
            table_vote(true);  // every warp has read the masks
            if (threadIdx.x == 0) st->acc[0] = st->acc[1] = 0;
        }
    }
};

// Float forward on the tensor cores, up to 64 bf16 vectors: as MmaCons<false> with kind::f16, bf16 W and x (int8
// weights are exact in bf16, every product is exact in fp32) and fp32 sums, 8 quads (32 columns, two K steps of 16) at
// a time: W tile 2 KB, x tiles (XTiles) 64 bytes per vector.  Unit u goes to warp u mod W, each warp's MMAs accumulate in order
// and the warps' sums are added in unit order, so results are reproducible bit for bit.
struct FwdCons {
    static constexpr bool kMma = true, kFloat = true, kStatic = true, kPrepare = false;
    static constexpr int kRed = 0, kAreas = 0;
    static constexpr int kLag = 2;  // accumulators
    static constexpr int kMaxDecode = 16;
    static constexpr uint32_t kWTile = 2048;
    static constexpr uint32_t tile_bytes(int xrows) { return kWTile + XTiles::bytes(xrows); }
    int seg_quads, qtot;
    XTiles xs;
    uint32_t wt, d_tmem, nmma, ndp;
    uint32_t mbar, dempty;
    uint64_t b_desc;
    int warp;
    bool any;
    __device__ __forceinline__ void init(const Q8WLaunch &L, unsigned char *sm, const Bars &B, uint32_t tmem, int w) {
        warp = w;
        wt = smem_u32(sm) + L.lay.tiles + (uint32_t)w * tile_bytes(L.xrows);
        xs.init(B, w, wt + kWTile);
        d_tmem = tmem + 32u * (uint32_t)w;
        b_desc = umma_smem_desc(wt, 512u, 128u);
        mbar = B.mma(w);
        dempty = B.dempty(w, 0);
        nmma = ndp = 0;
        any = false;
    }
    __device__ __forceinline__ void begin_item(const Q8WLaunch &, const ItemRec &I, int) {
        seg_quads = I.seg_quads;
        qtot = I.cols >> 2;
    }
    __device__ __forceinline__ void wait_acc(const Q8WLaunch &L, volatile uint32_t *failed) const {
        if (ndp >= 2) wait_bar(dempty + 8u * (ndp & 1u), (ndp / 2u - 1u) & 1u, L, failed);
    }
    // the previous MMAs are done with the tiles (x columns past the segment are never multiplied)
    __device__ __forceinline__ void refill_tiles(const Q8WLaunch &L, int col, bool next, int lane, volatile uint32_t *failed) {
        if (nmma) wait_bar(mbar, (nmma - 1) & 1u, L, failed);
        xs.refill(L, nmma, col, 32, next, lane, failed);
    }
    __device__ __forceinline__ void issue(const Q8WLaunch &L, bool two, int lane, volatile uint32_t *failed) {
        if (!any) wait_acc(L, failed);
        fence_proxy_async_smem();
        tcgen05_fence_before();
        __syncwarp();
        if (elect_one()) {
            tcgen05_fence_after();
            const uint32_t idesc = umma_idesc_bf16(64, 32, 0, 0);
            const uint32_t d = d_tmem + ((ndp & 1u) << 20);
            const uint64_t a = xs.wait(L, nmma, failed);
            umma_f16_ss(d, a, b_desc, idesc, any ? 1u : 0u);
            if (two) umma_f16_ss(d, a + 2u, b_desc + 64u, idesc, 1u);
            umma_commit(mbar);
        }
        __syncwarp();
        any = true;
        nmma++;
    }
    // two quads (8 columns) of the lane's row: piece c of the 32-column tile
    __device__ __forceinline__ void two_quads(Stream &s, const unsigned char *sm, uint32_t lw, uint32_t (&w)[4]) const {
        s.step_bf16(sm, lw, w[0], w[1]);
        s.step_bf16(sm, lw, w[2], w[3]);
    }
    __device__ __forceinline__ void store_w(uint32_t c, const uint32_t (&w)[4], int lane) const {
        asm volatile("st.shared.v4.u32 [%0], {%1,%2,%3,%4};" ::"r"(wt + c * 512u + (uint32_t)lane * 16u), "r"(w[0]),
                     "r"(w[1]), "r"(w[2]), "r"(w[3])
                     : "memory");
    }
    __device__ __forceinline__ void unit(const Q8WLaunch &L, const UnitDesc &d, const unsigned char *sm, uint32_t soff,
                                         uint32_t lw, int lane, volatile uint32_t *failed) {
        const int q0 = d.seg * seg_quads;
        const int nq = min(seg_quads, qtot - q0);
        xs.begin(L, nmma, 4 * q0, lane, failed);
        Stream s(sm, soff, d.rows, lane);
        uint32_t w[4];
        int q = 0;
        for (; q + 8 <= nq; q += 8) {
#pragma unroll
            for (int c = 0; c < 4; c++) {
                two_quads(s, sm, lw, w);
                if (c == 0) refill_tiles(L, 4 * (q0 + q), q + 8 < nq, lane, failed);
                store_w((uint32_t)c, w, lane);
                if (c & 1) s.clamp();
            }
            issue(L, true, lane, failed);
        }
        if (q < nq) {  // the segment's last 4 quads (segments are whole groups of 4: cols % 16 == 0)
            two_quads(s, sm, lw, w);
            refill_tiles(L, 4 * (q0 + q), false, lane, failed);
            store_w(0, w, lane);
            two_quads(s, sm, lw, w);
            store_w(1, w, lane);
            issue(L, false, lane, failed);
        }
        if (!s.ok()) atomicOr(L.status, MV_DEV_FINAL_STATE);
    }
    __device__ __forceinline__ void end_unit(const Q8WLaunch &L, int k, bool last, unsigned char *sm, const Bars &B,
                                             int lane, volatile uint32_t *failed) {
        if (nmma) wait_bar(mbar, (nmma - 1) & 1u, L, failed);
        tcgen05_fence_before();
        __syncwarp();
        if (lane == 0) {
            ItemState *st = reinterpret_cast<ItemState *>(sm + L.lay.cnt) + k % kRing;
            if (any) atomicOr(&st->acc[ndp & 1u], 1u << warp);
            arrive(B.tdone(k % kRing));
        }
        __syncwarp();
        if (last) {  // the sums stay where they are until the table warps have read them
            if (any) ndp++;
            any = false;
        }
    }
    __device__ __forceinline__ void drain(const Q8WLaunch &L) {
        xs.drain(L, threadIdx.x & 31);
        if (nmma)
            for (uint32_t it = 0; it < L.spin_limit; it++)
                if (mbar_try_wait(mbar, (nmma - 1) & 1u)) break;
    }
    // Table warps: y = s . sums, the warps' sums added in the order of their first units.
    static __device__ __forceinline__ void epilogue(const Q8WLaunch &L, const ItemRec &I, int k, unsigned char *sm,
                                                    const Bars &B, uint32_t tmem) {
        const int q = threadIdx.x >> 5, lane = threadIdx.x & 31;
        tcgen05_fence_after();
        ItemState *st = reinterpret_cast<ItemState *>(sm + L.lay.cnt) + k % kRing;
        const uint32_t m0 = *reinterpret_cast<volatile uint32_t *>(&st->acc[0]);
        const uint32_t m1 = *reinterpret_cast<volatile uint32_t *>(&st->acc[1]);
        const bool active = 16 * q < L.batch;
        const uint32_t W = (uint32_t)L.W, nc = min(I.n, W), first = I.u0 % W;
        const int v = 16 * q + lane;
        if (active) {
#pragma unroll 1
            for (int h = 0; h < 32; h += 16) {  // 16 stripe rows at a time (registers)
                float sum[16];
#pragma unroll
                for (int j = 0; j < 16; j++) sum[j] = 0.f;
                uint32_t w = first;
                for (uint32_t i = 0; i < nc; i++, w = w + 1 < W ? w + 1 : 0) {
                    if (!((m0 | m1) >> w & 1u)) continue;
                    uint32_t r[16];
                    tmem_ld_32x32b_x16(tmem + 32u * w + (uint32_t)h + (((uint32_t)q * 32u) << 16), r);
                    if (m1 >> w & 1u) {  // the second accumulator's sums are 16 lanes further
#pragma unroll
                        for (int j = 0; j < 16; j++) r[j] = __shfl_down_sync(0xffffffffu, r[j], 16);
                    }
#pragma unroll
                    for (int j = 0; j < 16; j++) sum[j] += __uint_as_float(r[j]);
                }
                const int row0 = I.stripe * 32 + h;
                if (lane < 16 && v < L.batch) {
                    float *dst = I.ys + (size_t)v * I.rows + row0;
                    float sc[16];
#pragma unroll
                    for (int j = 0; j < 16; j++) sc[j] = row_scale(I, row0 + j);
                    if (I.atomic) {  // even shares: the other CTA's part is added, and scaled with it afterwards
#pragma unroll
                        for (int j = 0; j < 16; j++)
                            if (row0 + j < I.rows) atomicAdd(dst + j, sum[j]);
                    } else if (row0 + 16 <= I.rows && (I.rows & 3) == 0 && ((uintptr_t)I.ys & 15) == 0) {
#pragma unroll
                        for (int j = 0; j < 16; j += 4)
                            *reinterpret_cast<float4 *>(dst + j) = make_float4(
                                sum[j] * sc[j], sum[j + 1] * sc[j + 1], sum[j + 2] * sc[j + 2], sum[j + 3] * sc[j + 3]);
                    } else {
#pragma unroll
                        for (int j = 0; j < 16; j++)
                            if (row0 + j < I.rows) dst[j] = sum[j] * sc[j];
                    }
                }
            }
            tcgen05_fence_before();
        }
        __syncwarp();
        if (lane == 0)
            for (uint32_t left = m0 | m1; left; left &= left - 1u) {
                const int w = __ffs((int)left) - 1;
                arrive(B.dempty(w, (int)(m1 >> w & 1u)));
            }
        table_vote(true);  // every warp has read the masks
        if (threadIdx.x == 0) st->acc[0] = st->acc[1] = 0;
    }
};

// Float forward on the CUDA cores, one bf16 vector, or (engine 1) up to 8 of them: fp32 multiply-adds of the table's bf16
// symbols, x behind the block in the slot (or from global memory when the segment is longer than kXQuads).  Unit u goes to
// warp u mod W, each warp adds its units of an item in order, and the warps' sums are added in the order of their first
// units: reproducible bit for bit, and for each vector what it is alone.  Measured on a B200, 1, 2, 4 and 8 vectors:
// 11008x4096 28, 33, 43 and 60 us; 4096x11008 26, 29, 41 and 63 (one vector through the MMAs of FwdCons, whose tiles cost
// more than its products: 40).
template <int NV>
struct FwdDot {
    static constexpr bool kMma = false, kFloat = true, kStatic = true, kPrepare = false;
    static constexpr int kLag = 1;
    static constexpr int kMaxDecode = NV <= 4 ? 16 : 12;  // (registers, and the slots' x)
    static constexpr int kRed = kMaxDecode * NV * 32;
    static constexpr int kAreas = 2;  // (with kLag 1 two items are open)
    static constexpr uint32_t tile_bytes(int) { return 0; }
    const uint16_t *x;
    int cols, seg_quads, qtot, warp;
    bool in_slot;
    float acc[NV];
    __device__ __forceinline__ void init(const Q8WLaunch &, unsigned char *, const Bars &, uint32_t, int w) {
        warp = w;
#pragma unroll
        for (int v = 0; v < NV; v++) acc[v] = 0.f;
    }
    __device__ __forceinline__ void begin_item(const Q8WLaunch &L, const ItemRec &I, int) {
        in_slot = x_in_slot(L, I.seg_quads);
        x = reinterpret_cast<const uint16_t *>(I.x);
        cols = I.cols;
        seg_quads = I.seg_quads;
        qtot = cols >> 2;
    }
    // one quad of one vector: x as two bf16 pairs
    static __device__ __forceinline__ void fma4(float &a, const uint32_t (&e)[4], uint32_t x01, uint32_t x23) {
        a = fmaf(__uint_as_float(e[0] & 0xFFFF0000u), __uint_as_float(x01 << 16), a);
        a = fmaf(__uint_as_float(e[1] & 0xFFFF0000u), __uint_as_float(x01 & 0xFFFF0000u), a);
        a = fmaf(__uint_as_float(e[2] & 0xFFFF0000u), __uint_as_float(x23 << 16), a);
        a = fmaf(__uint_as_float(e[3] & 0xFFFF0000u), __uint_as_float(x23 & 0xFFFF0000u), a);
    }
    // two quads of every vector
    __device__ __forceinline__ void pair(Stream &s, const unsigned char *sm, uint32_t lw, const uint4 (&xv)[NV]) {
        uint32_t e[4];
        s.step_f(sm, lw, e);
#pragma unroll
        for (int v = 0; v < NV; v++) fma4(acc[v], e, xv[v].x, xv[v].y);
        s.step_f(sm, lw, e);
#pragma unroll
        for (int v = 0; v < NV; v++) fma4(acc[v], e, xv[v].z, xv[v].w);
    }
    // eight columns of every vector at p (past the batch: its last vector again)
    __device__ __forceinline__ void load_x(const uint16_t *p, int batch, uint4 (&xv)[NV]) const {
#pragma unroll
        for (int v = 0; v < NV; v++) {
            xv[v] = ldx_u4(p);
            if (NV <= 2 || v + 1 < batch) p += cols;
        }
    }
    __device__ __forceinline__ void unit(const Q8WLaunch &L, const UnitDesc &d, const unsigned char *sm, uint32_t soff,
                                         uint32_t lw, int lane, volatile uint32_t *) {
        const int q0 = d.seg * seg_quads;
        const int nq = min(seg_quads, qtot - q0);
        Stream s(sm, soff, d.rows, lane);
        if (in_slot) {
            const unsigned char *xs = sm + soff + L.x_off;
            constexpr int kUnroll = NV == 1 ? 2 : 1;
#pragma unroll kUnroll
            for (int i = 0; i < nq; i += 4, xs += 32) {
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    uint4 xv[NV];
#pragma unroll
                    for (int v = 0; v < NV; v++) xv[v] = *reinterpret_cast<const uint4 *>(xs + 8 * v * seg_quads + 16 * h);
                    pair(s, sm, lw, xv);
                }
                s.clamp();
            }
        } else {
            const uint16_t *xp = x + 4 * q0;
            uint4 xn[NV];
            load_x(xp, L.batch, xn);
            for (int i = 0; i < nq; i += 2) {
                uint4 xv[NV];
#pragma unroll
                for (int v = 0; v < NV; v++) xv[v] = xn[v];
                xp += i + 2 < nq ? 8 : 0;
                load_x(xp, L.batch, xn);
                pair(s, sm, lw, xv);
                if (i & 2) s.clamp();
            }
        }
        if (!s.ok()) atomicOr(L.status, MV_DEV_FINAL_STATE);
    }
    __device__ __forceinline__ void end_unit(const Q8WLaunch &L, int k, bool last, unsigned char *sm, const Bars &B,
                                             int lane, volatile uint32_t *) {
        if (last) {
            float *red = reinterpret_cast<float *>(sm + L.lay.red) + (k % kAreas) * kRed + warp * NV * 32 + lane;
#pragma unroll
            for (int v = 0; v < NV; v++) {
                red[v * 32] = acc[v];
                acc[v] = 0.f;
            }
        }
        __syncwarp();
        if (lane == 0) arrive(B.tdone(k % kRing));
    }
    __device__ __forceinline__ void drain(const Q8WLaunch &) {}
    // Table warps: one vector per warp at a time, lane = stripe row.
    static __device__ __forceinline__ void epilogue(const Q8WLaunch &L, const ItemRec &I, int k, unsigned char *sm,
                                                    const Bars &, uint32_t) {
        const int lane = threadIdx.x & 31, row = I.stripe * 32 + lane;
        const float scale = row_scale(I, row);
        const uint32_t W = (uint32_t)L.W, nc = min(I.n, W), first = I.u0 % W;
        for (int v = threadIdx.x >> 5; v < min(NV, L.batch); v += kTableWarps) {
            const volatile float *red = reinterpret_cast<const volatile float *>(sm + L.lay.red) + (k % kAreas) * kRed + v * 32 + lane;
            uint32_t w = first;
            float sum = 0.f;
            for (uint32_t i = 0; i < nc; i++, w = w + 1 < W ? w + 1 : 0) sum += red[w * NV * 32];
            if (row >= I.rows) continue;
            float *dst = I.ys + (size_t)v * I.rows + row;
            if (I.atomic) atomicAdd(dst, sum);  // even shares: scaled together with the other CTA's part afterwards
            else *dst = sum * scale;
        }
    }
};

// Float backward on the tensor cores: dX = W^T (s . dY), up to 32 bf16 vectors a pass, added to dX (fp32, zeroed by the
// launcher) with 16-byte reductions.
//   A = G = s . dY of the stripe's 32 rows (K), in TMEM: the table warps write it with the item's decode table, vector v
//       in lane v of every quarter, as bf16 terms hi + lo (g to 2^-17);
//   B = W: 8 quads at a time, each lane storing its row's four 16-byte pieces (the tile is W^T's transpose as it
//       stands: MN-major, N = 32 columns, K = 32 rows);
//   D: 32 TMEM columns per decode warp, vector v in lane v of the warp's own quarter.
// The sums of a tile are read while the next one decodes.  From 5 vectors on they pass through shared memory so that
// eight lanes cover the 128 bytes of a vector's row: reductions from one lane per vector ran at 2.6 TB/s, these at 5.4,
// and they bound the larger batches (4 bytes per vector, column and stripe).
// Measured on a B200 against the form this replaced (the same passes, terms and MMAs in a CTA with barriers between its
// items): 11008x4096, 64 vectors 219 -> 120 us, 16 vectors 87 -> 52 us, 2 vectors 75 -> 45 us; 4096x11008, 64 vectors
// 251 -> 120 us, 16 vectors 104 -> 52 us.
struct BwdCons {
    static constexpr bool kMma = true, kFloat = true, kStatic = false, kPrepare = true;
    static constexpr int kRed = 0, kAreas = 0;
    static constexpr int kLag = 1;  // two buffers of G, written with the item's table
    static constexpr int kMaxDecode = 12;
    static constexpr uint32_t kWTile = 2048, kTr = 4096;
    static constexpr uint32_t kGCols = 32;  // TMEM columns of an item's G: two terms of two K steps
    static constexpr uint32_t tile_bytes(int) { return kWTile + kTr; }
    float *dx;
    int cols, seg_quads, qtot, batch;
    uint32_t wt, tr, d_tmem, g_tmem, g_base, nmma, mbar, quarter;
    int pend_col, pend_n;  // the tile whose sums are still in D: first column, columns
    __device__ __forceinline__ void init(const Q8WLaunch &L, unsigned char *sm, const Bars &B, uint32_t tmem, int w) {
        wt = smem_u32(sm) + L.lay.tiles + (uint32_t)w * tile_bytes(0);
        tr = wt + kWTile;
        quarter = ((uint32_t)(w + kFirstDecode) & 3u) << 21;
        g_base = tmem;
        d_tmem = tmem + 2u * kGCols + 32u * (uint32_t)w;
        mbar = B.mma(w);
        nmma = 0;
        batch = L.batch;
        pend_n = 0;
    }
    __device__ __forceinline__ void begin_item(const Q8WLaunch &, const ItemRec &I, int k) {
        dx = I.ys;
        cols = I.cols;
        seg_quads = I.seg_quads;
        qtot = cols >> 2;
        g_tmem = g_base + (uint32_t)(k & 1) * kGCols;
        tcgen05_fence_after();  // G was written by the table warps
    }
    // Table warps: G of item k (into one of two buffers: the item before the previous one is finished).
    static __device__ __forceinline__ void prepare(const Q8WLaunch &L, const ItemRec &I, int k, unsigned char *, uint32_t tmem) {
        const int q = threadIdx.x >> 5, v = threadIdx.x & 31, row0 = I.stripe * 32;
        const uint16_t *dy = reinterpret_cast<const uint16_t *>(I.x) + (size_t)v * I.rows + row0;
        const float sl = row0 + v < I.rows ? ldp(I.scales + row0 + v) : 0.f;  // lane = row
        float g[32];
        if (v < L.batch && row0 + 32 <= I.rows && ((uintptr_t)dy & 15) == 0) {
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const uint4 d = ldp(reinterpret_cast<const uint4 *>(dy) + j);
                const uint32_t w[4] = {d.x, d.y, d.z, d.w};
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    g[8 * j + 2 * i] = __uint_as_float(w[i] << 16);
                    g[8 * j + 2 * i + 1] = __uint_as_float(w[i] & 0xFFFF0000u);
                }
            }
        } else {
#pragma unroll
            for (int j = 0; j < 32; j++)
                g[j] = v < L.batch && row0 + j < I.rows ? __uint_as_float((uint32_t)ldp(dy + j) << 16) : 0.f;
        }
#pragma unroll
        for (int j = 0; j < 32; j++) g[j] *= __shfl_sync(0xffffffffu, sl, j);
        const uint32_t dst = tmem + (uint32_t)(k & 1) * kGCols + ((uint32_t)q << 21);
#pragma unroll
        for (int t = 0; t < 2; t++) {
            uint32_t r[16];
#pragma unroll
            for (int j = 0; j < 32; j += 2) {
                uint32_t h[2];
#pragma unroll
                for (int i = 0; i < 2; i++) {
                    // term t, and what it leaves (nothing of an infinity or NaN)
                    const float x = g[j + i];
                    h[i] = (uint32_t)__bfloat16_as_ushort(__float2bfloat16_rn(x));
                    g[j + i] = isfinite(x) ? x - __uint_as_float(h[i] << 16) : 0.f;
                }
                r[j >> 1] = h[0] | h[1] << 16;
            }
            tmem_st_32x32b_x16_nowait(dst + 16u * (uint32_t)t, r);
        }
        tmem_wait_st();
        tcgen05_fence_before();
    }
    // the sums of the pending tile, added to dX
    __device__ __forceinline__ void flush(const Q8WLaunch &L, int lane, volatile uint32_t *failed) {
        if (nmma) wait_bar(mbar, (nmma - 1) & 1u, L, failed);
        if (!pend_n) return;
        tcgen05_fence_after();
        uint32_t r[32];
        tmem_ld_32x32b_x32(d_tmem + quarter, r);  // lane = vector, r[j] = column pend_col + j
        tcgen05_fence_before();
        if (batch <= 4) {
            float *dst = dx + (size_t)lane * cols + pend_col;
            if (lane < batch) {
#pragma unroll
                for (int j = 0; j < 32; j += 4)
                    if (j < pend_n) red4(dst + j, r[j], r[j + 1], r[j + 2], r[j + 3]);
            }
        } else {
            // piece j of vector v at 16 (j ^ v % 8): conflict-free both ways
#pragma unroll
            for (int j = 0; j < 8; j++)
                asm volatile("st.shared.v4.u32 [%0], {%1,%2,%3,%4};" ::"r"(tr + 128u * (uint32_t)lane +
                                                                           16u * (uint32_t)(j ^ (lane & 7))),
                             "r"(r[4 * j]), "r"(r[4 * j + 1]), "r"(r[4 * j + 2]), "r"(r[4 * j + 3])
                             : "memory");
            __syncwarp();
            const int c = 4 * (lane & 7);
            float *dst = dx + (size_t)(lane >> 3) * cols + pend_col + c;
            uint32_t src = tr + 128u * (uint32_t)(lane >> 3);
            for (int v = lane >> 3; v < batch; v += 4) {
                uint32_t a0, a1, a2, a3;
                asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];"
                             : "=r"(a0), "=r"(a1), "=r"(a2), "=r"(a3)
                             : "r"(src + 16u * (uint32_t)((lane & 7) ^ (v & 7)))
                             : "memory");
                if (c < pend_n) red4(dst, a0, a1, a2, a3);
                dst += 4 * (size_t)cols;
                src += 512u;
            }
            __syncwarp();
        }
        pend_n = 0;
    }
    static __device__ __forceinline__ void red4(float *p, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
        asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(p), "f"(__uint_as_float(a)),
                     "f"(__uint_as_float(b)), "f"(__uint_as_float(c)), "f"(__uint_as_float(d))
                     : "memory");
    }
    __device__ __forceinline__ void unit(const Q8WLaunch &L, const UnitDesc &d, const unsigned char *sm, uint32_t soff,
                                         uint32_t lw, int lane, volatile uint32_t *failed) {
        const int q0 = d.seg * seg_quads;
        const int nq = min(seg_quads, qtot - q0);
        Stream s(sm, soff, d.rows, lane);
        // lane = stripe row r: K step r / 16, K group (r / 8) % 2, row r % 8; N group c (8 columns) at 256 c
        const uint32_t wdst = wt + (uint32_t)(lane >> 4) * 1024u + (uint32_t)((lane >> 3) & 1) * 128u + (uint32_t)(lane & 7) * 16u;
#pragma unroll 1
        for (int q = 0; q < nq; q += 8) {
            const int n = min(4, (nq - q) >> 1);  // pieces of two quads (segments are whole groups of 4 quads)
#pragma unroll
            for (int c = 0; c < 4; c++) {
                if (c < n) {
                    uint32_t w[4];
                    s.step_bf16(sm, lw, w[0], w[1]);
                    s.step_bf16(sm, lw, w[2], w[3]);
                    if (c & 1) s.clamp();
                    if (c == 0) flush(L, lane, failed);  // (the W tile is free, too)
                    asm volatile("st.shared.v4.u32 [%0], {%1,%2,%3,%4};" ::"r"(wdst + 256u * c), "r"(w[0]), "r"(w[1]),
                                 "r"(w[2]), "r"(w[3])
                                 : "memory");
                }
            }
            fence_proxy_async_smem();
            tcgen05_fence_before();
            __syncwarp();
            if (elect_one()) {
                tcgen05_fence_after();
                const uint32_t idesc = umma_idesc_bf16(128, 32, 0, 1);
#pragma unroll
                for (int t = 0; t < 2; t++)
#pragma unroll
                    for (int kk = 0; kk < 2; kk++)
                        umma_f16_ts(d_tmem, g_tmem + 16u * (uint32_t)t + 8u * kk, umma_smem_desc(wt + 1024u * kk, 128u, 256u),
                                    idesc, t || kk ? 1u : 0u);
                umma_commit(mbar);
            }
            __syncwarp();
            nmma++;
            pend_col = 4 * (q0 + q);
            pend_n = 8 * n;
        }
        if (!s.ok()) atomicOr(L.status, MV_DEV_FINAL_STATE);
    }
    __device__ __forceinline__ void end_unit(const Q8WLaunch &L, int k, bool, unsigned char *, const Bars &B, int lane,
                                             volatile uint32_t *failed) {
        flush(L, lane, failed);
        __syncwarp();
        if (lane == 0) arrive(B.tdone(k % kRing));
    }
    __device__ __forceinline__ void drain(const Q8WLaunch &L) {
        if (nmma)
            for (uint32_t it = 0; it < L.spin_limit; it++)
                if (mbar_try_wait(mbar, (nmma - 1) & 1u)) break;
    }
    static __device__ __forceinline__ void epilogue(const Q8WLaunch &, const ItemRec &, int, unsigned char *, const Bars &,
                                                    uint32_t) {}
};

// Float backward on the CUDA cores, one vector, or (engine 1) up to 8 of them: fp32 products of the table's bf16 symbols
// with the row's g = s . dy (the tensor cores' sums of 32 rows are less exact than fp32 additions).  The products of 4 quads
// (16 columns) of the 32 rows change hands in shared memory, a vector at a time: a lane stores its row's four 16-byte pieces
// and reads one piece of four rows, which leaves eight partial sums a column for three shuffle steps.  (All sixteen columns
// by shuffles alone: 30 selects and 16 shuffles a group against 6 and 4.)  Bound by issue.  Measured on a B200, one vector,
// by shuffles between barriers and now: 4096x11008 47 -> 37 us, 11008x4096 50 -> 41 us (with BwdCons, 45 us and 2e-6 of
// error where this form has 2e-7); 8 vectors 141 and 150 us.
template <int NV>
struct BwdDot {
    static constexpr bool kMma = false, kFloat = true, kStatic = false, kPrepare = true;
    static constexpr int kLag = 1;
    static constexpr int kMaxDecode = 16;
    static constexpr int kRed = NV * 32;  // g of the item's rows
    static constexpr int kAreas = kRing;
    static constexpr uint32_t tile_bytes(int) { return 2048; }
    const float *gs;
    float *dx;
    float g[NV];
    int cols, seg_quads, qtot;
    uint32_t st, ld;  // this lane's row, and its piece of rows lane / 4, + 8, + 16, + 24
    __device__ __forceinline__ void init(const Q8WLaunch &L, unsigned char *sm, const Bars &, uint32_t, int w) {
        const uint32_t lane = threadIdx.x & 31u, t = smem_u32(sm) + L.lay.tiles + (uint32_t)w * tile_bytes(0);
        gs = reinterpret_cast<const float *>(sm + L.lay.red) + lane;
        // piece j of row r at 64 r + 16 (j ^ r / 2 % 4): conflict-free both ways
        st = t + 64u * lane + 16u * ((lane >> 1) & 3u);
        ld = t + 64u * (lane >> 2) + 16u * ((lane & 3u) ^ ((lane >> 3) & 3u));
    }
    __device__ __forceinline__ void begin_item(const Q8WLaunch &, const ItemRec &I, int k) {
        dx = I.ys;
        cols = I.cols;
        seg_quads = I.seg_quads;
        qtot = I.cols >> 2;
#pragma unroll
        for (int v = 0; v < NV; v++) g[v] = *reinterpret_cast<const volatile float *>(gs + (k % kAreas) * kRed + v * 32);
    }
    static __device__ __forceinline__ void prepare(const Q8WLaunch &L, const ItemRec &I, int k, unsigned char *sm, uint32_t) {
        const int lane = threadIdx.x & 31, row = I.stripe * 32 + lane;
        const float scale = row_scale(I, row);
        for (int v = threadIdx.x >> 5; v < NV; v += kTableWarps) {
            float gv = 0.f;
            if (row < I.rows && v < L.batch)
                gv = scale * __uint_as_float((uint32_t)ldp(reinterpret_cast<const uint16_t *>(I.x) + (size_t)v * I.rows + row) << 16);
            reinterpret_cast<float *>(sm + L.lay.red)[(k % kAreas) * kRed + v * 32 + lane] = gv;
        }
    }
    // the lane's products of quad j with its row's g
    __device__ __forceinline__ void store4(uint32_t j, const uint32_t (&e)[4], float gv) const {
        asm volatile("st.shared.v4.f32 [%0], {%1,%2,%3,%4};" ::"r"(st ^ (16u * j)), "f"(__uint_as_float(e[0] & 0xFFFF0000u) * gv),
                     "f"(__uint_as_float(e[1] & 0xFFFF0000u) * gv), "f"(__uint_as_float(e[2] & 0xFFFF0000u) * gv),
                     "f"(__uint_as_float(e[3] & 0xFFFF0000u) * gv)
                     : "memory");
    }
    // the 32 rows' products of 16 columns, summed and added to dst (which is this lane's column)
    __device__ __forceinline__ void reduce(float *dst, int lane) const {
        const bool b4 = lane & 16, b3 = lane & 8;
        __syncwarp();
        float a[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (uint32_t r = 0; r < 4; r++) {
            float v[4];
            asm volatile("ld.shared.v4.f32 {%0,%1,%2,%3}, [%4];"
                         : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3])
                         : "r"(ld + 512u * r)
                         : "memory");
#pragma unroll
            for (int c = 0; c < 4; c++) a[c] += v[c];
        }
        __syncwarp();
        float k0 = b4 ? a[2] : a[0], k1 = b4 ? a[3] : a[1];
        k0 += __shfl_xor_sync(0xffffffffu, b4 ? a[0] : a[2], 16);
        k1 += __shfl_xor_sync(0xffffffffu, b4 ? a[1] : a[3], 16);
        float c = b3 ? k1 : k0;
        c += __shfl_xor_sync(0xffffffffu, b3 ? k0 : k1, 8);
        c += __shfl_xor_sync(0xffffffffu, c, 4);
        if (!(lane & 4)) atomicAdd(dst, c);
    }
    __device__ __forceinline__ void unit(const Q8WLaunch &L, const UnitDesc &d, const unsigned char *sm, uint32_t soff,
                                         uint32_t lw, int lane, volatile uint32_t *) {
        const int q0 = d.seg * seg_quads;
        const int nq = min(seg_quads, qtot - q0);
        Stream s(sm, soff, d.rows, lane);
        float *dst = dx + 4 * q0 + 4 * (lane & 3) + (lane & 16 ? 2 : 0) + (lane & 8 ? 1 : 0);
        for (int i = 0; i < nq; i += 4, dst += 16) {  // segments are whole groups of 4 quads (cols % 16 == 0)
            if constexpr (NV == 1) {
#pragma unroll
                for (uint32_t j = 0; j < 4; j++) {
                    uint32_t e[4];
                    s.step_f(sm, lw, e);
                    store4(j, e, g[0]);
                }
                s.clamp();
                reduce(dst, lane);
            } else {
                uint32_t e[4][4];
#pragma unroll
                for (int j = 0; j < 4; j++) s.step_f(sm, lw, e[j]);
                s.clamp();
#pragma unroll
                for (int v = 0; v < NV; v++)
                    if (v < L.batch) {
#pragma unroll
                        for (uint32_t j = 0; j < 4; j++) store4(j, e[j], g[v]);
                        reduce(dst + (size_t)v * cols, lane);
                    }
            }
        }
        if (!s.ok()) atomicOr(L.status, MV_DEV_FINAL_STATE);
    }
    __device__ __forceinline__ void end_unit(const Q8WLaunch &L, int k, bool, unsigned char *, const Bars &B, int lane,
                                             volatile uint32_t *) {
        __syncwarp();
        if (lane == 0) arrive(B.tdone(k % kRing));
    }
    __device__ __forceinline__ void drain(const Q8WLaunch &) {}
    static __device__ __forceinline__ void epilogue(const Q8WLaunch &, const ItemRec &, int, unsigned char *, const Bars &,
                                                    uint32_t) {}
};

// An item's outputs, once all its units are decoded (table warps).
template <class Cons>
__device__ __forceinline__ bool finish_item(const Q8WLaunch &L, const ItemRec &I, int k, unsigned char *sm, const Bars &B,
                                            uint32_t tmem, volatile uint32_t *failed) {
    // one warp polls, the others wait at the barrier (no issue slots taken from the decode warps)
    if (!table_vote(threadIdx.x >= 32 || wait_bar(B.tdone(k % kRing), (uint32_t)(k / kRing) & 1u, L, failed))) return false;
    Cons::epilogue(L, I, k, sm, B, tmem);
    table_vote(true);
    if (threadIdx.x == 0) {
        if (L.chain_scales) {
            __threadfence();  // this item's outputs are visible before it is counted
            atomicAdd(const_cast<uint32_t *>(&L.jobs[I.job].pad), 1u);
        }
        arrive(B.idone(k % kRing));
    }
    return true;
}

template <class Cons>
__device__ __forceinline__ void serve_tables(const Q8WLaunch &L, unsigned char *sm, const Bars &B, uint32_t tmem,
                                             volatile uint32_t *failed) {
    const ItemRec *ring = reinterpret_cast<const ItemRec *>(sm + L.lay.ring);
    int done = 0;  // items whose epilogue is done
    const bool poll = threadIdx.x < 32;
    // Warp 0 waits, then all four vote: they leave together when a wait gives up, and the other three take no issue
    // slots from the decode warps meanwhile.
    for (int k = 0;; k++) {
        if (!table_vote(!poll || wait_bar(B.rfull(k % kRing), (uint32_t)(k / kRing) & 1u, L, failed))) return;
        const ItemRec &I = ring[k % kRing];
        if (I.it < 0) {
            for (; done < k; done++)
                if (!finish_item<Cons>(L, ring[done % kRing], done, sm, B, tmem, failed)) return;
            return;
        }
        if (I.build) {
            const int area = I.gen % kStages;
            // the table's previous users must be done (with kLag 1 they are among the items finished below)
            if (Cons::kLag > 1)
                for (; done < I.build - 1; done++)
                    if (!finish_item<Cons>(L, ring[done % kRing], done, sm, B, tmem, failed)) return;
            bool ok = !poll || wait_bar(B.staged(area), (uint32_t)(I.gen / kStages) & 1u, L, failed);
            if (!table_vote(ok)) return;
            const uint32_t *so = reinterpret_cast<const uint32_t *>(sm + L.lay.stage_o) + area * kStageOffs;
            const uint16_t *se = reinterpret_cast<const uint16_t *>(
                sm + L.lay.stage_e + (uint32_t)area * ((uint32_t)L.tbl_stage + kStagePad) * 2u);
            build_table<Cons::kFloat>(L, I.local, sm + 128 * I.tab, so, se + so[37]);
        }
        if (k == 0) grid_dependency_wait();  // (see produce; no bounded wait runs while the launch before this one does)
        if constexpr (Cons::kPrepare) Cons::prepare(L, I, k, sm, tmem);
        if (L.chain_scales && I.job > 0) {
            for (; done < k; done++)
                if (!finish_item<Cons>(L, ring[done % kRing], done, sm, B, tmem, failed)) return;
            if (threadIdx.x == 0) chain_wait(L, I.job - 1, failed);
        }
        if (!table_vote(true)) return;
        if (threadIdx.x == 0) arrive(B.tfull(k % kRing));
        // Earlier items' outputs, before the next record is waited for: this item's decode may need their accumulators
        // and, when it has more units than there are slots, holds that record up.  kLag items may be open: small ones
        // then decode side by side (16000x400, one table for all rows, 16 vectors: 17.3 -> 15.5 us; up to two vectors
        // gain nothing, and the second copy of the epilogue slowed their decode by 2 %).
        for (; done + Cons::kLag <= k; done++)
            if (!finish_item<Cons>(L, ring[done % kRing], done, sm, B, tmem, failed)) return;
    }
}

template <class Cons>
__device__ __forceinline__ void decode_units(const Q8WLaunch &L, unsigned char *sm, const Bars &B, uint32_t tmem,
                                             volatile uint32_t *failed) {
    const int lane = threadIdx.x & 31;
    const int w = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5) - kFirstDecode, 0);
    const ItemRec *ring = reinterpret_cast<const ItemRec *>(sm + L.lay.ring);
    const UnitDesc *desc = reinterpret_cast<const UnitDesc *>(sm + L.lay.desc);
    Cons cons;
    cons.init(L, sm, B, tmem, w);
    grid_dependency_wait();  // (see produce)
    uint32_t *unext = reinterpret_cast<uint32_t *>(sm + L.lay.misc) + 2;
    const uint32_t S = (uint32_t)L.S;
    int cur = -1;
    uint32_t lw = 0, taken = (uint32_t)w, last = 0;
    if (!Cons::kStatic && lane == 0) taken = atomicAdd(unext, 1u);
    for (;;) {
        // Units are taken as the warps get to them (their pace differs with the other warps of their scheduler), but
        // for sums whose order counts: there unit u goes to warp u mod W.
        const uint32_t u = Cons::kStatic ? taken : __shfl_sync(0xffffffffu, taken, 0);
        const uint32_t turn = S == 1u ? u : __umulhi(u, L.S_inv), slot = u - turn * S, ph = turn & 1u;
        // A slot passes from warp to warp, so its barrier may still be a phase behind, where the parity test would
        // pass too early: the unit number in the slot tells, and the copy is waited for again once it is right.
        bool ok = wait_bar(B.sfull((int)slot), ph, L, failed);
        const volatile uint32_t *un = &desc[slot].unit;
        for (uint32_t it = 0; ok && *un != u; it++) ok = it < L.spin_limit && !*failed;
        __syncwarp();
        ok = ok && wait_bar(B.sfull((int)slot), ph, L, failed);
        if (!__all_sync(0xffffffffu, ok)) break;
        const UnitDesc d = desc[slot];
        if (d.item < 0) break;
        if (d.item != cur) {
            cur = d.item;
            if (!__all_sync(0xffffffffu, wait_bar(B.tfull(cur % kRing), (uint32_t)(cur / kRing) & 1u, L, failed))) break;
            const ItemRec &I = ring[cur % kRing];
            cons.begin_item(L, I, cur);
            last = I.u0 + I.n;
            lw = (uint32_t)lane * 4u | (uint32_t)I.tab << 7;
        }
        if (d.rows) cons.unit(L, d, sm, L.lay.slots + slot * L.slot_bytes, lw, lane, failed);
        if (Cons::kStatic) taken += (uint32_t)L.W;
        else if (lane == 0) taken = atomicAdd(unext, 1u);  // (its latency passes while this unit is closed)
        __syncwarp();
        if (lane == 0) arrive(B.sempty((int)slot));
        cons.end_unit(L, cur, u + (uint32_t)L.W >= last, sm, B, lane, failed);
    }
    cons.drain(L);
}

// TMEM columns: 32 per decode warp, and the backward's G
template <class Cons>
__device__ __forceinline__ uint32_t tmem_cols(int W) {
    if (Cons::kPrepare) W += 2;
    return W <= 1 ? 32u : W <= 2 ? 64u : W <= 4 ? 128u : W <= 8 ? 256u : 512u;
}

template <class Cons>
__global__ void __launch_bounds__(32 * (kFirstDecode + Cons::kMaxDecode), 1) q8w_kernel(const __grid_constant__ Q8WLaunch L) {
    extern __shared__ __align__(1024) unsigned char smem[];
    const int warp = threadIdx.x >> 5;
    Bars B{smem_u32(smem) + L.lay.bars, L.S, L.W};
    uint32_t *misc = reinterpret_cast<uint32_t *>(smem + L.lay.misc);  // [0] failure flag, [1] TMEM address, [2] next unit
    volatile uint32_t *failed = misc;
    if (threadIdx.x == 0) misc[0] = misc[2] = 0;
    {
        const int n = Bars::count(L.S, L.W, Cons::kMma);
        for (int i = threadIdx.x; i < n; i += blockDim.x) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(B.at(i)), "r"(B.arrivals(i)) : "memory");
        }
        uint32_t *z = reinterpret_cast<uint32_t *>(smem + L.lay.cnt);
        for (int i = threadIdx.x; i < kRing * 2; i += blockDim.x) z[i] = 0;
        UnitDesc *desc = reinterpret_cast<UnitDesc *>(smem + L.lay.desc);
        for (int i = threadIdx.x; i < L.S; i += blockDim.x) desc[i].unit = 0xFFFFFFFFu;
        uint32_t *red = reinterpret_cast<uint32_t *>(smem + L.lay.red);
        for (int i = threadIdx.x; i < Cons::kAreas * Cons::kRed; i += blockDim.x) red[i] = 0;
    }
    fence_mbar_init();
    uint32_t tmem = 0;
    if (Cons::kMma) {
        if (warp == 0) tmem_alloc(misc + 1, tmem_cols<Cons>(L.W));
        tcgen05_fence_before();
    }
    // The launch before this one may still be running (see launch_t).  Whatever the caller passes, matrices and job tables
    // too, may be what it writes, so nothing of that is read before it is complete and its writes are visible.  Where the
    // launch before is this library's own, made in the same call after everything the caller's memory depends on (a zeroing
    // launch, an earlier pass), the first item's record and table go ahead of it.
    if (!L.early) grid_dependency_wait();
    __syncthreads();
    if (Cons::kMma) {
        tcgen05_fence_after();
        tmem = misc[1];
    }
    if (warp < kTableWarps) serve_tables<Cons>(L, smem, B, tmem, failed);
    else if (warp == kProducer) produce(L, smem, B, failed);
    else if (warp == kStager) stage_tables(L, smem, B, failed);
    else if (warp < kFirstDecode + L.W) decode_units<Cons>(L, smem, B, tmem, failed);
    if (Cons::kMma) {
        tcgen05_fence_before();
        __syncthreads();
        if (warp == 0) tmem_dealloc(tmem, tmem_cols<Cons>(L.W));
    } else {
        __syncthreads();
    }
}

// Shared-memory layout for W decode warps and S slots.
template <class Cons>
Q8WLayout layout(const Q8WLaunch &L, int W, int S) {
    Q8WLayout o{};
    auto up = [](uint32_t p) { return (p + 127u) & ~127u; };
    uint32_t p = kLutBytes;
    o.tiles = p;
    p += (uint32_t)W * Cons::tile_bytes(L.xrows);
    o.slots = p = up(p);
    p += (uint32_t)S * L.slot_bytes;
    o.red = p;
    p += (uint32_t)(Cons::kAreas * Cons::kRed) * 4u;
    o.bars = p;
    p += 8u * (uint32_t)Bars::count(S, W, Cons::kMma);
    p = (p + 15u) & ~15u;
    o.desc = p;
    p += (uint32_t)S * (uint32_t)sizeof(UnitDesc);
    o.ring = p;
    p += (uint32_t)(kRing * sizeof(ItemRec));
    o.cnt = p;
    p += (uint32_t)(kRing * sizeof(ItemState));
    o.misc = p;
    p += 16u;
    o.stage_o = p;
    p += kStages * kStageOffs * 4u;
    o.stage_e = p = (p + 15u) & ~15u;
    p += kStages * ((uint32_t)L.tbl_stage + kStagePad) * 2u;
    // an x tile is read as 64 vectors, however many it holds: up to 4 KB past the last tile
    o.total = Cons::kMma ? std::max(p, o.slots + 4096u) : p;
    return o;
}

// The 32 rows' products of 16 columns (w: the lane's row of them, g its s . dy) summed over the lanes and added to dst: over
// lane bits 16, 8, 4 and 2 each half keeps half of the columns, then lanes 2 c and 2 c + 1 hold column c.
__device__ __forceinline__ void wide_reduce(const float (&w)[16], float g, float *dst, int lane) {
    float a[16];
#pragma unroll
    for (int j = 0; j < 16; j++) a[j] = w[j] * g;
#pragma unroll
    for (int n = 8; n > 0; n >>= 1) {
        const bool up = lane & (2 * n);
#pragma unroll
        for (int j = 0; j < 8; j++)
            if (j < n) {
                const float give = up ? a[j] : a[j + n], keep = up ? a[j + n] : a[j];
                a[j] = keep + __shfl_xor_sync(0xffffffffu, give, 2 * n);
            }
    }
    a[0] += __shfl_xor_sync(0xffffffffu, a[0], 1);
    if (!(lane & 1)) atomicAdd(dst + (lane >> 1), a[0]);
}

// The same products where one block leaves no room for q8w_kernel's two decode tables and staging areas (segments of some
// 900 quads and more at 8 bits a weight): a CTA is one warp with one table of 32 KB and one block at a time, no copy under
// way while it decodes.  A block of up to 195 KB fits, more than any launch shape asks for.  kMode 0: integer product, 1:
// float forward, 2: float backward; NV vectors a decode.  Items are q8w_kernel's, each CTA taking every G-th one (even
// shares: its share); of a chain, those of job `only`.  Bound by the lone warp's chain of steps, its x a group of 4 quads
// ahead.
template <int kMode, int NV>
__global__ void __launch_bounds__(32) q8_wide_kernel(const __grid_constant__ Q8WLaunch L, int only) {
    extern __shared__ __align__(1024) unsigned char smem[];
    __shared__ uint64_t bar;
    const int lane = threadIdx.x;
    uint32_t *lut = reinterpret_cast<uint32_t *>(smem) + lane;
    const uint32_t *buf = reinterpret_cast<const uint32_t *>(smem + 32768);
    if (lane == 0) mbar_init(&bar, 1);
    fence_mbar_init();
    __syncwarp();
    uint32_t phase = 0;
    int job = only >= 0 ? only : 0, tjob = -1, tstripe = -1;
    uint32_t next = only >= 0 ? L.jobs[job].item0 + blockIdx.x : blockIdx.x, limit = L.nitems;
    if (only >= 0 && job + 1 < L.njobs) limit = L.jobs[job + 1].item0;
    if (L.span) {
        next = (uint32_t)((uint64_t)blockIdx.x * L.span / gridDim.x);
        limit = (uint32_t)((uint64_t)(blockIdx.x + 1) * L.span / gridDim.x);
    }
    ItemRec r{};
    for (; next < limit; next += L.span ? r.n : gridDim.x) {
        r = ItemRec{};
        fill_item(L, next, limit, job, r);
        const mv_q8_view &m = job_at(L, job).m;
        if (job != tjob || (r.local && r.stripe != tstripe)) {  // the lane's column of the decode table
            tjob = job;
            tstripe = r.stripe;
            const uint32_t t = r.local ? (uint32_t)r.stripe * 32u + (uint32_t)lane : 0u;
            const uint32_t o0 = ldp(m.tbl_off + t), o1 = min(ldp(m.tbl_off + t + 1), m.tbl_len);
            uint32_t q = 0;
            for (uint32_t k = o0; k < o1 && q < 256u; k++) {
                const uint32_t ent = ldp(m.tbl + k), f = ent >> 8;
                for (uint32_t i = 0; i < f && q < 256u; i++, q++) lut[q * 32u] = f | (ent & 0xFFu) << 16 | i << 24;
            }
            if (q < 256u) atomicOr(L.status, MV_DEV_BAD_TABLE);
            for (; q < 256u; q++) lut[q * 32u] = 1u;
        }
        const int row = r.stripe * 32 + lane;
        const float scale = row_scale(r, row);
        for (int v0 = 0; v0 < L.batch; v0 += NV) {
            const int nb = min(NV, L.batch - v0);
            int sum[NV];
            float fs[NV];  // sums, or g = s . dy
#pragma unroll
            for (int v = 0; v < NV; v++) {
                sum[v] = 0;
                fs[v] = 0.f;
                if (kMode == 2 && row < r.rows && v < nb)
                    fs[v] = scale * __uint_as_float((uint32_t)ldp(reinterpret_cast<const uint16_t *>(r.x) + (size_t)(v0 + v) * r.rows + row) << 16);
            }
            for (int seg = r.sb; seg < r.sb + (int)r.n; seg++) {
                const int b = r.stripe * m.nseg + seg;
                const uint32_t o0 = ldp(m.blk_off + b), o1 = ldp(m.blk_off + b + 1), rows = o1 - o0;
                if (o1 < o0 || o1 > m.blocks_rows || rows < 2 || rows >= L.block_bytes / 128u) {
                    if (lane == 0) atomicOr(L.status, MV_DEV_STREAM_OVERRUN);
                    continue;
                }
                __syncwarp();  // (the block before is decoded)
                if (lane == 0) {
                    mbar_arrive_expect_tx(&bar, rows * 128u);
                    if (!L.drop_copy) bulk_g2s(smem + 32768, m.blocks + (size_t)o0 * 32, rows * 128u, &bar);
                }
                const int q0 = seg * r.seg_quads, nq = min(r.seg_quads, (r.cols >> 2) - q0);
                // four quads of every vector (past the batch: its last vector again)
                constexpr int kX = kMode == 0 ? 1 : kMode == 1 ? 2 : 0;  // 16-byte pieces of them
                uint4 xn[NV][kX ? kX : 1];
                const int8_t *xp = r.x + ((size_t)v0 * r.cols + 4 * (size_t)q0) * kX;
                auto load_x = [&]() {
                    const int8_t *p = xp;
#pragma unroll
                    for (int v = 0; v < (kX ? NV : 0); v++) {
#pragma unroll
                        for (int h = 0; h < kX; h++) xn[v][h] = ldx_u4(p + 16 * h);
                        if (v + 1 < nb) p += (size_t)r.cols * kX;
                    }
                };
                load_x();
                const bool ok = mbar_wait_bounded(&bar, phase, L.status, L.spin_limit);
                if (!__all_sync(0xffffffffu, ok)) {
                    mbar_wait_bounded(&bar, phase, nullptr, L.spin_limit);  // let a late copy land before the exit
                    return;
                }
                phase ^= 1u;
                uint32_t lo = buf[lane], hi = buf[32 + lane], at = 64u + (uint32_t)lane, P = 0;
                const uint32_t end = rows * 32u + (uint32_t)lane;
                for (int q = 0; q < nq; q += 4) {  // segments are whole groups of 4 quads (cols % 16 == 0)
                    uint4 xv[NV][kX ? kX : 1];
#pragma unroll
                    for (int v = 0; v < (kX ? NV : 0); v++)
#pragma unroll
                        for (int h = 0; h < kX; h++) xv[v][h] = xn[v][h];
                    xp += q + 4 < nq ? 16 * kX : 0;
                    load_x();
                    float w[16];
#pragma unroll
                    for (int i = 0; i < 4; i++) {
                        const uint32_t word = buf[at];
                        if (hi == 0) {
                            hi = lo;
                            lo = word;
                            at = min(at + 32u, end);
                        }
                        uint32_t e[4];
#pragma unroll
                        for (int j = 0; j < 4; j++) e[j] = lut[((lo >> (8 * j)) & 0xFFu) * 32u];
                        const uint32_t f0 = e[0] & 0xFFu, f1 = e[1] & 0xFFu, f2 = e[2] & 0xFFu;
                        P = f0 * f1 * (f2 * (e[3] & 0xFFu));
                        const unsigned long long st = (unsigned long long)hi * P +
                                                      ((e[0] >> 24) + f0 * ((e[1] >> 24) + f1 * ((e[2] >> 24) + f2 * (e[3] >> 24))));
                        lo = (uint32_t)st;
                        hi = (uint32_t)(st >> 32);
                        const uint32_t wq = __byte_perm(__byte_perm(e[0], e[1], 0x0062), __byte_perm(e[2], e[3], 0x0062), 0x5410);
                        if constexpr (kMode == 0) {
#pragma unroll
                            for (int v = 0; v < NV; v++) {
                                const uint4 &x = xv[v][0];
                                sum[v] = __dp4a((int)wq, (int)(i == 0 ? x.x : i == 1 ? x.y : i == 2 ? x.z : x.w), sum[v]);
                            }
                        } else {
#pragma unroll
                            for (int j = 0; j < 4; j++) w[4 * i + j] = (float)(int8_t)(wq >> (8 * j));
                        }
                        if constexpr (kMode == 1) {
#pragma unroll
                            for (int v = 0; v < NV; v++) {
                                const uint4 &x = xv[v][i >> 1];
                                const uint32_t x01 = i & 1 ? x.z : x.x, x23 = i & 1 ? x.w : x.y;
                                fs[v] = fmaf(w[4 * i], __uint_as_float(x01 << 16), fs[v]);
                                fs[v] = fmaf(w[4 * i + 1], __uint_as_float(x01 & 0xFFFF0000u), fs[v]);
                                fs[v] = fmaf(w[4 * i + 2], __uint_as_float(x23 << 16), fs[v]);
                                fs[v] = fmaf(w[4 * i + 3], __uint_as_float(x23 & 0xFFFF0000u), fs[v]);
                            }
                        }
                    }
                    if constexpr (kMode == 2) {
#pragma unroll
                        for (int v = 0; v < NV; v++)
                            if (v < nb) wide_reduce(w, fs[v], r.ys + (size_t)(v0 + v) * r.cols + 4 * (q0 + q), lane);
                    }
                }
                if (nq > 0 && (hi != 0 || lo != P)) atomicOr(L.status, MV_DEV_FINAL_STATE);
            }
            if (kMode == 2 || row >= r.rows) continue;
#pragma unroll
            for (int v = 0; v < NV; v++) {
                if (v >= nb) break;
                if (kMode == 0) {
                    emit(r, v0 + v, row, sum[v], scale);
                } else {
                    float *dst = r.ys + (size_t)(v0 + v) * r.rows + row;
                    if (r.atomic) atomicAdd(dst, fs[v]);
                    else *dst = fs[v] * scale;
                }
            }
        }
    }
}

template <int kMode>
mv_status launch_wide(const Q8WLaunch &L0, cudaStream_t st) {
    Q8WLaunch L = L0;
    L.block_bytes = L.slot_bytes;
    const size_t smem = 32768 + (size_t)L.block_bytes;
    if (L.ragged || smem + 64 > (size_t)max_smem_optin())
        return fail(MV_ERR_UNSUPPORTED, "Q8 launch needs %zu B of shared memory (max %d)", smem + 64, max_smem_optin());
    auto kern = L.batch == 1 ? q8_wide_kernel<kMode, 1> : q8_wide_kernel<kMode, kMode == 0 ? 16 : 8>;
    mv_status rc = prepare_kernel((const void *)kern, smem, 32, nullptr);
    if (rc) return rc;
    const unsigned grid = (unsigned)std::max(1LL, std::min<long long>(L.nitems, sm_count()));
    for (int job = L.chain_scales ? 0 : -1; job < (L.chain_scales ? L.njobs : 0); job++) {  // a chain: job after job
        kern<<<grid, 32, smem, st>>>(L, job);
        MV_CUDA_TRY(cudaGetLastError(), "q8 wide kernel launch");
    }
    return MV_OK;
}

template <class Cons>
mv_status launch_t(const Q8WLaunch &L0, int warps, int units, cudaStream_t st) {
    Q8WLaunch L = L0;
    const uint32_t limit = (uint32_t)max_smem_optin();
    // CUDA-core consumers: x of a segment behind its block, but for chains, and for the backward, whose job0.x is dY
    L.block_bytes = L.slot_bytes;
    if (!Cons::kMma && !Cons::kPrepare && !L.chain_scales) {
        L.x_off = L.slot_bytes;
        L.x_quad = Cons::kFloat ? 8u : 4u;
        L.slot_bytes += L.x_quad * (uint32_t)(L.batch * kXQuads);
    }
    // Decode warps: as many as asked for (or the consumer's most), no more than a CTA has units for.  The slots
    // beyond one per warp hold the units that the warps take next: without any, a warp would wait for its copy
    // at every unit, so fewer warps with spare slots come before more warps without.
    int W = std::min(warps > 0 ? warps : Cons::kMaxDecode, Cons::kMaxDecode);
    W = std::max(1, std::min(W, units));
    int S = 0;
    for (; W >= 1; W--) {
        const int spare = W >= 4 ? W / 4 : 1;
        for (S = std::min(2 * W + 4, std::max(units, W)); S >= W; S--)
            if (layout<Cons>(L, W, S).total <= limit) break;
        if (S >= W + spare || (S >= W && (W == 1 || S >= units))) break;
        S = 0;
    }
    if (!S) return launch_wide<Cons::kPrepare ? 2 : Cons::kFloat ? 1 : 0>(L0, st);
    L.W = W;
    L.S = S;
    L.S_inv = (uint32_t)((0x100000000ull + (uint32_t)S - 1) / (uint32_t)S);
    L.lay = layout<Cons>(L, W, S);
    auto kern = q8w_kernel<Cons>;
    mv_status rc = prepare_kernel((const void *)kern, L.lay.total, 32 * (kFirstDecode + W), nullptr);
    if (rc) return rc;
    const unsigned grid = (unsigned)std::max(1LL, std::min<long long>(L.nitems, sm_count()));
    const dim3 block(32 * (kFirstDecode + W));
    if (L.chain_scales) {
        // the chained pipeline waits across CTAs: a cooperative launch guarantees that they are all resident
        void *args[] = {&L};
        MV_CUDA_TRY(cudaLaunchCooperativeKernel((const void *)kern, dim3(grid), block, args, L.lay.total, st),
                    "q8 chain cooperative launch");
        return MV_OK;
    }
    // Programmatic dependent launch: a CTA takes over an SM as soon as the launch before it has left it, and sets up its
    // barriers and tensor memory meanwhile; see q8w_kernel for what waits.  Measured on a B200, calls back to back without and
    // with it: a layer of seven matrices, one vector 77.3 -> 74.7 us, 16 vectors 110.3 -> 107.5; 4090x4100, 2 vectors
    // 15.3 -> 13.0; 11008x4096, 64 vectors 47.8 -> 46.4.  (With the first table fetched and built ahead of the wait, 72, 104,
    // 12.1 and 42.6 us; but then a matrix that the launch before writes would be read too early.)
    MV_CUDA_TRY(launch_dependent(kern, dim3(grid), block, L.lay.total, st, L), "q8 kernel launch");
    return MV_OK;
}

}  // namespace

namespace {

// The tensor map of XTiles: job0.x as batch rows of 64-byte pieces.
mv_status x_map(Q8WLaunch &L, bool bf16) {
    typedef CUresult (*Encode)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *, const cuuint64_t *,
                               const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave, CUtensorMapSwizzle,
                               CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
    static const Encode encode = [] {
        void *f = nullptr;
        cudaDriverEntryPointQueryResult r;
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &f, 12000, cudaEnableDefault, &r) != cudaSuccess ||
            r != cudaDriverEntryPointSuccess)
            f = nullptr;
        return reinterpret_cast<Encode>(f);
    }();
    if (!encode) return fail(MV_ERR_CUDA, "cuTensorMapEncodeTiled is not available");
    const cuuint64_t cols = (cuuint64_t)L.job0.m.cols, row = cols * (bf16 ? 2 : 1);
    const cuuint64_t dims[2] = {cols, (cuuint64_t)L.batch};
    const cuuint32_t box[2] = {bf16 ? 32u : 64u, (cuuint32_t)L.xrows}, ones[2] = {1u, 1u};
    const CUresult r = encode(&L.xmap, bf16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_UINT8, 2,
                              const_cast<int8_t *>(L.job0.x), dims, &row, box, ones, CU_TENSOR_MAP_INTERLEAVE_NONE,
                              CU_TENSOR_MAP_SWIZZLE_64B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return fail(MV_ERR_CUDA, "cuTensorMapEncodeTiled: error %d", (int)r);
    return MV_OK;
}

}  // namespace

mv_status q8w_launch_int(const Q8WLaunch &L0, int nv, bool mma, int warps, int units, cudaStream_t st) {
    Q8WLaunch L = L0;
    if (mma) {
        L.xrows = (L.batch + 7) & ~7;
        if (L.ragged)
            return L.batch <= 16 ? launch_t<MmaCons<true, true>>(L, warps, units, st)
                                 : launch_t<MmaCons<false, true>>(L, warps, units, st);
        if (L.batch <= 16) return launch_t<MmaCons<true>>(L, warps, units, st);
        mv_status rc = x_map(L, false);
        return rc ? rc : launch_t<MmaCons<false>>(L, warps, units, st);
    }
    if (L.ragged) switch (nv) {
            case 1: return launch_t<DotCons<1, true>>(L, warps, units, st);
            case 2: return launch_t<DotCons<2, true>>(L, warps, units, st);
            case 4: return launch_t<DotCons<4, true>>(L, warps, units, st);
            default: return launch_t<DotCons<8, true>>(L, warps, units, st);  // (more go to the tensor cores)
        }
    switch (nv) {
        case 1: return launch_t<DotCons<1>>(L, warps, units, st);
        case 2: return launch_t<DotCons<2>>(L, warps, units, st);
        case 4: return launch_t<DotCons<4>>(L, warps, units, st);
        case 8: return launch_t<DotCons<8>>(L, warps, units, st);
        default: return launch_t<DotCons<16>>(L, warps, units, st);
    }
}

bool q8w_ragged_fits(const Q8WLaunch &L0, bool mma) {
    Q8WLaunch L = L0;
    L.xrows = (L.batch + 7) & ~7;
    if (!mma) L.slot_bytes += 4u * (uint32_t)(std::min(L.batch, 8) * kXQuads);
    const uint32_t need = mma ? std::max(layout<MmaCons<true, true>>(L, 1, 1).total, layout<MmaCons<false, true>>(L, 1, 1).total)
                              : layout<DotCons<8, true>>(L, 1, 1).total;
    return need <= (uint32_t)max_smem_optin();
}

mv_status q8w_launch_fwd(const Q8WLaunch &L0, bool dot, int warps, int units, cudaStream_t st) {
    Q8WLaunch L = L0;
    if (L.batch == 1) return launch_t<FwdDot<1>>(L, warps, units, st);
    if (dot)
        return L.batch == 2  ? launch_t<FwdDot<2>>(L, warps, units, st)
               : L.batch <= 4 ? launch_t<FwdDot<4>>(L, warps, units, st)
                              : launch_t<FwdDot<8>>(L, warps, units, st);
    L.xrows = (L.batch + 7) & ~7;
    mv_status rc = x_map(L, true);
    return rc ? rc : launch_t<FwdCons>(L, warps, units, st);
}

mv_status q8w_launch_bwd(const Q8WLaunch &L, bool dot, int warps, int units, cudaStream_t st) {
    if (L.batch == 1) return launch_t<BwdDot<1>>(L, warps, units, st);
    if (dot)
        return L.batch == 2  ? launch_t<BwdDot<2>>(L, warps, units, st)
               : L.batch <= 4 ? launch_t<BwdDot<4>>(L, warps, units, st)
                              : launch_t<BwdDot<8>>(L, warps, units, st);
    return launch_t<BwdCons>(L, warps, units, st);
}

}  // namespace mv

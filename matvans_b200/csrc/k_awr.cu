// Decode + int8 matvec for the reference's "ans-warp-rows" (AWR) layout on
// sm_100a.  Parity target: buffered/ans-warp-rows-kernel.cu:7-221.
//
// The layout makes the 32 lanes of a row share one word stream: at every quad
// step the lanes whose 64-bit state dropped below 2^32 take the next words in
// lane order (ballot + prefix popcount), from a 128-word warp-wide cache that
// holds one uint4 per lane and is read field by field (x, then y, z, w) --
// see ans-warp-rows-kernel.cu:76-139.  That consumption order is part of the
// format, so this kernel keeps one warp per row and reproduces it exactly.
// What changes on B200:
//   * the word stream of a row passes through a ring in shared memory, in
//     consumption order, filled a 128-word block (one 16-byte load per lane) at a
//     time and requested a block ahead when the stream's length is known; a lane's
//     word is then one load at cursor + prefix popcount.  (A block is taken only
//     when a lane actually consumes one of its words: with an unknown length
//     nothing past the row's words is read.  The reference also reloads when the
//     cursor lands exactly on a block boundary, which can read past the row.)
//   * the three 32-entry packed tables become one 4-byte entry {p, 0, symbol,
//     q - cum} per (quantile, lane) at byte q*128 + lane*4: four conflict-free
//     loads per quad instead of twelve warp shuffles
//     (ans-warp-rows-kernel.cu:147-189);
//   * the state update forms the reference's r0 + p0 r1 + p0p1 r2 + p0p1p2 r3
//     (ans-warp-rows-kernel.cu:198-202) as (r0 + p0 r1) + (p0 p1)(r2 + p2 r3)
//     with byte dot products: the same integer, fewer instructions;
//   * one CTA per SM, with as many warps (up to 28) as spread the rows evenly, so
//     that the table is built and x staged once per SM;
//   * any number of vectors per pass (1..16) share one decode, and the int32
//     result is exact (requantisation optional).
// What bounds it: issue, ~45 instructions a step (98 in the form this replaced,
// which kept the words in registers and moved them by shuffles).  Measured on a
// B200, 4096x4096, one vector: 19.4 us before, 12.0 us now; calls back to back,
// launched after one another and while the one before ends, 13.3 and 11.4 us.
//
// The "ans-warp-stripes" layout (ans-warp-stripes-kernel.cu:21-227, encoder.py:
// 323-391) has the same coder and word stream with lane = row of a 32-row stripe:
// one sequential chain per stripe, bound by the latency of a step.  aws_kernel
// shortens the chain: what a word decodes to depends on its low 28 bits alone, so
// helper warps look up every word of the stream ahead of the decode, and a lane
// that refills takes its four symbols and products from there, in parallel with
// the lanes that look up their own state.
#include <algorithm>
#include <cstdio>

#include "mv_device.cuh"

namespace mv {

struct AwrLaunch {
    const uint4 *comp;
    size_t n_u4;  // 0 = unknown (reference shim): no prefetch, no bounds checks
    const uint32_t *offs, *ppf, *cum, *prob;
    int rows, cols;
    const int8_t *x;
    int batch;
    int32_t *y;
    const float *scales;
    float *ys;
    int8_t *out8;  // requantised output (one vector)
    float scale;
    uint32_t *status;
    uint32_t spin_limit;
    int warps;  // awr_kernel: of a CTA, those that take units; the others help with the table and x alone
};

constexpr uint32_t kAwrLut = 128 * 128;    // decode table
constexpr uint32_t kAwrRing = 512 * 4;     // words in shared memory per warp (at most 31 + 128 are waiting)
template <int NV>
constexpr int kAwrWarps = NV <= 4 ? 28 : 20;

// Decode table by the whole CTA: four threads per quantile, eight lane columns each.
__device__ __forceinline__ void awr_table(const AwrLaunch &L, unsigned char *lut) {
    bool bad = false;
    for (uint32_t i = threadIdx.x; i < 128 * 4; i += blockDim.x) {
        const uint32_t q = i >> 2, sh = 8 * (q & 3);
        const uint32_t sym = (ldp(L.ppf + (q >> 2)) >> sh) & 0xFF;
        const uint32_t c = (ldp(L.cum + (q >> 2)) >> sh) & 0xFF;
        const uint32_t p = (ldp(L.prob + (q >> 2)) >> sh) & 0xFF;
        bad |= c > q || p == 0;
        const uint32_t e = p | sym << 16 | ((q - c) & 0xFFu) << 24;
        uint4 *dst = reinterpret_cast<uint4 *>(lut + q * 128u + (i & 3u) * 32u);
        dst[0] = dst[1] = make_uint4(e, e, e, e);
    }
    if (bad) atomicOr(L.status, MV_DEV_BAD_TABLE);
}

// x as quads [cols/4][NV] by the whole CTA
template <int NV>
__device__ __forceinline__ void awr_stage_x(const AwrLaunch &L, uint32_t *xs) {
    const int nq = L.cols >> 2;
    const bool xal = (reinterpret_cast<uintptr_t>(L.x) & 3) == 0;
    for (int i = threadIdx.x; i < nq * NV; i += blockDim.x) {
        const int v = i / nq, c = i - v * nq;  // consecutive threads read consecutive quads
        uint32_t val = 0;
        if (v < L.batch) {
            const int8_t *p = L.x + (size_t)v * L.cols + 4 * c;
            if (xal) val = *reinterpret_cast<const uint32_t *>(p);
            else for (int j = 0; j < 4; j++) val |= (uint32_t)(uint8_t)p[j] << (8 * j);
        }
        xs[c * NV + v] = val;
    }
}

// What the low 28 bits of a state (or of a word) decode to: the packed symbols, the product P of the four
// probabilities and the mixed-radix remainder t < P.
__device__ __forceinline__ uint32_t awr_lookup(const unsigned char *lut, uint32_t lane4, uint32_t lo, uint32_t &P, uint32_t &t) {
    const uint32_t e0 = *reinterpret_cast<const uint32_t *>(lut + (((lo << 7) & 0x3F80u) | lane4));
    const uint32_t e1 = *reinterpret_cast<const uint32_t *>(lut + ((lo & 0x3F80u) | lane4));
    const uint32_t e2 = *reinterpret_cast<const uint32_t *>(lut + (((lo >> 7) & 0x3F80u) | lane4));
    const uint32_t e3 = *reinterpret_cast<const uint32_t *>(lut + (((lo >> 14) & 0x3F80u) | lane4));
    const uint32_t u01 = __dp4a(e0, __byte_perm(e1, 1u, 0x4553), 0u);  // r0 + p0 r1 = (p0, 0, sym, r0) . (r1, 0, 0, 1)
    const uint32_t u23 = __dp4a(e2, __byte_perm(e3, 1u, 0x4553), 0u);
    const uint32_t p01 = __dp2a_lo(e1, e0, 0u), p23 = __dp2a_lo(e3, e2, 0u);
    P = p01 * p23;
    t = u01 + p01 * u23;
    return __byte_perm(__byte_perm(e0, e1, 0x0062), __byte_perm(e2, e3, 0x0062), 0x5410);
}

// state = (state >> 28) * P + t
__device__ __forceinline__ void awr_update(uint32_t &lo, uint32_t &hi, uint32_t P, uint32_t t) {
    const uint32_t a = __funnelshift_r(lo, hi, 28), b = hi >> 28;
    const unsigned long long s = (unsigned long long)a * P + t;
    lo = (uint32_t)s;
    hi = (uint32_t)(s >> 32) + b * P;
}

template <bool REQUANT, int NV>
__device__ __forceinline__ void awr_store(const AwrLaunch &L, int r, const int (&acc)[NV]) {
    if (REQUANT) {
        const int q = __float2int_rn((float)acc[0] * L.scale);  // ans-warp-rows-kernel.cu:212-220
        L.out8[r] = (int8_t)max(-128, min(127, q));
    } else {
#pragma unroll
        for (int v = 0; v < NV; v++)
            if (v < L.batch) {
                L.y[(size_t)v * L.rows + r] = acc[v];
                if (L.ys) L.ys[(size_t)v * L.rows + r] = (float)acc[v] * L.scales[r];
            }
    }
}

// STRIPES: lane l is row 32u + l of stripe u, decodes its quad j (columns 4j..4j+3) at step j and keeps its own sums
// (no warp reduction); one offset per stripe.
// BOUNDED: the stream's length is known, so words may be staged ahead: the ring is looked after once in four steps
// (a warp-wide branch costs ~50 cycles of a step's latency).  Otherwise (the reference's launchers do not pass the
// length) a block is read when a lane takes its first word and not before.
template <int NV, bool REQUANT, bool STRIPES, bool BOUNDED>
__global__ void __launch_bounds__(32 * kAwrWarps<NV>) awr_kernel(const AwrLaunch L) {
    extern __shared__ __align__(1024) unsigned char smem[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, W = L.warps;
    const int nq = L.cols >> 2;
    uint32_t *ring = reinterpret_cast<uint32_t *>(smem + kAwrLut + (uint32_t)warp * kAwrRing);
    uint32_t *xs = reinterpret_cast<uint32_t *>(smem + kAwrLut + (uint32_t)W * kAwrRing);
    grid_dependency_wait();  // (the launch before this one may have written the tables, the stream or x)
    grid_launch_dependents();
    awr_table(L, smem);
    awr_stage_x<NV>(L, xs);
    __syncthreads();
    if (warp >= W) return;

    const uint32_t lt_mask = (1u << lane) - 1u, lane4 = (uint32_t)lane << 2;
    const int units = STRIPES ? L.rows / 32 : L.rows;  // warps' work units: rows or 32-row stripes
    for (int row = blockIdx.x * W + warp; row < units; row += gridDim.x * W) {
        // The first block holds the initial states (fields z, w) and the first 64 words of the stream (x, y); every
        // later block 128 words, field by field (ans-warp-rows-kernel.cu:76-139).
        size_t bi = ldp(L.offs + row);  // uint4 index of the latest block in the ring
        auto block = [&](size_t at) {
            return !BOUNDED || at + 32 <= L.n_u4 ? L.comp[at + lane] : make_uint4(0, 0, 0, 0);
        };
        // words of the stream that can be read (from the first block's x on), for the overrun check
        const unsigned long long have = BOUNDED ? (bi + 32 <= L.n_u4 ? (L.n_u4 - bi) / 32 * 128 - 64 : 0) : ~0ull;
        const uint4 first = block(bi);
        uint4 nxt = BOUNDED ? block(bi + 32) : first;
        uint32_t lo = first.z, hi = first.w;
        __syncwarp();
        ring[lane] = first.x;
        ring[32 + lane] = first.y;
        uint32_t cur = 0, staged = 64;  // words consumed, words in the ring
        auto stage = [&]() {
            bi += 32;
            if (!BOUNDED) nxt = block(bi);
            const uint32_t s = staged + (uint32_t)lane;
            ring[s & 511u] = nxt.x;
            ring[(s + 32u) & 511u] = nxt.y;
            ring[(s + 64u) & 511u] = nxt.z;
            ring[(s + 96u) & 511u] = nxt.w;
            staged += 128u;
            if (BOUNDED) nxt = block(bi + 32);
            __syncwarp();
        };
        __syncwarp();
        int acc[NV];
#pragma unroll
        for (int v = 0; v < NV; v++) acc[v] = 0;
        const uint32_t *xq = xs + (STRIPES ? 0 : lane * NV);  // stripes: one x quad for all lanes
        auto step = [&]() {
            const bool need = hi == 0;
            const uint32_t ballot = __ballot_sync(0xffffffffu, need);
            const uint32_t at = cur + __popc(ballot & lt_mask);
            cur += __popc(ballot);
            if (!BOUNDED && cur > staged) stage();  // a lane takes a word of the next block (128 > 32: one is enough)
            const uint32_t w = ring[at & 511u];
            hi = need ? lo : hi;
            lo = need ? w : lo;
            uint32_t P, t;
            const uint32_t wq = awr_lookup(smem, lane4, lo, P, t);
            awr_update(lo, hi, P, t);
#pragma unroll
            for (int v = 0; v < NV; v++) acc[v] = __dp4a((int)wq, (int)xq[v], acc[v]);
            xq += STRIPES ? NV : 32 * NV;
        };
        const int steps = STRIPES ? nq : nq / 32;
        int j = 0;
        for (; j + 4 <= steps; j += 4) {
            if (BOUNDED)
                while (staged < cur + 128u) stage();  // at most twice: 384 words wait in the ring at most
            step();
            step();
            step();
            step();
        }
        for (; j < steps; j++) {
            if (BOUNDED && staged < cur + 32u) stage();
            step();
        }
        if (BOUNDED && (cur > have || have == 0)) atomicOr(L.status, MV_DEV_STREAM_OVERRUN);
        if (STRIPES) {
            awr_store<REQUANT>(L, row * 32 + lane, acc);  // rows % 32 == 0
        } else {
#pragma unroll
            for (int v = 0; v < NV; v++) acc[v] = __reduce_add_sync(0xffffffffu, acc[v]);
            if (lane == 0) awr_store<REQUANT>(L, row, acc);
        }
    }
}

// Stripes with a stream of known length: one CTA per stripe, warp 0 decodes, kAwsHelpers warps look up the stream's
// words ahead.  The words go through a ring of kAwsBlocks blocks of 128 entries {P, t, symbols, word} (16 bytes); full
// and empty mbarriers per block.  A step of the decode is: vote, prefix popcount, one 16-byte load, two selects and the
// state's multiply-add, beside it the four lookups of the lanes that do not refill.  (Measured on a B200, 4096x4096, one vector: 174.7 us with
// the words in registers and the lookups behind the refill, 340 cycles a step; 107.2 us now, 204 cycles a step.)
constexpr int kAwsHelpers = 3, kAwsBlocks = 8;
constexpr uint32_t kAwsRing = kAwsBlocks * 2048;

template <int NV, bool REQUANT>
__global__ void __launch_bounds__(32 * (1 + kAwsHelpers)) aws_kernel(const AwrLaunch L) {
    extern __shared__ __align__(1024) unsigned char smem[];
    __shared__ uint64_t full[kAwsBlocks], empty[kAwsBlocks];
    __shared__ uint32_t stop;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int nq = L.cols >> 2;
    const uint32_t lane4 = (uint32_t)lane << 2;
    unsigned char *ring = smem + kAwrLut;
    uint32_t *xs = reinterpret_cast<uint32_t *>(smem + kAwrLut + kAwsRing);
    if (threadIdx.x < kAwsBlocks) {
        mbar_init(&full[threadIdx.x], 1);
        mbar_init(&empty[threadIdx.x], 1);
    }
    if (threadIdx.x == 0) stop = 0;
    fence_mbar_init();
    grid_dependency_wait();  // (as in awr_kernel)
    grid_launch_dependents();
    awr_table(L, smem);
    awr_stage_x<NV>(L, xs);
    __syncthreads();

    const int stripe = blockIdx.x;
    const size_t b0 = ldp(L.offs + stripe);  // uint4 index of the stripe's first block
    const size_t nblk = b0 + 32 <= L.n_u4 ? (L.n_u4 - b0) / 32 : 0;  // whole blocks that can be read
    volatile uint32_t *done = &stop;

    if (warp > 0) {
        // helpers: block b (0: the 64 words behind the states) to ring slot b % kAwsBlocks, warp b % kAwsHelpers
        uint4 v = make_uint4(0, 0, 0, 0);
        uint32_t b = (uint32_t)warp - 1u;
        if (b < nblk) v = L.comp[b0 + 32 * (size_t)b + lane];
        for (; b < nblk; b += kAwsHelpers) {
            const uint4 c = v;
            if (b + kAwsHelpers < nblk) v = L.comp[b0 + 32 * (size_t)(b + kAwsHelpers) + lane];
            const uint32_t slot = b % kAwsBlocks, turn = b / kAwsBlocks;
            if (turn > 0) {
                bool ok = false;
                for (uint32_t it = 0; !ok && it < L.spin_limit; it++) {
                    ok = mbar_try_wait(&empty[slot], (turn - 1u) & 1u);
                    if (!ok && *done) break;
                }
                if (!__all_sync(0xffffffffu, ok)) return;  // the decode is over (or gave up)
            }
            uint4 *dst = reinterpret_cast<uint4 *>(ring + slot * 2048u) + lane;
            // (block 0: its two fields of words go to the slot's upper half, before block 1)
            const uint32_t w[4] = {c.x, c.y, b ? c.z : c.x, b ? c.w : c.y};
#pragma unroll
            for (int j = 0; j < 4; j++) {
                uint32_t P, t;
                const uint32_t wq = awr_lookup(smem, lane4, w[j], P, t);
                dst[32 * j] = make_uint4(P, t, wq, w[j]);
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(&full[slot]);
        }
        return;
    }

    const uint32_t lt_mask = (1u << lane) - 1u;
    const uint4 first = nblk ? L.comp[b0 + lane] : make_uint4(0, 0, 0, 0);
    uint32_t lo = first.z, hi = first.w;
    // words consumed, words in the ring so far, blocks they came from, blocks given back; word w is entry w + 64
    uint32_t cur = 0, limit = 0, blocks = 0, freed = 0;
    bool ok = true;
    int acc[NV];
#pragma unroll
    for (int v = 0; v < NV; v++) acc[v] = 0;
    const uint32_t *xq = xs;
    auto step = [&]() {
        const bool need = hi == 0;
        uint32_t P, t;
        uint32_t wq = awr_lookup(smem, lane4, lo, P, t);  // of the lanes that do not refill
        const uint32_t ballot = __ballot_sync(0xffffffffu, need);
        const uint32_t at = cur + __popc(ballot & lt_mask);
        cur += __popc(ballot);
        const uint4 e = *reinterpret_cast<const uint4 *>(ring + (((at + 64u) * 16u) & (kAwsRing - 1u)));
        hi = need ? lo : hi;
        lo = need ? e.w : lo;
        P = need ? e.x : P;
        t = need ? e.y : t;
        wq = need ? e.z : wq;
        awr_update(lo, hi, P, t);
#pragma unroll
        for (int v = 0; v < NV; v++) acc[v] = __dp4a((int)wq, (int)xq[v], acc[v]);
        xq += NV;
    };
    for (int j = 0; j < nq; j += 8) {
        // Eight steps take at most 256 words: their blocks are waited for, and the blocks before them given back.  (Once
        // in eight steps: a warp-wide branch costs ~50 cycles, a step of the chain ~130.)
        while (limit < cur + 256u && blocks < nblk) {
            ok &= mbar_wait_bounded(&full[blocks % kAwsBlocks], (blocks / kAwsBlocks) & 1u, L.status, ok ? L.spin_limit : 1u);
            limit += blocks ? 128u : 64u;
            blocks++;
        }
        const uint32_t over = min((cur + 64u) >> 7, blocks ? blocks - 1u : 0u);  // blocks whose words are all consumed
        __syncwarp();  // (every lane has loaded its words of the steps before: one lane's arrival gives a block back)
        if (freed + (uint32_t)lane < over) mbar_arrive(&empty[(freed + (uint32_t)lane) % kAwsBlocks]);
        freed = max(freed, over);
        if (j + 8 <= nq) {
#pragma unroll
            for (int i = 0; i < 8; i++) step();
        } else {
            for (int i = j; i < nq; i++) step();
        }
    }
    __syncwarp();
    if (lane == 0) *done = 1u;
    if (nblk == 0 || cur > 128ull * nblk - 64ull) atomicOr(L.status, MV_DEV_STREAM_OVERRUN);
    awr_store<REQUANT>(L, stripe * 32 + lane, acc);  // rows % 32 == 0
}

namespace {

template <int NV, bool REQUANT, bool STRIPES = false>
mv_status launch_awr(const AwrLaunch &L0, cudaStream_t st) {
    AwrLaunch L = L0;
    const size_t xb = (size_t)(L.cols / 4) * NV * 4;
    if (128 * 32 * 8 + xb > (size_t)max_smem_optin())
        return fail(MV_ERR_UNSUPPORTED, "AWR: %d columns x %d vectors exceed shared memory", L.cols, NV);
    if (STRIPES && L.n_u4 && kAwrLut + kAwsRing + xb + 2048 <= (size_t)max_smem_optin()) {  // (2 KB: barriers)
        const size_t smem = kAwrLut + kAwsRing + xb;
        auto kern = aws_kernel<NV, REQUANT>;
        mv_status rc = prepare_kernel((const void *)kern, smem, 32 * (1 + kAwsHelpers), nullptr);
        if (rc) return rc;
        MV_CUDA_TRY(launch_dependent(kern, dim3(L.rows / 32), dim3(32 * (1 + kAwsHelpers)), smem, st, L), "aws kernel launch");
        return MV_OK;
    }
    // warps: stripes are few (rows / 32) and long, one to a CTA spreads them over the SMs; rows in even rounds over the
    // SMs, as many as fit beside x
    const int units = STRIPES ? L.rows / 32 : L.rows, sms = sm_count();
    int wmax = STRIPES ? 1 : kAwrWarps<NV>;
    while (wmax > 1 && kAwrLut + (size_t)wmax * kAwrRing + xb > (size_t)max_smem_optin()) wmax--;
    const int rounds = (units + sms * wmax - 1) / (sms * wmax);
    const int W = STRIPES ? 1 : std::max(1, (units + sms * rounds - 1) / (sms * rounds));
    const size_t smem = kAwrLut + (size_t)W * kAwrRing + xb;
    auto kern = L.n_u4 ? awr_kernel<NV, REQUANT, STRIPES, true> : awr_kernel<NV, REQUANT, STRIPES, false>;
    // (rows: the table and x by 8 warps at least; 512x1024, 4 vectors, 4 rows a CTA: 6.2 us with 4 warps, 5.0 with 8)
    const int threads = 32 * (STRIPES ? 1 : std::max(W, 8));
    mv_status rc = prepare_kernel((const void *)kern, smem, threads, nullptr);
    if (rc) return rc;
    L.warps = W;
    const int grid = STRIPES ? units : std::max(1, std::min((units + W - 1) / W, sms));
    MV_CUDA_TRY(launch_dependent(kern, dim3(grid), dim3(threads), smem, st, L), "awr kernel launch");
    return MV_OK;
}

mv_status awr_common(const uint32_t *comp, size_t n_words, const uint32_t *offs, const uint32_t *ppf,
                     const uint32_t *cum, const uint32_t *prob, int rows, int cols, const int8_t *x,
                     AwrLaunch &L, bool stripes = false) {
    if (!comp || !offs || !ppf || !cum || !prob || !x) return fail(MV_ERR_ARG, "mv_awr: NULL pointer");
    if (rows <= 0 || cols <= 0) return fail(MV_ERR_ARG, "mv_awr: rows/cols must be positive");
    if (stripes) {
        if (rows % 32 || cols % 4)
            return fail(MV_ERR_SHAPE, "stripes layout needs rows %% 32 == 0 and cols %% 4 == 0 (%dx%d)", rows, cols);
    } else if (cols % 128) {
        return fail(MV_ERR_SHAPE, "AWR layout needs cols %% 128 == 0 (cols=%d)", cols);
    }
    if (((uintptr_t)comp & 15) != 0) return fail(MV_ERR_ARG, "mv_awr: compressed not 16-byte aligned");
    mv_status rc;
    L.status = device_status_word(&rc);
    if (rc) return rc;
    L.comp = reinterpret_cast<const uint4 *>(comp);
    L.n_u4 = n_words / 4;
    L.spin_limit = wait_spin_limit();
    L.offs = offs;
    L.ppf = ppf;
    L.cum = cum;
    L.prob = prob;
    L.rows = rows;
    L.cols = cols;
    L.x = x;
    return MV_OK;
}

}  // namespace

mv_status awr_matvec(const uint32_t *comp, size_t n_words, const uint32_t *offs, const uint32_t *ppf,
                     const uint32_t *cum, const uint32_t *prob, int rows, int cols, const int8_t *x,
                     int batch, int32_t *y, const float *scales, float *ys, cudaStream_t st) {
    AwrLaunch L{};
    mv_status rc = awr_common(comp, n_words, offs, ppf, cum, prob, rows, cols, x, L);
    if (rc) return rc;
    if (!y || batch <= 0) return fail(MV_ERR_ARG, "mv_awr_matvec: bad y/batch");
    if (n_words == 0) return fail(MV_ERR_ARG, "mv_awr_matvec: n_words must be given");
    if (ys && !scales) return fail(MV_ERR_ARG, "mv_awr_matvec: y_scaled needs row scales");
    for (int v0 = 0; v0 < batch; v0 += 16) {
        const int nb = std::min(16, batch - v0);
        AwrLaunch P = L;
        P.x = x + (size_t)v0 * cols;
        P.batch = nb;
        P.y = y + (size_t)v0 * rows;
        P.scales = scales;
        P.ys = ys ? ys + (size_t)v0 * rows : nullptr;
        if (nb == 1) rc = launch_awr<1, false>(P, st);
        else if (nb == 2) rc = launch_awr<2, false>(P, st);
        else if (nb <= 4) rc = launch_awr<4, false>(P, st);
        else if (nb <= 8) rc = launch_awr<8, false>(P, st);
        else rc = launch_awr<16, false>(P, st);
        if (rc) return rc;
    }
    return MV_OK;
}

mv_status aws_matvec(const uint32_t *comp, size_t n_words, const uint32_t *offs, const uint32_t *ppf,
                     const uint32_t *cum, const uint32_t *prob, int rows, int cols, const int8_t *x,
                     int batch, int32_t *y, const float *scales, float *ys, cudaStream_t st) {
    AwrLaunch L{};
    mv_status rc = awr_common(comp, n_words, offs, ppf, cum, prob, rows, cols, x, L, true);
    if (rc) return rc;
    if (!y || batch <= 0) return fail(MV_ERR_ARG, "mv_aws_matvec: bad y/batch");
    if (n_words == 0) return fail(MV_ERR_ARG, "mv_aws_matvec: n_words must be given");
    if (ys && !scales) return fail(MV_ERR_ARG, "mv_aws_matvec: y_scaled needs row scales");
    for (int v0 = 0; v0 < batch; v0 += 16) {
        const int nb = std::min(16, batch - v0);
        AwrLaunch P = L;
        P.x = x + (size_t)v0 * cols;
        P.batch = nb;
        P.y = y + (size_t)v0 * rows;
        P.scales = scales;
        P.ys = ys ? ys + (size_t)v0 * rows : nullptr;
        if (nb == 1) rc = launch_awr<1, false, true>(P, st);
        else if (nb == 2) rc = launch_awr<2, false, true>(P, st);
        else if (nb <= 4) rc = launch_awr<4, false, true>(P, st);
        else if (nb <= 8) rc = launch_awr<8, false, true>(P, st);
        else rc = launch_awr<16, false, true>(P, st);
        if (rc) return rc;
    }
    return MV_OK;
}

mv_status aws_requant(const uint32_t *comp, size_t n_words, const uint32_t *offs, const uint32_t *ppf,
                      const uint32_t *cum, const uint32_t *prob, int rows, int cols, const int8_t *x,
                      float scale, int8_t *out8, cudaStream_t st) {
    AwrLaunch L{};
    mv_status rc = awr_common(comp, n_words, offs, ppf, cum, prob, rows, cols, x, L, true);
    if (rc) return rc;
    if (!out8) return fail(MV_ERR_ARG, "mv_aws_matvec_requant: NULL output");
    L.batch = 1;
    L.out8 = out8;
    L.scale = scale;
    return launch_awr<1, true, true>(L, st);
}

mv_status awr_requant(const uint32_t *comp, size_t n_words, const uint32_t *offs, const uint32_t *ppf,
                      const uint32_t *cum, const uint32_t *prob, int rows, int cols, const int8_t *x,
                      float scale, int8_t *out8, cudaStream_t st) {
    AwrLaunch L{};
    mv_status rc = awr_common(comp, n_words, offs, ppf, cum, prob, rows, cols, x, L);
    if (rc) return rc;
    if (!out8) return fail(MV_ERR_ARG, "mv_awr_matvec_requant: NULL output");
    L.batch = 1;
    L.out8 = out8;
    L.scale = scale;
    return launch_awr<1, true>(L, st);
}

}  // namespace mv

extern "C" {

mv_status mv_awr_matvec(const uint32_t *compressed_dev, size_t n_words, const uint32_t *warp_offsets_dev,
                        const uint32_t *ppf_dev, const uint32_t *ppf_cum_dev,
                        const uint32_t *ppf_prob_dev, int rows, int cols, const int8_t *x_dev,
                        int batch, int32_t *y_dev, const float *row_scales_dev, float *y_scaled_dev,
                        void *stream) {
    return mv::awr_matvec(compressed_dev, n_words, warp_offsets_dev, ppf_dev, ppf_cum_dev, ppf_prob_dev,
                          rows, cols, x_dev, batch, y_dev, row_scales_dev, y_scaled_dev,
                          (cudaStream_t)stream);
}

mv_status mv_awr_matvec_requant(const uint32_t *compressed_dev, size_t n_words,
                                const uint32_t *warp_offsets_dev, const uint32_t *ppf_dev,
                                const uint32_t *ppf_cum_dev, const uint32_t *ppf_prob_dev, int rows,
                                int cols, const int8_t *x_dev, float scale, int8_t *out8_dev,
                                void *stream) {
    return mv::awr_requant(compressed_dev, n_words, warp_offsets_dev, ppf_dev, ppf_cum_dev, ppf_prob_dev,
                           rows, cols, x_dev, scale, out8_dev, (cudaStream_t)stream);
}

// buffered/ans-warp-rows.cu:38-60: same arguments, same int8 output, legacy
// default stream.  The stream length is unknown here, so no bounds checks.
void mat_vec_mul_coalesced(const void *in_vector_gpu, void *out_vector_gpu, size_t in_dim, size_t out_dim,
                           float scale, const void *compressed, const uint32_t *warp_offsets,
                           const uint32_t *ppf, const uint32_t *ppf_cum, const uint32_t *ppf_prob) {
    mv_status rc = mv::awr_requant(reinterpret_cast<const uint32_t *>(compressed), 0, warp_offsets, ppf,
                                   ppf_cum, ppf_prob, (int)out_dim, (int)in_dim,
                                   reinterpret_cast<const int8_t *>(in_vector_gpu), scale,
                                   reinterpret_cast<int8_t *>(out_vector_gpu), 0);
    if (rc) std::fprintf(stderr, "mat_vec_mul_coalesced: %s\n", mv_last_error());
}

mv_status mv_aws_matvec(const uint32_t *compressed_dev, size_t n_words, const uint32_t *warp_offsets_dev,
                        const uint32_t *ppf_dev, const uint32_t *ppf_cum_dev,
                        const uint32_t *ppf_prob_dev, int rows, int cols, const int8_t *x_dev,
                        int batch, int32_t *y_dev, const float *row_scales_dev, float *y_scaled_dev,
                        void *stream) {
    return mv::aws_matvec(compressed_dev, n_words, warp_offsets_dev, ppf_dev, ppf_cum_dev, ppf_prob_dev,
                          rows, cols, x_dev, batch, y_dev, row_scales_dev, y_scaled_dev,
                          (cudaStream_t)stream);
}

mv_status mv_aws_matvec_requant(const uint32_t *compressed_dev, size_t n_words,
                                const uint32_t *warp_offsets_dev, const uint32_t *ppf_dev,
                                const uint32_t *ppf_cum_dev, const uint32_t *ppf_prob_dev, int rows,
                                int cols, const int8_t *x_dev, float scale, int8_t *out8_dev,
                                void *stream) {
    return mv::aws_requant(compressed_dev, n_words, warp_offsets_dev, ppf_dev, ppf_cum_dev, ppf_prob_dev,
                           rows, cols, x_dev, scale, out8_dev, (cudaStream_t)stream);
}

// buffered/ans-warp-stripes.cu:38-60 (the launcher of the stripes program, which has the same name as the
// rows program's; renamed here so that both live in one library): same arguments, same int8 output,
// legacy default stream, no bounds checks (the stream length is unknown).
void mat_vec_mul_coalesced_stripes(const void *in_vector_gpu, void *out_vector_gpu, size_t in_dim,
                                   size_t out_dim, float scale, const void *compressed,
                                   const uint32_t *warp_offsets, const uint32_t *ppf, const uint32_t *ppf_cum,
                                   const uint32_t *ppf_prob) {
    mv_status rc = mv::aws_requant(reinterpret_cast<const uint32_t *>(compressed), 0, warp_offsets, ppf,
                                   ppf_cum, ppf_prob, (int)out_dim, (int)in_dim,
                                   reinterpret_cast<const int8_t *>(in_vector_gpu), scale,
                                   reinterpret_cast<int8_t *>(out_vector_gpu), 0);
    if (rc) std::fprintf(stderr, "mat_vec_mul_coalesced_stripes: %s\n", mv_last_error());
}

}  // extern "C"

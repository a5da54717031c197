// Planning and launching of the Q8-stripe products: single matrices, stacks (many
// matrices in one launch), the chained pipeline and the float form, all through
// the kernels of k_q8w.cu.
#include <algorithm>

#include "mv_device.cuh"
#include "q8w.cuh"

namespace mv {

__global__ void scale_rows_kernel(const int32_t *y, const float *s, float *ys, int rows, int batch, int ldy);

__global__ void q8s_chain_reset(Q8Job *jobs, int njobs) {
    for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < njobs; j += gridDim.x * blockDim.x) jobs[j].pad = 0;
}

__global__ void q8s_zero_atomic_y(const Q8Job *jobs, int njobs, int batch) {
    for (int j = blockIdx.y; j < njobs; j += gridDim.y) {
        const Q8Job &J = jobs[j];
        if (!J.atomic) continue;
        const size_t n = (size_t)batch * J.m.rows;
        for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
            J.y[i] = 0;
    }
}

__global__ void q8s_scale_atomic_y(const Q8Job *jobs, int njobs, int batch) {
    for (int j = blockIdx.y; j < njobs; j += gridDim.y) {
        const Q8Job &J = jobs[j];
        if (!J.atomic || !J.ys) continue;
        const size_t n = (size_t)batch * J.m.rows;
        for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
            J.ys[i] = (float)J.y[i] * J.scales[i % J.m.rows];
    }
}

// n 32-bit zeros.  (A memset between kernels costs more than a small kernel: 500x2992 and 160x4096, one vector, four
// parts, 12.3 us with cudaMemsetAsync, 9.6 with this.)
__global__ void __launch_bounds__(256) zero_words(uint32_t *p, size_t n) {
    grid_launch_dependents();  // (the product behind it waits for these zeros before its first sum)
    const size_t head = min(n, (size_t)((16 - ((uintptr_t)p & 15)) & 15) / 4), n4 = (n - head) / 4;
    const size_t i0 = blockIdx.x * (size_t)blockDim.x + threadIdx.x, step = (size_t)gridDim.x * blockDim.x;
    uint4 *q = reinterpret_cast<uint4 *>(p + head);
    for (size_t i = i0; i < n4; i += step) q[i] = make_uint4(0, 0, 0, 0);
    if (i0 < head) p[i0] = 0;
    const size_t t = head + 4 * n4 + i0;
    if (t < n) p[t] = 0;
}

namespace {

mv_status zero_launch(void *p, size_t words, cudaStream_t st) {
    const unsigned grid = (unsigned)std::min<size_t>((words + 1023) / 1024, 4 * (size_t)sm_count());
    zero_words<<<std::max(1u, grid), 256, 0, st>>>(static_cast<uint32_t *>(p), words);
    MV_CUDA_TRY(cudaGetLastError(), "zero_words launch");
    return MV_OK;
}

// Integer batches of at least this many vectors go to the tensor-core consumer with engine 0, whose cost hardly depends
// on the batch, while the dp4a consumer's grows with it.  Measured on a B200, dp4a | tensor cores: 11008x4096, 4 vectors
// 30.2 | 32.6 us, 6 vectors 36.4 | 31.4; 6000x6000, 25.5 | 29.5 and 30.8 | 29.5; a layer of seven matrices, 4 vectors
// 92.7 | 97.1, 8 vectors 115.4 | 97.5.
constexpr int kMmaMinVectors = 5;
// Where the dp4a consumer reads x from global memory, a load per vector and group in its loop (chains, whose x is not there
// any earlier, and segments of more than kXQuads quads), from 3 vectors: a chain of 7B matrices, 3 vectors 94.6 | 73.5 us,
// of hidden size 512 22.3 | 21.9; 4096x4096 in segments of 128 quads 17.3 | 15.9, of 256 25.3 | 20.7.
constexpr int kMmaMinGlobalX = 3;
// A single matrix that gives no warp a second segment is bound by a lone warp's pace, which the tensor cores' tiles slow
// down: dp4a up to 8 vectors (500x2992, 8 vectors: 10.0 | 12.4 us; 1024x1024: 8.8 | 9.0).
constexpr int kMmaMinLone = 9;
// check_shape: the batch from which a launch shape is taken as a tensor-core one.
constexpr int kMmaShape = MV_MMA_MIN_VECTORS;

int nv_round(int nb) { return nb <= 2 ? nb : nb <= 4 ? 4 : nb <= 8 ? 8 : 16; }

}  // namespace

mv_status stack_plan(mv_q8_job *jobs, int njobs, const mv_q8_tuning *tuning, mv_q8_stack_info *info);

namespace {

mv_q8_tuning resolve(const mv_q8_tuning *t) {
    mv_q8_tuning r{8, 2, 1, 0, 0, MV_ENGINE_AUTO};
    if (t) {
        if (t->engine == MV_ENGINE_DP4A) r.engine = MV_ENGINE_DP4A;
        if (t->parts > 0) r.parts = t->parts;
        if (t->warps > 0) r.warps = std::min(16, t->warps);  // more than 8: the integer CUDA-core consumer only
        if (t->ilp == 1 || t->ilp == 2) r.ilp = t->ilp;
        if (t->depth == 1 || t->depth == 2) r.depth = t->depth;
        if (t->ctas_per_sm > 0) r.ctas_per_sm = t->ctas_per_sm;
    }
    return r;
}

// Decode warps of a launch (0: as many as fit).  Up to 8 warps a CTA once meant two CTAs to an SM, and callers hold tuned
// shapes of that kind: the one CTA per SM gets as many warps as the two had.  (12 matrices of a 7B layer, 8 warps: 191 us
// with 8 decode warps an SM, 147 with 16.)
int decode_warps(const mv_q8_tuning *asked, const mv_q8_tuning &t) {
    if (!asked || asked->warps <= 0) return 0;
    return t.warps <= 8 ? 2 * t.warps : t.warps;
}

// parts = 0: whole stripes (stacks); otherwise split each stripe's segments into `parts`
void plan_job(Q8Job &J, const mv_q8_tuning &t, uint32_t &item, int parts) {
    J.ngroups = std::max(1, std::min(parts > 0 ? parts : 1, J.m.nseg));
    const int spp = (J.m.nseg + J.ngroups - 1) / J.ngroups;
    J.ngroups = (J.m.nseg + spp - 1) / spp;  // no empty part
    J.atomic = J.ngroups > 1;
    J.item0 = item;
    J.pad = 0;  // work-queue counter (job 0 of a stack) or item counter (chains)
    item += (uint32_t)((J.m.rows + 31) / 32) * (uint32_t)J.ngroups;
}

}  // namespace

bool q8s_supports(const mv_q8_view *m, const int8_t *x) {
    return (m->cols & 15) == 0 && ((uintptr_t)x & 15) == 0 && (m->seg_quads & 3) == 0;
}

// The launch shape a caller asks for (or the default one) has to fit shared memory: a decode table, `warps` x ilp x depth
// stream buffers and the tiles or sums of `warps`, whatever shape the kernel then runs in.  (Callers that try shapes count on
// the refusal; where a shape passes, the kernel finds one of its own.)
mv_status check_shape(const mv_q8_tuning &t, int ilp, int max_blk_rows, size_t table, size_t warp_bytes) {
    const size_t need = table + (size_t)t.warps * ilp * t.depth * (size_t)(max_blk_rows + 1) * 128 + warp_bytes;
    if (need > (size_t)max_smem_optin())
        return fail(MV_ERR_UNSUPPORTED, "Q8 launch: %d warps x %d segments x %d buffers need %zu B of shared memory (max %d)",
                    t.warps, ilp, t.depth, need, max_smem_optin());
    return MV_OK;
}
mv_status check_shape_int(const mv_q8_tuning &t, int nv, int max_blk_rows, uint32_t tbl_stripe_max) {
    const bool mma = t.engine == MV_ENGINE_AUTO && nv >= kMmaShape;
    return check_shape(t, mma ? 1 : t.ilp, max_blk_rows, 65536 + 2 * (size_t)tbl_stripe_max,
                       mma ? (size_t)std::max(0, t.warps - 8) * 4096 : (size_t)2 * t.warps * nv * 128);
}

// How one matrix is spread over the CTAs: whole stripes (parts = 1), every stripe in `parts` ranges of its segments, or
// the units in even shares (parts = 0), which only cuts the stripes at the borders between two CTAs' shares.
//
// Chosen by the time of the busiest CTA, in cycles: its units, at `step` a quad with all warps at work and `lone` a
// quad of a warp's own pace, and no less than its items' service by the table warps (a table build of ~6000 cycles, and
// the epilogue); to that, what joining cut stripes takes (zeroing launch, scaling launch, atomics).  Measured on a B200,
// whole stripes | even shares | the best aligned parts, 16 int8 vectors: 11008x4096 (3 items on some CTAs, 2 on others)
// 36.7 | 36.1 | 39.4 us, 6000x6000 33.1 | 28.8 | 30.6, 2400x11008 31.3 | 24.5 | 27.3, 500x2992 16.2 | 14.0 | 11.7; the
// same, one vector: 23.7 | 26.4 | 30.0, 23.0 | 22.3 | 23.4, 21.3 | 19.1 | 19.7, 11.2 | 11.6 | 9.3.  The backward adds to
// dX by atomics in any case: 11008x4096, 64 vectors, 132.8 | 121.9 us.
struct Cost {
    int step, lone;
    int service;     // cycles an item takes the table warps
    int join_parts;  // every stripe cut; and ~50 of a part's `outputs` a cycle are added
    long long outputs;
    int join_even;   // the stripes at the borders of the shares cut
};
int choose_parts(int nseg, int seg_quads, int stripes, const Cost &c) {
    constexpr long long kDecodeWarps = 14, kBuild = 4800;
    const long long G = sm_count();
    auto time = [&](long long units, long long items) {
        const long long rounds = (units + kDecodeWarps - 1) / kDecodeWarps;
        return std::max(seg_quads * std::max(rounds * c.lone, units * c.step) + items * kBuild, items * c.service) + c.service;
    };
    int best = 1;
    long long best_cost = -1;
    for (int p = 1; p <= 64 && p <= nseg; p++) {
        const long long items = ((long long)stripes * p + G - 1) / G;
        if (best_cost >= 0 && (items + 1) * c.service >= best_cost) break;  // (no larger p is better: time() is at least that)
        const long long cost = time(items * ((nseg + p - 1) / p), items) + (p > 1 ? c.join_parts + c.outputs * p / 50 : 0);
        if (best_cost < 0 || cost < best_cost) {
            best_cost = cost;
            best = p;
        }
    }
    const long long all = (long long)stripes * nseg;
    if (all > G && all < 0x7FFFFFFF) {
        const long long units = (all + G - 1) / G;
        if (time(units, units / nseg + 2) + c.join_even < best_cost) best = 0;
    }
    return best;
}

// The stripes that even shares cut: each border inside a stripe, the first of those in the same stripe.  kScale:
// the sums are complete, ys = y s (float form: in place); otherwise they are set to zero before the product.
template <typename T, bool kScale>
__global__ void __launch_bounds__(256) cut_stripes(T *y, float *ys, const float *scales, int rows, int batch, uint32_t nseg,
                                                   uint32_t span, uint32_t shares) {
    if (!kScale) grid_launch_dependents();
    const uint32_t b = blockIdx.x + 1, p = (uint32_t)((uint64_t)b * span / shares), stripe = p / nseg;
    const uint32_t q = (uint32_t)((uint64_t)(b - 1) * span / shares);
    if (p == stripe * nseg || q > stripe * nseg) return;
    const int row = (int)stripe * 32 + (int)(threadIdx.x & 31);
    if (row >= rows) return;
    const float s = kScale ? scales[row] : 0.f;
    for (int v = threadIdx.x >> 5; v < batch; v += 8) {
        const size_t i = (size_t)v * rows + row;
        if (kScale) ys[i] = (float)y[i] * s;
        else y[i] = 0;
    }
}
template <typename T, bool kScale>
mv_status cut_stripes_launch(const Q8WLaunch &L, T *y, float *ys, cudaStream_t st) {
    const uint32_t shares = std::min<uint32_t>(L.span, (uint32_t)sm_count());
    cut_stripes<T, kScale><<<shares - 1, 256, 0, st>>>(y, ys, L.job0.scales, L.job0.m.rows, L.batch, (uint32_t)L.job0.m.nseg,
                                                      L.span, shares);
    MV_CUDA_TRY(cudaGetLastError(), "cut_stripes launch");
    return MV_OK;
}

// Work items of a single-matrix launch: parts as asked for, or as chosen.  Returns the most units a CTA can get.
int plan_single(Q8WLaunch &L, const mv_q8_tuning &t, const Cost &c) {
    const mv_q8_view &m = L.job0.m;
    const int stripes = (m.rows + 31) / 32;
    const int parts = t.parts > 0 ? t.parts : choose_parts(m.nseg, m.seg_quads, stripes, c);
    uint32_t items = 0;
    plan_job(L.job0, t, items, parts > 0 ? parts : 1);
    L.jobs = nullptr;
    L.njobs = 1;
    L.nitems = items;
    L.span = 0;
    long long units;
    if (parts == 0) {
        L.nitems = L.span = (uint32_t)stripes * (uint32_t)m.nseg;
        units = (L.span + sm_count() - 1) / sm_count();
    } else {
        units = ((long long)items + sm_count() - 1) / sm_count() * ((m.nseg + L.job0.ngroups - 1) / L.job0.ngroups);
    }
    return (int)std::min<long long>(units, 1 << 20);
}

// Whether a product that q8s_supports refuses can run there all the same (q8s_matvec then takes it): its blocks must leave
// room for two decode tables.  The kernel for it is otherwise the CTA-per-stripe one of k_q8.cu.  Measured on a B200,
// that one | this: 4090x4100, 1, 2, 16 and 64 vectors 17.4 | 13.2, 19.9 | 13.9, 48.7 | 24.7, 193 | 82 us; 10001x5003,
// 41.8 | 29.3, 48.2 | 30.8, 93 | 61, 371 | 185; 12000x1602, 17.9 | 18.8, 21.0 | 20.0, 45.6 | 34.9, 181 | 78.
bool q8s_takes_ragged(const mv_q8_view *m, int batch) {
    Q8WLaunch L{};
    L.slot_bytes = (uint32_t)(m->max_blk_rows + 1) * 128u;
    L.tbl_stage = (int)((m->tbl_stripe_max + 7) & ~7u);
    L.batch = std::min(batch, 64);
    return m->max_blk_rows < (1 << 20) && q8w_ragged_fits(L, false) && (L.batch < kMmaMinVectors || q8w_ragged_fits(L, true));
}

// Single matrix through the persistent kernel (one inline job): passes of up to 64 vectors on the tensor cores, of
// up to 16 on the CUDA cores; ragged ones (see Q8WLaunch) too.
mv_status q8s_matvec(const mv_q8_view *m, const int8_t *x, int batch, int32_t *y, const float *scales, float *ys,
                     const mv_q8_tuning *tuning, cudaStream_t st) {
    mv_status rc;
    uint32_t *status = device_status_word(&rc);
    if (rc) return rc;
    const mv_q8_tuning t = resolve(tuning);
    const bool ragged = !q8s_supports(m, x);
    const int pass = t.engine == MV_ENGINE_AUTO ? 64 : 16;
    for (int v0 = 0; v0 < batch; v0 += pass) {
        const int nb = std::min(pass, batch - v0);
        const bool global_x = !ragged && m->seg_quads > kXQuads;
        bool mma = t.engine == MV_ENGINE_AUTO && nb >= (global_x ? kMmaMinGlobalX : kMmaMinVectors);
        if (!ragged) rc = check_shape_int(t, nv_round(nb), m->max_blk_rows, m->tbl_stripe_max);
        if (rc) return rc;
        Q8WLaunch L{};
        L.ragged = ragged;
        L.job0.m = *m;
        L.job0.x = x + (size_t)v0 * m->cols;
        L.job0.y = y + (size_t)v0 * m->rows;
        L.job0.scales = scales;
        L.job0.ys = ys ? ys + (size_t)v0 * m->rows : nullptr;
        const int nv = nv_round(nb);
        auto cost = [&](bool mma) {
            const int n = mma ? std::max(nb, kMmaMinVectors) : nb;  // (tuned from there on)
            return Cost{mma ? (n <= 16 ? 18 + n / 4 : 23) : 9 + nv, mma ? 220 : 90, 6000 + 100 * n, 3000 + 60 * n + (ys ? 1000 : 0),
                        (long long)n * m->rows, 6000 + 250 * n + (ys ? 4000 : 0)};
        };
        const bool choose = mma && nb < kMmaMinLone && !global_x;
        int units = plan_single(L, t, cost(mma && !choose));
        if (choose) {
            // More than a dp4a launch has warps for.  Not for ragged short rows, bound by their tables and outputs: dp4a |
            // tensor cores, 8 vectors, 16000x401 19.5 | 21.8 us, one table for all 14.2 | 15.3; 50000x129 42.6 | 45.8, one
            // table 22.9 | 29.9; 30000x803 33.8 | 36.9, one table 27.7 | 25.1.
            mma = units > 10 && !(ragged && m->cols <= (m->local ? 832 : 480));
            if (mma) units = plan_single(L, t, cost(true));
        }
        float *out = L.job0.ys;
        if (L.job0.atomic) L.job0.ys = nullptr;
        L.batch = nb;
        L.status = status;
        L.spin_limit = wait_spin_limit();
        L.drop_copy = inject_drop_copy();
        L.slot_bytes = (uint32_t)(m->max_blk_rows + 1) * 128u;
        L.tbl_stage = (int)((m->tbl_stripe_max + 7) & ~7u);
        L.early = v0 > 0 || L.job0.atomic || L.span;
        if (L.job0.atomic) {
            rc = zero_launch(L.job0.y, (size_t)nb * m->rows, st);
            if (rc) return rc;
        }
        if (L.span) {
            rc = cut_stripes_launch<int32_t, false>(L, L.job0.y, nullptr, st);
            if (rc) return rc;
        }
        rc = q8w_launch_int(L, nv, mma, decode_warps(tuning, t), units, st);
        if (rc) return rc;
        if (L.span && out) {
            rc = cut_stripes_launch<int32_t, true>(L, L.job0.y, out, st);
            if (rc) return rc;
        }
        if (ys && L.job0.atomic) {
            const size_t n = (size_t)nb * m->rows;
            scale_rows_kernel<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(L.job0.y, scales, ys + (size_t)v0 * m->rows, m->rows,
                                                               nb, m->rows);
            MV_CUDA_TRY(cudaGetLastError(), "scale_rows_kernel launch");
        }
    }
    return MV_OK;
}

// Float forward: passes of up to 64 vectors (8 with engine 1, on the CUDA cores) through the warp-specialised kernel.
mv_status q8_fwd(const mv_q8_view *m, const uint16_t *x, int batch, const float *scales, float *y,
                 const mv_q8_tuning *tuning, cudaStream_t st) {
    mv_status rc;
    uint32_t *status = device_status_word(&rc);
    if (rc) return rc;
    const mv_q8_tuning t = resolve(tuning);
    const bool asked = tuning && tuning->warps > 0;
    if (asked && t.warps > 8 && t.engine == MV_ENGINE_AUTO && batch >= 2)
        return fail(MV_ERR_ARG, "Q8 launch: %d warps per CTA; the float form on the tensor cores takes at most 8", t.warps);
    const bool dot = t.engine == MV_ENGINE_DP4A;
    rc = check_shape(t, 1, m->max_blk_rows, 32768, dot || batch == 1 ? 0 : (size_t)t.warps * 2048);
    if (rc) return rc;
    const int pass = dot ? 8 : 64;
    for (int v0 = 0; v0 < batch; v0 += pass) {
        Q8WLaunch L{};
        L.job0.m = *m;
        L.job0.x = reinterpret_cast<const int8_t *>(x + (size_t)v0 * m->cols);
        L.job0.scales = scales;
        L.job0.ys = y + (size_t)v0 * m->rows;
        L.batch = std::min(pass, batch - v0);
        // whole stripes, or even shares where no stripe is cut twice: a sum of two parts does not depend on their order
        // (whole | even: 11008x4096, one vector 28.3 | 31.4 us, 16 vectors 46.7 | 51.6, 64 vectors 54.5 | 63.1; 6000x6000, 16
        // vectors 46.7 | 45.1, 64 vectors 54.3 | 55.2)
        constexpr int kNever = 1 << 30;
        const bool cuda = dot || L.batch == 1;
        const Cost cost{cuda ? 11 + 4 * nv_round(L.batch) : 26 + L.batch / 16, cuda ? 90 : 220, 6000 + 100 * L.batch, kNever, 0,
                        t.parts <= 0 && (m->rows + 31) / 32 >= sm_count() ? 20000 : kNever};
        mv_q8_tuning by_rule = t;
        by_rule.parts = 0;
        const int units = plan_single(L, by_rule, cost);
        L.status = status;
        L.spin_limit = wait_spin_limit();
        L.drop_copy = inject_drop_copy();
        L.slot_bytes = (uint32_t)(m->max_blk_rows + 1) * 128u;
        L.tbl_stage = (int)((m->tbl_stripe_max + 7) & ~7u);
        L.early = v0 > 0 || L.span;
        if (L.span) {
            rc = cut_stripes_launch<float, false>(L, L.job0.ys, nullptr, st);
            if (rc) return rc;
        }
        rc = q8w_launch_fwd(L, dot, decode_warps(tuning, t), units, st);
        if (rc) return rc;
        if (L.span) {
            rc = cut_stripes_launch<float, true>(L, L.job0.ys, L.job0.ys, st);
            if (rc) return rc;
        }
    }
    return MV_OK;
}

// Transposed product: passes of 32 vectors (8 with engine 1, on the CUDA cores), added to dX by atomics, so that stripes may be split.  The tensor cores'
// sums leave by 16-byte reductions: a dX off that grid takes the one-vector form, whose reductions are scalars.
mv_status q8_bwd(const mv_q8_view *m, const uint16_t *dy, int batch, const float *scales, float *dx,
                 const mv_q8_tuning *tuning, cudaStream_t st) {
    mv_status rc;
    uint32_t *status = device_status_word(&rc);
    if (rc) return rc;
    mv_q8_tuning t = resolve(tuning);
    if (!tuning || (tuning->ilp != 1 && tuning->ilp != 2)) t.ilp = 1;  // the float form's default
    const bool mma = t.engine == MV_ENGINE_AUTO && batch >= 2;
    if (t.warps > 8) return fail(MV_ERR_ARG, "Q8 launch: %d warps per CTA; the float backward takes at most 8", t.warps);
    rc = check_shape(t, mma ? 1 : t.ilp, m->max_blk_rows, 32768, mma ? 4096 + (size_t)t.warps * 2048 : 0);
    if (rc) return rc;
    rc = zero_launch(dx, (size_t)batch * m->cols, st);
    if (rc) return rc;
    const bool dot = t.engine == MV_ENGINE_DP4A;
    const int pass = dot ? 8 : ((uintptr_t)dx & 15) ? 1 : 32;
    for (int v0 = 0; v0 < batch; v0 += pass) {
        Q8WLaunch L{};
        L.job0.m = *m;
        L.job0.x = reinterpret_cast<const int8_t *>(dy + (size_t)v0 * m->rows);
        L.job0.scales = scales;
        L.job0.ys = dx + (size_t)v0 * m->cols;
        L.batch = std::min(pass, batch - v0);
        const bool cuda = dot || L.batch == 1;
        const Cost cost{cuda ? 10 + 10 * nv_round(L.batch) : 28 + L.batch / 4, cuda ? 90 : 220, 6000, 0, 0, L.batch == 1 ? 10000 : 0};
        const int units = plan_single(L, t, cost);
        L.status = status;
        L.spin_limit = wait_spin_limit();
        L.drop_copy = inject_drop_copy();
        L.slot_bytes = (uint32_t)(m->max_blk_rows + 1) * 128u;
        L.tbl_stage = (int)((m->tbl_stripe_max + 7) & ~7u);
        L.early = 1;  // (dX has been zeroed)
        rc = q8w_launch_bwd(L, dot, decode_warps(tuning, t), units, st);
        if (rc) return rc;
    }
    return MV_OK;
}

}  // namespace mv

extern "C" {

mv_status mv_q8_matvec_bf16(const mv_q8_view *m, const uint16_t *x_dev, int batch, const float *row_scales_dev,
                            float *y_dev, const mv_q8_tuning *tuning, void *stream) {
    if (!m || !x_dev || !row_scales_dev || !y_dev || batch <= 0)
        return mv::fail(MV_ERR_ARG, "mv_q8_matvec_bf16: bad arguments");
    if ((m->cols & 15) || ((uintptr_t)x_dev & 15) || (m->seg_quads & 3))
        return mv::fail(MV_ERR_ARG, "mv_q8_matvec_bf16: needs cols %% 16 == 0, seg_quads %% 4 == 0, 16-byte aligned x");
    return mv::q8_fwd(m, x_dev, batch, row_scales_dev, y_dev, tuning, (cudaStream_t)stream);
}

mv_status mv_q8_matvec_t_bf16(const mv_q8_view *m, const uint16_t *dy_dev, int batch, const float *row_scales_dev,
                              float *dx_dev, const mv_q8_tuning *tuning, void *stream) {
    if (!m || !dy_dev || !row_scales_dev || !dx_dev || batch <= 0)
        return mv::fail(MV_ERR_ARG, "mv_q8_matvec_t_bf16: bad arguments");
    if ((m->cols & 15) || (m->seg_quads & 3))
        return mv::fail(MV_ERR_ARG, "mv_q8_matvec_t_bf16: needs cols %% 16 == 0 and seg_quads %% 4 == 0");
    return mv::q8_bwd(m, dy_dev, batch, row_scales_dev, dx_dev, tuning, (cudaStream_t)stream);
}

mv_status mv_q8_stack_plan(mv_q8_job *jobs, int njobs, const mv_q8_tuning *tuning, mv_q8_stack_info *info) {
    if (!jobs || njobs <= 0 || !info) return mv::fail(MV_ERR_ARG, "mv_q8_stack_plan: bad arguments");
    // The work queue hands out items in job order: jobs with the most work per item (decode steps of a
    // stripe's segment group) go first, so that the last items taken, which set the end of the launch, are
    // the shortest (stable: equal jobs keep their order).  Each job carries its own x and y, so the outputs
    // do not depend on the order.
    std::stable_sort(jobs, jobs + njobs, [&](const mv_q8_job &a, const mv_q8_job &b) {
        auto work = [&](const mv_q8_job &j) {
            const int parts = std::max(1, std::min(tuning && tuning->parts > 0 ? tuning->parts : 1, std::max(1, j.m.nseg)));
            return (long long)((std::max(1, j.m.nseg) + parts - 1) / parts) * std::max(1, j.m.seg_quads);
        };
        return work(a) > work(b);
    });
    return mv::stack_plan(jobs, njobs, tuning, info);
}

}  // extern "C"

namespace mv {

mv_status stack_plan(mv_q8_job *jobs, int njobs, const mv_q8_tuning *tuning, mv_q8_stack_info *info) {
    const mv_q8_tuning t = mv::resolve(tuning);
    uint32_t item = 0;
    info->max_blk_rows = 2;
    info->tbl_stripe_max = 2;
    for (int j = 0; j < njobs; j++) {
        const mv_q8_view &m = jobs[j].m;
        if (m.rows <= 0 || m.cols <= 0 || (m.cols & 15) || m.nseg <= 0 || m.seg_quads <= 0 || (m.seg_quads & 3) ||
            ((uintptr_t)jobs[j].x & 15))
            return mv::fail(MV_ERR_ARG,
                            "mv_q8_stack_plan: job %d: needs cols %% 16 == 0, seg_quads %% 4 == 0 and a "
                            "16-byte aligned x",
                            j);
        if ((uint64_t)item + (uint64_t)((m.rows + 31) / 32) * (uint64_t)m.nseg > 0xFFFFFFFFull)
            return mv::fail(MV_ERR_SHAPE, "mv_q8_stack_plan: too many work items");
        mv::plan_job(jobs[j], t, item, t.parts);
        info->max_blk_rows = std::max(info->max_blk_rows, m.max_blk_rows);
        info->tbl_stripe_max = std::max(info->tbl_stripe_max, m.tbl_stripe_max);
    }
    info->nitems = item;
    info->atomic_jobs = 0;
    for (int j = 0; j < njobs; j++) info->atomic_jobs += jobs[j].atomic ? 1 : 0;
    info->warps = t.warps;
    info->ilp = t.ilp;
    info->depth = t.depth;
    return MV_OK;
}

}  // namespace mv

extern "C" {

size_t mv_q8_x_tiles_bytes(const mv_q8_view *m) {
    if (!m || m->nseg <= 0 || m->seg_quads <= 0) return 0;
    return (size_t)m->nseg * (size_t)((m->seg_quads + 31) / 32) * 2048;
}

mv_status mv_q8_chain_plan(mv_q8_job *jobs, int njobs, const mv_q8_tuning *tuning, mv_q8_stack_info *info) {
    if (!jobs || njobs <= 0 || !info) return mv::fail(MV_ERR_ARG, "mv_q8_chain_plan: bad arguments");
    for (int j = 0; j + 1 < njobs; j++)
        if (jobs[j].m.rows != jobs[j + 1].m.cols)
            return mv::fail(MV_ERR_SHAPE, "mv_q8_chain_plan: job %d has %d rows but job %d has %d columns", j,
                            jobs[j].m.rows, j + 1, jobs[j + 1].m.cols);
    mv_q8_tuning t = mv::resolve(tuning);
    if (t.parts > 1) return mv::fail(MV_ERR_ARG, "mv_q8_chain_plan: a chain needs whole stripes (parts <= 1)");
    t.parts = 0;
    return mv::stack_plan(jobs, njobs, &t, info);  // a chain keeps its order
}

mv_status mv_q8_chain_matvec(mv_q8_job *jobs_dev, int njobs, const mv_q8_stack_info *info, int batch,
                             const float *chain_scales_dev, int8_t *out8_dev, const mv_q8_tuning *tuning,
                             void *stream) {
    if (!jobs_dev || njobs <= 0 || !info || batch <= 0 || batch > 16 || !chain_scales_dev || !out8_dev)
        return mv::fail(MV_ERR_ARG, "mv_q8_chain_matvec: bad arguments (batch must be 1..16)");
    mv_q8_tuning t = mv::resolve(tuning);
    if (t.parts > 1) return mv::fail(MV_ERR_ARG, "mv_q8_chain_matvec: a chain needs whole stripes (parts <= 1)");
    if (t.warps != info->warps || t.ilp != info->ilp)
        return mv::fail(MV_ERR_ARG, "mv_q8_chain_matvec: tuning differs from the one the jobs were planned with");
    cudaStream_t st = (cudaStream_t)stream;
    mv_status rc;
    mv::Q8WLaunch L{};
    L.status = mv::device_status_word(&rc);
    if (rc) return rc;
    L.jobs = jobs_dev;
    L.njobs = njobs;
    L.nitems = info->nitems;
    L.batch = batch;
    L.spin_limit = mv::wait_spin_limit();
    L.drop_copy = mv::inject_drop_copy();
    L.slot_bytes = (uint32_t)(info->max_blk_rows + 1) * 128u;
    L.tbl_stage = (int)((info->tbl_stripe_max + 7) & ~7u);
    L.chain_scales = chain_scales_dev;
    L.chain_out8 = out8_dev;
    const int nv = mv::nv_round(batch);
    const bool mma = t.engine == MV_ENGINE_AUTO && batch >= mv::kMmaMinGlobalX;
    rc = mv::check_shape_int(t, nv, info->max_blk_rows, info->tbl_stripe_max);
    if (rc) return rc;
    mv::q8s_chain_reset<<<(njobs + 255) / 256, 256, 0, st>>>(reinterpret_cast<mv::Q8Job *>(jobs_dev), njobs);
    MV_CUDA_TRY(cudaGetLastError(), "q8s_chain_reset launch");
    return mv::q8w_launch_int(L, nv, mma, mv::decode_warps(tuning, t), 1 << 20, st);
}

mv_status mv_q8_stack_matvec(const mv_q8_job *jobs_dev, int njobs, const mv_q8_stack_info *info, int batch,
                             const mv_q8_tuning *tuning, void *stream) {
    if (!jobs_dev || njobs <= 0 || !info || batch <= 0 || batch > 16)
        return mv::fail(MV_ERR_ARG, "mv_q8_stack_matvec: bad arguments (batch must be 1..16)");
    const mv_q8_tuning t = mv::resolve(tuning);
    if (t.warps != info->warps || t.ilp != info->ilp)
        return mv::fail(MV_ERR_ARG, "mv_q8_stack_matvec: tuning differs from the one the jobs were planned with");
    cudaStream_t st = (cudaStream_t)stream;
    mv_status rc;
    mv::Q8WLaunch L{};
    L.status = mv::device_status_word(&rc);
    if (rc) return rc;
    L.jobs = jobs_dev;
    L.njobs = njobs;
    L.nitems = info->nitems;
    L.batch = batch;
    L.spin_limit = mv::wait_spin_limit();
    L.drop_copy = mv::inject_drop_copy();
    L.slot_bytes = (uint32_t)(info->max_blk_rows + 1) * 128u;
    L.tbl_stage = (int)((info->tbl_stripe_max + 7) & ~7u);
    // work queue: jobs_dev[0].pad, zero after planning and after every completed launch
    if (info->nitems < 0x7FFFFFFFu) L.queue = const_cast<uint32_t *>(&jobs_dev[0].pad);
    const int nv = mv::nv_round(batch);
    const bool mma = t.engine == MV_ENGINE_AUTO && nv >= mv::kMmaMinVectors;
    rc = mv::check_shape_int(t, nv, info->max_blk_rows, info->tbl_stripe_max);
    if (rc) return rc;
    dim3 zg(64, std::min(njobs, 1024));
    L.early = info->atomic_jobs > 0;
    if (info->atomic_jobs > 0) {
        mv::q8s_zero_atomic_y<<<zg, 256, 0, st>>>(jobs_dev, njobs, batch);
        MV_CUDA_TRY(cudaGetLastError(), "q8s_zero_atomic_y launch");
    }
    rc = mv::q8w_launch_int(L, nv, mma, mv::decode_warps(tuning, t), 1 << 20, st);
    if (rc) return rc;
    if (info->atomic_jobs > 0) {
        mv::q8s_scale_atomic_y<<<zg, 256, 0, st>>>(jobs_dev, njobs, batch);
        MV_CUDA_TRY(cudaGetLastError(), "q8s_scale_atomic_y launch");
    }
    return MV_OK;
}

mv_status mv_q8_matvec_tuned(const mv_q8_view *m, const int8_t *x_dev, int batch, int32_t *y_dev,
                             const float *row_scales_dev, float *y_scaled_dev, const mv_q8_tuning *tuning,
                             void *stream) {
    if (!m || !x_dev || !y_dev || batch <= 0) return mv::fail(MV_ERR_ARG, "mv_q8_matvec_tuned: bad arguments");
    if (y_scaled_dev && !row_scales_dev) return mv::fail(MV_ERR_ARG, "mv_q8_matvec_tuned: y_scaled needs scales");
    if (!mv::q8s_supports(m, x_dev))
        return mv::fail(MV_ERR_ARG,
                        "mv_q8_matvec_tuned: needs cols %% 16 == 0, seg_quads %% 4 == 0 and 16-byte aligned x");
    return mv::q8s_matvec(m, x_dev, batch, y_dev, row_scales_dev, y_scaled_dev, tuning, (cudaStream_t)stream);
}

}  // extern "C"

// Decode + int8 matvec for the reference's matvansWarpPerRow (WPR) layout on
// sm_100a.  Parity target: matvansWarpPerRow/matvansWarpPerRow-kernel.cu:46-175.
//
// One warp per row; lane l owns columns 512k + 16l .. 512k + 16l + 15 and its
// own 16-bit word stream (word k at payload[cursor + (k/8)*256 + 8l + k%8],
// create_matrices_WarpPerRow.py:405-420).  Decode step: q = head & 0xFF,
// r = ppf[q], w = min + r, head = (head >> 8) * prob(r) + (q - cdf[r]), refill
// 16 bits when head < 2^16 (kernel.cu:120-157).
//
// What bounds it: issue.  A step (one symbol per lane) takes ~13 instructions
// against 34 in the form this replaced, whose refill recomputed a global word
// index, checked it and reloaded a word at every symbol:
//   * the lane's stream passes through a ring of its own in shared memory, word k
//     at byte 64 k + 2 lane, filled 8 words (one 16-byte load, requested a chunk
//     ahead) at a time between groups of 16 symbols, so that a refill is a merge,
//     a 16-bit load and an add, all predicated; bounds are checked per chunk, and
//     an overrun once per row from the number of words taken;
//   * decode table: one 4-byte entry {prob, 0, symbol, q - cdf} per (quantile,
//     lane) at byte q*256 + lane*4, one byte permute per address;
//   * one CTA per SM with as many warps (up to 28) as spread the rows evenly over
//     the SMs: 4096 rows are 28 warps on each, all in one round.
// Measured on a B200, 4096x4096, one vector: 29.4 us before, 14.8 us with the ring
// and the packed entries.
// Four decoded symbols go through one dp4a; any number of vectors share a decode.
#include <cooperative_groups.h>

#include <algorithm>

#include "mv_device.cuh"

namespace mv {

struct WprLaunch {
    const uint16_t *payload;
    size_t payload_size;
    const uint32_t *cursors;
    int8_t min_value;
    const uint8_t *cdf;
    int G;
    const uint8_t *ppf;
    int rows, cols;
    const int8_t *x;
    int batch;
    int32_t *y;
    const float *scales;
    float *ys;
    uint32_t *status;
    int warps;  // of a CTA, those that take rows; the others help with the table alone
};

constexpr uint32_t kRingBytes = 32 * 64;               // 32 words of 32 lanes
constexpr uint32_t kRingAlloc = kRingBytes + 16 * 64;  // the first 16 words again behind the ring: a group of 16
                                                       // symbols runs past its end without wrapping
template <int NV>
constexpr int kWprWarps = NV <= 4 ? 28 : NV <= 8 ? 16 : 12;

// Words [ix, ix + 8) of the payload; zeros past its end.
__device__ __forceinline__ uint4 wpr_chunk(const WprLaunch &L, uint64_t ix) {
    if (ix + 8 <= L.payload_size && (ix & 7) == 0) return ldp(reinterpret_cast<const uint4 *>(L.payload + ix));
    uint32_t w[4];
#pragma unroll
    for (int j = 0; j < 4; j++) {
        const uint64_t i = ix + 2 * j;
        w[j] = (i < L.payload_size ? (uint32_t)ldp(L.payload + i) : 0u) |
               (i + 1 < L.payload_size ? (uint32_t)ldp(L.payload + i + 1) << 16 : 0u);
    }
    return make_uint4(w[0], w[1], w[2], w[3]);
}

template <int NV>
__global__ void __launch_bounds__(32 * kWprWarps<NV>) wpr_kernel(const WprLaunch L) {
    extern __shared__ __align__(1024) unsigned char smem[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, W = L.warps;
    grid_dependency_wait();  // (the launch before this one may have written the tables, the payload or x)
    grid_launch_dependents();
    // decode table: eight threads per quantile, four lane columns each
    bool bad = false;
#pragma unroll 4
    for (uint32_t i = threadIdx.x; i < 256 * 8; i += blockDim.x) {
        const uint32_t q = i >> 3, r = ldp(L.ppf + q);
        uint32_t e = 0;
        if ((int)r + 1 > L.G) {
            bad = true;
        } else {
            const uint32_t c0 = ldp(L.cdf + r), c1 = ldp(L.cdf + r + 1);
            bad |= c0 > q;  // (q - c0 is never negative for a valid table)
            e = ((c1 - c0) & 0xFFu) | (uint32_t)(uint8_t)(int8_t)(L.min_value + (int)r) << 16 | (q - c0) << 24;
        }
        const uint4 e4 = make_uint4(e, e, e, e);
        uint4 *dst = reinterpret_cast<uint4 *>(smem + 256u * q + 16u * (i & 7u));
        *dst = e4;
    }
    if (bad) atomicOr(L.status, MV_DEV_BAD_TABLE);
    __syncthreads();
    if (warp >= W) return;

    const uint32_t lane4 = (uint32_t)lane * 4u;
    const uint32_t ring = smem_u32(smem) + 65536u + (uint32_t)warp * kRingAlloc + (uint32_t)lane * 2u;
    const int groups = L.cols / 512;
    for (int row = blockIdx.x * W + warp; row < L.rows; row += gridDim.x * W) {
        const uint64_t ix0 = (uint64_t)ldp(L.cursors + row) + 8u * (uint32_t)lane;
        uint32_t staged = 0;  // words in the ring so far; the chunk behind them is in `nxt`
        uint4 nxt = wpr_chunk(L, ix0);
        const uint4 c0 = nxt;
        auto stage = [&]() {
            const uint32_t s = staged & 31u, d = ring + s * 64u;
            const uint32_t w[4] = {nxt.x, nxt.y, nxt.z, nxt.w};
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const uint16_t lo = (uint16_t)w[j], hi = (uint16_t)(w[j] >> 16);
                asm volatile("st.shared.u16 [%0], %1;" ::"r"(d + 128u * j), "h"(lo) : "memory");
                asm volatile("st.shared.u16 [%0], %1;" ::"r"(d + 128u * j + 64u), "h"(hi) : "memory");
                if (s < 16u) {
                    asm volatile("st.shared.u16 [%0], %1;" ::"r"(d + 128u * j + kRingBytes), "h"(lo) : "memory");
                    asm volatile("st.shared.u16 [%0], %1;" ::"r"(d + 128u * j + 64u + kRingBytes), "h"(hi) : "memory");
                }
            }
            staged += 8u;
            nxt = wpr_chunk(L, ix0 + 32ull * staged);  // 256 words a chunk of 8
        };
        stage();
        stage();
        stage();
        // head from words 0 and 1; nw is the next word, a the place of the one after it
        uint32_t head = __byte_perm(c0.x, 0u, 0x1032), nw = c0.y & 0xFFFFu, a = ring + 3u * 64u;
        uint32_t left = staged - 3u;  // staged words from a on
        int acc[NV];
#pragma unroll
        for (int v = 0; v < NV; v++) acc[v] = 0;
        const int8_t *xp = L.x + 16 * lane;
        for (int g = 0; g < groups; g++, xp += 512) {
            uint4 xv[NV];
#pragma unroll
            for (int v = 0; v < NV; v++)
                xv[v] = v < L.batch ? ldp(reinterpret_cast<const uint4 *>(xp + (size_t)v * L.cols)) : make_uint4(0, 0, 0, 0);
            const uint32_t a0 = a;
#pragma unroll
            for (int k = 0; k < 4; k++) {
                uint32_t e[4];
#pragma unroll
                for (int t = 0; t < 4; t++) {
                    e[t] = *reinterpret_cast<const uint32_t *>(smem + __byte_perm(head, lane4, 0x7604));
                    // entry bytes (prob, 0, symbol, bias): two of them by dot products, off the permutes' pipe
                    head = (head >> 8) * (e[t] & 0xFFu) + __dp4a(e[t], 0x01000000u, 0u);
                    asm volatile(
                        "{\n\t.reg .pred p;\n\t.reg .u16 h;\n\t"
                        "setp.lo.u32 p, %0, 0x10000;\n\t"
                        "@p prmt.b32 %0, %1, %0, 0x5410;\n\t"  // (head << 16) | nw
                        "@p ld.shared.u16 %1, [%2];\n\t"
                        "@p add.u32 %2, %2, 64;\n\t}"
                        : "+r"(head), "+r"(nw), "+r"(a)::"memory");
                }
                const uint32_t wq = __byte_perm(__byte_perm(e[0], e[1], 0x0062), __byte_perm(e[2], e[3], 0x0062), 0x5410);
#pragma unroll
                for (int v = 0; v < NV; v++) {
                    const uint32_t xw = k == 0 ? xv[v].x : k == 1 ? xv[v].y : k == 2 ? xv[v].z : xv[v].w;
                    acc[v] = __dp4a((int)wq, (int)xw, acc[v]);
                }
            }
            // a group takes at most 16 words; with 18 left the next one cannot run dry
            left -= (a - a0) >> 6;
            if (a - ring >= kRingBytes) a -= kRingBytes;
            if (__any_sync(0xffffffffu, left < 18u)) {
                if (left < 18u) stage(), left += 8u;
                if (__any_sync(0xffffffffu, left < 18u)) {
                    if (left < 18u) stage(), left += 8u;
                }
            }
        }
        // the coder ends in its initial head 1 << 16 (create_matrices_WarpPerRow.py:271,372)
        if (head != (1u << 16)) atomicOr(L.status, MV_DEV_FINAL_STATE);
        const uint32_t k = staged - left - 2u;  // the last word taken into the head
        if (ix0 + 256ull * (k >> 3) + (k & 7u) >= L.payload_size) atomicOr(L.status, MV_DEV_STREAM_OVERRUN);
#pragma unroll
        for (int v = 0; v < NV; v++) acc[v] = __reduce_add_sync(0xffffffffu, acc[v]);
        if (lane == 0) {
#pragma unroll
            for (int v = 0; v < NV; v++)
                if (v < L.batch) {
                    L.y[(size_t)v * L.rows + row] = acc[v];
                    if (L.ys) L.ys[(size_t)v * L.rows + row] = (float)acc[v] * L.scales[row];
                }
        }
    }
}

// matvansWarpPerRow.cu:51-72 + 167-172 without the host round trip.
__global__ void absmax_kernel(const int32_t *y, int n, uint32_t *m) {
    uint32_t local = 0;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const int v = y[i];
        const uint32_t a = v < 0 ? (uint32_t)(-(int64_t)v) : (uint32_t)v;
        local = max(local, a);
    }
    for (int o = 16; o > 0; o >>= 1) local = max(local, __shfl_xor_sync(0xffffffffu, local, o));
    if ((threadIdx.x & 31) == 0) atomicMax(m, local);
}

__global__ void requant_kernel(const int32_t *y, int n, const uint32_t *m, int8_t *out8, float *delta) {
    // thrust's transform_reduce there yields float(max |y|) (AbsValue returns float)
    const float absmax = (float)(int)(float)*m;
    const float d = absmax / 127.0f;
    if (blockIdx.x == 0 && threadIdx.x == 0 && delta) *delta = d;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        out8[i] = (int8_t)__float2int_rn((float)y[i] / d);
}

// The same in one launch for n up to kRequantMax: one cluster of up to 8 CTAs holds y in registers, exchanges the CTAs'
// maxima through their shared memory and quantises.  Bound by launch latency, which a memset and two kernels pay three
// times: on a B200, 4096 elements 6.4 -> 3.7 us, 131072 9.3 -> 5.1 us.  Launched while the kernel before it ends (it waits
// for it before it reads): WPR 4096x4096 and this, the calls, 22.5 -> 20.3 us.
constexpr int kRequantEach = 16, kRequantMax = 8 * 1024 * kRequantEach;

__global__ void __launch_bounds__(1024) requant_cluster_kernel(const int32_t *y, int n, uint32_t *m, int8_t *out8, float *delta) {
    namespace cg = cooperative_groups;
    cg::cluster_group cluster = cg::this_cluster();
    __shared__ uint32_t warp_max[32], cta_max[8];
    const int step = (int)gridDim.x * 1024, i0 = (int)(blockIdx.x * 1024 + threadIdx.x);
    cluster_arrive_relaxed();  // (this CTA runs; waited for before the others' shared memory is written)
    grid_dependency_wait();    // y may be the launch before's
    int v[kRequantEach];
    uint32_t local = 0;
#pragma unroll
    for (int j = 0; j < kRequantEach; j++) {
        const int i = i0 + j * step;
        v[j] = i < n ? y[i] : 0;
        local = max(local, v[j] < 0 ? (uint32_t)(-(int64_t)v[j]) : (uint32_t)v[j]);
    }
    local = __reduce_max_sync(0xffffffffu, local);
    if ((threadIdx.x & 31) == 0) warp_max[threadIdx.x >> 5] = local;
    __syncthreads();
    cluster_wait();
    if (threadIdx.x < 32) {
        const uint32_t mine = __reduce_max_sync(0xffffffffu, warp_max[threadIdx.x]);
        if (threadIdx.x < gridDim.x) *cluster.map_shared_rank(&cta_max[blockIdx.x], threadIdx.x) = mine;
    }
    cluster.sync();
    uint32_t total = 0;
    for (unsigned c = 0; c < gridDim.x; c++) total = max(total, cta_max[c]);
    const float absmax = (float)(int)(float)total;
    const float d = absmax / 127.0f;
    if (i0 == 0) {
        *m = total;
        if (delta) *delta = d;
    }
#pragma unroll
    for (int j = 0; j < kRequantEach; j++) {
        const int i = i0 + j * step;
        if (i < n) out8[i] = (int8_t)__float2int_rn((float)v[j] / d);
    }
}

namespace {

template <int NV>
mv_status launch_wpr(const WprLaunch &L0, cudaStream_t st) {
    WprLaunch L = L0;
    // (the limit of the form that kept x in shared memory)
    if (256 * 32 * 4 + (size_t)NV * L.cols > (size_t)max_smem_optin())
        return fail(MV_ERR_UNSUPPORTED, "WPR: %d columns x %d vectors exceed shared memory", L.cols, NV);
    // rows in even rounds over the SMs
    const int sms = sm_count(), rounds = (L.rows + sms * kWprWarps<NV> - 1) / (sms * kWprWarps<NV>);
    const int W = std::max(1, (L.rows + sms * rounds - 1) / (sms * rounds));
    const size_t smem = 65536 + (size_t)W * kRingAlloc;
    auto kern = wpr_kernel<NV>;
    // a table by fewer than 8 warps takes longer than short rows (512x1024, 4 rows a CTA: 7.2 us with 4 warps, 5.3 with 8)
    const int threads = 32 * std::max(W, 8);
    mv_status rc = prepare_kernel((const void *)kern, smem, threads, nullptr);
    if (rc) return rc;
    L.warps = W;
    const int grid = std::max(1, std::min((L.rows + W - 1) / W, sms));
    MV_CUDA_TRY(launch_dependent(kern, dim3(grid), dim3(threads), smem, st, L), "wpr kernel launch");
    return MV_OK;
}

}  // namespace

mv_status wpr_matvec(const uint16_t *payload, size_t payload_size, const uint32_t *cursors,
                     int8_t min_value, const uint8_t *cdf, int G, const uint8_t *ppf, int rows, int cols,
                     const int8_t *x, int batch, int32_t *y, const float *scales, float *ys,
                     cudaStream_t st) {
    if (!payload || !cursors || !cdf || !ppf || !x || !y) return fail(MV_ERR_ARG, "mv_wpr_matvec: NULL pointer");
    if (rows <= 0 || cols <= 0 || batch <= 0 || G < 1) return fail(MV_ERR_ARG, "mv_wpr_matvec: bad sizes");
    if (cols % 512) return fail(MV_ERR_SHAPE, "WPR layout needs cols %% 512 == 0 (cols=%d)", cols);
    if (((uintptr_t)payload & 15) || ((uintptr_t)x & 15))
        return fail(MV_ERR_ARG, "mv_wpr_matvec: payload and x must be 16-byte aligned");
    if (ys && !scales) return fail(MV_ERR_ARG, "mv_wpr_matvec: y_scaled needs row scales");
    if (payload_size >= 0xF0000000u) return fail(MV_ERR_UNSUPPORTED, "mv_wpr_matvec: payload of 0xF0000000 words or more");
    mv_status rc;
    WprLaunch L{};
    L.status = device_status_word(&rc);
    if (rc) return rc;
    L.payload = payload;
    L.payload_size = payload_size;
    L.cursors = cursors;
    L.min_value = min_value;
    L.cdf = cdf;
    L.G = G;
    L.ppf = ppf;
    L.rows = rows;
    L.cols = cols;
    for (int v0 = 0; v0 < batch; v0 += 16) {
        const int nb = std::min(16, batch - v0);
        WprLaunch P = L;
        P.x = x + (size_t)v0 * cols;
        P.batch = nb;
        P.y = y + (size_t)v0 * rows;
        P.scales = scales;
        P.ys = ys ? ys + (size_t)v0 * rows : nullptr;
        if (nb == 1) rc = launch_wpr<1>(P, st);
        else if (nb == 2) rc = launch_wpr<2>(P, st);
        else if (nb <= 4) rc = launch_wpr<4>(P, st);
        else if (nb <= 8) rc = launch_wpr<8>(P, st);
        else rc = launch_wpr<16>(P, st);
        if (rc) return rc;
    }
    return MV_OK;
}

mv_status requant_absmax(const int32_t *y, int n, int8_t *out8, float *delta, uint32_t *scratch,
                         cudaStream_t st) {
    if (!y || !out8 || !scratch || n <= 0) return fail(MV_ERR_ARG, "mv_requant_absmax: bad arguments");
    if (n <= kRequantMax) {
        unsigned ctas = 1;
        while (ctas < 8 && n > (int)ctas * 4096) ctas *= 2;
        cudaLaunchAttribute attr[2];
        attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[1].val.programmaticStreamSerializationAllowed = 1;
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = ctas;
        attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
        cudaLaunchConfig_t cfg{};
        cfg.gridDim = dim3(ctas);
        cfg.blockDim = dim3(1024);
        cfg.stream = st;
        cfg.attrs = attr;
        cfg.numAttrs = 2;
        MV_CUDA_TRY(cudaLaunchKernelEx(&cfg, requant_cluster_kernel, y, n, scratch, out8, delta), "requant launch");
        return MV_OK;
    }
    MV_CUDA_TRY(cudaMemsetAsync(scratch, 0, sizeof(uint32_t), st), "cudaMemsetAsync(absmax)");
    const int grid = std::max(1, std::min((n + 255) / 256, 4 * sm_count()));
    absmax_kernel<<<grid, 256, 0, st>>>(y, n, scratch);
    requant_kernel<<<grid, 256, 0, st>>>(y, n, scratch, out8, delta);
    MV_CUDA_TRY(cudaGetLastError(), "requant kernels launch");
    return MV_OK;
}

}  // namespace mv

extern "C" {

mv_status mv_wpr_matvec(const uint16_t *payload_dev, size_t payload_size, const uint32_t *cursors_dev,
                        int8_t min_value, const uint8_t *cdf_dev, int G, const uint8_t *ppf_dev, int rows,
                        int cols, const int8_t *x_dev, int batch, int32_t *y_dev,
                        const float *row_scales_dev, float *y_scaled_dev, void *stream) {
    return mv::wpr_matvec(payload_dev, payload_size, cursors_dev, min_value, cdf_dev, G, ppf_dev, rows, cols,
                          x_dev, batch, y_dev, row_scales_dev, y_scaled_dev, (cudaStream_t)stream);
}

mv_status mv_requant_absmax(const int32_t *y_dev, int n, int8_t *out8_dev, float *delta_dev,
                            uint32_t *absmax_scratch_dev, void *stream) {
    return mv::requant_absmax(y_dev, n, out8_dev, delta_dev, absmax_scratch_dev, (cudaStream_t)stream);
}

}  // extern "C"

// fp32 projections of a multi-head attention layer on the fp16 tensor cores of sm_100a: out = x @ W^T + bias for up to
// three (x, W) pairs in one launch, operands carried as hi + lo fp16 pairs and every product as three tcgen05 MMAs.
//
// It stands where tensorax runs F.linear four times around its attention (tensorax/nn/attention/layers.py:112-128,
// tensorax/functional.py:105-110); the single-call form of that function stays on linear_tc.cuh.  Against that kernel
// (three TF32 products, split inside the GEMM): fp16 MMAs run at twice the TF32 rate, and the split is done once per
// tensor instead of once per tile, so shared memory -- which bounded the TF32 form: 16 KB of tile became 96 KB of
// traffic per k-step -- carries the operands and nothing else.
//
//   split_rows_kernel   one warp per row of x or W: the row is scaled by a power of two that brings its largest element
//                       to [2^13, 2^14), then hi = rn16(x), lo = rn16(x - hi).  With the scale a pair is exact to 2^-39
//                       of the row's maximum and to 22 bits down to 2^-17 of it, whatever the row's magnitude.  A row in
//                       which more than one element in 16 lies below that (an outlier and little else) raises a flag.
//   gemm_x3_kernel      persistent, one CTA per SM, 128 x BN tiles.  The tensor core's fp32 accumulation truncates, so a
//                       tensor-memory accumulator takes two stages (K = 128) only, a stage's small products first, so
//                       that few of its 24 MMAs add at full magnitude; two accumulators ping-pong and two warpgroups
//                       fold them into fp32 register sums, rounded to nearest.
//                       warp 0 TMA producer, warp 1 MMA issuer, warps 4-7 / 8-11 sums and results of the left / right
//                       half of a tile's columns (thread = row); results are turned through shared memory so that a
//                       warp stores whole 128-byte pieces of rows, head-split, fp32 or fp16.
//                       With the flag raised the CTA computes its tiles from the fp32 operands on CUDA cores instead.
// Bound: L2 -> SM traffic (a 128 x 256 tile brings 96 KB per 64 k, 128 FLOP per byte) next to the tensor pipe.  Measured, B4
// S1024 E1024 (three projections, then the output's): 94 us together = 1.1 PFLOP/s of fp16 MMAs; folding after every stage
// 103 us, after four 93; CTA pairs on 256 x 256 tiles (cta_group::2, 64 KB per 64 k and SM) 95 us, 128 x 128 tiles 99 us.
// Every mbarrier wait is bounded.
#pragma once
#include "linear_simt.cuh"
#include "ptx.cuh"

namespace txb {

enum : int { GX3_ERR_PRODUCER = 42, GX3_ERR_MMA = 43, GX3_ERR_SUMS = 44 };

// ------------------------------------------------------------------ split
struct SplitRowsSeg {
    const float *x;           // [rows, K], or [rows / S, heads, S, K / heads] when heads > 0
    __half *hi, *lo;          // [rows, K]
    float *inv;               // [rows] the factor that undoes the row's scale
    int rows, heads, S;
    int first;                // rows of the segments before this one
};
constexpr int kSplitRowsSegs = 7;          // q, k, v inputs and four weights
struct SplitRowsParams {
    SplitRowsSeg seg[kSplitRowsSegs];
    int n_segs, rows, K;      // rows: of all segments
    int *outliers;            // set where some row is not carried well
};

__global__ void __launch_bounds__(256) split_rows_kernel(const SplitRowsParams p)
{
    const int lane = threadIdx.x & 31;
    const int g = (int)blockIdx.x * 8 + (threadIdx.x >> 5);
    ptx::grid_trigger();
    ptx::grid_wait();
    if (g >= p.rows) return;
    int t = 0;
#pragma unroll
    for (int i = 1; i < kSplitRowsSegs; ++i)
        if (i < p.n_segs && g >= p.seg[i].first) t = i;
    const SplitRowsSeg s = p.seg[t];
    const int row = g - s.first;
    const int dh = s.heads > 0 ? p.K / s.heads : p.K;
    const float *base = s.heads > 0 ? s.x + ((size_t)(row / s.S) * s.heads * s.S + row % s.S) * dh : s.x + (size_t)row * p.K;
    const size_t head_step = (size_t)s.S * dh;
    auto load = [&](int k) {
        return *reinterpret_cast<const float4 *>(s.heads > 0 ? base + (size_t)(k / dh) * head_step + k % dh : base + k);
    };
    // rows of up to 1024 elements stay in registers between the two passes, longer ones are read again (from L1)
    float4 keep[8];
    int mx = 0;                                   // bits of the largest magnitude: integers order as the floats do
    auto big = [](float4 v) {
        return max(max(__float_as_int(fabsf(v.x)), __float_as_int(fabsf(v.y))), max(__float_as_int(fabsf(v.z)), __float_as_int(fabsf(v.w))));
    };
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int k = (i * 32 + lane) * 4;
        if (k < p.K) { keep[i] = load(k); mx = max(mx, big(keep[i])); }
    }
    for (int k = 1024 + lane * 4; k < p.K; k += 128) mx = max(mx, big(load(k)));
    mx = __reduce_max_sync(0xffffffffu, mx);
    // 2^e: exponent that brings the maximum to [2^13, 2^14); both 2^e and 2^-e are normal floats
    const int e = mx == 0 ? 0 : min(126, max(-126, 13 - ((mx >> 23) - 127)));
    const float scale = __int_as_float((e + 127) << 23);
    if (lane == 0) s.inv[row] = __int_as_float((127 - e) << 23);
    int small = 0;                                // elements that keep fewer than 22 bits
    auto is_small = [](float v) { return v != 0.f && fabsf(v) < 0.125f; };
    auto put = [&](int k, float4 v) {
        v.x *= scale; v.y *= scale; v.z *= scale; v.w *= scale;
        small += (int)is_small(v.x) + (int)is_small(v.y) + (int)is_small(v.z) + (int)is_small(v.w);
        const __half2 h01 = __floats2half2_rn(v.x, v.y), h23 = __floats2half2_rn(v.z, v.w);
        const float2 b01 = __half22float2(h01), b23 = __half22float2(h23);
        const __half2 l01 = __floats2half2_rn(v.x - b01.x, v.y - b01.y), l23 = __floats2half2_rn(v.z - b23.x, v.w - b23.y);
        uint2 hh, ll;
        hh.x = *reinterpret_cast<const uint32_t *>(&h01); hh.y = *reinterpret_cast<const uint32_t *>(&h23);
        ll.x = *reinterpret_cast<const uint32_t *>(&l01); ll.y = *reinterpret_cast<const uint32_t *>(&l23);
        *reinterpret_cast<uint2 *>(s.hi + (size_t)row * p.K + k) = hh;
        *reinterpret_cast<uint2 *>(s.lo + (size_t)row * p.K + k) = ll;
    };
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int k = (i * 32 + lane) * 4;
        if (k < p.K) put(k, keep[i]);
    }
    for (int k = 1024 + lane * 4; k < p.K; k += 128) put(k, load(k));
    small = __reduce_add_sync(0xffffffffu, small);
    if (lane == 0 && small > p.K / 16) atomicOr(p.outliers, 1);
}

// ------------------------------------------------------------------ GEMM
struct GemmX3Problem {
    const float *inv_x, *inv_w;            // [M], [N] row factors of the operands
    const float *bias;                     // optional [N]
    void *out;                             // [M, N], or [M / S, heads, S, N / heads] when heads > 0
    int M, S, heads;
    const float *x, *w;                    // the operands as they were: [M, K] or [M / S, x_heads, S, K / x_heads], [N, K]
    int x_heads;
    int w_row;                             // first row of this problem's W inside the W map
    int first_tile, tiles_n;
};
struct GemmX3Params {
    GemmX3Problem prob[3];
    int n_probs, n_tiles, N, K;
    int out_f16;
    const int *outliers;                   // the split passes' flag
    int *status;
};
// Which of the products a tile belongs to
__device__ __forceinline__ int problem_of(const GemmX3Params &p, int tile)
{
    int i = 0;
    if (p.n_probs > 1 && tile >= p.prob[1].first_tile) i = 1;
    if (p.n_probs > 2 && tile >= p.prob[2].first_tile) i = 2;
    return i;
}

struct GemmX3Maps {
    CUtensorMap xh[3], xl[3], wh, wl;
};

template <int BN_>
struct GemmX3Cfg {
    static constexpr int BM = 128, BN = BN_, BK = 64, CHUNK = 2;          // CHUNK: stages per accumulator
    static constexpr int THREADS = 384, REGS_LIGHT = 56, REGS_SUMS = 224; // 128 * 56 + 256 * 224 = 64512 = 384 * 168
    static constexpr uint32_t X_BYTES = BM * BK * 2, W_BYTES = BN * BK * 2;
    static constexpr uint32_t STAGE = 2 * X_BYTES + 2 * W_BYTES;          // x hi | x lo | W hi | W lo
    static constexpr int NS = BN == 256 ? 2 : (BN == 128 ? 3 : 4);
    static constexpr uint32_t OFF_TURN = NS * STAGE;                      // 8 warps x 32 rows x 128 bytes
    static constexpr uint32_t OFF_BAR = OFF_TURN + 8 * 4096;              // full[NS] empty[NS] acc_full[2] acc_free[2]
    static constexpr uint32_t OFF_TMEM = OFF_BAR + (2 * NS + 4) * 8, OFF_ABORT = OFF_TMEM + 4;
    static constexpr uint32_t SMEM_BYTES = ((OFF_ABORT + 4 + 127) / 128) * 128;
    static constexpr uint32_t TMEM_COLS = 2 * BN < 128 ? 128 : 2 * BN;
    static_assert(BN == 64 || BN == 128 || BN == 256, "tile width");
    static_assert(SMEM_BYTES <= 232448, "more than the 227 KB a CTA may have");
};

// This CTA's tiles from the fp32 operands, where some row's halves would not do.  A function of its own: inside the kernel
// its code cost the ordinary path 13 us a launch (B4 S1024 E1024: 78 -> 92 and 29 -> 44 us).
template <class Cfg>
__device__ __noinline__ void gemm_exact_tiles(const GemmX3Params &p, uint8_t *smem)
{
    auto a_s = reinterpret_cast<float (*)[LIN_BM + 4]>(smem);
    auto w_s = reinterpret_cast<float (*)[LIN_BN + 4]>(smem + LIN_BK * (LIN_BM + 4) * sizeof(float));
    for (int tile = blockIdx.x; tile < p.n_tiles; tile += gridDim.x) {
        const GemmX3Problem &pr = p.prob[problem_of(p, tile)];
        const int local = tile - pr.first_tile;
        LinearParams lp;
        lp.x = pr.x; lp.w = pr.w; lp.bias = pr.bias; lp.out = nullptr;
        lp.B = pr.M / pr.S; lp.S = pr.S; lp.K = p.K; lp.N = p.N; lp.heads_in = pr.x_heads; lp.heads_out = pr.heads;
        for (int m = 0; m < Cfg::BM; m += LIN_BM)
            for (int n = 0; n < Cfg::BN; n += LIN_BN)
                linear_simt_tile(lp, local / pr.tiles_n * Cfg::BM + m, local % pr.tiles_n * Cfg::BN + n, threadIdx.x, a_s, w_s,
                                 [&](int64_t row, int64_t col, float v) {
                                     const int64_t at = lin_index(row, col, lp.S, lp.N, lp.heads_out);
                                     if (p.out_f16) static_cast<__half *>(pr.out)[at] = __float2half_rn(v);
                                     else static_cast<float *>(pr.out)[at] = v;
                                 });
    }
}

template <class Cfg>
__global__ void __launch_bounds__(Cfg::THREADS, 1)
gemm_x3_kernel(const __grid_constant__ GemmX3Maps maps, const __grid_constant__ GemmX3Params p)
{
    constexpr int BM = Cfg::BM, BN = Cfg::BN, BK = Cfg::BK, NS = Cfg::NS, HALF = BN / 2;
    extern __shared__ __align__(1024) uint8_t smem[];
    const uint32_t sbase = ptx::smem_u32(smem);
    const uint32_t full = sbase + Cfg::OFF_BAR, empty = full + 8 * NS, acc_full = empty + 8 * NS, acc_free = acc_full + 16;
    volatile uint32_t *tmem_slot = reinterpret_cast<volatile uint32_t *>(smem + Cfg::OFF_TMEM);
    volatile int *abort_flag = reinterpret_cast<volatile int *>(smem + Cfg::OFF_ABORT);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int k_stages = (p.K + BK - 1) / BK, chunks = (k_stages + Cfg::CHUNK - 1) / Cfg::CHUNK;

    if (tid == 0) {
        *abort_flag = 0;
        for (int s = 0; s < NS; ++s) {
            ptx::mbar_init(full + 8 * s, 1);
            ptx::mbar_init(empty + 8 * s, 1);
        }
        for (int a = 0; a < 2; ++a) {
            ptx::mbar_init(acc_full + 8 * a, 1);
            ptx::mbar_init(acc_free + 8 * a, 8);                          // one arrival per summing warp
        }
        ptx::fence_mbar_init();
        if (sbase & 1023u) { *abort_flag = 1; ptx::report(p.status, 1); }
        if (*reinterpret_cast<volatile int *>(p.status) != 0) *abort_flag = 1;
    }
    if (warp == 1) {
        ptx::tmem_alloc(ptx::smem_u32(const_cast<uint32_t *>(tmem_slot)), Cfg::TMEM_COLS);
        ptx::tmem_relinquish();
    }
    ptx::tc_fence_before_sync();
    __syncthreads();
    ptx::tc_fence_after_sync();
    const uint32_t tmem = *tmem_slot;
    const bool run = *abort_flag == 0;
    ptx::grid_trigger();
    ptx::grid_wait();                                                     // the split pass; the start above ran under its end
    if (*reinterpret_cast<const volatile int *>(p.outliers) != 0) {
        gemm_exact_tiles<Cfg>(p, smem);
        ptx::tc_fence_before_sync();
        __syncthreads();
        if (warp == 1) {
            ptx::tc_fence_after_sync();
            ptx::tmem_dealloc(tmem, Cfg::TMEM_COLS);
        }
        return;
    }

    if (warp < 4) {
    ptx::setmaxnreg_dec<Cfg::REGS_LIGHT>();
    if (warp == 0) {
        if (run) {
            const bool leader = ptx::elect_one();
            bool ok = true;
            int n = 0;                                                    // stages so far, over all tiles
            for (int tile = blockIdx.x; tile < p.n_tiles && ok; tile += gridDim.x) {
                const int i = problem_of(p, tile), local = tile - p.prob[i].first_tile;
                const int m0 = local / p.prob[i].tiles_n * BM, n0 = p.prob[i].w_row + local % p.prob[i].tiles_n * BN;
                for (int j = 0; j < k_stages && ok; ++j, ++n) {
                    const int s = n % NS;
                    ok = ptx::mbar_wait(empty + 8 * s, ((uint32_t)(n / NS) & 1u) ^ 1u, abort_flag);
                    if (!ok) break;
                    if (leader) {
                        const uint32_t dst = sbase + (uint32_t)s * Cfg::STAGE, bar = full + 8 * s;
                        ptx::mbar_arrive_expect_tx(bar, Cfg::STAGE);
                        ptx::tma_load_3d(dst, &maps.xh[i], bar, j * BK, m0, 0);
                        ptx::tma_load_3d(dst + Cfg::X_BYTES, &maps.xl[i], bar, j * BK, m0, 0);
                        ptx::tma_load_3d(dst + 2 * Cfg::X_BYTES, &maps.wh, bar, j * BK, n0, 0);
                        ptx::tma_load_3d(dst + 2 * Cfg::X_BYTES + Cfg::W_BYTES, &maps.wl, bar, j * BK, n0, 0);
                    }
                    __syncwarp();
                }
            }
            if (!ok && leader) { *abort_flag = 1; ptx::report(p.status, GX3_ERR_PRODUCER); }
        }
    } else if (warp == 1) {
        if (run) {
            const bool leader = ptx::elect_one();
            constexpr uint32_t idesc = ptx::idesc_f16(BM, BN, false);
            constexpr uint32_t desc_hi = ptx::smem_desc_sw128_hi(1024);
            const uint32_t base_lo = ptx::smem_desc_sw128_lo(sbase, 16);
            bool ok = true;
            int n = 0, c = 0;                                             // stages and chunks so far
            for (int tile = blockIdx.x; tile < p.n_tiles && ok; tile += gridDim.x) {
                for (int j = 0; j < k_stages && ok; ++j, ++n) {
                    const int s = n % NS, a = c & 1;
                    const bool first = j % Cfg::CHUNK == 0, last = j % Cfg::CHUNK == Cfg::CHUNK - 1 || j == k_stages - 1;
                    if (first && c >= 2) ok = ptx::mbar_wait(acc_free + 8 * a, (uint32_t)((c - 2) >> 1) & 1u, abort_flag);
                    if (ok) ok = ptx::mbar_wait(full + 8 * s, (uint32_t)(n / NS) & 1u, abort_flag);
                    if (!ok) break;
                    ptx::tc_fence_after_sync();
                    if (leader) {
                        const uint32_t xh = base_lo + (uint32_t)s * (Cfg::STAGE >> 4), xl = xh + (Cfg::X_BYTES >> 4);
                        const uint32_t wh = xl + (Cfg::X_BYTES >> 4), wl = wh + (Cfg::W_BYTES >> 4);
                        const uint32_t acc = tmem + (uint32_t)a * BN;
#pragma unroll
                        for (int kk = 0; kk < BK / 16; ++kk) {
                            const uint32_t o = (kk * 32) >> 4;
                            ptx::mma_ss(acc, ptx::make_desc(xh + o, desc_hi), ptx::make_desc(wl + o, desc_hi), idesc, (!first || kk > 0) ? 1u : 0u);
                            ptx::mma_ss(acc, ptx::make_desc(xl + o, desc_hi), ptx::make_desc(wh + o, desc_hi), idesc, 1u);
                        }
#pragma unroll
                        for (int kk = 0; kk < BK / 16; ++kk) {
                            const uint32_t o = (kk * 32) >> 4;
                            ptx::mma_ss(acc, ptx::make_desc(xh + o, desc_hi), ptx::make_desc(wh + o, desc_hi), idesc, 1u);
                        }
                        ptx::mma_commit(empty + 8 * s);
                        if (last) ptx::mma_commit(acc_full + 8 * a);
                    }
                    __syncwarp();
                    if (last) ++c;
                }
            }
            if (!ok && leader) { *abort_flag = 1; ptx::report(p.status, GX3_ERR_MMA); }
        }
    }
    } else {
        ptx::setmaxnreg_inc<Cfg::REGS_SUMS>();
        const int quarter = warp & 3, half = (warp - 4) >> 2;
        const uint32_t lane_base = (uint32_t)(quarter * 32) << 16;
        const uint32_t turn = sbase + Cfg::OFF_TURN + (uint32_t)(warp - 4) * 4096;
        bool ok = run;
        int c = 0;
        for (int tile = blockIdx.x; tile < p.n_tiles && ok; tile += gridDim.x) {
            float sum[HALF];
#pragma unroll
            for (int i = 0; i < HALF; ++i) sum[i] = 0.f;
            for (int ch = 0; ch < chunks && ok; ++ch, ++c) {
                const int a = c & 1;
                ok = ptx::mbar_wait(acc_full + 8 * a, (uint32_t)(c >> 1) & 1u, abort_flag);
                if (!ok) break;
                ptx::tc_fence_after_sync();
                const uint32_t acc = tmem + lane_base + (uint32_t)(a * BN + half * HALF);
#pragma unroll
                for (int q = 0; q < HALF / 32; ++q) {
                    uint32_t t[32];
                    ptx::tmem_ld32(acc + q * 32, t);
                    ptx::tmem_wait_ld();
                    ptx::reg_fence32(t);
#pragma unroll
                    for (int i = 0; i < 32; ++i) sum[q * 32 + i] += __uint_as_float(t[i]);
                }
                ptx::tc_fence_before_sync();
                __syncwarp();
                if (lane == 0) ptx::mbar_arrive(acc_free + 8 * a);
            }
            if (!ok) break;
            // result: 32 rows x 32 columns at a time through shared memory (16-byte pieces at piece ^ (row & 7)), then
            // eight lanes store 128 bytes of one row
            const GemmX3Problem &pr = p.prob[problem_of(p, tile)];
            const int local = tile - pr.first_tile;
            const int row0 = local / pr.tiles_n * BM + quarter * 32, col0 = local % pr.tiles_n * BN + half * HALF;
            // The result is sum * inv_x * inv_w + bias; the factor below 1 comes first where the other one is above, so that
            // the product in between is in range whenever the result is (x of 1e36 and weights of 1e-30: sum * inv_x alone
            // overflowed).  Rows that need inv_x last are rare: a warp without one does nothing more.
            const float inv_x = row0 + lane < pr.M ? pr.inv_x[row0 + lane] : 0.f, inv = fminf(inv_x, 1.f), inv_last = fmaxf(inv_x, 1.f);
            const bool any_last = __any_sync(0xffffffffu, inv_x > 1.f);
            const int dh = pr.heads > 0 ? p.N / pr.heads : p.N;
#pragma unroll
            for (int q = 0; q < HALF / 32; ++q) {
                __syncwarp();
#pragma unroll
                for (int i = 0; i < 32; i += 4)
                    ptx::st_shared_v4(turn + (uint32_t)lane * 128 + ((uint32_t)((i >> 2) ^ (lane & 7)) << 4),
                                      __float_as_uint(sum[q * 32 + i] * inv), __float_as_uint(sum[q * 32 + i + 1] * inv),
                                      __float_as_uint(sum[q * 32 + i + 2] * inv), __float_as_uint(sum[q * 32 + i + 3] * inv));
                __syncwarp();
                const int n = col0 + q * 32 + (lane & 7) * 4;
                float last[8];                                            // of the rows this lane stores
                if (any_last)
#pragma unroll
                    for (int i = 0; i < 8; ++i) last[i] = __shfl_sync(0xffffffffu, inv_last, i * 4 + (lane >> 3));
                if (n < p.N) {
                    const float4 iw = *reinterpret_cast<const float4 *>(pr.inv_w + n);
                    const float4 bb = pr.bias ? __ldg(reinterpret_cast<const float4 *>(pr.bias + n)) : make_float4(0.f, 0.f, 0.f, 0.f);
                    const int h = n / dh, cc = n % dh;
#pragma unroll
                    for (int r4 = 0; r4 < 32; r4 += 4) {
                        const int r = r4 + (lane >> 3), m = row0 + r;
                        if (m >= pr.M) break;
                        uint32_t x, y, z, w;
                        ptx::ld_shared_v4(turn + (uint32_t)r * 128 + ((uint32_t)((lane & 7) ^ (r & 7)) << 4), x, y, z, w);
                        float4 f = make_float4(fmaf(__uint_as_float(x), iw.x, bb.x), fmaf(__uint_as_float(y), iw.y, bb.y),
                                               fmaf(__uint_as_float(z), iw.z, bb.z), fmaf(__uint_as_float(w), iw.w, bb.w));
                        if (any_last) {
                            const float a = last[r4 / 4];
                            f = make_float4(fmaf(__uint_as_float(x) * iw.x, a, bb.x), fmaf(__uint_as_float(y) * iw.y, a, bb.y),
                                            fmaf(__uint_as_float(z) * iw.z, a, bb.z), fmaf(__uint_as_float(w) * iw.w, a, bb.w));
                        }
                        const size_t at = pr.heads > 0 ? (((size_t)(m / pr.S) * pr.heads + h) * pr.S + m % pr.S) * dh + cc
                                                       : (size_t)m * p.N + n;
                        if (p.out_f16) {
                            uint2 u;
                            u.x = ptx::pack_half2(f.x, f.y); u.y = ptx::pack_half2(f.z, f.w);
                            *reinterpret_cast<uint2 *>(static_cast<__half *>(pr.out) + at) = u;
                        } else {
                            *reinterpret_cast<float4 *>(static_cast<float *>(pr.out) + at) = f;
                        }
                    }
                }
            }
        }
        if (run && !ok) { *abort_flag = 1; ptx::report(p.status, GX3_ERR_SUMS); }
    }

    ptx::tc_fence_before_sync();
    __syncthreads();
    if (*abort_flag) {
        for (int i = 0; i < 64; ++i) __nanosleep(2000);                   // let copies in flight land
        __syncthreads();
    }
    if (warp == 1) {
        ptx::tc_fence_after_sync();
        ptx::tmem_dealloc(tmem, Cfg::TMEM_COLS);
    }
}

}  // namespace txb

// SDPA backward on sm_100a: dQ, dK, dV from Q, K, V (fp16), dO and the forward's row statistics.
//
// The math is the reference's autograd rule for 'scaled_dot_product_attention'
// (tensorax/tensor.py:806-827):
//     P  = softmax(Q K^T * scale [+ mask])          dV = P^T dO
//     dP = dO V^T                                   D  = rowsum(dP o P)  (= rowsum(dO o O))
//     dS = P o (dP - D) * scale                     dQ = dS K,   dK = dS^T Q
// done flash-style: P is rebuilt tile by tile from the forward's per-row log-sum-exp, nothing of
// size Sq x Sk ever reaches global memory.  Two kernels, so that no gradient needs atomics and the
// result is bitwise reproducible:
//
//   sdpa_bwd_dq_kernel   one CTA = one 128-row query tile; loops over key tiles:
//                        S = Q K^T, dP = dO V^T (SS MMAs) -> registers -> dS (fp16, TMEM) ->
//                        dQ += dS K (TS MMA, K read MN-major from the same stage)
//   sdpa_bwd_dkv_kernel  one CTA = one 128-row key tile of one K/V head; loops over the query heads
//                        of its group and their query tiles: S^T = K Q^T, dP^T = V dO^T ->
//                        registers -> P^T, dS^T (fp16, TMEM) -> dV += P^T dO, dK += dS^T Q
//
// Roles per CTA as in the forward kernel: warp 0 TMA producer, warp 1 MMA issuer and TMEM owner,
// then one or two row warpgroups (4 warps each, one thread per TMEM lane; two warpgroups split a
// tile's columns).  Head dims 64, 128 and 256 (at 256 the dK/dV kernel runs two CTAs per key tile,
// each accumulating half of the gradient columns).  Every wait is bounded (ptx::mbar_wait); a wait that runs out
// sets the CTA's abort flag and a code in the device status word.
//
// Bound, d = 128: shared-memory traffic in the dQ kernel (operands of the SS MMAs and the TMA writes: about 1 800 of 2 000
// cycles per 128 x 128 tile), MMA issue in the dK/dV kernel (about 1 300 cycles per 128 x 64 tile); a CTA's start and end
// are 15 to 25 % of a causal one.  B4 H16 S2048 d128 causal: 148 -> 141 us and 218 -> 182 us; B2 Hq12 Hkv4 S921 d64 causal:
// dK/dV 79 -> 27 us, its items cut over clusters (split_k).
#pragma once

#include <cooperative_groups.h>

#include "ptx.cuh"
#include "sdpa_tc.cuh"

namespace txb {

enum : int { BWD_ERR_PRODUCER = 22, BWD_ERR_MMA = 23, BWD_ERR_ROWS = 24 };

struct BwdParams {
    const float *lse;         // [B,Hq,Sq] log2-domain row statistic written by the forward
    const float *delta;       // [B,Hq,Sq] rowsum(dO o O)
    KvLens kv_lens;           // optional [B]
    float *dq, *dk, *dv;      // [B,Hq,Sq,D], [B,Hkv,Sk,D], [B,Hkv,Sk,D] fp32
    int *status;
    int *prepared;            // word of the workspace: 1 once the dQ kernel has the preprocess behind it
    int Hq, Hkv, Sq, Sk;
    int causal;
    float scale;              // 1/sqrt(d)
    float scale_log2;         // scale * log2(e)
    // Launch order of the 1-D grids (as in the forward's two-tile kernel): slabs are walked in groups, inside a
    // group every slab's longest items first.  *_q: the dQ kernel (slab = (batch, query head), item = query tile);
    // *_k: the dK/dV kernel (slab = (batch, K/V head), item = key tile; its ZS column parts stay side by side).
    int group_q, items_q, slabs_q;
    int group_k, items_k, slabs_k;
    // CTAs (a thread-block cluster, neighbours in the 1-D grid) that share one work item: CTA z of `split_*` takes the
    // item's tiles z, z + split, z + 2 split ... and the cluster adds the partial gradients in rank order.
    int split_q, split_k;
};

// ------------------------------------------------------------------ result
// Gradient tiles leave tensor memory through shared memory, so that global memory is written in whole lines (one row a
// thread straight from tensor memory, 32 rows an instruction, cost 5 900 cycles a CTA in the dQ kernel and 9 800 in the
// dK/dV kernel at d = 128, of 31 000 and 58 000 in all), and so that the CTAs of a cluster can add theirs up.
// A staged tile is [128 rows][W floats]; 16-byte chunk c of row r sits at chunk c ^ (r % 8) (both sides conflict-free).
template <int W>
__device__ __forceinline__ uint32_t grad_chunk(int r, int c) { return (uint32_t)(r * (W / 4) + (c ^ (r & 7))) * 16u; }

// 32 accumulator columns of the thread's row (TMEM lane) to the staged tile; zeros where the CTA had no tile to walk
template <int W>
__device__ __forceinline__ void stage_grad32(uint32_t tile, uint32_t taddr, int r, int col, bool any)
{
    uint32_t o[32];
    if (any) {
        ptx::tmem_ld32(taddr, o);
        ptx::tmem_wait_ld();
        ptx::reg_fence32(o);
    } else {
#pragma unroll
        for (int i = 0; i < 32; ++i) o[i] = 0u;
    }
#pragma unroll
    for (int i = 0; i < 32; i += 4)
        ptx::st_shared_v4(tile + grad_chunk<W>(r, (col + i) / 4), o[i], o[i + 1], o[i + 2], o[i + 3]);
}

// This CTA's share of the tile's rows: summed over the cluster's CTAs in rank order, written to dst[row * ld + column].
// `fill` stands in for the sum where no CTA of the item had anything to walk.
template <int W, int THREADS>
__device__ __forceinline__ void store_grad(const uint8_t *tile, float *dst, int64_t ld, int rows_ok, int rank, int split,
                                           bool filled, float fill, int tid)
{
    namespace cg = cooperative_groups;
    constexpr int C = W / 4;
    if (split == 1 && !filled) {
        // unrolled: several rows under way at once
        constexpr int N = 128 * C;
#pragma unroll 8
        for (int n = 0; n < (N + THREADS - 1) / THREADS; ++n) {
            const int i = n * THREADS + tid, r = i / C, c = i % C;
            if (i < N && r < rows_ok)
                *reinterpret_cast<float4 *>(dst + (int64_t)r * ld + c * 4) =
                    *reinterpret_cast<const float4 *>(tile + grad_chunk<W>(r, c));
        }
        return;
    }
    const int rows = 128 / split, r0 = rank * rows;
    for (int i = tid; i < rows * C; i += THREADS) {
        const int r = r0 + i / C, c = i % C;
        if (r >= rows_ok) break;
        float4 v = make_float4(fill, fill, fill, fill);
        if (!filled) {
            cg::cluster_group cluster = cg::this_cluster();
            const uint8_t *at = tile + grad_chunk<W>(r, c);
            float4 part[8];                                        // all remote loads first: they take as long as one
#pragma unroll
            for (int z = 0; z < 8; ++z)
                if (z < split) part[z] = *reinterpret_cast<const float4 *>(cluster.map_shared_rank(at, z));
            v = part[0];
#pragma unroll
            for (int z = 1; z < 8; ++z)
                if (z < split) { v.x += part[z].x; v.y += part[z].y; v.z += part[z].z; v.w += part[z].w; }
        }
        *reinterpret_cast<float4 *>(dst + (int64_t)r * ld + c * 4) = v;
    }
}

// ------------------------------------------------------------------ preprocess
// dO fp32 -> fp16 (MMA operand) and delta = rowsum(dO o O).  Bound: HBM (10 d + 4 or 8 d + 4 bytes a row).  Sixteen lanes a row
// at d = 64, 32 otherwise, four values a lane and step; a warp requests two steps of rows at a time.  One row a warp and
// eight bytes a lane took 30.3 us at B4 H16 S2048 d128, this 23.4 (6.9 TB/s; dO and O partly in L2).
template <typename OT, int D>
__global__ void __launch_bounds__(256) sdpa_bwd_prep_kernel(const float *__restrict__ dout, const OT *__restrict__ out,
                                                            __half *__restrict__ dout_h, float *__restrict__ delta, int64_t rows,
                                                            int *prepared)
{
    ptx::grid_trigger();
    if (blockIdx.x == 0 && threadIdx.x == 0) *prepared = 0;
    constexpr int LPR = D / 4 < 32 ? D / 4 : 32, RPW = 32 / LPR, STEPS = 2, PIECES = D / 4 / LPR;   // lanes a row, rows a warp step
    const int lane = threadIdx.x & 31, gl = lane % LPR;
    const int64_t row0 = ((int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)) * (RPW * STEPS) + lane / LPR;
    float4 g[STEPS][PIECES], o[STEPS][PIECES];
#pragma unroll
    for (int t = 0; t < STEPS; ++t)
#pragma unroll
        for (int c = 0; c < PIECES; ++c) {
            const int64_t row = row0 + t * RPW;
            g[t][c] = o[t][c] = make_float4(0.f, 0.f, 0.f, 0.f);
            if (row >= rows) continue;
            const int64_t at = row * D + (c * LPR + gl) * 4;
            g[t][c] = *reinterpret_cast<const float4 *>(dout + at);
            if constexpr (sizeof(OT) == 2) {
                const uint2 h = *reinterpret_cast<const uint2 *>(out + at);
                const float2 lo = __half22float2(*reinterpret_cast<const __half2 *>(&h.x)), hi = __half22float2(*reinterpret_cast<const __half2 *>(&h.y));
                o[t][c] = make_float4(lo.x, lo.y, hi.x, hi.y);
            } else {
                o[t][c] = *reinterpret_cast<const float4 *>(out + at);
            }
        }
#pragma unroll
    for (int t = 0; t < STEPS; ++t) {
        const int64_t row = row0 + t * RPW;
        float acc = 0.f;
#pragma unroll
        for (int c = 0; c < PIECES; ++c) {
            const float4 a = g[t][c], b = o[t][c];
            acc = fmaf(a.x, b.x, acc); acc = fmaf(a.y, b.y, acc); acc = fmaf(a.z, b.z, acc); acc = fmaf(a.w, b.w, acc);
            if (row < rows)
                *reinterpret_cast<uint2 *>(dout_h + row * D + (c * LPR + gl) * 4) = make_uint2(ptx::pack_half2(a.x, a.y), ptx::pack_half2(a.z, a.w));
        }
#pragma unroll
        for (int w = LPR / 2; w > 0; w >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, w);
        if (gl == 0 && row < rows) delta[row] = acc;
    }
}

// ------------------------------------------------------------------ dQ
// WGS: row warpgroups (4 warps, one thread per TMEM lane each); with 2, each takes half of a tile's columns.
// NS / NSV: depth of the K / V ring.  A K stage is read twice (S = Q K^T, later dQ += dS K) and only
// then freed, so its ring is one deeper than V's, whose stage goes back right after dP = dO V^T.
template <int D_, int BN_, int NS_, int WGS_ = 1, int NSV_ = 2>
struct BwdDqCfg {
    static constexpr int D = D_, BN = BN_, NS = NS_, NSV = NSV_, BM = 128, WGS = WGS_;
    static constexpr int CW = BN / WGS;                      // tile columns per warpgroup
    static constexpr int THREADS = 64 + 128 * WGS;
    static constexpr int KP = D / 64;
    static constexpr uint32_t Q_BYTES = BM * D * 2;          // Q tile, dO tile
    static constexpr uint32_t KV_BYTES = BN * D * 2;         // one K or V stage
    static constexpr uint32_t KV_PANEL = BN * 128;
    static constexpr uint32_t OFF_Q = 0, OFF_DO = Q_BYTES, OFF_K = 2 * Q_BYTES, OFF_V = OFF_K + NS * KV_BYTES;
    static constexpr uint32_t OFF_BAR = OFF_V + NSV * KV_BYTES;
    // barriers: qdo_full, s_full, dp_full, s_free, ds_full, dq_done, k_full/k_empty[NS], v_full/v_empty[NSV]
    static constexpr int N_BARS = 6 + 2 * NS + 2 * NSV;
    static constexpr uint32_t OFF_TMEM = OFF_BAR + N_BARS * 8;
    static constexpr uint32_t OFF_ABORT = OFF_TMEM + 4;
    static constexpr uint32_t SMEM_BYTES = ((OFF_ABORT + 4 + 127) / 128) * 128;
    // tensor memory: S [BN] | dP [BN] | dQ [D] | dS fp16 pairs [BN/2]
    static constexpr uint32_t COL_S = 0, COL_DP = BN, COL_DQ = 2 * BN, COL_DS = 2 * BN + D;
    static constexpr uint32_t COLS_USED = 2 * BN + D + BN / 2;
    static constexpr uint32_t TMEM_COLS = COLS_USED <= 256 ? 256 : 512;
    static constexpr int CTAS_PER_SM = (SMEM_BYTES <= 115712 && TMEM_COLS <= 256) ? 2 : 1;
    static_assert(D % 64 == 0 && CW % 32 == 0 && (D / 32) % WGS == 0 && COLS_USED <= 512 && SMEM_BYTES <= 232448,
                  "tile shape");
    static_assert(BM * D * 4 <= OFF_BAR, "the staged dQ tile lies over the operand tiles");
};

template <class Cfg>
__global__ void __launch_bounds__(Cfg::THREADS, Cfg::CTAS_PER_SM)
sdpa_bwd_dq_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_do,
                   const __grid_constant__ CUtensorMap tm_k, const __grid_constant__ CUtensorMap tm_v,
                   const BwdParams p)
{
    constexpr int D = Cfg::D, BN = Cfg::BN, NS = Cfg::NS, NSV = Cfg::NSV, BM = Cfg::BM;
    extern __shared__ __align__(1024) uint8_t smem[];
    const uint32_t sbase = ptx::smem_u32(smem);
    const uint32_t q_s = sbase + Cfg::OFF_Q, do_s = sbase + Cfg::OFF_DO, k_s = sbase + Cfg::OFF_K,
                   v_s = sbase + Cfg::OFF_V;
    const uint32_t bar0 = sbase + Cfg::OFF_BAR;
    const uint32_t qdo_full = bar0, s_full = bar0 + 8, dp_full = bar0 + 16, s_free = bar0 + 24,
                   ds_full = bar0 + 32, dq_done = bar0 + 40;
    const uint32_t k_full = bar0 + 48, k_empty = k_full + 8 * NS, v_full = k_empty + 8 * NS,
                   v_empty = v_full + 8 * NSV;
    volatile uint32_t *tmem_slot = reinterpret_cast<volatile uint32_t *>(smem + Cfg::OFF_TMEM);
    volatile int *abort_flag = reinterpret_cast<volatile int *>(smem + Cfg::OFF_ABORT);

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    // work item: group-major, then longest first over all slabs of the group (late causal query tiles walk most keys)
    const int split = p.split_q, rank = (int)blockIdx.x % split;
    const int item = (int)blockIdx.x / split;
    const int span = p.group_q * p.items_q;
    const int grp = item / span, rem = item % span;
    const int in_grp = min(p.group_q, p.slabs_q - grp * p.group_q);
    const int q_tile = p.items_q - 1 - rem / in_grp;
    const int q0 = q_tile * BM;
    const int bh = grp * p.group_q + rem % in_grp;
    const int b = bh / p.Hq, h = bh % p.Hq;
    const int kvh = b * p.Hkv + h / (p.Hq / p.Hkv);
    int kv_limit = p.Sk;
    kv_limit = p.kv_lens.limit(b, kv_limit);
    int kv_end = kv_limit;
    if (p.causal) kv_end = min(kv_end, q0 + BM);
    const int n_all = (kv_end + BN - 1) / BN;
    const int n_tiles = n_all > rank ? (n_all - rank + split - 1) / split : 0;      // tiles rank, rank + split, ...

    auto load_k = [&](int j) {
        const int s = j % NS;
        ptx::mbar_arrive_expect_tx(k_full + 8 * s, Cfg::KV_BYTES);
#pragma unroll
        for (int pn = 0; pn < Cfg::KP; ++pn)
            ptx::tma_load_3d(k_s + s * Cfg::KV_BYTES + pn * Cfg::KV_PANEL, &tm_k, k_full + 8 * s, pn * 64,
                             (rank + j * split) * BN, kvh);
    };
    auto load_v = [&](int j) {
        const int s = j % NSV;
        ptx::mbar_arrive_expect_tx(v_full + 8 * s, Cfg::KV_BYTES);
#pragma unroll
        for (int pn = 0; pn < Cfg::KP; ++pn)
            ptx::tma_load_3d(v_s + s * Cfg::KV_BYTES + pn * Cfg::KV_PANEL, &tm_v, v_full + 8 * s, pn * 64,
                             (rank + j * split) * BN, kvh);
    };
    if (tid == 0) {
        *abort_flag = 0;
        ptx::mbar_init(qdo_full, 1);
        ptx::mbar_init(s_full, 1);
        ptx::mbar_init(dp_full, 1);
        ptx::mbar_init(s_free, 4 * Cfg::WGS);
        ptx::mbar_init(ds_full, 4 * Cfg::WGS);
        ptx::mbar_init(dq_done, 1);
        for (int s = 0; s < NS; ++s) {
            ptx::mbar_init(k_full + 8 * s, 1);
            ptx::mbar_init(k_empty + 8 * s, 1);
        }
        for (int s = 0; s < NSV; ++s) {
            ptx::mbar_init(v_full + 8 * s, 1);
            ptx::mbar_init(v_empty + 8 * s, 1);
        }
        ptx::fence_mbar_init();
        if (sbase & 1023u) {
            *abort_flag = 1;
            ptx::report(p.status, TC_ERR_ALIGN);
        } else if (n_tiles > 0) {
            ptx::grid_wait();                    // the preprocess: dO in fp16 and the row sums
            // the first loads run under the tensor-memory allocation and the meeting
            ptx::mbar_arrive_expect_tx(qdo_full, 2 * Cfg::Q_BYTES);
#pragma unroll
            for (int pn = 0; pn < Cfg::KP; ++pn)
                ptx::tma_load_3d(q_s + pn * (BM * 128), &tm_q, qdo_full, pn * 64, q0, bh);
            load_k(0);
#pragma unroll
            for (int pn = 0; pn < Cfg::KP; ++pn)
                ptx::tma_load_3d(do_s + pn * (BM * 128), &tm_do, qdo_full, pn * 64, q0, bh);
            load_v(0);
        }
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
    const bool run = (*abort_flag == 0) && n_tiles > 0;
    // The dK/dV kernel starts under this one and reads what the preprocess wrote.  The wait makes that visible to this
    // kernel, the word hands it on, and no CTA lets the dK/dV kernel start before its own thread 0 is past both.
    ptx::grid_wait();
    if (tid == 0) {
        if (blockIdx.x == 0) ptx::store_release(p.prepared, 1);
        ptx::grid_trigger();
    }

    if (warp == 0) {
        if (run) {
            const bool leader = ptx::elect_one();
            bool ok = true;
            // tile 0 went out before the meeting: no wait is taken on its behalf (its stages may be released already)
            for (int j = 1; j < n_tiles && ok; ++j) {
                ok = ptx::mbar_wait(k_empty + 8 * (j % NS), ((uint32_t)(j / NS) & 1u) ^ 1u, abort_flag);
                if (!ok) break;
                if (leader) load_k(j);
                __syncwarp();
                ok = ptx::mbar_wait(v_empty + 8 * (j % NSV), ((uint32_t)(j / NSV) & 1u) ^ 1u, abort_flag);
                if (!ok) break;
                if (leader) load_v(j);
                __syncwarp();
            }
            if (!ok && leader) { *abort_flag = 1; ptx::report(p.status, BWD_ERR_PRODUCER); }
        }
    } else if (warp == 1) {
        if (run) {
            const bool leader = ptx::elect_one();
            constexpr uint32_t idesc_s = ptx::idesc_f16(BM, BN, false);     // S, dP: both operands K-major
            constexpr uint32_t idesc_dq = ptx::idesc_f16(BM, D, true);      // dQ: B = K tile read MN-major
            constexpr uint32_t desc_hi = ptx::smem_desc_sw128_hi(1024);
            const uint32_t q_lo = ptx::smem_desc_sw128_lo(q_s, 16);
            const uint32_t do_lo = ptx::smem_desc_sw128_lo(do_s, 16);
            const uint32_t k_lo = ptx::smem_desc_sw128_lo(k_s, 16);
            const uint32_t v_lo = ptx::smem_desc_sw128_lo(v_s, 16);
            const uint32_t kmn_lo = ptx::smem_desc_sw128_lo(k_s, Cfg::KV_PANEL);
            const uint32_t t_s = tmem + Cfg::COL_S, t_dp = tmem + Cfg::COL_DP, t_dq = tmem + Cfg::COL_DQ,
                           t_ds = tmem + Cfg::COL_DS;
            bool ok = ptx::mbar_wait(qdo_full, 0, abort_flag);
            auto issue_s_dp = [&](int j) -> bool {
                const int s = j % NS;
                const uint32_t ph = (uint32_t)(j / NS) & 1u;
                if (!ptx::mbar_wait(k_full + 8 * s, ph, abort_flag)) return false;
                ptx::tc_fence_after_sync();
                const uint32_t st_off = (uint32_t)s * (Cfg::KV_BYTES >> 4);
                if (leader) {
#pragma unroll
                    for (int kk = 0; kk < D / 16; ++kk) {
                        const uint32_t a = ((kk >> 2) * (BM * 128) + (kk & 3) * 32) >> 4;
                        const uint32_t bb = ((kk >> 2) * Cfg::KV_PANEL + (kk & 3) * 32) >> 4;
                        ptx::mma_ss(t_s, ptx::make_desc(q_lo + a, desc_hi), ptx::make_desc(k_lo + st_off + bb, desc_hi),
                                    idesc_s, kk > 0);
                    }
                    ptx::mma_commit(s_full);
                }
                __syncwarp();
                const int sv_ = j % NSV;
                const uint32_t phv = (uint32_t)(j / NSV) & 1u;
                const uint32_t sv_off = (uint32_t)sv_ * (Cfg::KV_BYTES >> 4);
                if (!ptx::mbar_wait(v_full + 8 * sv_, phv, abort_flag)) return false;
                ptx::tc_fence_after_sync();
                if (leader) {
#pragma unroll
                    for (int kk = 0; kk < D / 16; ++kk) {
                        const uint32_t a = ((kk >> 2) * (BM * 128) + (kk & 3) * 32) >> 4;
                        const uint32_t bb = ((kk >> 2) * Cfg::KV_PANEL + (kk & 3) * 32) >> 4;
                        ptx::mma_ss(t_dp, ptx::make_desc(do_lo + a, desc_hi), ptx::make_desc(v_lo + sv_off + bb, desc_hi),
                                    idesc_s, kk > 0);
                    }
                    ptx::mma_commit(v_empty + 8 * sv_);
                    ptx::mma_commit(dp_full);
                }
                __syncwarp();
                return true;
            };
            if (ok) ok = issue_s_dp(0);
            for (int j = 0; j < n_tiles && ok; ++j) {
                if (j + 1 < n_tiles) {
                    ok = ptx::mbar_wait(s_free, (uint32_t)j & 1u, abort_flag);
                    if (!ok) break;
                    ptx::tc_fence_after_sync();
                    ok = issue_s_dp(j + 1);
                    if (!ok) break;
                }
                ok = ptx::mbar_wait(ds_full, (uint32_t)j & 1u, abort_flag);
                if (!ok) break;
                ptx::tc_fence_after_sync();
                const int s = j % NS;
                const uint32_t ks = kmn_lo + (uint32_t)s * (Cfg::KV_BYTES >> 4);
                if (leader) {
#pragma unroll
                    for (int kk = 0; kk < BN / 16; ++kk)
                        ptx::mma_ts(t_dq, t_ds + kk * 8, ptx::make_desc(ks + kk * ((16 * 128) >> 4), desc_hi), idesc_dq,
                                    (j > 0 || kk > 0) ? 1u : 0u);
                    ptx::mma_commit(k_empty + 8 * s);
                    ptx::mma_commit(dq_done);
                }
                __syncwarp();
            }
            if (!ok && leader) { *abort_flag = 1; ptx::report(p.status, BWD_ERR_MMA); }
        }
    } else {
        constexpr int CW = Cfg::CW;
        const int quarter = warp & 3;
        const int wg = (warp - 2) >> 2;
        const int c0 = wg * CW;                     // this warpgroup's first column of every tile
        const int r = quarter * 32 + lane;
        const int row = q0 + r;
        const uint32_t lane_base = (uint32_t)(quarter * 32) << 16;
        const uint32_t t_s = tmem + lane_base + Cfg::COL_S + c0, t_dp = tmem + lane_base + Cfg::COL_DP + c0,
                       t_dq = tmem + lane_base + Cfg::COL_DQ, t_ds = tmem + lane_base + Cfg::COL_DS + c0 / 2;
        const bool row_ok = row < p.Sq;
        // a row outside the problem gets lse = +inf: every P of it is 2^(-inf) = 0
        const float lse = row_ok ? p.lse[(size_t)bh * p.Sq + row] : INFINITY;
        const float delta = row_ok ? p.delta[(size_t)bh * p.Sq + row] : 0.f;
        bool ok = run;
        auto arrive_warp = [&](uint32_t bar) {
            ptx::tc_fence_before_sync();
            __syncwarp();
            if (lane == 0) ptx::mbar_arrive(bar);
        };
        for (int j = 0; j < n_tiles && ok; ++j) {
            const int kv0 = (rank + j * split) * BN + c0;
            ok = ptx::mbar_wait(s_full, (uint32_t)j & 1u, abort_flag);
            if (!ok) break;
            ptx::tc_fence_after_sync();
            uint32_t sv[CW], dpv[CW];
            ptx::tmem_ld_cols<CW>(t_s, sv);
            ok = ptx::mbar_wait(dp_full, (uint32_t)j & 1u, abort_flag);
            if (!ok) break;
            ptx::tc_fence_after_sync();
            ptx::tmem_ld_cols<CW>(t_dp, dpv);
            ptx::tmem_wait_ld();
            ptx::reg_fence_cols<CW>(sv);
            ptx::reg_fence_cols<CW>(dpv);
            arrive_warp(s_free);
            const bool need_mask = (kv0 + CW > kv_limit) || (p.causal && (kv0 + CW - 1 > q0));
            const int lim = min(kv_limit - kv0, p.causal ? row - kv0 + 1 : CW);
            uint32_t pk[CW / 2];
            // packed fp32 pairs: x = s*c - lse, t = dP*scale - D*scale, dS = P*t
            const float2 c2 = make_float2(p.scale_log2, p.scale_log2), nl2 = make_float2(-lse, -lse);
            const float2 s2 = make_float2(p.scale, p.scale), nd2 = make_float2(-delta * p.scale, -delta * p.scale);
#pragma unroll
            for (int i = 0; i < CW; i += 2) {
                const float2 x = __ffma2_rn(make_float2(__uint_as_float(sv[i]), __uint_as_float(sv[i + 1])), c2, nl2);
                float2 pr = make_float2(ptx::ex2_approx(x.x), ptx::ex2_approx(x.y));
                if (need_mask) {                 // visible keys of this row are a prefix of the tile: [0, lim)
                    pr.x = ptx::zero_unless_lt(pr.x, i, lim);
                    pr.y = ptx::zero_unless_lt(pr.y, i + 1, lim);
                }
                const float2 tt = __ffma2_rn(make_float2(__uint_as_float(dpv[i]), __uint_as_float(dpv[i + 1])), s2, nd2);
                const float2 ds = __fmul2_rn(pr, tt);
                pk[i / 2] = ptx::pack_half2(ds.x, ds.y);
            }
            if (j > 0) {
                ok = ptx::mbar_wait(dq_done, (uint32_t)(j - 1) & 1u, abort_flag);   // dS of tile j-1 consumed
                if (!ok) break;
                ptx::tc_fence_after_sync();
            }
            ptx::tmem_st_cols<CW / 2>(t_ds, pk);
            ptx::tmem_wait_st();
            arrive_warp(ds_full);
        }
        if (run && ok) {
            ok = ptx::mbar_wait(dq_done, (uint32_t)(n_tiles - 1) & 1u, abort_flag);
            ptx::tc_fence_after_sync();
        }
        if (run && !ok) { *abort_flag = 1; ptx::report(p.status, BWD_ERR_ROWS); }
        // every load and MMA of this CTA is done: the operand tiles make room for the result
        if (ok || (split > 1 && n_tiles == 0)) {
#pragma unroll
            for (int cc = 0; cc < D / 32 / Cfg::WGS; ++cc) {
                const int c = (cc * Cfg::WGS + wg) * 32;       // the warpgroups share the row's chunks
                stage_grad32<D>(sbase, t_dq + c, r, c, ok);
            }
        }
    }

    ptx::tc_fence_before_sync();
    if (split > 1) cooperative_groups::this_cluster().sync();
    else __syncthreads();
    // a row without any visible key: the forward row is 0/0, and so is its gradient
    if (*abort_flag == 0)
        store_grad<D, Cfg::THREADS>(smem, p.dq + ((size_t)bh * p.Sq + q0) * D, D, p.Sq - q0, rank, split, n_all == 0,
                                    __int_as_float(0x7fc00000), tid);
    else
        for (int i = 0; i < 64; ++i) __nanosleep(2000);
    if (warp == 1) {
        ptx::tc_fence_after_sync();
        ptx::tmem_dealloc(tmem, Cfg::TMEM_COLS);
    }
    if (split > 1) cooperative_groups::this_cluster().sync();       // nobody leaves while its shared memory is read
}

// ------------------------------------------------------------------ dK, dV
// PS_SMEM: P^T and dS^T are staged in shared memory (SS-form MMAs) instead of tensor memory, which
// brings the CTA down to 256 tensor-memory columns at d = 64 so that two CTAs share an SM.
// NS / NSD: depth of the Q / dO ring; both stages are read twice (K-major for S^T / dP^T, MN-major for
// dK / dV) and stay occupied until the second read is done.
// ZS: CTAs (side by side in the 1-D grid) that share one key tile, each accumulating D/ZS columns of dK and dV (both form the whole
// S^T and dP^T): at d = 256 the two accumulators of one CTA would need all 512 tensor-memory columns.
template <int D_, int BQ_, int NS_, int WGS_ = 1, bool PS_SMEM_ = false, int NSD_ = NS_, int ZS_ = 1>
struct BwdDkvCfg {
    static constexpr int D = D_, BQ = BQ_, NS = NS_, NSD = NSD_, BMK = 128, WGS = WGS_, ZS = ZS_;
    static constexpr int DA = D / ZS;                        // gradient columns this CTA accumulates
    static constexpr bool PS_SMEM = PS_SMEM_;
    static constexpr int CW = BQ / WGS;                      // tile columns (queries) per warpgroup
    static constexpr int THREADS = 64 + 128 * WGS;
    static constexpr int KP = D / 64;
    static constexpr uint32_t KV_BYTES = BMK * D * 2;        // resident K tile, V tile
    static constexpr uint32_t Q_BYTES = BQ * D * 2;          // one Q or dO stage
    static constexpr uint32_t Q_PANEL = BQ * 128;
    static constexpr uint32_t OFF_K = 0, OFF_V = KV_BYTES, OFF_Q = 2 * KV_BYTES, OFF_DO = OFF_Q + NS * Q_BYTES;
    static constexpr uint32_t PS_BYTES = PS_SMEM ? BMK * BQ * 2 : 0;  // P^T / dS^T tile when staged in shared memory
    static constexpr uint32_t OFF_PS = OFF_DO + NSD * Q_BYTES, OFF_DSS = OFF_PS + PS_BYTES;
    static constexpr uint32_t OFF_STAT = OFF_DSS + PS_BYTES;          // float lse[2][BQ], delta[2][BQ]
    static constexpr uint32_t OFF_BAR = OFF_STAT + 4 * BQ * 4;
    // barriers: kv_full, s_full, dp_full, s_free, pds_full, pds_done, q_full/q_empty[NS], do_full/do_empty[NSD]
    static constexpr int N_BARS = 6 + 2 * NS + 2 * NSD;
    static constexpr uint32_t OFF_TMEM = OFF_BAR + N_BARS * 8;
    static constexpr uint32_t OFF_ABORT = OFF_TMEM + 4;
    static constexpr uint32_t SMEM_BYTES = ((OFF_ABORT + 4 + 127) / 128) * 128;
    // tensor memory: S^T [BQ] | dP^T [BQ] | dK [D] | dV [D] | P^T fp16 [BQ/2] | dS^T fp16 [BQ/2]
    static constexpr uint32_t COL_S = 0, COL_DP = BQ, COL_DK = 2 * BQ, COL_DV = 2 * BQ + DA, COL_P = 2 * BQ + 2 * DA,
                              COL_DS = 2 * BQ + 2 * DA + BQ / 2;
    static constexpr uint32_t COLS_USED = (PS_SMEM ? 2 : 3) * BQ + 2 * DA;
    static constexpr uint32_t TMEM_COLS = COLS_USED <= 256 ? 256 : 512;
    static constexpr int CTAS_PER_SM = (SMEM_BYTES <= 115712 && TMEM_COLS <= 256) ? 2 : 1;
    static_assert(D % 64 == 0 && DA % 64 == 0 && CW % 32 == 0 && (DA / 32) % WGS == 0 && 2 * BQ <= 128 * WGS &&
                      COLS_USED <= 512 && SMEM_BYTES <= 232448 && (!PS_SMEM || BQ == 64), "tile shape");
    static_assert(2 * BMK * DA * 4 <= OFF_STAT, "the staged dK and dV tiles lie over the operand tiles");
    static_assert(NS >= 2 && NSD >= 2, "Q and dO stages are held from their first read to their second");
};

template <class Cfg>
__global__ void __launch_bounds__(Cfg::THREADS, Cfg::CTAS_PER_SM)
sdpa_bwd_dkv_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_do,
                    const __grid_constant__ CUtensorMap tm_k, const __grid_constant__ CUtensorMap tm_v,
                    const BwdParams p)
{
    constexpr int D = Cfg::D, DA = Cfg::DA, BQ = Cfg::BQ, NS = Cfg::NS, NSD = Cfg::NSD, BMK = Cfg::BMK;
    extern __shared__ __align__(1024) uint8_t smem[];
    const uint32_t sbase = ptx::smem_u32(smem);
    const uint32_t k_s = sbase + Cfg::OFF_K, v_s = sbase + Cfg::OFF_V, q_s = sbase + Cfg::OFF_Q,
                   do_s = sbase + Cfg::OFF_DO;
    float *stat = reinterpret_cast<float *>(smem + Cfg::OFF_STAT);   // [stage][0: -lse, 1: -delta*scale][BQ]
    const uint32_t bar0 = sbase + Cfg::OFF_BAR;
    const uint32_t kv_full = bar0, s_full = bar0 + 8, dp_full = bar0 + 16, s_free = bar0 + 24,
                   pds_full = bar0 + 32, pds_done = bar0 + 40;
    const uint32_t q_full = bar0 + 48, q_empty = q_full + 8 * NS, do_full = q_empty + 8 * NS,
                   do_empty = do_full + 8 * NSD;
    volatile uint32_t *tmem_slot = reinterpret_cast<volatile uint32_t *>(smem + Cfg::OFF_TMEM);
    volatile int *abort_flag = reinterpret_cast<volatile int *>(smem + Cfg::OFF_ABORT);

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    // work item: column part fastest, then group-major and longest first over the group's slabs (with a causal
    // mask the FIRST key tiles are seen by most queries)
    const int split = p.split_k, rank = (int)blockIdx.x % split, part = (int)blockIdx.x / split;
    const int item = part / Cfg::ZS;
    const int span = p.group_k * p.items_k;
    const int grp = item / span, rem = item % span;
    const int in_grp = min(p.group_k, p.slabs_k - grp * p.group_k);
    const int key0 = (rem / in_grp) * BMK;
    const int col0 = (part % Cfg::ZS) * DA;          // first dK / dV column of this CTA
    const int kvh = grp * p.group_k + rem % in_grp;             // b * Hkv + kv head
    const int b = kvh / p.Hkv;
    const int group = p.Hq / p.Hkv;
    const int bh0 = b * p.Hq + (kvh % p.Hkv) * group;           // first query head of the group
    int kv_limit = p.Sk;
    kv_limit = p.kv_lens.limit(b, kv_limit);
    const int nq = (p.Sq + BQ - 1) / BQ;
    // causal: query rows below the tile's first key see none of its keys
    const int i_start = p.causal ? min(key0 / BQ, nq) : 0;
    const int per_head = (key0 < kv_limit) ? nq - i_start : 0;  // a tile beyond the valid keys gets zero gradients
    const int n_all = per_head * group;
    const int n_it = n_all > rank ? (n_all - rank + split - 1) / split : 0;         // tiles rank, rank + split, ...
    auto tile_of = [&](int t, int &head, int &row0) {           // query head and first query row of this CTA's tile t
        const int g = rank + t * split, hd = g / per_head;
        head = bh0 + hd;
        row0 = (i_start + g - hd * per_head) * BQ;
    };
    auto load_q = [&](int t) {
        const int s = t % NS;
        int bhq, qr0;
        tile_of(t, bhq, qr0);
        ptx::mbar_arrive_expect_tx(q_full + 8 * s, Cfg::Q_BYTES);
#pragma unroll
        for (int pn = 0; pn < Cfg::KP; ++pn)
            ptx::tma_load_3d(q_s + s * Cfg::Q_BYTES + pn * Cfg::Q_PANEL, &tm_q, q_full + 8 * s, pn * 64, qr0, bhq);
    };
    auto load_do = [&](int t) {
        const int s = t % NSD;
        int bhq, qr0;
        tile_of(t, bhq, qr0);
        ptx::mbar_arrive_expect_tx(do_full + 8 * s, Cfg::Q_BYTES);
#pragma unroll
        for (int pn = 0; pn < Cfg::KP; ++pn)
            ptx::tma_load_3d(do_s + s * Cfg::Q_BYTES + pn * Cfg::Q_PANEL, &tm_do, do_full + 8 * s, pn * 64, qr0, bhq);
    };

    if (tid == 0) {
        *abort_flag = 0;
        ptx::mbar_init(kv_full, 1);
        ptx::mbar_init(s_full, 1);
        ptx::mbar_init(dp_full, 1);
        ptx::mbar_init(s_free, 4 * Cfg::WGS);
        ptx::mbar_init(pds_full, 4 * Cfg::WGS);
        ptx::mbar_init(pds_done, 1);
        for (int s = 0; s < NS; ++s) {
            ptx::mbar_init(q_full + 8 * s, 1);
            ptx::mbar_init(q_empty + 8 * s, 1);
        }
        for (int s = 0; s < NSD; ++s) {
            ptx::mbar_init(do_full + 8 * s, 1);
            ptx::mbar_init(do_empty + 8 * s, 1);
        }
        ptx::fence_mbar_init();
        if (sbase & 1023u) {
            *abort_flag = 1;
            ptx::report(p.status, TC_ERR_ALIGN);
        } else if (n_it > 0) {
            // the first loads run under the tensor-memory allocation and the meeting
            ptx::mbar_arrive_expect_tx(kv_full, 2 * Cfg::KV_BYTES);
#pragma unroll
            for (int pn = 0; pn < Cfg::KP; ++pn)
                ptx::tma_load_3d(k_s + pn * (BMK * 128), &tm_k, kv_full, pn * 64, key0, kvh);
            load_q(0);
#pragma unroll
            for (int pn = 0; pn < Cfg::KP; ++pn)
                ptx::tma_load_3d(v_s + pn * (BMK * 128), &tm_v, kv_full, pn * 64, key0, kvh);
            // From here on the preprocess' results are read (by the row warps behind the meeting).  The word stands: every
            // CTA of the dQ kernel let this one start after it was stored.  Were it not seen, waiting for that kernel's end
            // would do as well.
            if (ptx::load_acquire(p.prepared) != 1) ptx::grid_wait();
            ptx::fence_proxy_async();
            load_do(0);
        }
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
    const bool run = (*abort_flag == 0) && n_it > 0;

    if (warp == 0) {
        if (run) {
            const bool leader = ptx::elect_one();
            bool ok = true;
            // tile 0 went out before the meeting: no wait is taken on its behalf (its stages may be released already)
            for (int t = 1; t < n_it && ok; ++t) {
                ok = ptx::mbar_wait(q_empty + 8 * (t % NS), ((uint32_t)(t / NS) & 1u) ^ 1u, abort_flag);
                if (!ok) break;
                if (leader) load_q(t);
                __syncwarp();
                ok = ptx::mbar_wait(do_empty + 8 * (t % NSD), ((uint32_t)(t / NSD) & 1u) ^ 1u, abort_flag);
                if (!ok) break;
                if (leader) load_do(t);
                __syncwarp();
            }
            if (!ok && leader) { *abort_flag = 1; ptx::report(p.status, BWD_ERR_PRODUCER); }
        }
    } else if (warp == 1) {
        if (run) {
            const bool leader = ptx::elect_one();
            constexpr uint32_t idesc_s = ptx::idesc_f16(BMK, BQ, false);    // S^T, dP^T: both operands K-major
            constexpr uint32_t idesc_g = ptx::idesc_f16(BMK, DA, true);     // dV, dK: B = dO / Q tile read MN-major
            constexpr uint32_t desc_hi = ptx::smem_desc_sw128_hi(1024);
            const uint32_t k_lo = ptx::smem_desc_sw128_lo(k_s, 16);
            const uint32_t v_lo = ptx::smem_desc_sw128_lo(v_s, 16);
            const uint32_t q_lo = ptx::smem_desc_sw128_lo(q_s, 16);
            const uint32_t do_lo = ptx::smem_desc_sw128_lo(do_s, 16);
            // MN-major reads start at this CTA's first 64-column panel
            const uint32_t pan0 = (uint32_t)(col0 / 64) * Cfg::Q_PANEL;
            const uint32_t qmn_lo = ptx::smem_desc_sw128_lo(q_s + pan0, Cfg::Q_PANEL);
            const uint32_t domn_lo = ptx::smem_desc_sw128_lo(do_s + pan0, Cfg::Q_PANEL);
            const uint32_t ps_lo = ptx::smem_desc_sw128_lo(sbase + Cfg::OFF_PS, 16);
            const uint32_t dss_lo = ptx::smem_desc_sw128_lo(sbase + Cfg::OFF_DSS, 16);
            const uint32_t t_s = tmem + Cfg::COL_S, t_dp = tmem + Cfg::COL_DP, t_dk = tmem + Cfg::COL_DK,
                           t_dv = tmem + Cfg::COL_DV, t_p = tmem + Cfg::COL_P, t_ds = tmem + Cfg::COL_DS;
            bool ok = ptx::mbar_wait(kv_full, 0, abort_flag);
            auto issue_s_dp = [&](int t) -> bool {
                const int s = t % NS;
                const uint32_t ph = (uint32_t)(t / NS) & 1u;
                const uint32_t st_off = (uint32_t)s * (Cfg::Q_BYTES >> 4);
                if (!ptx::mbar_wait(q_full + 8 * s, ph, abort_flag)) return false;
                ptx::tc_fence_after_sync();
                if (leader) {
#pragma unroll
                    for (int kk = 0; kk < D / 16; ++kk) {
                        const uint32_t a = ((kk >> 2) * (BMK * 128) + (kk & 3) * 32) >> 4;
                        const uint32_t bb = ((kk >> 2) * Cfg::Q_PANEL + (kk & 3) * 32) >> 4;
                        ptx::mma_ss(t_s, ptx::make_desc(k_lo + a, desc_hi), ptx::make_desc(q_lo + st_off + bb, desc_hi),
                                    idesc_s, kk > 0);
                    }
                    ptx::mma_commit(s_full);
                }
                __syncwarp();
                const int sd = t % NSD;
                const uint32_t phd = (uint32_t)(t / NSD) & 1u;
                const uint32_t sd_off = (uint32_t)sd * (Cfg::Q_BYTES >> 4);
                if (!ptx::mbar_wait(do_full + 8 * sd, phd, abort_flag)) return false;
                ptx::tc_fence_after_sync();
                if (leader) {
#pragma unroll
                    for (int kk = 0; kk < D / 16; ++kk) {
                        const uint32_t a = ((kk >> 2) * (BMK * 128) + (kk & 3) * 32) >> 4;
                        const uint32_t bb = ((kk >> 2) * Cfg::Q_PANEL + (kk & 3) * 32) >> 4;
                        ptx::mma_ss(t_dp, ptx::make_desc(v_lo + a, desc_hi), ptx::make_desc(do_lo + sd_off + bb, desc_hi),
                                    idesc_s, kk > 0);
                    }
                    ptx::mma_commit(dp_full);
                }
                __syncwarp();
                return true;
            };
            if (ok) ok = issue_s_dp(0);
            for (int t = 0; t < n_it && ok; ++t) {
                if (t + 1 < n_it) {
                    ok = ptx::mbar_wait(s_free, (uint32_t)t & 1u, abort_flag);
                    if (!ok) break;
                    ptx::tc_fence_after_sync();
                    ok = issue_s_dp(t + 1);
                    if (!ok) break;
                }
                ok = ptx::mbar_wait(pds_full, (uint32_t)t & 1u, abort_flag);
                if (!ok) break;
                ptx::tc_fence_after_sync();
                const int s = t % NS, sd = t % NSD;
                const uint32_t st_off = (uint32_t)s * (Cfg::Q_BYTES >> 4), sd_off = (uint32_t)sd * (Cfg::Q_BYTES >> 4);
                if (leader) {
#pragma unroll
                    for (int kk = 0; kk < BQ / 16; ++kk) {
                        const uint64_t bdesc = ptx::make_desc(domn_lo + sd_off + kk * ((16 * 128) >> 4), desc_hi);
                        const uint32_t acc = (t > 0 || kk > 0) ? 1u : 0u;
                        if constexpr (Cfg::PS_SMEM)
                            ptx::mma_ss(t_dv, ptx::make_desc(ps_lo + ((kk * 32) >> 4), desc_hi), bdesc, idesc_g, acc);
                        else
                            ptx::mma_ts(t_dv, t_p + kk * 8, bdesc, idesc_g, acc);
                    }
                    ptx::mma_commit(do_empty + 8 * sd);
#pragma unroll
                    for (int kk = 0; kk < BQ / 16; ++kk) {
                        const uint64_t bdesc = ptx::make_desc(qmn_lo + st_off + kk * ((16 * 128) >> 4), desc_hi);
                        const uint32_t acc = (t > 0 || kk > 0) ? 1u : 0u;
                        if constexpr (Cfg::PS_SMEM)
                            ptx::mma_ss(t_dk, ptx::make_desc(dss_lo + ((kk * 32) >> 4), desc_hi), bdesc, idesc_g, acc);
                        else
                            ptx::mma_ts(t_dk, t_ds + kk * 8, bdesc, idesc_g, acc);
                    }
                    ptx::mma_commit(q_empty + 8 * s);
                    ptx::mma_commit(pds_done);
                }
                __syncwarp();
            }
            if (!ok && leader) { *abort_flag = 1; ptx::report(p.status, BWD_ERR_MMA); }
        }
    } else {
        constexpr int CW = Cfg::CW;
        const int quarter = warp & 3;
        const int wg = (warp - 2) >> 2;
        const int c0 = wg * CW;                     // this warpgroup's first query column of every tile
        const int r = quarter * 32 + lane;          // key row inside the tile = TMEM lane
        const int key = key0 + r;
        const int st = tid - 64;                    // 0 .. 128*WGS-1 among the row warps
        const uint32_t lane_base = (uint32_t)(quarter * 32) << 16;
        const uint32_t t_s = tmem + lane_base + Cfg::COL_S + c0, t_dp = tmem + lane_base + Cfg::COL_DP + c0,
                       t_dk = tmem + lane_base + Cfg::COL_DK, t_dv = tmem + lane_base + Cfg::COL_DV,
                       t_p = tmem + lane_base + Cfg::COL_P + c0 / 2, t_ds = tmem + lane_base + Cfg::COL_DS + c0 / 2;
        const bool key_ok = key < kv_limit;
        bool ok = run;
        auto arrive_warp = [&](uint32_t bar) {
            ptx::tc_fence_before_sync();
            __syncwarp();
            if (lane == 0) ptx::mbar_arrive(bar);
        };
        // The row statistics of a tile's queries: requested one tile ahead (a thread holds one of them; asking for them
        // where they are needed cost 870 of 2 310 cycles a tile at d = 128), through shared memory to all row warps.
        // The value stays as it was loaded until it is stored: arithmetic on it here would wait for it here.
        const float *stat_src = st < BQ ? p.lse : p.delta;
        const float stat_mul = st < BQ ? -1.f : -p.scale;                        // -lse, -D*scale
        int head_n = 0, i_n = rank;                                              // tile t + 1: head of the group, query tile
        auto settle = [&]() { while (i_n >= per_head && per_head > 0) { i_n -= per_head; ++head_n; } };
        auto fetch_stat = [&]() -> float {
            float v = st < BQ ? INFINITY : 0.f;                                  // no such query: -lse = -inf, P = 0
            const int qrow = (i_start + i_n) * BQ + (st < BQ ? st : st - BQ);
            if (head_n < group && st < 2 * BQ && qrow < p.Sq) v = stat_src[(size_t)(bh0 + head_n) * p.Sq + qrow];
            return v;
        };
        settle();
        float next_stat = fetch_stat();
        for (int t = 0; t < n_it; ++t) {
            // All row warps take every iteration's named barrier, also after a failed wait, so
            // that none of them is left behind at it.
            const int qr0 = (i_start + i_n) * BQ;
            float *st_lse = stat + (t & 1) * 2 * BQ, *st_delta = st_lse + BQ;
            if (st < 2 * BQ) st_lse[st] = stat_mul * next_stat;
            if constexpr (Cfg::WGS == 1) asm volatile("bar.sync 1, 128;" ::: "memory");
            else asm volatile("bar.sync 1, 256;" ::: "memory");
            i_n += split;
            settle();
            next_stat = fetch_stat();
            if (!ok) continue;
            ok = ptx::mbar_wait(s_full, (uint32_t)t & 1u, abort_flag);
            if (!ok) continue;
            ptx::tc_fence_after_sync();
            uint32_t sv[CW], dpv[CW];
            ptx::tmem_ld_cols<CW>(t_s, sv);
            ok = ptx::mbar_wait(dp_full, (uint32_t)t & 1u, abort_flag);
            if (!ok) continue;
            ptx::tc_fence_after_sync();
            ptx::tmem_ld_cols<CW>(t_dp, dpv);
            ptx::tmem_wait_ld();
            ptx::reg_fence_cols<CW>(sv);
            ptx::reg_fence_cols<CW>(dpv);
            arrive_warp(s_free);
            const int qc0 = qr0 + c0;               // first query of this warpgroup's columns
            const bool need_mask = p.causal && (key0 + BMK - 1 > qc0);
            const int key_lo = key - qc0 - 1;
            uint32_t pp[CW / 2], pd[CW / 2];
            const float2 c2 = make_float2(p.scale_log2, p.scale_log2), s2 = make_float2(p.scale, p.scale);
#pragma unroll
            for (int i = 0; i < CW; i += 2) {
                // packed fp32 pairs; the two queries' statistics sit side by side in shared memory
                const float2 l2 = *reinterpret_cast<const float2 *>(st_lse + c0 + i);
                const float2 dl = *reinterpret_cast<const float2 *>(st_delta + c0 + i);
                const float2 x = __ffma2_rn(make_float2(__uint_as_float(sv[i]), __uint_as_float(sv[i + 1])), c2, l2);
                float2 pr = make_float2(ptx::ex2_approx(x.x), ptx::ex2_approx(x.y));
                if (!key_ok) pr = make_float2(0.f, 0.f);
                if (need_mask) {                 // query qc0 + i sees this key when key <= qc0 + i
                    pr.x = ptx::zero_unless_lt(pr.x, key_lo, i);
                    pr.y = ptx::zero_unless_lt(pr.y, key_lo, i + 1);
                }
                const float2 tt = __ffma2_rn(make_float2(__uint_as_float(dpv[i]), __uint_as_float(dpv[i + 1])), s2,
                                             dl);
                const float2 ds = __fmul2_rn(pr, tt);
                pp[i / 2] = ptx::pack_half2(pr.x, pr.y);
                pd[i / 2] = ptx::pack_half2(ds.x, ds.y);
            }
            if (t > 0) {
                ok = ptx::mbar_wait(pds_done, (uint32_t)(t - 1) & 1u, abort_flag);
                if (!ok) continue;
                ptx::tc_fence_after_sync();
            }
            if constexpr (Cfg::PS_SMEM) {
                // row r of the [128 keys][64 queries] tile: 128 bytes = 8 chunks of 8 halves, chunk ^= r % 8
                const uint32_t prow = sbase + Cfg::OFF_PS + (uint32_t)r * 128, drow = sbase + Cfg::OFF_DSS + (uint32_t)r * 128;
#pragma unroll
                for (int ch = 0; ch < 8; ++ch) {
                    const uint32_t sw = ((uint32_t)ch ^ (uint32_t)(r & 7)) << 4;
                    ptx::st_shared_v4(prow + sw, pp[ch * 4], pp[ch * 4 + 1], pp[ch * 4 + 2], pp[ch * 4 + 3]);
                    ptx::st_shared_v4(drow + sw, pd[ch * 4], pd[ch * 4 + 1], pd[ch * 4 + 2], pd[ch * 4 + 3]);
                }
                ptx::fence_proxy_async_smem();
            } else {
                ptx::tmem_st_cols<CW / 2>(t_p, pp);
                ptx::tmem_st_cols<CW / 2>(t_ds, pd);
                ptx::tmem_wait_st();
            }
            arrive_warp(pds_full);
        }
        if (run && ok) {
            ok = ptx::mbar_wait(pds_done, (uint32_t)(n_it - 1) & 1u, abort_flag);
            ptx::tc_fence_after_sync();
        }
        if (run && !ok) { *abort_flag = 1; ptx::report(p.status, BWD_ERR_ROWS); }
        // every load and MMA of this CTA is done: the operand tiles make room for the result
        if (ok || (split > 1 && n_it == 0)) {
#pragma unroll
            for (int cc = 0; cc < DA / 32 / Cfg::WGS; ++cc) {
                const int c = (cc * Cfg::WGS + wg) * 32;       // the warpgroups share the row's chunks
                stage_grad32<DA>(sbase, t_dk + c, r, c, ok);
                stage_grad32<DA>(sbase + BMK * DA * 4, t_dv + c, r, c, ok);
            }
        }
    }

    ptx::tc_fence_before_sync();
    if (split > 1) cooperative_groups::this_cluster().sync();
    else __syncthreads();
    if (*abort_flag == 0) {
        // keys no query sees: zero gradients -- unless the batch element has no valid key at
        // all, where the forward rows are 0/0 and the reference's rule propagates NaN to every gradient
        const float fill = kv_limit == 0 ? __int_as_float(0x7fc00000) : 0.f;
        const size_t gbase = ((size_t)kvh * p.Sk + key0) * D + col0;
        store_grad<DA, Cfg::THREADS>(smem, p.dk + gbase, D, p.Sk - key0, rank, split, n_all == 0, fill, tid);
        store_grad<DA, Cfg::THREADS>(smem + BMK * DA * 4, p.dv + gbase, D, p.Sk - key0, rank, split, n_all == 0, fill, tid);
    } else {
        for (int i = 0; i < 64; ++i) __nanosleep(2000);
    }
    // This kernel reads nothing the dQ kernel writes and starts under its last CTAs; it must not end before it, though:
    // what follows in the stream takes both for done.
    if (tid == 0) ptx::grid_wait();
    if (warp == 1) {
        ptx::tc_fence_after_sync();
        ptx::tmem_dealloc(tmem, Cfg::TMEM_COLS);
    }
    if (split > 1) cooperative_groups::this_cluster().sync();       // nobody leaves while its shared memory is read
}

}  // namespace txb

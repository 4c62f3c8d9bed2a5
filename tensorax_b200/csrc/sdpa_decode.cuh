// Attention for few query rows per K/V head -- one decoding step against a K/V cache -- for sm_100a, fp16 and fp32.
//
// Bound: HBM.  Every key and value is used by at most a handful of query rows, so the tensor-core kernels (128 query
// rows per tile, one CTA walking all keys of a head, fp32 operands split into hi / lo copies first) spend their time on
// padding, on one serial chain of key tiles and on extra passes over the cache.  Here the keys of one (batch, K/V head)
// are cut over the CTAs of a thread-block cluster, each key and value is read from memory once for all query rows that
// share the head, and the partial results meet in distributed shared memory: no workspace, no second launch.
//
//   warp 7      producer: consecutive keys of a head are one contiguous block, so a stage is two bulk copies (K, V)
//   warps 0-6   LPK lanes share one key: each holds EPL elements of every query row and of every output row in
//               registers; scores are summed over the LPK lanes by shuffles (the sum then sits in all of them, so
//               P needs no exchange before P V); fp32 FMAs throughout, online softmax per lane group with the rescale of
//               O skipped while no lane of the warp saw a larger score
// Group, warp and CTA partials (max, sum, O) are merged at the end, CTAs of the cluster through ld.shared::cluster in
// rank order: results are the same bits on every run.
//
// Measured on B200, fp32, B8 Hq32 Hkv8 d128, 4096 keys of which three quarters are valid (202 MB): 42 us = 4.8 TB/s, where
// the split pass + tensor-core kernel took 253 us; d64, one query head per K/V head: 5.5 TB/s.  The rest is latency: 127
// registers a thread leave 14 row warps per SM, which issue in 0.34 of the cycles at four rows a head, and about 6 us of
// start, cluster barriers and merge are outside the loop.
//
// Semantics as in the other kernels (tensorax csrc/cpu/tensor_cpu.cpp:489-515): scores are dot * scale + mask in the
// natural-log domain with the running max starting at -FLT_MAX, a row without a visible key ends in 0/0.
// Every mbarrier wait is bounded.
#pragma once
#include <cfloat>
#include <cooperative_groups.h>

#include "ptx.cuh"

namespace txb {

enum : int { DEC_ERR_PRODUCER = 32, DEC_ERR_ROWS = 34 };

struct DecodeParams {
    const void *q, *k, *v;    // [B,Hq,Sq,D], [B,Hkv,Sk,D] x 2
    const float *mask;        // optional dense additive [B,Hq,Sq,Sk]
    KvLens kv_lens;           // optional [B]
    void *out;                // [B,Hq,Sq,D] fp32, or fp16 when out_f16
    float *lse;               // optional [B,Hq,Sq], as the tensor-core kernels write it (log2 domain)
    int *status;
    int Hkv, Sq, Sk;
    int rows;                 // query rows of one K/V head: (Hq / Hkv) * Sq
    int row_parts;            // CTAs (per split) that share them, R rows each
    int causal, out_f16;
    float scale;              // 1/sqrt(d)
};

template <typename T_, int D_, int R_>
struct DecodeCfg {
    using T = T_;
    static constexpr int D = D_, R = R_, WARPS = 7;
    static constexpr int VEC = 16 / (int)sizeof(T);                      // elements of one 16-byte load
    // a lane keeps R x EPL query and R x EPL output elements in registers; LPK * 16 bytes are read side by side
    static constexpr int EPL = (D == 64 || R == 4) ? 8 : 16, LPK = D / EPL, NV = EPL / VEC;
    static constexpr int GROUPS = 32 / LPK;                              // keys a warp works on at a time
    static constexpr int U = 2;                                          // such keys per lane group and stage
    static constexpr int N = U * R;                                      // scores of a lane group per stage
    static constexpr int KEYS = WARPS * GROUPS * U;
    static constexpr uint32_t ROW = D * sizeof(T), TILE = KEYS * ROW;    // one of K, V
    static constexpr uint32_t MERGE = (WARPS + 1) * R * D * 4;           // [WARPS + 1][R][D] partial sums
    static constexpr uint32_t WANT = MERGE > 65536 ? MERGE : 65536;
    static constexpr int NS_WANT = (WANT + 2 * TILE - 1) / (2 * TILE), NS = NS_WANT < 3 ? 3 : NS_WANT;
    static constexpr uint32_t RING = NS * 2 * TILE;
    static constexpr uint32_t OFF_BAR = RING;                            // full[NS], empty[NS]
    static constexpr uint32_t OFF_ABORT = OFF_BAR + 2 * NS * 8;
    static constexpr uint32_t OFF_ML = OFF_ABORT + 16;                   // float [WARPS + 1][R][2]: warps, then the CTA
    static constexpr uint32_t SMEM = OFF_ML + (WARPS + 1) * R * 8;
    static constexpr int THREADS = (WARPS + 1) * 32, MAX_SPLITS = 16;
    // CTAs an SM holds (228 KB, 1 KB of it per CTA taken): one in fp32 at d = 128 and 256 with up to two rows.  Counting on two
    // there cut the keys into two waves of clusters: B4 Hkv8 Sk1000 d128 24.6 us, 16.4 with one; B9 Hkv8 Sk4096 75.8 and 66.7.
    static constexpr int CTAS_PER_SM = 2 * (SMEM + 1024) <= 233472 ? 2 : 1;
    static_assert(R == 1 || R == 2 || R == 4, "more rows are shared out over CTAs (eight in one: slower at every size)");
    static_assert(LPK >= 8 && LPK <= 32 && NV >= 1 && NV * VEC == EPL, "lane layout");
    static_assert(MERGE <= RING, "partial results are merged in the drained ring");
};

__device__ __forceinline__ void dec_unpack(const uint4 &u, float *f, float)
{
    f[0] = __uint_as_float(u.x); f[1] = __uint_as_float(u.y); f[2] = __uint_as_float(u.z); f[3] = __uint_as_float(u.w);
}
__device__ __forceinline__ void dec_unpack(const uint4 &u, float *f, __half)
{
    const __half2 *h = reinterpret_cast<const __half2 *>(&u);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const float2 x = __half22float2(h[i]);
        f[2 * i] = x.x; f[2 * i + 1] = x.y;
    }
}

// The log2(N) low bits of x in reverse order
template <int N>
__device__ __forceinline__ constexpr int dec_reverse(int x)
{
    int r = 0;
    for (int b = 1; b < N; b <<= 1, x >>= 1) r = 2 * r + (x & 1);
    return r;
}

template <class Cfg>
__global__ void __launch_bounds__(Cfg::THREADS, 2)
sdpa_decode_kernel(const DecodeParams p)
{
    using T = typename Cfg::T;
    constexpr int D = Cfg::D, R = Cfg::R, EPL = Cfg::EPL, LPK = Cfg::LPK, NV = Cfg::NV, VEC = Cfg::VEC, U = Cfg::U, N = Cfg::N, NS = Cfg::NS;
    constexpr float kLog2e = 1.4426950408889634f;
    namespace cg = cooperative_groups;
    extern __shared__ __align__(1024) uint8_t smem[];
    const uint32_t sbase = ptx::smem_u32(smem), full = sbase + Cfg::OFF_BAR, empty = full + 8 * NS;
    volatile int *abort_flag = reinterpret_cast<volatile int *>(smem + Cfg::OFF_ABORT);
    float *ml = reinterpret_cast<float *>(smem + Cfg::OFF_ML);
    float *part = reinterpret_cast<float *>(smem);                       // [WARPS + 1][R][D], once the ring is drained
    cg::cluster_group cluster = cg::this_cluster();
    const int split = (int)cluster.block_rank(), splits = (int)cluster.num_blocks();
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;

    const int item = (int)blockIdx.x / splits;
    const int kvh = item / p.row_parts, row0 = (item % p.row_parts) * R; // (batch, K/V head), first of this CTA's rows
    const int b = kvh / p.Hkv;
    int limit = p.kv_lens.limit(b, p.Sk);
    if (p.causal) limit = min(limit, p.Sq);
    // equal shares of the visible keys, whole warp rounds each
    const int share = ((limit + splits - 1) / splits + Cfg::KEYS - 1) / Cfg::KEYS * Cfg::KEYS;
    const int key0 = min(split * share, limit), n_keys = min(share, limit - key0);
    const int n_stages = (n_keys + Cfg::KEYS - 1) / Cfg::KEYS;

    auto load_stage = [&](int j) {
        const int s = j % NS;
        const uint32_t bytes = (uint32_t)min(Cfg::KEYS, n_keys - j * Cfg::KEYS) * Cfg::ROW;
        const uint32_t dst = sbase + (uint32_t)s * 2 * Cfg::TILE;
        const size_t from = ((size_t)kvh * p.Sk + key0) * Cfg::ROW + (size_t)j * Cfg::TILE;
        ptx::mbar_arrive_expect_tx(full + 8 * s, 2 * bytes);
        ptx::bulk_load(dst, static_cast<const char *>(p.k) + from, bytes, full + 8 * s);
        ptx::bulk_load(dst + Cfg::TILE, static_cast<const char *>(p.v) + from, bytes, full + 8 * s);
    };
    // the producer fills the ring before anything else; the CTA meets, and asks whether an earlier one gave up, under
    // the loads' latency
    if (tid == Cfg::WARPS * 32) {
        *abort_flag = 0;
        for (int s = 0; s < NS; ++s) {
            ptx::mbar_init(full + 8 * s, 1);
            ptx::mbar_init(empty + 8 * s, Cfg::WARPS);
        }
        ptx::fence_mbar_init();
        for (int j = 0; j < min(NS, n_stages); ++j) load_stage(j);
        if (*reinterpret_cast<volatile int *>(p.status) != 0) *abort_flag = 1;
    }
    __syncthreads();
    const bool run = *abort_flag == 0;

    if (warp == Cfg::WARPS) {
        if (run && lane == 0) {
            bool ok = true;
            for (int j = NS; j < n_stages; ++j) {
                ok = ptx::mbar_wait(empty + 8 * (j % NS), ((uint32_t)(j / NS) & 1u) ^ 1u, abort_flag);
                if (!ok) break;
                load_stage(j);
            }
            if (!ok) { *abort_flag = 1; ptx::report(p.status, DEC_ERR_PRODUCER); }
        }
        __syncthreads();            // the ring is drained
        __syncthreads();            // warp partials are in shared memory
    } else {
        const int group = lane / LPK, gl = lane % LPK;
        // Of the N scores of a round (U keys x R rows) each lane ends up with one, number `mine` = key * R + row
        // (N divides LPK; the lanes LPK / N apart hold the same one).
        const int mine = dec_reverse<N>(gl), my_u = mine / R, my_r = mine % R;
        float q[R][EPL], o[R][EPL];
        float m = -FLT_MAX, l = 0.f;                                     // of row my_r; l over this lane's key slot only
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const int row = min(row0 + r, p.rows - 1);                   // a row beyond the last repeats it, never written
            // rows of one K/V head follow each other in [B,Hq,Sq,D]: head kvh * group + row / Sq, position row % Sq
            const T *qr = static_cast<const T *>(p.q) + ((size_t)kvh * p.rows + row) * D;
#pragma unroll
            for (int j = 0; j < NV; ++j) {
                const uint4 x = *reinterpret_cast<const uint4 *>(qr + (j * LPK + gl) * VEC);
                dec_unpack(x, &q[r][j * VEC], T());
            }
#pragma unroll
            for (int i = 0; i < EPL; ++i) o[r][i] = 0.f;
        }
        const int my_row = min(row0 + my_r, p.rows - 1);
        const int my_lim = p.causal ? min(limit, my_row % p.Sq + 1) : limit;
        const float *my_mask = p.mask ? p.mask + ((size_t)kvh * p.rows + my_row) * p.Sk : nullptr;
        const int kl = warp * Cfg::GROUPS * U + group;                   // this lane group's keys of a stage: kl + u * GROUPS
        const int my_kl = kl + my_u * Cfg::GROUPS;
        bool ok = run;
        for (int j = 0; j < n_stages && ok; ++j) {
            const int s = j % NS;
            float mk = 0.f;
            if (p.mask) mk = __ldg(my_mask + min(key0 + j * Cfg::KEYS + my_kl, p.Sk - 1));
            ok = ptx::mbar_wait(full + 8 * s, (uint32_t)(j / NS) & 1u, abort_flag);
            if (!ok) break;
            const uint8_t *kt = smem + (size_t)s * 2 * Cfg::TILE + (size_t)kl * Cfg::ROW + gl * 16;
            const uint8_t *vt = kt + Cfg::TILE;
            float sc[N];
#pragma unroll
            for (int u = 0; u < U; ++u) {
                float kf[EPL];
#pragma unroll
                for (int i = 0; i < NV; ++i)
                    dec_unpack(*reinterpret_cast<const uint4 *>(kt + (size_t)u * Cfg::GROUPS * Cfg::ROW + i * LPK * 16), &kf[i * VEC], T());
#pragma unroll
                for (int r = 0; r < R; ++r) {
                    float2 a = make_float2(0.f, 0.f);
#pragma unroll
                    for (int i = 0; i < EPL; i += 2)
                        a = __ffma2_rn(make_float2(q[r][i], q[r][i + 1]), make_float2(kf[i], kf[i + 1]), a);
                    sc[u * R + r] = a.x + a.y;
                }
            }
            // Sums over the group's lanes.  Each step hands half of the values to the partner and keeps the other half,
            // so N values cost N - 1 + log2(LPK / N) shuffles instead of N * log2(LPK), and the softmax below is done
            // once per score instead of in every lane.
#pragma unroll
            for (int w = 1, n = N / 2; n > 0; w <<= 1, n >>= 1)
#pragma unroll
                for (int i = 0; i < n; ++i) {
                    const bool up = (gl & w) != 0;
                    const float keep = up ? sc[i + n] : sc[i], send = up ? sc[i] : sc[i + n];
                    sc[i] = keep + __shfl_xor_sync(0xffffffffu, send, w);
                }
#pragma unroll
            for (int w = N; w < LPK; w <<= 1) sc[0] += __shfl_xor_sync(0xffffffffu, sc[0], w);
            float x = sc[0] * p.scale + mk;
            // also true for the rows of a stage that were never filled: whatever they hold is dropped here
            if (key0 + j * Cfg::KEYS + my_kl >= my_lim) x = -INFINITY;
            float mn = fmaxf(m, x);
#pragma unroll
            for (int w = 1; w < U; w <<= 1) mn = fmaxf(mn, __shfl_xor_sync(0xffffffffu, mn, w));   // the row's other keys
            if (__any_sync(0xffffffffu, mn > m)) {
                const float a = ptx::ex2_approx((m - mn) * kLog2e);
                m = mn;
                l *= a;
#pragma unroll
                for (int r = 0; r < R; ++r) {
                    const float ar = __shfl_sync(0xffffffffu, a, dec_reverse<N>(r), LPK);
#pragma unroll
                    for (int i = 0; i < EPL; ++i) o[r][i] *= ar;
                }
            }
            const float pr = ptx::ex2_approx((x - m) * kLog2e);
            l += pr;
#pragma unroll
            for (int u = 0; u < U; ++u) {
                float pu[R];
#pragma unroll
                for (int r = 0; r < R; ++r) pu[r] = __shfl_sync(0xffffffffu, pr, dec_reverse<N>(u * R + r), LPK);
                // keys past the share were not copied: their stage rows may hold anything, NaN included
                if (j * Cfg::KEYS + kl + u * Cfg::GROUPS < n_keys) {
                    float vf[EPL];
#pragma unroll
                    for (int i = 0; i < NV; ++i)
                        dec_unpack(*reinterpret_cast<const uint4 *>(vt + (size_t)u * Cfg::GROUPS * Cfg::ROW + i * LPK * 16), &vf[i * VEC], T());
#pragma unroll
                    for (int r = 0; r < R; ++r) {
                        const float2 p2 = make_float2(pu[r], pu[r]);
#pragma unroll
                        for (int i = 0; i < EPL; i += 2) {
                            const float2 y = __ffma2_rn(p2, make_float2(vf[i], vf[i + 1]), make_float2(o[r][i], o[r][i + 1]));
                            o[r][i] = y.x; o[r][i + 1] = y.y;
                        }
                    }
                }
            }
            __syncwarp();
            if (lane == 0) ptx::mbar_arrive(empty + 8 * s);
        }
        if (run && !ok) { *abort_flag = 1; ptx::report(p.status, DEC_ERR_ROWS); }
        // key slots of the lane group, then the lane groups of the warp
#pragma unroll
        for (int w = 1; w < U; w <<= 1) l += __shfl_xor_sync(0xffffffffu, l, w);
        float mr[R], lr[R];
#pragma unroll
        for (int r = 0; r < R; ++r) {
            mr[r] = __shfl_sync(0xffffffffu, m, dec_reverse<N>(r), LPK);
            lr[r] = __shfl_sync(0xffffffffu, l, dec_reverse<N>(r), LPK);
        }
#pragma unroll
        for (int w = LPK; w < 32; w <<= 1) {
#pragma unroll
            for (int r = 0; r < R; ++r) {
                const float mo = __shfl_xor_sync(0xffffffffu, mr[r], w), lo = __shfl_xor_sync(0xffffffffu, lr[r], w);
                const float mx = fmaxf(mr[r], mo);
                const float fa = ptx::ex2_approx((mr[r] - mx) * kLog2e), fb = ptx::ex2_approx((mo - mx) * kLog2e);
                lr[r] = lr[r] * fa + lo * fb;
                mr[r] = mx;
#pragma unroll
                for (int i = 0; i < EPL; ++i) o[r][i] = o[r][i] * fa + __shfl_xor_sync(0xffffffffu, o[r][i], w) * fb;
            }
        }
        __syncthreads();                                                 // every warp is past its last stage
        if (lane < LPK) {
#pragma unroll
            for (int r = 0; r < R; ++r) {
                if (lane == 0) { ml[(warp * R + r) * 2] = mr[r]; ml[(warp * R + r) * 2 + 1] = lr[r]; }
#pragma unroll
                for (int i = 0; i < EPL; ++i)
                    part[(warp * R + r) * D + ((i / VEC) * LPK + gl) * VEC + i % VEC] = o[r][i];
            }
        }
        __syncthreads();
    }
    // warps of the CTA
    float *cta_part = part + Cfg::WARPS * R * D, *cta_ml = ml + Cfg::WARPS * R * 2;
    for (int i = tid; i < R * D; i += Cfg::THREADS) {
        const int r = i / D;
        float mn = -FLT_MAX;
#pragma unroll
        for (int w = 0; w < Cfg::WARPS; ++w) mn = fmaxf(mn, ml[(w * R + r) * 2]);
        float acc = 0.f, ls = 0.f;
#pragma unroll
        for (int w = 0; w < Cfg::WARPS; ++w) {
            const float f = ptx::ex2_approx((ml[(w * R + r) * 2] - mn) * kLog2e);
            acc += f * part[w * R * D + i];
            ls += f * ml[(w * R + r) * 2 + 1];
        }
        cta_part[i] = acc;
        if (i % D == 0) { cta_ml[r * 2] = mn; cta_ml[r * 2 + 1] = *abort_flag ? __int_as_float(0x7fc00000) : ls; }
    }
    // CTAs of the cluster: each writes an equal share of the rows' elements
    cluster.sync();
    for (int i = split * Cfg::THREADS + tid; i < R * D; i += splits * Cfg::THREADS) {
        const int r = i / D;
        if (row0 + r >= p.rows) break;
        // all remote loads first: they take as long as one
        constexpr int S = Cfg::MAX_SPLITS;
        float mc[S], lc[S], pc[S], mn = -FLT_MAX;
#pragma unroll
        for (int c = 0; c < S; ++c) {
            const int from = min(c, splits - 1);
            const float *ml_c = cluster.map_shared_rank(cta_ml, from);
            mc[c] = ml_c[r * 2];
            lc[c] = ml_c[r * 2 + 1];
            pc[c] = cluster.map_shared_rank(cta_part, from)[i];
        }
#pragma unroll
        for (int c = 0; c < S; ++c) mn = fmaxf(mn, mc[c]);
        float acc = 0.f, ls = 0.f;
#pragma unroll
        for (int c = 0; c < S; ++c) {
            if (c < splits) {
                const float f = ptx::ex2_approx((mc[c] - mn) * kLog2e);
                acc += f * pc[c];
                ls += f * lc[c];
            }
        }
        const size_t flat = (size_t)kvh * p.rows + row0 + r;
        const float val = acc / ls;                                      // ls == 0 (no visible key): NaN, as the reference
        if (p.out_f16) static_cast<__half *>(p.out)[flat * D + i % D] = __float2half_rn(val);
        else static_cast<float *>(p.out)[flat * D + i % D] = val;
        if (p.lse && i % D == 0) p.lse[flat] = ls > 0.f ? mn * kLog2e + __log2f(ls) : __int_as_float(0x7fc00000);
    }
    if (*abort_flag)
        for (int i = 0; i < 64; ++i) __nanosleep(2000);                  // let copies in flight land
    cluster.sync();                                                      // nobody leaves while its shared memory is read
}

}  // namespace txb

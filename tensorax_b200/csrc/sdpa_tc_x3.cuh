// fp32 flash-attention forward on the fp16 tensor cores of sm_100a: every fp32 operand is carried as the sum of
// two fp16 numbers (hi = rn(x), lo = rn(x - hi): 22 significand bits) and every product is three tcgen05 MMAs,
//     S  = Qhi Klo^T + Qlo Khi^T + Qhi Khi^T          O += Phi Vlo + Plo Vhi + Phi Vhi
// accumulated in fp32 in tensor memory (the lo*lo term is below fp32's own rounding).  It stands where the
// reference's fp32 kernels do (tensorax csrc/cuda/kernels/attn.cu:296-656 sdpa_kernel_mma and the naive / tiled /
// flash forms before it) for head dims up to 128 (multiples of 4; d_k and d_v may differ), with or without a dense
// additive mask, at any magnitude: the split pass scales every row of Q and every 64-key tile of K and V by a power of two
// that brings its largest element to [2^13, 2^14), and writes the factors.  A pair is then exact to 22 bits down to 2^-17
// of that largest element and to 2^-39 of it below.  Q's and K's factors join the softmax scale of a (row, tile), V's the
// accumulation; both are exact.  Where that is not enough (x3_declines) this kernel returns at once and the exact
// CUDA-core kernel, launched behind it, does the work.
//
// One CTA per SM and 128-row query tile, 64 keys per tile:
//   warp 0        TMA producer: Q hi / lo once, then K hi / lo and V hi / lo of every key tile through an NS-deep ring
//   warp 1        issues the MMAs: QK^T of tile j+1 as soon as the softmax warps have S_j in registers, then PV of tile j
//   warps 2-3     idle, or bring the dense mask's [128 rows][64 keys] tile to shared memory (cp.async: any row length)
//   warps 4-7     softmax, thread = row = tensor-memory lane: fp32 online softmax with the exact running max
//                 (full-precision `ex2.approx`, no polynomial), 2^14 P split into hi / lo in registers and stored to
//                 tensor memory as two fp16 operands; the row's rescale factor of the tile goes to shared memory
//   warps 8-11    accumulators, thread = row: O lives in REGISTERS.  Each tile's P V is a fresh tensor-memory
//                 accumulator (12 MMAs) that these warps fold in with O = O * alpha + PV, rounded to nearest.  The
//                 tensor core's own fp32 accumulation truncates, and carried over hundreds of key tiles that bias
//                 grows with the sequence length; twelve steps of it stay below fp32's rounding of the result.
//                 They also write the result (staged bulk tensor stores).
// The operands are the split pass's fp16 copies, their rows padded to a multiple of 8; the last 64-column panel is
// filled with zeros by the TMA unit, QK^T runs ceil(d_k / 16) steps and PV's N is d_v rounded up to 16, so a head dim
// between the two template sizes costs what it needs (fp32 B2 H8 S1000 d80: 608 -> 62 us a call against the CUDA-core kernel).
// Dense mask: scores stay in the natural-log domain (x = s * scale + mask, p = 2^((x - m) log2 e)) with the running max
// starting at -FLT_MAX, so that rows masked by the lowest floats average V and rows masked by -inf are 0/0, as in the
// reference (fp32 B4 H8 S512 d64: 275 -> 56 us a call).
// Tensor memory: S 64 | Phi 32 | Plo 32 | PV_0 D | PV_1 D columns.
// Every mbarrier wait is bounded, as in the fp16 kernels.
#pragma once
#include <cfloat>

#include "ptx.cuh"
#include "sdpa_tc.cuh"

namespace txb {

constexpr int X3_TILE = 64;      // keys per tile, each tile of K and V with a factor of its own; the split pass's CTAs

template <int D_, int NS_, bool MASK_ = false>
struct X3Cfg {
    static constexpr int D = D_, NS = NS_;                 // D: 64 or 128, at least d_k and d_v
    static constexpr bool MASK = MASK_;
    // Stages of the mask tile, as many as shared memory has room for: the mask comes from memory, 32 KB a tile, and with two
    // stages and a rolled copy loop the softmax warps waited 1 480 of 3 060 cycles a tile for it (B4 H8 S512 d64: 49.6 -> 49.2 us
    // a call with four, 48.4 with the loop unrolled as well).
    static constexpr int NM = D_ == 64 ? 4 : 1;
    static constexpr int BM = 128, BN = X3_TILE;
    static constexpr int THREADS = 384;
    // registers: producer / MMA warpgroup, softmax warpgroup, accumulator warpgroup (128 * (56 + 192 + 248) <= 384 * 168)
    static constexpr int REGS_LIGHT = 56, REGS_SOFTMAX = 192, REGS_ACC = 248;
    static constexpr int KP = D / 64;                      // 64-column panels per row
    static constexpr uint32_t Q_BYTES = BM * D * 2;        // one of hi / lo
    static constexpr uint32_t KV_BYTES = BN * D * 2;       // one of K hi, K lo, V hi, V lo
    static constexpr uint32_t KV_PANEL = BN * 128;
    static constexpr uint32_t OFF_QH = 0, OFF_QL = Q_BYTES;
    static constexpr uint32_t OFF_K = 2 * Q_BYTES;         // per stage: K hi | K lo
    static constexpr uint32_t OFF_V = OFF_K + NS * 2 * KV_BYTES;
    static constexpr uint32_t MASK_BYTES = BM * BN * 4;
    static constexpr uint32_t OFF_MASK = OFF_V + NS * 2 * KV_BYTES;
    static constexpr uint32_t OFF_BAR = OFF_MASK + (MASK ? NM * MASK_BYTES : 0);
    // q_full s_full s_free p_full l_full pv_done[2] pv_free[2] alpha_full[4] k_full[NS] k_empty[NS] v_full[NS] v_empty[NS]
    // mask_full[NM] mask_empty[NM]
    static constexpr int N_BARS = 13 + 4 * NS + (MASK ? 2 * NM : 0);
    static constexpr uint32_t OFF_ALPHA = OFF_BAR + ((N_BARS * 8 + 15) / 16) * 16;   // [4][BM] rescale factors, then [BM] row sums
    static constexpr uint32_t OFF_TMEM = OFF_ALPHA + 5 * BM * 4;
    static constexpr uint32_t OFF_ABORT = OFF_TMEM + 4;
    static constexpr uint32_t SMEM_BYTES = ((OFF_ABORT + 4 + 127) / 128) * 128;
    static constexpr uint32_t COL_S = 0, COL_PH = BN, COL_PL = BN + BN / 2, COL_PV0 = 2 * BN, COL_PV1 = 2 * BN + D;
    static constexpr uint32_t TMEM_COLS = 512;
    static_assert(D == 64 || D == 128, "operand width");
    static_assert(2 * BN + 2 * D <= TMEM_COLS, "tensor memory");
    static_assert(SMEM_BYTES <= 232448, "more than the 227 KB a CTA may have");
    static_assert(Q_BYTES / 4 >= 4096, "a softmax warp stages its results in its quarter of the Q buffers");
};

// P is carried as 2^14 p (p <= 1), so that its pairs too are exact to 2^-39 absolutely and not to 2^-25: keys of small weight
// and large V count.  The split pass takes the factor out of V's (X3Params::vf).
constexpr float X3_P_SCALE = 16384.f;

// range[0]: some value is not finite (the split pass), or the largest elements of two keys of a head's V lie more than 2^13
// apart (this kernel, on its way; the exact kernel then does the whole call once more), so that the rounding of P and V at
// the large ones would show beside the small ones.  range[1], range[2]: the bits of max |q| and max |k|: what scaling leaves
// of a row or tile below 2^-39 of its maximum is worth up to 2^-39 max |q| max |k| in a score (sqrt(d) such terms, times
// 1 / sqrt(d)), which stays below 2^-20 here.
__device__ __forceinline__ bool x3_declines(const int *range)
{
    const volatile int *w = range;
    return w[0] != 0 || __int_as_float(w[1]) * __int_as_float(w[2]) > 524288.f;
}

struct X3Params {
    float *out;               // [B,Hq,Sq,dv] fp32
    const float *mask;        // dense additive [B,Hq,Sq,Sk] (MASK instantiations)
    KvLens kv_lens;           // optional [B]
    int *range;               // three words (see x3_declines)
    const float *qf;          // [B,Hq,Sq] what undoes the scale of a row of Q
    const float *kf, *vf;     // [B,Hkv,ceil(Sk / 64)] the same of a tile of K and V (V: and of P)
    const int *vr;            // [B,Hkv,ceil(Sk / 64)] exponent fields of the largest and the smallest key of a tile of V: max | min << 8
    int *status;              // device word: 0 = ok, else first failing wait's code
    int Hq, Hkv, Sq, Sk;
    int dk, dv;
    int causal;
    float scale;              // 1/sqrt(d_k)
    float scale_log2;         // scale * log2(e)
    int group, n_tiles_q, BH; // work-item order, as in sdpa_tc_pair_kernel (query tiles in place of pairs)
};

template <class Cfg>
__global__ void __launch_bounds__(Cfg::THREADS, 1)
sdpa_tc_x3_kernel(const __grid_constant__ CUtensorMap tm_qh, const __grid_constant__ CUtensorMap tm_ql,
                  const __grid_constant__ CUtensorMap tm_kh, const __grid_constant__ CUtensorMap tm_kl,
                  const __grid_constant__ CUtensorMap tm_vh, const __grid_constant__ CUtensorMap tm_vl,
                  const __grid_constant__ CUtensorMap tm_o, const X3Params p)
{
    constexpr int D = Cfg::D, BN = Cfg::BN, NS = Cfg::NS, BM = Cfg::BM;
    ptx::grid_trigger();
    ptx::grid_wait();                                            // the split pass
    if (x3_declines(p.range)) return;                            // the exact kernel takes this call

    extern __shared__ __align__(1024) uint8_t smem[];
    const uint32_t sbase = ptx::smem_u32(smem);
    const uint32_t qh_s = sbase + Cfg::OFF_QH, ql_s = sbase + Cfg::OFF_QL, k_s = sbase + Cfg::OFF_K, v_s = sbase + Cfg::OFF_V;
    const uint32_t bar0 = sbase + Cfg::OFF_BAR;
    const uint32_t q_full = bar0, s_full = bar0 + 8, s_free = bar0 + 16, p_full = bar0 + 24, l_full = bar0 + 32;
    const uint32_t pv_done = bar0 + 40, pv_free = bar0 + 56;     // one pair each: PV accumulator j & 1
    float *alpha_s = reinterpret_cast<float *>(smem + Cfg::OFF_ALPHA);       // [4][BM]: tile j's factors in slot j & 3
    float *l_s = alpha_s + 4 * BM;
    // Four slots and four barriers for the factors: the softmax warps reach tile j + 4 only after PV_{j+2} was
    // issued, which waited for the accumulator warps to be done with tile j -- so a slot is never rewritten, and
    // its barrier never a phase ahead, while its reader still needs it.
    const uint32_t alpha_full = bar0 + 72;
    const uint32_t k_full = bar0 + 104, k_empty = k_full + 8 * NS, v_full = k_empty + 8 * NS, v_empty = v_full + 8 * NS;
    const uint32_t mask_full = v_empty + 8 * NS, mask_empty = mask_full + 8 * Cfg::NM;
    const int kp_k = (p.dk + 63) / 64, kp_v = (p.dv + 63) / 64;  // 64-column panels that hold something
    volatile uint32_t *tmem_slot = reinterpret_cast<volatile uint32_t *>(smem + Cfg::OFF_TMEM);
    volatile int *abort_flag = reinterpret_cast<volatile int *>(smem + Cfg::OFF_ABORT);

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;

    // work item: groups of slabs, each group's longest items first (see sdpa_tc_pair_kernel)
    const int span = p.group * p.n_tiles_q;
    const int grp = (int)blockIdx.x / span, rem = (int)blockIdx.x % span;
    const int slabs = min(p.group, p.BH - grp * p.group);
    const int q_tile = p.n_tiles_q - 1 - rem / slabs;
    const int q0 = q_tile * BM;
    const int bh = grp * p.group + rem % slabs;
    const int b = bh / p.Hq, h = bh % p.Hq;
    const int kvh = b * p.Hkv + h / (p.Hq / p.Hkv);

    int kv_limit = p.Sk;                                         // keys any row of this batch may see
    kv_limit = p.kv_lens.limit(b, kv_limit);
    const int kv_end = p.causal ? min(kv_limit, q0 + BM) : kv_limit;
    const int nt = (kv_end + BN - 1) / BN;

    auto load_kv = [&](uint32_t dst, const CUtensorMap *hi, const CUtensorMap *lo, uint32_t bar, int j, int panels) {
        ptx::mbar_arrive_expect_tx(bar, 2 * Cfg::KV_PANEL * (uint32_t)panels);
#pragma unroll
        for (int pn = 0; pn < Cfg::KP; ++pn) {
            if (pn >= panels) break;
            ptx::tma_load_3d(dst + pn * Cfg::KV_PANEL, hi, bar, pn * 64, j * BN, kvh);
            ptx::tma_load_3d(dst + Cfg::KV_BYTES + pn * Cfg::KV_PANEL, lo, bar, pn * 64, j * BN, kvh);
        }
    };

    // warp 0 sets the barriers up and sends Q and the first key tile on their way before the CTA meets
    if (warp == 0) {
        if (lane == 0) {
            *abort_flag = 0;
            ptx::mbar_init(q_full, 1);
            ptx::mbar_init(s_full, 1);
            ptx::mbar_init(s_free, 4);                           // one arrival per softmax warp
            ptx::mbar_init(p_full, 4);
            ptx::mbar_init(l_full, 4);
            for (int t = 0; t < 2; ++t) {
                ptx::mbar_init(pv_done + 8 * t, 1);
                ptx::mbar_init(pv_free + 8 * t, 4);              // one arrival per accumulator warp
            }
            for (int t = 0; t < 4; ++t) ptx::mbar_init(alpha_full + 8 * t, 4);
            for (int s = 0; s < NS; ++s) {
                ptx::mbar_init(k_full + 8 * s, 1);
                ptx::mbar_init(k_empty + 8 * s, 1);
                ptx::mbar_init(v_full + 8 * s, 1);
                ptx::mbar_init(v_empty + 8 * s, 1);
            }
            if constexpr (Cfg::MASK)
                for (int t = 0; t < Cfg::NM; ++t) {
                    ptx::mbar_init(mask_full + 8 * t, 64);       // every loading thread's copies
                    ptx::mbar_init(mask_empty + 8 * t, 4);
                }
            ptx::fence_mbar_init();
            if (sbase & 1023u) {
                *abort_flag = 1;
                ptx::report(p.status, TC_ERR_ALIGN);
            } else if (nt > 0) {
                ptx::prefetch_tmap(&tm_qh);
                ptx::prefetch_tmap(&tm_kh);
                ptx::mbar_arrive_expect_tx(q_full, 2 * BM * 128 * (uint32_t)kp_k);
#pragma unroll
                for (int pn = 0; pn < Cfg::KP; ++pn) {
                    if (pn >= kp_k) break;
                    ptx::tma_load_3d(qh_s + pn * (BM * 128), &tm_qh, q_full, pn * 64, q0, bh);
                    ptx::tma_load_3d(ql_s + pn * (BM * 128), &tm_ql, q_full, pn * 64, q0, bh);
                }
                load_kv(k_s, &tm_kh, &tm_kl, k_full, 0, kp_k);
                load_kv(v_s, &tm_vh, &tm_vl, v_full, 0, kp_v);
            }
            if (*reinterpret_cast<volatile int *>(p.status) != 0) *abort_flag = 1;   // an earlier CTA gave up
        }
        __syncwarp();
    }
    if (warp == 1) {
        ptx::tmem_alloc(ptx::smem_u32(const_cast<uint32_t *>(tmem_slot)), Cfg::TMEM_COLS);
        ptx::tmem_relinquish();
    }
    ptx::tc_fence_before_sync();
    __syncthreads();
    ptx::tc_fence_after_sync();
    const uint32_t tmem = *tmem_slot;
    const bool run = (*abort_flag == 0) && nt > 0;

    if (warp < 4) {
    ptx::setmaxnreg_dec<Cfg::REGS_LIGHT>();
    if (warp == 0) {
        // ------------------------------------------------------------ TMA producer
        if (run) {
            const bool leader = ptx::elect_one();
            bool ok = true;
            for (int j = 1; j < nt && ok; ++j) {                 // key tile 0 went out before the meeting
                const int s = j % NS;
                const uint32_t ph = (uint32_t)(j / NS) & 1u;
                ok = ptx::mbar_wait(k_empty + 8 * s, ph ^ 1u, abort_flag);
                if (!ok) break;
                if (leader) load_kv(k_s + s * 2 * Cfg::KV_BYTES, &tm_kh, &tm_kl, k_full + 8 * s, j, kp_k);
                __syncwarp();
                ok = ptx::mbar_wait(v_empty + 8 * s, ph ^ 1u, abort_flag);
                if (!ok) break;
                if (leader) load_kv(v_s + s * 2 * Cfg::KV_BYTES, &tm_vh, &tm_vl, v_full + 8 * s, j, kp_v);
                __syncwarp();
            }
            if (!ok && leader) { *abort_flag = 1; ptx::report(p.status, TC_ERR_PRODUCER); }
        }
    } else if (warp == 1) {
        // ------------------------------------------------------------ MMA issuer
        // Three products per GEMM, the small ones first; the tensor pipe runs them in issue order.
        if (run) {
            const bool leader = ptx::elect_one();
            constexpr uint32_t idesc_qk = ptx::idesc_f16(BM, BN, false);
            const uint32_t idesc_pv = ptx::idesc_f16(BM, (p.dv + 15) / 16 * 16, true);
            const int steps = (p.dk + 15) / 16;
            constexpr uint32_t desc_hi = ptx::smem_desc_sw128_hi(1024);
            const uint32_t qh_lo = ptx::smem_desc_sw128_lo(qh_s, 16), ql_lo = ptx::smem_desc_sw128_lo(ql_s, 16);
            const uint32_t k_lo = ptx::smem_desc_sw128_lo(k_s, 16);
            const uint32_t v_lo = ptx::smem_desc_sw128_lo(v_s, Cfg::KV_PANEL);
            const uint32_t t_s = tmem + Cfg::COL_S;
            const uint32_t t_ph = tmem + Cfg::COL_PH, t_pl = tmem + Cfg::COL_PL;
            bool ok = true;
            auto issue_qk = [&](int j) -> bool {
                const int s = j % NS;
                const uint32_t ph = (uint32_t)(j / NS) & 1u;
                if (!ptx::mbar_wait(k_full + 8 * s, ph, abort_flag)) return false;
                ptx::tc_fence_after_sync();
                const uint32_t kh = k_lo + (uint32_t)s * ((2 * Cfg::KV_BYTES) >> 4), kl = kh + (Cfg::KV_BYTES >> 4);
                if (leader) {
#pragma unroll
                    for (int c = 0; c < 3; ++c) {
                        const uint32_t qa0 = c == 1 ? ql_lo : qh_lo;         // Qhi Klo, Qlo Khi, Qhi Khi
                        const uint32_t kb0 = c == 0 ? kl : kh;
#pragma unroll
                        for (int kk = 0; kk < D / 16; ++kk) {
                            if (kk >= steps) break;
                            const uint32_t qa = ((kk >> 2) * (BM * 128) + (kk & 3) * 32) >> 4;
                            const uint32_t kb = ((kk >> 2) * Cfg::KV_PANEL + (kk & 3) * 32) >> 4;
                            ptx::mma_ss(t_s, ptx::make_desc(qa0 + qa, desc_hi), ptx::make_desc(kb0 + kb, desc_hi),
                                        idesc_qk, (c > 0 || kk > 0) ? 1u : 0u);
                        }
                    }
                    ptx::mma_commit(k_empty + 8 * s);
                    ptx::mma_commit(s_full);
                }
                __syncwarp();
                return true;
            };
            // PV_j = P_j V_j into the fresh accumulator j & 1, once the accumulator warps have taken PV_{j-2} out of it
            auto issue_pv = [&](int j) -> bool {
                const int s = j % NS;
                const uint32_t ph = (uint32_t)(j / NS) & 1u;
                const int a = j & 1;
                if (!ptx::mbar_wait(v_full + 8 * s, ph, abort_flag)) return false;
                if (j >= 2 && !ptx::mbar_wait(pv_free + 8 * a, (uint32_t)((j - 2) >> 1) & 1u, abort_flag)) return false;
                if (!ptx::mbar_wait(p_full, (uint32_t)j & 1u, abort_flag)) return false;
                ptx::tc_fence_after_sync();
                const uint32_t vh = v_lo + (uint32_t)s * ((2 * Cfg::KV_BYTES) >> 4), vl = vh + (Cfg::KV_BYTES >> 4);
                const uint32_t t_pv = tmem + (a ? Cfg::COL_PV1 : Cfg::COL_PV0);
                if (leader) {
#pragma unroll
                    for (int c = 0; c < 3; ++c) {
                        const uint32_t pa0 = c == 1 ? t_pl : t_ph;           // Phi Vlo, Plo Vhi, Phi Vhi
                        const uint32_t vb0 = c == 0 ? vl : vh;
#pragma unroll
                        for (int kk = 0; kk < BN / 16; ++kk) {
                            const uint64_t bdesc = ptx::make_desc(vb0 + kk * ((16 * 128) >> 4), desc_hi);
                            ptx::mma_ts(t_pv, pa0 + kk * 8, bdesc, idesc_pv, (c > 0 || kk > 0) ? 1u : 0u);
                        }
                    }
                    ptx::mma_commit(v_empty + 8 * s);
                    ptx::mma_commit(pv_done + 8 * a);
                }
                __syncwarp();
                return true;
            };
            ok = ptx::mbar_wait(q_full, 0, abort_flag);
            if (ok) ok = issue_qk(0);
            for (int j = 0; j < nt && ok; ++j) {
                if (j + 1 < nt) {
                    ok = ptx::mbar_wait(s_free, (uint32_t)j & 1u, abort_flag);
                    if (ok) { ptx::tc_fence_after_sync(); ok = issue_qk(j + 1); }
                }
                if (ok) ok = issue_pv(j);
            }
            if (!ok && leader) { *abort_flag = 1; ptx::report(p.status, TC_ERR_MMA); }
        }
    } else if constexpr (Cfg::MASK) {
        // ------------------------------------------------------------ mask loader (warps 2, 3)
        // 16-byte copies where the mask's rows are 16-byte aligned, 4-byte ones otherwise; a 256-byte tile row keeps its
        // 16-byte chunks at chunk ^ (row & 7), which is what lets 8 softmax threads read 8 rows without bank conflicts.
        if (run) {
            const int t = (warp - 2) * 32 + lane;                // 0..63
            const float *base = p.mask + ((size_t)bh * p.Sq + q0) * p.Sk;
            const bool wide = (p.Sk & 3) == 0 && (reinterpret_cast<uintptr_t>(p.mask) & 15u) == 0;
            const int rows = min(BM, p.Sq - q0);
            bool ok = true;
            for (int j = 0; j < nt && ok; ++j) {
                const int s = j % Cfg::NM;
                if (j >= Cfg::NM) ok = ptx::mbar_wait(mask_empty + 8 * s, ((uint32_t)(j / Cfg::NM) & 1u) ^ 1u, abort_flag);
                if (!ok) break;
                const uint32_t dst = sbase + Cfg::OFF_MASK + (uint32_t)s * Cfg::MASK_BYTES;
                const int kv0 = j * BN;
                if (wide) {
                    const int c = t & 15;                        // chunk of the row: 16 threads a row, 4 rows a step
                    const bool in = kv0 + c * 4 < p.Sk;
                    const int r0 = t >> 4;
                    // rows r0, r0 + 4, r0 + 8 ...: the swizzle alternates between two places, all else advances evenly
                    const uint32_t d0 = dst + (uint32_t)r0 * 256;
                    const uint32_t sw[2] = {(uint32_t)(c ^ r0) << 4, (uint32_t)(c ^ (r0 + 4)) << 4};
                    const float *src = base + (size_t)r0 * p.Sk + kv0 + c * 4;
                    const size_t step = (size_t)4 * p.Sk;
                    const int n = in ? (rows - r0 + 3) / 4 : 0;
                    if (n == BM / 4) {
#pragma unroll
                        for (int i = 0; i < BM / 4; ++i, src += step) ptx::cp_async16(d0 + (uint32_t)i * 1024 + sw[i & 1], src);
                    } else {
                        for (int i = 0; i < n; ++i, src += step) ptx::cp_async16(d0 + (uint32_t)i * 1024 + sw[i & 1], src);
                    }
                } else {
                    const bool in = kv0 + t < p.Sk;
                    for (int row = 0; row < rows; ++row)
                        if (in) ptx::cp_async4(dst + (uint32_t)row * 256 + ((uint32_t)((t >> 2) ^ (row & 7)) << 4) + (t & 3) * 4,
                                               base + (size_t)row * p.Sk + kv0 + t);
                }
                ptx::cp_async_arrive(mask_full + 8 * s);
            }
            if (!ok && lane == 0) { *abort_flag = 1; ptx::report(p.status, TC_ERR_PRODUCER); }
            ptx::cp_async_wait_all();
        }
    }
    } else if (warp < 8) {
        ptx::setmaxnreg_inc<Cfg::REGS_SOFTMAX>();
        // ------------------------------------------------------------ softmax
        const int quarter = warp & 3;                    // tensor-memory lanes this warp may touch
        const int r = quarter * 32 + lane;               // row inside the tile
        const int row = q0 + r;
        const uint32_t lane_base = (uint32_t)(quarter * 32) << 16;
        const uint32_t t_s = tmem + lane_base + Cfg::COL_S;
        const uint32_t t_ph = tmem + lane_base + Cfg::COL_PH, t_pl = tmem + lane_base + Cfg::COL_PL;
        constexpr float kLog2e = 1.4426950408889634f;
        const float row_scale = (Cfg::MASK ? p.scale : p.scale_log2) * (row < p.Sq ? p.qf[(size_t)bh * p.Sq + row] : 1.f);
        const int f0 = kvh * ((p.Sk + BN - 1) / BN);     // factor of the head's first tile
        float m_run = Cfg::MASK ? -FLT_MAX : -1.0e30f;           // finite stand-in for "no key seen yet"
        float l = 0.f;
        bool ok = run;
        if (run && warp == 4) {                          // how far V's keys lie apart, while the first tiles are on their way
            int most = 0, least = 255;
            for (int j = lane; j < nt; j += 32) {
                const int f = p.vr[f0 + j];
                most = max(most, f & 255);
                least = min(least, f >> 8);
            }
            most = __reduce_max_sync(0xffffffffu, most);
            least = __reduce_min_sync(0xffffffffu, least);
            if (lane == 0 && most - least > 13) atomicOr(p.range, 1);
        }
        auto arrive_warp = [&](uint32_t bar) {
            ptx::tc_fence_before_sync();
            __syncwarp();
            if (lane == 0) ptx::mbar_arrive(bar);
        };
        for (int j = 0; j < nt && ok; ++j) {
            const int kv0 = j * BN;
            // not 0, however small the factors: -inf * 0 would make a NaN of a key that is not seen
            const float tile_scale = fmaxf(row_scale * p.kf[f0 + j], FLT_MIN), scale = Cfg::MASK ? kLog2e : tile_scale;
            ok = ptx::mbar_wait(s_full, (uint32_t)j & 1u, abort_flag);
            if (!ok) break;
            ptx::tc_fence_after_sync();
            uint32_t sv[BN];
            ptx::tmem_ld_cols<BN>(t_s, sv);
            ptx::tmem_wait_ld();
            ptx::reg_fence_cols<BN>(sv);
            arrive_warp(s_free);                         // S belongs to the MMA warp again
            if constexpr (Cfg::MASK) {
                const int sm_ = j % Cfg::NM;
                ok = ptx::mbar_wait(mask_full + 8 * sm_, (uint32_t)(j / Cfg::NM) & 1u, abort_flag);
                if (!ok) break;
                const uint32_t mrow = sbase + Cfg::OFF_MASK + (uint32_t)sm_ * Cfg::MASK_BYTES + (uint32_t)r * 256;
#pragma unroll
                for (int i = 0; i < BN; i += 4) {
                    uint32_t a, b2, c, d;
                    ptx::ld_shared_v4(mrow + ((uint32_t)((i >> 2) ^ (r & 7)) << 4), a, b2, c, d);
                    sv[i] = __float_as_uint(fmaf(__uint_as_float(sv[i]), tile_scale, __uint_as_float(a)));
                    sv[i + 1] = __float_as_uint(fmaf(__uint_as_float(sv[i + 1]), tile_scale, __uint_as_float(b2)));
                    sv[i + 2] = __float_as_uint(fmaf(__uint_as_float(sv[i + 2]), tile_scale, __uint_as_float(c)));
                    sv[i + 3] = __float_as_uint(fmaf(__uint_as_float(sv[i + 3]), tile_scale, __uint_as_float(d)));
                }
                __syncwarp();
                if (lane == 0) ptx::mbar_arrive(mask_empty + 8 * sm_);
            }
            const bool need_mask = (kv0 + BN > kv_limit) || (p.causal && (kv0 + BN - 1 > q0));
            if (need_mask) {
                // visible keys of this row are a prefix of the tile: columns [0, lim)
                const int lim = min(kv_limit - kv0, p.causal ? row - kv0 + 1 : BN);
#pragma unroll
                for (int i = 0; i < BN; ++i) sv[i] = ptx::keep_if_below(sv[i], i, lim);
            }
            float mx0 = -INFINITY, mx1 = -INFINITY, mx2 = -INFINITY, mx3 = -INFINITY;
#pragma unroll
            for (int i = 0; i < BN; i += 8) {
                mx0 = ptx::max3(mx0, __uint_as_float(sv[i]), __uint_as_float(sv[i + 1]));
                mx1 = ptx::max3(mx1, __uint_as_float(sv[i + 2]), __uint_as_float(sv[i + 3]));
                mx2 = ptx::max3(mx2, __uint_as_float(sv[i + 4]), __uint_as_float(sv[i + 5]));
                mx3 = ptx::max3(mx3, __uint_as_float(sv[i + 6]), __uint_as_float(sv[i + 7]));
            }
            const float mx = fmaxf(fmaxf(mx0, mx1), fmaxf(mx2, mx3));
            const float m_next = fmaxf(m_run, Cfg::MASK ? mx : mx * scale);   // exact running max: every p <= 1
            const float alpha = ptx::ex2_approx(Cfg::MASK ? (m_run - m_next) * kLog2e : m_run - m_next);
            m_run = m_next;
            alpha_s[(j & 3) * BM + r] = alpha;                      // for the accumulator thread of this row
            __syncwarp();
            if (lane == 0) ptx::mbar_arrive(alpha_full + 8 * (j & 3));
            // p = 2^(s*scale - m): a masked score is -inf and gives exactly 0
            const float2 scale2 = make_float2(scale, scale), negm2 = make_float2(-m_next, -m_next);
            const float2 p_scale2 = make_float2(X3_P_SCALE, X3_P_SCALE);
            float2 sum_a = make_float2(0.f, 0.f), sum_b = make_float2(0.f, 0.f);
            uint32_t pkh[BN / 2], pkl[BN / 2];
#pragma unroll
            for (int i = 0; i < BN; i += 4) {
                const float2 sa = make_float2(__uint_as_float(sv[i]), __uint_as_float(sv[i + 1]));
                const float2 sb = make_float2(__uint_as_float(sv[i + 2]), __uint_as_float(sv[i + 3]));
                // masked: the difference first, then the scaling (both terms may be as large as floats get)
                const float2 xa = Cfg::MASK ? __fmul2_rn(__fadd2_rn(sa, negm2), scale2) : __ffma2_rn(sa, scale2, negm2);
                const float2 xb = Cfg::MASK ? __fmul2_rn(__fadd2_rn(sb, negm2), scale2) : __ffma2_rn(sb, scale2, negm2);
                const float2 ea = make_float2(ptx::ex2_approx(xa.x), ptx::ex2_approx(xa.y));
                const float2 eb = make_float2(ptx::ex2_approx(xb.x), ptx::ex2_approx(xb.y));
                sum_a = __fadd2_rn(sum_a, ea);
                sum_b = __fadd2_rn(sum_b, eb);
                const float2 pa = __fmul2_rn(ea, p_scale2), pb = __fmul2_rn(eb, p_scale2);
                const __half2 ha = __floats2half2_rn(pa.x, pa.y), hb = __floats2half2_rn(pb.x, pb.y);
                const float2 ba = __half22float2(ha), bb = __half22float2(hb);
                const __half2 la = __floats2half2_rn(pa.x - ba.x, pa.y - ba.y), lb = __floats2half2_rn(pb.x - bb.x, pb.y - bb.y);
                pkh[i / 2] = *reinterpret_cast<const uint32_t *>(&ha);
                pkh[i / 2 + 1] = *reinterpret_cast<const uint32_t *>(&hb);
                pkl[i / 2] = *reinterpret_cast<const uint32_t *>(&la);
                pkl[i / 2 + 1] = *reinterpret_cast<const uint32_t *>(&lb);
            }
            l = l * alpha + ((sum_a.x + sum_a.y) + (sum_b.x + sum_b.y));
            if (j > 0) {
                // PV of the previous tile must have read P before it is overwritten
                ok = ptx::mbar_wait(pv_done + 8 * ((j - 1) & 1), (uint32_t)((j - 1) >> 1) & 1u, abort_flag);
                if (!ok) break;
                ptx::tc_fence_after_sync();
            }
            ptx::tmem_st_cols<BN / 2>(t_ph, pkh);
            ptx::tmem_st_cols<BN / 2>(t_pl, pkl);
            ptx::tmem_wait_st();
            arrive_warp(p_full);
        }
        if (run && ok) {
            l_s[r] = l;
            __syncwarp();
            if (lane == 0) ptx::mbar_arrive(l_full);
        }
        if (run && !ok) { *abort_flag = 1; ptx::report(p.status, TC_ERR_SOFTMAX); }
        if (nt == 0 && *abort_flag == 0 && row < p.Sq) {
            // no visible key at all for this tile: the reference's 0/0
            float *orow = p.out + ((size_t)bh * p.Sq + row) * p.dv;
            for (int i = 0; i < p.dv; ++i) orow[i] = __int_as_float(0x7fc00000);
        }
    } else {
        ptx::setmaxnreg_inc<Cfg::REGS_ACC>();
        // ------------------------------------------------------------ accumulators + epilogue
        const int quarter = warp & 3;
        const int r = quarter * 32 + lane;
        const uint32_t lane_base = (uint32_t)(quarter * 32) << 16;
        float o[D];
#pragma unroll
        for (int i = 0; i < D; ++i) o[i] = 0.f;
        bool ok = run;
        const int f0 = kvh * ((p.Sk + BN - 1) / BN);
        for (int j = 0; j < nt && ok; ++j) {
            const int a = j & 1;
            const float beta = p.vf[f0 + j];             // asked for before the waits
            ok = ptx::mbar_wait(alpha_full + 8 * (j & 3), (uint32_t)(j >> 2) & 1u, abort_flag);
            if (!ok) break;
            const float alpha = alpha_s[(j & 3) * BM + r];
            const float2 alpha2 = make_float2(alpha, alpha), beta2 = make_float2(beta, beta);
            ok = ptx::mbar_wait(pv_done + 8 * a, (uint32_t)(j >> 1) & 1u, abort_flag);
            if (!ok) break;
            ptx::tc_fence_after_sync();
            const uint32_t t_pv = tmem + lane_base + (a ? Cfg::COL_PV1 : Cfg::COL_PV0);
#pragma unroll
            for (int c = 0; c < D / 32; ++c) {
                if (c * 32 >= p.dv) break;
                uint32_t t[32];
                ptx::tmem_ld32(t_pv + c * 32, t);
                ptx::tmem_wait_ld();
                ptx::reg_fence32(t);
#pragma unroll
                for (int i = 0; i < 32; i += 2) {
                    const float2 pv = __fmul2_rn(make_float2(__uint_as_float(t[i]), __uint_as_float(t[i + 1])), beta2);
                    const float2 y = __ffma2_rn(make_float2(o[c * 32 + i], o[c * 32 + i + 1]), alpha2, pv);
                    o[c * 32 + i] = y.x; o[c * 32 + i + 1] = y.y;
                }
            }
            ptx::tc_fence_before_sync();
            __syncwarp();
            if (lane == 0) ptx::mbar_arrive(pv_free + 8 * a);
        }
        if (run && ok) {
            ok = ptx::mbar_wait(l_full, 0, abort_flag);
            if (ok) {
                const float inv_l = 1.0f / l_s[r];   // l == 0 (no visible key) -> inf -> NaN rows, as the reference
                // staging: two 4 KB chunk buffers in this warp's quarter of the Q buffers (all QK^T have completed)
                constexpr uint32_t CHUNK_BYTES = 32 * 128;
                const uint32_t buf_a = qh_s + (uint32_t)quarter * (Cfg::Q_BYTES / 4);
                const uint32_t buf_b = ql_s + (uint32_t)quarter * (Cfg::Q_BYTES / 4);
                static_assert(CHUNK_BYTES <= Cfg::Q_BYTES / 4, "chunk buffer");
                const int row0 = q0 + quarter * 32;
                const uint32_t my_line = (uint32_t)lane * 128u;
                const uint32_t sw = (uint32_t)(lane & 7);
                auto put = [&](uint32_t buf, int piece, float x, float y, float z, float w) {
                    ptx::st_shared_v4(buf + my_line + (((uint32_t)piece ^ sw) << 4), __float_as_uint(x * inv_l),
                                      __float_as_uint(y * inv_l), __float_as_uint(z * inv_l), __float_as_uint(w * inv_l));
                };
                auto send = [&](uint32_t buf, int col) {
                    ptx::fence_proxy_async_smem();
                    __syncwarp();
                    if (lane == 0 && row0 < p.Sq && col < p.dv) {
                        ptx::tma_store_3d(&tm_o, buf, col, row0, bh);
                        ptx::tma_store_commit();
                    }
                };
#pragma unroll
                for (int c = 0; c < D / 64; ++c) {
                    if (c > 0) {                                        // both buffers were sent in the step before
                        if (lane == 0) ptx::tma_store_wait_read<0>();
                        __syncwarp();
                    }
#pragma unroll
                    for (int i = 0; i < 32; i += 4)
                        put(buf_a, i / 4, o[c * 64 + i], o[c * 64 + i + 1], o[c * 64 + i + 2], o[c * 64 + i + 3]);
                    send(buf_a, c * 64);
#pragma unroll
                    for (int i = 0; i < 32; i += 4)
                        put(buf_b, i / 4, o[c * 64 + 32 + i], o[c * 64 + 33 + i], o[c * 64 + 34 + i], o[c * 64 + 35 + i]);
                    send(buf_b, c * 64 + 32);
                }
                if (lane == 0) ptx::tma_store_wait_read<0>();   // shared memory must outlive the stores' reads
                __syncwarp();
            }
        }
        if (run && !ok) { *abort_flag = 1; ptx::report(p.status, TC_ERR_SOFTMAX); }
    }

    // ---------------------------------------------------------------- teardown
    ptx::tc_fence_before_sync();
    __syncthreads();
    if (*abort_flag) {
        // a wait ran out in this CTA (or in an earlier one of the launch): its rows are not valid and say so
        if (warp >= 4 && warp < 8) {
            const int row_a = q0 + (warp & 3) * 32 + lane;
            if (row_a < p.Sq) {
                float *orow = p.out + ((size_t)bh * p.Sq + row_a) * p.dv;
                for (int i = 0; i < p.dv; ++i) orow[i] = __int_as_float(0x7fc00000);
            }
        }
        for (int i = 0; i < 64; ++i) __nanosleep(2000);   // let copies in flight land
        __syncthreads();
    }
    if (warp == 1) {
        ptx::tc_fence_after_sync();
        ptx::tmem_dealloc(tmem, Cfg::TMEM_COLS);
    }
}

// The split pass: hi = rn_fp16(2^e x), lo = rn_fp16(2^e x - hi) of Q, K and V in one launch, rows padded with zeros to a
// multiple of 8, the factors 2^-e, and the words that decide between the tensor-core kernel above and the exact one.
// Bound: HBM.  One CTA takes 64 rows of Q (a factor each) or a 64-key tile of K or V, all of it in registers between the
// maximum and the scaling.  Four lanes share a row, each with every fourth group of eight elements: a row's maximum is two
// shuffles away, and a CTA is small enough for the whole launch to be one wave (with 8, 16 or 32 lanes a row, up to eight
// rows a thread, B2 H8 S1000 d80 took 11.5 us and B4 H16 S1024 d64 23; now 7.2 and 14.7; eight CTAs an SM at d = 64 spill: 15.9).
struct SplitSeg {
    const float *x;
    __half *hi, *lo;
    float *factor;            // Q: [rows], K and V: [tiles]
    int *fields;              // V: [tiles], see X3Params::vr
    long long S;              // rows of a slab, cut into `tiles` tiles (Q: all rows are one slab)
    int tiles, first;         // `first`: CTAs of the segments before this one
    int q4, p8;               // a row: quads of the source, groups of eight of the padded copy
};
struct SplitParams {
    SplitSeg seg[3];          // Q, K, V
    int *range;               // three words, zero
};

template <int N>              // groups of eight a lane, 4 N at least p8
__global__ void __launch_bounds__(256, N == 1 ? 8 : N == 2 ? 6 : 5) split_f32_hi_lo_kernel(const SplitParams sp)
{
    ptx::grid_trigger();
    constexpr int kInf = 0x7f800000;
    __shared__ int warp_max[8], warp_min[8];
    const int t = (int)blockIdx.x >= sp.seg[2].first ? 2 : ((int)blockIdx.x >= sp.seg[1].first ? 1 : 0);
    const SplitSeg &s = sp.seg[t];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, part = lane & 3, row = warp * 8 + (lane >> 2);
    const int tile = (int)blockIdx.x - s.first, slab = tile / s.tiles;
    const long long r0 = (long long)(tile - slab * s.tiles) * X3_TILE, at = (long long)slab * s.S + r0 + row;
    const bool in = r0 + row < s.S;
    const float4 *src = reinterpret_cast<const float4 *>(s.x) + at * s.q4;
    ptx::grid_wait();                                                            // where the tensors come from the launch before
    float4 x[2 * N];
#pragma unroll
    for (int i = 0; i < 2 * N; ++i) {
        const int c = ((i >> 1) * 4 + part) * 2 + (i & 1);
        x[i] = in && c < s.q4 ? src[c] : make_float4(0.f, 0.f, 0.f, 0.f);
    }
    // the largest magnitude of the row and of the tile, as bits: integers order as the floats do, NaN above everything
    int m = 0;
#pragma unroll
    for (int i = 0; i < 2 * N; ++i)
        m = max(m, max(max(__float_as_int(fabsf(x[i].x)), __float_as_int(fabsf(x[i].y))), max(__float_as_int(fabsf(x[i].z)), __float_as_int(fabsf(x[i].w)))));
    m = max(m, __shfl_xor_sync(0xffffffffu, m, 1));
    m = max(m, __shfl_xor_sync(0xffffffffu, m, 2));
    int most = __reduce_max_sync(0xffffffffu, m), least = __reduce_min_sync(0xffffffffu, m != 0 ? m : kInf);
    if (lane == 0) { warp_max[warp] = most; warp_min[warp] = least; }
    __syncthreads();
#pragma unroll
    for (int w = 0; w < 8; ++w) { most = max(most, warp_max[w]); least = min(least, warp_min[w]); }
    // exponent that brings the maximum to [2^13, 2^14); both 2^e and 2^-e are normal floats
    const int e = min(126, 140 - ((t == 0 ? m : most) >> 23));
    const float scale = __int_as_float((e + 127) << 23), factor = __int_as_float((127 - e) << 23);
    if (threadIdx.x == 0) {
        if (most >= kInf) atomicOr(sp.range, 1);
        if (t == 0) atomicMax(sp.range + 1, most);
        if (t == 1) atomicMax(sp.range + 2, most);
        if (t == 1) s.factor[tile] = factor;
        if (t == 2) { s.factor[tile] = factor / X3_P_SCALE; s.fields[tile] = most >> 23 | (least >> 23) << 8; }
    }
    if (!in) return;
    if (t == 0 && part == 0) s.factor[at] = factor;
    uint4 *hi = reinterpret_cast<uint4 *>(s.hi) + at * s.p8, *lo = reinterpret_cast<uint4 *>(s.lo) + at * s.p8;
    auto halves = [&](float a, float b, uint32_t &h, uint32_t &l) {
        a *= scale; b *= scale;
        const __half2 hh = __floats2half2_rn(a, b);
        const float2 back = __half22float2(hh);
        const __half2 ll = __floats2half2_rn(a - back.x, b - back.y);
        h = *reinterpret_cast<const uint32_t *>(&hh);
        l = *reinterpret_cast<const uint32_t *>(&ll);
    };
#pragma unroll
    for (int i = 0; i < N; ++i) {
        const int c = i * 4 + part;
        if (c >= s.p8) continue;
        uint4 h, l;
        halves(x[2 * i].x, x[2 * i].y, h.x, l.x);
        halves(x[2 * i].z, x[2 * i].w, h.y, l.y);
        halves(x[2 * i + 1].x, x[2 * i + 1].y, h.z, l.z);
        halves(x[2 * i + 1].z, x[2 * i + 1].w, h.w, l.w);
        hi[c] = h;
        lo[c] = l;
    }
}

}  // namespace txb

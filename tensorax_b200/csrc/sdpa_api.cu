// C ABI of the B200 SDPA forward path: validation, kernel selection, launch.
// Declarations and the reference interfaces they replace: include/tensorax_b200.h.
#include "../../include/tensorax_b200.h"

#include <cuda.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstdarg>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <mutex>
#include <string>
#include <type_traits>
#include <unordered_map>
#include <vector>

// NVTX ranges around the entry points, as the reference's launchers have them
// (csrc/cuda/profiling.cuh:7-18: scoped ranges when the NVTX header is present, nothing otherwise).
#if defined(__has_include)
#if __has_include(<nvtx3/nvtx3.hpp>)
#include <nvtx3/nvtx3.hpp>
#define TX_NVTX_RANGE(name) ::nvtx3::scoped_range tx_nvtx_range_{(name)}
#endif
#endif
#ifndef TX_NVTX_RANGE
#define TX_NVTX_RANGE(name) ((void)0)
#endif

#include "gemm_x3.cuh"
#include "linear_simt.cuh"
#include "linear_tc.cuh"
#include "sdpa_tc.cuh"
#include "sdpa_tc_pair.cuh"
#include "sdpa_tc_x3.cuh"
#include "sdpa_simt.cuh"
#include "sdpa_bwd.cuh"
#include "sdpa_decode.cuh"

namespace {

thread_local std::string g_err;
std::atomic<int64_t> g_launches{0};

int fail(int code, const char *fmt, ...)
{
    char buf[512];
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(buf, sizeof buf, fmt, ap);
    va_end(ap);
    g_err = buf;
    return code;
}

#define TX_CUDA(call)                                                                     \
    do {                                                                                  \
        cudaError_t e_ = (call);                                                          \
        if (e_ != cudaSuccess)                                                            \
            return fail(TX_ERR_CUDA, "%s failed: %s", #call, cudaGetErrorString(e_));     \
    } while (0)

int ensure_device()
{
    int n = 0;
    cudaError_t e = cudaGetDeviceCount(&n);
    if (e != cudaSuccess || n <= 0) {
        (void)cudaGetLastError();
        return fail(TX_ERR_NO_DEVICE, "no CUDA device available (%s)",
                    e == cudaSuccess ? "device count is 0" : cudaGetErrorString(e));
    }
    return TX_OK;
}

constexpr int kMaxDevices = 64;

int current_device(int *dev)
{
    TX_CUDA(cudaGetDevice(dev));
    if (*dev < 0 || *dev >= kMaxDevices) return fail(TX_ERR_INVALID, "device index %d out of range", *dev);
    return TX_OK;
}

int pool_ready();
void pool_took(void *ptr, size_t bytes);
void pool_gave(void *ptr);

// Workspace of one call from the device's stream-ordered pool.  pool_ready() first: with the pool's default release
// threshold of zero every synchronisation hands the freed workspace back to the driver, and the next call pays for
// mapping it again (2.5 ms for 400 MB).
int pool_alloc(char **p, size_t bytes, cudaStream_t st)
{
    if (int rc = pool_ready()) return rc;
    TX_CUDA(cudaMallocAsync(reinterpret_cast<void **>(p), bytes, st));
    pool_took(*p, bytes);
    return TX_OK;
}

void pool_free(char *p, cudaStream_t st)
{
    pool_gave(p);
    (void)cudaFreeAsync(p, st);
}

// One status word per device, written by kernels whose bounded waits run out, and its mirror in pinned host memory
// (the device address of the mirror sits behind the word, see ptx::report): asking for it after a synchronise is a
// load, where copying the word back was a second trip to the device on every call (7 us of a 47 us call).
struct Status {
    int *word = nullptr;
    volatile int *mirror = nullptr;
};
Status g_status[kMaxDevices];
std::atomic<bool> g_status_ready[kMaxDevices] = {};
std::mutex g_status_mu;

int status_word(int **out)
{
    int dev = 0;
    if (int rc = current_device(&dev)) return rc;
    if (!g_status_ready[dev].load(std::memory_order_acquire)) {
        std::lock_guard<std::mutex> lk(g_status_mu);
        if (!g_status_ready[dev].load(std::memory_order_relaxed)) {
            Status s;
            int *mirror = nullptr, *mirror_dev = nullptr;
            TX_CUDA(cudaMalloc(&s.word, 256));
            TX_CUDA(cudaHostAlloc(&mirror, 64, cudaHostAllocMapped));
            *mirror = 0;
            s.mirror = mirror;
            TX_CUDA(cudaHostGetDevicePointer(reinterpret_cast<void **>(&mirror_dev), mirror, 0));
            TX_CUDA(cudaMemset(s.word, 0, 256));
            TX_CUDA(cudaMemcpy(s.word + 2, &mirror_dev, sizeof mirror_dev, cudaMemcpyHostToDevice));
            g_status[dev] = s;
            g_status_ready[dev].store(true, std::memory_order_release);
        }
    }
    *out = g_status[dev].word;
    return TX_OK;
}

// ------------------------------------------------------------------ TMA descriptors
using EncodeTiledFn = CUresult (*)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *,
                                   const cuuint64_t *, const cuuint64_t *, const cuuint32_t *,
                                   const cuuint32_t *, CUtensorMapInterleave, CUtensorMapSwizzle,
                                   CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

int get_encode_fn(EncodeTiledFn *fn)
{
    static EncodeTiledFn cached = nullptr;
    if (!cached) {
        void *sym = nullptr;
        cudaDriverEntryPointQueryResult q;
        TX_CUDA(cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &sym, cudaEnableDefault, &q));
        if (!sym || q != cudaDriverEntryPointSuccess)
            return fail(TX_ERR_CUDA, "driver does not provide cuTensorMapEncodeTiled");
        cached = reinterpret_cast<EncodeTiledFn>(sym);
    }
    *fn = cached;
    return TX_OK;
}

// fp16 (or fp32: elem_bytes 4) tensor [slabs, rows, d] -> 3-D map (d, rows, slabs); box = 128 bytes of a row x
// box_rows, 128B swizzle.
// A map is a pure function of (base, slabs, rows, d, box_rows): the last few are kept per host thread, so a
// caller that runs the same buffers again (a decoding loop, a benchmark) does not pay the driver's encode
// call three times per launch.
struct MapKey {
    const void *base;
    int64_t slabs, rows, d;
    int box_rows, elem_bytes;
    bool operator==(const MapKey &o) const
    {
        return base == o.base && slabs == o.slabs && rows == o.rows && d == o.d && box_rows == o.box_rows &&
               elem_bytes == o.elem_bytes;
    }
};
constexpr int kMapCache = 16;
struct MapCache {
    MapKey key[kMapCache] = {};
    CUtensorMap map[kMapCache];
    bool used[kMapCache] = {};
    int next = 0;
};
thread_local MapCache g_map_cache;

int make_map(CUtensorMap *m, const void *base, int64_t slabs, int64_t rows, int64_t d, int box_rows, int elem_bytes = 2)
{
    const MapKey key{base, slabs, rows, d, box_rows, elem_bytes};
    MapCache &mc = g_map_cache;
    for (int i = 0; i < kMapCache; ++i)
        if (mc.used[i] && mc.key[i] == key) {
            *m = mc.map[i];
            return TX_OK;
        }
    EncodeTiledFn enc;
    if (int rc = get_encode_fn(&enc)) return rc;
    cuuint64_t dims[3] = {(cuuint64_t)d, (cuuint64_t)rows, (cuuint64_t)slabs};
    const cuuint64_t eb = (cuuint64_t)elem_bytes;
    cuuint64_t strides[2] = {(cuuint64_t)d * eb, (cuuint64_t)rows * (cuuint64_t)d * eb};
    cuuint32_t box[3] = {(cuuint32_t)(128 / elem_bytes), (cuuint32_t)box_rows, 1};
    cuuint32_t estr[3] = {1, 1, 1};
    CUresult r = enc(m, elem_bytes == 4 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 3,
                     const_cast<void *>(base), dims, strides,
                     box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                     CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return fail(TX_ERR_CUDA, "cuTensorMapEncodeTiled failed with code %d", (int)r);
    mc.key[mc.next] = key;
    mc.map[mc.next] = *m;
    mc.used[mc.next] = true;
    mc.next = (mc.next + 1) % kMapCache;
    return TX_OK;
}

// cudaFuncSetAttribute(MaxDynamicSharedMemorySize) once per kernel and device: one bit per device beside each kernel.
// LARGE_CLUSTERS: the kernel may be launched in clusters of more than eight CTAs.
template <auto Kernel, bool LARGE_CLUSTERS = false>
int allow_smem(int bytes)
{
    static std::atomic<uint64_t> done{0};
    static_assert(kMaxDevices <= 64, "one bit per device");
    int dev = 0;
    if (int rc = current_device(&dev)) return rc;
    if (done.load(std::memory_order_acquire) >> dev & 1u) return TX_OK;
    TX_CUDA(cudaFuncSetAttribute(Kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes));
    if (LARGE_CLUSTERS) TX_CUDA(cudaFuncSetAttribute(Kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
    done.fetch_or(uint64_t{1} << dev, std::memory_order_release);
    return TX_OK;
}

// Multiprocessors of the current device (asked once per device).
int sm_count(int *n)
{
    static std::atomic<int> seen[kMaxDevices] = {};
    int dev = 0;
    if (int rc = current_device(&dev)) return rc;
    int v = seen[dev].load(std::memory_order_relaxed);
    if (v == 0) {
        TX_CUDA(cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev));
        seen[dev].store(v, std::memory_order_relaxed);
    }
    *n = v;
    return TX_OK;
}

// fp32 tensor maps of the linear layer: 128-byte-swizzled boxes of 32 floats x `box_rows` rows.
int make_map_f32(CUtensorMap *m, const void *base, int rank, const cuuint64_t *dims, const cuuint64_t *strides,
                 int box_rows)
{
    EncodeTiledFn enc;
    if (int rc = get_encode_fn(&enc)) return rc;
    cuuint32_t box[4] = {32, (cuuint32_t)box_rows, 1, 1};
    cuuint32_t estr[4] = {1, 1, 1, 1};
    CUresult r = enc(m, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, (cuuint32_t)rank, const_cast<void *>(base), dims, strides,
                     box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                     CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return fail(TX_ERR_CUDA, "cuTensorMapEncodeTiled (fp32) failed with code %d", (int)r);
    return TX_OK;
}

// ------------------------------------------------------------------ validation
bool tc_eligible(const tx_sdpa_desc *d);

int validate(const tx_sdpa_desc *d)
{
    if (!d) return fail(TX_ERR_INVALID, "SDPA: null descriptor");
    if (!d->q || !d->k || !d->v || !d->out)
        return fail(TX_ERR_INVALID, "SDPA: Query, Key, Value and output pointers must not be null");
    if (d->batch <= 0 || d->q_heads <= 0 || d->kv_heads <= 0 || d->seq_q <= 0 || d->seq_k <= 0 ||
        d->d_k <= 0 || d->d_v <= 0)
        return fail(TX_ERR_INVALID, "SDPA: every dimension must be positive");
    if (d->q_heads % d->kv_heads != 0)
        return fail(TX_ERR_INVALID, "SDPA: Key dimensions don't match Query (q_heads %lld not a multiple of kv_heads %lld)",
                    (long long)d->q_heads, (long long)d->kv_heads);
    if (d->dtype != TX_DTYPE_F32 && d->dtype != TX_DTYPE_F16)
        return fail(TX_ERR_INVALID, "SDPA: dtype must be float32 or float16");
    if (d->batch * d->q_heads > 0x7fffffffLL / 2 || d->seq_q > 0x3fffffffLL || d->seq_k > 0x3fffffffLL)
        return fail(TX_ERR_UNSUPPORTED, "SDPA: dimension too large");
    if (d->lse && !tc_eligible(d))
        return fail(TX_ERR_UNSUPPORTED, "SDPA: the log-sum-exp output is written by the tensor-core kernel only "
                                        "(fp16, no dense mask, d_k == d_v in {64,128,256,512})");
    return TX_OK;
}

bool tc_eligible(const tx_sdpa_desc *d)
{
    if (d->flags & TX_SDPA_FORCE_SIMT) return false;
    if (d->dtype != TX_DTYPE_F16 || d->mask) return false;
    if (d->d_k != d->d_v) return false;
    if (d->d_k != 64 && d->d_k != 128 && d->d_k != 256 && d->d_k != 512) return false;
    auto al = [](const void *p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; };
    if (!al(d->q) || !al(d->k) || !al(d->v) || !al(d->out)) return false;
    if (d->batch * d->q_heads > 65535) return false;   // grid.y
    return true;
}

// ------------------------------------------------------------------ launches
// Key lengths as a kernel parameter.  Host arrays of more than KvLens::kInline lengths never get here (with_device_lens).
txb::KvLens lens_of(const int32_t *lens, int flags, int64_t batch)
{
    txb::KvLens k;
    if (lens && (flags & TX_SDPA_KV_LENS_HOST)) {
        k.n_inline = (int)batch;
        std::copy(lens, lens + batch, k.val);
    } else {
        k.ptr = lens;
    }
    return k;
}

void pool_free(char *p, cudaStream_t st);

// `call(desc)` with the key lengths where the kernels can read them: a host array too long for the parameter block is
// written to the device first, by launches that carry it (it has been read when the call returns).
template <class Desc, class Call>
int with_device_lens(const Desc *d, Call call)
{
    if (!d->kv_lens || !(d->flags & TX_SDPA_KV_LENS_HOST) || d->batch <= txb::KvLens::kInline) return call(d);
    cudaStream_t st = static_cast<cudaStream_t>(d->stream);
    char *ws = nullptr;
    if (int rc = pool_alloc(&ws, (size_t)d->batch * 4, st)) return rc;
    int32_t *lens = reinterpret_cast<int32_t *>(ws);
    auto body = [&]() -> int {
        for (int64_t at = 0; at < d->batch; at += txb::KvLensChunk::kMax) {
            txb::KvLensChunk c;
            c.n = (int32_t)std::min<int64_t>(txb::KvLensChunk::kMax, d->batch - at);
            std::copy(d->kv_lens + at, d->kv_lens + at + c.n, c.val);
            txb::put_kv_lens_kernel<<<1, 256, 0, st>>>(c, lens + at);
            g_launches++;
            TX_CUDA(cudaGetLastError());
        }
        Desc on_device = *d;
        on_device.kv_lens = lens;
        on_device.flags &= ~TX_SDPA_KV_LENS_HOST;
        return call(&on_device);
    };
    const int rc = body();
    pool_free(ws, st);
    return rc;
}

// A launch that may start under the end of the one before it in the stream (ptx::grid_wait inside the kernel orders what
// has to be ordered), in clusters of `cluster` CTAs.  A plain launch starts 1 to 2 us after its predecessor has ended.
template <class... Params, class... Args>
int launch_behind(void (*kernel)(Params...), dim3 grid, int threads, size_t smem, cudaStream_t st, int cluster, const Args &...args)
{
    cudaLaunchAttribute at[2];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    at[1].id = cudaLaunchAttributeClusterDimension;
    at[1].val.clusterDim.x = (unsigned)cluster; at[1].val.clusterDim.y = 1; at[1].val.clusterDim.z = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3((unsigned)threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cfg.attrs = at;
    cfg.numAttrs = cluster > 1 ? 2 : 1;
    TX_CUDA(cudaLaunchKernelEx(&cfg, kernel, args...));
    g_launches++;
    return TX_OK;
}

template <typename T, int DVC, bool PROF>
int launch_simt_t(const txb::SimtParams &p, cudaStream_t st)
{
    dim3 grid((unsigned)((p.dv + 32 * DVC - 1) / (32 * DVC)),
              (unsigned)((p.Sq + txb::SIMT_BR - 1) / txb::SIMT_BR), (unsigned)(p.B * p.Hq));
    if (p.only_if) {
        // a stand-in that nearly always has nothing to do: one wave of CTAs that walk the items if they must (a CTA
        // each took 6.7 us to find that out at 2048 items)
        static std::atomic<int> fit{0};
        int sms = 0, per_sm = fit.load(std::memory_order_relaxed);
        if (int rc = sm_count(&sms)) return rc;
        if (per_sm == 0) {
            TX_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, txb::sdpa_simt_kernel<T, DVC, PROF>, txb::SIMT_THREADS, 0));
            fit.store(per_sm = std::max(per_sm, 1), std::memory_order_relaxed);
        }
        const int64_t items = (int64_t)grid.x * grid.y * grid.z;
        grid = dim3((unsigned)std::min<int64_t>(items, (int64_t)sms * per_sm));
        return launch_behind(txb::sdpa_simt_kernel<T, DVC, PROF>, grid, txb::SIMT_THREADS, 0, st, 1, p);
    }
    txb::sdpa_simt_kernel<T, DVC, PROF><<<grid, txb::SIMT_THREADS, 0, st>>>(p);
    g_launches++;
    TX_CUDA(cudaGetLastError());
    return TX_OK;
}

template <typename T, bool PROF = false>
int launch_simt(const txb::SimtParams &p, cudaStream_t st)
{
    if (p.B * p.Hq > 65535) return fail(TX_ERR_UNSUPPORTED, "SDPA: batch*heads > 65535");
    if ((p.Sq + txb::SIMT_BR - 1) / txb::SIMT_BR > 65535) return fail(TX_ERR_UNSUPPORTED, "SDPA: seq_len_q too large");
    if (p.dv <= 32) return launch_simt_t<T, 1, PROF>(p, st);
    if (p.dv <= 64) return launch_simt_t<T, 2, PROF>(p, st);
    if (p.dv <= 128) return launch_simt_t<T, 4, PROF>(p, st);
    return launch_simt_t<T, 8, PROF>(p, st);   // wider heads: one CTA column per 256 value columns
}

// Elements (bit e = element e of each group of 16) whose exponential is evaluated by the FMA-pipe
// polynomial at d = 64: two whole pairs of 16 (the polynomial is evaluated two-wide); measured round-robin
// against 0, 1, 3 and 4 pairs of 8.
constexpr int kPolyPairsD64 = 0x0303;
// d = 128: one pair of 16 (0.896 -> 0.880 ms at B4 H8 S8192 against none, 0.884 with two pairs; the medians of
// back-to-back runs move by 4-5 %: fewer special-function instructions also means a cooler part)
constexpr int kPolyPairsD128 = 0x0003;

int causal_group(const tx_sdpa_desc *d, int64_t items_per_slab, int64_t *group);

template <class Cfg>
int launch_tc_t(const tx_sdpa_desc *d, cudaStream_t st, int *status, long long *prof = nullptr)
{
    CUtensorMap tq, tk, tv, to;
    const bool out_f16 = (d->flags & TX_SDPA_OUT_F16) != 0;
    if (int rc = make_map(&tq, d->q, d->batch * d->q_heads, d->seq_q, d->d_k, Cfg::BM)) return rc;
    if (int rc = make_map(&tk, d->k, d->batch * d->kv_heads, d->seq_k, d->d_k, Cfg::BN)) return rc;
    if (int rc = make_map(&tv, d->v, d->batch * d->kv_heads, d->seq_k, d->d_v, Cfg::BN)) return rc;
    // the result leaves in boxes of one softmax warp's 32 rows x 128 bytes
    if (int rc = make_map(&to, d->out, d->batch * d->q_heads, d->seq_q, d->d_v, 32, out_f16 ? 2 : 4)) return rc;
    txb::TcParams p;
    p.out = d->out;
    p.out_f16 = out_f16 ? 1 : 0;
    p.lse = d->lse;
    p.kv_lens = lens_of(d->kv_lens, d->flags, d->batch);
    p.status = status;
    p.Hq = (int)d->q_heads;
    p.Hkv = (int)d->kv_heads;
    p.Sq = (int)d->seq_q;
    p.Sk = (int)d->seq_k;
    p.dv_total = (int)d->d_v;
    p.causal = d->causal ? 1 : 0;
    p.scale_log2 = (1.0f / std::sqrt((float)d->d_k)) * 1.4426950408889634f;
    p.prof = prof;
    p.skip_k_tile = -1;
    const int64_t n_tiles = (d->seq_q + Cfg::BM - 1) / Cfg::BM, slabs = d->batch * d->q_heads, zparts = d->d_v / Cfg::DV;
    int64_t group = 1;
    if (int rc = causal_group(d, n_tiles * zparts, &group)) return rc;
    p.group = (int)group; p.n_pairs = (int)n_tiles; p.BH = (int)slabs;
    if (n_tiles * slabs * zparts > 0x7fffffffLL) return fail(TX_ERR_UNSUPPORTED, "SDPA: more than 2^31 work items");
    if (int rc = allow_smem<txb::sdpa_tc_kernel<Cfg>>((int)Cfg::SMEM_BYTES)) return rc;
    dim3 grid((unsigned)(n_tiles * slabs * zparts), 1, 1);
    txb::sdpa_tc_kernel<Cfg><<<grid, Cfg::THREADS, Cfg::SMEM_BYTES, st>>>(tq, tk, tv, to, p);
    g_launches++;
    TX_CUDA(cudaGetLastError());
    return TX_OK;
}

// Slabs per group of the launch order of a causal call (see launch_two_tiles); 1 = slab-major.  `bytes_per_slab`: what
// the CTAs of one slab stream through L2; `multiple`: slabs that share those bytes and should stay together.
std::atomic<long long> g_group_l2_bytes{48ll << 20};

int launch_group(bool causal, int64_t slabs, int64_t items_per_slab, double bytes_per_slab, int64_t multiple, int64_t *group,
                 int64_t max_waves = 0)
{
    *group = 1;
    int sms = 0;
    if (int rc = sm_count(&sms)) return rc;
    if (!causal || slabs <= 1) return TX_OK;
    if (max_waves > 0 && items_per_slab * slabs > max_waves * sms) return TX_OK;   // a long launch: its tail is small anyway
    const int64_t by_l2 = std::max<int64_t>(1, (int64_t)((double)g_group_l2_bytes.load() / bytes_per_slab));
    const int64_t two_waves = (2 * sms + items_per_slab - 1) / items_per_slab;
    const int64_t want = std::min<int64_t>(slabs, std::max(by_l2, two_waves));
    const int64_t n_groups = (slabs + want - 1) / want;
    const int64_t g = (slabs + n_groups - 1) / n_groups;          // equal groups, none left small at the end
    *group = std::min<int64_t>(slabs, (g + multiple - 1) / multiple * multiple);
    return TX_OK;
}

int causal_group(const tx_sdpa_desc *d, int64_t items_per_slab, int64_t *group)
{
    const int64_t ratio = d->q_heads / d->kv_heads;
    return launch_group(d->causal != 0, d->batch * d->q_heads, items_per_slab,
                        2.0 * (double)d->seq_k * (double)(d->d_k + d->d_v) / (double)ratio, ratio, group);
}

template <class Cfg>
int launch_pair_t(const tx_sdpa_desc *d, cudaStream_t st, int *status, long long *prof = nullptr, int skip_k_tile = -1)
{
    CUtensorMap tq, tk, tv, to;
    const bool out_f16 = (d->flags & TX_SDPA_OUT_F16) != 0;
    if (int rc = make_map(&tq, d->q, d->batch * d->q_heads, d->seq_q, d->d_k, Cfg::BM)) return rc;
    if (int rc = make_map(&tk, d->k, d->batch * d->kv_heads, d->seq_k, d->d_k, Cfg::BN)) return rc;
    if (int rc = make_map(&tv, d->v, d->batch * d->kv_heads, d->seq_k, d->d_v, Cfg::BN)) return rc;
    // the result leaves in boxes of one softmax warp's 32 rows x 128 bytes
    if (int rc = make_map(&to, d->out, d->batch * d->q_heads, d->seq_q, d->d_v, 32, out_f16 ? 2 : 4)) return rc;
    txb::TcParams p;
    p.out = d->out;
    p.out_f16 = out_f16 ? 1 : 0;
    p.lse = d->lse;
    p.kv_lens = lens_of(d->kv_lens, d->flags, d->batch);
    p.status = status;
    p.Hq = (int)d->q_heads;
    p.Hkv = (int)d->kv_heads;
    p.Sq = (int)d->seq_q;
    p.Sk = (int)d->seq_k;
    p.dv_total = (int)d->d_v;
    p.causal = d->causal ? 1 : 0;
    p.scale_log2 = (1.0f / std::sqrt((float)d->d_k)) * 1.4426950408889634f;
    p.prof = prof;
    p.skip_k_tile = skip_k_tile;
    // Work items in launch order.  Slab-major (group = 1: a slab's CTAs, which share its K/V, start side by side)
    // unless the mask is causal: then the slabs are taken in groups, and inside a group every slab's longest items
    // come before any shorter one, so that the SMs do not end on a late slab's long items.  A group is as large as
    // its K/V may be while staying in L2 (48 MB; K/V heads shared by several query heads count once), at least two
    // waves of CTAs, a whole number of K/V heads, and the groups are equal (a small last group is the same tail
    // again: 32 slabs as 10 + 10 + 10 + 2 were slower than slab-major, as 4 x 8 or as one group 12-24 % faster).
    // Measured on B200, causal, slab-major -> grouped: d = 128 B1 Hq32 Hkv8 S8192 0.514 -> 0.468 ms, B1 H16 S8192
    // 0.333 -> 0.253, d = 64 B4 H8 S8192 0.388 -> 0.342, B4 H16 S4096 d = 128 0.286 -> 0.268, d = 64 0.220 -> 0.199,
    // B8 H16 S2048 0.170 -> 0.162; long launches gain less but gain (B8 Hq32 Hkv8 S8192, 55 waves: 3.80 -> 3.73 ms).
    const int64_t n_pairs = (d->seq_q + 2 * Cfg::BM - 1) / (2 * Cfg::BM);
    const int64_t slabs = d->batch * d->q_heads;
    int64_t group = 1;
    if (int rc = causal_group(d, n_pairs, &group)) return rc;
    p.group = (int)group;
    p.n_pairs = (int)n_pairs;
    p.BH = (int)slabs;
    if (n_pairs * slabs > 0x7fffffffLL) return fail(TX_ERR_UNSUPPORTED, "SDPA: more than 2^31 work items");
    if (int rc = allow_smem<txb::sdpa_tc_pair_kernel<Cfg>>((int)Cfg::SMEM_BYTES)) return rc;
    dim3 grid((unsigned)(n_pairs * slabs), 1, 1);
    txb::sdpa_tc_pair_kernel<Cfg><<<grid, Cfg::THREADS, Cfg::SMEM_BYTES, st>>>(tq, tk, tv, to, p);
    g_launches++;
    TX_CUDA(cudaGetLastError());
    return TX_OK;
}

// Kernel and tile shape per head dim.
//   d = 64, 128   sdpa_tc_pair_kernel: one CTA per SM, two 128-row query tiles, 128 keys per tile
//                 (d = 64: four-deep K/V ring, P in its own tensor-memory columns, a quarter of the
//                 exponentials on the FMA pipe; d = 128: two-deep ring, P over S)
//   d = 256       sdpa_tc_kernel, 64 keys per tile, one CTA per SM, Q in tensor memory
//   d = 512       sdpa_tc_kernel, 64 keys per tile, two CTAs split the value columns
// `prof` (section profile) selects the instrumented instantiation of the same shape.
using PairD64 = txb::PairCfg<64, 128, 4, kPolyPairsD64, false>;
using PairD64Prof = txb::PairCfg<64, 128, 4, kPolyPairsD64, false, true>;
using PairD128 = txb::PairCfg<128, 128, 2, kPolyPairsD128, true>;
using PairD128Prof = txb::PairCfg<128, 128, 2, kPolyPairsD128, true, true>;

int launch_tc(const tx_sdpa_desc *d, cudaStream_t st, int *status, long long *prof = nullptr)
{
    const bool p_smem = (d->flags & TX_SDPA_P_IN_SMEM) != 0;
    switch (d->d_k) {
    case 64:
        if (p_smem) return launch_tc_t<txb::TcCfg<64, 64, 128, 2, false>>(d, st, status);
        return prof ? launch_pair_t<PairD64Prof>(d, st, status, prof) : launch_pair_t<PairD64>(d, st, status);
    case 128:
        if (p_smem) return launch_tc_t<txb::TcCfg<128, 128, 64, 2, false>>(d, st, status);
        return prof ? launch_pair_t<PairD128Prof>(d, st, status, prof) : launch_pair_t<PairD128>(d, st, status);
    case 256:
        if (p_smem) return launch_tc_t<txb::TcCfg<256, 256, 64, 2, false>>(d, st, status);
        // Narrow key tiles make the A (Q) read the busiest user of the shared-memory port: Q lives
        // in tensor memory instead, and K / V are fetched as two independent queues.
        if (prof) return launch_tc_t<txb::TcCfg<256, 256, 64, 2, true, true, 0, 2, true, 128>>(d, st, status, prof);
        return launch_tc_t<txb::TcCfg<256, 256, 64, 2, true, false, 0, 2, true, 128>>(d, st, status);
    case 512:
        // All 512 tensor-memory columns: S 64 | O 256 | P 32 | first 320 elements of Q 160.  Those five Q panels
        // are staged in the empty K/V ring, so shared memory holds only Q's last three panels (48 KB) beside
        // two 64-key K stages (128 KB) and one V stage (32 KB): 64-key tiles where 32 fitted before.
        if (prof) return launch_tc_t<txb::TcCfg<512, 256, 64, 2, true, true, 0, 1, true, 160, true>>(d, st, status, prof);
        return launch_tc_t<txb::TcCfg<512, 256, 64, 2, true, false, 0, 1, true, 160, true>>(d, st, status);
    }
    return fail(TX_ERR_UNSUPPORTED, "SDPA: no tensor-core tile shape for d = %lld", (long long)d->d_k);
}

// Few query rows per K/V head (a decoding step): the kernel that reads the cache once and cuts the keys over a cluster.
// fp16 up to 16 rows a head (CTAs of four rows each, side by side, read the same keys through L2; beyond that the
// tensor-core kernel's 128-row tile is the better use of a CTA) and from one whole tile of keys on; fp32 up to 32 rows,
// because the tensor-core form first writes and reads back hi / lo copies of the whole cache.
// Small fp32 calls go there too: one launch without a workspace against three and a memset.  Up to 2^23 products (B1 H2
// S128 d64 44 -> 31 us a call, B1 H8 S128 d64 38 -> 28, B4 H8 S64 d64 37 -> 33; at 2^24 products and 1024 row groups it
// was 37 against 43) or up to two query rows per SM in all (B1 H4 Sq64 Sk2048 d128 84 -> 42: four CTAs' work otherwise;
// 148 SMs where there is no device to ask).
bool decode_eligible(const tx_sdpa_desc *d)
{
    if (d->flags & (TX_SDPA_FORCE_SIMT | TX_SDPA_P_IN_SMEM)) return false;
    if (d->d_k != d->d_v || (d->d_k != 64 && d->d_k != 128 && d->d_k != 256)) return false;
    auto al = [](const void *p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; };
    if (!al(d->q) || !al(d->k) || !al(d->v)) return false;
    const int64_t rows = d->q_heads / d->kv_heads * d->seq_q;
    if (d->dtype == TX_DTYPE_F16) return rows <= 16 && d->seq_k >= 128;
    int sms = 0;
    if (sm_count(&sms) != TX_OK) sms = 148;
    const double all_rows = (double)(d->batch * d->kv_heads * rows);
    return rows <= 32 || all_rows <= 2.0 * sms || all_rows * (double)d->seq_k * (double)d->d_k <= 8388608.0;
}

template <class Cfg>
int launch_decode_t(const tx_sdpa_desc *d, cudaStream_t st, int *status)
{
    txb::DecodeParams p;
    p.q = d->q; p.k = d->k; p.v = d->v; p.mask = d->mask;
    p.kv_lens = lens_of(d->kv_lens, d->flags, d->batch);
    p.out = d->out; p.lse = d->lse; p.status = status;
    p.out_f16 = (d->flags & TX_SDPA_OUT_F16) ? 1 : 0;
    p.Hkv = (int)d->kv_heads; p.Sq = (int)d->seq_q; p.Sk = (int)d->seq_k;
    p.rows = (int)(d->q_heads / d->kv_heads * d->seq_q);
    p.row_parts = (p.rows + Cfg::R - 1) / Cfg::R;
    p.causal = d->causal ? 1 : 0;
    p.scale = 1.0f / std::sqrt((float)d->d_k);
    int sms = 0;
    if (int rc = sm_count(&sms)) return rc;
    // CTAs per head: as many as one wave holds, as long as each still has a stage of keys; sixteen (a cluster size that
    // costs 1.4 us more to start and merge) only where each then has four stages
    const int64_t items = d->batch * d->kv_heads * p.row_parts;
    if (items * Cfg::MAX_SPLITS > 0x7fffffffLL) return fail(TX_ERR_UNSUPPORTED, "SDPA: more than 2^31 work items");
    int splits = 1;
    const int most = d->seq_k >= 4 * Cfg::MAX_SPLITS * Cfg::KEYS ? Cfg::MAX_SPLITS : 8;
    while (splits < most && items * splits * 2 <= Cfg::CTAS_PER_SM * sms && splits * Cfg::KEYS < d->seq_k) splits *= 2;
    if (int rc = allow_smem<txb::sdpa_decode_kernel<Cfg>, true>((int)Cfg::SMEM)) return rc;
    cudaLaunchAttribute at;
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim.x = (unsigned)splits; at.val.clusterDim.y = 1; at.val.clusterDim.z = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(items * splits));
    cfg.blockDim = dim3(Cfg::THREADS);
    cfg.dynamicSmemBytes = Cfg::SMEM;
    cfg.stream = st;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    TX_CUDA(cudaLaunchKernelEx(&cfg, txb::sdpa_decode_kernel<Cfg>, p));
    g_launches++;
    return TX_OK;
}

template <typename T, int D>
int launch_decode_d(const tx_sdpa_desc *d, cudaStream_t st, int *status)
{
    const int64_t rows = d->q_heads / d->kv_heads * d->seq_q;
    if (rows == 1) return launch_decode_t<txb::DecodeCfg<T, D, 1>>(d, st, status);
    if (rows == 2) return launch_decode_t<txb::DecodeCfg<T, D, 2>>(d, st, status);
    return launch_decode_t<txb::DecodeCfg<T, D, 4>>(d, st, status);
}

template <typename T>
int launch_decode(const tx_sdpa_desc *d, cudaStream_t st, int *status)
{
    if (d->d_k == 64) return launch_decode_d<T, 64>(d, st, status);
    if (d->d_k == 128) return launch_decode_d<T, 128>(d, st, status);
    return launch_decode_d<T, 256>(d, st, status);
}

// fp16 without a dense mask, at the shapes tc_eligible names
int launch_f16(const tx_sdpa_desc *d, cudaStream_t st, int *status)
{
    return decode_eligible(d) ? launch_decode<__half>(d, st, status) : launch_tc(d, st, status);
}

// One kernel of the backward as its launch sees it: items, tiles of the longest and of the mean one, the time of a tile.
struct BwdWork {
    double items, longest, mean, tile;
};

// CTAs per work item of a backward kernel on `sms` multiprocessors of `per_sm` CTAs (two on one get through half as much
// again as one does).  Time in tiles, a CTA's start and end counting as three, five with the sum over the cluster: the longest
// CTA, or all of them spread over the places, in whole waves where the items are equal.  An item is cut (in two, four or
// eight, a cluster) where that shortens the launch by a fifth or more; a CTA keeps two tiles at least.  B2 Hq12 Hkv4 S921
// d64 causal: the dK/dV kernel 67 us uncut, 42 us in two, 28 us in four, 35 us in eight; the dQ kernel 20 us uncut, 22 in two.
int bwd_split(const BwdWork &w, int sms, int per_sm)
{
    const double places = per_sm == 2 ? 1.5 * sms : (double)sms;
    auto cost = [&](int z) {
        const double fixed = z > 1 ? 5.0 : 3.0, one = std::ceil(w.longest / z) + fixed, waves = w.items * z / places;
        return std::max(one, w.mean < w.longest ? waves * (w.mean / z + fixed) : std::ceil(waves) * one);
    };
    int best = 1;
    for (int z = 2; z <= 8 && w.longest >= 2.0 * z; z *= 2)
        if (cost(z) < 0.8 * cost(best)) best = z;
    return best;
}

// Both kernels as they run, the dK/dV kernel beside the dQ kernel's CTAs wherever those leave an SM free (one CTA each):
// all the work spread over the SMs, or the longest dK/dV CTA behind the dQ CTAs that go before it, or the longest dQ CTA.
double bwd_together(const BwdWork &q, int zq, const BwdWork &k, int zk, int sms)
{
    auto share = [](const BwdWork &w, int z, double tiles) { return (tiles / z + (z > 1 ? 5.0 : 2.0)) * w.tile; };
    auto chain = [&](const BwdWork &w, int z) { return share(w, z, z * std::ceil(w.longest / z)); };
    const double q1 = share(q, zq, q.mean), k1 = share(k, zk, k.mean);
    const double work = (q.items * zq * q1 + k.items * zk * k1) / sms, behind = std::max(0.0, q.items * zq / sms - 1.0) * q1;
    return std::max({work, behind + chain(k, zk), chain(q, zq)});
}

template <int D, class DqCfg, class DkvCfg>
int launch_bwd(const tx_sdpa_bwd_desc *d, cudaStream_t st, int *status, const __half *dout_h, const float *delta, int *prepared)
{
    txb::BwdParams p;
    p.lse = d->lse; p.delta = delta; p.kv_lens = lens_of(d->kv_lens, d->flags, d->batch);
    p.dq = d->dq; p.dk = d->dk; p.dv = d->dv;
    p.status = status; p.prepared = prepared;
    p.Hq = (int)d->q_heads; p.Hkv = (int)d->kv_heads; p.Sq = (int)d->seq_q; p.Sk = (int)d->seq_k;
    p.causal = d->causal ? 1 : 0;
    p.scale = 1.0f / std::sqrt((float)D);
    p.scale_log2 = p.scale * 1.4426950408889634f;
    p.group_q = p.group_k = 1;
    p.items_q = p.items_k = p.slabs_q = p.slabs_k = 1;
    p.split_q = p.split_k = 1;
    int sms = 0;
    if (int rc = sm_count(&sms)) return rc;
    {
        auto up = [](int64_t n, int64_t by) { return (double)((n + by - 1) / by); };
        const double ratio = (double)(d->q_heads / d->kv_heads), tq = up(d->seq_k, DqCfg::BN), tk = up(d->seq_q, DkvCfg::BQ) * ratio;
        // a dK/dV tile against a dQ tile, one CTA per SM: 1.2 and 1.7 us at d = 128, 1.8 and 2.2 at d = 256
        const BwdWork q = {up(d->seq_q, DqCfg::BM) * (double)(d->batch * d->q_heads), tq, d->causal ? 0.5 * (tq + 1) : tq, 1.0};
        const BwdWork k = {up(d->seq_k, DkvCfg::BMK) * (double)(d->batch * d->kv_heads * DkvCfg::ZS), tk, d->causal ? 0.5 * (tk + ratio) : tk,
                           D == 128 ? 0.7 : 0.82};
        p.split_q = bwd_split(q, sms, DqCfg::CTAS_PER_SM);
        p.split_k = bwd_split(k, sms, DkvCfg::CTAS_PER_SM);
        // Each kernel alone gains by that; together, uncut, they may fill the chip as it is.  B1 H8 S1000 d256 causal: kernels
        // of 41 + 59 us uncut and 29 + 51 in two, the call 72 and 78; B1 H4 S2048 d128 32 + 42 and 22 + 30, the call 51.5 and
        // 55.6.  (58 shapes measured with every pair of cuts: none slower than uncut by this, four by up to 9 % without it.)
        if (DqCfg::CTAS_PER_SM == 1 && p.split_q * p.split_k > 1 &&
            bwd_together(q, p.split_q, k, p.split_k, sms) >= 0.9 * bwd_together(q, 1, k, 1, sms))
            p.split_q = p.split_k = 1;
    }
    {
        CUtensorMap tq, tdo, tk, tv;
        if (int rc = make_map(&tq, d->q, d->batch * d->q_heads, d->seq_q, D, DqCfg::BM)) return rc;
        if (int rc = make_map(&tdo, dout_h, d->batch * d->q_heads, d->seq_q, D, DqCfg::BM)) return rc;
        if (int rc = make_map(&tk, d->k, d->batch * d->kv_heads, d->seq_k, D, DqCfg::BN)) return rc;
        if (int rc = make_map(&tv, d->v, d->batch * d->kv_heads, d->seq_k, D, DqCfg::BN)) return rc;
        if (int rc = allow_smem<txb::sdpa_bwd_dq_kernel<DqCfg>>((int)DqCfg::SMEM_BYTES)) return rc;
        // 1-D grid, grouped longest-first order for causal calls (a slab's CTAs stream its K and V)
        const int64_t items = (d->seq_q + DqCfg::BM - 1) / DqCfg::BM, slabs = d->batch * d->q_heads;
        const int64_t ratio = d->q_heads / d->kv_heads;
        int64_t group = 1;
        // (beyond 32 waves the slab-major order was the better one here: B8 Hq32 Hkv8 S4096 d128 4.24 against 4.35 ms)
        if (int rc = launch_group(d->causal != 0, slabs, items, 4.0 * (double)d->seq_k * (double)D / (double)ratio, ratio, &group, 32))
            return rc;
        p.group_q = (int)group; p.items_q = (int)items; p.slabs_q = (int)slabs;
        if (items * slabs * p.split_q > 0x7fffffffLL) return fail(TX_ERR_UNSUPPORTED, "SDPA backward: more than 2^31 work items");
        if (int rc = launch_behind(txb::sdpa_bwd_dq_kernel<DqCfg>, dim3((unsigned)(items * slabs * p.split_q)), DqCfg::THREADS,
                                   DqCfg::SMEM_BYTES, st, p.split_q, tq, tdo, tk, tv, p))
            return rc;
    }
    {
        CUtensorMap tq, tdo, tk, tv;
        if (int rc = make_map(&tq, d->q, d->batch * d->q_heads, d->seq_q, D, DkvCfg::BQ)) return rc;
        if (int rc = make_map(&tdo, dout_h, d->batch * d->q_heads, d->seq_q, D, DkvCfg::BQ)) return rc;
        if (int rc = make_map(&tk, d->k, d->batch * d->kv_heads, d->seq_k, D, DkvCfg::BMK)) return rc;
        if (int rc = make_map(&tv, d->v, d->batch * d->kv_heads, d->seq_k, D, DkvCfg::BMK)) return rc;
        if (int rc = allow_smem<txb::sdpa_bwd_dkv_kernel<DkvCfg>>((int)DkvCfg::SMEM_BYTES)) return rc;
        // 1-D grid: (slab of (batch, K/V head)) x key tile x column part; a slab's CTAs stream the Q and dO of its
        // query heads
        const int64_t items = (d->seq_k + DkvCfg::BMK - 1) / DkvCfg::BMK, slabs = d->batch * d->kv_heads;
        const int64_t ratio = d->q_heads / d->kv_heads;
        int64_t group = 1;
        if (int rc = launch_group(d->causal != 0, slabs, items * DkvCfg::ZS, 4.0 * (double)ratio * (double)d->seq_q * (double)D, 1, &group, 32))
            return rc;
        p.group_k = (int)group; p.items_k = (int)items; p.slabs_k = (int)slabs;
        const int64_t ctas = items * slabs * DkvCfg::ZS * p.split_k;
        if (ctas > 0x7fffffffLL) return fail(TX_ERR_UNSUPPORTED, "SDPA backward: more than 2^31 work items");
        if (int rc = launch_behind(txb::sdpa_bwd_dkv_kernel<DkvCfg>, dim3((unsigned)ctas), DkvCfg::THREADS, DkvCfg::SMEM_BYTES, st,
                                   p.split_k, tq, tdo, tk, tv, p))
            return rc;
    }
    return TX_OK;
}

__global__ void cast_f32_to_f16_kernel(const float *__restrict__ in, __half *__restrict__ out, int64_t n);
__global__ void copy_out_kernel(const uint4 *__restrict__ src, uint4 *__restrict__ dst, size_t n16);
size_t align_up(size_t x, size_t a);

// fp32 inputs through the tensor-core kernel: fp16 copies of Q, K, V in stream-ordered pool memory.
int forward_f32_via_f16(const tx_sdpa_desc *d, cudaStream_t st)
{
    const int64_t nq = d->batch * d->q_heads * d->seq_q * d->d_k, nk = d->batch * d->kv_heads * d->seq_k * d->d_k,
                  nv = d->batch * d->kv_heads * d->seq_k * d->d_v;
    const size_t oq = 0, ok = align_up((size_t)nq * 2, 256), ov = ok + align_up((size_t)nk * 2, 256);
    char *ws = nullptr;
    if (int rc = pool_alloc(&ws, ov + (size_t)nv * 2, st)) return rc;
    const void *src[3] = {d->q, d->k, d->v};
    const int64_t n[3] = {nq, nk, nv};
    const size_t off[3] = {oq, ok, ov};
    int rc = TX_OK;
    for (int i = 0; i < 3 && rc == TX_OK; ++i) {
        const int64_t blocks = (n[i] + 1023) / 1024;
        if (blocks > 0x7fffffffLL) { rc = fail(TX_ERR_UNSUPPORTED, "SDPA: tensor too large"); break; }
        cast_f32_to_f16_kernel<<<(unsigned)blocks, 256, 0, st>>>(static_cast<const float *>(src[i]),
                                                               reinterpret_cast<__half *>(ws + off[i]), n[i]);
        g_launches++;
        if (cudaGetLastError() != cudaSuccess) rc = fail(TX_ERR_CUDA, "SDPA: cast launch failed");
    }
    if (rc == TX_OK) {
        tx_sdpa_desc h = *d;
        h.q = ws + oq; h.k = ws + ok; h.v = ws + ov;
        h.dtype = TX_DTYPE_F16;
        int *status = nullptr;
        rc = status_word(&status);
        if (rc == TX_OK) rc = launch_f16(&h, st, status);
    }
    pool_free(ws, st);
    return rc;
}

// fp32 in, fp32 out on the fp16 tensor cores (three products per GEMM, sdpa_tc_x3.cuh) for the calls that fit it.
bool x3_eligible(const tx_sdpa_desc *d)
{
    if (d->dtype != TX_DTYPE_F32 || d->lse) return false;
    if (d->flags & (TX_SDPA_FORCE_SIMT | TX_SDPA_OUT_F16 | TX_SDPA_P_IN_SMEM)) return false;
    // rows of whole 16-byte pieces (the split pass reads them, bulk tensor stores write the result)
    if (d->d_k > 128 || d->d_v > 128 || d->d_k % 4 || d->d_v % 4) return false;
    auto al = [](const void *p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; };
    if (!al(d->q) || !al(d->k) || !al(d->v) || !al(d->out)) return false;
    // the exact kernel stands behind it and must be launchable for the same call
    if (d->batch * d->q_heads > 65535 || (d->seq_q + txb::SIMT_BR - 1) / txb::SIMT_BR > 65535) return false;
    return true;
}

void fill_simt_params(txb::SimtParams *p, const tx_sdpa_desc *d)
{
    p->q = d->q; p->k = d->k; p->v = d->v;
    p->mask = d->mask;
    p->kv_lens = lens_of(d->kv_lens, d->flags, d->batch);
    p->out = d->out;
    p->out_f16 = (d->flags & TX_SDPA_OUT_F16) ? 1 : 0;
    p->B = d->batch; p->Hq = d->q_heads; p->Hkv = d->kv_heads;
    p->Sq = d->seq_q; p->Sk = d->seq_k; p->dk = d->d_k; p->dv = d->d_v;
    p->causal = d->causal ? 1 : 0;
    p->scale = 1.0f / std::sqrt((float)d->d_k);
    p->prof = nullptr;
}

// `zeroed`: three words of device memory that are zero behind a launch of this library that lets its successor start under
// its end (the layer); without them the call brings its own.
template <class Cfg>
int launch_x3_t(const tx_sdpa_desc *d, cudaStream_t st, int *status, int *zeroed)
{
    const int64_t rows_q = d->batch * d->q_heads * d->seq_q, rows_k = d->batch * d->kv_heads * d->seq_k;
    const int64_t dk8 = (d->d_k + 7) / 8 * 8, dv8 = (d->d_v + 7) / 8 * 8;       // row length of the fp16 copies
    const int64_t slabs_k = d->batch * d->kv_heads, tiles_k = (d->seq_k + txb::X3_TILE - 1) / txb::X3_TILE;
    const int64_t tiles_q = (rows_q + txb::X3_TILE - 1) / txb::X3_TILE;
    if (tiles_q + 2 * slabs_k * tiles_k > 0x7fffffffLL) return fail(TX_ERR_UNSUPPORTED, "SDPA: more than 2^31 work items");
    // workspace: hi and lo fp16 copies of Q, K and V, their factors and the range words, stream-ordered pool memory
    size_t total = 0;
    auto take = [&](int64_t bytes) { const size_t at = total; total += align_up((size_t)bytes, 256); return at; };
    const size_t o_qh = take(rows_q * dk8 * 2), o_ql = take(rows_q * dk8 * 2), o_kh = take(rows_k * dk8 * 2), o_kl = take(rows_k * dk8 * 2),
                 o_vh = take(rows_k * dv8 * 2), o_vl = take(rows_k * dv8 * 2);
    const size_t o_qf = take(rows_q * 4), o_kf = take(slabs_k * tiles_k * 4), o_vf = take(slabs_k * tiles_k * 4), o_vr = take(slabs_k * tiles_k * 4), o_range = take(3 * sizeof(int));
    char *ws = nullptr;
    if (int rc = pool_alloc(&ws, total, st)) return rc;
    auto float_at = [&](size_t at) { return reinterpret_cast<float *>(ws + at); };
    int rc = TX_OK;
    auto body = [&]() -> int {
        int *range = zeroed ? zeroed : reinterpret_cast<int *>(ws + o_range);
        if (!zeroed) TX_CUDA(cudaMemsetAsync(range, 0, 3 * sizeof(int), st));
        txb::SplitParams sp;
        auto seg = [&](int i, const void *x, size_t hi, size_t lo, size_t factor, int64_t S, int64_t tiles, int64_t first, int64_t n, int64_t n8) {
            sp.seg[i] = {static_cast<const float *>(x), reinterpret_cast<__half *>(ws + hi), reinterpret_cast<__half *>(ws + lo),
                         float_at(factor), i == 2 ? reinterpret_cast<int *>(ws + o_vr) : nullptr, (long long)S, (int)tiles, (int)first, (int)(n / 4), (int)(n8 / 8)};
        };
        seg(0, d->q, o_qh, o_ql, o_qf, rows_q, tiles_q, 0, d->d_k, dk8);
        seg(1, d->k, o_kh, o_kl, o_kf, d->seq_k, tiles_k, tiles_q, d->d_k, dk8);
        seg(2, d->v, o_vh, o_vl, o_vf, d->seq_k, tiles_k, tiles_q + slabs_k * tiles_k, d->d_v, dv8);
        sp.range = range;
        const dim3 ctas((unsigned)(tiles_q + 2 * slabs_k * tiles_k));
        const int64_t groups = std::max(dk8, dv8) / 8;
        auto kernel = groups <= 4 ? txb::split_f32_hi_lo_kernel<1> : (groups <= 8 ? txb::split_f32_hi_lo_kernel<2> :
                      (groups <= 12 ? txb::split_f32_hi_lo_kernel<3> : txb::split_f32_hi_lo_kernel<4>));
        if (zeroed) {
            if (int r = launch_behind(kernel, ctas, 256, 0, st, 1, sp)) return r;
        } else {
            kernel<<<ctas, 256, 0, st>>>(sp);                            // behind whatever the caller enqueued: a plain launch
            g_launches++;
            TX_CUDA(cudaGetLastError());
        }

        CUtensorMap qh, ql, kh, kl, vh, vl, to;
        const int64_t sq = d->batch * d->q_heads, sk = d->batch * d->kv_heads;
        if (int r = make_map(&qh, ws + o_qh, sq, d->seq_q, dk8, Cfg::BM)) return r;
        if (int r = make_map(&ql, ws + o_ql, sq, d->seq_q, dk8, Cfg::BM)) return r;
        if (int r = make_map(&kh, ws + o_kh, sk, d->seq_k, dk8, Cfg::BN)) return r;
        if (int r = make_map(&kl, ws + o_kl, sk, d->seq_k, dk8, Cfg::BN)) return r;
        if (int r = make_map(&vh, ws + o_vh, sk, d->seq_k, dv8, Cfg::BN)) return r;
        if (int r = make_map(&vl, ws + o_vl, sk, d->seq_k, dv8, Cfg::BN)) return r;
        if (int r = make_map(&to, d->out, sq, d->seq_q, d->d_v, 32, 4)) return r;
        txb::X3Params p;
        p.out = static_cast<float *>(d->out);
        p.mask = d->mask;
        p.kv_lens = lens_of(d->kv_lens, d->flags, d->batch);
        p.range = range;
        p.qf = float_at(o_qf); p.kf = float_at(o_kf); p.vf = float_at(o_vf); p.vr = reinterpret_cast<const int *>(ws + o_vr);
        p.status = status;
        p.Hq = (int)d->q_heads; p.Hkv = (int)d->kv_heads; p.Sq = (int)d->seq_q; p.Sk = (int)d->seq_k;
        p.dk = (int)d->d_k; p.dv = (int)d->d_v;
        p.causal = d->causal ? 1 : 0;
        p.scale = 1.0f / std::sqrt((float)d->d_k);
        p.scale_log2 = p.scale * 1.4426950408889634f;
        const int64_t n_tiles = (d->seq_q + Cfg::BM - 1) / Cfg::BM;
        int64_t group = 1;
        if (int r = causal_group(d, n_tiles, &group)) return r;
        p.group = (int)group; p.n_tiles_q = (int)n_tiles; p.BH = (int)sq;
        if (n_tiles * sq > 0x7fffffffLL) return fail(TX_ERR_UNSUPPORTED, "SDPA: more than 2^31 work items");
        if (int r = allow_smem<txb::sdpa_tc_x3_kernel<Cfg>>((int)Cfg::SMEM_BYTES)) return r;
        if (int r = launch_behind(txb::sdpa_tc_x3_kernel<Cfg>, dim3((unsigned)(n_tiles * sq)), Cfg::THREADS, Cfg::SMEM_BYTES, st, 1,
                                  qh, ql, kh, kl, vh, vl, to, p))
            return r;
        // the exact kernel behind it: works only where the fp16 pairs would not do
        txb::SimtParams sp2;
        fill_simt_params(&sp2, d);
        sp2.only_if = range;
        return launch_simt<float>(sp2, st);
    };
    rc = body();
    pool_free(ws, st);
    return rc;
}

int launch_x3(const tx_sdpa_desc *d, cudaStream_t st, int *status, int *zeroed = nullptr)
{
    auto on = [&](auto cfg) { return launch_x3_t<decltype(cfg)>(d, st, status, zeroed); };
    const bool narrow = d->d_k <= 64 && d->d_v <= 64;
    if (d->mask) return narrow ? on(txb::X3Cfg<64, 2, true>{}) : on(txb::X3Cfg<128, 2, true>{});
    return narrow ? on(txb::X3Cfg<64, 4>{}) : on(txb::X3Cfg<128, 2>{});
}

// Which kernel takes a (valid) call.
enum class Route { Decode, TensorCores, Pairs, CudaCores };
Route route_of(const tx_sdpa_desc *d)
{
    if (decode_eligible(d)) return Route::Decode;
    if (tc_eligible(d)) return Route::TensorCores;
    return x3_eligible(d) ? Route::Pairs : Route::CudaCores;
}

// fp32 tensors to be rounded to fp16 first: the call as the fp16 path gets it, if it takes it
bool via_f16(const tx_sdpa_desc *d, tx_sdpa_desc *h)
{
    if (d->dtype != TX_DTYPE_F32 || !(d->flags & TX_SDPA_F32_VIA_F16)) return false;
    *h = *d;
    h->dtype = TX_DTYPE_F16;
    return tc_eligible(h);
}

int forward_launch(const tx_sdpa_desc *d)
{
    cudaStream_t st = static_cast<cudaStream_t>(d->stream);
    tx_sdpa_desc h;
    if (via_f16(d, &h)) return forward_f32_via_f16(d, st);
    const Route route = route_of(d);
    if (route == Route::CudaCores) {
        txb::SimtParams p;
        fill_simt_params(&p, d);
        return d->dtype == TX_DTYPE_F16 ? launch_simt<__half>(p, st) : launch_simt<float>(p, st);
    }
    int *status = nullptr;
    if (int rc = status_word(&status)) return rc;
    if (route == Route::Decode) return d->dtype == TX_DTYPE_F16 ? launch_decode<__half>(d, st, status) : launch_decode<float>(d, st, status);
    return route == Route::TensorCores ? launch_tc(d, st, status) : launch_x3(d, st, status);
}

int forward(const tx_sdpa_desc *d)
{
    if (int rc = validate(d)) return rc;
    if (int rc = ensure_device()) return rc;
    return with_device_lens(d, forward_launch);
}

int finish(cudaStream_t st)
{
    TX_CUDA(cudaStreamSynchronize(st));
    int dev = 0;
    if (int rc = current_device(&dev)) return rc;
    if (!g_status_ready[dev].load(std::memory_order_acquire) || *g_status[dev].mirror == 0) return TX_OK;
    std::lock_guard<std::mutex> lk(g_status_mu);
    const int code = txb::take_report(
        [&](int v) { return __atomic_exchange_n(const_cast<int *>(g_status[dev].mirror), v, __ATOMIC_SEQ_CST); },
        // the word only: the mirror's address stays behind it
        [&] { return cudaMemset(g_status[dev].word, 0, sizeof(int)) == cudaSuccess && cudaStreamSynchronize(nullptr) == cudaSuccess; });
    if (code != 0)
        return fail(TX_ERR_KERNEL, "SDPA kernel gave up on a bounded wait (stage code %d); output is not valid", code);
    return TX_OK;
}

// ------------------------------------------------------------------ multi-head attention layer
template <class Cfg>
int launch_gemm_x3_t(const txb::GemmX3Params &p0, const __half *const *xh, const __half *const *xl, const __half *wh, const __half *wl,
                     int64_t w_rows, cudaStream_t st)
{
    txb::GemmX3Params p = p0;
    txb::GemmX3Maps maps;
    p.n_tiles = 0;
    for (int i = 0; i < p.n_probs; ++i) {
        txb::GemmX3Problem &pr = p.prob[i];
        pr.tiles_n = (p.N + Cfg::BN - 1) / Cfg::BN;
        pr.first_tile = p.n_tiles;
        p.n_tiles += (pr.M + Cfg::BM - 1) / Cfg::BM * pr.tiles_n;
        if (int rc = make_map(&maps.xh[i], xh[i], 1, pr.M, p.K, Cfg::BM)) return rc;
        if (int rc = make_map(&maps.xl[i], xl[i], 1, pr.M, p.K, Cfg::BM)) return rc;
    }
    if (int rc = make_map(&maps.wh, wh, 1, w_rows, p.K, Cfg::BN)) return rc;
    if (int rc = make_map(&maps.wl, wl, 1, w_rows, p.K, Cfg::BN)) return rc;
    int sms = 0;
    if (int rc = sm_count(&sms)) return rc;
    if (int rc = allow_smem<txb::gemm_x3_kernel<Cfg>>((int)Cfg::SMEM_BYTES)) return rc;
    return launch_behind(txb::gemm_x3_kernel<Cfg>, dim3((unsigned)std::min(p.n_tiles, sms)), Cfg::THREADS, Cfg::SMEM_BYTES, st, 1, maps, p);
}

// Tile width by the number of rounds the persistent CTAs need: a 128 x 128 tile takes about 0.53 of a 128 x 256 one and
// 128 x 64 about 0.37 (the narrower the tile, the more of its time goes to bringing x).
int launch_gemm_x3(const txb::GemmX3Params &p, const __half *const *xh, const __half *const *xl, const __half *wh, const __half *wl,
                   int64_t w_rows, cudaStream_t st)
{
    int sms = 0;
    if (int rc = sm_count(&sms)) return rc;
    auto time = [&](int bn, double tile) {
        int64_t tiles = 0;
        for (int i = 0; i < p.n_probs; ++i) tiles += (int64_t)((p.prob[i].M + 127) / 128) * ((p.N + bn - 1) / bn);
        return (double)((tiles + sms - 1) / sms) * tile;
    };
    const double t256 = time(256, 1.0), t128 = time(128, 0.53), t64 = time(64, 0.37);
    if (t256 <= t128 && t256 <= t64) return launch_gemm_x3_t<txb::GemmX3Cfg<256>>(p, xh, xl, wh, wl, w_rows, st);
    if (t128 <= t64) return launch_gemm_x3_t<txb::GemmX3Cfg<128>>(p, xh, xl, wh, wl, w_rows, st);
    return launch_gemm_x3_t<txb::GemmX3Cfg<64>>(p, xh, xl, wh, wl, w_rows, st);
}

// The whole layer on one stream: operands split, three projections in one launch (head-split, fp32 or fp16), attention,
// its result split (heads merged on the way), output projection.  One workspace from the pool.
int mha_launch(const tx_mha_desc *d)
{
    cudaStream_t st = static_cast<cudaStream_t>(d->stream);
    int *status = nullptr;
    if (int rc = status_word(&status)) return rc;
    const int64_t E = d->embed, Mq = d->batch * d->seq_q, Mk = d->batch * d->seq_k;
    const bool f16 = (d->flags & TX_MHA_F16_ATTENTION) != 0;
    const int64_t M[3] = {Mq, Mk, Mk};
    const float *x[3] = {d->xq, d->xk, d->xv}, *w[4] = {d->wq, d->wk, d->wv, d->wo}, *bias[3] = {d->bq, d->bk, d->bv};
    const int64_t seq[3] = {d->seq_q, d->seq_k, d->seq_k};

    size_t total = 0;
    auto take = [&](size_t bytes) { const size_t at = total; total += align_up(bytes, 256); return at; };
    int from[3];                                                  // inputs passed more than once are split once
    size_t o_xh[3], o_xl[3], o_xi[3];
    for (int i = 0; i < 3; ++i) {
        from[i] = i;
        for (int j = 0; j < i; ++j)
            if (x[j] == x[i] && M[j] == M[i]) { from[i] = j; break; }
        if (from[i] != i) { o_xh[i] = o_xh[from[i]]; o_xl[i] = o_xl[from[i]]; o_xi[i] = o_xi[from[i]]; continue; }
        o_xh[i] = take((size_t)(M[i] * E) * 2); o_xl[i] = take((size_t)(M[i] * E) * 2); o_xi[i] = take((size_t)M[i] * 4);
    }
    const size_t o_wh = take((size_t)(4 * E * E) * 2), o_wl = take((size_t)(4 * E * E) * 2), o_wi = take((size_t)(4 * E) * 4);
    const size_t es = f16 ? 2 : 4;
    const size_t o_p[3] = {take((size_t)(Mq * E) * es), take((size_t)(Mk * E) * es), take((size_t)(Mk * E) * es)};
    const size_t o_a = take((size_t)(Mq * E) * 4), o_range = take(4 * sizeof(int));
    // the attention result's halves go where the inputs' were (none is needed any more and Q's are as large)
    const size_t o_ah = o_xh[0], o_al = o_xl[0], o_ai = o_xi[0];

    char *ws = nullptr;
    if (int rc = pool_alloc(&ws, total, st)) return rc;
    auto half_at = [&](size_t at) { return reinterpret_cast<__half *>(ws + at); };
    auto float_at = [&](size_t at) { return reinterpret_cast<float *>(ws + at); };
    auto body = [&]() -> int {
        txb::SplitRowsParams sp;
        int *range = reinterpret_cast<int *>(ws + o_range), *outliers = range + 3;     // of the attention step, of the projections
        TX_CUDA(cudaMemsetAsync(range, 0, 4 * sizeof(int), st));
        sp.n_segs = 0; sp.rows = 0; sp.K = (int)E; sp.outliers = outliers;
        auto add = [&](const float *src, size_t hi, size_t lo, size_t inv, int64_t rows, int64_t first_row, int heads, int64_t S) {
            txb::SplitRowsSeg &s = sp.seg[sp.n_segs++];
            s.x = src; s.hi = half_at(hi) + first_row * E; s.lo = half_at(lo) + first_row * E; s.inv = float_at(inv) + first_row;
            s.rows = (int)rows; s.heads = heads; s.S = (int)S; s.first = sp.rows;
            sp.rows += (int)rows;
        };
        auto split_grid = [&]() { return dim3((unsigned)((sp.rows + 7) / 8)); };
        for (int i = 0; i < 3; ++i)
            if (from[i] == i) add(x[i], o_xh[i], o_xl[i], o_xi[i], M[i], 0, 0, 1);
        for (int i = 0; i < 4; ++i) add(w[i], o_wh, o_wl, o_wi, E, i * E, 0, 1);
        txb::split_rows_kernel<<<split_grid(), 256, 0, st>>>(sp);          // behind whatever the caller enqueued: a plain launch
        g_launches++;
        TX_CUDA(cudaGetLastError());

        txb::GemmX3Params g;
        g.N = g.K = (int)E; g.status = status; g.out_f16 = f16 ? 1 : 0; g.n_probs = 3; g.outliers = outliers;
        const __half *xh[3], *xl[3];
        for (int i = 0; i < 3; ++i) {
            xh[i] = half_at(o_xh[i]); xl[i] = half_at(o_xl[i]);
            g.prob[i] = {float_at(o_xi[i]), float_at(o_wi) + i * E, bias[i], ws + o_p[i], (int)M[i], (int)seq[i], (int)d->heads,
                         x[i], w[i], 0, (int)(i * E), 0, 0};
        }
        if (int rc = launch_gemm_x3(g, xh, xl, half_at(o_wh), half_at(o_wl), 3 * E, st)) return rc;

        tx_sdpa_desc a;
        std::memset(&a, 0, sizeof a);
        a.q = ws + o_p[0]; a.k = ws + o_p[1]; a.v = ws + o_p[2]; a.out = ws + o_a;
        a.mask = d->mask; a.kv_lens = d->kv_lens;
        a.batch = d->batch; a.q_heads = a.kv_heads = d->heads;
        a.seq_q = d->seq_q; a.seq_k = d->seq_k; a.d_k = a.d_v = E / d->heads;
        a.dtype = f16 ? TX_DTYPE_F16 : TX_DTYPE_F32;
        a.causal = d->causal; a.flags = d->flags & TX_SDPA_KV_LENS_HOST; a.stream = d->stream;
        if (x3_eligible(&a) && !decode_eligible(&a)) {
            if (int rc = validate(&a)) return rc;
            if (int rc = with_device_lens(&a, [&](const tx_sdpa_desc *e) { return launch_x3(e, st, status, range); })) return rc;
        } else if (int rc = forward(&a)) {
            return rc;
        }

        sp.n_segs = 0; sp.rows = 0;
        add(float_at(o_a), o_ah, o_al, o_ai, Mq, 0, (int)d->heads, d->seq_q);
        if (int rc = launch_behind(txb::split_rows_kernel, split_grid(), 256, 0, st, 1, sp)) return rc;
        g.n_probs = 1; g.out_f16 = 0;
        g.prob[0] = {float_at(o_ai), float_at(o_wi) + 3 * E, d->bo, d->out, (int)Mq, (int)d->seq_q, 0,
                     float_at(o_a), d->wo, (int)d->heads, 0, 0, 0};
        xh[0] = half_at(o_ah); xl[0] = half_at(o_al);
        return launch_gemm_x3(g, xh, xl, half_at(o_wh) + 3 * E * E, half_at(o_wl) + 3 * E * E, E, st);
    };
    const int rc = body();
    pool_free(ws, st);
    return rc;
}

int sync_f32(const float *Q, const float *K, const float *V, const float *mask, float *out,
             int64_t B, int64_t H, int64_t Sq, int64_t Sk, int64_t dk, int64_t dv)
{
    tx_sdpa_desc d;
    std::memset(&d, 0, sizeof d);
    d.q = Q; d.k = K; d.v = V; d.mask = mask; d.out = out;
    d.batch = B; d.q_heads = H; d.kv_heads = H; d.seq_q = Sq; d.seq_k = Sk; d.d_k = dk; d.d_v = dv;
    d.dtype = TX_DTYPE_F32;
    if (int rc = forward(&d)) return rc;
    return finish(nullptr);
}

// The fp32 launchers' section profile: one instrumented launch of the exact-fp32 kernel, 32 clock64
// stamps of thread 0 of CTA (0,0,0) (txb::SimtStamp; unused entries stay 0), as the reference's
// sdpa_*_profile_sections_cuda return them (csrc/cuda/kernels/attn.cu:1113-1140,1617-1722).
int profile_f32(const float *Q, const float *K, const float *V, const float *mask, float *out,
                int64_t B, int64_t H, int64_t Sq, int64_t Sk, int64_t dk, int64_t dv, long long *ticks32)
{
    if (!ticks32) return fail(TX_ERR_INVALID, "profile_sections: null output");
    tx_sdpa_desc d;
    std::memset(&d, 0, sizeof d);
    d.q = Q; d.k = K; d.v = V; d.mask = mask; d.out = out;
    d.batch = B; d.q_heads = H; d.kv_heads = H; d.seq_q = Sq; d.seq_k = Sk; d.d_k = dk; d.d_v = dv;
    d.dtype = TX_DTYPE_F32;
    if (int rc = validate(&d)) return rc;
    if (int rc = ensure_device()) return rc;
    long long *dev = nullptr;
    TX_CUDA(cudaMalloc(&dev, 32 * sizeof(long long)));
    int rc = cudaMemset(dev, 0, 32 * sizeof(long long)) == cudaSuccess ? TX_OK : fail(TX_ERR_CUDA, "cudaMemset failed");
    if (rc == TX_OK) {
        txb::SimtParams p;
        p.q = Q; p.k = K; p.v = V; p.mask = mask; p.out = out; p.out_f16 = 0;
        p.B = B; p.Hq = H; p.Hkv = H; p.Sq = Sq; p.Sk = Sk; p.dk = dk; p.dv = dv;
        p.causal = 0;
        p.scale = 1.0f / std::sqrt((float)dk);
        p.prof = dev;
        rc = launch_simt<float, true>(p, nullptr);
    }
    if (rc == TX_OK) rc = finish(nullptr);
    if (rc == TX_OK && cudaMemcpy(ticks32, dev, 32 * sizeof(long long), cudaMemcpyDeviceToHost) != cudaSuccess)
        rc = fail(TX_ERR_CUDA, "cudaMemcpy of the section profile failed");
    (void)cudaFree(dev);
    return rc;
}

__global__ void cast_f32_to_f16_kernel(const float *__restrict__ in, __half *__restrict__ out, int64_t n)
{
    const int64_t i = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) * 4;
    if (i + 3 < n && ((reinterpret_cast<uintptr_t>(in) | reinterpret_cast<uintptr_t>(out)) & 15u) == 0) {
        const float4 f = *reinterpret_cast<const float4 *>(in + i);
        __half2 a = __floats2half2_rn(f.x, f.y), b = __floats2half2_rn(f.z, f.w);
        uint2 u;
        u.x = *reinterpret_cast<uint32_t *>(&a);
        u.y = *reinterpret_cast<uint32_t *>(&b);
        *reinterpret_cast<uint2 *>(out + i) = u;
    } else {
        for (int64_t j = i; j < n && j < i + 4; ++j) out[j] = __float2half_rn(in[j]);
    }
}

// Result slab of one chunk of the host form, written by a few CTAs straight into the caller's pinned (device-mapped)
// buffer: 16 bytes per thread, a warp's 512 bytes contiguous.
__global__ void __launch_bounds__(1024) copy_out_kernel(const uint4 *__restrict__ src, uint4 *__restrict__ dst, size_t n16)
{
    const size_t stride = (size_t)gridDim.x * blockDim.x;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n16; i += stride) dst[i] = src[i];
}

template <typename T>
__global__ void repeat_interleave_kernel(const T *__restrict__ in, T *__restrict__ out, int64_t total,
                                         int64_t dim_size, int64_t inner, int64_t repeats)
{
    for (int64_t o = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; o < total;
         o += (int64_t)gridDim.x * blockDim.x) {
        const int64_t k = o % inner;
        const int64_t jr = (o / inner) % (dim_size * repeats);
        const int64_t i = o / (inner * dim_size * repeats);
        out[o] = in[(i * dim_size + jr / repeats) * inner + k];
    }
}

// ------------------------------------------------------------------ host-buffer form
struct Workspace {
    void *ptr = nullptr;
    size_t bytes = 0;
};
Workspace g_ws[kMaxDevices];
std::mutex g_ws_mu;

int workspace(size_t bytes, void **out)
{
    int dev = 0;
    TX_CUDA(cudaGetDevice(&dev));
    if (dev < 0 || dev >= kMaxDevices) return fail(TX_ERR_INVALID, "device index %d out of range", dev);
    Workspace &w = g_ws[dev];
    if (w.bytes < bytes) {
        if (w.ptr) TX_CUDA(cudaFree(w.ptr));
        w.ptr = nullptr;
        w.bytes = 0;
        TX_CUDA(cudaMalloc(&w.ptr, bytes));
        w.bytes = bytes;
    }
    *out = w.ptr;
    return TX_OK;
}

size_t align_up(size_t x, size_t a) { return (x + a - 1) / a * a; }

std::atomic<int> g_linear_force_simt{0};
bool flags_linear_force_simt() { return g_linear_force_simt.load() != 0; }

// Streams and events of the host-buffer form, created once per device.
constexpr int kHostChunks = 16;
struct HostPipe {
    bool ready = false;
    cudaStream_t in = nullptr, out = nullptr;
    cudaEvent_t start = nullptr, out_done = nullptr, in_done[kHostChunks] = {}, k_done[kHostChunks] = {};
};
HostPipe g_pipe[kMaxDevices];

int host_pipe(HostPipe **out)
{
    int dev = 0;
    TX_CUDA(cudaGetDevice(&dev));
    if (dev < 0 || dev >= kMaxDevices) return fail(TX_ERR_INVALID, "device index %d out of range", dev);
    HostPipe &p = g_pipe[dev];
    if (!p.ready) {
        TX_CUDA(cudaStreamCreateWithFlags(&p.in, cudaStreamNonBlocking));
        TX_CUDA(cudaStreamCreateWithFlags(&p.out, cudaStreamNonBlocking));
        TX_CUDA(cudaEventCreateWithFlags(&p.start, cudaEventDisableTiming));
        TX_CUDA(cudaEventCreateWithFlags(&p.out_done, cudaEventDisableTiming));
        for (int i = 0; i < kHostChunks; ++i) {
            TX_CUDA(cudaEventCreateWithFlags(&p.in_done[i], cudaEventDisableTiming));
            TX_CUDA(cudaEventCreateWithFlags(&p.k_done[i], cudaEventDisableTiming));
        }
        p.ready = true;
    }
    *out = &p;
    return TX_OK;
}

// ------------------------------------------------------------------ allocation-free form
// Scratch of tx_sdpa_fp16_static_scratch: [0,256) status word (+ padding), then up to
// TX_STATIC_SCRATCH_MAX_BATCH key lengths.  It is part of the module image on every GPU that
// loads the library.  In host code the name below is only a handle for
// cudaGetSymbolAddress; kernels are given the address that call returns.
static __device__ __align__(256) unsigned char g_static_scratch[TX_STATIC_SCRATCH_BYTES];
unsigned char *g_static_scratch_addr[kMaxDevices] = {};
std::mutex g_static_mu;

// Device address of the array on the current device, looked up once per device.
int static_scratch(unsigned char **out)
{
    int dev = 0;
    TX_CUDA(cudaGetDevice(&dev));
    if (dev < 0 || dev >= kMaxDevices) return fail(TX_ERR_INVALID, "device index %d out of range", dev);
    std::lock_guard<std::mutex> lk(g_static_mu);
    if (!g_static_scratch_addr[dev]) {
        unsigned char *ptr = nullptr;
        TX_CUDA(cudaGetSymbolAddress(reinterpret_cast<void **>(&ptr), g_static_scratch));
        if (!ptr) return fail(TX_ERR_CUDA, "cudaGetSymbolAddress returned a null address for the static scratch");
        g_static_scratch_addr[dev] = ptr;
    }
    *out = g_static_scratch_addr[dev];
    return TX_OK;
}

// Output tensors are allocated per call by the dispatchers (csrc/tensor_ops.cpp:901-907), and in the
// reference every one of them is a cudaMalloc / cudaFree pair -- device-wide synchronisations that
// dominate short calls (docs/profiling/RESULTS.md:149-152).  Here the pair goes through the device's
// stream-ordered memory pool with a release threshold that keeps freed blocks cached, so a steady
// sequence of calls stops touching the driver's allocator after the first one.
// Freed blocks stay cached up to kPoolKeep bytes BEYOND what the program holds; more goes back to the driver at the
// next synchronisation, so a process on a shared GPU does not sit on everything it ever touched.  CUDA's release
// threshold counts the blocks in use too, so it follows them: with a fixed 4 GiB a program that held more than that
// in tensors had every freed block unmapped at each synchronisation and mapped again by the next call (a 1 GiB result:
// 4.6 ms to 24 ms per call around 3.7 ms of kernel).
constexpr unsigned long long kPoolKeep = 4ull << 30, kPoolStep = 1ull << 30;
struct PoolBooks {
    std::mutex mu;
    std::unordered_map<void *, std::pair<int, size_t>> blocks;     // pointer -> (device, bytes)
    unsigned long long live[kMaxDevices] = {}, steps[kMaxDevices] = {};
    cudaMemPool_t pool[kMaxDevices] = {};
};
PoolBooks &books()
{
    static PoolBooks *b = new PoolBooks;     // never destroyed: tensors may be freed while the process ends
    return *b;
}

// Called with the books locked: the release threshold in whole steps, so that it is set only now and then.
void pool_threshold(PoolBooks &bk, int dev)
{
    const unsigned long long steps = bk.live[dev] / kPoolStep + 1;
    if (steps == bk.steps[dev]) return;
    unsigned long long keep = steps * kPoolStep + kPoolKeep;
    if (cudaMemPoolSetAttribute(bk.pool[dev], cudaMemPoolAttrReleaseThreshold, &keep) == cudaSuccess) bk.steps[dev] = steps;
    else (void)cudaGetLastError();
}

void pool_took(void *ptr, size_t bytes)
{
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return;
    PoolBooks &bk = books();
    std::lock_guard<std::mutex> lk(bk.mu);
    bk.blocks[ptr] = {dev, bytes};
    bk.live[dev] += bytes;
    pool_threshold(bk, dev);
}

void pool_gave(void *ptr)
{
    PoolBooks &bk = books();
    std::lock_guard<std::mutex> lk(bk.mu);
    const auto it = bk.blocks.find(ptr);
    if (it == bk.blocks.end()) return;
    const int dev = it->second.first;
    bk.live[dev] -= it->second.second;
    bk.blocks.erase(it);
    pool_threshold(bk, dev);
}

int pool_ready()
{
    static std::atomic<bool> ready[kMaxDevices] = {};
    int dev = 0;
    if (int rc = current_device(&dev)) return rc;
    if (!ready[dev].load(std::memory_order_acquire)) {
        PoolBooks &bk = books();
        std::lock_guard<std::mutex> lk(bk.mu);
        TX_CUDA(cudaDeviceGetDefaultMemPool(&bk.pool[dev], dev));
        unsigned long long keep = kPoolStep + kPoolKeep;
        TX_CUDA(cudaMemPoolSetAttribute(bk.pool[dev], cudaMemPoolAttrReleaseThreshold, &keep));
        bk.steps[dev] = 1;
        ready[dev].store(true, std::memory_order_release);
    }
    return TX_OK;
}

}  // namespace

extern "C" {

const char *tx_last_error(void) { return g_err.c_str(); }
int tx_version(void) { return 100; }

int tx_cuda_is_available(void)
{
    int n = 0;
    if (cudaGetDeviceCount(&n) != cudaSuccess) {
        (void)cudaGetLastError();
        return 0;
    }
    return n > 0 ? 1 : 0;
}

int tx_cuda_device_count(void)
{
    int n = 0;
    if (cudaGetDeviceCount(&n) != cudaSuccess) {
        (void)cudaGetLastError();
        return 0;
    }
    return n;
}

int tx_cuda_set_device(int device)
{
    TX_CUDA(cudaSetDevice(device));
    return TX_OK;
}

void *tx_cuda_malloc(size_t bytes)
{
    void *p = nullptr;
    if (pool_ready() != TX_OK) return nullptr;
    cudaError_t e = cudaMallocAsync(&p, bytes ? bytes : 1, (cudaStream_t)0);
    if (e != cudaSuccess) {
        fail(TX_ERR_CUDA, "cudaMallocAsync(%zu) failed: %s", bytes, cudaGetErrorString(e));
        (void)cudaGetLastError();
        return nullptr;
    }
    pool_took(p, bytes ? bytes : 1);
    return p;
}

int tx_cuda_free(void *ptr)
{
    if (!ptr) return TX_OK;
    pool_gave(ptr);
    TX_CUDA(cudaFreeAsync(ptr, (cudaStream_t)0));
    return TX_OK;
}

int tx_cuda_free_on(void *ptr, void *stream)
{
    if (!ptr) return TX_OK;
    pool_gave(ptr);
    TX_CUDA(cudaFreeAsync(ptr, static_cast<cudaStream_t>(stream)));
    return TX_OK;
}

int tx_cuda_pool_trim(void)
{
    int dev = 0;
    TX_CUDA(cudaGetDevice(&dev));
    cudaMemPool_t pool;
    TX_CUDA(cudaDeviceGetDefaultMemPool(&pool, dev));
    TX_CUDA(cudaDeviceSynchronize());
    TX_CUDA(cudaMemPoolTrimTo(pool, 0));
    return TX_OK;
}

int tx_cuda_memcpy_h2d(void *dst, const void *src, size_t bytes)
{
    TX_CUDA(cudaMemcpy(dst, src, bytes, cudaMemcpyHostToDevice));
    return TX_OK;
}

int tx_cuda_memcpy_d2h(void *dst, const void *src, size_t bytes)
{
    TX_CUDA(cudaMemcpy(dst, src, bytes, cudaMemcpyDeviceToHost));
    return TX_OK;
}

int tx_cuda_memcpy_d2d(void *dst, const void *src, size_t bytes)
{
    TX_CUDA(cudaMemcpy(dst, src, bytes, cudaMemcpyDeviceToDevice));
    return TX_OK;
}

int tx_cuda_synchronize(void)
{
    TX_CUDA(cudaDeviceSynchronize());
    return TX_OK;
}

void *tx_host_alloc_pinned(size_t bytes)
{
    void *p = nullptr;
    cudaError_t e = cudaHostAlloc(&p, bytes ? bytes : 1, cudaHostAllocDefault);
    if (e != cudaSuccess) {
        fail(TX_ERR_CUDA, "cudaHostAlloc(%zu) failed: %s", bytes, cudaGetErrorString(e));
        (void)cudaGetLastError();
        return nullptr;
    }
    return p;
}

int tx_host_free_pinned(void *ptr)
{
    if (!ptr) return TX_OK;
    TX_CUDA(cudaFreeHost(ptr));
    return TX_OK;
}

int tx_sdpa_naive_cuda(const float *Q, const float *K, const float *V, const float *mask, float *out,
                       int64_t B, int64_t H, int64_t Sq, int64_t Sk, int64_t dk, int64_t dv)
{
    TX_NVTX_RANGE("sdpa.naive");
    return sync_f32(Q, K, V, mask, out, B, H, Sq, Sk, dk, dv);
}
int tx_sdpa_tiled_cuda(const float *Q, const float *K, const float *V, const float *mask, float *out,
                       int64_t B, int64_t H, int64_t Sq, int64_t Sk, int64_t dk, int64_t dv)
{
    TX_NVTX_RANGE("sdpa.tiled");
    return sync_f32(Q, K, V, mask, out, B, H, Sq, Sk, dk, dv);
}
int tx_sdpa_flash_cuda(const float *Q, const float *K, const float *V, const float *mask, float *out,
                       int64_t B, int64_t H, int64_t Sq, int64_t Sk, int64_t dk, int64_t dv)
{
    TX_NVTX_RANGE("sdpa.flash");
    return sync_f32(Q, K, V, mask, out, B, H, Sq, Sk, dk, dv);
}
int tx_sdpa_optimized_flash_cuda(const float *Q, const float *K, const float *V, const float *mask,
                                 float *out, int64_t B, int64_t H, int64_t Sq, int64_t Sk, int64_t dk,
                                 int64_t dv)
{
    TX_NVTX_RANGE("sdpa.flash_optimized");
    return sync_f32(Q, K, V, mask, out, B, H, Sq, Sk, dk, dv);
}
int tx_sdpa_mma_cuda(const float *Q, const float *K, const float *V, const float *mask, float *out,
                     int64_t B, int64_t H, int64_t Sq, int64_t Sk, int64_t dk, int64_t dv)
{
    TX_NVTX_RANGE("sdpa.mma");
    // The reference computes this variant with fp16 operands; the exact-fp32 kernel
    // is used here, which is strictly closer to the CPU path.
    return sync_f32(Q, K, V, mask, out, B, H, Sq, Sk, dk, dv);
}

int tx_sdpa_mma_fp16_cuda(const void *Q_h, const void *K_h, const void *V_h, float *out, int64_t B,
                          int64_t H, int64_t Sq, int64_t Sk, int64_t dk, int64_t dv)
{
    TX_NVTX_RANGE("sdpa.mma.fp16");
    tx_sdpa_desc d;
    std::memset(&d, 0, sizeof d);
    d.q = Q_h; d.k = K_h; d.v = V_h; d.out = out;
    d.batch = B; d.q_heads = H; d.kv_heads = H; d.seq_q = Sq; d.seq_k = Sk; d.d_k = dk; d.d_v = dv;
    d.dtype = TX_DTYPE_F16;
    if (int rc = forward(&d)) return rc;
    return finish(nullptr);
}

int tx_sdpa_naive_profile_sections_cuda(const float *Q, const float *K, const float *V, const float *mask, float *out,
        int64_t B, int64_t H, int64_t Sq, int64_t Sk, int64_t dk, int64_t dv, long long *ticks32)
{
    TX_NVTX_RANGE("sdpa.naive.profile");
    return profile_f32(Q, K, V, mask, out, B, H, Sq, Sk, dk, dv, ticks32);
}
int tx_sdpa_tiled_profile_sections_cuda(const float *Q, const float *K, const float *V, const float *mask, float *out,
        int64_t B, int64_t H, int64_t Sq, int64_t Sk, int64_t dk, int64_t dv, long long *ticks32)
{
    TX_NVTX_RANGE("sdpa.tiled.profile");
    return profile_f32(Q, K, V, mask, out, B, H, Sq, Sk, dk, dv, ticks32);
}
int tx_sdpa_flash_profile_sections_cuda(const float *Q, const float *K, const float *V, const float *mask, float *out,
        int64_t B, int64_t H, int64_t Sq, int64_t Sk, int64_t dk, int64_t dv, long long *ticks32)
{
    TX_NVTX_RANGE("sdpa.flash.profile");
    return profile_f32(Q, K, V, mask, out, B, H, Sq, Sk, dk, dv, ticks32);
}
int tx_sdpa_optimized_flash_profile_sections_cuda(const float *Q, const float *K, const float *V, const float *mask, float *out,
        int64_t B, int64_t H, int64_t Sq, int64_t Sk, int64_t dk, int64_t dv, long long *ticks32)
{
    TX_NVTX_RANGE("sdpa.flash_optimized.profile");
    return profile_f32(Q, K, V, mask, out, B, H, Sq, Sk, dk, dv, ticks32);
}
int tx_sdpa_mma_profile_sections_cuda(const float *Q, const float *K, const float *V, const float *mask, float *out,
        int64_t B, int64_t H, int64_t Sq, int64_t Sk, int64_t dk, int64_t dv, long long *ticks32)
{
    TX_NVTX_RANGE("sdpa.mma.profile");
    return profile_f32(Q, K, V, mask, out, B, H, Sq, Sk, dk, dv, ticks32);
}

int tx_cast_f32_to_f16_cuda(const float *in, void *out, int64_t size)
{
    if (size < 0 || (size > 0 && (!in || !out))) return fail(TX_ERR_INVALID, "cast_to_fp16: bad arguments");
    if (int rc = ensure_device()) return rc;
    if (size == 0) return TX_OK;
    const int threads = 256;
    const int64_t blocks = (size + threads * 4 - 1) / (threads * 4);
    if (blocks > 0x7fffffffLL) return fail(TX_ERR_UNSUPPORTED, "cast_to_fp16: tensor too large");
    cast_f32_to_f16_kernel<<<(unsigned)blocks, threads>>>(in, static_cast<__half *>(out), size);
    g_launches++;
    TX_CUDA(cudaGetLastError());
    return TX_OK;
}

int tx_repeat_interleave_cuda(const void *in, void *out, int64_t outer, int64_t dim_size,
                              int64_t inner, int64_t repeats, int32_t elem_bytes)
{
    if (!in || !out || outer <= 0 || dim_size <= 0 || inner <= 0 || repeats <= 0)
        return fail(TX_ERR_INVALID, "repeat_interleave: bad arguments");
    if (elem_bytes != 2 && elem_bytes != 4) return fail(TX_ERR_INVALID, "repeat_interleave: element size must be 2 or 4");
    if (int rc = ensure_device()) return rc;
    const int64_t total = outer * dim_size * repeats * inner;
    const int threads = 256;
    const unsigned blocks = (unsigned)std::min<int64_t>((total + threads - 1) / threads, 148 * 16);
    if (elem_bytes == 2)
        repeat_interleave_kernel<uint16_t><<<blocks, threads>>>(static_cast<const uint16_t *>(in),
                                                               static_cast<uint16_t *>(out), total, dim_size, inner, repeats);
    else
        repeat_interleave_kernel<uint32_t><<<blocks, threads>>>(static_cast<const uint32_t *>(in),
                                                               static_cast<uint32_t *>(out), total, dim_size, inner, repeats);
    g_launches++;
    TX_CUDA(cudaGetLastError());
    return TX_OK;
}

int tx_sdpa_set_group_l2_bytes(int64_t bytes)
{
    g_group_l2_bytes.store(bytes > 0 ? (long long)bytes : (48ll << 20));
    return TX_OK;
}

int tx_linear_set_cuda_cores_only(int on)
{
    g_linear_force_simt.store(on ? 1 : 0);
    return TX_OK;
}

int tx_linear_f32_cuda(const float *x, const float *w, const float *bias, float *out, int64_t batch,
                       int64_t seq, int64_t in_features, int64_t out_features, int32_t heads_in,
                       int32_t heads_out)
{
    if (!x || !w || !out || batch <= 0 || seq <= 0 || in_features <= 0 || out_features <= 0)
        return fail(TX_ERR_INVALID, "linear: bad arguments");
    if (heads_in < 0 || heads_out < 0 || (heads_in > 0 && in_features % heads_in) ||
        (heads_out > 0 && out_features % heads_out))
        return fail(TX_ERR_INVALID, "linear: feature count must be a multiple of the head count");
    if (int rc = ensure_device()) return rc;
    const int64_t dh_in = heads_in > 0 ? in_features / heads_in : in_features;
    const int64_t dh_out = heads_out > 0 ? out_features / heads_out : out_features;
    auto al = [](const void *q) { return (reinterpret_cast<uintptr_t>(q) & 15u) == 0; };
    const bool tensor_cores = !(flags_linear_force_simt()) && in_features % 32 == 0 && dh_in % 32 == 0 &&
                              out_features % 32 == 0 && dh_out % 32 == 0 && al(x) && al(w) && al(out) &&
                              (!bias || al(bias)) && batch <= 65535 && (seq + 127) / 128 <= 65535;
    if (tensor_cores) {
        int *status = nullptr;
        if (int rc = status_word(&status)) return rc;
        CUtensorMap tx_map, tw_map;
        const int64_t hin = heads_in > 0 ? heads_in : 1;
        cuuint64_t xd[4] = {(cuuint64_t)dh_in, (cuuint64_t)seq, (cuuint64_t)hin, (cuuint64_t)batch};
        cuuint64_t xs[3];
        if (heads_in > 0) {        // [B, H, S, dh]
            xs[0] = (cuuint64_t)dh_in * 4; xs[1] = (cuuint64_t)seq * dh_in * 4; xs[2] = (cuuint64_t)hin * seq * dh_in * 4;
        } else {                   // [B, S, K] seen as one head
            xs[0] = (cuuint64_t)in_features * 4; xs[1] = (cuuint64_t)seq * in_features * 4; xs[2] = (cuuint64_t)seq * in_features * 4;
        }
        if (int rc = make_map_f32(&tx_map, x, 4, xd, xs, txb::LTC_BM)) return rc;
        cuuint64_t wd[3] = {(cuuint64_t)in_features, (cuuint64_t)out_features, 1};
        cuuint64_t ws[2] = {(cuuint64_t)in_features * 4, (cuuint64_t)in_features * out_features * 4};
        if (int rc = make_map_f32(&tw_map, w, 3, wd, ws, txb::LTC_BN)) return rc;
        txb::LinearTcParams lp;
        lp.bias = bias; lp.out = out; lp.status = status;
        lp.S = (int)seq; lp.N = (int)out_features; lp.K = (int)in_features;
        lp.dh_in = (int)dh_in; lp.heads_out = heads_out;
        if (int rc = allow_smem<txb::linear_tc_kernel>((int)txb::LTC_SMEM)) return rc;
        dim3 grid((unsigned)((out_features + txb::LTC_BN - 1) / txb::LTC_BN), (unsigned)((seq + txb::LTC_BM - 1) / txb::LTC_BM),
                  (unsigned)batch);
        txb::linear_tc_kernel<<<grid, txb::LTC_THREADS, txb::LTC_SMEM>>>(tx_map, tw_map, lp);
        g_launches++;
        TX_CUDA(cudaGetLastError());
        return TX_OK;
    }
    txb::LinearParams p;
    p.x = x; p.w = w; p.bias = bias; p.out = out;
    p.B = batch; p.S = seq; p.K = in_features; p.N = out_features;
    p.heads_in = heads_in; p.heads_out = heads_out;
    const int64_t gy = (batch * seq + txb::LIN_BM - 1) / txb::LIN_BM, gx = (out_features + txb::LIN_BN - 1) / txb::LIN_BN;
    if (gy > 65535 || gx > 0x7fffffffLL) return fail(TX_ERR_UNSUPPORTED, "linear: too many rows for one launch");
    txb::linear_simt_kernel<<<dim3((unsigned)gx, (unsigned)gy), txb::LIN_THREADS>>>(p);
    g_launches++;
    TX_CUDA(cudaGetLastError());
    return TX_OK;
}

int tx_mha_forward_f32(const tx_mha_desc *d)
{
    TX_NVTX_RANGE("mha.forward");
    if (!d || !d->xq || !d->xk || !d->xv || !d->wq || !d->wk || !d->wv || !d->wo || !d->out)
        return fail(TX_ERR_INVALID, "MHA: inputs, weights and output must not be null");
    if (d->batch <= 0 || d->seq_q <= 0 || d->seq_k <= 0 || d->embed <= 0 || d->heads <= 0 || d->embed % d->heads)
        return fail(TX_ERR_INVALID, "MHA: every dimension must be positive and embed a multiple of heads");
    const void *ptrs[] = {d->xq, d->xk, d->xv, d->wq, d->wk, d->wv, d->wo, d->bq, d->bk, d->bv, d->bo, d->out};
    bool aligned = true;
    for (const void *q : ptrs) aligned = aligned && (reinterpret_cast<uintptr_t>(q) & 15u) == 0;
    const int64_t M = d->batch * std::max(d->seq_q, d->seq_k);
    if (!aligned || d->embed % 8 || d->embed / d->heads % 4 || 4 * d->embed > 0x7fffffff || 3 * M > 0x7fffffff - 4 * d->embed)
        return fail(TX_ERR_UNSUPPORTED, "MHA: built for 16-byte aligned tensors, embed a multiple of 8 and head dims of 4");
    if (int rc = ensure_device()) return rc;
    return mha_launch(d);
}

int tx_sdpa_forward(const tx_sdpa_desc *desc)
{
    TX_NVTX_RANGE("sdpa.forward");
    return forward(desc);
}

int tx_profile_sections_sdpa(const tx_sdpa_desc *d, long long *ticks64)
{
    TX_NVTX_RANGE("sdpa.mma.fp16.profile");
    if (!ticks64) return fail(TX_ERR_INVALID, "profile_sections: null output");
    if (int rc = validate(d)) return rc;
    if (!tc_eligible(d))
        return fail(TX_ERR_UNSUPPORTED, "profile_sections: built for the tensor-core kernel only");
    if (d->flags & TX_SDPA_P_IN_SMEM)
        return fail(TX_ERR_UNSUPPORTED, "profile_sections: not built for the P-in-shared-memory variant");
    if (int rc = ensure_device()) return rc;
    int *status = nullptr;
    if (int rc = status_word(&status)) return rc;
    long long *dev = nullptr;
    TX_CUDA(cudaMalloc(&dev, 64 * sizeof(long long)));
    cudaStream_t st = static_cast<cudaStream_t>(d->stream);
    int rc = TX_OK;
    if (cudaMemsetAsync(dev, 0, 64 * sizeof(long long), st) != cudaSuccess) rc = fail(TX_ERR_CUDA, "cudaMemsetAsync failed");
    if (rc == TX_OK) rc = with_device_lens(d, [&](const tx_sdpa_desc *e) { return launch_tc(e, st, status, dev); });
    if (rc == TX_OK) rc = finish(st);
    if (rc == TX_OK && cudaMemcpy(ticks64, dev, 64 * sizeof(long long), cudaMemcpyDeviceToHost) != cudaSuccess)
        rc = fail(TX_ERR_CUDA, "cudaMemcpy of the section profile failed");
    (void)cudaFree(dev);
    return rc;
}

int tx_selftest_wait_timeout(const tx_sdpa_desc *d, int32_t skip_k_tile)
{
    if (int rc = validate(d)) return rc;
    if (!tc_eligible(d) || d->d_k != 64 || (d->flags & TX_SDPA_P_IN_SMEM))
        return fail(TX_ERR_UNSUPPORTED, "wait-timeout self-test: built for the fp16 d = 64 tensor-core kernel");
    if (int rc = ensure_device()) return rc;
    int *status = nullptr;
    if (int rc = status_word(&status)) return rc;
    cudaStream_t st = static_cast<cudaStream_t>(d->stream);
    if (int rc = with_device_lens(d, [&](const tx_sdpa_desc *e) {
            return launch_pair_t<txb::PairCfg<64, 128, 4, kPolyPairsD64, false, false, true>>(e, st, status, nullptr, skip_k_tile);
        }))
        return rc;
    return finish(st);
}

static int backward_launch(const tx_sdpa_bwd_desc *d);

int tx_sdpa_backward(const tx_sdpa_bwd_desc *d)
{
    if (!d) return fail(TX_ERR_INVALID, "SDPA backward: null descriptor");
    if (!d->q || !d->k || !d->v || !d->out || !d->dout || !d->lse || !d->dq || !d->dk || !d->dv)
        return fail(TX_ERR_INVALID, "SDPA backward: q, k, v, out, dout, lse, dq, dk, dv must not be null");
    if (d->batch <= 0 || d->q_heads <= 0 || d->kv_heads <= 0 || d->seq_q <= 0 || d->seq_k <= 0)
        return fail(TX_ERR_INVALID, "SDPA backward: every dimension must be positive");
    if (d->q_heads % d->kv_heads != 0)
        return fail(TX_ERR_INVALID, "SDPA backward: q_heads %lld not a multiple of kv_heads %lld",
                    (long long)d->q_heads, (long long)d->kv_heads);
    if (d->d != 64 && d->d != 128 && d->d != 256)
        return fail(TX_ERR_UNSUPPORTED, "SDPA backward: built for d in {64, 128, 256}, got %lld", (long long)d->d);
    if (d->batch * d->q_heads > 65535 || d->seq_q > 0x3fffffffLL || d->seq_k > 0x3fffffffLL)
        return fail(TX_ERR_UNSUPPORTED, "SDPA backward: dimension too large");
    auto al = [](const void *p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; };
    if (!al(d->q) || !al(d->k) || !al(d->v) || !al(d->out) || !al(d->dout) || !al(d->dq) || !al(d->dk) || !al(d->dv))
        return fail(TX_ERR_INVALID, "SDPA backward: pointers must be 16-byte aligned");
    if (int rc = ensure_device()) return rc;
    return with_device_lens(d, backward_launch);
}

static int backward_launch(const tx_sdpa_bwd_desc *d)
{
    int *status = nullptr;
    if (int rc = status_word(&status)) return rc;
    cudaStream_t st = static_cast<cudaStream_t>(d->stream);
    const int64_t rows = d->batch * d->q_heads * d->seq_q;
    const size_t h_bytes = align_up((size_t)rows * (size_t)d->d * 2, 256), delta_bytes = align_up((size_t)rows * 4, 256);
    char *ws = nullptr;
    if (int rc = pool_alloc(&ws, h_bytes + delta_bytes + sizeof(int), st)) return rc;
    __half *dout_h = reinterpret_cast<__half *>(ws);
    float *delta = reinterpret_cast<float *>(ws + h_bytes);
    int *prepared = reinterpret_cast<int *>(ws + h_bytes + delta_bytes);
    auto prep = [&](auto out, auto dim) {
        constexpr int D = decltype(dim)::value, rows_per_cta = 8 * 2 * (D == 64 ? 2 : 1);
        txb::sdpa_bwd_prep_kernel<std::remove_const_t<std::remove_pointer_t<decltype(out)>>, D>
            <<<(unsigned)((rows + rows_per_cta - 1) / rows_per_cta), 256, 0, st>>>(d->dout, out, dout_h, delta, rows, prepared);
    };
    auto prep_of = [&](auto out) {
        if (d->d == 64) prep(out, std::integral_constant<int, 64>{});
        else if (d->d == 128) prep(out, std::integral_constant<int, 128>{});
        else prep(out, std::integral_constant<int, 256>{});
    };
    if (d->flags & TX_SDPA_OUT_F16) prep_of(static_cast<const __half *>(d->out));
    else prep_of(static_cast<const float *>(d->out));
    g_launches++;
    int rc = (cudaGetLastError() == cudaSuccess) ? TX_OK : fail(TX_ERR_CUDA, "SDPA backward: preprocess launch failed");
    if (rc == TX_OK) {
        // d = 64: two CTAs per SM for both kernels (64-key / 64-query tiles; dK/dV stages P^T and dS^T in shared
        // memory to stay inside 256 tensor-memory columns: 3.23 ms against 3.51 ms with 128-query tiles, one CTA
        // per SM and two row warpgroups, config-2 size).
        // d = 128: one CTA per SM for both, two row warpgroups, 128-key / 64-query tiles (all of tensor memory).
        if (d->d == 64)
            rc = launch_bwd<64, txb::BwdDqCfg<64, 64, 3, 1, 2>, txb::BwdDkvCfg<64, 64, 3, 1, true, 2>>(d, st, status, dout_h, delta, prepared);
        else if (d->d == 128)
            rc = launch_bwd<128, txb::BwdDqCfg<128, 128, 3, 2, 2>, txb::BwdDkvCfg<128, 64, 3, 2, false, 3>>(d, st, status, dout_h, delta, prepared);
        else
            // d = 256: dQ alone takes 256 tensor-memory columns (64-key tiles, single V stage: 224 KB of shared
            // memory); two CTAs per key tile each own 128 columns of dK and dV, with 32-query tiles so that two
            // stages each of Q and dO fit beside the resident K and V (a stage stays occupied from its first
            // read to its second, so one stage per ring would deadlock the MMA warp).
            rc = launch_bwd<256, txb::BwdDqCfg<256, 64, 2, 1, 1>, txb::BwdDkvCfg<256, 32, 2, 1, false, 2, 2>>(d, st, status, dout_h, delta, prepared);
    }
    pool_free(ws, st);        // ordered after the kernels on `st`
    return rc;
}

int tx_sdpa_finish(void *stream) { return finish(static_cast<cudaStream_t>(stream)); }

int tx_sdpa_uses_tensor_cores(const tx_sdpa_desc *desc)
{
    if (validate(desc) != TX_OK) return 0;
    tx_sdpa_desc h;
    const Route route = route_of(via_f16(desc, &h) ? &h : desc);
    return route == Route::TensorCores || route == Route::Pairs ? 1 : 0;
}

int64_t tx_kernel_launch_count(void) { return g_launches.load(); }

// Host-buffer form.  `with_kernel == false` runs the same copy schedule with the kernels left out: what the
// host <-> device path alone takes (the benchmark reports it beside the full call).
static int forward_host(const tx_sdpa_desc *h, bool with_kernel)
{
    if (int rc = validate(h)) return rc;
    if (h->mask) return fail(TX_ERR_UNSUPPORTED, "SDPA host form: dense masks are not taken; use causal / kv_lens");
    if (h->lse) return fail(TX_ERR_UNSUPPORTED, "SDPA host form: no log-sum-exp output");
    if (int rc = ensure_device()) return rc;
    // The call is cut into chunks of whole (batch, K/V head) units -- contiguous slabs of Q, K, V and
    // O -- so that the upload of chunk i+1, the kernel of chunk i and the download of chunk i-1 run
    // at the same time on three streams (PCIe is full duplex; with pinned host buffers the copies
    // are asynchronous).  Chunks are about an eighth of the call: smaller ones start the first kernel and
    // the first download earlier but pay the fixed cost of a copy (some microseconds) more often.
    const int64_t units = h->batch * h->kv_heads, group = h->q_heads / h->kv_heads;
    const size_t es = h->dtype == TX_DTYPE_F16 ? 2 : 4;
    const size_t uq = (size_t)(group * h->seq_q * h->d_k) * es;       // bytes of one unit
    const size_t uk = (size_t)(h->seq_k * h->d_k) * es;
    const size_t uv = (size_t)(h->seq_k * h->d_v) * es;
    const size_t uo = (size_t)(group * h->seq_q * h->d_v) * ((h->flags & TX_SDPA_OUT_F16) ? 2 : 4);
    const size_t nl = h->kv_lens ? (size_t)units * 4 : 0;
    const size_t oq = 0, ok = align_up(oq + uq * units, 256), ov = align_up(ok + uk * units, 256),
                 oo = align_up(ov + uv * units, 256), ol = align_up(oo + uo * units, 256);
    const size_t total = align_up(ol + nl, 256);
    std::lock_guard<std::mutex> lk(g_ws_mu);
    void *base = nullptr;
    if (int rc = workspace(total, &base)) return rc;
    char *w = static_cast<char *>(base);
    HostPipe *hp = nullptr;
    if (int rc = host_pipe(&hp)) return rc;
    cudaStream_t st = static_cast<cudaStream_t>(h->stream);

    // chunk boundaries in units
    int64_t bounds[kHostChunks + 1];
    int n_chunks = 0;
    bounds[0] = 0;
    const size_t bytes_total = (uq + uk + uv + uo) * (size_t)units;
    if (bytes_total < (8u << 20) || units < 2) {                       // too small to be worth cutting
        bounds[1] = units;
        n_chunks = 1;
    } else {
        // A small first chunk (the first kernel and the first download start early), large middle chunks (every
        // copy costs about 10 us of set-up and small opposite copies disturb each other), a small last chunk (its
        // kernel and its download are the tail nothing overlaps).  Measured on B200 + PCIe 5 with the copies alone
        // (96 MiB in, 64 MiB out; units 4 8 8 6 4 2 of 32): 2.35 ms; eight eighths 2.49, 4 6 4 4 4 4 4 2 2.44,
        // quarters 2.39, sixteenths 2.81, one chunk 3.00; two big opposite copies 1.93, the upload alone 1.82.
        static const double cum[] = {0.125, 0.375, 0.625, 0.8125, 0.9375, 1.0};
        int64_t u = 0;
        for (double f : cum) {
            const int64_t to = std::min<int64_t>(units, std::max<int64_t>(u + 1, (int64_t)std::llround(f * (double)units)));
            if (to > u) { u = to; bounds[++n_chunks] = u; }
            if (u >= units) break;
        }
        if (u < units) bounds[n_chunks] = units;
    }
    // The result goes back either by the copy engine or, when the caller's buffer is pinned memory the device can
    // address (what tx_host_alloc_pinned returns), by a small kernel that writes it there: next to the uploads the
    // copy engine's many small downloads disturbed them more (copies alone, 96 MiB in and 64 MiB out in eight chunks:
    // 2.19 ms with the kernel, 2.44 ms with download copies; two big opposite copies 1.93 ms).
    uint4 *out_mapped = nullptr;
    {
        cudaPointerAttributes at;
        if (cudaPointerGetAttributes(&at, h->out) == cudaSuccess && at.type == cudaMemoryTypeHost && at.devicePointer &&
            (reinterpret_cast<uintptr_t>(at.devicePointer) & 15u) == 0 && (uo & 15u) == 0)
            out_mapped = static_cast<uint4 *>(at.devicePointer);
        else
            (void)cudaGetLastError();
    }
    // everything below is ordered after what the caller already put on its stream
    TX_CUDA(cudaEventRecord(hp->start, st));
    TX_CUDA(cudaStreamWaitEvent(hp->in, hp->start, 0));
    TX_CUDA(cudaStreamWaitEvent(hp->out, hp->start, 0));
    std::vector<int32_t> unit_lens;
    if (nl) {
        unit_lens.resize((size_t)units);
        for (int64_t u = 0; u < units; ++u) unit_lens[(size_t)u] = h->kv_lens[u / h->kv_heads];
        TX_CUDA(cudaMemcpyAsync(w + ol, unit_lens.data(), nl, cudaMemcpyHostToDevice, hp->in));
    }
    for (int c = 0; c < n_chunks; ++c) {
        const int64_t u0 = bounds[c], u1 = bounds[c + 1], nu = u1 - u0;
        if (nu <= 0) continue;
        TX_CUDA(cudaMemcpyAsync(w + oq + uq * u0, static_cast<const char *>(h->q) + uq * u0, uq * nu, cudaMemcpyHostToDevice, hp->in));
        TX_CUDA(cudaMemcpyAsync(w + ok + uk * u0, static_cast<const char *>(h->k) + uk * u0, uk * nu, cudaMemcpyHostToDevice, hp->in));
        TX_CUDA(cudaMemcpyAsync(w + ov + uv * u0, static_cast<const char *>(h->v) + uv * u0, uv * nu, cudaMemcpyHostToDevice, hp->in));
        TX_CUDA(cudaEventRecord(hp->in_done[c], hp->in));
        TX_CUDA(cudaStreamWaitEvent(st, hp->in_done[c], 0));
        if (with_kernel) {
            tx_sdpa_desc d = *h;                   // the chunk as a problem of its own: one K/V head per "batch"
            d.q = w + oq + uq * u0; d.k = w + ok + uk * u0; d.v = w + ov + uv * u0;
            d.out = w + oo + uo * u0;
            d.kv_lens = nl ? reinterpret_cast<const int32_t *>(w + ol) + u0 : nullptr;
            d.flags &= ~TX_SDPA_KV_LENS_HOST;
            d.batch = nu; d.q_heads = group; d.kv_heads = 1;
            if (int rc = forward(&d)) return rc;
        }
        TX_CUDA(cudaEventRecord(hp->k_done[c], st));
        TX_CUDA(cudaStreamWaitEvent(hp->out, hp->k_done[c], 0));
        if (out_mapped) {
            copy_out_kernel<<<8, 1024, 0, hp->out>>>(reinterpret_cast<const uint4 *>(w + oo + uo * u0),
                                                     out_mapped + (uo * u0) / 16, (uo * (size_t)nu) / 16);
            g_launches++;
            TX_CUDA(cudaGetLastError());
        } else {
            TX_CUDA(cudaMemcpyAsync(reinterpret_cast<char *>(h->out) + uo * u0, w + oo + uo * u0, uo * nu, cudaMemcpyDeviceToHost, hp->out));
        }
    }
    TX_CUDA(cudaEventRecord(hp->out_done, hp->out));
    TX_CUDA(cudaStreamWaitEvent(st, hp->out_done, 0));      // the caller's stream ends after the last download
    return finish(st);
}

int tx_sdpa_forward_host(const tx_sdpa_desc *h)
{
    TX_NVTX_RANGE("sdpa.forward_host");
    return forward_host(h, true);
}

int tx_sdpa_forward_host_copies_only(const tx_sdpa_desc *h) { return forward_host(h, false); }

int tx_sdpa_fp16_static_scratch(const void *Q_h, const void *K_h, const void *V_h, float *out,
                                int64_t batch, int64_t q_heads, int64_t kv_heads, int64_t seq_q,
                                int64_t seq_k, int64_t d, int32_t causal, const int32_t *kv_lens_host,
                                void *stream)
{
    tx_sdpa_desc desc;
    std::memset(&desc, 0, sizeof desc);
    desc.q = Q_h; desc.k = K_h; desc.v = V_h; desc.out = out;
    desc.batch = batch; desc.q_heads = q_heads; desc.kv_heads = kv_heads;
    desc.seq_q = seq_q; desc.seq_k = seq_k; desc.d_k = d; desc.d_v = d;
    desc.dtype = TX_DTYPE_F16;
    desc.causal = causal;
    desc.stream = stream;
    if (int rc = validate(&desc)) return rc;
    if (kv_lens_host && batch > TX_STATIC_SCRATCH_MAX_BATCH)
        return fail(TX_ERR_INVALID, "static-scratch SDPA: batch %lld exceeds the %d key lengths the fixed scratch holds",
                    (long long)batch, TX_STATIC_SCRATCH_MAX_BATCH);
    if (!tc_eligible(&desc))
        return fail(TX_ERR_UNSUPPORTED,
                    "static-scratch SDPA: only the tensor-core shapes are taken (fp16, d_k == d_v in {64,128,256,512}, "
                    "16-byte aligned pointers, batch*heads <= 65535)");
    if (int rc = ensure_device()) return rc;
    unsigned char *scratch = nullptr;
    if (int rc = static_scratch(&scratch)) return rc;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    int *status = reinterpret_cast<int *>(scratch);
    TX_CUDA(cudaMemsetAsync(status, 0, 256, st));            // the array keeps the last call's contents
    if (kv_lens_host) {
        TX_CUDA(cudaMemcpyAsync(scratch + 256, kv_lens_host, (size_t)batch * 4, cudaMemcpyHostToDevice, st));
        desc.kv_lens = reinterpret_cast<const int32_t *>(scratch + 256);
    }
    if (int rc = launch_f16(&desc, st, status)) return rc;
    int code = 0;
    TX_CUDA(cudaMemcpyAsync(&code, status, sizeof code, cudaMemcpyDeviceToHost, st));
    TX_CUDA(cudaStreamSynchronize(st));
    if (code != 0)
        return fail(TX_ERR_KERNEL, "SDPA kernel gave up on a bounded wait (stage code %d); output is not valid", code);
    return TX_OK;
}

}  // extern "C"

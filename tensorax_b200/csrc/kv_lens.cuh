// Valid keys per batch element, as a kernel parameter: a device array, or up to 32 lengths inside the parameter block
// itself.  The second form is for callers that have the lengths on the host (a serving loop, the Python layer): they
// travel with the launch instead of in a buffer of their own that is allocated, filled by a copy the host waits for,
// and freed on every call.
#pragma once
#include <cstdint>

namespace txb {

struct KvLens {
    static constexpr int kInline = 32;
    const int32_t *ptr = nullptr;      // optional device array [B]
    int32_t n_inline = 0;              // B when the lengths are in `val`
    int32_t val[kInline];

    // `all`, or the batch element's length where one was given and is smaller (a negative one counts as 0)
    __device__ __forceinline__ int limit(int b, int all) const
    {
        if (n_inline > 0) return min(all, max(val[b], 0));
        if (ptr) return min(all, max(ptr[b], 0));
        return all;
    }
};

// Longer host arrays are brought to the device by value too, a chunk per launch: a copy would read the caller's array when
// the stream gets to it -- after the call, where the array is pinned, and again at every replay, where the call was captured.
struct KvLensChunk {
    static constexpr int kMax = 960;   // with the rest of the parameters inside 4 KB
    int32_t n, val[kMax];
};

__global__ void __launch_bounds__(256) put_kv_lens_kernel(const __grid_constant__ KvLensChunk c, int32_t *__restrict__ dst)
{
    for (int i = threadIdx.x; i < c.n; i += blockDim.x) dst[i] = c.val[i];
}

}  // namespace txb

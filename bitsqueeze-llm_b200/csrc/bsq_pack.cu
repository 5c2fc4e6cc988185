// Moving the sections of a packed object between their aligned device buffers and a device-resident object (sm_100a).
//
// The reference assembles its object on the host, one cudaMemcpy per piece (src/bitsqz_llm.cu:1237-1277).  A
// device-resident object consists of up to a dozen device pieces at unpadded offsets plus the headers that the host
// knows.  As stream copies those are a dozen operations of ~2 us each whatever their size, and the object's own header,
// which depends on the error flag, needed a host round trip; here they are ONE launch:
//   * the device pieces go through 16-byte stores; where source and destination are not aligned alike, 16 bytes are put
//     together from five aligned words (the pieces are 2- or 1-byte aligned only for ragged shapes);
//   * the section headers and the object's header travel in the kernel's parameters; the error section's entry and flag
//     are dropped on the device when the error flag says so, and the whole header is zeroed when a kernel of the call has
//     reported an error (the call fails then, and nothing that could pass for an object is left in the buffer);
//   * the status words go to the caller's page-locked mirror and are cleared for the next call.
// Bound by launch latency up to a few MB, by memory above (9.7 MB of a 4096 x 4096 NF4_DQ object: 6.7 us).  Measured with
// the calls around it: compress 256 x 1024 NF4_DQ 71 -> 40 us, 4096 x 4096 114 -> 75 us; decompress 4096 x 4096, which also
// reads aligned sections where they lie, 78 -> 56 us.
#include "bsq_device.cuh"
#include "bsq_internal.hpp"

#include <cuda.h>

#include <mutex>

namespace bsq {
namespace {

// cuPointerGetAttributes from the driver, looked up once (the library links the runtime only).
typedef CUresult (*PointerAttributesFn)(unsigned, CUpointer_attribute *, void **, CUdeviceptr);
PointerAttributesFn pointer_attributes() {
    static PointerAttributesFn fn = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        void *p = nullptr;
        cudaDriverEntryPointQueryResult q = cudaDriverEntryPointSymbolNotFound;
        if (cudaGetDriverEntryPoint("cuPointerGetAttributes", &p, cudaEnableDefault, &q) == cudaSuccess && q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<PointerAttributesFn>(p);
        else
            cudaGetLastError();
    });
    return fn;
}

constexpr int kCopyThreads = 256;
constexpr unsigned kCopyUnits = 2048;                        // 16-byte units per CTA: 32 KB, eight per thread

struct CopyArgs {
    CopySegment seg[kMaxCopySegments];
    unsigned first_cta[kMaxCopySegments + 1];
    int segments;
};

// `bytes` bytes; CTA `part` of the segment takes units part * kCopyUnits .. of the 16-byte units of dst, the first CTA
// also the bytes in front of and behind them.
__device__ __forceinline__ void copy_part(const CopySegment &s, unsigned part) {
    uint8_t *dst = static_cast<uint8_t *>(s.dst);
    const uint8_t *src = static_cast<const uint8_t *>(s.src);
    uint64_t lead = (16u - (unsigned)(reinterpret_cast<uintptr_t>(dst) & 15u)) & 15u;
    if (lead > s.bytes) lead = s.bytes;
    uint64_t units = (s.bytes - lead) / 16;
    const unsigned m = (unsigned)(reinterpret_cast<uintptr_t>(src + lead) & 15u);
    if ((m & 3u) && units) --units;                          // the word behind the last unit stays inside the segment
    if (part == 0) {
        for (uint64_t i = threadIdx.x; i < lead; i += kCopyThreads) dst[i] = src[i];
        for (uint64_t i = lead + units * 16 + threadIdx.x; i < s.bytes; i += kCopyThreads) dst[i] = src[i];
    }
    const uint64_t u0 = (uint64_t)part * kCopyUnits + threadIdx.x;
    const uint8_t *from = src + lead;
    uint4 *to = reinterpret_cast<uint4 *>(dst + lead);
    uint4 v[kCopyUnits / kCopyThreads];
#pragma unroll
    for (int j = 0; j < (int)(kCopyUnits / kCopyThreads); ++j) {
        const uint64_t u = u0 + (uint64_t)j * kCopyThreads;
        if (u >= units) continue;
        if (m == 0) {
            v[j] = reinterpret_cast<const uint4 *>(from)[u];
        } else if ((m & 7u) == 0) {
            const uint2 a = reinterpret_cast<const uint2 *>(from)[2 * u], b = reinterpret_cast<const uint2 *>(from)[2 * u + 1];
            v[j] = make_uint4(a.x, a.y, b.x, b.y);
        } else {
            const unsigned *w = reinterpret_cast<const unsigned *>(from - (m & 3u)) + 4 * u;
            const unsigned sh = (m & 3u) * 8u, w0 = w[0], w1 = w[1], w2 = w[2], w3 = w[3];
            const unsigned w4 = sh ? w[4] : 0u;
            v[j] = make_uint4(__funnelshift_r(w0, w1, sh), __funnelshift_r(w1, w2, sh), __funnelshift_r(w2, w3, sh),
                              __funnelshift_r(w3, w4, sh));
        }
    }
#pragma unroll
    for (int j = 0; j < (int)(kCopyUnits / kCopyThreads); ++j) {
        const uint64_t u = u0 + (uint64_t)j * kCopyThreads;
        if (u < units) to[u] = v[j];
    }
}

__device__ __forceinline__ void copy_all(const CopyArgs &c) {
    int s = 0;
    while (s + 1 < c.segments && blockIdx.x >= c.first_cta[s + 1]) ++s;
    if (s < c.segments && blockIdx.x < c.first_cta[c.segments]) copy_part(c.seg[s], blockIdx.x - c.first_cta[s]);
}

__global__ void __launch_bounds__(kCopyThreads) copy_segments_kernel(const __grid_constant__ CopyArgs c) { copy_all(c); }

__global__ void __launch_bounds__(kCopyThreads) pack_object_kernel(const __grid_constant__ CopyArgs c, const __grid_constant__ PackHeaders h,
                                                                   unsigned *status, unsigned *mirror) {
    chain_begin();
    copy_all(c);
    if (blockIdx.x != gridDim.x - 1) return;
    // the last CTA: headers and status (its share of the pieces is the smallest)
    for (int p = 0; p < h.pieces; ++p) {
        const PackHeaders::Piece &q = h.piece[p];
        for (int i = threadIdx.x; i < q.length; i += kCopyThreads) {
            uint8_t b = h.bytes[q.at + i];
            if (q.patch && i >= q.patch_at && i < q.patch_at + 4) b = static_cast<const uint8_t *>(q.patch)[i - q.patch_at];
            q.dst[i] = b;
        }
    }
    const bool failed = status[kWordStatus] != 0, no_error = status[kWordError] == 0;
    for (int i = threadIdx.x; i < (int)sizeof(h.object); i += kCopyThreads) {
        uint8_t b = failed ? 0 : h.object[i];
        if (no_error) {
            if (i >= h.error_entry_at && i < h.error_entry_at + h.error_entry_length) b = 0;
            if (i == h.flags_at) b &= (uint8_t)~h.error_flag;
        }
        h.object_dst[i] = b;
    }
    __syncthreads();                                         // (everybody has read the two words above)
    if (threadIdx.x < kStatusWords) {
        reinterpret_cast<volatile unsigned *>(mirror)[threadIdx.x] = status[threadIdx.x];
        status[threadIdx.x] = 0;
    }
}

// One CTA: the small headers inside a device-resident payload into page-locked host memory, 64 bytes apart; clears the
// status words of the call that reads them.
__global__ void __launch_bounds__(64 * kMaxHeads) fetch_heads_kernel(const __grid_constant__ HeadList h, uint8_t *host, unsigned *status) {
    const int which = threadIdx.x >> 6, i = threadIdx.x & 63;
    if (which < h.count && i < h.length[which]) reinterpret_cast<volatile uint8_t *>(host)[which * 64 + i] = h.src[which][i];
    if (threadIdx.x < kStatusWords) status[threadIdx.x] = 0;
}

unsigned fill(CopyArgs &c, const CopySegment *segments, int count) {
    unsigned ctas = 0;
    c.segments = 0;
    for (int i = 0; i < count; ++i) {
        if (segments[i].bytes == 0) continue;
        c.seg[c.segments] = segments[i];
        c.first_cta[c.segments++] = ctas;
        ctas += (unsigned)((segments[i].bytes / 16 + kCopyUnits - 1) / kCopyUnits);
        if (segments[i].bytes < 16) ++ctas;
    }
    c.first_cta[c.segments] = ctas;
    return ctas;
}

}  // namespace

// A buffer may consist of several mappings (an allocator's expandable segments): each of them is asked for.
Reach memory_reach(const void *p, uint64_t bytes) {
    const PointerAttributesFn ask = pointer_attributes();
    int device = 0;
    if (!ask || cudaGetDevice(&device) != cudaSuccess) return Reach::kCopies;
    bool kernels = true;
    const CUdeviceptr end = reinterpret_cast<CUdeviceptr>(p) + bytes;
    CUdeviceptr at = reinterpret_cast<CUdeviceptr>(p);
    do {
        unsigned type = 0, managed = 0;
        int ordinal = -1;
        CUdeviceptr start = 0;
        size_t size = 0;
        CUpointer_attribute what[5] = {CU_POINTER_ATTRIBUTE_MEMORY_TYPE, CU_POINTER_ATTRIBUTE_IS_MANAGED, CU_POINTER_ATTRIBUTE_DEVICE_ORDINAL,
                                       CU_POINTER_ATTRIBUTE_RANGE_START_ADDR, CU_POINTER_ATTRIBUTE_RANGE_SIZE};
        void *into[5] = {&type, &managed, &ordinal, &start, &size};
        if (ask(5, what, into, at) != CUDA_SUCCESS || type == 0) return Reach::kNone;
        if (type != CU_MEMORYTYPE_DEVICE || managed || ordinal != device) kernels = false;
        if (start > at || start + size <= at) return Reach::kCopies;     // no range to go by: the copies check it themselves
        at = start + size;
    } while (at < end);
    return kernels ? Reach::kKernels : Reach::kCopies;
}

cudaError_t copy_segments(const CopySegment *segments, int count, cudaStream_t stream) {
    if (count < 0 || count > kMaxCopySegments) return cudaErrorInvalidValue;
    CopyArgs c;
    const unsigned ctas = fill(c, segments, count);
    if (ctas == 0) return cudaSuccess;
    copy_segments_kernel<<<ctas, kCopyThreads, 0, stream>>>(c);
    return cudaGetLastError();
}

cudaError_t pack_object(const CopySegment *segments, int count, const PackHeaders &headers, unsigned *d_status, unsigned *mirror,
                        cudaStream_t stream) {
    if (count < 0 || count > kMaxCopySegments) return cudaErrorInvalidValue;
    CopyArgs c;
    const unsigned ctas = fill(c, segments, count);
    return launch_chained(pack_object_kernel, ctas + 1, kCopyThreads, 0, stream, c, headers, d_status, mirror);
}

cudaError_t fetch_heads(const HeadList &heads, uint8_t *host, unsigned *d_status, cudaStream_t stream) {
    fetch_heads_kernel<<<1, 64 * kMaxHeads, 0, stream>>>(heads, host, d_status);
    return cudaGetLastError();
}

}  // namespace bsq

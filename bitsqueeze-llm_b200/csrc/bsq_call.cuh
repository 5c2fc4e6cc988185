// What the first and the last kernel of a call on a device-resident object do beside their work (sm_100a): reading sections at
// whatever address they lie, checking the headers inside the payload, reporting.
#pragma once

#include "bsq_device.cuh"
#include "bsq_internal.hpp"

namespace bsq {

__device__ __forceinline__ unsigned load_u16_any(const uint8_t *p) {
    return (reinterpret_cast<uintptr_t>(p) & 1u) ? (unsigned)p[0] | ((unsigned)p[1] << 8) : *reinterpret_cast<const uint16_t *>(p);
}
__device__ __forceinline__ float load_f32_any(const uint8_t *p) {
    if ((reinterpret_cast<uintptr_t>(p) & 3u) == 0) return *reinterpret_cast<const float *>(p);
    return __uint_as_float((unsigned)p[0] | ((unsigned)p[1] << 8) | ((unsigned)p[2] << 16) | ((unsigned)p[3] << 24));
}

// Every CTA checks for itself (a byte per thread; the headers come from the L2 after the first): nobody waits for another CTA, and
// nothing of a refused object is decoded.  All threads of the CTA call it; the result is uniform.
__device__ __forceinline__ bool heads_match(const HeadCheck &h) {
    if (h.count == 0) return true;
    int differs = 0;
    for (int t = threadIdx.x; t < h.count * kMaxHeadBytes; t += blockDim.x) {
        const int which = t / kMaxHeadBytes, i = t % kMaxHeadBytes;
        if (i >= h.length[which]) continue;
        differs |= ((h.mask[which] >> i) & 1u) && h.src[which][i] != h.want[which][i];
    }
    differs = __syncthreads_or(differs);
    // (one store that says it all: a fence between several, out to the host's memory and back, held the CTA's first warp for 2 us)
    if (blockIdx.x == 0 && threadIdx.x == 0) *reinterpret_cast<volatile unsigned *>(h.answer) = h.number + (differs ? 1u : 0u);
    return differs == 0;
}

// A kernel's report of an index out of range: into the status word, or straight into the host's mirror of it where the kernel is its
// call's last one and nothing else is reported there.  (Words that each call's last CTA handed over and cleared, found by a ticket,
// made that kernel 8 us longer; a report is never made in a call that goes well, so there is nothing to hand over then.)
__device__ __forceinline__ void report_bad_index(unsigned *status, bool host) {
    if (status == nullptr) return;
    if (host) *reinterpret_cast<volatile unsigned *>(status) = kStatusBadIndex;
    else atomicOr(status, kStatusBadIndex);
}

}  // namespace bsq

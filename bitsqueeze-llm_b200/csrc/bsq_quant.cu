// NF4 / NF4_DQ blockwise quantiser and dequantiser over a flat FP32 array (sm_100a).
//
// Replaces the reference kernels nf4_compress_kernel, compute_block_absmax_kernel,
// cub::DeviceReduce::Max, store_dq_scale_kernel, nf4_dq_compress_kernel,
// nf4_decompress_kernel and nf4_dq_decompress_kernel
// (modules/quantization_cuda/src/quantization_cuda.cu:130-341, launched from :564-663).
//
// Work decomposition: a warp takes a batch of 1024 consecutive elements = 16 blocks of 64.
// In each of 4 iterations a lane owns 8 consecutive elements (two 128-bit loads, one 32-bit
// store of 8 nibbles), so a block is 8 adjacent lanes and its absmax is 3 shuffles.  The
// per-block scale work (IEEE reciprocal, E4M3 coding) is done once per block by lanes 0..15
// and handed to the owning lanes by shuffle.  Codes come from the bucket-table encoder in
// bsq_device.cuh.  HBM-bound: 4 B read + 0.5 B + (4 or 1)/64 B written per element.
#include "bsq_call.cuh"
#include "bsq_device.cuh"
#include "bsq_internal.hpp"

#include <algorithm>
#include <mutex>

namespace bsq {
namespace {

// Scratch of nf4dq_quantize_static(): global-max word (16 bytes) + one float per 64-element
// block, for at most kStaticMaxElems elements.  Lives in the module image of every device that
// loads the library, from load to exit.
constexpr uint64_t kStaticMaxElems = 1ull << 24;
static __device__ __align__(256) unsigned char g_static_scratch[16 + (kStaticMaxElems / 64) * sizeof(float)];

constexpr int kBatch = 1024;
constexpr int kThreads = 256;

struct Lane8 {
    float v[8];
};

__device__ __forceinline__ Lane8 load8(const float *x, uint64_t e, uint64_t n, bool vec) {
    Lane8 r;
    if (vec && e + 8 <= n) {
        const float4 a = __ldcs(reinterpret_cast<const float4 *>(x + e));
        const float4 b = __ldcs(reinterpret_cast<const float4 *>(x + e) + 1);
        r.v[0] = a.x; r.v[1] = a.y; r.v[2] = a.z; r.v[3] = a.w;
        r.v[4] = b.x; r.v[5] = b.y; r.v[6] = b.z; r.v[7] = b.w;
    } else {
#pragma unroll
        for (int j = 0; j < 8; ++j) r.v[j] = (e + j < n) ? x[e + j] : 0.0f;
    }
    return r;
}

__device__ __forceinline__ float absmax8(const Lane8 &r) {
    float m = 0.0f;
#pragma unroll
    for (int j = 0; j < 8; ++j) m = fmaxf(m, fabsf(sanitize(r.v[j])));
    return m;
}

__device__ __forceinline__ float group8_max(float v) {
    v = fmaxf(v, __shfl_xor_sync(kFullMask, v, 1));
    v = fmaxf(v, __shfl_xor_sync(kFullMask, v, 2));
    v = fmaxf(v, __shfl_xor_sync(kFullMask, v, 4));
    return v;
}

// Lane l (< 16) receives the value that block l of the batch holds: block j = 4*it + g lives
// in am[it] of lanes 8g..8g+7.
__device__ __forceinline__ float gather_block_value(const float (&am)[4], int lane) {
    float s = 0.0f;
#pragma unroll
    for (int it = 0; it < 4; ++it) {
        const float t = __shfl_sync(kFullMask, am[it], (lane & 3) * 8);
        if ((lane >> 2) == it) s = t;
    }
    return s;
}

// One array of a launch, or two side by side: CTAs from `second` on take the second.
struct EncodeJob {
    const float *x;
    uint64_t n;
    bool vec;
    const float *absmax_in;
    unsigned *gmax_bits;
    float *scales_f32;
    uint8_t *scale_codes;
    float *dq_out;
    uint8_t *data;
    float *deq_out;                                           // may alias x (in-place write-back)
    unsigned *flag;
    const float *colscale;
    unsigned cols;
    unsigned *max_bits;
};
struct EncodeJobs {
    EncodeJob job[2];
    unsigned second;
};

// ---- NF4_DQ pass 1: per-block absmax (1.0 for an all-zero block) and the global maximum ----
__global__ void __launch_bounds__(kThreads) absmax_flat_kernel(const __grid_constant__ EncodeJobs jobs) {
    chain_begin();
    const int lane = threadIdx.x & 31;
    const bool other = blockIdx.x >= jobs.second;
    const EncodeJob &job = jobs.job[other];
    const float *x = job.x;
    const uint64_t n = job.n;
    const bool vec = job.vec;
    float *absmax_out = const_cast<float *>(job.absmax_in);
    const uint64_t warp = (uint64_t)(blockIdx.x - (other ? jobs.second : 0u)) * (kThreads / 32) + (threadIdx.x >> 5);
    const uint64_t nwarps = (uint64_t)(other ? gridDim.x - jobs.second : jobs.second) * (kThreads / 32);
    const uint64_t nb = (n + 63) / 64;
    float run = 0.0f;
    for (uint64_t base = warp * kBatch; base < n; base += nwarps * kBatch) {
        float am[4];
#pragma unroll
        for (int it = 0; it < 4; ++it) {
            const Lane8 r = load8(x, base + it * 256 + lane * 8, n, vec);
            am[it] = group8_max(absmax8(r));
        }
        float s = gather_block_value(am, lane);
        s = s > 0.0f ? s : 1.0f;
        const uint64_t blk = base / 64 + lane;
        if (lane < 16 && blk < nb) {
            absmax_out[blk] = s;
            run = fmaxf(run, s);
        }
    }
    run = warp_max(run);
    if (lane == 0 && run > 0.0f) atomicMax(job.gmax_bits, __float_as_uint(run));
}

// ---- encode: NF4 (DQ == false: computes its own absmax) or NF4_DQ pass 2 -----------------
// What the encoder writes beside codes and scales: nothing, the dequantised values, or what the quantiser got wrong,
// x - dequantised, with *flag |= any(|.| > FLT_EPSILON) (the reference's subtract_kernel + has_nonzero_kernel,
// src/bitsqz_llm.cu:164-184: without a pass of its own over two matrices).
enum : int { kWriteNone = 0, kWriteDeq = 1, kWriteError = 2 };
template <bool DQ, int WRITE>
__global__ void __launch_bounds__(kThreads) encode_flat_kernel(const __grid_constant__ EncodeJobs jobs) {
    chain_begin();
    bool any = false;
    unsigned largest = 0;
    const int lane = threadIdx.x & 31;
    const bool other = blockIdx.x >= jobs.second;
    const EncodeJob &job = jobs.job[other];
    const float *x = job.x;
    const uint64_t n = job.n;
    const bool vec = job.vec;
    float *scales_f32 = job.scales_f32, *deq_out = job.deq_out;
    uint8_t *scale_codes = job.scale_codes, *data = job.data;
    const uint64_t warp = (uint64_t)(blockIdx.x - (other ? jobs.second : 0u)) * (kThreads / 32) + (threadIdx.x >> 5);
    const uint64_t nwarps = (uint64_t)(other ? gridDim.x - jobs.second : jobs.second) * (kThreads / 32);
    const uint64_t nb = (n + 63) / 64;
    Nf4Lut lut;
    lut.load();
    float dq = 1.0f;
    if (DQ) {
        dq = dq_from_max(__uint_as_float(*job.gmax_bits));
        if (warp == 0 && lane == 0) *job.dq_out = dq;
    }
    for (uint64_t base = warp * kBatch; base < n; base += nwarps * kBatch) {
        Lane8 r[4];
#pragma unroll
        for (int it = 0; it < 4; ++it) r[it] = load8(x, base + it * 256 + lane * 8, n, vec);

        const uint64_t blk = base / 64 + lane;
        const bool owns_block = lane < 16 && blk < nb;
        float scale = 1.0f, blk_absmax = 0.0f;
        if (!DQ) {
            float am[4];
#pragma unroll
            for (int it = 0; it < 4; ++it) am[it] = group8_max(absmax8(r[it]));
            blk_absmax = gather_block_value(am, lane);
            scale = blk_absmax > 0.0f ? blk_absmax : 1.0f;
            if (owns_block) scales_f32[blk] = scale;
        } else {
            if (owns_block) {
                blk_absmax = job.absmax_in[blk];
                unsigned code;
                scale = dq_block_scale(blk_absmax, dq, &code);
                scale_codes[blk] = (uint8_t)code;
            }
        }
        const float inv = __fdiv_rn(1.0f, scale);
        // A scaled value leaves the encoder's exact range (|v| < 2^23) only in two corners: a DQ
        // block that fell back to scale 1.0 while holding a huge element, and a block whose scale
        // is so small (denormal) that 1/scale overflows; such blocks take the literal scan.
        const unsigned slow_blocks = __ballot_sync(kFullMask, !(__fmul_rn(blk_absmax, inv) < 8388608.0f));

#pragma unroll
        for (int it = 0; it < 4; ++it) {
            const int j = it * 4 + (lane >> 3);
            const float invb = __shfl_sync(kFullMask, inv, j);
            const uint64_t e = base + it * 256 + lane * 8;
            unsigned c[8];
#pragma unroll
            for (int q = 0; q < 8; ++q) c[q] = lut.encode(__fmul_rn(sanitize(r[it].v[q]), invb));
            if ((slow_blocks >> j) & 1u) {
#pragma unroll
                for (int q = 0; q < 8; ++q) c[q] = nf4_code_scan(__fmul_rn(sanitize(r[it].v[q]), invb));
            }
            if (WRITE != kWriteNone) {
                const float sb = __shfl_sync(kFullMask, scale, j);
                float d[8];
#pragma unroll
                for (int q = 0; q < 8; ++q) d[q] = __fmul_rn(sb, lut.decode(c[q]));
                if (WRITE == kWriteError) {
#pragma unroll
                    for (int q = 0; q < 8; ++q) {
                        d[q] = __fsub_rn(r[it].v[q], d[q]);
                        any |= e + q < n && fabsf(d[q]) > 1.1920928955078125e-07f;
                    }
                }
                if (WRITE == kWriteDeq && job.max_bits && e < n) {
                    unsigned c = job.colscale ? (unsigned)e % job.cols : 0u;   // (a factor has fewer than 2^32 elements)
#pragma unroll
                    for (int q = 0; q < 8; ++q) {
                        const float v = job.colscale ? d[q] * job.colscale[c] : d[q];
                        if (e + q < n) largest = max(largest, __float_as_uint(v) & 0x7fffffffu);
                        if (++c == job.cols) c = 0;
                    }
                }
                if (vec && e + 8 <= n) {
                    reinterpret_cast<float4 *>(deq_out + e)[0] = make_float4(d[0], d[1], d[2], d[3]);
                    reinterpret_cast<float4 *>(deq_out + e)[1] = make_float4(d[4], d[5], d[6], d[7]);
                } else {
#pragma unroll
                    for (int q = 0; q < 8; ++q)
                        if (e + q < n) deq_out[e + q] = d[q];
                }
            }
            if (e + 8 <= n) {
                const unsigned w = ((c[0] << 4) | c[1]) | (((c[2] << 4) | c[3]) << 8) | (((c[4] << 4) | c[5]) << 16) |
                                   (((c[6] << 4) | c[7]) << 24);
                if (vec) {
                    *reinterpret_cast<unsigned *>(data + e / 2) = w;
                } else {
#pragma unroll
                    for (int q = 0; q < 4; ++q) data[e / 2 + q] = (uint8_t)(w >> (8 * q));
                }
            } else if (e < n) {
#pragma unroll
                for (int q = 0; q < 8; q += 2) {
                    if (e + q < n) {
                        const unsigned lo = (e + q + 1 < n) ? c[q + 1] : 0u;   // odd tail: low nibble 0
                        data[(e + q) / 2] = (uint8_t)((c[q] << 4) | lo);
                    }
                }
            }
        }
    }
    if (WRITE == kWriteError && __any_sync(kFullMask, any) && lane == 0) atomicOr(job.flag, 1u);
    if (WRITE == kWriteDeq && job.max_bits) {
        largest = __reduce_max_sync(kFullMask, largest);
        if (lane == 0 && largest) atomicMax(job.max_bits, largest);
    }
}

// ---- decode ----------------------------------------------------------------------------------
// Row-wise top-k lists to add onto the decoded rows x cols matrix in the same pass, one after the other (idx: u16, val: f32, any
// alignment; k = 0: none).
struct TopkList {
    const uint8_t *idx, *val;
    unsigned k;
};
struct TopkLists {
    TopkList list[2];
    unsigned cols;
    unsigned *status;
    bool status_on_host;
};
// What a batch of kBatch elements needs from memory.  The first 64 entries of each list's row come with it.
struct DecodeBatch {
    unsigned w[4];
    float scale;
    unsigned c[2][2];
    float v[2][2];
};

// A warp decodes kBatch consecutive elements into shared memory, adds the lists' entries there and sends the batch out by one bulk
// store; what the next batch needs is on its way meanwhile.  scales (NF4: f32), dq_in and data may lie at any address
// (vec_in: data at a multiple of 4); out off a 16-byte boundary, and the last batch, go out by lanes.
// Bound by the bytes written (a plain fill of as many: 10.1 us) and the trip for the first batch.  4096 x 4096 NF4_DQ with a list of 41
// per row 16.9 us, without 14.9, 19 with the check of the headers; two buffers and three CTAs per SM 17.9, five and six CTAs 17.9 and
// 20.1; entries added in global memory behind the batch's own stores 17.1.  As a whole call, against a kernel that fetches the headers,
// a wait, this kernel and a copy of the status words: 56.3 -> 40.1 us; 2505 x 3085 with two lists, off its alignment, 69.1 -> 34.5.
constexpr int kDecodeCtas = 4;
constexpr size_t kDecodeSmem = (size_t)(kThreads / 32) * kBatch * sizeof(float);
template <bool DQ>
__global__ void __launch_bounds__(kThreads, kDecodeCtas)
    decode_flat_kernel(const uint8_t *__restrict__ scales_f32, const uint8_t *__restrict__ scale_codes,
                       const uint8_t *__restrict__ dq_in, const uint8_t *__restrict__ data, uint64_t n, bool vec_in, bool bulk_out,
                       float *out, const __grid_constant__ TopkLists add, const __grid_constant__ HeadCheck heads) {
    extern __shared__ __align__(128) float stage_raw[];
    const int lane = threadIdx.x & 31;
    const uint64_t warp = (uint64_t)blockIdx.x * (kThreads / 32) + (threadIdx.x >> 5);
    const uint64_t nwarps = (uint64_t)gridDim.x * (kThreads / 32);
    const uint64_t nb = (n + 63) / 64;
    float *const stage = stage_raw + (threadIdx.x >> 5) * kBatch;
    Nf4Lut lut;
    lut.load();
    float dq = 1.0f;
    if (DQ) {
        dq = load_f32_any(dq_in);
        if (dq == 0.0f || !isfinite(dq)) dq = 1.0f;   // quantization_cuda.cu:325-328
    }
    const bool listed = add.list[0].k + add.list[1].k != 0, small = n <= 0xFFFFFFFFull;
    const auto row_of = [&](uint64_t e) { return small ? (uint64_t)((unsigned)e / add.cols) : e / add.cols; };
    auto fetch = [&](uint64_t base, DecodeBatch &b) {
        if (base >= n) return;
#pragma unroll
        for (int it = 0; it < 4; ++it) {
            const uint64_t e = base + it * 256 + lane * 8;
            if (vec_in && e + 8 <= n) {
                b.w[it] = __ldcs(reinterpret_cast<const unsigned *>(data + e / 2));
            } else {
                b.w[it] = 0;
#pragma unroll
                for (int q = 0; q < 4; ++q)
                    if (e + 2 * q < n) b.w[it] |= (unsigned)data[e / 2 + q] << (8 * q);
            }
        }
        const uint64_t blk = base / 64 + lane;
        b.scale = 1.0f;
        if (lane < 16 && blk < nb) {
            b.scale = DQ ? __fmul_rn(dq, e4m3_decode(scale_codes[blk])) : load_f32_any(scales_f32 + 4 * blk);
            if (b.scale == 0.0f || !isfinite(b.scale)) b.scale = 1.0f;
        }
        if (!listed) return;
        const uint64_t r = row_of(base);
#pragma unroll
        for (int l = 0; l < 2; ++l) {
            const TopkList t = add.list[l];
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                const unsigned j = lane + 32 * u;
                if (j < t.k) {
                    b.c[l][u] = load_u16_any(t.idx + 2 * (r * t.k + j));
                    b.v[l][u] = load_f32_any(t.val + 4 * (r * t.k + j));
                }
            }
        }
    };
    DecodeBatch now, next;
    fetch(warp * kBatch, now);                                // (all inside the object, whatever its headers say)
    if (!heads_match(heads)) n = 0;                           // (uniform over the CTA)
    for (uint64_t base = warp * kBatch; base < n; base += nwarps * kBatch) {
        fetch(base + nwarps * kBatch, next);
        if (lane == 0) bulk_wait_read_all();                  // the batch before has left the buffer
        __syncwarp();
#pragma unroll
        for (int it = 0; it < 4; ++it) {
            const float sb = __shfl_sync(kFullMask, now.scale, it * 4 + (lane >> 3));
            float d[8];
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const unsigned byte = (now.w[it] >> (8 * q)) & 0xFFu;
                d[2 * q] = __fmul_rn(sb, lut.decode(byte >> 4));
                d[2 * q + 1] = __fmul_rn(sb, lut.decode(byte & 0xFu));
            }
            float4 *to = reinterpret_cast<float4 *>(stage + it * 256 + lane * 8);
            to[0] = make_float4(d[0], d[1], d[2], d[3]);
            to[1] = make_float4(d[4], d[5], d[6], d[7]);
        }
        __syncwarp();
        const uint64_t end = base + kBatch <= n ? base + kBatch : n;
        if (listed) {
            // dense[row, idx] += value (topk_cuda.cuh:83-86) for the entries that fall into this batch: its row or rows, in full
            const uint64_t r0 = row_of(base), r1 = row_of(end - 1);
#pragma unroll
            for (int l = 0; l < 2; ++l) {
                const TopkList t = add.list[l];
                if (t.k == 0) continue;
                // at: where the entry's row starts, counted from the batch's first element (modulo 2^32)
                auto put = [&](unsigned at, unsigned c, float v) {
                    if (c >= add.cols) {
                        report_bad_index(add.status, add.status_on_host);
                    } else if (at + c < (unsigned)(end - base)) {
                        stage[at + c] += v;
                    }
                };
                unsigned at = (unsigned)(r0 * add.cols - base);
#pragma unroll
                for (int u = 0; u < 2; ++u)
                    if (lane + 32 * u < t.k) put(at, now.c[l][u], now.v[l][u]);
                for (uint64_t r = r0; r <= r1; ++r, at += add.cols)
                    for (unsigned j = lane + (r == r0 ? 64u : 0u); j < t.k; j += 32)
                        put(at, load_u16_any(t.idx + 2 * (r * t.k + j)), load_f32_any(t.val + 4 * (r * t.k + j)));
                __syncwarp();
            }
        }
        if (bulk_out && end - base == kBatch) {
            fence_proxy_async_smem();
            __syncwarp();
            if (lane == 0) {
                bulk_s2g(out + base, stage, kBatch * sizeof(float));
                bulk_commit();
            }
        } else {
            for (unsigned i = lane; i < (unsigned)(end - base); i += 32) out[base + i] = stage[i];
            __syncwarp();
        }
        now = next;
    }
    if (lane == 0) bulk_wait_all();
}

// ---- the factors of a low-rank object --------------------------------------------------------------
struct FactorArgs {
    SectionSource f[2];                                       // U, V
    float *out[2];
    unsigned *max_bits[2];
    const uint8_t *s;
    float *s_out;
    unsigned rank, first_cta_v;
};
constexpr unsigned kSharedS = 1024;                          // singular values kept in shared memory
// U, V and S out of an object, and the two maxima that the reconstruction's scales come from.  Bound by latency (4096 x 14336 at rank 256: 3 MB
// of codes in, 19 MB out, 9.8 us; 7.2 to 7.6 us where there is next to nothing to do), so it is one launch: with the split of both operands
// behind it 18 us to the product, where a fetch of the headers and a wait, two decoding kernels, a copy of S, two memsets, two passes for the
// maxima and two for the split took 60.  Whole decompress calls of that shape 209 -> 171 us.
__global__ void __launch_bounds__(kThreads) open_factors_kernel(const __grid_constant__ FactorArgs a, const __grid_constant__ HeadCheck heads) {
    __shared__ float s_s[kSharedS];
    const int lane = threadIdx.x & 31, which = blockIdx.x >= a.first_cta_v;
    const unsigned first = which ? a.first_cta_v : 0u, ctas = which ? gridDim.x - a.first_cta_v : a.first_cta_v;
    const SectionSource &f = a.f[which];
    const uint64_t n = f.n, nb = (n + 63) / 64;
    const bool coded = f.scales != nullptr, coded_dq = f.dq != nullptr;
    const bool words = (reinterpret_cast<uintptr_t>(f.data) & 3u) == 0, pairs = (reinterpret_cast<uintptr_t>(f.data) & 7u) == 0;
    Nf4Lut lut;
    lut.load();
    float dq = 1.0f;
    if (coded_dq) {
        dq = load_f32_any(f.dq);
        if (dq == 0.0f || !isfinite(dq)) dq = 1.0f;           // as decode_flat_kernel
    }
    struct Coded {
        unsigned w[4];
        float scale;
    };
    const auto fetch = [&](uint64_t base, Coded &c) {
        c.scale = 1.0f;
        if (!coded || base >= n) return;
        const uint64_t blk = base / 64 + lane;
#pragma unroll
        for (int it = 0; it < 4; ++it) {
            const uint64_t e = base + it * 256 + lane * 8;
            c.w[it] = 0u;
            if (words && e + 8 <= n) {
                c.w[it] = *reinterpret_cast<const unsigned *>(f.data + e / 2);
            } else {
#pragma unroll
                for (int q = 0; q < 4; ++q)
                    if (e + 2 * q < n) c.w[it] |= (unsigned)f.data[e / 2 + q] << (8 * q);
            }
        }
        if (lane < 16 && blk < nb) {
            c.scale = coded_dq ? __fmul_rn(dq, e4m3_decode(f.scales[blk])) : load_f32_any(f.scales + 4 * blk);
            if (c.scale == 0.0f || !isfinite(c.scale)) c.scale = 1.0f;
        }
    };
    // what the CTA reads first is on its way while the headers are checked (all inside the object, whatever its headers say)
    const uint64_t step = (uint64_t)ctas * (kThreads / 32) * kBatch;
    uint64_t base = ((uint64_t)(blockIdx.x - first) * (kThreads / 32) + (threadIdx.x >> 5)) * kBatch;
    Coded now, next;
    fetch(base, now);
    if (!which)
        for (unsigned t = threadIdx.x; t < a.rank && t < kSharedS; t += kThreads) s_s[t] = load_f32_any(a.s + 4 * t);
    if (!heads_match(heads)) return;
    if (which && blockIdx.x == first)
        for (unsigned t = threadIdx.x; t < a.rank; t += kThreads) a.s_out[t] = load_f32_any(a.s + 4ull * t);
    __syncthreads();
    unsigned largest = 0;
    for (; base < n; base += step) {
        fetch(base + step, next);
#pragma unroll
        for (int it = 0; it < 4; ++it) {
            const uint64_t e = base + it * 256 + lane * 8;
            float d[8];
            if (coded) {
                const float sb = __shfl_sync(kFullMask, now.scale, it * 4 + (lane >> 3));
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    const unsigned byte = (now.w[it] >> (8 * q)) & 0xFFu;
                    d[2 * q] = __fmul_rn(sb, lut.decode(byte >> 4));
                    d[2 * q + 1] = __fmul_rn(sb, lut.decode(byte & 0xFu));
                }
            } else if (pairs && e + 8 <= n) {
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    const float2 v = reinterpret_cast<const float2 *>(f.data + 4 * e)[q];
                    d[2 * q] = v.x;
                    d[2 * q + 1] = v.y;
                }
            } else {
#pragma unroll
                for (int q = 0; q < 8; ++q) d[q] = e + q < n ? load_f32_any(f.data + 4 * (e + q)) : 0.0f;
            }
            if (e + 8 <= n) {
                float4 *to = reinterpret_cast<float4 *>(a.out[which] + e);
                to[0] = make_float4(d[0], d[1], d[2], d[3]);
                to[1] = make_float4(d[4], d[5], d[6], d[7]);
            } else {
#pragma unroll
                for (int q = 0; q < 8; ++q)
                    if (e + q < n) a.out[which][e + q] = d[q];
            }
            unsigned c = which ? 0u : (unsigned)e % a.rank;   // (a factor has fewer than 2^32 elements)
#pragma unroll
            for (int q = 0; q < 8; ++q) {
                if (!which) {
                    d[q] *= a.rank <= kSharedS ? s_s[c] : load_f32_any(a.s + 4ull * c);
                    if (++c == a.rank) c = 0;
                }
                if (e + q < n) largest = max(largest, __float_as_uint(d[q]) & 0x7fffffffu);
            }
        }
        now = next;
    }
    largest = __reduce_max_sync(kFullMask, largest);
    if (lane == 0 && largest) atomicMax(a.max_bits[which], largest);
}

inline const uint8_t *bytes(const void *p) { return static_cast<const uint8_t *>(p); }
inline bool aligned(const void *p, size_t a) { return (reinterpret_cast<uintptr_t>(p) % a) == 0; }

inline int grid_for(uint64_t n, int sm_count) {
    const uint64_t batches = (n + kBatch - 1) / kBatch;
    const uint64_t blocks = (batches + (kThreads / 32) - 1) / (kThreads / 32);
    const uint64_t cap = (uint64_t)sm_count * 8;      // 8 resident CTAs of 256 threads per SM
    return (int)(blocks < cap ? (blocks ? blocks : 1) : cap);
}

}  // namespace

// Both arrays of `jobs` (the second possibly empty) in one launch per pass.
static cudaError_t launch_encode(bool dq, EncodeJobs &jobs, int sm_count, cudaStream_t stream) {
    unsigned grid = 0;
    for (int i = 0; i < 2; ++i) {
        EncodeJob &j = jobs.job[i];
        if (i == 1) jobs.second = grid;
        if (j.n == 0) continue;
        j.vec = aligned(j.x, 16) && aligned(j.data, 4) && (!j.deq_out || aligned(j.deq_out, 16));
        grid += (unsigned)grid_for(j.n, sm_count);
    }
    if (dq) {
        const cudaError_t err = launch_chained(absmax_flat_kernel, grid, kThreads, 0, stream, jobs);
        if (err != cudaSuccess) return err;
    }
    const EncodeJob &j = jobs.job[0];
    if (j.deq_out && j.flag)
        return dq ? launch_chained(encode_flat_kernel<true, kWriteError>, grid, kThreads, 0, stream, jobs)
                  : launch_chained(encode_flat_kernel<false, kWriteError>, grid, kThreads, 0, stream, jobs);
    if (j.deq_out)
        return dq ? launch_chained(encode_flat_kernel<true, kWriteDeq>, grid, kThreads, 0, stream, jobs)
                  : launch_chained(encode_flat_kernel<false, kWriteDeq>, grid, kThreads, 0, stream, jobs);
    return dq ? launch_chained(encode_flat_kernel<true, kWriteNone>, grid, kThreads, 0, stream, jobs)
              : launch_chained(encode_flat_kernel<false, kWriteNone>, grid, kThreads, 0, stream, jobs);
}

cudaError_t nf4_quantize(const float *d_x, uint64_t n, float *d_scales, uint8_t *d_data, float *d_deq_out, int sm_count,
                         cudaStream_t stream, unsigned *d_error_flag) {
    EncodeJobs jobs{};
    EncodeJob &j = jobs.job[0];
    j.x = d_x;
    j.n = n;
    j.scales_f32 = d_scales;
    j.data = d_data;
    j.deq_out = d_deq_out;
    j.flag = d_error_flag;
    return launch_encode(false, jobs, sm_count, stream);
}

size_t nf4dq_scratch_bytes(uint64_t n) { return (size_t)((n + 63) / 64) * sizeof(float) + 16; }

cudaError_t nf4dq_quantize(const float *d_x, uint64_t n, float *d_dq, uint8_t *d_scale_codes, uint8_t *d_data,
                           float *d_deq_out, void *d_scratch, int sm_count, cudaStream_t stream, unsigned *d_error_flag, unsigned *d_gmax) {
    // scratch layout: [0,16) global-max word (+ padding), then one float per block
    unsigned *gmax = d_gmax ? d_gmax : static_cast<unsigned *>(d_scratch);
    if (!d_gmax) {
        const cudaError_t err = cudaMemsetAsync(gmax, 0, 4, stream);
        if (err != cudaSuccess) return err;
    }
    EncodeJobs jobs{};
    EncodeJob &j = jobs.job[0];
    j.x = d_x;
    j.n = n;
    j.absmax_in = reinterpret_cast<float *>(static_cast<uint8_t *>(d_scratch) + 16);
    j.gmax_bits = gmax;
    j.scale_codes = d_scale_codes;
    j.dq_out = d_dq;
    j.data = d_data;
    j.deq_out = d_deq_out;
    j.flag = d_error_flag;
    return launch_encode(true, jobs, sm_count, stream);
}

cudaError_t quantize_pair(int method, const QuantTarget &a, const QuantTarget &b, void *d_scratch, int sm_count, cudaStream_t stream) {
    const bool dq = method == 10;
    EncodeJobs jobs{};
    uint8_t *room = static_cast<uint8_t *>(d_scratch);
    for (int i = 0; i < 2; ++i) {
        const QuantTarget &t = i ? b : a;
        EncodeJob &j = jobs.job[i];
        if (!t.x || !t.n || !t.data || (dq ? !t.dq || !t.scale_codes || !t.gmax || !d_scratch : !t.scales) || (t.deq == nullptr) != (a.deq == nullptr))
            return cudaErrorInvalidValue;
        j.x = t.x;
        j.n = t.n;
        j.scales_f32 = t.scales;
        j.scale_codes = t.scale_codes;
        j.dq_out = t.dq;
        j.data = t.data;
        j.deq_out = t.deq;
        j.gmax_bits = t.gmax;
        j.colscale = t.colscale;
        j.cols = t.cols;
        j.max_bits = t.max_bits;
        if (dq) {
            j.absmax_in = reinterpret_cast<float *>(room + 16);
            room += nf4dq_scratch_bytes(t.n);
        }
    }
    return launch_encode(dq, jobs, sm_count, stream);
}

uint64_t nf4dq_static_max_elements() { return kStaticMaxElems; }

// NF4_DQ quantiser that allocates nothing: its scratch is the file-scope array above.  The device
// address of that array is looked up once per device (cudaGetSymbolAddress, with that device
// current) the first time the function runs there; that first call should therefore come before
// any stream capture.  All calls on a device share the array: work from two calls that overlaps
// on the GPU (different streams) races on it.  Stale contents are harmless: the global-max word is
// cleared at the start of every call and every block maximum that is read was written by the same call.
cudaError_t nf4dq_quantize_static(const float *d_x, uint64_t n, float *d_dq, uint8_t *d_scale_codes, uint8_t *d_data,
                                  int sm_count, cudaStream_t stream) {
    static std::mutex mu;
    static void *scratch_of_device[64] = {};
    if (n == 0 || n > kStaticMaxElems) return cudaErrorInvalidValue;
    int dev = 0;
    cudaError_t err = cudaGetDevice(&dev);
    if (err != cudaSuccess) return err;
    if (dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
    void *scratch = nullptr;
    {
        std::lock_guard<std::mutex> g(mu);
        if (!scratch_of_device[dev]) {
            void *p = nullptr;
            err = cudaGetSymbolAddress(&p, g_static_scratch);     // host code must not pass the symbol itself
            if (err != cudaSuccess) return err;
            scratch_of_device[dev] = p;
        }
        scratch = scratch_of_device[dev];
    }
    return nf4dq_quantize(d_x, n, d_dq, d_scale_codes, d_data, nullptr, scratch, sm_count, stream);
}

static cudaError_t launch_decode(const SectionSource &q, const TopkLists &add, float *d_out, const HeadCheck &heads, int sm_count,
                                 cudaStream_t stream) {
    const bool vec_in = aligned(q.data, 4), bulk_out = aligned(d_out, 16);
    const auto go = [&](auto kernel, const uint8_t *f32, const uint8_t *codes) {
        const cudaError_t err = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kDecodeSmem);
        if (err != cudaSuccess) return err;
        const uint64_t ctas = (q.n + (uint64_t)kBatch * (kThreads / 32) - 1) / ((uint64_t)kBatch * (kThreads / 32));
        const uint64_t most = (uint64_t)sm_count * kDecodeCtas;
        kernel<<<(unsigned)(ctas < most ? ctas : most), kThreads, kDecodeSmem, stream>>>(f32, codes, q.dq, q.data, q.n, vec_in, bulk_out, d_out, add, heads);
        return cudaGetLastError();
    };
    return q.dq ? go(decode_flat_kernel<true>, nullptr, q.scales) : go(decode_flat_kernel<false>, q.scales, nullptr);
}

cudaError_t nf4_dequantize(const float *d_scales, const uint8_t *d_data, uint64_t n, float *d_out, int sm_count,
                           cudaStream_t stream) {
    return launch_decode(SectionSource{bytes(d_scales), nullptr, d_data, n}, TopkLists{}, d_out, HeadCheck{}, sm_count, stream);
}

cudaError_t nf4dq_dequantize(const float *d_dq, const uint8_t *d_scale_codes, const uint8_t *d_data, uint64_t n,
                             float *d_out, int sm_count, cudaStream_t stream) {
    return launch_decode(SectionSource{d_scale_codes, bytes(d_dq), d_data, n}, TopkLists{}, d_out, HeadCheck{}, sm_count, stream);
}

// Dequantise a rows x cols matrix and add its row-wise top-k list in the same pass (quantization_cuda_decompress
// followed by topk_apply in the reference, src/bitsqz_llm.cu:1304-1393).  d_scales: FP32 block scales (NF4) or null;
// d_dq + d_scale_codes: NF4_DQ or null.
cudaError_t nf4_dequantize_add_topk(const float *d_scales, const float *d_dq, const uint8_t *d_scale_codes, const uint8_t *d_data,
                                    uint32_t rows, uint32_t cols, const uint16_t *d_idx, const float *d_val, uint32_t k,
                                    float *d_out, unsigned *d_status, int sm_count, cudaStream_t stream) {
    if (!d_data || !d_out || !d_idx || !d_val || rows == 0 || cols == 0 || k == 0) return cudaErrorInvalidValue;
    if ((d_scales != nullptr) == (d_dq != nullptr && d_scale_codes != nullptr)) return cudaErrorInvalidValue;
    const SectionSource q{d_scales ? bytes(d_scales) : d_scale_codes, d_scales ? nullptr : bytes(d_dq), d_data, (uint64_t)rows * cols};
    return launch_decode(q, TopkLists{{{bytes(d_idx), bytes(d_val), k}, {}}, cols, d_status, false}, d_out, HeadCheck{}, sm_count, stream);
}

// In the pass a warp looks through the whole lists of a row for each batch that it decodes there, 32 entries a trip of 0.25 to 0.4 us; behind it the
// lists cost a launch and a wait, of which 6 us show, and about 8 us for a million entries, each read once.  us a call, in the pass / behind
// it: 8 x 9216 with 68 + 14 entries a row 22.6 / 29.7, 384 x 1792 with 46 + 270 27.6 / 33.1, 4928 x 768 with one list of 489 31.0 / 47.8, 1856 x 4608 with
// one of 1781 71 / 95; on the other side 64 x 3136 with 343 + 1040 41.7 / 28.7, 158 x 14175 with one of 1113 51.0 / 27.8, 2897 x 5492 with one of 446 73 / 46,
// 69 x 11924 with 4664 + 3463 143 / 37, 3673 x 5182 with 1900 + 2380 468 / 254.  Of 400 shapes the choice costs 1.3 % in the mean.
bool decode_lists_apart(uint32_t rows, uint32_t cols, uint32_t k0, uint32_t k1, int sm_count) {
    const uint64_t batches = ((uint64_t)rows * cols + kBatch - 1) / kBatch, warps = (uint64_t)sm_count * kDecodeCtas * (kThreads / 32);
    const double per_warp = batches > warps ? (double)batches / warps : 1.0;
    const double rows_of_batch = cols < kBatch ? std::min<uint32_t>(rows, (kBatch - 1) / cols + 2) : 1.0 + (double)(kBatch - 1) / cols;
    const double trips = ((k0 + 31) / 32 + (k1 + 31) / 32) * rows_of_batch * per_warp;
    return 0.25 * trips > 6.0 + 8.0e-6 * rows * ((double)k0 + k1);
}

cudaError_t decode_matrix(const SectionSource &q, uint32_t rows, uint32_t cols, const ListSource &first, const ListSource &second, float *d_out,
                          unsigned *mirror, const HeadCheck &heads, int sm_count, cudaStream_t stream) {
    if (!q.scales || !q.data || !d_out || q.n != (uint64_t)rows * cols || q.n == 0) return cudaErrorInvalidValue;
    const TopkLists add{{{first.idx, first.val, first.k}, {second.idx, second.val, second.k}}, cols, mirror, true};
    return launch_decode(q, add, d_out, heads, sm_count, stream);
}

cudaError_t open_factors(const SectionSource &u, const SectionSource &v, const uint8_t *s, uint32_t rank, float *d_u, float *d_v, float *d_s,
                         unsigned *d_max_us, unsigned *d_max_v, const HeadCheck &heads, int sm_count, cudaStream_t stream) {
    if (!u.n || !v.n || !u.data || !v.data || !s || !rank || !aligned(d_u, 16) || !aligned(d_v, 16)) return cudaErrorInvalidValue;
    FactorArgs a{};
    a.f[0] = u; a.f[1] = v;
    a.out[0] = d_u; a.out[1] = d_v;
    a.max_bits[0] = d_max_us; a.max_bits[1] = d_max_v;
    a.s = s;
    a.s_out = d_s;
    a.rank = rank;
    // a warp per batch up to four CTAs per SM for each factor: all of them are in flight at once
    const auto ctas = [&](uint64_t n) {
        const uint64_t c = (n + kBatch * (kThreads / 32) - 1) / (kBatch * (kThreads / 32));
        return (unsigned)(c < (uint64_t)sm_count * 4 ? c : (uint64_t)sm_count * 4);
    };
    a.first_cta_v = ctas(u.n);
    open_factors_kernel<<<a.first_cta_v + ctas(v.n), kThreads, 0, stream>>>(a, heads);
    return cudaGetLastError();
}

}  // namespace bsq

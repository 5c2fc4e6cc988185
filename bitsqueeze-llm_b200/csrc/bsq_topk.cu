// Per-row ordered top-k of |x| (outlier separation and error-correction extraction), the
// scatter-add that undoes it, and the residual/any-nonzero helper (sm_100a).
//
// Replaces build_sort_inputs_kernel + cub::DeviceSegmentedRadixSort::SortPairsDescending +
// gather_topk_kernel + zero_selected_entries_kernel and scatter_add_topk_kernel
// (modules/topk_cuda/src/topk_cuda_utils.cuh:51-149,254-295; entry points
// modules/topk_cuda/src/topk_cuda.cu:186-233), and subtract_kernel / has_nonzero_kernel
// (src/bitsqz_llm.cu:164-184).  The reference sorts every row completely to keep ~1 % of it;
// here a row is read once from HBM into shared memory by a bulk (TMA) copy, selected and
// sorted there (bsq_topk.cuh), and only the k pairs -- and, for separation, the row with the
// selected entries zeroed -- are written back.  HBM-bound: 4 B read per element, 6k B written
// per row (+ 4 B per element when the zeroed copy is wanted).
#include "bsq_call.cuh"
#include "bsq_internal.hpp"
#include "bsq_rowgroup.cuh"
#include "bsq_topk.cuh"

#include <math.h>

namespace bsq {
namespace {

// ---- rows that fit shared memory, k <= kCandCap (ragged_rows_fit for rows off 16 bytes) --------
// One group of G warps per row (bsq_rowgroup.cuh); a CTA holds several groups, rows are dealt out
// round-robin over all groups of the grid.  kBulk: 16-byte aligned rows, which a bulk copy moves; other rows (cols not a
// multiple of 4, or a matrix that starts off a 16-byte boundary) are moved by the lanes, four bytes at a time, eight loads
// in flight per lane: 16 us against 49 us of the generic kernel's six passes over the row for 1501 x 3001, k = 30.
template <int G, bool kBulk>
__global__ void __launch_bounds__(512)
    topk_rows_group_kernel(const float *in, float *residual, unsigned rows, unsigned cols, unsigned k,
                           uint16_t *__restrict__ out_idx, float *__restrict__ out_val, unsigned *status, unsigned group_bytes,
                           unsigned ctl_off, unsigned *bound) {
    chain_begin();
    extern __shared__ __align__(128) unsigned char smem_raw[];
    const RowGroup<G> g;
    unsigned char *base = smem_raw + (size_t)g.gid * group_bytes;
    float *row = reinterpret_cast<float *>(base);
    GroupCtl &c = *reinterpret_cast<GroupCtl *>(base + ctl_off);
    uint64_t *bar = reinterpret_cast<uint64_t *>(&c.bar);
    const unsigned bytes = cols * 4u;
    const unsigned groups_per_cta = blockDim.x / RowGroup<G>::L;
    if (g.lane == 0) {
        mbar_init(bar, 1);
        mbar_fence_init();
        c.wait_failed = 0;
    }
    g.sync();
    unsigned phase = 0;
    float hint = 0.0f;
    const unsigned row_step = gridDim.x * groups_per_cta;
    bool next_loading = false;                               // uniform over the group: the copy of row r is already on its way
    for (unsigned r = blockIdx.x * groups_per_cta + g.gid; r < rows; r += row_step) {
        if (!kBulk) {
            const float *src = in + (size_t)r * cols;
            constexpr unsigned L = RowGroup<G>::L;
            unsigned i = g.lane;
            for (; i + 7 * L < cols; i += 8 * L) {
                float v[8];
#pragma unroll
                for (unsigned u = 0; u < 8; ++u) v[u] = src[i + u * L];
#pragma unroll
                for (unsigned u = 0; u < 8; ++u) row[i + u * L] = v[u];
            }
            for (; i < cols; i += L) row[i] = src[i];
            if (g.lane < ((4u - cols % 4u) & 3u)) row[cols + g.lane] = 0.0f;
        } else if (g.lane == 0 && !next_loading) {
            mbar_expect_tx(bar, bytes);
            bulk_g2s(row, in + (size_t)r * cols, bytes, bar);
        }
        next_loading = false;
        // the outcome of the wait must be the same for every lane of the group (they meet at group barriers below):
        // a lane whose wait ran out says so, and all lanes read the same flag after a group barrier
        if (kBulk && !mbar_wait_bounded(bar, phase, status)) c.wait_failed = 1;
        g.sync();
        if (c.wait_failed) break;
        phase ^= 1u;
        bool special = false;
        // Extraction only (no zeroed copy wanted): once the candidates and their values are out of the row, the next
        // row's copy starts into the same buffer while this row's candidates are still ranked and written out.
        auto row_free = [&]() {
            if (kBulk && r + row_step < rows) {
                fence_proxy_async_smem();
                g.sync();
                if (g.lane == 0) {
                    mbar_expect_tx(bar, bytes);
                    bulk_g2s(row, in + (size_t)(r + row_step) * cols, bytes, bar);
                }
                next_loading = true;
            }
        };
        hint = group_topk_row<G>(g, c, row, cols, k, out_idx + (size_t)r * k, out_val + (size_t)r * k, residual != nullptr,
                                 hint, &special, row_free);
        if (bound && g.lane == 0) atomicMax(bound, c.kth_bits);          // (published before the function's last group sync)
        fence_proxy_async_smem();
        g.sync();
        if (!kBulk) {
            if (residual != nullptr)
                for (unsigned i = g.lane; i < cols; i += RowGroup<G>::L) residual[(size_t)r * cols + i] = row[i];
        } else if (residual != nullptr && g.lane == 0) {
            bulk_s2g(residual + (size_t)r * cols, row, bytes);
            bulk_commit();
            bulk_wait_read_all();
        }
        g.sync();
    }
    if (kBulk && g.lane == 0) bulk_wait_all();
}

// ---- any shape: row stays in global memory (L2), k up to cols -----------------------------------
constexpr int kGenericThreads = 256;
constexpr int kGenericSortCap = 2048;

struct GenericSmem {
    TopkScratch s;
    unsigned long long list[kGenericSortCap];
};

// CTA-wide bitonic sort (descending) of n2 (power of two, <= kGenericSortCap) composites.
__device__ void block_bitonic_desc(unsigned long long *a, unsigned n2) {
    for (unsigned size = 2; size <= n2; size <<= 1) {
        for (unsigned stride = size >> 1; stride > 0; stride >>= 1) {
            __syncthreads();
            for (unsigned t = threadIdx.x; t < n2 / 2; t += blockDim.x) {
                const unsigned i = 2 * t - (t & (stride - 1));      // lower index of the pair
                const unsigned j = i + stride;
                const bool desc = (i & size) == 0;
                const unsigned long long x = a[i], y = a[j];
                if (desc ? (x < y) : (x > y)) { a[i] = y; a[j] = x; }
            }
        }
    }
    __syncthreads();
}

__global__ void __launch_bounds__(kGenericThreads)
    topk_rows_generic_kernel(const float *in, float *residual, unsigned rows, unsigned cols, unsigned k,
                             uint16_t *__restrict__ out_idx, float *__restrict__ out_val) {
    __shared__ GenericSmem g;
    TopkScratch &s = g.s;
    const int tid = threadIdx.x;
    for (unsigned r = blockIdx.x; r < rows; r += gridDim.x) {
        const float *row = in + (size_t)r * cols;
        uint16_t *oi = out_idx + (size_t)r * k;
        float *ov = out_val + (size_t)r * k;
        // radix select over the 48-bit composite, most significant byte first
        unsigned long long prefix = 0;
        unsigned need = k;
        for (int pass = 0; pass < 6; ++pass) {
            const int shift = 40 - 8 * pass;
            for (int i = tid; i < 256; i += kGenericThreads) s.hist[i] = 0;
            __syncthreads();
            for (unsigned c = tid; c < cols; c += kGenericThreads) {
                const unsigned long long comp = topk_composite(row[c], c);
                if (pass == 0 || (comp >> (shift + 8)) == (prefix >> (shift + 8)))
                    atomicAdd(&s.hist[(unsigned)(comp >> shift) & 0xFFu], 1u);
            }
            __syncthreads();
            if (tid < 32) hist_select_warp(s, need);
            __syncthreads();
            prefix |= (unsigned long long)s.sel_bin << shift;
            need = s.sel_need;
        }
        if (k <= kGenericSortCap) {
            unsigned n2 = 2;
            while (n2 < k) n2 <<= 1;
            for (unsigned i = tid; i < n2; i += kGenericThreads) g.list[i] = 0ull;
            if (tid == 0) s.count = 0;
            __syncthreads();
            for (unsigned c = tid; c < cols; c += kGenericThreads) {
                const unsigned long long comp = topk_composite(row[c], c);
                if (comp >= prefix) {
                    const unsigned pos = atomicAdd(&s.count, 1u);
                    if (pos < kGenericSortCap) g.list[pos] = comp;
                }
            }
            block_bitonic_desc(g.list, n2);
            for (unsigned j = tid; j < k; j += kGenericThreads) {
                const unsigned col = 0xFFFFu - (unsigned)(g.list[j] & 0xFFFFull);
                oi[j] = (uint16_t)col;
                ov[j] = row[col];
            }
        } else {
            // very large k: rank every selected element by counting the composites above it
            for (unsigned c = tid; c < cols; c += kGenericThreads) {
                const unsigned long long comp = topk_composite(row[c], c);
                if (comp < prefix) continue;
                unsigned rank = 0;
                for (unsigned d = 0; d < cols; ++d) rank += topk_composite(row[d], d) > comp ? 1u : 0u;
                oi[rank] = (uint16_t)c;
                ov[rank] = row[c];
            }
        }
        __syncthreads();
        if (residual != nullptr) {
            float *dst = residual + (size_t)r * cols;
            if (dst != row) {
                for (unsigned c = tid; c < cols; c += kGenericThreads) dst[c] = row[c];
                __syncthreads();
            }
            for (unsigned j = tid; j < k; j += kGenericThreads) dst[oi[j]] = 0.0f;
        }
        __syncthreads();
    }
}

// ---- scatter-add ----------------------------------------------------------------------------------
// Lists may lie at any address.  The last kernel of a decompress call also takes the words of its earlier kernels: what they reported goes
// to the host's mirror, all are cleared (the one report that this kernel can make goes there directly).
struct ApplyReport {
    unsigned *status;                                        // nullable; device word, or the mirror itself (on_host)
    bool on_host;
    unsigned *words;                                         // nullable: this is not a call's last kernel
};
__device__ __forceinline__ void end_call(const ApplyReport &r) {
    if (r.words == nullptr || blockIdx.x != 0 || threadIdx.x >= kStatusWords) return;
    const unsigned w = r.words[threadIdx.x];
    if (threadIdx.x == kWordStatus && w) *reinterpret_cast<volatile unsigned *>(r.status) = w;
    r.words[threadIdx.x] = 0;
}
__global__ void __launch_bounds__(32) end_call_kernel(ApplyReport report) {
    chain_begin();
    end_call(report);
}
__global__ void topk_apply_kernel(ListSource list, unsigned rows, unsigned cols, float *dense, ApplyReport report) {
    chain_begin();
    end_call(report);
    const unsigned k = list.k;
    const size_t total = (size_t)rows * k;
    for (size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x; e < total; e += (size_t)gridDim.x * blockDim.x) {
        const unsigned r = (unsigned)(e / k);
        const unsigned c = load_u16_any(list.idx + 2 * e);
        if (c < cols) dense[(size_t)r * cols + c] += load_f32_any(list.val + 4 * e);
        else report_bad_index(report.status, report.on_host);
    }
}

// Two lists of the same rows, the first added before the second (the reference applies its error list, then its outliers,
// src/bitsqz_llm.cu:1372-1387): one warp per row, so that the order holds without a launch between the lists and the row's
// sectors are fetched while everything about both lists is.  Four entries of each list in flight per lane; a trip of a warp
// (128 entries of a list) is a chain of two loads and a store, 1 us, which is what bounds it while the device has rows to
// spare for few warps.  topk_apply_two says where it stands in for two launches.
__device__ __forceinline__ void apply_row(const ListSource &list, unsigned r, unsigned cols, float *row, unsigned lane, const ApplyReport &report) {
    const unsigned k = list.k;
    const uint8_t *idx = list.idx + 2 * (size_t)r * k, *val = list.val + 4 * (size_t)r * k;
    for (unsigned j0 = lane; j0 < k; j0 += 128) {
        unsigned c[4];
        float v[4], d[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            c[u] = j0 + 32 * u < k ? load_u16_any(idx + 2 * (j0 + 32 * u)) : 0xFFFFFFFFu;
            v[u] = j0 + 32 * u < k ? load_f32_any(val + 4 * (j0 + 32 * u)) : 0.0f;
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) d[u] = c[u] < cols ? row[c[u]] : 0.0f;
        // (a list's entries have columns of their own; what a list that names one twice leaves there is open, as it is when
        // the entries are spread over threads)
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            if (c[u] < cols) row[c[u]] = d[u] + v[u];
            else if (c[u] != 0xFFFFFFFFu) report_bad_index(report.status, report.on_host);
        }
    }
}
__global__ void __launch_bounds__(256) topk_apply_two_kernel(ListSource first, ListSource second, unsigned rows, unsigned cols, float *dense,
                                                             ApplyReport report) {
    chain_begin();
    end_call(report);
    const unsigned lane = threadIdx.x & 31, r = blockIdx.x * 8 + (threadIdx.x >> 5);
    if (r >= rows) return;
    float *row = dense + (size_t)r * cols;
    apply_row(first, r, cols, row, lane, report);
    __syncwarp();
    apply_row(second, r, cols, row, lane, report);
}

// ---- e = a - b, flag |= any(|e| > FLT_EPSILON) ----------------------------------------------------
__global__ void __launch_bounds__(256)
    residual_error_kernel(const float *__restrict__ a, const float *__restrict__ b, uint64_t n, bool vec,
                          float *__restrict__ e, unsigned *flag) {
    bool any = false;
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    const uint64_t t0 = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (vec) {
        const uint64_t n4 = n / 4;
        for (uint64_t i = t0; i < n4; i += stride) {
            const float4 x = __ldcs(reinterpret_cast<const float4 *>(a) + i);
            const float4 y = __ldcs(reinterpret_cast<const float4 *>(b) + i);
            const float4 d = make_float4(__fsub_rn(x.x, y.x), __fsub_rn(x.y, y.y), __fsub_rn(x.z, y.z), __fsub_rn(x.w, y.w));
            any |= abs4max(d) > 1.1920928955078125e-07f;
            reinterpret_cast<float4 *>(e)[i] = d;
        }
        for (uint64_t i = n4 * 4 + t0; i < n; i += stride) {
            const float d = __fsub_rn(a[i], b[i]);
            any |= fabsf(d) > 1.1920928955078125e-07f;
            e[i] = d;
        }
    } else {
        for (uint64_t i = t0; i < n; i += stride) {
            const float d = __fsub_rn(a[i], b[i]);
            any |= fabsf(d) > 1.1920928955078125e-07f;
            e[i] = d;
        }
    }
    if (__any_sync(kFullMask, any) && (threadIdx.x & 31) == 0) atomicOr(flag, 1u);
}

}  // namespace

int device_sm_count() {
    int dev = 0, sms = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return 148;
    if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms <= 0) return 148;
    return sms;
}

int topk_num_columns(uint16_t cols, float ratio) {
    if (cols == 0) return 0;
    if (!(ratio >= 0.0f && ratio <= 1.0f)) return -1;
    const float raw = (float)cols * ratio;
    uint16_t k = (uint16_t)roundf(raw);
    if (k > cols) k = cols;
    else if (k == 0 && ratio > 0.0f) k = 1;
    return k;
}

// Geometry of the group kernel: G warps per row (a group never holds more than 16 KiB of row per warp
// pair), as many groups per CTA as fit half of an SM's shared memory.
struct GroupGeometry {
    int G, groups, threads;
    unsigned group_bytes, ctl_off;
};
static GroupGeometry group_geometry(uint32_t cols) {
    GroupGeometry f;
    f.G = cols <= 4096 ? 2 : (cols <= 8192 ? 4 : 8);
    f.ctl_off = (cols * 4u + 15u) & ~15u;
    f.group_bytes = (f.ctl_off + (unsigned)sizeof(GroupCtl) + 127u) & ~127u;
    int groups = (int)((110u * 1024u) / f.group_bytes);
    if (groups < 1) groups = 1;
    if (groups > 512 / (32 * f.G)) groups = 512 / (32 * f.G);
    if (groups > 15) groups = 15;
    f.groups = groups;
    f.threads = groups * 32 * f.G;
    return f;
}

static bool topk_rows_fit_smem(uint32_t cols, uint32_t k) {
    return k > 0 && k <= (uint32_t)kCandCap && cols <= 24576u && group_geometry(cols).group_bytes <= 110u * 1024u;
}
// Rows that no bulk copy can move: up to how many entries the group kernel is the faster one.  Its bound is the k-th largest of
// the two largest float4 of every lane; as k comes near the number of those (two per lane, or the row's float4) more elements
// reach it than there is room for, and the row is done once more the slow way: 2 to 3 times the generic kernel's time.
// us, group / generic: 148 x 1001 k = 80 16 / 16, k = 128 51 / 16; 2000 x 3001 k = 96 29 / 68, k = 128 125 / 70; 8192 x 8190 k = 160
// 139 / 563, k = 192 718 / 565; 2000 x 14335 k = 208 74 / 211, k = 240 395 / 211; 600 x 63 k = 16 10 / 12, k = 24 35 / 12.
// With many rows the generic kernel's passes weigh more, so the line lies a little higher.
static bool ragged_rows_fit(uint32_t rows, uint32_t cols, uint32_t k) {
    const int G = group_geometry(cols).G;
    if (k > (cols + 3) / 4) return false;
    if (G == 8) return k <= 216;
    const uint32_t most = G == 2 ? (rows >= 2000 ? 112 : rows >= 1024 ? 108 : rows >= 700 ? 100 : 80)
                                 : (rows >= 2000 ? 176 : rows >= 1024 ? 168 : 160);
    return k <= most && (rows >= 1024 || k <= 32 || 5 * k <= cols);
}
// rows that a bulk copy can move: whole 16-byte pieces at 16-byte boundaries
static bool bulk_rows(const void *d_in, const void *d_residual, uint32_t cols) {
    return cols % 4 == 0 && reinterpret_cast<uintptr_t>(d_in) % 16 == 0 && reinterpret_cast<uintptr_t>(d_residual) % 16 == 0;
}

template <int G, bool kBulk>
static cudaError_t launch_group(const float *d_in, float *d_residual, uint32_t rows, uint32_t cols, uint32_t k,
                                uint16_t *d_idx, float *d_val, unsigned *d_status, int sm_count, cudaStream_t stream, unsigned *d_bound) {
    const GroupGeometry f = group_geometry(cols);
    const size_t smem = (size_t)f.group_bytes * f.groups;
    cudaError_t err = cudaFuncSetAttribute(topk_rows_group_kernel<G, kBulk>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (err != cudaSuccess) return err;
    err = cudaFuncSetAttribute(topk_rows_group_kernel<G, kBulk>, cudaFuncAttributePreferredSharedMemoryCarveout,
                               cudaSharedmemCarveoutMaxShared);
    if (err != cudaSuccess) return err;
    int per_sm = 0;
    err = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, topk_rows_group_kernel<G, kBulk>, f.threads, smem);
    if (err != cudaSuccess) return err;
    if (per_sm < 1) per_sm = 1;
    unsigned grid = (unsigned)sm_count * (unsigned)per_sm;
    const unsigned needed = (rows + f.groups - 1) / f.groups;
    if (grid > needed) grid = needed;
    return launch_chained(topk_rows_group_kernel<G, kBulk>, grid, f.threads, smem, stream, d_in, d_residual, rows, cols, k, d_idx, d_val, d_status,
                          f.group_bytes, f.ctl_off, d_bound);
}

cudaError_t topk_rows(const float *d_in, float *d_residual, uint32_t rows, uint32_t cols, uint32_t k, uint16_t *d_idx,
                      float *d_val, unsigned *d_status, int sm_count, cudaStream_t stream, unsigned *d_bound, bool *bound_written) {
    if (bound_written) *bound_written = false;
    if (!d_in || rows == 0 || cols == 0 || cols > 65535u || k > cols) return cudaErrorInvalidValue;
    if (k == 0) {
        if (d_residual && d_residual != d_in)
            return cudaMemcpyAsync(d_residual, d_in, (size_t)rows * cols * 4, cudaMemcpyDeviceToDevice, stream);
        return cudaSuccess;
    }
    if (!d_idx || !d_val) return cudaErrorInvalidValue;
    const bool bulk = bulk_rows(d_in, d_residual, cols);
    if (topk_rows_fit_smem(cols, k) && (bulk || ragged_rows_fit(rows, cols, k))) {
        if (d_bound && bound_written) *bound_written = true;
#define BSQ_TOPK(G_)                                                                                                             \
    (bulk ? launch_group<G_, true>(d_in, d_residual, rows, cols, k, d_idx, d_val, d_status, sm_count, stream, d_bound) \
          : launch_group<G_, false>(d_in, d_residual, rows, cols, k, d_idx, d_val, d_status, sm_count, stream, d_bound))
        switch (group_geometry(cols).G) {
            case 2: return BSQ_TOPK(2);
            case 4: return BSQ_TOPK(4);
            default: return BSQ_TOPK(8);
        }
#undef BSQ_TOPK
    }
    unsigned grid = (unsigned)sm_count * 8u;
    if (grid > rows) grid = rows;
    topk_rows_generic_kernel<<<grid, kGenericThreads, 0, stream>>>(d_in, d_residual, rows, cols, k, d_idx, d_val);
    return cudaGetLastError();
}

static cudaError_t launch_apply(const ListSource &list, uint32_t rows, uint32_t cols, float *d_dense, const ApplyReport &report, cudaStream_t stream) {
    const size_t total = (size_t)rows * list.k;
    size_t grid = (total + 255) / 256;
    if (grid > 148 * 16) grid = 148 * 16;
    return launch_chained(topk_apply_kernel, (unsigned)grid, 256, 0, stream, list, rows, cols, d_dense, report);
}
static ListSource as_list(const uint16_t *d_idx, const float *d_val, uint32_t k) {
    ListSource l;
    l.idx = reinterpret_cast<const uint8_t *>(d_idx);
    l.val = reinterpret_cast<const uint8_t *>(d_val);
    l.k = k;
    return l;
}

cudaError_t topk_apply(const uint16_t *d_idx, const float *d_val, uint32_t rows, uint32_t cols, uint32_t k,
                       float *d_dense, unsigned *d_status, cudaStream_t stream) {
    if (!d_dense || rows == 0 || cols == 0) return cudaErrorInvalidValue;
    if (k == 0) return cudaSuccess;
    if (!d_idx || !d_val) return cudaErrorInvalidValue;
    return launch_apply(as_list(d_idx, d_val, k), rows, cols, d_dense, ApplyReport{d_status, false, nullptr}, stream);
}

static cudaError_t launch_apply_two(const ListSource &a, const ListSource &b, uint32_t rows, uint32_t cols, float *d_dense, const ApplyReport &report,
                                    cudaStream_t stream) {
    // A decompress call is 2 to 6 us shorter with one launch than with two, until a warp's trips take longer than that (few
    // rows), or a matrix beyond the L2 wants the two launches' larger grids; and lists that name a good part of a row find it in
    // the L1 cache when one warp walks it.  us a call, one / two launches, calls of either taken in turn: 300 x 4096
    // with 41 + 20 entries a row 38 / 41, 64 x 8192 with 82 + 164 39 / 41; 4001 x 4096 with 41 + 82 56 / 59; 2048 x 4096 with
    // 41 + 819 55 / 67, 1000 x 8192 with 3277 + 3277 112 / 189; on the other side 8 x 14336 with 5734 + 5734 125 / 39, 64 x 14336 with
    // 717 + 717 43 / 41, 4001 x 14336 with 717 + 717 267 / 225, 6144 x 8192 with 82 + 1638 352 / 281.
    const uint64_t listed = (uint64_t)a.k + b.k, entries = rows * listed, elements = (uint64_t)rows * cols;
    const uint32_t trips = (a.k + 127) / 128 + (b.k + 127) / 128;
    bool one_launch;
    if (rows >= 512 && 5 * listed >= cols) one_launch = elements <= (32u << 20) || 2 * listed >= cols;
    else if (entries > 1400000) one_launch = trips <= 3;
    else one_launch = trips <= (rows >= 512 ? 8u : 5u);
    if (!one_launch) {
        // (the words are for the call's last kernel; the first one reports where that one does)
        const cudaError_t err = launch_apply(a, rows, cols, d_dense, ApplyReport{report.status, report.on_host, nullptr}, stream);
        return err != cudaSuccess ? err : launch_apply(b, rows, cols, d_dense, report, stream);
    }
    return launch_chained(topk_apply_two_kernel, (rows + 7) / 8, 256, 0, stream, a, b, rows, cols, d_dense, report);
}

cudaError_t topk_apply_two(const uint16_t *d_idx0, const float *d_val0, uint32_t k0, const uint16_t *d_idx1, const float *d_val1,
                           uint32_t k1, uint32_t rows, uint32_t cols, float *d_dense, unsigned *d_status, cudaStream_t stream) {
    if (!d_dense || rows == 0 || cols == 0) return cudaErrorInvalidValue;
    if ((k0 && (!d_idx0 || !d_val0)) || (k1 && (!d_idx1 || !d_val1))) return cudaErrorInvalidValue;
    if (k0 == 0) return topk_apply(d_idx1, d_val1, rows, cols, k1, d_dense, d_status, stream);
    if (k1 == 0) return topk_apply(d_idx0, d_val0, rows, cols, k0, d_dense, d_status, stream);
    return launch_apply_two(as_list(d_idx0, d_val0, k0), as_list(d_idx1, d_val1, k1), rows, cols, d_dense, ApplyReport{d_status, false, nullptr}, stream);
}

cudaError_t apply_lists_end(const ListSource &a, const ListSource &b, uint32_t rows, uint32_t cols, float *d_dense, unsigned *d_status,
                            unsigned *mirror, cudaStream_t stream) {
    const ApplyReport report{mirror, true, d_status};
    if (a.k && b.k) return launch_apply_two(a, b, rows, cols, d_dense, report, stream);
    if (a.k || b.k) return launch_apply(a.k ? a : b, rows, cols, d_dense, report, stream);
    return launch_chained(end_call_kernel, 1, 32, 0, stream, report);
}

cudaError_t residual_error(const float *d_a, const float *d_b, uint64_t n, float *d_e, unsigned *d_flag, int sm_count,
                           cudaStream_t stream) {
    if (!d_a || !d_b || !d_e || !d_flag || n == 0) return cudaErrorInvalidValue;
    const bool vec = ((reinterpret_cast<uintptr_t>(d_a) | reinterpret_cast<uintptr_t>(d_b) |
                       reinterpret_cast<uintptr_t>(d_e)) % 16) == 0;
    uint64_t grid = (n / 4 + 255) / 256;
    const uint64_t cap = (uint64_t)sm_count * 8;
    if (grid > cap) grid = cap;
    if (grid == 0) grid = 1;
    residual_error_kernel<<<(unsigned)grid, 256, 0, stream>>>(d_a, d_b, n, vec, d_e, d_flag);
    return cudaGetLastError();
}

}  // namespace bsq

// Host-side launchers of the sm_100a kernels.  Internal to the library: the public surfaces
// are include/bitsqz_llm.hpp (C++ interface of the reference) and include/bitsqz_llm_c.h
// (C ABI).  Every launcher enqueues work on `stream` and returns without synchronising.
#pragma once

#include <cuda_runtime.h>
#include <stddef.h>
#include <stdint.h>

namespace bsq {

// ---- a call's first and last kernel -------------------------------------------------------------
constexpr int kMaxHeads = 6;
// The headers inside a device-resident payload, checked by the kernel that reads the sections: it is launched before the host has seen
// them (a wait of 12 us between a small kernel that fetched them and the one that decodes), writes nothing unless every byte under
// `mask` is the one that the host expects, and its first CTA leaves the outcome in page-locked memory, where the host waits for it
// before it goes on.
constexpr int kMaxHeadBytes = 48;
struct HeadCheck {
    const uint8_t *src[kMaxHeads];
    uint64_t mask[kMaxHeads];                                // bit i: byte i has to match
    uint8_t length[kMaxHeads];
    uint8_t want[kMaxHeads][kMaxHeadBytes];
    int count = 0;
    unsigned *answer = nullptr, number = 0;                  // receives `number` (even), + 1 where a header differs
};

// ---- NF4 / NF4_DQ over a flat array (bsq_quant.cu) ----------------------------------------
// d_deq_out (nullable): also write the dequantised values, which is what the reference's
// compress path feeds into its error-correction stage (src/bitsqz_llm.cu:506-511).  With d_error_flag (a device word) the
// second output is x - dequantised instead, and the word is set to 1 when some |difference| > FLT_EPSILON.
cudaError_t nf4_quantize(const float *d_x, uint64_t n, float *d_scales, uint8_t *d_data, float *d_deq_out, int sm_count,
                         cudaStream_t stream, unsigned *d_error_flag = nullptr);
size_t nf4dq_scratch_bytes(uint64_t n);
// d_gmax (nullable): a device word that is zero, for the largest magnitude; without it the call clears one in d_scratch.
cudaError_t nf4dq_quantize(const float *d_x, uint64_t n, float *d_dq, uint8_t *d_scale_codes, uint8_t *d_data,
                           float *d_deq_out, void *d_scratch, int sm_count, cudaStream_t stream, unsigned *d_error_flag = nullptr,
                           unsigned *d_gmax = nullptr);
// Variant for callers that must not allocate: scratch is a fixed array inside the library.
uint64_t nf4dq_static_max_elements();
cudaError_t nf4dq_quantize_static(const float *d_x, uint64_t n, float *d_dq, uint8_t *d_scale_codes, uint8_t *d_data,
                                  int sm_count, cudaStream_t stream);
cudaError_t nf4_dequantize(const float *d_scales, const uint8_t *d_data, uint64_t n, float *d_out, int sm_count,
                           cudaStream_t stream);
cudaError_t nf4dq_dequantize(const float *d_dq, const uint8_t *d_scale_codes, const uint8_t *d_data, uint64_t n,
                             float *d_out, int sm_count, cudaStream_t stream);
// Two arrays of one format at once (the factors U and V), each with what it is quantised into; NF4_DQ: gmax is a device word that is
// zero, scratch holds nf4dq_scratch_bytes of both.  deq (nullable, may be x): the dequantised values; max_bits (nullable, with deq; zero before)
// receives the bits of the largest |deq(i) colscale(i mod cols)|, colscale nullable.
struct QuantTarget {
    const float *x = nullptr;
    uint64_t n = 0;
    float *scales = nullptr;              // NF4
    float *dq = nullptr;                  // NF4_DQ
    uint8_t *scale_codes = nullptr;
    uint8_t *data = nullptr;
    float *deq = nullptr;
    unsigned *gmax = nullptr;
    const float *colscale = nullptr;
    uint32_t cols = 1;
    unsigned *max_bits = nullptr;
};
cudaError_t quantize_pair(int method, const QuantTarget &a, const QuantTarget &b, void *d_scratch, int sm_count, cudaStream_t stream);
// A section as it lies in a device-resident object, whatever its alignment.
struct SectionSource {
    const uint8_t *scales = nullptr;      // NF4: FP32, NF4_DQ: E4M3
    const uint8_t *dq = nullptr;          // NF4_DQ only
    const uint8_t *data = nullptr;        // nibbles, or FP32 values where scales is null
    uint64_t n = 0;
};
// A row-wise top-k list as it lies in an object (idx: u16, val: f32, any alignment).
struct ListSource {
    const uint8_t *idx = nullptr, *val = nullptr;
    uint32_t k = 0;
};
// A quantised matrix section -> d_out, and its lists (k > 0), one after the other, added in the same pass: the whole decompress call
// of such an object.  Nothing is written where the object's headers are not what `heads` expects.  mirror: page-locked, zero; receives
// kStatusBadIndex where a list names a column that the matrix does not have.
cudaError_t decode_matrix(const SectionSource &q, uint32_t rows, uint32_t cols, const ListSource &first, const ListSource &second, float *d_out,
                          unsigned *mirror, const HeadCheck &heads, int sm_count, cudaStream_t stream);
// Whether lists of k0 and k1 entries a row are better added behind that pass (apply_lists_end).
bool decode_lists_apart(uint32_t rows, uint32_t cols, uint32_t k0, uint32_t k1, int sm_count);
// Dequantise a rows x cols matrix and add a row-wise top-k list in one pass; d_scales (NF4) or d_dq + d_scale_codes (NF4_DQ).
cudaError_t nf4_dequantize_add_topk(const float *d_scales, const float *d_dq, const uint8_t *d_scale_codes, const uint8_t *d_data,
                                    uint32_t rows, uint32_t cols, const uint16_t *d_idx, const float *d_val, uint32_t k,
                                    float *d_out, unsigned *d_status, int sm_count, cudaStream_t stream);

// The factors U (rows x rank), V and S (rank FP32 values) of an object into 16-byte aligned buffers, in one launch; *d_max_us and *d_max_v
// (zero before) receive the bits of the largest |U(i, t) S(t)| and |V|.  What the buffers hold is of no use where `heads` finds a difference.
cudaError_t open_factors(const SectionSource &u, const SectionSource &v, const uint8_t *s, uint32_t rank, float *d_u, float *d_v, float *d_s,
                         unsigned *d_max_us, unsigned *d_max_v, const HeadCheck &heads, int sm_count, cudaStream_t stream);

// ---- per-row top-k (bsq_topk.cu) ------------------------------------------------------------
// k = (uint16)roundf(cols * ratio) clamped to cols, at least 1 for ratio > 0; -1 for a ratio
// outside [0, 1] (reference topk_cuda.cu:53-69).
int topk_num_columns(uint16_t cols, float ratio);

// Per row: the k entries of largest |x| ordered by (|x| descending, column ascending), NaN
// ranking below every number.  d_idx / d_val are [rows][k].  d_residual (nullable): receives
// the row with the selected entries set to +0.0f; may alias d_in (in-place separation).
// d_status: device word that receives kStatus* bits.
// d_bound (nullable device word, zero when the call runs) receives, where the shared-memory path runs (*bound_written says
// so), the bits of the largest k-th |x| over the rows: an upper bound of every |x| that is left in d_residual.
cudaError_t topk_rows(const float *d_in, float *d_residual, uint32_t rows, uint32_t cols, uint32_t k, uint16_t *d_idx,
                      float *d_val, unsigned *d_status, int sm_count, cudaStream_t stream, unsigned *d_bound = nullptr,
                      bool *bound_written = nullptr);

// dense[row, idx] += val for every entry; indices >= cols are skipped and reported in d_status.
cudaError_t topk_apply(const uint16_t *d_idx, const float *d_val, uint32_t rows, uint32_t cols, uint32_t k,
                       float *d_dense, unsigned *d_status, cudaStream_t stream);

// Two lists, the first before the second where they name the same element, in one launch or two.
cudaError_t topk_apply_two(const uint16_t *d_idx0, const float *d_val0, uint32_t k0, const uint16_t *d_idx1, const float *d_val1,
                           uint32_t k1, uint32_t rows, uint32_t cols, float *d_dense, unsigned *d_status, cudaStream_t stream);
// The same with the lists where they lie in an object, either or both possibly empty, as the end of a decompress call: status words of the
// call's earlier kernels (d_status, null where they report to the mirror themselves), and columns out of range, are reported in the page-locked, zero
// `mirror`; the words are cleared.
cudaError_t apply_lists_end(const ListSource &a, const ListSource &b, uint32_t rows, uint32_t cols, float *d_dense, unsigned *d_status,
                            unsigned *mirror, cudaStream_t stream);

// ---- fused front end of the no-SVD path (bsq_frontend.cu) -----------------------------------
// outlier separation + NF4 or NF4_DQ of the remainder, reading the input once from HBM (the
// NF4_DQ second pass re-reads it through L2).  Needs cols % 64 == 0, k <= 256 and a row that
// fits shared memory; frontend_supported() says whether a shape qualifies.
bool frontend_supported(uint32_t rows, uint32_t cols, uint32_t k);
size_t frontend_scratch_bytes(uint32_t rows, uint32_t cols);
// method: 11 = NF4 (d_scales_f32 used), 10 = NF4_DQ (d_dq, d_scale_codes used).
// d_words (nullable): kFrontWords device words that are zero; without them the call clears words in d_scratch.
cudaError_t frontend_quantize(int method, const float *d_in, uint32_t rows, uint32_t cols, uint32_t k, uint16_t *d_idx,
                              float *d_val, float *d_scales_f32, float *d_dq, uint8_t *d_scale_codes, uint8_t *d_data,
                              void *d_scratch, unsigned *d_status, int sm_count, cudaStream_t stream,
                              cudaEvent_t *events = nullptr,    // events[3]: before pass 1, between, after pass 2
                              unsigned *d_words = nullptr);
constexpr int kFrontWords = 3;

// ---- residual / error helpers ---------------------------------------------------------------
// e = a - b and *d_flag |= 1 when some |e| > FLT_EPSILON (reference src/bitsqz_llm.cu:164-184).
cudaError_t residual_error(const float *d_a, const float *d_b, uint64_t n, float *d_e, unsigned *d_flag, int sm_count,
                           cudaStream_t stream);

// ---- device-resident objects (bsq_pack.cu) ---------------------------------------------------
constexpr int kMaxCopySegments = 12;
// The words of a runtime's status block.  All are zero when a call's first kernel starts: the kernel that ends a call hands
// them to the host and clears them for the next one, where a memset in front of each of them cost the chain of a call
// 4.3 us (its own 1.6 and the gap to the next operation).
constexpr int kStatusWords = 16;
enum : int {
    kWordStatus = 0,                                         // kernel status bits
    kWordError = 1,                                          // something is left for the error list
    kWordFront = 2,                                          // kFrontWords of the fused front end
    kWordMaxU = 5,                                           // NF4_DQ: the largest magnitude of a section
    kWordMaxV = 6,
    kWordMaxOne = 7,                                         // (the matrix or S)
    kWordBound = 8,                                          // bound of the residual for the SVD's products
    kWordMaxUS = 9,                                          // the largest |U S| and |V|: scales of the reconstruction's operands
    kWordMaxVR = 10
};
struct CopySegment {
    void *dst;
    const void *src;
    uint64_t bytes;
};
// Headers that the host knows, on their way into a device-resident object.
struct PackHeaders {
    struct Piece {
        uint8_t *dst;
        const void *patch;                                   // nullable: device word that replaces the four bytes at patch_at
        uint16_t at, length, patch_at;
    } piece[kMaxHeads];
    int pieces;
    uint8_t bytes[256];                                      // the pieces' contents
    uint8_t object[200];                                     // the object's header as it is with an error section
    uint8_t *object_dst;
    int flags_at, error_entry_at, error_entry_length;        // cleared where status word 1 says that there is none
    uint8_t error_flag;
};
struct HeadList {
    const uint8_t *src[kMaxHeads];
    int length[kMaxHeads];                                   // at most 64
    int count;
};
// How [p, p + bytes) may be reached from the current device.  Kernels fault where a stream copy works (another GPU's memory) or
// returns an error (memory that CUDA does not know), so the caller's pointer is looked at before one is launched on it.
enum class Reach {
    kNone,                                                   // some of it is not CUDA memory
    kCopies,                                                 // stream copies only: another device's memory, page-locked, managed
    kKernels                                                 // this device's memory from one end to the other
};
Reach memory_reach(const void *p, uint64_t bytes);
// Copies up to kMaxCopySegments pieces of device memory, of any alignment, in one launch.
cudaError_t copy_segments(const CopySegment *segments, int count, cudaStream_t stream);
// The same together with the headers and, into page-locked `mirror`, the status words, which it clears.
cudaError_t pack_object(const CopySegment *segments, int count, const PackHeaders &headers, unsigned *d_status, unsigned *mirror,
                        cudaStream_t stream);
// Small headers out of a device-resident payload into page-locked `host`, 64 bytes apart; clears the status words.
cudaError_t fetch_heads(const HeadList &heads, uint8_t *host, unsigned *d_status, cudaStream_t stream);

int device_sm_count();
// A block for a packed object that the caller will release with bitsqz_llm_free: page-locked from the library's pool
// when one can be had, plain heap memory otherwise (bsq_api.cu).
void *host_block_take(size_t bytes);

// ---- randomized low-rank SVD and reconstruction (bsq_svd.cu, bsq_gemm.cu) -------------------
// Replaces svd_lowrank_cuda_initialize / svd_lowrank_cuda / svd_lowrank_cuda_release
// (modules/svd_lowrank_cuda/src/svd_lowrank_cuda.cu:541-581) and reconstruct_lowrank_cuda
// (modules/reconstruct_lowrank_cuda/src/reconstruct_lowrank_cuda.cu:153-171).
// C[M x N] = opA[M x K] * opB[K x N] in FP32 (bsq_gemm.cu).  a_kmajor: opA(i,kk) = A[i*lda+kk], else A[kk*lda+i];
// b_kmajor: opB(kk,j) = B[j*ldb+kk], else B[kk*ldb+j].  kscale (nullable) scales opA along K.  minuend (nullable):
// C = minuend - product, *flag |= 1 when some |C| > FLT_EPSILON.  workspace (nullable) enables a deterministic K split.
// Skinny products (N = 16..256, no fused epilogue) run on the tensor cores (bsq_gemm_tc.cu); `status` (nullable device
// word) receives kStatusBarrierTimeout if one of that kernel's bounded waits gives up.
cudaError_t gemm(bool a_kmajor, bool b_kmajor, const float *A, long lda, const float *B, long ldb, float *C, long ldc, int M,
                 int N, int K, const float *kscale, const float *minuend, long ldm, unsigned *flag, unsigned *status,
                 float *workspace, size_t workspace_bytes, int sm_count, cudaStream_t stream, const unsigned *a_absmax_bits = nullptr,
                 float b_bound = 0.0f, bool device_full = false,
                 const unsigned *b_absmax_bits = nullptr);
// The same with the kernel choice explicit: allow_tensor_cores = false keeps the product on the FP32 pipes.
cudaError_t gemm_select(bool allow_tensor_cores, bool a_kmajor, bool b_kmajor, const float *A, long lda, const float *B, long ldb,
                        float *C, long ldc, int M, int N, int K, const float *kscale, const float *minuend, long ldm,
                        unsigned *flag, unsigned *status, float *workspace, size_t workspace_bytes, int sm_count,
                        cudaStream_t stream, const unsigned *a_absmax_bits = nullptr, float b_bound = 0.0f, bool device_full = false,
                        const unsigned *b_absmax_bits = nullptr);
// (a_absmax_bits: device word with the bits of an upper bound of |A|, b_bound: an upper bound of |B| known on the host,
// 0 = none -- with a bound on |A| the 256-column products split their operands into FP16 halves, bsq_gemm_tc.cuh;
// a_absmax_bits and b_absmax_bits together: the largest |A kscale| and |B| for a wide product's split)

struct SvdWorkspace;
// sums `count` floats at `buf` over all ranks, enqueued on `stream`
typedef cudaError_t (*SvdAllReduce)(void *ctx, float *buf, size_t count, cudaStream_t stream);
// coded_factors: U, S, V are quantised afterwards or an error list is made from them, so that the order of rotations in the
// core's SVD shows in an object's bytes (bsq_svd.cu)
SvdWorkspace *svd_workspace_create(int m, int n, int k, int niter, int sm_count, bool coded_factors = false);
SvdWorkspace *svd_workspace_create_sharded(int m_local, int n, int k, int niter, int sm_count, SvdAllReduce allreduce,
                                           void *allreduce_ctx, int m_total, bool coded_factors = false);
void svd_workspace_destroy(SvdWorkspace *ws);
// whether other work fills the device beside the calls that follow (chooses tile widths, not results; no until set)
void svd_workspace_device_full(SvdWorkspace *ws, bool full);
// A row-major m x n -> U (m x k row-major), S (k, descending), V (n x k row-major).
// The random matrix is the first N x k normals of cuRAND's XORWOW sequence of `seed`, starting `offset` values in.
cudaError_t svd_lowrank(SvdWorkspace *ws, const float *d_A, float *d_U, float *d_S, float *d_V,
                        unsigned long long seed, unsigned *d_status, cudaStream_t stream, unsigned long long offset = 0,
                        const unsigned *d_abs_bound = nullptr);
// (d_abs_bound, nullable: device word with the bits of an upper bound of |A|, e.g. from topk_rows; without it the call
// makes a pass over A for the largest |A| where it needs one.)
// Optional timing of a call's products with the big matrix (kind 0) and, row-sharded, its all-reduces (kind 1).
cudaError_t svd_workspace_profile(SvdWorkspace *ws, bool on);
int svd_workspace_spans(SvdWorkspace *ws, float *ms, int *kinds, int capacity);
// For calls made with d_status == nullptr: waits for the stream and returns an error if a bounded wait gave up.
cudaError_t svd_workspace_finish(SvdWorkspace *ws, cudaStream_t stream);
// out = (U diag(S)) V^T, row-major m x n.  d_minuend (nullable): write minuend - out instead and
// OR 1 into *d_flag when some |difference| > FLT_EPSILON.
// d_status (nullable): device word that receives kStatusBarrierTimeout if a bounded wait of the product kernel gives up
// (the output is then incomplete).
// d_workspace (nullable, reconstruct_workspace_bytes, 128-byte aligned): room for V and U diag(S) split once into the
// tensor cores' operand format, shared by all tiles; without it every tile splits its pieces itself.
// d_max_us, d_max_v (nullable): device words with the bits of the largest |U(i, t) S(t)| and |V|; without them the call makes a pass
// over each.
size_t reconstruct_workspace_bytes(int m, int n, int k);
cudaError_t reconstruct_lowrank(const float *d_U, const float *d_S, const float *d_V, int m, int n, int k,
                                const float *d_minuend, float *d_out, unsigned *d_flag, unsigned *d_status, float *d_workspace,
                                size_t workspace_bytes, int sm_count, cudaStream_t stream, const unsigned *d_max_us = nullptr,
                                const unsigned *d_max_v = nullptr);

}  // namespace bsq

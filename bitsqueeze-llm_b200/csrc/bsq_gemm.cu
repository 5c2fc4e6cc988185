// FP32 GEMM building block of the low-rank stages (sm_100a).
//
// Replaces the cublasSgemm / cublasSdgmm call sites of the reference
// (modules/svd_lowrank_cuda/src/svd_lowrank_cuda.cu:293-309,319-335,344-360,370-386,409-425 and
// modules/reconstruct_lowrank_cuda/src/reconstruct_lowrank_cuda.cu:31-61) with one kernel that reads
// the caller's row-major matrices in whichever orientation a product needs, so the reference's
// explicit transposes of the input and of U, V (svd_lowrank_cuda_utils.cuh:91-109) disappear:
//
//   C[M x N] = opA[M x K] * opB[K x N]
//   A_KMAJOR  : opA(i, kk) = A[i * lda + kk]   (A used as stored)      else opA(i, kk) = A[kk * lda + i]  (A^T)
//   B_KMAJOR  : opB(kk, j) = B[j * ldb + kk]   (B^T of a row-major B)  else opB(kk, j) = B[kk * ldb + j]
//
// All the products of the randomized SVD are "skinny": one of M, N is the rank k (<= 256), the other
// one matrix dimension, and K is the other matrix dimension, so there are few output tiles; the grid's
// third dimension splits K and a second kernel adds the partial tiles in a fixed order (deterministic).
// Optional fusions: a per-k scale on opA (U * diag(S) of reconstruct), and in the epilogue
// "minuend - C" with an any(|.| > FLT_EPSILON) flag (the reference's subtract_kernel + has_nonzero_kernel,
// src/bitsqz_llm.cu:164-184).
//
// This version computes on the FP32 pipes (tiles of 128 x 128, 128 x 64 or 64 x 64 outputs, pieces of 16 of K by asynchronous copies).
#include "bsq_device.cuh"
#include "bsq_gemm.hpp"
#include "bsq_internal.hpp"

#include <cstdlib>

namespace bsq {
namespace {

constexpr int BM = 128, BN = 128, BK = 16, GT = 256;         // (what K is split by; the tiles themselves are TM x TN)

// One operand's piece of a step: kRows rows or columns of the output tile by BK of K, as it lies in memory: contiguous along K
// (kKMajor: row r at r (BK + 4)) or along the rows (k at k (kRows + 4)).
template <bool kKMajor, int kRows>
struct Piece {
    static constexpr int kLd = kKMajor ? BK + 4 : kRows + 4;
    static constexpr int kFloats = kKMajor ? kRows * kLd : BK * kLd;

    // Starts the copies of rows row0 .. and k0 .. (zero outside the matrix and the split).  kVec: rows are 16-byte aligned.
    template <bool kVec>
    static __device__ __forceinline__ void fetch(float *S, const float *__restrict__ P, long ld, int rows_total, int row0, int k0, int k_end) {
        constexpr int kW = kVec ? 4 : 1;                     // floats per copy
        constexpr int kInner = (kKMajor ? BK : kRows) / kW, kCopies = kRows * BK / kW;
        static_assert(kCopies % GT == 0, "whole copies per thread");
#pragma unroll
        for (int u = 0; u < kCopies / GT; ++u) {
            const int e = threadIdx.x + u * GT, outer = e / kInner, inner = e % kInner * kW;
            const int r = row0 + (kKMajor ? outer : inner), k = k0 + (kKMajor ? inner : outer);
            // what of the copy lies inside, in bytes
            const int left = kKMajor ? (r < rows_total ? k_end - k : 0) : (k < k_end ? rows_total - r : 0);
            const int bytes = min(max(left, 0), kW) * 4;
            const float *src = bytes ? P + (kKMajor ? (long)r * ld + k : (long)k * ld + r) : P;
            const unsigned dst = smem_u32(S + outer * kLd + inner);
            if (kVec) asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
            else asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
        }
    }
};

// TM x TN outputs per CTA, TM / 16 x TN / 16 per thread; thread (ty, tx) has rows ty + 16 i of an operand that lies along K
// (neighbouring rows then start 20 floats apart: no bank twice in eight lanes) and 4 ty .. + 3 of every 64 of one that lies along
// the rows.  Pieces come in by asynchronous copies kStages - 1 steps ahead.  Each output is one chain of multiply-adds over its split's
// K, whatever the tile.
template <bool A_KMAJOR, bool B_KMAJOR, int TM, int TN, int kStages, bool kVecA, bool kVecB>
__global__ void __launch_bounds__(GT, A_KMAJOR && B_KMAJOR && TM * TN == 128 * 128 ? 1 : 2) gemm_kernel(GemmArgs g) {
    using PA = Piece<A_KMAJOR, TM>;
    using PB = Piece<B_KMAJOR, TN>;
    constexpr int MI = TM / 16, NI = TN / 16;
    __shared__ __align__(16) float As[kStages][PA::kFloats];
    __shared__ __align__(16) float Bs[kStages][PB::kFloats];
    const int t = threadIdx.x, tx = t & 15, ty = t >> 4;
    chain_begin();
    const int m0 = blockIdx.y * TM, n0 = blockIdx.x * TN;
    const int k_begin = blockIdx.z * g.k_per_split;
    const int k_end = min(g.K, k_begin + g.k_per_split);
    const int steps = k_end > k_begin ? (k_end - k_begin + BK - 1) / BK : 0;
    float acc[MI][NI];
#pragma unroll
    for (int i = 0; i < MI; ++i)
#pragma unroll
        for (int j = 0; j < NI; ++j) acc[i][j] = 0.0f;
    auto fetch = [&](int step) {
        if (step < steps) {
            const int k0 = k_begin + step * BK, s = step % kStages;
            PA::template fetch<kVecA>(As[s], g.A, g.lda, g.M, m0, k0, k_end);
            PB::template fetch<kVecB>(Bs[s], g.B, g.ldb, g.N, n0, k0, k_end);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
#pragma unroll
    for (int s = 0; s < kStages - 1; ++s) fetch(s);
    for (int step = 0; step < steps; ++step) {
        asm volatile("cp.async.wait_group %0;" ::"n"(kStages - 2) : "memory");
        __syncthreads();                                     // this step's pieces are here, and nobody reads the ones before
        fetch(step + kStages - 1);
        const float *A = As[step % kStages], *B = Bs[step % kStages];
        const int k0 = k_begin + step * BK;
#pragma unroll
        for (int k4 = 0; k4 < BK; k4 += 4) {
            float4 aq[A_KMAJOR ? MI : 1], bq[B_KMAJOR ? NI : 1];         // four of K of an operand that lies along it
            if (A_KMAJOR) {
#pragma unroll
                for (int i = 0; i < MI; ++i) aq[i] = *reinterpret_cast<const float4 *>(A + (ty + 16 * i) * PA::kLd + k4);
            }
            if (B_KMAJOR) {
#pragma unroll
                for (int j = 0; j < NI; ++j) bq[j] = *reinterpret_cast<const float4 *>(B + (tx + 16 * j) * PB::kLd + k4);
            }
#pragma unroll
            for (int kk = 0; kk < 4; ++kk) {
                float a[MI], b[NI];
#pragma unroll
                for (int i = 0; i < MI; i += A_KMAJOR ? 1 : 4) {
                    if (A_KMAJOR) {
                        a[i] = kk == 0 ? aq[i].x : (kk == 1 ? aq[i].y : (kk == 2 ? aq[i].z : aq[i].w));
                    } else {
                        const float4 q = *reinterpret_cast<const float4 *>(A + (k4 + kk) * PA::kLd + 16 * i + 4 * ty);
                        a[i] = q.x; a[i + 1] = q.y; a[i + 2] = q.z; a[i + 3] = q.w;
                    }
                }
#pragma unroll
                for (int j = 0; j < NI; j += B_KMAJOR ? 1 : 4) {
                    if (B_KMAJOR) {
                        b[j] = kk == 0 ? bq[j].x : (kk == 1 ? bq[j].y : (kk == 2 ? bq[j].z : bq[j].w));
                    } else {
                        const float4 q = *reinterpret_cast<const float4 *>(B + (k4 + kk) * PB::kLd + 16 * j + 4 * tx);
                        b[j] = q.x; b[j + 1] = q.y; b[j + 2] = q.z; b[j + 3] = q.w;
                    }
                }
                if (g.kscale) {
                    const float ks = k0 + k4 + kk < k_end ? g.kscale[k0 + k4 + kk] : 0.0f;
#pragma unroll
                    for (int i = 0; i < MI; ++i) a[i] = __fmul_rn(a[i], ks);
                }
#pragma unroll
                for (int i = 0; i < MI; ++i)
#pragma unroll
                    for (int j = 0; j < NI; ++j) acc[i][j] = fmaf(a[i], b[j], acc[i][j]);
            }
        }
    }

    float *C = g.C + (long)blockIdx.z * g.split_stride;
    bool any = false;
#pragma unroll
    for (int i = 0; i < MI; ++i) {
        const int gm = m0 + (A_KMAJOR ? ty + 16 * i : 64 * (i / 4) + 4 * ty + i % 4);
        if (gm >= g.M) continue;
        float *row = C + (long)gm * g.ldc;
#pragma unroll
        for (int j0 = 0; j0 < NI; j0 += 4) {
            // four columns: neighbours, or 16 apart
            const int step = B_KMAJOR ? 16 : 1, gn = n0 + (B_KMAJOR ? tx + 16 * j0 : 16 * j0 + 4 * tx);
            float v[4] = {acc[i][j0], acc[i][j0 + 1], acc[i][j0 + 2], acc[i][j0 + 3]};
            if (g.minuend) {
#pragma unroll
                for (int j = 0; j < 4; ++j)
                    if (gn + j * step < g.N) {
                        v[j] = __fsub_rn(g.minuend[(long)gm * g.ldm + gn + j * step], v[j]);
                        any |= fabsf(v[j]) > 1.1920928955078125e-07f;
                    }
            }
            if (!B_KMAJOR && gn + 3 < g.N && (reinterpret_cast<uintptr_t>(row + gn) % 16 == 0)) {
                *reinterpret_cast<float4 *>(row + gn) = make_float4(v[0], v[1], v[2], v[3]);
            } else {
#pragma unroll
                for (int j = 0; j < 4; ++j)
                    if (gn + j * step < g.N) row[gn + j * step] = v[j];
            }
        }
    }
    if (g.flag && __any_sync(0xffffffffu, any) && (t & 31) == 0) atomicOr(g.flag, 1u);
}

template <bool A_KMAJOR, bool B_KMAJOR, int TM, int TN, int kStages>
void launch_fp32(const GemmArgs &g, cudaStream_t stream) {
    const bool va = reinterpret_cast<uintptr_t>(g.A) % 16 == 0 && g.lda % 4 == 0, vb = reinterpret_cast<uintptr_t>(g.B) % 16 == 0 && g.ldb % 4 == 0;
    const dim3 grid((g.N + TN - 1) / TN, (g.M + TM - 1) / TM, g.splits);
    if (va && vb) launch_chained(gemm_kernel<A_KMAJOR, B_KMAJOR, TM, TN, kStages, true, true>, grid, GT, 0, stream, g);
    else if (va) launch_chained(gemm_kernel<A_KMAJOR, B_KMAJOR, TM, TN, kStages, true, false>, grid, GT, 0, stream, g);
    else if (vb) launch_chained(gemm_kernel<A_KMAJOR, B_KMAJOR, TM, TN, kStages, false, true>, grid, GT, 0, stream, g);
    else launch_chained(gemm_kernel<A_KMAJOR, B_KMAJOR, TM, TN, kStages, false, false>, grid, GT, 0, stream, g);
}
// Tiles: 128 columns unless there are at most 64; 64 rows where there are no more, or where 128 leave the device idle.  What bounds a
// small product is the way of its few steps from memory: copies that are waited for one by one and 128 x 128 tiles for everything took
// 14 to 18 us for each product of 777 x 1031 at rank 48, whole compress and decompress calls of that shape 0.79 ms, now 0.64;
// 2048 x 5120 at rank 64, whose Gram matrices run here, 1.14 and 1.08 ms.
// Wider products, reconstructions above all, take 64 x 64 tiles as well where those of 128 x 128 are no more than half the SMs: us, 128 / 64,
// 396 x 557 x 19 7.5 / 3.8, 777 x 1031 x 48 9.6 / 6.1, 777 x 1031 x 200 32.0 / 18.6, 65 x 8000 x 20 6.7 / 4.6 (63 tiles and fewer); 144 tiles, on the
// other side: 1500 x 1500 x 48 9.9 / 10.8, 2000 x 1030 x 33 10.3 / 12.3.
template <bool A_KMAJOR, bool B_KMAJOR>
void launch_fp32(const GemmArgs &g, int sm_count, cudaStream_t stream) {
    const long tiles = (long)((g.M + 127) / 128) * ((g.N + 127) / 128) * g.splits;
    if (g.N > 64 && 2 * tiles > sm_count) launch_fp32<A_KMAJOR, B_KMAJOR, 128, 128, 2>(g, stream);
    else if (g.N > 64) launch_fp32<A_KMAJOR, B_KMAJOR, 64, 64, 4>(g, stream);
    else if (g.M <= 64 || (long)((g.M + 127) / 128) * g.splits < sm_count) launch_fp32<A_KMAJOR, B_KMAJOR, 64, 64, 4>(g, stream);
    else launch_fp32<A_KMAJOR, B_KMAJOR, 128, 64, 3>(g, stream);
}

// C = sum over splits of the partial results, in split order (the order fixes the result bit for bit).  VEC = 4: four
// neighbouring elements per thread, where rows of C allow it and the result is large enough to fill the device that way.
// A thread keeps 32 (VEC 1) or 8 (VEC 4) partials in flight; rows and columns are worked out only where C has gaps.
// 48 partials of 256 x 256: 4.6 us, 4 of 4096 x 256: 7.2 us; before, with a 64-bit division per element and eight loads in
// flight, 5.8 us in the mean over a rank-256 call's fourteen reductions, 5.3 us now.
template <int VEC>
__global__ void __launch_bounds__(256) reduce_splits_kernel(const float *part, float *__restrict__ C, unsigned total, int N, long ldc,
                                                            int splits, size_t split_stride) {
    constexpr int U = VEC == 4 ? 8 : 32;
    chain_begin();
    const unsigned e = (blockIdx.x * 256u + threadIdx.x) * VEC;
    if (e >= total) return;
    float s[VEC] = {};
    const float *p = part + e;
    int z = 0;
    for (; z < splits; z += U) {
        float v[U][VEC];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            if (z + u < splits) {
                if constexpr (VEC == 4) {
                    const float4 q = *reinterpret_cast<const float4 *>(p + (size_t)(z + u) * split_stride);
                    v[u][0] = q.x; v[u][1] = q.y; v[u][2] = q.z; v[u][3] = q.w;
                } else {
                    v[u][0] = p[(size_t)(z + u) * split_stride];
                }
            }
        }
#pragma unroll
        for (int u = 0; u < U; ++u)
            if (z + u < splits) {
#pragma unroll
                for (int q = 0; q < VEC; ++q) s[q] += v[u][q];
            }
    }
    const unsigned row = ldc == N ? 0u : e / (unsigned)N, col = ldc == N ? e : e % (unsigned)N;
    float *dst = C + (size_t)row * ldc + col;
    if constexpr (VEC == 4) *reinterpret_cast<float4 *>(dst) = make_float4(s[0], s[1], s[2], s[3]);
    else dst[0] = s[0];
}

cudaError_t launch_reduce(const float *workspace, float *C, int M, int N, long ldc, int splits, int sm_count,
                          cudaStream_t stream) {
    const size_t total = (size_t)M * N;                      // (K is only split for fewer tiles than the device has slots: a few million elements)
    const bool aligned = ((reinterpret_cast<uintptr_t>(workspace) | reinterpret_cast<uintptr_t>(C)) & 15) == 0 && N % 4 == 0 && ldc % 4 == 0;
    if (aligned && total >= (size_t)sm_count * 1024)
        return launch_chained(reduce_splits_kernel<4>, (unsigned)((total / 4 + 255) / 256), 256, 0, stream, workspace, C, (unsigned)total, N, ldc, splits, total);
    return launch_chained(reduce_splits_kernel<1>, (unsigned)((total + 255) / 256), 256, 0, stream, workspace, C, (unsigned)total, N, ldc, splits, total);
}

// BSQ_GEMM_IMAGE=0 keeps the tensor-core kernel that splits B inside every CTA, =2 uses the kernel with B split
// beforehand wherever it can run (for A/B comparisons and tests); default 1: where it is faster.
int b_image_mode() {
    static const int mode = [] {
        const char *e = std::getenv("BSQ_GEMM_IMAGE");
        return e && e[0] >= '0' && e[0] <= '2' ? e[0] - '0' : 1;
    }();
    return mode;
}

// BSQ_GEMM_AIMAGE=0: the persistent product splits A in the kernel (transform warps) instead of beforehand.
bool a_image_enabled() {
    static const bool on = [] {
        const char *e = std::getenv("BSQ_GEMM_AIMAGE");
        return !(e && e[0] == '0');
    }();
    return on;
}

// BSQ_GEMM_WIDE=0: the persistent product keeps 128-column tiles (two accumulators per tile) when A is split beforehand.
bool wide_tiles_enabled() {
    static const bool on = [] {
        const char *e = std::getenv("BSQ_GEMM_WIDE");
        return !(e && e[0] == '0');
    }();
    return on;
}

// BSQ_GEMM_F16: 0 TF32 halves everywhere; 1 (default): FP16 halves where the caller gives a bound on |A|; 2: also where it
// does not (a pass over A per product).
int f16_mode() {
    static const int mode = [] {
        const char *e = std::getenv("BSQ_GEMM_F16");
        return e && e[0] >= '0' && e[0] <= '2' ? e[0] - '0' : 1;
    }();
    return mode;
}

// BSQ_GEMM_TC=0 keeps every product on the FP32 pipes (for A/B comparisons of the two kernels).
bool tensor_cores_enabled() {
    static const bool on = [] {
        const char *e = std::getenv("BSQ_GEMM_TC");
        return !(e && e[0] == '0');
    }();
    return on;
}

}  // namespace

size_t gemm_workspace_bytes(int M, int N, int max_splits) { return (size_t)M * N * max_splits * sizeof(float); }

// Picks the K split so that about two CTAs per SM are busy; partials go to `workspace` (may be null: no split).
cudaError_t gemm(bool a_kmajor, bool b_kmajor, const float *A, long lda, const float *B, long ldb, float *C, long ldc, int M,
                 int N, int K, const float *kscale, const float *minuend, long ldm, unsigned *flag, unsigned *status,
                 float *workspace, size_t workspace_bytes, int sm_count, cudaStream_t stream, const unsigned *a_absmax_bits, float b_bound,
                 bool device_full, const unsigned *b_absmax_bits) {
    return gemm_select(tensor_cores_enabled(), a_kmajor, b_kmajor, A, lda, B, ldb, C, ldc, M, N, K, kscale, minuend, ldm, flag,
                       status, workspace, workspace_bytes, sm_count, stream, a_absmax_bits, b_bound, device_full, b_absmax_bits);
}

cudaError_t gemm_select(bool allow_tensor_cores, bool a_kmajor, bool b_kmajor, const float *A, long lda, const float *B, long ldb,
                        float *C, long ldc, int M, int N, int K, const float *kscale, const float *minuend, long ldm,
                        unsigned *flag, unsigned *status, float *workspace, size_t workspace_bytes, int sm_count,
                        cudaStream_t stream, const unsigned *a_absmax_bits, float b_bound, bool device_full,
                        const unsigned *b_absmax_bits) {
    if (M <= 0 || N <= 0 || K <= 0) return cudaErrorInvalidValue;
    if (allow_tensor_cores) {
        // tensor-core path: one 128-row tile per CTA, two CTAs per SM up to N = 128; K is split so that the tiles fill
        // the SMs once
        GemmArgs t{};
        t.A = A; t.B = B; t.M = M; t.N = N; t.K = K; t.lda = lda; t.ldb = ldb;
        t.kscale = kscale; t.minuend = minuend; t.ldm = ldm;
        // N up to 256 is one tile; wider products (the reconstruction) are cut into 128-column tiles
        t.n_tile = N <= 256 ? N : 128;
        t.flag = minuend ? flag : nullptr;
        // B split beforehand when several row tiles share it and the workspace has room for its images (at its end)
        const size_t image_bytes = gemm_tc_image_bytes(N, t.n_tile, K);
        // (measured: the products are then bound by what the CTAs draw from L2, A once and B's images once per row
        // tile; that pays for tiles wider than 128 columns, where splitting B in every CTA is two thirds of the
        // staging work, and for long K)
        // (up to 128 columns the register-staged kernel with two CTAs per SM measured faster than either image kernel:
        // 67 against 80-88 us for 8192 x 128 x 4096)
        bool with_image = workspace && image_bytes + 128 <= workspace_bytes &&
                          (b_image_mode() == 2 ? M >= 256 : (b_image_mode() == 1 && M >= 512 && t.n_tile > 128 && K >= 1024));
        // a wide product (the reconstruction: N = a matrix dimension, K = the rank) in 256-column tiles, B's images
        // made once and shared by all row tiles, when the workspace has room for them; otherwise every CTA of a
        // 128-column tile splits its piece of B itself
        if (!with_image && N > 256 && workspace && b_image_mode() >= 1 && M >= 512 && K >= 64 &&
            gemm_tc_image_bytes(N, 256, K) + 128 <= workspace_bytes) {
            t.n_tile = 256;
            with_image = true;
        }
        const size_t image_room = with_image ? gemm_tc_image_bytes(N, t.n_tile, K) : 0;
        if (with_image) workspace_bytes = (workspace_bytes - image_room) & ~(size_t)127;
        // Few row tiles and a short K (a panel times a k x k factor, a Gram matrix of a short panel): narrower tiles until
        // three quarters of the SMs have one.  A CTA's time is the chain of its chunks of K whatever its width, but
        // splitting its piece of B is most of a chunk; below 64 columns, or with more CTAs than that, every tile splits A
        // once more and the time goes up again.  8192 x 256 x 256: 22.8 -> 19.0 us, 4096 x 256 x 256: 22.8 -> 16.7 us, the
        // Gram matrix of 4096 x 256 with its reduction 26.9 -> 20.8 us, 8192 x 128 x 128: 12.5 -> 11.0 us; tiles for twice
        // the SMs measured 37.3 us (14336 x 256 x 256, 24.7 with one 256-column tile per row tile).  Narrow tiles take more SM
        // time in all (4096 x 256 x 256: 32 CTAs for 22.8 us, 128 for 16.7), so not where other matrices fill the device
        // (`device_full`: eight compress calls of 4096 x 14336, rank 256, side by side: 10.30 ms with narrow tiles, 10.11 with wide ones).
        // Every width splits K alike (as often as K / 256 allows), so results are the same bits.
        if (!device_full && !with_image && !kscale && !minuend && N <= 256) {
            const int most_splits = workspace ? max(1, K / 256) : 1;
            while (t.n_tile >= 128 && ((M + 127) / 128) * ((N + t.n_tile - 1) / t.n_tile) * most_splits * 4 < sm_count * 3)
                t.n_tile = (t.n_tile / 2 + 15) / 16 * 16;
        }
        const int tiles_tc = ((M + 127) / 128) * ((N + t.n_tile - 1) / t.n_tile);
        int splits_tc = 1;
        if (with_image) {
            // A contiguous along K comes in by TMA (one CTA per SM); the other orientation is staged through registers
            t.b_image = reinterpret_cast<const float4 *>(workspace);      // placeholder for the check; set for good below
            t.k_per_split = 32;
            t.use_tma = gemm_tc_tma_usable(t, a_kmajor);
            t.b_image = nullptr;
            t.sm_count = sm_count;
            if (t.use_tma && N > 256 && (minuend || kscale || tiles_tc >= sm_count)) {       // (no K split then)
                // a wide product on the TMA-fed kernel: 128-column tiles (two accumulator sets fit tensor memory), walked
                // by a persistent grid
                t.n_tile = 128;
                t.persistent = true;
                // a small A read again by every column tile: split once beforehand too, when the workspace has the room
                // (in front of B's images; a persistent product has no K split and so no partial results there)
                const size_t a_room = (gemm_tc_a_image_bytes(M, K) + 127) & ~(size_t)127;
                if (a_kmajor && K % 4 == 0 && a_image_enabled() && workspace_bytes >= a_room && reinterpret_cast<uintptr_t>(workspace) % 128 == 0) {
                    t.a_image = workspace;
                    t.a_image_rows = (M + 127) / 128 * 128;
                    if (wide_tiles_enabled()) {
                        t.n_tile = 256;                                 // (B's images were given room for 256-column tiles above)
                        t.wide_tiles = true;
                        // ... and both operands as FP16 halves (low halves without their factor: the tile's products share
                        // one accumulator); the scales come from the largest |A kscale| and |B|, the caller's or found by a
                        // pass over each (the FP16 images take half the room, its last words hold the two maxima)
                        if (f16_mode() >= 1 && K % 8 == 0) {
                            unsigned *words = reinterpret_cast<unsigned *>(reinterpret_cast<unsigned char *>(workspace) + a_room - 256);
                            t.f16 = true;
                            t.lo_unscaled = true;
                            t.maxima_given = a_absmax_bits && b_absmax_bits;
                            t.a_absmax_bits = t.maxima_given ? a_absmax_bits : words;
                            t.b_absmax_bits = t.maxima_given ? b_absmax_bits : words + 1;
                        }
                    }
                }
            }
        }
        const int slots = (t.use_tma ? 1 : with_image ? gemm_tc_image_ctas_per_sm(t.n_tile) : (t.n_tile <= 128 ? 2 : 1)) * sm_count;
        // the FP16 form of the split (BSQ_GEMM_F16=1; =2 also without a given bound on |A|: it is then worked out here, a pass over A):
        // 256-column products on the TMA-fed kernel.  Narrower ones keep TF32 halves: 8192 x 128 x 4096 takes 67 us with them and 45 with FP16 halves, but one
        // scale for the whole of A leaves rows far below its largest element fewer bits (error over the row's own norm 4e-5 at 2^-24, 2e-2 at 2^-32;
        // 7e-7 with TF32 halves), and U and V of such rows with them.
        if (t.use_tma && !t.persistent && t.n_tile == 256 && !kscale && !minuend && workspace_bytes >= 4096 &&
            (f16_mode() == 2 || (f16_mode() == 1 && a_absmax_bits))) {
            unsigned *words = reinterpret_cast<unsigned *>(workspace);      // [0]: |B| max, [1]: |A| max when not given
            workspace += 64;
            workspace_bytes -= 256;
            t.f16 = true;
            t.b_absmax_bits = words;
            if (b_bound > 0.0f && b_bound < 1.0e30f) t.b_scale_fixed = std::exp2((float)(14 - std::ilogb(b_bound)));
            t.a_absmax_bits = a_absmax_bits;
            if (!a_absmax_bits) {
                const cudaError_t e = gemm_absmax_bits(A, lda, a_kmajor ? M : K, a_kmajor ? K : M, words + 1, stream);
                if (e != cudaSuccess) return e;
                t.a_absmax_bits = words + 1;
            }
        }
        t.boxed_c = t.wide_tiles && t.f16;
        if (t.use_tma) gemm_tc_tma_rings(t.n_tile, a_kmajor, &t.raw_stages, &t.a_stages, &t.b_stages, t.f16 && !t.a_image, t.boxed_c);
        else if (with_image) gemm_tc_image_rings(t.n_tile, &t.a_stages, &t.b_stages);
        if (workspace && !minuend && !kscale && tiles_tc < slots) {
            const int max_by_k = max(1, K / 256);             // a split below 256 of K costs more in the reduction than it gains
            const int max_by_ws = (int)(workspace_bytes / ((size_t)M * N * sizeof(float)));
            splits_tc = max(1, min(slots / tiles_tc, min(max_by_k, max_by_ws)));
        }
        if (with_image) t.b_image = reinterpret_cast<const float4 *>(reinterpret_cast<unsigned char *>(workspace) + workspace_bytes);
        t.splits = splits_tc;
        t.k_per_split = t.f16 ? ((K + splits_tc - 1) / splits_tc + 63) / 64 * 64 : ((K + splits_tc - 1) / splits_tc + 31) / 32 * 32;
        t.splits = (K + t.k_per_split - 1) / t.k_per_split;                    // no empty split
        if (t.splits > 1) {
            t.C = workspace; t.ldc = N; t.split_stride = (long)M * N;
        } else {
            t.C = C; t.ldc = ldc; t.split_stride = 0;
        }
        if (gemm_tc_eligible(t, a_kmajor, b_kmajor)) {
            cudaError_t err = gemm_tc_launch(t, a_kmajor, b_kmajor, status, stream);
            if (err != cudaSuccess || t.splits == 1) return err;
            return launch_reduce(workspace, C, M, N, ldc, t.splits, sm_count, stream);
        }
    }
    const int tiles = ((M + BM - 1) / BM) * ((N + BN - 1) / BN);
    int splits = 1;
    if (workspace && !minuend && tiles < 2 * sm_count) {
        splits = (2 * sm_count + tiles - 1) / tiles;
        const int max_by_k = (K + 4 * BK - 1) / (4 * BK);                      // at least 64 of K per split
        const int max_by_ws = (int)(workspace_bytes / ((size_t)M * N * sizeof(float)));
        splits = max(1, min(splits, min(max_by_k, max_by_ws)));
    }
    GemmArgs g{};
    g.A = A; g.B = B; g.M = M; g.N = N; g.K = K; g.lda = lda; g.ldb = ldb;
    g.kscale = kscale;
    g.splits = splits;
    g.k_per_split = ((K + splits - 1) / splits + BK - 1) / BK * BK;
    g.minuend = minuend; g.ldm = ldm; g.flag = minuend ? flag : nullptr;
    if (splits > 1) {
        g.C = workspace; g.ldc = N; g.split_stride = (long)M * N;
    } else {
        g.C = C; g.ldc = ldc; g.split_stride = 0;
    }
    if (a_kmajor && b_kmajor) launch_fp32<true, true>(g, sm_count, stream);
    else if (a_kmajor) launch_fp32<true, false>(g, sm_count, stream);
    else if (b_kmajor) launch_fp32<false, true>(g, sm_count, stream);
    else launch_fp32<false, false>(g, sm_count, stream);
    cudaError_t err = cudaGetLastError();
    if (err != cudaSuccess || splits == 1) return err;
    return launch_reduce(workspace, C, M, N, ldc, splits, sm_count, stream);
}

}  // namespace bsq

// Cholesky factor and its inverse for the Gram matrices of the randomized SVD, k <= kCholeskyBlockedMaxK (sm_100a).
//
// Stands where the reference orthonormalises with cusolverDnSgeqrf + Sorgqr (svd_lowrank_cuda.cu:196-281): a panel Y
// with Gram matrix G = Y^T Y is multiplied by R^-1, G + s I = R^T R.  The shift (s = 1e-5 max(diag G)) and a floor of
// s / 2 under every pivot keep a rank-deficient panel from dividing by zero or taking the root of a negative number:
// deficient directions just come out shorter than unit length (an all-zero panel gives R = R^-1 = 0).
//
// Work by 32 x 32 blocks, k padded to a multiple of 32 with an identity, in two kernels:
//   cholesky_factor_kernel   one CTA.  What bounds it is the chain of k pivots: while one warp factors the diagonal block of
//       step J, the other warps apply step J - 1 to the rest of the matrix; only the block that the next pivots need is
//       updated first.
//   cholesky_inverse_blocked_kernel  one CTA per block row of R^-1, which needs nothing from the other rows:
//       T_IJ = -(sum_{L=I..J-1} T_IL R_LJ) T_JJ from left to right.
// Every value is the same sum in the same order as in the one-CTA kernel that did both before, so results are too, bit for
// bit.  That one (cholesky_small_kernel) stays for k <= 64.  In launch lists of whole calls, both kernels against it: k = 256
// 78 + 26 against 138 us, k = 128 30 + 12 against 49 us.
#pragma once

#include "bsq_device.cuh"

namespace bsq {
namespace {

constexpr int kCholeskyBlockedMaxK = 256;
constexpr int kCB = 32;
constexpr int kCBB = kCB * kCB;
constexpr int kCTs = kCB + 4;
__host__ __device__ constexpr int chol_blocks(int k) { return (k + kCB - 1) / kCB; }
__host__ __device__ constexpr size_t cholesky_factor_smem_bytes(int k) {
    return ((size_t)(chol_blocks(k) * (chol_blocks(k) + 1) / 2 + chol_blocks(k)) * kCBB + kCBB + 3 * kCB + 64) * sizeof(float);
}
__device__ __forceinline__ int blk_id(int I, int J, int nb) { return I * nb - (I * (I - 1)) / 2 + (J - I); }
// Block products, 64 threads each, 4 x 4 outputs per thread (rows 4 ti .. + 3, columns 4 tc .. + 3): acc -= A^T B, both
// operands with the contraction index in rows (lda, ldb apart), which is the form in which a warp's reads of either are one
// conflict-free float4 per 16 multiply-adds.
template <int lda, int ldb>
__device__ __forceinline__ void block_mac(float (&acc)[4][4], const float *__restrict__ A, const float *__restrict__ B, int ti, int tc) {
#pragma unroll 8
    for (int l = 0; l < kCB; ++l) {
        const float4 a = *reinterpret_cast<const float4 *>(A + l * lda + 4 * ti);
        const float4 b = *reinterpret_cast<const float4 *>(B + l * ldb + 4 * tc);
        const float av[4] = {a.x, a.y, a.z, a.w}, bv[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
        for (int r = 0; r < 4; ++r)
#pragma unroll
            for (int q = 0; q < 4; ++q) acc[r][q] = fmaf(-av[r], bv[q], acc[r][q]);
    }
}
// a thread's 4 x 4 tile of a block, as four float4
__device__ __forceinline__ void tile_load(float (&acc)[4][4], const float *O, int ti, int tc) {
#pragma unroll
    for (int r = 0; r < 4; ++r) {
        const float4 v = *reinterpret_cast<const float4 *>(O + (4 * ti + r) * kCB + 4 * tc);
        acc[r][0] = v.x; acc[r][1] = v.y; acc[r][2] = v.z; acc[r][3] = v.w;
    }
}
__device__ __forceinline__ void tile_store(const float (&acc)[4][4], float *O, int ti, int tc) {
#pragma unroll
    for (int r = 0; r < 4; ++r)
        *reinterpret_cast<float4 *>(O + (4 * ti + r) * kCB + 4 * tc) = make_float4(acc[r][0], acc[r][1], acc[r][2], acc[r][3]);
}

// R (row-major k x k, upper triangular, zeros below the diagonal) from G (only read); Dinv: 1 / its diagonal, as the pivots
// were worked out.
constexpr int kCholStep = 8;                              // pivots per trip of the diagonal block's loop
constexpr int kCholThreads = 512;
__global__ void __launch_bounds__(kCholThreads) cholesky_factor_kernel(const float *__restrict__ G, int k, float *__restrict__ R,
                                                               float *__restrict__ Dinv) {
    extern __shared__ __align__(16) float sm[];
    const int nb = chol_blocks(k), nbt = nb * (nb + 1) / 2;
    float *blocks = sm;                                    // nbt blocks of 32 x 32, row-major
    float *row = blocks + (size_t)nbt * kCBB;              // block row J of R: block C at C
    float *dia = row + (size_t)nb * kCBB;                  // the diagonal block of R
    float *dinv = dia + kCBB;                              // 1 / its diagonal
    float *piv = dinv + kCB;                         // pivot rows of the diagonal block, two in turn
    float *red = piv + 2 * kCB;                            // 32 + 1
    constexpr int kParts = kCholThreads / 64;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int part = tid >> 6, ti = (tid & 63) >> 3, tc = tid & 7;         // this thread's 4 x 4 tile of its part's block
    // load block by block (four elements of a row per thread), padded with an identity; what lies below the diagonal of
    // a diagonal block is never read.  Four loads in flight per thread.
    float md = 0.0f;
    for (int b0 = 0; b0 < nbt; b0 += 8) {
        float4 v[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const int b = b0 + 2 * u + (tid >> 8);
            float x[4] = {0.0f, 0.0f, 0.0f, 0.0f};
            if (b < nbt) {
                int I = 0, rem = b;
                while (rem >= nb - I) { rem -= nb - I; ++I; }      // block (I, I + rem)
                const int i = I * kCB + ((tid & 255) >> 3), c = (I + rem) * kCB + 4 * (tid & 7);
                if ((k & 3) == 0 && i < k && c < k) {
                    const float4 g = *reinterpret_cast<const float4 *>(G + (size_t)i * k + c);
                    x[0] = g.x; x[1] = g.y; x[2] = g.z; x[3] = g.w;
                } else {
#pragma unroll
                    for (int q = 0; q < 4; ++q) x[q] = (i < k && c + q < k) ? G[(size_t)i * k + c + q] : (i == c + q ? 1.0f : 0.0f);
                }
#pragma unroll
                for (int q = 0; q < 4; ++q)
                    if (i == c + q && i < k) md = fmaxf(md, x[q]);
            }
            v[u] = make_float4(x[0], x[1], x[2], x[3]);
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const int b = b0 + 2 * u + (tid >> 8);
            if (b < nbt) reinterpret_cast<float4 *>(blocks + (size_t)b * kCBB)[tid & 255] = v[u];
        }
    }
    for (int d = 16; d > 0; d >>= 1) md = fmaxf(md, __shfl_xor_sync(0xffffffffu, md, d));
    if (lane == 0) red[warp] = md;
    __syncthreads();
    if (tid == 0) {
        float m = 0.0f;
        for (int w = 0; w < kCholThreads / 32; ++w) m = fmaxf(m, red[w]);
        red[32] = m > 0.0f ? m * 1.0e-5f : 0.0f;
    }
    // zeros below R's diagonal blocks
    for (int i = kCB + warp; i < k; i += kCholThreads / 32)
        for (int c = lane; c < i / kCB * kCB; c += 32) R[(size_t)i * k + c] = 0.0f;
    __syncthreads();
    const float shift = red[32];
    for (int i = tid; i < k; i += kCholThreads) blocks[(size_t)blk_id(i / kCB, i / kCB, nb) * kCBB + (i % kCB) * (kCB + 1)] += shift;
    __syncthreads();
    for (int J = 0; J < nb; ++J) {
        const int rest = nb - J - 1;                        // blocks to the right of the diagonal block
        if (warp == 0) {
            const float *D = blocks + (size_t)blk_id(J, J, nb) * kCBB;
            // lane c keeps column c; the scaled pivot row goes through shared memory, four of its values per load; rows move up
            // after every eight pivots, so that the loop's code is short enough to stay in the instruction cache
            float a[kCB];
#pragma unroll
            for (int i = 0; i < kCB; ++i) a[i] = D[i * kCB + lane];
            float my_inv = 0.0f;
#pragma unroll 1
            for (int j0 = 0; j0 < kCB; j0 += kCholStep) {
#pragma unroll
                for (int j = 0; j < kCholStep; ++j) {
                    float d = a[j];                         // valid in lane j0 + j
                    if (!(d > 0.5f * shift)) d = 0.5f * shift;
                    float inv = 0.0f;
                    if (d > 0.0f) {
                        inv = rsqrtf(d);
                        inv = inv * (1.5f - 0.5f * d * inv * inv);
                    }
                    const float r = d * inv;
                    const bool mine = lane == j0 + j;
                    if (mine) my_inv = inv;
                    inv = __shfl_sync(0xffffffffu, inv, j0 + j);
                    a[j] = mine ? r : a[j] * inv;
                    float *pj = piv + (j & 1) * kCB;        // the scaled pivot row from column j0 on
                    pj[(lane - j0) & 31] = a[j];
                    dia[(j0 + j) * kCB + lane] = (j0 + j <= lane) ? a[j] : 0.0f;
                    __syncwarp();
#pragma unroll
                    for (int i4 = (j + 1) / 4 * 4; i4 < kCB; i4 += 4) {
                        const float4 p = *reinterpret_cast<const float4 *>(pj + i4);
                        const float pv[4] = {p.x, p.y, p.z, p.w};
#pragma unroll
                        for (int q = 0; q < 4; ++q)
                            if (i4 + q > j) a[i4 + q] -= pv[q] * a[j];
                    }
                }
#pragma unroll
                for (int i = 0; i + kCholStep < kCB; ++i) a[i] = a[i + kCholStep];
            }
            dinv[lane] = my_inv;
            Dinv[J * kCB + lane] = my_inv;
        } else if (J > 0 && part > 0) {
            // the rest of step J - 1: G_AB -= R_{J-1,A}^T R_{J-1,B} for J <= A <= B except the diagonal block (J, J)
            const int r1 = rest + 1, pairs = r1 * (r1 + 1) / 2;
            for (int pr = part; pr < pairs; pr += kParts - 1) {
                int A = 0, rem = pr;
                while (rem >= r1 - A) { rem -= r1 - A; ++A; }
                float *O = blocks + (size_t)blk_id(J + A, J + A + rem, nb) * kCBB;
                float acc[4][4];
                tile_load(acc, O, ti, tc);
                block_mac<kCB, kCB>(acc, row + (size_t)(J + A) * kCBB, row + (size_t)(J + A + rem) * kCBB, ti, tc);
                tile_store(acc, O, ti, tc);
            }
        }
        __syncthreads();
        {   // diagonal block out
            for (int e = tid; e < kCBB; e += kCholThreads) {
                const int i = J * kCB + e / kCB, c = J * kCB + e % kCB;
                if (i < k && c < k) R[(size_t)i * k + c] = dia[e];
            }
        }
        if (rest == 0) break;
        // block row J, one thread per column: forward substitution with R_JJ^T, every value into the rows below as soon as it is known
        for (int col = tid; col < rest * kCB; col += kCholThreads) {
            const float *X = blocks + (size_t)blk_id(J, J + 1 + col / kCB, nb) * kCBB + col % kCB;
            float *Yr = row + (size_t)(J + 1 + col / kCB) * kCBB + col % kCB;
            const int c = (J + 1) * kCB + col;
            float *out = R + (size_t)J * kCB * k + c;
            float y[kCB];
#pragma unroll
            for (int i = 0; i < kCB; ++i) y[i] = X[i * kCB];
#pragma unroll
            for (int l = 0; l < kCB; ++l) {
                const float v = y[l] * dinv[l];
                Yr[l * kCB] = v;
                if (c < k && J * kCB + l < k) out[(size_t)l * k] = v;
#pragma unroll
                for (int i4 = (l + 1) / 4 * 4; i4 < kCB; i4 += 4) {
                    const float4 p = *reinterpret_cast<const float4 *>(dia + l * kCB + i4);
                    const float pv[4] = {p.x, p.y, p.z, p.w};
#pragma unroll
                    for (int q = 0; q < 4; ++q)
                        if (i4 + q > l) y[i4 + q] -= pv[q] * v;
                }
            }
        }
        __syncthreads();
        // the block of the next pivots first, two elements per thread
        {
            const float *RA = row + (size_t)(J + 1) * kCBB;
            float *O = blocks + (size_t)blk_id(J + 1, J + 1, nb) * kCBB;
            float s0 = O[warp * kCB + lane], s1 = O[(warp + 16) * kCB + lane];
#pragma unroll
            for (int l = 0; l < kCB; ++l) {
                const float x = RA[l * kCB + lane];
                s0 = fmaf(-RA[l * kCB + warp], x, s0);
                s1 = fmaf(-RA[l * kCB + warp + 16], x, s1);
            }
            O[warp * kCB + lane] = s0;
            O[(warp + 16) * kCB + lane] = s1;
        }
        __syncthreads();
    }
}

// T = R^-1 (row-major k x k, zeros below the diagonal); CTA I makes block row I.  Everything it needs of R comes in at once.
// The transposes of T_IL and of the sums are what is kept, so that every product has the form A^T B of block_mac:
//   T_IJ^T = -(T_JJ)^T S_J^T with S_J = sum_L T_IL R_LJ, and S_C^T += (R_JC)^T T_IJ^T for the columns C still to come.
constexpr int kCholInvThreads = 512;
__host__ __device__ constexpr size_t cholesky_inverse_smem_bytes(int k) {
    return (size_t)(chol_blocks(k) * (chol_blocks(k) + 1) / 2 + 2 * chol_blocks(k)) * kCBB * sizeof(float) + kCB * kCTs * sizeof(float);
}
__global__ void __launch_bounds__(kCholInvThreads, 1) cholesky_inverse_blocked_kernel(const float *__restrict__ R, const float *__restrict__ Dinv, int k, float *__restrict__ T) {
    extern __shared__ __align__(16) float sm[];
    const int nb = chol_blocks(k), I = blockIdx.x, n = nb - I;           // blocks I .. nb - 1 of rows and columns
    float *rb = sm;                                        // block (L, C) of R, L, C counted from I: at blk_id(L, C, n)
    float *tj = rb + (size_t)(n * (n + 1) / 2) * kCBB;     // T_JJ, J counted from I
    float *sum = tj + (size_t)n * kCBB;                    // -S_C^T
    float *tij = sum + (size_t)n * kCBB;                   // T_IJ^T, rows kCTs apart
    const int tid = threadIdx.x, part = tid >> 6, ti = (tid & 63) >> 3, tc = tid & 7;
#pragma unroll 4
    for (int b = tid >> 8; b < n * (n + 1) / 2; b += kCholInvThreads / 256) {
        int L = 0, rem = b;
        while (rem >= n - L) { rem -= n - L; ++L; }
        const int i = (I + L) * kCB + ((tid & 255) >> 3), c = (I + L + rem) * kCB + 4 * (tid & 7);
        float x[4] = {0.0f, 0.0f, 0.0f, 0.0f};
        if ((k & 3) == 0 && i < k && c < k) {
            const float4 g = *reinterpret_cast<const float4 *>(R + (size_t)i * k + c);
            x[0] = g.x; x[1] = g.y; x[2] = g.z; x[3] = g.w;
        } else {
#pragma unroll
            for (int q = 0; q < 4; ++q)
                if (i < k && c + q < k) x[q] = R[(size_t)i * k + c + q];
#pragma unroll
            for (int q = 0; q < 4; ++q)
                if (i == c + q && i >= k) x[q] = 1.0f;          // padding: an identity
        }
        reinterpret_cast<float4 *>(rb + (size_t)b * kCBB)[tid & 255] = make_float4(x[0], x[1], x[2], x[3]);
    }
    for (int i = tid >> 5; i < kCB; i += kCholInvThreads / 32)           // zeros left of the diagonal block
        for (int c = tid & 31; c < I * kCB; c += 32)
            if (I * kCB + i < k) T[(size_t)(I * kCB + i) * k + c] = 0.0f;
    __syncthreads();
    // the diagonal blocks' inverses, one warp each: lane c keeps column c, rows from the bottom up
    if ((tid >> 5) < n) {
        const int b = tid >> 5, lane = tid & 31;
        const float *D = rb + (size_t)blk_id(b, b, n) * kCBB;
        float t[kCB];
        const float my_inv = Dinv[(I + b) * kCB + lane];
#pragma unroll
        for (int i = kCB - 1; i >= 0; --i) {
            float acc = (lane == i) ? 1.0f : 0.0f;
#pragma unroll
            for (int l4 = (i + 1) / 4 * 4; l4 < kCB; l4 += 4) {
                const float4 p = *reinterpret_cast<const float4 *>(D + i * kCB + l4);
                const float pv[4] = {p.x, p.y, p.z, p.w};
#pragma unroll
                for (int q = 0; q < 4; ++q)
                    if (l4 + q > i) acc -= pv[q] * t[l4 + q];
            }
            const float inv = __shfl_sync(0xffffffffu, my_inv, i);
            t[i] = (lane >= i) ? acc * inv : 0.0f;
        }
#pragma unroll
        for (int i = 0; i < kCB; ++i) tj[(size_t)b * kCBB + i * kCB + lane] = t[i];
    }
    __syncthreads();
    for (int J = 0; J < n; ++J) {
        // T_IJ^T = (T_JJ)^T (-S_J^T), two elements per thread
        {
            const int i = tid & 31, c0 = tid >> 5;          // elements (c0, i) and (c0 + 16, i) of the transposed block
            float o0 = 0.0f, o1 = 0.0f;
            if (J == 0) {
                o0 = tj[i * kCB + c0];
                o1 = tj[i * kCB + c0 + 16];
            } else {
                const float *A = tj + (size_t)J * kCBB, *B = sum + (size_t)J * kCBB;
#pragma unroll 8
                for (int l = 0; l < kCB; ++l) {
                    const float b = B[l * kCB + i];
                    o0 = fmaf(A[l * kCB + c0], b, o0);
                    o1 = fmaf(A[l * kCB + c0 + 16], b, o1);
                }
            }
            tij[c0 * kCTs + i] = o0;
            tij[(c0 + 16) * kCTs + i] = o1;
        }
        __syncthreads();
        // out, a row of T at a time (its column index is the row index of the transposed block)
        for (int r = tid >> 5; r < kCB; r += kCholInvThreads / 32) {
            const int i = I * kCB + r, c = (I + J) * kCB + (tid & 31);
            if (i < k && c < k) T[(size_t)i * k + c] = tij[(tid & 31) * kCTs + r];
        }
        for (int C = J + 1 + part; C < n; C += kCholInvThreads / 64) {
            float acc[4][4] = {};
            float *S = sum + (size_t)C * kCBB;
            if (J > 0) tile_load(acc, S, ti, tc);
            block_mac<kCB, kCTs>(acc, rb + (size_t)blk_id(J, C, n) * kCBB, tij, ti, tc);
            tile_store(acc, S, ti, tc);
        }
        __syncthreads();                                   // the sums of the next column are whole, tij may be overwritten
    }
}

// Sixteen 32 x 32 block products at a time: 64 threads per product, 4 x 4 outputs per thread (rows 4 ti .. + 3,
// columns 4 tc .. + 3), operands read as float4: 2 shared-memory loads per 16 multiply-adds (with 2 x 2 outputs
// per thread the loads, not the arithmetic, filled the issue slots of the one SM this kernel runs on).
//   out -= A^T B  (AT = true:  A, B hold the contraction index in rows)
//   out += A B    (AT = false: A holds it in columns)
template <bool AT>
__device__ __forceinline__ void block_mac_any(float (&acc)[4][4], const float *__restrict__ A, const float *__restrict__ B, int ti, int tc) {
    if (AT) {
#pragma unroll 4
        for (int l = 0; l < kCB; ++l) {
            const float4 a = *reinterpret_cast<const float4 *>(A + l * kCB + 4 * ti);
            const float4 b = *reinterpret_cast<const float4 *>(B + l * kCB + 4 * tc);
            const float av[4] = {a.x, a.y, a.z, a.w}, bv[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
            for (int r = 0; r < 4; ++r)
#pragma unroll
                for (int q = 0; q < 4; ++q) acc[r][q] = fmaf(-av[r], bv[q], acc[r][q]);
        }
    } else {
#pragma unroll 2
        for (int l0 = 0; l0 < kCB; l0 += 4) {
            float4 a[4];
#pragma unroll
            for (int r = 0; r < 4; ++r) a[r] = *reinterpret_cast<const float4 *>(A + (4 * ti + r) * kCB + l0);
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const float4 b = *reinterpret_cast<const float4 *>(B + (l0 + u) * kCB + 4 * tc);
                const float bv[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
                for (int r = 0; r < 4; ++r) {
                    const float ar = u == 0 ? a[r].x : (u == 1 ? a[r].y : (u == 2 ? a[r].z : a[r].w));
#pragma unroll
                    for (int q = 0; q < 4; ++q) acc[r][q] += ar * bv[q];
                }
            }
        }
    }
}
__device__ __forceinline__ void tile_store_signed(const float (&acc)[4][4], float *O, int ti, int tc, float sign) {
#pragma unroll
    for (int r = 0; r < 4; ++r)
        *reinterpret_cast<float4 *>(O + (4 * ti + r) * kCB + 4 * tc) =
            make_float4(sign * acc[r][0], sign * acc[r][1], sign * acc[r][2], sign * acc[r][3]);
}

// Up to kCholeskySmallMaxK columns, where a second launch costs more than it spreads (k = 64: 19 us here, 15 + 8 in the two
// kernels above; k = 32: 11 against 6.5 + 6.5), one CTA factors and inverts: forward substitutions per block row, then the
// inverse block column by block column.
constexpr int kCholeskySmallMaxK = 64;
__host__ __device__ constexpr size_t cholesky_small_smem_bytes(int k) {
    // packed blocks + inverted diagonal blocks + one temporary block column + 1 / diagonal + scalars
    return ((size_t)(chol_blocks(k) * (chol_blocks(k) + 1) / 2 + 2 * chol_blocks(k)) * kCB * kCB + (size_t)chol_blocks(k) * kCB + 64) *
           sizeof(float);
}
__global__ void __launch_bounds__(1024) cholesky_small_kernel(const float *__restrict__ G, int k, float *__restrict__ T,
                                                                        float *__restrict__ Rcpy) {
    extern __shared__ __align__(16) float sm[];
    const int nb = chol_blocks(k), nbt = nb * (nb + 1) / 2;
    float *blocks = sm;                                    // nbt blocks of 32 x 32, row-major
    float *tinv = blocks + (size_t)nbt * kCB * kCB;        // nb inverted diagonal blocks
    float *tmp = tinv + (size_t)nb * kCB * kCB;            // nb blocks: one block column of partial products
    float *dinv = tmp + (size_t)nb * kCB * kCB;            // 1 / R(i, i)
    float *red = dinv + nb * kCB;                          // 32 + 1
    const int tid = threadIdx.x, nt = blockDim.x, lane = tid & 31, warp = tid >> 5, nwarps = nt >> 5;
    const int bi = tid >> 5, bc = tid & 31;               // this thread's element of a block when the CTA walks blocks
    const int part = tid >> 6, ti = (tid & 63) >> 3, tc = tid & 7;         // ... and its 4 x 4 tile of its sixteenth's block
    // load block by block (row bi, column bc of each), padded with an identity; what lies below the diagonal of a
    // diagonal block is never read.  Four blocks per trip, so that four global loads are in flight per thread.
    float md = 0.0f;
    for (int b0 = 0; b0 < nbt; b0 += 4) {
        float v[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const int b = b0 + u;
            v[u] = 0.0f;
            if (b < nbt) {
                int I = 0, rem = b;
                while (rem >= nb - I) { rem -= nb - I; ++I; }      // block (I, I + rem)
                const int i = I * kCB + bi, c = (I + rem) * kCB + bc;
                v[u] = (i == c) ? 1.0f : 0.0f;
                if (i < k && c < k) v[u] = G[(size_t)i * k + c];
                if (i == c && i < k) md = fmaxf(md, v[u]);
            }
        }
#pragma unroll
        for (int u = 0; u < 4; ++u)
            if (b0 + u < nbt) blocks[(size_t)(b0 + u) * kCB * kCB + tid] = v[u];
    }
    for (int d = 16; d > 0; d >>= 1) md = fmaxf(md, __shfl_xor_sync(0xffffffffu, md, d));
    if (lane == 0) red[warp] = md;
    __syncthreads();
    if (tid == 0) {
        float m = 0.0f;
        for (int w = 0; w < nwarps; ++w) m = fmaxf(m, red[w]);
        red[32] = m > 0.0f ? m * 1.0e-5f : 0.0f;
    }
    __syncthreads();
    const float shift = red[32];
    for (int i = tid; i < k; i += nt) blocks[(size_t)blk_id(i / kCB, i / kCB, nb) * kCB * kCB + (i % kCB) * (kCB + 1)] += shift;
    __syncthreads();

    for (int J = 0; J < nb; ++J) {
        float *D = blocks + (size_t)blk_id(J, J, nb) * kCB * kCB;
        if (warp == 0) {                                    // diagonal block: lane c keeps column c
            float a[kCB];
#pragma unroll
            for (int i = 0; i < kCB; ++i) a[i] = D[i * kCB + lane];
            float my_inv = 0.0f;
#pragma unroll
            for (int j = 0; j < kCB; ++j) {
                float d = __shfl_sync(0xffffffffu, a[j], j);
                if (!(d > 0.5f * shift)) d = 0.5f * shift;
                // the 32 pivots of a block are one dependent chain: reciprocal square root from the special-function
                // unit plus one Newton step (a relative error of ~1e-7 in R(j, j) and 1 / R(j, j) alike) instead of
                // an IEEE square root followed by an IEEE division
                float inv = 0.0f;
                if (d > 0.0f) {
                    inv = rsqrtf(d);
                    inv = inv * (1.5f - 0.5f * d * inv * inv);
                }
                const float r = d * inv;
                a[j] = (lane == j) ? r : a[j] * inv;
                if (lane == j) my_inv = inv;
#pragma unroll
                for (int i = j + 1; i < kCB; ++i) {
                    const float rji = __shfl_sync(0xffffffffu, a[j], i);
                    a[i] -= rji * a[j];
                }
            }
#pragma unroll
            for (int i = 0; i < kCB; ++i) D[i * kCB + lane] = (i <= lane) ? a[i] : 0.0f;
            dinv[J * kCB + lane] = my_inv;
        }
        __syncthreads();
        // block row J: one thread per column, forward substitution with R_JJ^T
        for (int col = tid; col < (nb - J - 1) * kCB; col += nt) {
            float *X = blocks + (size_t)blk_id(J, J + 1 + col / kCB, nb) * kCB * kCB + col % kCB;
            float y[kCB];
#pragma unroll
            for (int i = 0; i < kCB; ++i) {
                float acc = X[i * kCB];
#pragma unroll
                for (int l = 0; l < i; ++l) acc -= D[l * kCB + i] * y[l];
                y[i] = acc * dinv[J * kCB + i];
            }
#pragma unroll
            for (int i = 0; i < kCB; ++i) X[i * kCB] = y[i];
        }
        __syncthreads();
        // trailing blocks (A, B), J < A <= B: G_AB -= R_JA^T R_JB, sixteen blocks per trip
        {
            const int rest = nb - J - 1, pairs = rest * (rest + 1) / 2;
            for (int pr0 = 0; pr0 < pairs; pr0 += 16) {
                const int pr = pr0 + part;
                if (pr < pairs) {
                    int A = 0, rem = pr;
                    while (rem >= rest - A) { rem -= rest - A; ++A; }
                    const int B = A + rem;
                    const float *RA = blocks + (size_t)blk_id(J, J + 1 + A, nb) * kCB * kCB;
                    const float *RB = blocks + (size_t)blk_id(J, J + 1 + B, nb) * kCB * kCB;
                    float *O = blocks + (size_t)blk_id(J + 1 + A, J + 1 + B, nb) * kCB * kCB;
                    float acc[4][4];
                    tile_load(acc, O, ti, tc);
                    block_mac_any<true>(acc, RA, RB, ti, tc);
                    tile_store_signed(acc, O, ti, tc, 1.0f);
                }
            }
        }
        __syncthreads();
    }
    // R out and the zeros below the diagonal of R and T, block by block; the diagonal blocks' inverses, one warp each
    for (int I = 0; I < nb; ++I) {
        for (int Jb = 0; Jb < nb; ++Jb) {
            const int i = I * kCB + bi, c = Jb * kCB + bc;
            if (i < k && c < k) {
                const size_t e = (size_t)i * k + c;
                if (c < i) {
                    if (T) T[e] = 0.0f;
                    if (Rcpy) Rcpy[e] = 0.0f;
                } else if (Rcpy) {
                    Rcpy[e] = blocks[(size_t)blk_id(I, Jb, nb) * kCB * kCB + tid];
                }
            }
        }
    }
    if (!T) return;                                         // only the factor was wanted (uniform over the CTA)
    if (warp < nb) {
        const float *D = blocks + (size_t)blk_id(warp, warp, nb) * kCB * kCB;
        float a[kCB], t[kCB];
#pragma unroll
        for (int i = 0; i < kCB; ++i) { a[i] = D[i * kCB + lane]; t[i] = 0.0f; }
        const float my_inv = dinv[warp * kCB + lane];
#pragma unroll
        for (int i = kCB - 1; i >= 0; --i) {
            float acc = (lane == i) ? 1.0f : 0.0f;
#pragma unroll
            for (int l = i + 1; l < kCB; ++l) acc -= __shfl_sync(0xffffffffu, a[i], l) * t[l];
            const float inv = __shfl_sync(0xffffffffu, my_inv, i);
            t[i] = (lane >= i) ? acc * inv : 0.0f;
        }
#pragma unroll
        for (int i = 0; i < kCB; ++i) tinv[(size_t)warp * kCB * kCB + i * kCB + lane] = t[i];
    }
    __syncthreads();
    // block column J of T, from the left: needs T_IL for L < J (already in place) and R_LJ (still in place)
    for (int J = 1; J < nb; ++J) {
        for (int I0 = 0; I0 < J; I0 += 16) {
            const int I = I0 + part;
            if (I < J) {
                float acc[4][4] = {};
                for (int L = I; L < J; ++L) {
                    const float *TL = (L == I) ? tinv + (size_t)I * kCB * kCB : blocks + (size_t)blk_id(I, L, nb) * kCB * kCB;
                    block_mac_any<false>(acc, TL, blocks + (size_t)blk_id(L, J, nb) * kCB * kCB, ti, tc);
                }
                tile_store_signed(acc, tmp + (size_t)I * kCB * kCB, ti, tc, 1.0f);
            }
        }
        __syncthreads();
        const float *TJ = tinv + (size_t)J * kCB * kCB;
        for (int I0 = 0; I0 < J; I0 += 16) {
            const int I = I0 + part;
            if (I < J) {
                float acc[4][4] = {};
                block_mac_any<false>(acc, tmp + (size_t)I * kCB * kCB, TJ, ti, tc);
                tile_store_signed(acc, blocks + (size_t)blk_id(I, J, nb) * kCB * kCB, ti, tc, -1.0f);
            }
        }
        __syncthreads();
    }
    for (int I = 0; I < nb; ++I) {
        for (int Jb = I; Jb < nb; ++Jb) {
            const int i = I * kCB + bi, c = Jb * kCB + bc;
            if (i < k && c < k && c >= i) {
                const float *src = (I == Jb) ? tinv + (size_t)I * kCB * kCB : blocks + (size_t)blk_id(I, Jb, nb) * kCB * kCB;
                T[(size_t)i * k + c] = src[tid];
            }
        }
    }
}

}  // namespace
}  // namespace bsq

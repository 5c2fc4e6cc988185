// Cholesky factor and its inverse for the Gram matrices of the randomized SVD, k <= kCholeskyBlockedMaxK (sm_100a); above 32 columns
// usually by way of bsq_cholesky_cluster.cuh.
//
// Stands where the reference orthonormalises with cusolverDnSgeqrf + Sorgqr (svd_lowrank_cuda.cu:196-281): a panel Y
// with Gram matrix G = Y^T Y is multiplied by R^-1, G + s I = R^T R.  The shift (s = 1e-5 max(diag G)) and a floor of
// s / 2 under every pivot keep a rank-deficient panel from dividing by zero or taking the root of a negative number:
// deficient directions just come out shorter than unit length (an all-zero panel gives R = R^-1 = 0).
//
// Work by 32 x 32 blocks in shared memory, k padded to a multiple of 32 with an identity.  What bounds it is the chain of k pivots:
// root, shuffle and multiply-add of about 70 clocks each; everything else is arranged around the warp that walks it.
//   * That warp has a scheduler (almost) to itself.  It takes the next pivot's row by shuffle and the rows below through shared memory,
//     behind its own shuffles: 105 clocks per pivot (a round trip through shared memory on the chain, roots that scale for
//     subnormal arguments and stores to global memory in between: 230).
//   * The block row is a forward substitution right behind the pivots, eight at a time (named barriers), the block of the next
//     pivots is updated right behind that, and all other updates run beside the chain.  From about 200 columns on those are
//     what an SM's multiply-adds take: 53 us at 256 columns for 8 blocks, 16 us at 128 for 4.
//   * R and the inverses of its diagonal blocks go out block row by block row, and other CTAs make the rows of the inverse
//     from them while the factor goes on: T_IJ = -(sum_{L=I..J-1} T_IL R_LJ) T_JJ from left to right.
// Every value is the same sum in the same order whatever the number of CTAs.  Above 32 columns the kernel of bsq_cholesky_cluster.cuh takes the
// place of this one wherever its cluster can be placed; both share what is above cholesky_factor.  Back to back, factor and inverse, this
// kernel / that one, us: k = 256 71 / 32, 128 31.5 / 20, 64 14.4 / 11.2, 48 15.3 / 10.7; up to 32 columns 7.
#pragma once

#include "bsq_device.cuh"

namespace bsq {
namespace {

constexpr int kCholeskyBlockedMaxK = 256;
constexpr int kCB = 32;
constexpr int kCBB = kCB * kCB;
constexpr int kCTs = kCB + 4;
__host__ __device__ constexpr int chol_blocks(int k) { return (k + kCB - 1) / kCB; }
__device__ __forceinline__ int blk_id(int I, int J, int nb) { return I * nb - (I * (I - 1)) / 2 + (J - I); }
// 16 bytes of shared memory; volatile, so that the loads of a step stay in front of the work that is meant to hide them
__device__ __forceinline__ float4 lds4(unsigned at) {
    float4 v;
    asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(at) : "memory");
    return v;
}
// Two FP32 multiply-adds per instruction; each half rounds as the scalar instruction does.
__device__ __forceinline__ float2 chol_fma2(float2 a, float2 b, float2 c) {
    float2 r;
    asm volatile("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(reinterpret_cast<unsigned long long &>(r))
                 : "l"(reinterpret_cast<unsigned long long &>(a)), "l"(reinterpret_cast<unsigned long long &>(b)),
                 "l"(reinterpret_cast<unsigned long long &>(c)));
    return r;
}
// Block products, acc -= A^T B: both operands with the contraction index in rows (lda, ldb apart).  A 16-byte load of shared memory
// takes four clocks of the SM however many lanes read the same, so what bounds these is loads per multiply-add: 16 threads take
// a block, 8 x 8 outputs each (rows 8 ti .. + 7, columns 8 tc .. + 7), four loads per 64 multiply-adds.  The next row is on its
// way while one is multiplied.
struct MacRow {
    float4 a0, a1, b0, b1;
};
__device__ __forceinline__ void mac_fetch(MacRow &m, unsigned A, unsigned B) {
    m.a0 = lds4(A);
    m.a1 = lds4(A + 16);
    m.b0 = lds4(B);
    m.b1 = lds4(B + 16);
}
__device__ __forceinline__ void mac_row(float2 (&acc)[8][4], const MacRow &m) {
    const float av[8] = {m.a0.x, m.a0.y, m.a0.z, m.a0.w, m.a1.x, m.a1.y, m.a1.z, m.a1.w};
    const float2 bv[4] = {make_float2(m.b0.x, m.b0.y), make_float2(m.b0.z, m.b0.w), make_float2(m.b1.x, m.b1.y), make_float2(m.b1.z, m.b1.w)};
#pragma unroll
    for (int r = 0; r < 8; ++r)
#pragma unroll
        for (int q = 0; q < 4; ++q) acc[r][q] = chol_fma2(make_float2(-av[r], -av[r]), bv[q], acc[r][q]);
}
template <int lda, int ldb>
__device__ __forceinline__ void block_mac(float2 (&acc)[8][4], const float *A_, const float *B_, int ti, int tc) {
    unsigned A = smem_u32(A_ + 8 * ti), B = smem_u32(B_ + 8 * tc);
    MacRow m0, m1;
    mac_fetch(m0, A, B);
#pragma unroll 2
    for (int l = 0; l < kCB; l += 2) {
        mac_fetch(m1, A + 4 * lda, B + 4 * ldb);
        mac_row(acc, m0);
        if (l + 2 < kCB) {
            A += 8 * lda;
            B += 8 * ldb;
        }
        mac_fetch(m0, A, B);                                // (the last trip reads a row again)
        mac_row(acc, m1);
    }
}
// a thread's 8 x 8 tile of a block
__device__ __forceinline__ void tile_load(float2 (&acc)[8][4], const float *O, int ti, int tc) {
#pragma unroll
    for (int r = 0; r < 8; ++r)
#pragma unroll
        for (int q = 0; q < 4; q += 2) {
            const float4 v = *reinterpret_cast<const float4 *>(O + (8 * ti + r) * kCB + 8 * tc + 2 * q);
            acc[r][q] = make_float2(v.x, v.y);
            acc[r][q + 1] = make_float2(v.z, v.w);
        }
}
__device__ __forceinline__ void tile_store(const float2 (&acc)[8][4], float *O, int ti, int tc) {
#pragma unroll
    for (int r = 0; r < 8; ++r)
#pragma unroll
        for (int q = 0; q < 4; q += 2)
            *reinterpret_cast<float4 *>(O + (8 * ti + r) * kCB + 8 * tc + 2 * q) = make_float4(acc[r][q].x, acc[r][q].y, acc[r][q + 1].x, acc[r][q + 1].y);
}
// The same by 64 threads, 4 x 4 outputs each, where there are more warps than blocks: a third of the time for twice the loads.
// kRows rows of the product.
template <int lda, int ldb, int kRows>
__device__ __forceinline__ void block_mac_wide(float2 (&acc)[4][2], const float *A_, const float *B_, int t) {
    const unsigned A = smem_u32(A_ + 4 * (t >> 3)), B = smem_u32(B_ + 4 * (t & 7));
    constexpr int kG = 8;
#pragma unroll
    for (int l0 = 0; l0 < kRows; l0 += kG) {
        float4 x[kG], y[kG];
#pragma unroll
        for (int l = 0; l < kG; ++l) {
            x[l] = lds4(A + (l0 + l) * lda * 4);
            y[l] = lds4(B + (l0 + l) * ldb * 4);
        }
#pragma unroll
        for (int l = 0; l < kG; ++l) {
            const float av[4] = {x[l].x, x[l].y, x[l].z, x[l].w};
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                const float2 n = make_float2(-av[r], -av[r]);
                acc[r][0] = chol_fma2(n, make_float2(y[l].x, y[l].y), acc[r][0]);
                acc[r][1] = chol_fma2(n, make_float2(y[l].z, y[l].w), acc[r][1]);
            }
        }
    }
}
__device__ __forceinline__ void tile_load_wide(float2 (&acc)[4][2], const float *O, int t) {
#pragma unroll
    for (int r = 0; r < 4; ++r) {
        const float4 v = *reinterpret_cast<const float4 *>(O + (4 * (t >> 3) + r) * kCB + 4 * (t & 7));
        acc[r][0] = make_float2(v.x, v.y);
        acc[r][1] = make_float2(v.z, v.w);
    }
}
__device__ __forceinline__ void tile_store_wide(const float2 (&acc)[4][2], float *O, int t) {
#pragma unroll
    for (int r = 0; r < 4; ++r)
        *reinterpret_cast<float4 *>(O + (4 * (t >> 3) + r) * kCB + 4 * (t & 7)) = make_float4(acc[r][0].x, acc[r][0].y, acc[r][1].x, acc[r][1].y);
}

// Named CTA barriers: `threads` threads in all, whole warps.
__device__ __forceinline__ void bar_sync(int id, int threads) { asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory"); }
__device__ __forceinline__ void bar_arrive(int id, int threads) { asm volatile("bar.arrive %0, %1;" ::"r"(id), "r"(threads) : "memory"); }
__device__ __forceinline__ void copy16_async(void *dst_smem, const void *src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(dst_smem)), "l"(src) : "memory");
}

// The dynamic shared memory of the kernel below: functions that are not inlined take offsets into it, so that their accesses are
// known to be to shared memory.
__device__ __forceinline__ float *chol_smem() {
    extern __shared__ __align__(16) float sm[];
    return sm;
}

constexpr int kCholStep = 8;                              // pivots per trip of the loops below
constexpr int kCholThreads = 384;
constexpr int kCholWarps = kCholThreads / 32;
constexpr int kCholWorkers = kCholWarps / 4 * 3, kCholPanel = 4, kCholTrail = kCholWorkers - kCholPanel;       // warps beside the pivots' scheduler: for the block row, for updates that can wait
// What the CTAs of one launch share in global memory; all zero between launches (the last CTA to leave clears it).
struct CholeskySync {
    unsigned ticket;                                       // roles are taken in the order in which CTAs start
    unsigned rows;                                         // block rows of R that are out
    unsigned done;
};
__host__ __device__ constexpr size_t cholesky_blocked_smem_bytes(int k) {
    // the factor's blocks (the inverse: a row of blocks, sums, two blocks), the diagonal block and 1 / diagonal twice, scalars
    return ((size_t)(chol_blocks(k) * (chol_blocks(k) + 1) / 2 > 2 * chol_blocks(k) + 2 ? chol_blocks(k) * (chol_blocks(k) + 1) / 2 : 2 * chol_blocks(k) + 2) * kCBB +
            2 * (kCBB + 3 * kCB) + kCB * kCTs + 2 * kCB + 64) *
           sizeof(float);
}

// A step of the elimination for the 32 rows that a lane keeps of its column (pairs of rows): every row i > j loses row[i] v.
// row: the step's row of the diagonal block of R, fetched before what is to hide the way.
struct StepRow {
    float4 q[kCB / 4];
};
__device__ __forceinline__ void step_fetch(StepRow &s, unsigned row, int j) {
#pragma unroll
    for (int i4 = (j + 1) / 4; i4 < kCB / 4; ++i4) s.q[i4] = lds4(row + 16 * i4);
}
__device__ __forceinline__ void eliminate(float2 (&y)[kCB / 2], const StepRow &s, int j, float v) {
    const float2 v2 = make_float2(-v, -v);
#pragma unroll
    for (int i4 = (j + 1) / 4 * 4; i4 < kCB; i4 += 4) {
        const float4 p = s.q[i4 / 4];
        if (i4 > j) y[i4 / 2] = chol_fma2(make_float2(p.x, p.y), v2, y[i4 / 2]);
        else if (i4 + 1 > j) y[i4 / 2].y = fmaf(p.y, -v, y[i4 / 2].y);
        if (i4 + 2 > j) y[i4 / 2 + 1] = chol_fma2(make_float2(p.z, p.w), v2, y[i4 / 2 + 1]);
        else if (i4 + 3 > j) y[i4 / 2 + 1].y = fmaf(p.w, -v, y[i4 / 2 + 1].y);
    }
}
__device__ __forceinline__ float row_of(const float2 (&y)[kCB / 2], int j) { return j & 1 ? y[j / 2].y : y[j / 2].x; }
__device__ __forceinline__ void rows_up(float2 (&y)[kCB / 2]) {
#pragma unroll
    for (int i = 0; i + kCholStep / 2 < kCB / 2; ++i) y[i] = y[i + kCholStep / 2];
}
__device__ __forceinline__ float chol_rsqrt_ftz(float x) {
    float r;
    asm volatile("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

// The pivots of a diagonal block, one warp: lane c keeps column c.  Row j of R goes to dia, 1 / R(j, j) to dinv; every kCholStep rows the
// warps of the block row (panel threads with this one) are let on.  The row in front of dia is zero.
// kNormal: the floor under the pivots is a normal number, so every pivot is, and its root needs no scaling.
// Rows move up after every kCholStep pivots, in a lane and in what is read of dia.  steps: times kCholStep pivots.
template <bool kNormal>
__device__ __forceinline__ void factor_diagonal(int at_d, int at_dia, int at_dinv, float half, int panel, int steps = kCB / kCholStep) {
    const float *D = chol_smem() + at_d;
    float *dia = chol_smem() + at_dia, *dinv = chol_smem() + at_dinv;
    const int lane = threadIdx.x & 31;
    float2 a[kCB / 2];
#pragma unroll
    for (int i = 0; i < kCB / 2; ++i) a[i] = make_float2(D[2 * i * kCB + lane], D[(2 * i + 1) * kCB + lane]);
    float d = a[0].x, v = 0.0f;                             // the next pivot before its root, valid in its lane
    const unsigned dia_at = smem_u32(dia);
#pragma unroll 1
    for (int j0 = 0; j0 < kCholStep * steps; j0 += kCholStep) {
#pragma unroll
        for (int j = 0; j < kCholStep; ++j) {
            d = fmaxf(d, half);                             // (a NaN as well)
            float inv = kNormal ? chol_rsqrt_ftz(d) : rsqrtf(d);
            // row j of the other columns takes what the pivot before takes from it by shuffle, the rows below by way of shared memory
            // behind this pivot's own shuffle: neither waits for more than it needs
            const float p = __shfl_sync(kFullMask, v, j0 + j);
            StepRow before;
            step_fetch(before, dia_at + ((j0 + j - 1) * kCB + j0) * 4, j);
            if (j & 1) a[j / 2].y = fmaf(p, -v, a[j / 2].y);
            else a[j / 2].x = fmaf(p, -v, a[j / 2].x);
            const bool mine = lane == j0 + j;
            const float aj = mine ? d : row_of(a, j);
            inv = inv * (1.5f - 0.5f * d * inv * inv);
            if (!kNormal) inv = d > 0.0f ? inv : 0.0f;
            const float inv_all = __shfl_sync(kFullMask, inv, j0 + j);
            eliminate(a, before, j, v);
            v = aj * inv_all;
            d = fmaf(-v, v, row_of(a, j + 1));              // the next pivot, in its lane
            dia[(j0 + j) * kCB + lane] = v;
            if (mine) dinv[j0 + j] = inv;
            __syncwarp();
        }
        if (panel > 32) bar_arrive(1 + j0 / kCholStep, panel);
        rows_up(a);
    }
}

// kCols columns of a block row per thread (in blocks beside one another): forward substitution with R_JJ^T, behind the pivots (await(s)
// waits for the s-th eight).  X: the columns, in place.
template <int kCols, class Await>
__device__ __forceinline__ void block_row(int at_x, int at_dia, int at_dinv, bool first, Await await) {
    float *X = chol_smem() + at_x;
    const unsigned dia_at = smem_u32(chol_smem() + at_dia), dinv_at = smem_u32(chol_smem() + at_dinv);
    float2 y[kCols][kCB / 2];
#pragma unroll
    for (int u = 0; u < kCols; ++u)
#pragma unroll
        for (int i = 0; i < kCB / 2; ++i) y[u][i] = make_float2(X[u * kCBB + 2 * i * kCB], X[u * kCBB + (2 * i + 1) * kCB]);
#pragma unroll 1
    for (int j0 = 0; j0 < kCB; j0 += kCholStep) {
        await(j0 / kCholStep);
        const float4 d0 = lds4(dinv_at + 4 * j0), d1 = lds4(dinv_at + 4 * j0 + 16);
        const float dv[kCholStep] = {d0.x, d0.y, d0.z, d0.w, d1.x, d1.y, d1.z, d1.w};
#pragma unroll
        for (int j = 0; j < kCholStep; ++j) {
            StepRow now;
            step_fetch(now, dia_at + ((j0 + j) * kCB + j0) * 4, j);
#pragma unroll
            for (int u = 0; u < kCols; ++u) {
                const float v = row_of(y[u], j) * dv[j];
                X[u * kCBB + (j0 + j) * kCB] = v;
                eliminate(y[u], now, j, v);
            }
        }
        if (first) bar_arrive(6 + j0 / kCholStep, 32 + 64);
#pragma unroll
        for (int u = 0; u < kCols; ++u) rows_up(y[u]);
    }
}

// The inverse of a diagonal block of R, one warp: lane c keeps column c, rows from the bottom up.  A row's sum begins with what the row
// below has just given, so all 496 multiply-adds are one chain; a row of R and its reciprocal are fetched while the row below is summed.
__device__ __forceinline__ void invert_diagonal(const float *D, float my_inv, float (&t)[kCB], int lane) {
    const unsigned at = smem_u32(D);
    StepRow row, next;
    float inv = __shfl_sync(kFullMask, my_inv, kCB - 1), next_inv = 0.0f;
#pragma unroll
    for (int i = kCB - 1; i >= 0; --i) {
        if (i > 0) {
            step_fetch(next, at + (i - 1) * kCB * 4, i - 1);
            next_inv = __shfl_sync(kFullMask, my_inv, i - 1);
        }
        float acc = (lane == i) ? 1.0f : 0.0f;
#pragma unroll
        for (int l4 = (i + 1) / 4 * 4; l4 < kCB; l4 += 4) {
            const float4 p = row.q[l4 / 4];
            if (l4 > i) acc -= p.x * t[l4];
            if (l4 + 1 > i) acc -= p.y * t[l4 + 1];
            if (l4 + 2 > i) acc -= p.z * t[l4 + 2];
            if (l4 + 3 > i) acc -= p.w * t[l4 + 3];
        }
        t[i] = (lane >= i) ? acc * inv : 0.0f;
        row = next;
        inv = next_inv;
    }
}

// Block (A, B) loses R_LA^T R_LB; a lane of 16.
__device__ __noinline__ void chol_update(int nb, int A, int B, int L) {
    float *blocks = chol_smem(), *O = blocks + blk_id(A, B, nb) * kCBB;
    const int ti = (threadIdx.x & 15) >> 2, tc = threadIdx.x & 3;
    float2 acc[8][4];
    tile_load(acc, O, ti, tc);
    block_mac<kCB, kCB>(acc, blocks + blk_id(L, A, nb) * kCBB, blocks + blk_id(L, B, nb) * kCBB, ti, tc);
    tile_store(acc, O, ti, tc);
}
// ... thread t of 64
__device__ __noinline__ void chol_update_wide(int nb, int A, int B, int L, int t) {
    float *blocks = chol_smem(), *O = blocks + blk_id(A, B, nb) * kCBB;
    float2 acc[4][2];
    tile_load_wide(acc, O, t);
    block_mac_wide<kCB, kCB, kCB>(acc, blocks + blk_id(L, A, nb) * kCBB, blocks + blk_id(L, B, nb) * kCBB, t);
    tile_store_wide(acc, O, t);
}

// R (row-major k x k, upper triangular, zeros below the diagonal) from G, and the diagonal blocks of T = R^-1 if T is given.
// sync (may be null): told which block rows are out.
__device__ __forceinline__ void cholesky_factor(const float *G, int k, float *R, float *T, CholeskySync *sync) {
    float *sm = chol_smem();
    const int nb = chol_blocks(k), nbt = nb * (nb + 1) / 2;
    float *blocks = sm;                                    // nbt blocks of 32 x 32, row-major; those above the diagonal end as R's
    float *dia = blocks + (size_t)nbt * kCBB + kCB;        // the diagonal block of R (what lies below its diagonal is never used), behind a row of zeros
    float *dinv = dia + kCBB + kCB;                        // 1 / its diagonal (reads of dia run on for up to 23 floats)
    constexpr int kDia = kCBB + 3 * kCB;                   // two of each in turn, from step to step
    float *red = dinv + kDia + kCB;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    // load block by block (four elements of a row per thread), padded with an identity; what lies below the diagonal of
    // a diagonal block is never used
    for (int e = tid; e < nbt * (kCBB / 4); e += kCholThreads) {
        int I = 0, rem = e / (kCBB / 4);
        while (rem >= nb - I) { rem -= nb - I; ++I; }      // block (I, I + rem)
        const int at = e % (kCBB / 4), i = I * kCB + (at >> 3), c = (I + rem) * kCB + 4 * (at & 7);
        float *dst = blocks + (size_t)4 * e;
        if ((k & 3) == 0 && i < k && c < k) {
            copy16_async(dst, G + (size_t)i * k + c);
        } else {
#pragma unroll
            for (int q = 0; q < 4; ++q) dst[q] = (i < k && c + q < k) ? G[(size_t)i * k + c + q] : (i == c + q ? 1.0f : 0.0f);
        }
    }
    if (tid < 2 * kCB) dia[(tid >> 5) * kDia + lane - kCB] = 0.0f;
    float md = tid < k ? fmaxf(G[(size_t)tid * k + tid], 0.0f) : 0.0f;
    for (int d = 16; d > 0; d >>= 1) md = fmaxf(md, __shfl_xor_sync(0xffffffffu, md, d));
    if (lane == 0) red[warp] = md;
    // zeros below R's diagonal blocks
    for (int i = kCB + warp; i < k; i += kCholWarps)
        for (int c = lane; c < i / kCB * kCB; c += 32) R[(size_t)i * k + c] = 0.0f;
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
    float m = 0.0f;
#pragma unroll
    for (int w = 0; w < kCholeskyBlockedMaxK / 32; ++w) m = fmaxf(m, red[w]);
    const float shift = m > 0.0f ? m * 1.0e-5f : 0.0f, half = 0.5f * shift;
    if (tid < k) blocks[(size_t)blk_id(tid / kCB, tid / kCB, nb) * kCBB + (tid % kCB) * (kCB + 1)] += shift;
    __syncthreads();
    // Warp 0 has a scheduler to itself but for the two warps that finish rows.  Of the warps on the other three, the first four take
    // the block row, the others the updates that are not urgent and the block of the next pivots.
    const int wi = (warp & 3) ? (warp >> 2) * 3 + (warp & 3) - 1 : -1;
    const int half_warp = 2 * wi + (lane >> 4);
    // Two warps finish a block row while the next one is made: one writes it out -- on another scheduler than warp 0's where a small
    // matrix leaves a worker free --, the other inverts its diagonal block, which is the diagonal block of the inverse.  (A store per
    // pivot, behind the comparisons that a ragged edge needs, cost the pivots' warp 60 of 185 clocks each.)
    const int writer = nb <= kCholPanel ? kCholWarps - 1 : 4, inverter = 8;
    auto finish_row = [&](int J) {
        const float *d = dia + (J & 1) * kDia;
        const int row0 = J * kCB, col = row0 + lane;
        const bool whole = row0 + kCB <= k;
        if (warp == writer) {
            for (int b = 0; b < nb - J; ++b) {
                const float *src = b == 0 ? d + lane : blocks + (size_t)blk_id(J, J + b, nb) * kCBB + lane;
                float *out = R + (size_t)row0 * k + col + b * kCB;
                const bool in = col + b * kCB < k;
#pragma unroll 1
                for (int l0 = 0; l0 < kCB; l0 += 8) {
                    float v[8];
#pragma unroll
                    for (int l = 0; l < 8; ++l) {
                        v[l] = src[(l0 + l) * kCB];
                        if (b == 0 && lane < l0 + l) v[l] = 0.0f;
                    }
                    if (in) {
#pragma unroll
                        for (int l = 0; l < 8; ++l)
                            if (whole || row0 + l0 + l < k) out[(size_t)(l0 + l) * k] = v[l];
                    }
                }
            }
        } else if (T != nullptr) {
            float t[kCB];
            invert_diagonal(d, dinv[(J & 1) * kDia + lane], t, lane);
            float *out = T + (size_t)row0 * k + col;
            if (col < k) {
#pragma unroll
                for (int i = 0; i < kCB; ++i)
                    if (whole || row0 + i < k) out[(size_t)i * k] = t[i];
            }
        }
        if (sync) {
            bar_sync(11, 64);
            if (warp == writer && lane == 0) {
                __threadfence();
                asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(&sync->rows), "r"(J + 1) : "memory");
            }
        }
    };
    for (int J = 0; J < nb; ++J) {
        const int at_dia = (int)(dia - sm) + (J & 1) * kDia, at_dinv = at_dia + kCBB + kCB;
        const int rest = nb - J - 1;                        // blocks to the right of the diagonal block
        const int panel_warps = rest ? 1 + rest / 2 : 0;    // one for the next pivots' columns, two blocks for each of the others
        const int panel = 32 * (1 + panel_warps);           // threads of the barriers between the pivots and the block row
        if (warp == 0) {
            if (half >= 1.17549435e-38f) factor_diagonal<true>(blk_id(J, J, nb) * kCBB, at_dia, at_dinv, half, panel);
            else factor_diagonal<false>(blk_id(J, J, nb) * kCBB, at_dia, at_dinv, half, panel);
        } else if (warp == writer || warp == inverter) {
            if (J > 0) {
                if (warp == kCholWarps - 1) bar_arrive(5, 32 * kCholWorkers);
                finish_row(J - 1);
            }
        } else if (wi >= 0) {
            // ---- G_AB -= R_{J-1,A}^T R_{J-1,B}: row J first, for the block row that follows ----
            if (J > 0) {
                if (rest <= kCholWorkers / 2) {
                    if (wi / 2 < rest) chol_update_wide(nb, J, J + 1 + wi / 2, J - 1, (wi & 1) * 32 + lane);
                } else if (half_warp < rest) {
                    chol_update(nb, J, J + 1 + half_warp, J - 1);
                }
                __syncwarp();
                if (wi < panel_warps) bar_sync(5, 32 * kCholWorkers);
                else bar_arrive(5, 32 * kCholWorkers);
            }
            if (wi < panel_warps) {
                const int b = wi == 0 ? 1 : 2 * wi;         // first block, counted from the diagonal
                const int at_x = blk_id(J, J + b, nb) * kCBB + lane;
                const auto await = [panel](int s) { bar_sync(1 + s, panel); };
                if (wi > 0 && b < rest) block_row<2>(at_x, at_dia, at_dinv, false, await);
                else block_row<1>(at_x, at_dia, at_dinv, wi == 0, await);
            } else if (wi >= kCholPanel && rest) {
                // ---- then the blocks below, that of the next pivots before all others ----
                constexpr int kTasks = 2 * kCholTrail;      // at a time
                const int h = half_warp - 2 * kCholPanel;
                if (J > 0) {
                    if (rest <= 2) {                        // at most three blocks, for two pairs of warps
                        for (int t = h >> 2; h < kTasks / 4 * 4 && t < rest * (rest + 1) / 2; t += kTasks / 4)
                            chol_update_wide(nb, J + 1 + t / 2, J + 1 + (t + 1) / 2, J - 1, ((wi - kCholPanel) & 1) * 32 + lane);
                    } else {
                        for (int t = h; t < rest * (rest + 1) / 2; t = t < kTasks ? 2 * kTasks - 1 - h : t + kTasks) {
                            int A = 0, rem = t;
                            while (rem >= rest - A) { rem -= rest - A; ++A; }
                            chol_update(nb, J + 1 + A, J + 1 + A + rem, J - 1);
                        }
                    }
                    __syncwarp();
                }
                if (wi < kCholPanel + 2) {
                    // ---- the block of the next pivots, 4 x 4 outputs per thread of two warps, behind its block row ----
                    if (J > 0) bar_sync(10, 64);
                    const float *RA = blocks + (size_t)blk_id(J, J + 1, nb) * kCBB;
                    float *O = blocks + (size_t)blk_id(J + 1, J + 1, nb) * kCBB;
                    const int t = (wi - kCholPanel) * 32 + lane;
                    float2 acc[4][2];
                    tile_load_wide(acc, O, t);
#pragma unroll 1
                    for (int j0 = 0; j0 < kCB; j0 += kCholStep) {
                        bar_sync(6 + j0 / kCholStep, 32 + 64);
                        block_mac_wide<kCB, kCB, kCholStep>(acc, RA + j0 * kCB, RA + j0 * kCB, t);
                    }
                    tile_store_wide(acc, O, t);
                }
            }
        }
        __syncthreads();
    }
    if (warp == writer || warp == inverter) finish_row(nb - 1);
}

// Block row I of T = R^-1 (row-major k x k, zeros below the diagonal) right of its diagonal block, from left to right, behind the
// factor's block rows and the diagonal blocks of T.  The transposes of T_IL and of the sums are what is kept, so that every product
// has the form A^T B of block_mac:
//   T_IJ^T = -(T_JJ)^T S_J^T with S_J = sum_L T_IL R_LJ, and S_C^T += (R_JC)^T T_IJ^T for the columns C still to come.
// sync: waited on for the block rows.  Gives up if they do not come.
__device__ __forceinline__ void cholesky_inverse_row(int I, int k, const float *R, float *T, CholeskySync *sync, unsigned *status) {
    const int nb = chol_blocks(k);
    float *rb = chol_smem();                               // block row J of R right of its diagonal block
    float *sum = rb + (size_t)nb * kCBB;                   // -S_C^T, at C
    float *tj = sum + (size_t)nb * kCBB;                   // T_JJ
    float *tij = tj + kCBB;                                // T_IJ^T, rows kCTs apart
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, half_warp = tid >> 4, ti = (tid & 15) >> 2, tc = tid & 3;
    for (int row = I; row < (I == nb - 2 ? nb : I + 1); ++row)           // zeros left of the diagonal block; the last row's as well
        for (int i = warp; i < kCB; i += kCholWarps)
            for (int c = lane; c < row * kCB; c += 32)
                if (row * kCB + i < k) T[(size_t)(row * kCB + i) * k + c] = 0.0f;
    for (int J = I; J < nb; ++J) {
        bool here = true;
        if (tid == 0) {
            unsigned rows = 0;
            for (unsigned i = 0; i < kMbarSpinLimit; ++i) {
                asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(rows) : "l"(&sync->rows) : "memory");
                if (rows > (unsigned)J) break;
                __nanosleep(32);
            }
            here = rows > (unsigned)J;
            if (!here && status) atomicOr(status, kStatusBarrierTimeout);
        }
        if (!__syncthreads_and(here)) return;
        // T_JJ and the blocks of R (past the first-level cache, which may hold older rows' lines)
        for (int e = tid; e < (nb - J) * (kCBB / 4); e += kCholThreads) {
            const int b = e / (kCBB / 4), at = e % (kCBB / 4), i = J * kCB + (at >> 3), c = (J + b) * kCB + 4 * (at & 7);
            const float *src = (b == 0 ? T : R) + (size_t)i * k + c;
            float x[4] = {0.0f, 0.0f, 0.0f, 0.0f};
            if ((k & 3) == 0 && i < k && c < k) {
                const float4 g = __ldcg(reinterpret_cast<const float4 *>(src));
                x[0] = g.x; x[1] = g.y; x[2] = g.z; x[3] = g.w;
            } else {
#pragma unroll
                for (int q = 0; q < 4; ++q)
                    if (i < k && c + q < k) x[q] = __ldcg(src + q);
            }
            reinterpret_cast<float4 *>(b == 0 ? tj : rb + (size_t)(b - 1) * kCBB)[at] = make_float4(x[0], x[1], x[2], x[3]);
        }
        __syncthreads();
        // T_IJ^T = (T_JJ)^T (-S_J^T), four elements of a column per thread of eight warps
        if (warp < 8) {
            const int c0 = 4 * warp;                        // elements (c0 .. + 3, lane) of the transposed block
            float o[4] = {0.0f, 0.0f, 0.0f, 0.0f};
            if (J == I) {
#pragma unroll
                for (int q = 0; q < 4; ++q) o[q] = tj[lane * kCB + c0 + q];
            } else {
                const float *B = sum + (size_t)J * kCBB + lane;
                const unsigned at_t = smem_u32(tj + c0);
#pragma unroll
                for (int l = 0; l < kCB; ++l) {
                    const float4 t = lds4(at_t + l * kCB * 4);
                    const float b = B[l * kCB];
                    o[0] = fmaf(t.x, b, o[0]);
                    o[1] = fmaf(t.y, b, o[1]);
                    o[2] = fmaf(t.z, b, o[2]);
                    o[3] = fmaf(t.w, b, o[3]);
                }
            }
#pragma unroll
            for (int q = 0; q < 4; ++q) tij[(c0 + q) * kCTs + lane] = o[q];
        }
        __syncthreads();
        // out, a row of T at a time (its column index is the row index of the transposed block)
        if (J > I)
            for (int r = warp; r < kCB; r += kCholWarps) {
                const int i = I * kCB + r, c = J * kCB + lane;
                if (i < k && c < k) T[(size_t)i * k + c] = tij[lane * kCTs + r];
            }
        if (nb - J - 1 <= kCholWarps / 2) {
            if (J + 1 + warp / 2 < nb) {
                const int C = J + 1 + warp / 2, t = (warp & 1) * 32 + lane;
                float2 acc[4][2] = {};
                float *S = sum + (size_t)C * kCBB;
                if (J > I) tile_load_wide(acc, S, t);
                block_mac_wide<kCB, kCTs, kCB>(acc, rb + (size_t)(C - J - 1) * kCBB, tij, t);
                tile_store_wide(acc, S, t);
            }
        } else if (J + 1 + half_warp < nb) {
            const int C = J + 1 + half_warp;
            float2 acc[8][4] = {};
            float *S = sum + (size_t)C * kCBB;
            if (J > I) tile_load(acc, S, ti, tc);
            block_mac<kCB, kCTs>(acc, rb + (size_t)(C - J - 1) * kCBB, tij, ti, tc);
            tile_store(acc, S, ti, tc);
        }
        __syncthreads();                                   // the sums of the next column are whole, rb, tj and tij may be overwritten
    }
}

// The CTA that starts first factors; where the inverse is wanted there is a CTA per block, and the others follow with its rows.
__global__ void __launch_bounds__(kCholThreads, 1) cholesky_kernel(const float *G, int k, float *R, float *T, CholeskySync *sync,
                                                                   unsigned *status) {
    __shared__ unsigned s_role;
    chain_begin();
    int role = 0;
    const bool together = gridDim.x > 1;
    if (together) {
        if (threadIdx.x == 0) s_role = atomicAdd(&sync->ticket, 1u);
        __syncthreads();
        role = (int)s_role;
    }
    if (role == 0) cholesky_factor(G, k, R, T, together ? sync : nullptr);
    else cholesky_inverse_row(role - 1, k, R, T, sync, status);
    if (!together) return;
    // The factor's last row is still on its way out when this thread gets here: if the other CTAs have given up on it, this CTA is the last
    // to leave, and a row announced behind the clearing would stand as the next launch's.
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        if (atomicAdd(&sync->done, 1u) + 1 == gridDim.x) {               // everybody has read, and written, what is cleared here
            sync->ticket = 0;
            sync->rows = 0;
            sync->done = 0;
        }
    }
}

}  // namespace
}  // namespace bsq

// SVD of the k x k core of the randomized SVD: one-sided (Hestenes) Jacobi over blocks of columns (sm_100a), for factors that
// stay in FP32 (bsq_svd.cu says why coded ones keep another order of rotations).
//
// The reference runs cusolverDnSgesvd on the k x n matrix B (svd_lowrank_cuda.cu:399-440); here only the k x k
// triangular factor is left to decompose.
//   in : C, row-major k x k; read as the column-major matrix M = C^T (column j = row j of C)
//   out: M = U diag(S) V^T with S descending; U column-major k x k; Vcol column-major k x k: V itself (kWithV), or
//        column j of M V divided by S(j)^2 -- the matrix that turns the panel the core came from into its singular
//        vectors (B^T v_j / S(j) with v_j = (M V)(:, j) / S(j)), for which nothing has to accumulate the rotations.
// Column pairs (p, q) are rotated until all columns of M V are orthogonal to tol, |m_p . m_q| <= tol |m_p| |m_q| with
// tol = sqrt(len) eps / 4: a quarter of LAPACK's sgesvj criterion, which costs no sweep (the last one is recognised by
// kJacobiLastSweepCos) and leaves the vectors that much closer to orthogonal.
//
// What bounds it is one dependent chain -- dot product, angle, rotation -- per round of disjoint pairs, k - 1 rounds per
// sweep and 6 to 9 sweeps whatever the split.  So the columns, not the rows, are dealt over the CTAs: CTA c of a cluster
// holds two blocks of whole columns, most often 16 (block_jacobi_shape), and the blocks move on over distributed shared memory only after
// as many rounds of one against the other.  (Rows dealt over the CTAs, as before, needs the partial dot products of every round
// from every CTA.)  Inside a CTA a warp holds two columns of one block and two of the other in registers and does two
// rounds on them (the straight pairs, then the crossed ones), each round two independent rotations whose angles are worked
// out side by side in the halves of the warp: half as many trips through shared memory and CTA barriers per round, which
// otherwise cost as much as the rotations (16 lanes per pair and a trip per round: 0.46 us per round at 256 columns).
// A sweep: the pairs inside the blocks (a tournament of their column pairs), then 2 x CTAs - 1 steps of a tournament of the blocks.
//   Measured against the kernels that deal rows over the CTAs (above 64 columns) or keep the core in one CTA, on 50 cores per
//   rank (flat, 1/i, geometric, rank-3 and 1e-9-scaled spectra), time and distance from 64 bits of the singular values:
//     k = 256 1323 -> 800 us, 2.3e-5 -> 5.4e-8; k = 128 461 -> 287 us, 1.3e-5 -> 5.7e-8; k = 64 222 -> 129 us, 5.3e-6 -> 5.5e-8;
//     k = 32 91 -> 62 us, 2.3e-6 -> 5.7e-8; k = 16 42 -> 32 us, 6.7e-7 -> 5.4e-8
//   and of U diag(S) V^T 3.5e-5 -> 1.0e-6, 1.6e-5 -> 5.0e-7, 7.7e-7 -> 9.5e-8, 7.7e-7 -> 4.8e-8, 5.0e-7 -> 4.8e-8.  (Below 12 and
//   from 17 to 20 columns the other kernel is 3 to 9 us faster, and as much further off.)
#pragma once

#include "bsq_device.cuh"

#include <cooperative_groups.h>

namespace bsq {
namespace {

constexpr int kBlockJacobiMaxK = 256;
constexpr int kJacobiMaxSweeps = 30;
// A sweep in which no visited pair had |cos(m_p, m_q)| above this is the last one: Jacobi converges quadratically,
// so what such a sweep's rotations leave between the columns is of the order of the square of what it met
// (<= 1e-8, below tol), and the sweep that would only confirm it (a full sweep's time for no rotation) is not run.
// Pairs between tol and this bound are still rotated when they are met.
constexpr float kJacobiLastSweepCos = 1.0e-4f;
__host__ __device__ constexpr int block_jacobi_len(int k) { return (k + 63) / 64 * 64; }           // padded column length: two floats per lane
// How a core is dealt: CTAs of the cluster, columns of a block (two blocks per CTA, a warp per pair of a block's columns).
struct BlockShape {
    int ctas, cols;
};
// A sweep takes as many rounds as the blocks have columns, padding among them, so the shape follows the rank where 16 columns per block leave
// much of that: us, 16 columns per block / as it is: k = 48 122 / 89, 24 61 / 47, 20 59 / 46, 72 185 / 166, 16 28 / 26.  Not taken, because
// twice the CTAs gain little: 32 on 2 x 8 63 / 58, 96 on 6 x 8 218 / 210, 128 on 8 x 8 289 / 277; slower: 48 on 2 x 12 105, 64 on 4 x 8 136
// against 124, 144 on 8 x 12 502 against 422.
constexpr BlockShape block_jacobi_shape(int k) {
    if (k <= 24) return {1, k <= 16 ? 8 : 12};
    if (k > 32 && k <= 48) return {3, 8};
    if (k > 64 && k <= 72) return {3, 12};
    return {(k + 31) / 32, 16};
}
__host__ __device__ constexpr size_t block_jacobi_smem_bytes(BlockShape b, int len, bool with_v) {
    // two parities x two blocks of columns and of squared norms, all singular values, votes and largest entries, ranks
    return ((size_t)4 * b.cols * len * (with_v ? 2 : 1) + 4 * b.cols + 2 * b.cols * b.ctas + 2 * 8 + 8 + 2 * b.cols) * sizeof(float);
}

// two FP32 multiplications / multiply-adds per instruction; each half rounds as the scalar instruction does
__device__ __forceinline__ float2 mul2(float2 a, float2 b) {
    float2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(reinterpret_cast<unsigned long long &>(r))
        : "l"(reinterpret_cast<unsigned long long &>(a)), "l"(reinterpret_cast<unsigned long long &>(b)));
    return r;
}
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) {
    float2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(reinterpret_cast<unsigned long long &>(r))
        : "l"(reinterpret_cast<unsigned long long &>(a)), "l"(reinterpret_cast<unsigned long long &>(b)),
          "l"(reinterpret_cast<unsigned long long &>(c)));
    return r;
}

// A lane's share of a column: kPairs float2, taken from the column 16 or 8 bytes per lane at a time (the same split of
// the rows for every column).
template <int kPairs>
__device__ __forceinline__ void column_load(float2 (&x)[kPairs], const float *col, int l) {
    if constexpr (kPairs % 2 == 0) {
#pragma unroll
        for (int u = 0; u < kPairs / 2; ++u) {
            const float4 v = reinterpret_cast<const float4 *>(col)[u * 32 + l];
            x[2 * u] = make_float2(v.x, v.y);
            x[2 * u + 1] = make_float2(v.z, v.w);
        }
    } else {
#pragma unroll
        for (int u = 0; u < kPairs; ++u) x[u] = reinterpret_cast<const float2 *>(col)[u * 32 + l];
    }
}
template <int kPairs>
__device__ __forceinline__ void column_store(const float2 (&x)[kPairs], float *col, int l) {
    if constexpr (kPairs % 2 == 0) {
#pragma unroll
        for (int u = 0; u < kPairs / 2; ++u)
            reinterpret_cast<float4 *>(col)[u * 32 + l] = make_float4(x[2 * u].x, x[2 * u].y, x[2 * u + 1].x, x[2 * u + 1].y);
    } else {
#pragma unroll
        for (int u = 0; u < kPairs; ++u) reinterpret_cast<float2 *>(col)[u * 32 + l] = x[u];
    }
}
// this lane's part of x . y
template <int kPairs>
__device__ __forceinline__ float column_dot(const float2 (&x)[kPairs], const float2 (&y)[kPairs]) {
    float2 s0 = mul2(x[0], y[0]), s1 = make_float2(0.0f, 0.0f);
#pragma unroll
    for (int u = 1; u < kPairs; ++u) {
        if (u & 1) s1 = fma2(x[u], y[u], s1);
        else s0 = fma2(x[u], y[u], s0);
    }
    return (s0.x + s1.x) + (s0.y + s1.y);
}
// x' = c x - s y, y' = s x + c y as corrections, x - s (y + h x) and y + s (x - h y) with h = s / (1 + c), the tangent of half
// the angle (Rutishauser's form): what is rounded besides x' and y' themselves is a multiple of s, where a rounded cosine
// lengthens or shortens both columns in every rotation.
template <int kPairs>
__device__ __forceinline__ void column_rotate(float2 (&x)[kPairs], float2 (&y)[kPairs], float h, float s) {
    const float2 h2 = make_float2(h, h), m2 = make_float2(-h, -h), s2 = make_float2(s, s), n2 = make_float2(-s, -s);
#pragma unroll
    for (int u = 0; u < kPairs; ++u) {
        const float2 p = fma2(n2, fma2(h2, x[u], y[u]), x[u]);
        y[u] = fma2(s2, fma2(m2, y[u], x[u]), y[u]);
        x[u] = p;
    }
}
// the warp's sums of two values: the lower half gets the first, the upper half the second
__device__ __forceinline__ float sum_two(float v0, float v1, bool upper) {
    float s = (upper ? v1 : v0) + __shfl_xor_sync(0xffffffffu, upper ? v0 : v1, 16);
#pragma unroll
    for (int d = 8; d > 0; d >>= 1) s += __shfl_xor_sync(0xffffffffu, s, d);
    return s;
}
__device__ __forceinline__ float rsqrt_ftz(float x) {
    float r;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}
__device__ __forceinline__ float rcp_ftz(float x) {
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

// Four columns of one warp: two from each side, their lanes' shares in registers, with their squared norms.
template <int kPairs, bool kWithV>
struct Quad {
    float2 a[2][kPairs], b[2][kPairs], av[2][kPairs], bv[2][kPairs];
    float na[2], nb[2];
};

// Makes p0 orthogonal to q0 and p1 to q1 (squared norms np., nq., updated): two rotations at once.  Returns whether one of
// the pairs was above the bound of the last sweep (this half's pair).  The core is scaled so that nothing here leaves FP32's
// range; pairs whose product is below 1e-19 (both columns below about 4e-17 of the largest entry) are left as they are.
template <int kPairs, bool kWithV>
__device__ __forceinline__ bool rotate_two(float2 (&p0)[kPairs], float2 (&q0)[kPairs], float2 (&p1)[kPairs], float2 (&q1)[kPairs],
                                           float2 (&vp0)[kPairs], float2 (&vq0)[kPairs], float2 (&vp1)[kPairs], float2 (&vq1)[kPairs],
                                           float &np0, float &nq0, float &np1, float &nq1, float tol2, bool upper) {
    const float g = sum_two(column_dot<kPairs>(p0, q0), column_dot<kPairs>(p1, q1), upper);
    const float alpha = upper ? np1 : np0, beta = upper ? nq1 : nq0;
    const float ab = alpha * beta, gg = g * g;
    const bool turn = gg > fmaxf(tol2 * ab, 1.2e-38f);
    // the angle from that of twice its size, whose cosine and sine are |d| / r and 2 g / r with d = beta - alpha,
    // r^2 = d^2 + 4 g^2: with q = 1 + |d| / r and e = 1 / sqrt(2 q), sin = 2 g / r e, 1 + cos = 1 + q e, tan = 2 (2 g / r) e^2,
    // and h = sin / (1 + cos).  All to a few units in the last place, far below the tolerance in what that leaves of the pair's product.
    // The rotation is as orthogonal as s = 2 h / (1 + h^2) is true for the h that is used, whatever that is: s gets a correction
    // that makes it so to the last place.  (IEEE divisions and roots throughout give the same distances from 64 bits and take half
    // as long again.)
    const float d = beta - alpha, ir = turn ? rsqrt_ftz(fmaf(d, d, 4.0f * gg)) : 0.0f;
    const float sin2 = copysignf(2.0f, d) * g * ir, q = fmaf(fabsf(d), ir, 1.0f), e = rsqrt_ftz(q + q);
    const float sin0 = sin2 * e, cos1 = fmaf(q, e, 1.0f), h = sin0 * rcp_ftz(cos1);
    const float s = fmaf(fmaf(-sin0, fmaf(h, h, 1.0f), h + h), 0.5f * cos1, sin0), tg = 2.0f * sin2 * e * e * g;
    const float oh = __shfl_xor_sync(0xffffffffu, h, 16), os = __shfl_xor_sync(0xffffffffu, s, 16), otg = __shfl_xor_sync(0xffffffffu, tg, 16);
    const float s0 = upper ? os : s, s1 = upper ? s : os;
    if (s0 != 0.0f || s1 != 0.0f) {                           // (uniform over the warp)
        const float h0 = upper ? oh : h, h1 = upper ? h : oh, tg0 = upper ? otg : tg, tg1 = upper ? tg : otg;
        column_rotate<kPairs>(p0, q0, h0, s0);
        column_rotate<kPairs>(p1, q1, h1, s1);
        if (kWithV) {
            column_rotate<kPairs>(vp0, vq0, h0, s0);
            column_rotate<kPairs>(vp1, vq1, h1, s1);
        }
        np0 = fmaxf(np0 - tg0, 0.0f);
        nq0 += tg0;
        np1 = fmaxf(np1 - tg1, 0.0f);
        nq1 += tg1;
    }
    return turn && gg > kJacobiLastSweepCos * kJacobiLastSweepCos * ab;
}

template <int kLen, int kCtas, int kJbCols, bool kWithV>
__global__ void __launch_bounds__(16 * kJbCols, 1) block_jacobi_kernel(const float *C, int k, float *__restrict__ S,
                                                                   float *__restrict__ Ucol, float *__restrict__ Vcol) {
    constexpr int kJbThreads = 16 * kJbCols, kCol = kLen * (kWithV ? 2 : 1);           // floats per column (V's below M's)
    constexpr int kPairs = kLen / 64;                                    // float2 per lane and column
    constexpr int kBlock = kJbCols * kCol, kAll = 2 * kJbCols * kCtas;
    namespace cg = cooperative_groups;
    cg::cluster_group cluster = cg::this_cluster();
    const int cr = kCtas > 1 ? (int)cluster.block_rank() : 0;
    extern __shared__ __align__(16) float sm[];
    float *cols = sm;                                         // [parity][block][column][kCol]
    float *nrm = cols + 4 * kBlock;                           // [parity][block][column]
    float *sall = nrm + 4 * kJbCols;                          // [CTA][block][column]
    unsigned *votes = reinterpret_cast<unsigned *>(sall + kAll);         // [parity of the sweep][CTA]
    float *maxes = reinterpret_cast<float *>(votes + 16);     // [CTA]
    int *rank_of = reinterpret_cast<int *>(maxes + 8);        // [block][column]
    const int tid = threadIdx.x, w = tid >> 5, l = tid & 31;
    const bool upper = l >= 16;
    chain_begin();
    cluster.sync();                                           // every CTA runs before anybody stores into its shared memory

    // ---- the two blocks of this CTA, zero-padded; V = identity ----
    float mx = 0.0f;
    for (int e0 = tid; e0 < 2 * kJbCols * kLen; e0 += 4 * kJbThreads) {
        float v[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {                         // four global loads in flight per thread
            const int e = e0 + u * kJbThreads, jj = e / kLen, i = e % kLen;
            const int j = (jj < kJbCols ? cr : kCtas + cr) * kJbCols + jj % kJbCols;
            v[u] = (j < k && i < k) ? C[(size_t)j * k + i] : 0.0f;
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const int e = e0 + u * kJbThreads, jj = e / kLen, i = e % kLen;
            const int j = (jj < kJbCols ? cr : kCtas + cr) * kJbCols + jj % kJbCols;
            cols[(size_t)jj * kCol + i] = v[u];
            if (kWithV) cols[(size_t)jj * kCol + kLen + i] = (i == j && j < k) ? 1.0f : 0.0f;
            mx = fmaxf(mx, fabsf(v[u]));
        }
    }
    static_assert(2 * kJbCols * kLen % (4 * kJbThreads) == 0, "whole trips");
    // power of two that brings the largest entry into [2^23, 2^24): squared norms and their squares then stay inside
    // FP32's range for columns down to 1e-15 of the largest (exact, taken out of S at the end)
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, d));
    if (l == 0) sall[w] = mx;
    __syncthreads();
    if (tid < kCtas) {
        float m = 0.0f;
#pragma unroll
        for (int i = 0; i < kJbThreads / 32; ++i) m = fmaxf(m, sall[i]);
        cluster.map_shared_rank(maxes, tid)[cr] = m;
    }
    cluster.sync();
    mx = 0.0f;
#pragma unroll
    for (int d = 0; d < kCtas; ++d) mx = fmaxf(mx, maxes[d]);
    const int shift = (mx > 0.0f && mx < INFINITY) ? min(100, max(-104, 23 - ilogbf(mx))) : 0;
    const float scale = exp2f((float)shift);

    const float tol = sqrtf((float)kLen) * (0.25f * 5.9604645e-08f), tol2 = tol * tol;
    Quad<kPairs, kWithV> c4;
    auto straight = [&]() {                                   // (a0, b0) and (a1, b1)
        return rotate_two<kPairs, kWithV>(c4.a[0], c4.b[0], c4.a[1], c4.b[1], c4.av[0], c4.bv[0], c4.av[1], c4.bv[1], c4.na[0], c4.nb[0],
                                          c4.na[1], c4.nb[1], tol2, upper);
    };
    auto crossed = [&]() {                                    // (a0, b1) and (a1, b0)
        return rotate_two<kPairs, kWithV>(c4.a[0], c4.b[1], c4.a[1], c4.b[0], c4.av[0], c4.bv[1], c4.av[1], c4.bv[0], c4.na[0], c4.nb[1],
                                          c4.na[1], c4.nb[0], tol2, upper);
    };
    auto inside = [&]() {                                     // (a0, a1) and (b0, b1)
        return rotate_two<kPairs, kWithV>(c4.a[0], c4.a[1], c4.b[0], c4.b[1], c4.av[0], c4.av[1], c4.bv[0], c4.bv[1], c4.na[0], c4.na[1],
                                          c4.nb[0], c4.nb[1], tol2, upper);
    };
    auto take = [&](float2 (&m)[2][kPairs], float2 (&v)[2][kPairs], float (&n)[2], const float *col, const float *norm) {
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            column_load<kPairs>(m[i], col + (size_t)i * kCol, l);
            if (kWithV) column_load<kPairs>(v[i], col + (size_t)i * kCol + kLen, l);
            n[i] = norm[i];
        }
    };
    auto give = [&](const float2 (&m)[2][kPairs], const float2 (&v)[2][kPairs], const float (&n)[2], float *col, float *norm) {
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            column_store<kPairs>(m[i], col + (size_t)i * kCol, l);
            if (kWithV) column_store<kPairs>(v[i], col + (size_t)i * kCol + kLen, l);
        }
        if (l < 2) norm[l] = l ? n[1] : n[0];
    };
    int cur = 0;
    const int steps = k > kJbCols ? 2 * kCtas - 1 : 0;        // (one block has nothing to pair it with)
    // where a CTA's blocks go after a step: block 0 ("top") of CTA 0 stays, the others move one place around the ring
    //   top of CTA 1, 2, .. , last, bottom of the last, .. , 1, 0, top of CTA 1
    const int top_cta = (cr == 0 || cr == kCtas - 1) ? cr : cr + 1, top_blk = (cr == 0 || cr != kCtas - 1) ? 0 : 1;
    const int bot_cta = cr == 0 ? (kCtas > 1 ? 1 : 0) : cr - 1, bot_blk = (cr == 0 && kCtas > 1) ? 0 : 1;

    for (int sweep = 0;; ++sweep) {
        float *X = cols + (size_t)cur * 2 * kBlock, *Y = X + kBlock, *nx = nrm + cur * 2 * kJbCols, *ny = nx + kJbCols;
        // exact squared norms, once per sweep (in between they are carried along through the rotations)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            float *col = X + (size_t)h * kBlock + (size_t)(2 * w) * kCol;
            column_load<kPairs>(c4.a[0], col, l);
            column_load<kPairs>(c4.a[1], col + kCol, l);
            if (sweep == 0 && shift != 0) {
                const float2 s2 = make_float2(scale, scale);
#pragma unroll
                for (int i = 0; i < 2; ++i) {
#pragma unroll
                    for (int u = 0; u < kPairs; ++u) c4.a[i][u] = mul2(c4.a[i][u], s2);
                    column_store<kPairs>(c4.a[i], col + (size_t)i * kCol, l);
                }
            }
            const float q = sum_two(column_dot<kPairs>(c4.a[0], c4.a[0]), column_dot<kPairs>(c4.a[1], c4.a[1]), upper);
            if ((l & 15) == 0) nx[h * kJbCols + 2 * w + (upper ? 1 : 0)] = q;
        }
        __syncthreads();
        if (sweep > 0) {
            unsigned any = 0;
#pragma unroll
            for (int d = 0; d < kCtas; ++d) any |= votes[(sweep & 1) * 8 + d];
            if (!any || sweep == kJacobiMaxSweeps) break;     // the same votes in every CTA: all of them leave here
        }
        bool big = false;
        // ---- inside the blocks: a tournament of each block's column pairs, half the warps on either block ----
        {
            constexpr int kTeams = kJbCols / 2, kMatches = kTeams / 2;
            float *B = X + (size_t)(w / kMatches) * kBlock, *nb = nx + (w / kMatches) * kJbCols;
            const int m = w % kMatches;                       // match of the round
            for (int r = 0; r < kTeams - 1; ++r) {
                int p = kTeams - 1, q = r;
                if (m) {
                    p = r + m;
                    q = r + kTeams - 1 - m;
                    p -= p >= kTeams - 1 ? kTeams - 1 : 0;
                    q -= q >= kTeams - 1 ? kTeams - 1 : 0;
                }
                take(c4.a, c4.av, c4.na, B + (size_t)(2 * p) * kCol, nb + 2 * p);
                take(c4.b, c4.bv, c4.nb, B + (size_t)(2 * q) * kCol, nb + 2 * q);
                if (r == 0) big |= inside();
                big |= straight();
                big |= crossed();
                __syncwarp();                                 // every lane has read the norms
                give(c4.a, c4.av, c4.na, B + (size_t)(2 * p) * kCol, nb + 2 * p);
                give(c4.b, c4.bv, c4.nb, B + (size_t)(2 * q) * kCol, nb + 2 * q);
                __syncthreads();
            }
        }
        // ---- block against block ----
        for (int step = 0; step < steps; ++step) {
            X = cols + (size_t)cur * 2 * kBlock;
            Y = X + kBlock;
            nx = nrm + cur * 2 * kJbCols;
            ny = nx + kJbCols;
            const int nxt = cur ^ 1;
            take(c4.a, c4.av, c4.na, X + (size_t)(2 * w) * kCol, nx + 2 * w);
            for (int r = 0; r < kJbCols / 2; ++r) {
                const int j = 2 * ((w + r) % (kJbCols / 2));
                take(c4.b, c4.bv, c4.nb, Y + (size_t)j * kCol, ny + j);
                big |= straight();
                big |= crossed();
                if (r < kJbCols / 2 - 1) {
                    __syncwarp();
                    give(c4.b, c4.bv, c4.nb, Y + (size_t)j * kCol, ny + j);
                    __syncthreads();
                } else {
                    // last round of the step: all four columns go straight to where they are needed next
                    give(c4.b, c4.bv, c4.nb, cluster.map_shared_rank(cols, bot_cta) + (size_t)(nxt * 2 + bot_blk) * kBlock + (size_t)j * kCol,
                         cluster.map_shared_rank(nrm, bot_cta) + (nxt * 2 + bot_blk) * kJbCols + j);
                    give(c4.a, c4.av, c4.na, cluster.map_shared_rank(cols, top_cta) + (size_t)(nxt * 2 + top_blk) * kBlock + (size_t)(2 * w) * kCol,
                         cluster.map_shared_rank(nrm, top_cta) + (nxt * 2 + top_blk) * kJbCols + 2 * w);
                }
            }
            if (step == steps - 1) {
                const unsigned mine = __syncthreads_or(big) ? 1u : 0u;
                if (tid < kCtas) cluster.map_shared_rank(votes, tid)[((sweep + 1) & 1) * 8 + cr] = mine;
            }
            // A CTA reads one parity and its neighbours write the other: they write this one again only after the
            // next of these barriers, which this CTA reaches when it has read it.
            cluster.sync();
            cur = nxt;
        }
        if (steps == 0) {                                     // (one CTA)
            const unsigned mine = __syncthreads_or(big) ? 1u : 0u;
            if (tid == 0) votes[((sweep + 1) & 1) * 8] = mine;
            __syncthreads();
        }
    }

    // ---- singular values (the norms are fresh, nothing rotated since), order, output ----
    const float *X = cols + (size_t)cur * 2 * kBlock;
    float *nx = nrm + cur * 2 * kJbCols;
    if (kWithV) {
        // padding columns, whose V is zero, come after real ones of norm zero
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const float *col = X + (size_t)h * kBlock + (size_t)(2 * w) * kCol + kLen;
            column_load<kPairs>(c4.av[0], col, l);
            column_load<kPairs>(c4.av[1], col + kCol, l);
            const float q = sum_two(column_dot<kPairs>(c4.av[0], c4.av[0]), column_dot<kPairs>(c4.av[1], c4.av[1]), upper);
            if (q == 0.0f && (l & 15) == 0) nx[h * kJbCols + 2 * w + (upper ? 1 : 0)] = -1.0f;
        }
        __syncthreads();
    }
    for (int e = tid; e < kCtas * 2 * kJbCols; e += kJbThreads) {
        const float q = nx[e % (2 * kJbCols)];
        cluster.map_shared_rank(sall, e / (2 * kJbCols))[cr * 2 * kJbCols + e % (2 * kJbCols)] = q < 0.0f ? -1.0f : sqrtf(q);
    }
    cluster.sync();
    const float unscale = exp2f((float)-shift);
    {
        // eight threads per column count the values that come before it, by the bits (NaN first, then descending), ties by place
        const int jj = tid >> 3, me = cr * 2 * kJbCols + jj;
        const int mine = __float_as_int(sall[me]);
        int before = 0;
        for (int i = tid & 7; i < kAll; i += 8) {
            const int v = __float_as_int(sall[i]);
            before += (v > mine || (v == mine && i < me)) ? 1 : 0;
        }
#pragma unroll
        for (int d = 4; d > 0; d >>= 1) before += __shfl_xor_sync(0xffffffffu, before, d);
        if ((tid & 7) == 0) {
            rank_of[jj] = before;
            if (before < k) S[before] = __int_as_float(mine) * unscale;
        }
    }
    __syncthreads();
    for (int e = tid; e < 2 * kJbCols * kLen; e += kJbThreads) {
        const int jj = e / kLen, i = e % kLen, to = rank_of[jj];
        if (i >= k || to >= k) continue;                      // (padding: zero columns, which come last)
        const float sj = sall[cr * 2 * kJbCols + jj], u = sj > 0.0f ? X[(size_t)jj * kCol + i] / sj : 0.0f;
        const size_t o = (size_t)to * k + i;
        Ucol[o] = u;
        Vcol[o] = kWithV ? X[(size_t)jj * kCol + kLen + i] : (sj > 0.0f ? u / (sj * unscale) : 0.0f);
    }
}

typedef void (*BlockJacobiFn)(const float *, int, float *, float *, float *);
// The instance for a core of k columns (k <= kBlockJacobiMaxK; null: there is none).
template <int kLen, int kCtas, int kJbCols>
BlockJacobiFn block_jacobi_instance(bool with_v) {
    return with_v ? block_jacobi_kernel<kLen, kCtas, kJbCols, true> : block_jacobi_kernel<kLen, kCtas, kJbCols, false>;
}
BlockJacobiFn block_jacobi_fn(int k, bool with_v) {
    const BlockShape b = block_jacobi_shape(k);
    if (b.cols == 8) return b.ctas == 1 ? block_jacobi_instance<64, 1, 8>(with_v) : block_jacobi_instance<64, 3, 8>(with_v);
    if (b.cols == 12) return b.ctas == 1 ? block_jacobi_instance<64, 1, 12>(with_v) : block_jacobi_instance<128, 3, 12>(with_v);
    switch (b.ctas) {
        case 1: return block_jacobi_instance<64, 1, 16>(with_v);
        case 2: return block_jacobi_instance<64, 2, 16>(with_v);
        case 3: return block_jacobi_instance<128, 3, 16>(with_v);
        case 4: return block_jacobi_instance<128, 4, 16>(with_v);
        case 5: return block_jacobi_instance<192, 5, 16>(with_v);
        case 6: return block_jacobi_instance<192, 6, 16>(with_v);
        case 7: return block_jacobi_instance<256, 7, 16>(with_v);
        case 8: return block_jacobi_instance<256, 8, 16>(with_v);
    }
    return nullptr;
}

// Launch configuration: one cluster, behind the kernel before as launch_chained has it.
void block_jacobi_config(cudaLaunchConfig_t *cfg, cudaLaunchAttribute (&attr)[2], int k, bool with_v, cudaStream_t st) {
    const BlockShape b = block_jacobi_shape(k);
    cfg->gridDim = dim3(b.ctas, 1, 1);
    cfg->blockDim = dim3(16 * b.cols, 1, 1);
    cfg->dynamicSmemBytes = block_jacobi_smem_bytes(b, block_jacobi_len(k), with_v);
    cfg->stream = st;
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = b.ctas;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg->attrs = attr;
    cfg->numAttrs = 2;
}

}  // namespace
}  // namespace bsq

// Randomized low-rank SVD and low-rank reconstruction (sm_100a host driver + glue kernels).
//
// Replaces svd_lowrank_cuda_initialize / svd_lowrank_cuda / svd_lowrank_cuda_release
// (modules/svd_lowrank_cuda/src/svd_lowrank_cuda.cu:284-581) and reconstruct_lowrank_cuda
// (modules/reconstruct_lowrank_cuda/src/reconstruct_lowrank_cuda.cu:21-62).
//
// Same algorithm family as the reference (Halko-style range finder: Y = W Omega, niter power
// iterations with re-orthonormalisation, projection B = Q^T W, small SVD, U = Q U_hat; the working
// matrix W is A, or A^T when A has fewer rows than columns), different linear algebra:
//   * every product with the big matrix reads the caller's row-major A directly, in either
//     orientation (bsq_gemm.cu) -- no transposed copy of A, no transposes of U and V on the way out;
//   * tall panels are orthonormalised through their k x k Gram matrix instead of Householder QR
//     (Cholesky QR): G = Y^T Y = R^T R, Y <- Y R^-1 -- once inside the power iteration, twice for
//     the bases that the result is built from.  G is shifted by 1e-5 max(diag G) before factoring,
//     so rank-deficient panels (exactly low-rank inputs, all-zero inputs) only leave some columns
//     shorter than unit length instead of dividing by zero;
//   * the small SVD works on a k x k core: B^T = Q2 C with C = R2 R1 the product of the two
//     triangular factors, C = Uc S Vc^T, V_hat = Q2 Uc, U = Q Vc.
// The SVD of the k x k core is a one-sided Jacobi kernel of this library up to 256 columns (bsq_jacobi.cuh; where the factors
// are coded afterwards bsq_ring_jacobi.cuh, up to 48 columns the one-CTA kernel here); larger cores, and devices that cannot place the cluster, go to cuSOLVER's gesvdj on
// the k x k core.  Everything that touches an M- or N-sized array is a kernel of this library.
// Omega comes from cuRAND's XORWOW generator like the reference's (svd_lowrank_cuda.cu:143,289-291),
// seeded per call, column-major N x k.
#include "bsq_cholesky.cuh"
#include "bsq_cholesky_cluster.cuh"
#include "bsq_device.cuh"
#include "bsq_gemm.hpp"
#include "bsq_internal.hpp"
#include "bsq_jacobi.cuh"
#include "bsq_ring_jacobi.cuh"

#include <cooperative_groups.h>
#include <curand.h>
#include <cusolverDn.h>

#include <algorithm>
#include <cstdlib>
#include <new>

namespace bsq {

// Up to this rank the block Jacobi kernel accumulates the right factor of the core, which keeps V orthonormal for singular
// values down to rounding; above, V comes from the panel (what the accumulation would cost grows with the rank).
constexpr int kCoreWithVMaxK = 64;

struct SvdWorkspace {
    int m = 0, n = 0, k = 0, niter = 0, sm_count = 148;
    bool transposed = false;            // working matrix is A^T
    int M = 0, N = 0;                   // working dimensions, M >= N
    float *omega = nullptr;             // N x k, column-major
    float *y = nullptr, *y2 = nullptr;  // M x k
    float *z = nullptr, *z2 = nullptr;  // N x k
    float *g = nullptr;                 // k x k Gram / eigenvectors
    float *w = nullptr;                 // k eigenvalues
    float *t = nullptr, *tinv1 = nullptr, *tinv2 = nullptr, *core = nullptr;   // k x k
    float *uc = nullptr, *vc = nullptr; // k x k outputs of the core SVD
    float *rfac = nullptr;              // k x k factor that nobody asked for
    CholeskySync *chol_sync = nullptr;  // zero between launches
    bool chol_cluster = false;          // Gram matrices go to cholesky_cluster_kernel
    float *gemm_ws = nullptr;
    size_t gemm_ws_bytes = 0;
    float *solver_work = nullptr;
    int lwork = 0;
    int *dev_info = nullptr;
    curandGenerator_t rng = nullptr;
    cusolverDnHandle_t solver = nullptr;
    gesvdjInfo_t svdj = nullptr;
    // row-sharded mode: sum a device buffer over all ranks, in stream order (null: single GPU)
    SvdAllReduce allreduce = nullptr;
    void *allreduce_ctx = nullptr;
    unsigned *status = nullptr;         // device status word of the current call
    unsigned *own_status = nullptr;     // used when the caller passes none
    unsigned *a_absmax = nullptr;       // bits of the largest |A| of the current call (scale of the FP16 split of the big products)
    bool a_absmax_valid = false;
    const unsigned *a_absmax_use = nullptr;
    RingLaunch ring = {};               // the core's kernel for coded factors above kRingMinK columns
    bool jc_with_v = false;             // ... and whether it accumulates the right factor (else that comes from the panel)
    bool device_full = false;           // other work fills the device beside this (chooses tile widths, not results)
    bool block_core = false;            // the core goes to block_jacobi_kernel
    bool own_core_svd = false;          // k small enough for jacobi_svd_kernel (else cuSOLVER's gesvdj on the core)
    bool seeded = false;                // omega holds the draw for `seed`
    unsigned long long seed = 0, offset = 0;
    // optional timing of the spans that matter for a roofline: the products with the big matrix (kind 0) and the
    // all-reduces of the row-sharded mode (kind 1), bracketed by events on the call's stream
    static constexpr int kMaxSpans = 32;
    bool profile = false;
    int spans = 0;
    int span_kind[kMaxSpans] = {};
    cudaEvent_t span_ev[2 * kMaxSpans] = {};
};

namespace {

// One CTA factorises the shifted k x k Gram matrix G + s I = R^T R (Cholesky, R upper triangular, in
// place over the upper triangle of A; s = 1e-5 max(diag G)) and inverts R.  The shift, and a floor of
// s / 2 under every pivot, keep a rank-deficient panel from dividing by zero or taking the root of a
// negative number: deficient directions just come out shorter than unit length (an all-zero panel
// gives R = T = 0).  Any invertible R^-1 leaves the span of the panel unchanged; a second pass brings
// every direction above ~3e-5 of the largest singular value to unit length.
//   A    in: G (symmetric, row-major); out: R in the upper triangle, zeros below
//   T    out: R^-1 (upper triangular, row-major), so that Y T has orthonormal columns
//   Rcpy out (nullable): a copy of R, the inverse transform (Y = (Y T) R)
__global__ void __launch_bounds__(1024) cholesky_inverse_kernel(float *A, int k, float *T, float *Rcpy) {
    __shared__ float s_red[32];
    __shared__ float s_floor, s_r;
    const int tid = threadIdx.x, nt = blockDim.x, lane = tid & 31, warp = tid >> 5, nwarps = nt >> 5;
    float md = 0.0f;
    for (int i = tid; i < k; i += nt) md = fmaxf(md, A[(size_t)i * k + i]);
    for (int d = 16; d > 0; d >>= 1) md = fmaxf(md, __shfl_xor_sync(0xffffffffu, md, d));
    if (lane == 0) s_red[warp] = md;
    __syncthreads();
    if (tid == 0) {
        float m = 0.0f;
        for (int w = 0; w < nwarps; ++w) m = fmaxf(m, s_red[w]);
        s_floor = m > 0.0f ? m * 1.0e-5f : 0.0f;
    }
    __syncthreads();
    // shift: G + s I with s = 1e-5 max(diag G), far above the rounding noise of G, so that the Schur
    // complements of a rank-deficient G stay diagonally dominant and R^-1 cannot blow up
    for (int i = tid; i < k; i += nt) A[(size_t)i * k + i] += s_floor;
    __syncthreads();
    for (int j = 0; j < k; ++j) {
        if (tid == 0) {
            float d = A[(size_t)j * k + j];
            if (!(d > 0.5f * s_floor)) d = 0.5f * s_floor;
            s_r = d > 0.0f ? sqrtf(d) : 0.0f;
            A[(size_t)j * k + j] = s_r;
        }
        __syncthreads();
        const float inv = s_r > 0.0f ? 1.0f / s_r : 0.0f;
        for (int c = j + 1 + tid; c < k; c += nt) A[(size_t)j * k + c] *= inv;        // row j of R
        __syncthreads();
        for (int i = j + 1 + warp; i < k; i += nwarps) {                               // trailing update
            const float rji = A[(size_t)j * k + i];
            for (int c = i + lane; c < k; c += 32) A[(size_t)i * k + c] -= rji * A[(size_t)j * k + c];
        }
        __syncthreads();
    }
    for (int e = tid; e < k * k; e += nt) {                // clear below the diagonal, copy R, clear T
        const int i = e / k, c = e % k;
        if (c < i) A[e] = 0.0f;
        if (Rcpy) Rcpy[e] = c < i ? 0.0f : A[e];
        T[e] = 0.0f;
    }
    __syncthreads();
    // T = R^-1, row by row from the bottom: T(i,c) = (delta_ic - sum_{l=i+1..c} R(i,l) T(l,c)) / R(i,i)
    for (int i = k - 1; i >= 0; --i) {
        const float rii = A[(size_t)i * k + i];
        const float inv = rii > 0.0f ? 1.0f / rii : 0.0f;
        for (int c = i + tid; c < k; c += nt) {
            float acc = (c == i) ? 1.0f : 0.0f;
            for (int l = i + 1; l <= c; ++l) acc -= A[(size_t)i * k + l] * T[(size_t)l * k + c];
            T[(size_t)i * k + c] = acc * inv;
        }
        __syncthreads();
    }
}

// The same factorisation and inverse for k up to kCholeskySmemMaxK, entirely in shared memory: the upper
// triangle is held packed (row i at row_off(i) + c, c >= i), k (k + 1) / 2 floats, so k = 256 takes 129 KB.
// G is only read; R goes to Rcpy, R^-1 to T (both full row-major k x k with zeros below the diagonal).
// Two CTA barriers per column in the factorisation, two per row in the inversion.
constexpr int kCholeskySmemMaxK = 320;
__host__ __device__ constexpr size_t cholesky_smem_bytes(int k) { return ((size_t)k * (k + 1) / 2 + 2 * (size_t)k + 2 * 1024 + 64) * sizeof(float); }

__global__ void __launch_bounds__(1024) cholesky_inverse_smem_kernel(const float *__restrict__ G, int k, float *__restrict__ T,
                                                                     float *__restrict__ Rcpy) {
    extern __shared__ float sm[];
    float *P = sm;                                         // packed upper triangle
    float *vec = sm + (size_t)k * (k + 1) / 2;             // 2 x k: the scaled pivot row / the row of R being inverted
    float *part = vec + 2 * k;                             // 2 x 1024: partial sums of the split dot products
    float *red = part + 2 * 1024;                          // 32 + 1
    const int tid = threadIdx.x, nt = blockDim.x, lane = tid & 31, warp = tid >> 5, nwarps = nt >> 5;
    auto row_off = [k](int i) { return i * k - (i * (i - 1)) / 2 - i; };
    float md = 0.0f;
    for (int e = tid; e < k * k; e += nt) {
        const int i = e / k, c = e % k;
        if (c >= i) {
            const float v = G[e];
            P[row_off(i) + c] = v;
            if (c == i) md = fmaxf(md, v);
        }
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
    for (int i = tid; i < k; i += nt) P[row_off(i) + i] += shift;
    __syncthreads();
    for (int j = 0; j < k; ++j) {
        // pivot and scaled row j (every thread derives the pivot itself; it is stored in the next phase)
        const int oj = row_off(j);
        float d = P[oj + j];
        if (!(d > 0.5f * shift)) d = 0.5f * shift;
        const float r = d > 0.0f ? sqrtf(d) : 0.0f;
        const float inv = r > 0.0f ? 1.0f / r : 0.0f;
        for (int c = j + 1 + tid; c < k; c += nt) vec[c] = P[oj + c] * inv;
        __syncthreads();
        if (tid == 0) P[oj + j] = r;
        for (int c = j + 1 + tid; c < k; c += nt) P[oj + c] = vec[c];
        for (int i = j + 1 + warp; i < k; i += nwarps) {    // trailing update, one warp per row
            const float rji = vec[i];
            const int oi = row_off(i);
            for (int c = i + lane; c < k; c += 32) P[oi + c] -= rji * vec[c];
        }
        __syncthreads();
    }
    for (int e = tid; e < k * k; e += nt) {                // R out; T's zeros below the diagonal
        const int i = e / k, c = e % k;
        if (Rcpy) Rcpy[e] = c < i ? 0.0f : P[row_off(i) + c];
        if (c < i) T[e] = 0.0f;
    }
    __syncthreads();
    // T = R^-1 in place, row by row from the bottom: T(i,c) = (delta_ic - sum_{l=i+1..c} R(i,l) T(l,c)) / R(i,i).
    // Column c is served by `ways` threads (one per residue of l); their partial sums are added in a fixed order,
    // so the result is the same on every run.  vec and part alternate between two copies: the stores of row i - 1
    // may overtake the last reads of row i.
    const int ways = max(1, min(32, nt / k));              // 1024 / 256 = 4, 1024 / 128 = 8
    const int c_of = tid % k, way = tid / k;
    for (int i = k - 1; i >= 0; --i) {
        const int oi = row_off(i);
        float *v = vec + (i & 1) * k, *ps = part + (i & 1) * 1024;
        for (int c = i + tid; c < k; c += nt) v[c] = P[oi + c];
        __syncthreads();
        if (way < ways) {
            float acc = 0.0f;
            for (int l = i + 1 + way; l <= c_of; l += ways) acc += v[l] * P[row_off(l) + c_of];
            ps[way * k + c_of] = acc;
        }
        __syncthreads();
        const float rii = v[i];
        const float inv = rii > 0.0f ? 1.0f / rii : 0.0f;
        for (int c = i + tid; c < k; c += nt) {
            float sum = 0.0f;
            for (int w = 0; w < ways; ++w) sum += ps[w * k + c];
            P[oi + c] = ((c == i ? 1.0f : 0.0f) - sum) * inv;
        }
    }
    __syncthreads();
    for (int e = tid; e < k * k; e += nt) {
        const int i = e / k, c = e % k;
        if (c >= i) T[e] = P[row_off(i) + c];
    }
}

// The kernel below and that of bsq_ring_jacobi.cuh serve cores whose factors are coded afterwards (NF4 / NF4_DQ sections, error lists made from them):
// the codes of a singular pair depend on its sign and, in a flat spectrum, on how the last bits turn neighbouring vectors
// into one another, so another order of rotations than theirs changes most objects in most bytes (measured: 6 to 8 % of the
// reconstructed matrix, as large a change as a library solver makes).  An error list is whole numbers too: which elements of
// the residual are the largest and in which order changes with the last bits of factors that are themselves FP32.  Objects
// that hold codes or such a list keep their bytes; where all that can change is the rounding of FP32 values, the factors come
// from the block kernel of bsq_jacobi.cuh.
// SVD of the k x k core for k <= kRingMinK: one-sided (Hestenes) Jacobi in one CTA, everything in shared memory.
// The reference runs cusolverDnSgesvd on the k x n matrix B (svd_lowrank_cuda.cu:399-440); here only the k x k
// triangular factor is left to decompose.
//   in : C, row-major k x k; read as the column-major matrix M = C^T (column j = row j of C)
//   out: M = U diag(S) V^T with S descending; U and V column-major k x k
// Column pairs (p, q) are rotated until all columns of M V are orthogonal to tol (LAPACK's sgesvj criterion,
// |m_p . m_q| <= tol |m_p| |m_q|, tol = sqrt(len) eps); the k / 2 pairs of a round are disjoint (round-robin
// schedule), 8 lanes serve a pair, a CTA barrier separates the rounds.  Squared column norms are carried along
// through the rotations and recomputed exactly at the start of every sweep.  At the end S(j) = |column j|,
// U(:, j) = column j / S(j) (zero for S(j) = 0), and a rank by counting puts S in descending order.
constexpr int kJacobiSingleMaxK = 64;         // cores whose right factor is accumulated
constexpr int kJacobiClusterMaxK = 256;       // larger ones go to the library solver
constexpr int kJacobiLen = 64;                // padded column length
__host__ __device__ constexpr size_t jacobi_smem_bytes(int k) {
    return ((size_t)2 * ((k + 1) & ~1) * kJacobiLen + 2 * (size_t)((k + 1) & ~1) + 64) * sizeof(float);
}

// (One CTA per SM told to the compiler: without that it schedules as if other warps hid a chain's latencies; k = 48 163 -> 158 us.)
__global__ void __launch_bounds__(256, 1) jacobi_svd_kernel(const float *C, int k, float *__restrict__ S,
                                                         float *__restrict__ Ucol, float *__restrict__ Vcol) {
    extern __shared__ __align__(16) float sm[];
    chain_begin();
    constexpr int LEN = kJacobiLen;
    const int kp = (k + 1) & ~1, npairs = kp / 2;
    float *M = sm, *V = M + (size_t)kp * LEN, *nrm = V + (size_t)kp * LEN;
    int *rank_of = reinterpret_cast<int *>(nrm + kp);
    const int tid = threadIdx.x, nt = blockDim.x;
    const int slot = tid >> 3, l = tid & 7;                   // 8 lanes per pair, up to 24 pairs
    constexpr int F4 = LEN / 32;                              // float4 per lane and column
    for (int e0 = tid; e0 < kp * LEN; e0 += 4 * nt) {        // four global loads in flight per thread
        float v[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const int e = e0 + u * nt, j = e / LEN, i = e % LEN;
            v[u] = (e < kp * LEN && j < k && i < k) ? C[(size_t)j * k + i] : 0.0f;
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const int e = e0 + u * nt, j = e / LEN, i = e % LEN;
            if (e < kp * LEN) {
                M[e] = v[u];
                V[e] = (i == j && j < k) ? 1.0f : 0.0f;
            }
        }
    }
    __syncthreads();
    const float tol = sqrtf((float)LEN) * 5.9604645e-08f, tol2 = tol * tol;
    auto sum8 = [&](float x) {                                // sum over the 8 lanes of a pair slot
        x += __shfl_xor_sync(0xffffffffu, x, 4, 8);
        x += __shfl_xor_sync(0xffffffffu, x, 2, 8);
        x += __shfl_xor_sync(0xffffffffu, x, 1, 8);
        return x;
    };
    // squared norm of column j; every lane of a warp calls it together (columns past the end count as zero)
    auto norm2 = [&](int j) {
        float acc = 0.0f;
        if (j < kp) {
            for (int f = 0; f < F4; ++f) {
                const float4 a = reinterpret_cast<const float4 *>(M + (size_t)j * LEN)[f * 8 + l];
                acc += a.x * a.x + a.y * a.y + a.z * a.z + a.w * a.w;
            }
        }
        return sum8(acc);
    };
    for (int sweep = 0; sweep < kJacobiMaxSweeps; ++sweep) {
        for (int j0 = 0; j0 < kp; j0 += nt / 8) {             // exact squared norms (uniform trip count: shuffles inside)
            const float a = norm2(j0 + slot);
            if (l == 0 && j0 + slot < kp) nrm[j0 + slot] = a;
        }
        __syncthreads();
        bool rotated = false;
        for (int r = 0; r < kp - 1; ++r) {
            const bool active = slot < npairs;
            int p = 0, q = 0;
            if (active) {
                if (slot == 0) { p = kp - 1; q = r; }
                else { p = (r + slot) % (kp - 1); q = (r + kp - 1 - slot) % (kp - 1); }
            }
            float4 *mp = reinterpret_cast<float4 *>(M + (size_t)p * LEN), *mq = reinterpret_cast<float4 *>(M + (size_t)q * LEN);
            float4 ap[F4], aq[F4];
            float g = 0.0f;
#pragma unroll
            for (int f = 0; f < F4; ++f) {
                ap[f] = mp[f * 8 + l];
                aq[f] = mq[f * 8 + l];
                g += ap[f].x * aq[f].x + ap[f].y * aq[f].y + ap[f].z * aq[f].z + ap[f].w * aq[f].w;
            }
            g = sum8(g);
            const float alpha = nrm[p], beta = nrm[q];
            // |m_p . m_q| > tol |m_p| |m_q|, compared in squares
            if (active && alpha > 0.0f && beta > 0.0f && g * g > tol2 * alpha * beta) {
                const float zeta = (beta - alpha) / (2.0f * g);
                // 1 / (2 zeta) once zeta^2 would overflow: the rotation is then too small to change anything
                const float t = fabsf(zeta) > 1.0e8f ? 0.5f / zeta : copysignf(1.0f, zeta) / (fabsf(zeta) + sqrtf(1.0f + zeta * zeta));
                const float c = rsqrtf(1.0f + t * t), sn = c * t;
                float4 *vp = reinterpret_cast<float4 *>(V + (size_t)p * LEN), *vq = reinterpret_cast<float4 *>(V + (size_t)q * LEN);
#pragma unroll
                for (int f = 0; f < F4; ++f) {
                    const float4 x = ap[f], y = aq[f];
                    mp[f * 8 + l] = make_float4(c * x.x - sn * y.x, c * x.y - sn * y.y, c * x.z - sn * y.z, c * x.w - sn * y.w);
                    mq[f * 8 + l] = make_float4(sn * x.x + c * y.x, sn * x.y + c * y.y, sn * x.z + c * y.z, sn * x.w + c * y.w);
                    const float4 u = vp[f * 8 + l], w = vq[f * 8 + l];
                    vp[f * 8 + l] = make_float4(c * u.x - sn * w.x, c * u.y - sn * w.y, c * u.z - sn * w.z, c * u.w - sn * w.w);
                    vq[f * 8 + l] = make_float4(sn * u.x + c * w.x, sn * u.y + c * w.y, sn * u.z + c * w.z, sn * u.w + c * w.w);
                }
                if (l == 0) {
                    nrm[p] = fmaxf(alpha - t * g, 0.0f);
                    nrm[q] = beta + t * g;
                }
                rotated = rotated || g * g > kJacobiLastSweepCos * kJacobiLastSweepCos * alpha * beta;
            }
            __syncthreads();
        }
        if (!__syncthreads_or(rotated)) break;
    }
    // singular values, order, output
    for (int j0 = 0; j0 < kp; j0 += nt / 8) {
        const float a = norm2(j0 + slot);
        if (l == 0 && j0 + slot < kp) nrm[j0 + slot] = sqrtf(a);
    }
    __syncthreads();
    for (int j = tid; j < k; j += nt) {
        const float sj = nrm[j];
        int rk = 0;
        for (int i = 0; i < k; ++i) {
            const float si = nrm[i];
            rk += (si > sj || (si == sj && i < j)) ? 1 : 0;
        }
        rank_of[j] = rk;
        S[rk] = sj;
    }
    __syncthreads();
    for (int e = tid; e < k * k; e += nt) {
        const int j = e / k, i = e % k;
        const float sj = nrm[j];
        const size_t o = (size_t)rank_of[j] * k + i;
        Ucol[o] = sj > 0.0f ? M[(size_t)j * LEN + i] / sj : 0.0f;
        Vcol[o] = V[(size_t)j * LEN + i];
    }
}

// A timed span of the current call (no-ops unless the workspace's profiling is on).
int span_begin(SvdWorkspace *ws, int kind, cudaStream_t st) {
    if (!ws->profile || ws->spans >= SvdWorkspace::kMaxSpans) return -1;
    const int i = ws->spans++;
    ws->span_kind[i] = kind;
    cudaEventRecord(ws->span_ev[2 * i], st);
    return i;
}
void span_end(SvdWorkspace *ws, int i, cudaStream_t st) {
    if (i >= 0) cudaEventRecord(ws->span_ev[2 * i + 1], st);
}
cudaError_t timed_allreduce(SvdWorkspace *ws, float *buf, size_t count, cudaStream_t st) {
    const int sp = span_begin(ws, 1, st);
    const cudaError_t err = ws->allreduce(ws->allreduce_ctx, buf, count, st);
    span_end(ws, sp, st);
    return err;
}

bool alloc_f(float **p, size_t count) {
    if (cudaMalloc(reinterpret_cast<void **>(p), std::max<size_t>(count, 1) * sizeof(float)) != cudaSuccess) {
        cudaGetLastError();
        *p = nullptr;
        return false;
    }
    return true;
}

// Y (rows x k, row-major) <- Y with orthonormalised columns, `passes` (1 or 2) Gram/Cholesky passes:
// one is enough to keep a power iteration stable, two give orthonormality to rounding.  `tmp` is a
// second rows x k buffer; the result ends in Y for 2 passes and in tmp for 1 (returned through *out).
// r_a / r_b (nullable) receive the triangular factors of the passes (Y_in = Y_out * r_b * r_a).
// last_factor_only: the last pass stops after its Cholesky factor (no inverse, no panel product): the caller wants the
// triangular factors only, and Y itself is left as it was (k <= kCholeskyBlockedMaxK).
cudaError_t orthonormalise(SvdWorkspace *ws, float *Y, float *tmp, int rows, int passes, float *r_a, float *r_b,
                           float **out, bool sharded_rows, cudaStream_t st, bool last_factor_only = false) {
    const int k = ws->k;
    float *src = Y, *dst = tmp;
    for (int pass = 0; pass < passes; ++pass) {
        const bool factor_only = last_factor_only && pass + 1 == passes;
        // G = src^T src
        cudaError_t err = gemm(false, false, src, k, src, k, ws->g, k, k, k, rows, nullptr, nullptr, 0, nullptr, ws->status, ws->gemm_ws,
                               ws->gemm_ws_bytes, ws->sm_count, st, nullptr, 0.0f, ws->device_full);
        if (err != cudaSuccess) return err;
        // a row-sharded panel: its Gram matrix is the sum of the shards' (the one exchange per QR pass);
        // every rank then factors the same k x k matrix and gets bit-identical R
        if (sharded_rows && ws->allreduce && (err = timed_allreduce(ws, ws->g, (size_t)k * k, st)) != cudaSuccess) return err;
        if (k <= kCholeskyBlockedMaxK) {
            float *r_out = pass == 0 ? r_a : r_b;
            if (!r_out) r_out = ws->rfac;
            if (ws->chol_cluster) {
                cudaLaunchConfig_t cfg;
                cudaLaunchAttribute attr[2];
                cholesky_cluster_config(&cfg, attr, k, st);
                const float *g = ws->g;
                if ((err = cudaLaunchKernelEx(&cfg, cholesky_cluster_kernel, g, k, r_out, factor_only ? (float *)nullptr : ws->t, ws->status)) != cudaSuccess)
                    return err;
            } else {
                launch_chained(cholesky_kernel, factor_only ? 1 : chol_blocks(k), kCholThreads, cholesky_blocked_smem_bytes(k), st, ws->g, k, r_out,
                               factor_only ? nullptr : ws->t, ws->chol_sync, ws->status);
            }
        } else if (k <= kCholeskySmemMaxK) {
            cholesky_inverse_smem_kernel<<<1, 1024, cholesky_smem_bytes(k), st>>>(ws->g, k, ws->t, pass == 0 ? r_a : r_b);
        } else {
            cholesky_inverse_kernel<<<1, 1024, 0, st>>>(ws->g, k, ws->t, pass == 0 ? r_a : r_b);
        }
        err = cudaGetLastError();
        if (err != cudaSuccess) return err;
        if (factor_only) break;
        // dst = src T
        err = gemm(true, false, src, k, ws->t, k, dst, k, rows, k, k, nullptr, nullptr, 0, nullptr, ws->status, ws->gemm_ws,
                   ws->gemm_ws_bytes, ws->sm_count, st, nullptr, 0.0f, ws->device_full);
        if (err != cudaSuccess) return err;
        std::swap(src, dst);
    }
    *out = src;
    return cudaSuccess;
}

// C[rows_out x k] = W * X or W^T * X for the working matrix W of the workspace.
// X is row-major unless x_colmajor (Omega).
cudaError_t times_w(SvdWorkspace *ws, const float *A, bool w_transposed_product, const float *X, bool x_colmajor, float *C,
                    cudaStream_t st) {
    // W = A (not transposed) or A^T.  "W * X" contracts over W's columns, "W^T * X" over its rows.
    const bool use_a_as_stored = (w_transposed_product == ws->transposed);   // W*X with W=A, or W^T*X with W=A^T
    const int rows_out = w_transposed_product ? ws->N : ws->M;
    const int contract = w_transposed_product ? ws->M : ws->N;
    const long ldx = x_colmajor ? contract : ws->k;
    const int sp = span_begin(ws, 0, st);
    cudaError_t err = gemm(use_a_as_stored, x_colmajor, A, ws->n, X, ldx, C, ws->k, rows_out, ws->k, contract, nullptr,
                           nullptr, 0, nullptr, ws->status, ws->gemm_ws, ws->gemm_ws_bytes, ws->sm_count, st, ws->a_absmax_valid ? ws->a_absmax_use : nullptr,
                           // what X can hold: standard normal draws from 32-bit uniforms stay below 6.7, the columns of an
                           // orthonormalised panel have norm 1 (a loose bound costs FP16 range, not precision)
                           x_colmajor ? 16.0f : 1024.0f, ws->device_full);
    span_end(ws, sp, st);
    // row-sharded W: W^T X contracts over the sharded rows, so the shards' partial products are summed
    if (err == cudaSuccess && w_transposed_product && ws->allreduce) err = timed_allreduce(ws, C, (size_t)rows_out * ws->k, st);
    return err;
}

}  // namespace

SvdWorkspace *svd_workspace_create(int m, int n, int k, int niter, int sm_count, bool coded_factors) {
    return svd_workspace_create_sharded(m, n, k, niter, sm_count, nullptr, nullptr, 0, coded_factors);
}

// Row-sharded: this rank holds m of the m_total rows (all n columns); the working matrix is never the
// transpose, so that the sharded dimension is the tall one that only GEMMs touch.
SvdWorkspace *svd_workspace_create_sharded(int m, int n, int k, int niter, int sm_count, SvdAllReduce allreduce,
                                           void *allreduce_ctx, int m_total, bool coded_factors) {
    if (m <= 0 || n <= 0 || k <= 0 || niter < 0) return nullptr;
    SvdWorkspace *ws = new (std::nothrow) SvdWorkspace();
    if (!ws) return nullptr;
    ws->m = m; ws->n = n; ws->niter = niter; ws->sm_count = sm_count;
    ws->allreduce = allreduce;
    ws->allreduce_ctx = allreduce_ctx;
    ws->k = std::max(1, std::min(k, std::min(allreduce ? m_total : m, n)));
    ws->transposed = allreduce ? false : m < n;
    ws->M = ws->transposed ? n : m;
    ws->N = ws->transposed ? m : n;
    const size_t kk = (size_t)ws->k * ws->k;
    bool ok = alloc_f(&ws->omega, (size_t)ws->N * ws->k + 2) && alloc_f(&ws->y, (size_t)ws->M * ws->k) &&
              alloc_f(&ws->y2, (size_t)ws->M * ws->k) && alloc_f(&ws->z, (size_t)ws->N * ws->k) &&
              alloc_f(&ws->z2, (size_t)ws->N * ws->k) && alloc_f(&ws->g, kk) && alloc_f(&ws->w, ws->k) &&
              alloc_f(&ws->t, kk) && alloc_f(&ws->tinv1, kk) && alloc_f(&ws->tinv2, kk) && alloc_f(&ws->core, kk) &&
              alloc_f(&ws->uc, kk) && alloc_f(&ws->vc, kk) && alloc_f(&ws->rfac, kk);
    // split-K partials: up to 2 * SMs tiles' worth of the largest skinny product, and of the Gram matrix
    // K-split partials, and behind them room for the images of a product's second operand split beforehand
    ws->gemm_ws_bytes = std::max((size_t)ws->M * ws->k * 8, kk * 2 * (size_t)sm_count) * sizeof(float) +
                        gemm_tc_image_bytes(ws->k, ws->k <= 256 ? ws->k : 128, std::max(ws->M, ws->N)) + 256;
    ok = ok && alloc_f(&ws->gemm_ws, ws->gemm_ws_bytes / sizeof(float));
    ok = ok && cudaMalloc(reinterpret_cast<void **>(&ws->dev_info), sizeof(int)) == cudaSuccess;
    ok = ok && cudaMalloc(reinterpret_cast<void **>(&ws->chol_sync), sizeof(CholeskySync)) == cudaSuccess &&
         cudaMemset(ws->chol_sync, 0, sizeof(CholeskySync)) == cudaSuccess && cudaStreamSynchronize(nullptr) == cudaSuccess;
    ok = ok && cudaMalloc(reinterpret_cast<void **>(&ws->own_status), sizeof(unsigned)) == cudaSuccess;
    ok = ok && cudaMalloc(reinterpret_cast<void **>(&ws->a_absmax), sizeof(unsigned)) == cudaSuccess;
    ok = ok && curandCreateGenerator(&ws->rng, CURAND_RNG_PSEUDO_DEFAULT) == CURAND_STATUS_SUCCESS;
    ok = ok && cusolverDnCreate(&ws->solver) == CUSOLVER_STATUS_SUCCESS;
    ok = ok && cusolverDnCreateGesvdjInfo(&ws->svdj) == CUSOLVER_STATUS_SUCCESS;
    {
        // Jacobi stops when the columns are orthogonal to this tolerance; the library's default is machine epsilon.
        // The factors only have to carry FP32 products to ~1e-6, and every sweep over a 256 x 256 core costs 0.4 ms.
        double tol = 1.0e-6;
        if (const char *e = getenv("BSQ_CORE_SVD_TOL")) {
            const double v = atof(e);
            if (v >= 1.0e-8 && v <= 1.0e-2) tol = v;          // anything else: keep the default
        }
        ok = ok && cusolverDnXgesvdjSetTolerance(ws->svdj, tol) == CUSOLVER_STATUS_SUCCESS;
    }
    if (ok) {
        int l1 = 0, l2 = 0;
        ok = cusolverDnSsyevd_bufferSize(ws->solver, CUSOLVER_EIG_MODE_VECTOR, CUBLAS_FILL_MODE_LOWER, ws->k, ws->g, ws->k,
                                         ws->w, &l1) == CUSOLVER_STATUS_SUCCESS &&
             cusolverDnSgesvdj_bufferSize(ws->solver, CUSOLVER_EIG_MODE_VECTOR, 0, ws->k, ws->k, ws->core, ws->k, ws->w,
                                          ws->uc, ws->k, ws->vc, ws->k, &l2, ws->svdj) == CUSOLVER_STATUS_SUCCESS;
        ws->lwork = std::max(1, std::max(l1, l2));
        ok = ok && alloc_f(&ws->solver_work, (size_t)ws->lwork);
    }
    {
        const char *e = getenv("BSQ_CORE_SVD");              // "cusolver": keep the library solver (A/B comparisons)
        ws->own_core_svd = ws->k <= kJacobiClusterMaxK && !(e && e[0] == 'c');
    }
    if (ok && ws->own_core_svd && !coded_factors) {
        const char *v = getenv("BSQ_JACOBI_V");
        ws->jc_with_v = v ? v[0] == '1' : ws->k <= kCoreWithVMaxK;
        cudaLaunchConfig_t cfg = {};
        cudaLaunchAttribute attr[2];
        block_jacobi_config(&cfg, attr, ws->k, ws->jc_with_v, nullptr);
        const BlockJacobiFn fn = block_jacobi_fn(ws->k, ws->jc_with_v);
        int clusters = 0;
        ws->block_core = fn && cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)cfg.dynamicSmemBytes) == cudaSuccess &&
                         cudaOccupancyMaxActiveClusters(&clusters, fn, &cfg) == cudaSuccess && clusters >= 1;
        if (!ws->block_core) {                               // a device (or partition of one) that cannot place the cluster
            cudaGetLastError();
            ws->jc_with_v = false;
        }
    }
    if (ok && ws->own_core_svd && !ws->block_core && ws->k <= kRingMinK)
        ok = cudaFuncSetAttribute(jacobi_svd_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)jacobi_smem_bytes(ws->k)) == cudaSuccess;
    if (ok && ws->own_core_svd && !ws->block_core && ws->k > kRingMinK) {
        if (ws->k > kJacobiSingleMaxK) {
            const char *v = getenv("BSQ_JACOBI_V");           // 1 / 0: with / without the accumulated right factor (A/B comparisons)
            ws->jc_with_v = v ? v[0] == '1' : false;
        }
        ws->ring = ring_jacobi_launch(ws->k, ws->jc_with_v);
        ok = cudaFuncSetAttribute(ws->ring.fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)ws->ring.smem) == cudaSuccess;
        if (ok && ws->ring.ctas > 1) {
            // a device (or partition of one) that cannot place the cluster keeps the library solver
            cudaLaunchConfig_t cfg = {};
            cudaLaunchAttribute attr[2];
            ring_jacobi_config(&cfg, attr, ws->ring, nullptr);
            int clusters = 0;
            const cudaError_t q = cudaOccupancyMaxActiveClusters(&clusters, ws->ring.fn, &cfg);
            if (q != cudaSuccess || clusters < 1) {
                cudaGetLastError();
                ws->own_core_svd = false;
            }
        }
    }
    const char *chol = getenv("BSQ_CHOL_CLUSTER");           // 0: as a device that cannot place the cluster (A/B comparisons)
    if (ok && ws->k > kCB && ws->k <= kCholeskyBlockedMaxK && !(chol && chol[0] == '0') &&
        cudaFuncSetAttribute(cholesky_cluster_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)cholesky_cluster_smem_bytes(kCholeskyBlockedMaxK)) ==
            cudaSuccess) {
        cudaLaunchConfig_t cfg;
        cudaLaunchAttribute attr[2];
        cholesky_cluster_config(&cfg, attr, ws->k, nullptr);
        int clusters = 0;
        // (a device, or a partition of one, that cannot place the cluster keeps the kernel of up to 32 columns)
        ws->chol_cluster = cudaOccupancyMaxActiveClusters(&clusters, cholesky_cluster_kernel, &cfg) == cudaSuccess && clusters >= 1;
    }
    if (ok && !ws->chol_cluster) cudaGetLastError();
    if (ok && ws->k <= kCholeskyBlockedMaxK)
        ok = cudaFuncSetAttribute(cholesky_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)cholesky_blocked_smem_bytes(ws->k)) == cudaSuccess;
    else if (ok && ws->k <= kCholeskySmemMaxK)
        ok = cudaFuncSetAttribute(cholesky_inverse_smem_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)cholesky_smem_bytes(ws->k)) == cudaSuccess;
    if (!ok) {
        cudaGetLastError();
        svd_workspace_destroy(ws);
        return nullptr;
    }
    return ws;
}

void svd_workspace_device_full(SvdWorkspace *ws, bool full) { ws->device_full = full; }

void svd_workspace_destroy(SvdWorkspace *ws) {
    if (!ws) return;
    float *bufs[] = {ws->omega, ws->y, ws->y2, ws->z, ws->z2, ws->g, ws->w, ws->t, ws->tinv1, ws->tinv2,
                     ws->core, ws->uc, ws->vc, ws->rfac, ws->gemm_ws, ws->solver_work};
    for (float *p : bufs)
        if (p) cudaFree(p);
    if (ws->dev_info) cudaFree(ws->dev_info);
    if (ws->chol_sync) cudaFree(ws->chol_sync);
    if (ws->own_status) cudaFree(ws->own_status);
    if (ws->a_absmax) cudaFree(ws->a_absmax);
    for (cudaEvent_t e : ws->span_ev)
        if (e) cudaEventDestroy(e);
    if (ws->svdj) cusolverDnDestroyGesvdjInfo(ws->svdj);
    if (ws->solver) cusolverDnDestroy(ws->solver);
    if (ws->rng) curandDestroyGenerator(ws->rng);
    cudaGetLastError();
    delete ws;
}

// Timing of the big products and all-reduces of the calls that follow (events on the call's stream).
cudaError_t svd_workspace_profile(SvdWorkspace *ws, bool on) {
    if (!ws) return cudaErrorInvalidValue;
    if (on)
        for (cudaEvent_t &e : ws->span_ev)
            if (!e && cudaEventCreate(&e) != cudaSuccess) return cudaErrorUnknown;
    ws->profile = on;
    ws->spans = 0;
    return cudaSuccess;
}
// Durations of the last call's spans, in call order; the call's stream must have been waited for.
int svd_workspace_spans(SvdWorkspace *ws, float *ms, int *kinds, int capacity) {
    if (!ws || !ws->profile) return 0;
    int n = 0;
    for (int i = 0; i < ws->spans && n < capacity; ++i) {
        float t = 0.0f;
        if (cudaEventElapsedTime(&t, ws->span_ev[2 * i], ws->span_ev[2 * i + 1]) != cudaSuccess) { cudaGetLastError(); continue; }
        if (ms) ms[n] = t;
        if (kinds) kinds[n] = ws->span_kind[i];
        ++n;
    }
    return n;
}

// Waits for the stream and reads the workspace's own status word (calls made without a caller status word).
cudaError_t svd_workspace_finish(SvdWorkspace *ws, cudaStream_t st) {
    unsigned h = 0;
    cudaError_t err = cudaMemcpyAsync(&h, ws->own_status, sizeof(unsigned), cudaMemcpyDeviceToHost, st);
    if (err == cudaSuccess) err = cudaStreamSynchronize(st);
    if (err != cudaSuccess) return err;
    return h == 0 ? cudaSuccess : cudaErrorLaunchTimeout;
}

cudaError_t svd_lowrank(SvdWorkspace *ws, const float *d_A, float *d_U, float *d_S, float *d_V, unsigned long long seed,
                        unsigned *d_status, cudaStream_t st, unsigned long long offset, const unsigned *d_abs_bound) {
    if (!ws || !d_A || !d_U || !d_S || !d_V) return cudaErrorInvalidValue;
    const int k = ws->k;
    ws->spans = 0;
    ws->status = d_status ? d_status : ws->own_status;    // bounded waits of the tensor-core GEMMs report here
    if (!d_status && cudaMemsetAsync(ws->own_status, 0, sizeof(unsigned), st) != cudaSuccess) return cudaErrorUnknown;
    if (curandSetStream(ws->rng, st) != CURAND_STATUS_SUCCESS) return cudaErrorUnknown;
    if (cusolverDnSetStream(ws->solver, st) != CUSOLVER_STATUS_SUCCESS) return cudaErrorUnknown;
    // Omega depends on the seed and the shape only (the generator is set back to the start of the seed's sequence for
    // every call), so it is drawn once per workspace and seed and kept: re-seeding costs a kernel of its own.
    if (!ws->seeded || ws->seed != seed || ws->offset != offset) {
        if (curandSetPseudoRandomGeneratorSeed(ws->rng, seed) != CURAND_STATUS_SUCCESS) return cudaErrorUnknown;
        if (curandSetGeneratorOffset(ws->rng, offset) != CURAND_STATUS_SUCCESS) return cudaErrorUnknown;
        size_t count = (size_t)ws->N * k;
        count += count & 1;                               // the normal generator wants an even count
        if (curandGenerateNormal(ws->rng, ws->omega, count, 0.0f, 1.0f) != CURAND_STATUS_SUCCESS) return cudaErrorUnknown;
        ws->seeded = true;
        ws->seed = seed;
        ws->offset = offset;
    }

    cudaError_t err;
    float *q = nullptr, *qz = nullptr, *spare = nullptr;
    // the largest |A|, once per call: from 256 columns on the six products with A split it into FP16 halves scaled by a power of two
    // from it (or a bound that the caller already has)
    ws->a_absmax_use = d_abs_bound ? d_abs_bound : ws->a_absmax;
    ws->a_absmax_valid = k >= 256 && (d_abs_bound != nullptr ||
                                      (ws->n % 4 == 0 && reinterpret_cast<uintptr_t>(d_A) % 16 == 0 &&
                                       gemm_absmax_bits(d_A, ws->n, ws->m, ws->n, ws->a_absmax, st) == cudaSuccess));
    // Y = W Omega, Q = orth(Y).  Panels ping-pong between the two buffers of their size.
    if ((err = times_w(ws, d_A, false, ws->omega, true, ws->y, st)) != cudaSuccess) return err;
    const int last_passes = 2;
    if ((err = orthonormalise(ws, ws->y, ws->y2, ws->M, ws->niter == 0 ? last_passes : 1, nullptr, nullptr, &q, true, st)) != cudaSuccess)
        return err;
    for (int it = 0; it < ws->niter; ++it) {
        if ((err = times_w(ws, d_A, true, q, false, ws->z, st)) != cudaSuccess) return err;               // Z = W^T Q
        if ((err = orthonormalise(ws, ws->z, ws->z2, ws->N, 1, nullptr, nullptr, &qz, false, st)) != cudaSuccess) return err;
        spare = (q == ws->y) ? ws->y2 : ws->y;
        if ((err = times_w(ws, d_A, false, qz, false, spare, st)) != cudaSuccess) return err;             // Y = W Qz
        float *other = (spare == ws->y) ? ws->y2 : ws->y;
        if ((err = orthonormalise(ws, spare, other, ws->M, it + 1 == ws->niter ? last_passes : 1, nullptr, nullptr, &q, true, st)) !=
            cudaSuccess)
            return err;
    }
    // B^T = W^T Q = Q2 C with C = R2 R1.  Where the Jacobi kernel does not accumulate the right factor, that comes from the panel B^T
    // itself (B^T v_j / S(j)), so Q2 is never formed: the second pass only has to deliver R2.
    const bool from_panel = ws->own_core_svd && (k > kJacobiSingleMaxK || ws->block_core) && !ws->jc_with_v;
    if ((err = times_w(ws, d_A, true, q, false, ws->z, st)) != cudaSuccess) return err;
    if ((err = orthonormalise(ws, ws->z, ws->z2, ws->N, 2, ws->tinv1, ws->tinv2, &qz, false, st, from_panel)) != cudaSuccess) return err;
    if (from_panel) qz = ws->z;
    if ((err = gemm(true, false, ws->tinv2, k, ws->tinv1, k, ws->core, k, k, k, k, nullptr, nullptr, 0, nullptr, ws->status, nullptr, 0,
                    ws->sm_count, st, nullptr, 0.0f, ws->device_full)) != cudaSuccess)
        return err;
    // The row-major C read as column-major is C^T = Vc S Uc^T: the solver's "U" is Vc, its "V" is Uc.
    if (ws->block_core) {
        cudaLaunchConfig_t cfg = {};
        cudaLaunchAttribute attr[2];
        block_jacobi_config(&cfg, attr, k, ws->jc_with_v, st);
        const float *core = ws->core;
        float *vc = ws->vc, *uc = ws->uc;
        if ((err = cudaLaunchKernelEx(&cfg, block_jacobi_fn(k, ws->jc_with_v), core, k, d_S, vc, uc)) != cudaSuccess) return err;
    } else if (ws->own_core_svd && k > kRingMinK) {
        cudaLaunchConfig_t cfg = {};
        cudaLaunchAttribute attr[2];
        ring_jacobi_config(&cfg, attr, ws->ring, st);
        const float *core = ws->core;
        float *vc = ws->vc, *uc = ws->uc;
        unsigned *status = ws->status;
        if ((err = cudaLaunchKernelEx(&cfg, ws->ring.fn, core, k, d_S, vc, uc, status)) != cudaSuccess) return err;
    } else if (ws->own_core_svd) {
        // eight lanes per pair and no more: warps without a pair only make a round's barrier longer (k = 64: 301 -> 290 us)
        const int threads = std::max(1, ((k + 1) / 2 * 8 + 31) / 32) * 32;
        if ((err = launch_chained(jacobi_svd_kernel, 1, threads, jacobi_smem_bytes(k), st, ws->core, k, d_S, ws->vc, ws->uc)) != cudaSuccess)
            return err;
    } else if (cusolverDnSgesvdj(ws->solver, CUSOLVER_EIG_MODE_VECTOR, 0, k, k, ws->core, k, d_S, ws->vc, k, ws->uc, k,
                                 ws->solver_work, ws->lwork, ws->dev_info, ws->svdj) != CUSOLVER_STATUS_SUCCESS) {
        return cudaErrorUnknown;
    }
    // W = (Q Vc) S (Q2 Uc)^T; both k x k factors are column-major, i.e. K-major B operands.  (from_panel: qz is the
    // panel B^T itself and column j of uc is Vc(:, j) / S(j): B^T Vc(:, j) / S(j) is the vector Q2 Uc(:, j).)
    float *d_left = ws->transposed ? d_V : d_U;            // M x k factor
    float *d_right = ws->transposed ? d_U : d_V;           // N x k factor
    if ((err = gemm(true, true, q, k, ws->vc, k, d_left, k, ws->M, k, k, nullptr, nullptr, 0, nullptr, ws->status, ws->gemm_ws, ws->gemm_ws_bytes,
                    ws->sm_count, st, nullptr, 0.0f, ws->device_full)) != cudaSuccess)
        return err;
    return gemm(true, true, qz, k, ws->uc, k, d_right, k, ws->N, k, k, nullptr, nullptr, 0, nullptr, ws->status, ws->gemm_ws, ws->gemm_ws_bytes,
                ws->sm_count, st, nullptr, 0.0f, ws->device_full);
}

size_t reconstruct_workspace_bytes(int m, int n, int k) {
    // V's images, and in front of them U diag(S) split beforehand (the persistent product of bsq_gemm.cu)
    return n > 256 ? gemm_tc_image_bytes(n, 256, k) + ((gemm_tc_a_image_bytes(m, k) + 127) & ~(size_t)127) + 1024 : 0;
}

cudaError_t reconstruct_lowrank(const float *d_U, const float *d_S, const float *d_V, int m, int n, int k,
                                const float *d_minuend, float *d_out, unsigned *d_flag, unsigned *d_status, float *d_workspace,
                                size_t workspace_bytes, int sm_count, cudaStream_t st, const unsigned *d_max_us, const unsigned *d_max_v) {
    if (!d_U || !d_S || !d_V || !d_out || m <= 0 || n <= 0 || k <= 0) return cudaErrorInvalidValue;
    // out(i, j) = sum_t (U(i, t) S(t)) V(j, t): A = U as stored with a per-k scale, B = V^T (K-major)
    return gemm(true, true, d_U, k, d_V, k, d_out, n, m, n, k, d_S, d_minuend, n, d_flag, d_status, d_workspace, workspace_bytes, sm_count, st,
                d_max_us, 0.0f, false, d_max_v);
}

}  // namespace bsq

// SVD of the k x k core of the randomized SVD where the factors are coded afterwards (NF4 / NF4_DQ sections, error lists made
// from them): one-sided (Hestenes) Jacobi with the columns in registers, moving from warp to warp around a ring (sm_100a).
//
// The reference runs cusolverDnSgesvd on the k x n matrix B (svd_lowrank_cuda.cu:399-440); here only the k x k
// triangular factor is left to decompose.
//   in : C, row-major k x k; read as the column-major matrix M = C^T (column j = row j of C)
//   out: M = U diag(S) V^T with S descending; U column-major k x k; Vcol column-major k x k: V itself (kWithV), or
//        column j of M V divided by S(j)^2 -- the matrix that turns the panel the core came from into its singular vectors.
//
// Column pairs (p, q) are rotated until all columns of M V are orthogonal to tol, |m_p . m_q| <= tol |m_p| |m_q| with tol = sqrt(len) eps
// (LAPACK's sgesvj criterion), in the order of a round-robin tournament: codes and error lists are whole numbers that depend on the order
// of rotations and on every last bit, so this kernel takes the pairs in the order, and adds the products in the order, of the kernel
// that dealt the rows over a cluster of 8 CTAs (up to 64 columns: of jacobi_svd_kernel), and gives the same bits.
//
// What bounds it is one dependent chain -- dot product, angle, rotation -- per round of disjoint pairs, k - 1 rounds per sweep and 7 to
// 9 sweeps whatever the split.  In that order a column only ever moves to the neighbouring pair: as p one slot down, as q one slot up,
// turning at the ends.  So whole columns stay in a warp's registers, four pairs (slots) per warp, and per round two columns per warp go
// to the neighbours through shared memory, those at a CTA's border through distributed shared memory, with their norms.  A warp adds its
// four dot products in one butterfly whose halves end with different slots, so the four angles are worked out side by side.
// (Rows dealt over the CTAs: every column through shared memory in every round, and the partial products of every round from and to every CTA.)
// Four warps per CTA, one per scheduler: eight measured 10 to 20 % slower, sixteen on one CTA 45 % (128 columns).
//   Against the kernels that it stands for, core alone: k = 256 1545 -> 1008 us, 192 1150 -> 761, 131 799 -> 563, 128 517 -> 413, 65 258 -> 221,
//   64 249 -> 199.  Up to kRingMinK columns jacobi_svd_kernel is as fast or faster (48 160 / 158, 16 48 / 44).
#pragma once

#include "bsq_device.cuh"
#include "bsq_jacobi.cuh"

#include <cooperative_groups.h>

namespace bsq {
namespace {

constexpr int kRingMinK = 48, kRingMaxK = 256;              // used above the one and up to the other
constexpr int kRingSlots = 4;                                // column pairs of a warp
__host__ __device__ constexpr int ring_pairs(int k) { return (k + 1) / 2; }
__host__ __device__ constexpr int ring_warps(int k) { return (ring_pairs(k) + kRingSlots - 1) / kRingSlots; }
constexpr int kRingWarps = 4;                                // of a CTA, but for the one CTA that takes up to 64 columns
__host__ __device__ constexpr int ring_max_threads(int len) { return len == 64 ? 256 : 32 * kRingWarps; }

// ... and stores of some of a warp's lanes, without a branch
__device__ __forceinline__ void st1_async_if(unsigned at, float v, unsigned mbar, unsigned on) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %3, 0;\n\t@p st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.f32 [%0], %1, [%2];\n\t}" ::"r"(at),
                 "f"(v), "r"(mbar), "r"(on)
                 : "memory");
}
__device__ __forceinline__ void st1_if(unsigned at, float v, unsigned on) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %2, 0;\n\t@p st.shared.f32 [%0], %1;\n\t}" ::"r"(at), "f"(v), "r"(on) : "memory");
}
__device__ __forceinline__ float lds1(unsigned at) {
    float v;
    asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(at) : "memory");
    return v;
}
__device__ __forceinline__ float div_ftz(float a, float b) {
    float r;
    asm("div.approx.ftz.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
    return r;
}

template <int kLen, bool kWithV>
struct RingShape {
    static constexpr bool kSplitLanes = kLen == 64 && kWithV;            // V in the upper half of the warp
    static constexpr int kRows = kLen == 256 ? 8 : 4;                    // rows of M per lane
    static constexpr int kVals = kRows * (kWithV && !kSplitLanes ? 2 : 1);      // floats per lane and column
    static constexpr int kN2 = kVals / 2, kCol = 32 * kVals;             // float2 per lane; floats per column in shared memory
};
// dynamic shared memory of one CTA: boxes [2 parities][warps][2 sides], carried norms, all norms, votes, mbarriers
template <int kLen, bool kWithV>
__host__ __device__ constexpr size_t ring_smem_bytes(int warps) {
    return ((size_t)4 * warps * RingShape<kLen, kWithV>::kCol + 4 * warps * kRingSlots + 2 * kRingMaxK + 2 * 16) * sizeof(float) + 4 * sizeof(uint64_t);
}

template <int kLen, bool kWithV, bool kCluster>
__global__ void __launch_bounds__(ring_max_threads(kLen), 1) ring_jacobi_kernel(const float *C, int k, float *__restrict__ S,
                                                                                float *__restrict__ Ucol, float *__restrict__ Vcol,
                                                                                unsigned *__restrict__ status) {
    static_assert(kLen > 64 || kWithV, "one CTA keeps V in the upper half of its warps");
    using Shape = RingShape<kLen, kWithV>;
    constexpr int kRows = Shape::kRows, kN2 = Shape::kN2, kCol = Shape::kCol, kS = kRingSlots, kQ = Shape::kVals / 4;
    constexpr bool kSplit = Shape::kSplitLanes;
    namespace cg = cooperative_groups;
    cg::cluster_group cluster = cg::this_cluster();
    const int cr = kCluster ? (int)cluster.block_rank() : 0, ctas = kCluster ? (int)cluster.num_blocks() : 1;
    extern __shared__ __align__(16) float sm[];
    chain_begin();
    const int tid = threadIdx.x, lane = tid & 31, w = __shfl_sync(kFullMask, tid >> 5, 0), wpc = blockDim.x >> 5;
    const int spc = wpc * kS;                                 // slots of a CTA
    float *boxes = sm;                                        // [parity][warp][0: from above (p), 1: from below (q)][kCol]
    float *norms = boxes + 4 * wpc * kCol;                    // [parity][0: p, 1: q][slot of the CTA]
    float *nall = norms + 4 * spc;                            // [parity of the sweep][column]
    int *votes = reinterpret_cast<int *>(nall + 2 * kRingMaxK);          // [parity of the sweep][CTA]
    uint64_t *mbar = reinterpret_cast<uint64_t *>(votes + 32);           // [0: from above, 1: from below][parity]
    const int kp = (k + 1) & ~1, npairs = kp / 2, rounds = kp - 1;
    const int gw = cr * wpc + w, top_w = (npairs - 1) / kS, top_j = (npairs - 1) % kS;
    const bool is_top = gw == top_w, is_bot = gw == 0, is_end = is_top || is_bot, works = gw <= top_w;
    const bool rem_up = kCluster && w == wpc - 1 && gw < top_w;          // the warp above is in the next CTA
    const bool rem_dn = kCluster && w == 0 && gw > 0 && gw <= top_w;     // the warp below is in the CTA before

    // the slot whose angle this lane works out, and the lane that does it for slot j
    const bool hi = kLen == 64 ? (lane & 8) != 0 : (lane & 2) != 0, odd = kLen == 64 ? (lane & 4) != 0 : (lane & 1) != 0;
    const int own = (kLen == 256 ? (hi ? 0 : 2) : (hi ? 2 : 0)) + (odd ? 1 : 0);
    constexpr auto lane_of = [](int j) constexpr { return kLen == 256 ? ((j & 2) ? 0 : 2) + (j & 1) : (kLen == 128 ? j : 4 * j); };
    const bool leader = lane == lane_of(own);
    const int gs = gw * kS + own;                             // that slot, counted over the cluster
    const bool on = gs < npairs;
    // where the norms of this lane's slot go after a round
    unsigned np_to, nq_to;                                    // address for parity 0
    unsigned np_remote = 0, nq_remote = 0;
    {
        int ps = gs, pside = 0, qs = gs, qside = 1;
        if (gs == 0) ps = 0;
        else if (gs == 1) { ps = 0; pside = 1; }
        else ps = gs - 1;
        if (gs == npairs - 1) qside = 0;
        else qs = gs + 1;
        if (gs == 0 && npairs == 1) { qs = 0; qside = 1; }
        const int pc = kCluster ? min(ps / spc, ctas - 1) : 0, qc = kCluster ? min(qs / spc, ctas - 1) : 0;
        np_to = smem_u32(norms + pside * spc + (ps - pc * spc));
        nq_to = smem_u32(norms + qside * spc + (qs - qc * spc));
        if (kCluster && pc != cr) { np_remote = 1; np_to = cluster_addr(np_to, pc); }
        if (kCluster && qc != cr) { nq_remote = 1; nq_to = cluster_addr(nq_to, qc); }
    }
    const unsigned np_local = leader && on && !np_remote, nq_local = leader && on && !nq_remote;
    np_remote = np_remote && leader && on;
    nq_remote = nq_remote && leader && on;
    // outgoing columns: down (P of the warp's slot 0) into the box "from above" of the warp below -- the lowest warp's into its
    // own box "from below" -- and up (Q of the last slot) into the box "from below" of the warp above; the top warp's into its own
    // "from above"
    const unsigned lane_off = lane * 16;
    unsigned dn_to, up_to, dn_bar = 0, up_bar = 0;
    {
        const int dw = is_bot ? 0 : (rem_dn ? wpc - 1 : w - 1), uw = is_top ? w : (rem_up ? 0 : w + 1);
        dn_to = smem_u32(boxes + (max(dw, 0) * 2 + (is_bot ? 1 : 0)) * kCol) + lane_off;
        up_to = smem_u32(boxes + (min(uw, wpc - 1) * 2 + (is_top ? 0 : 1)) * kCol) + lane_off;
        if (kCluster) {
            dn_bar = smem_u32(mbar);
            up_bar = smem_u32(mbar + 2);
            if (rem_dn) { dn_to = cluster_addr(dn_to, (unsigned)(cr - 1)); dn_bar = cluster_addr(dn_bar, (unsigned)(cr - 1)); }
            if (rem_up) { up_to = cluster_addr(up_to, (unsigned)(cr + 1)); up_bar = cluster_addr(up_bar, (unsigned)(cr + 1)); }
        }
    }
    const unsigned box_par = 2 * wpc * kCol * sizeof(float), norm_par = 2 * spc * sizeof(float);
    const unsigned norm_at = smem_u32(norms + w * kS + own), box_at = smem_u32(boxes + w * 2 * kCol) + lane_off;
    constexpr unsigned kTx = kCol * sizeof(float) + sizeof(float);
    if (kCluster && tid == 0) {
#pragma unroll
        for (int i = 0; i < 4; ++i) mbar_init(&mbar[i], 1);
        mbar_fence_init();
#pragma unroll
        for (int i = 0; i < 4; ++i) mbar_expect_tx(&mbar[i], kTx);
    }
    if (kCluster) cluster.sync();                             // every CTA runs, its mbarriers ready, before anybody stores into its shared memory

    // ---- this warp's columns ----
    // slot s: p = s (the last column in slot 0), q = kp - 1 - s (column 0 in slot 0)
    float2 P[kS][kN2], Q[kS][kN2];
    auto col_of = [&](int j, int side) {
        const int s = gw * kS + j;
        return side == 0 ? (s == 0 ? kp - 1 : s) : (s == 0 ? 0 : kp - 1 - s);
    };
    // value v of this lane's share: row of M (or of V)
    auto row_of = [&](int v) {
        if (kLen == 256) {
            const int r = v % kRows;                          // pairs: element r / 2 of float4 number 2 h + (r & 1) of the slice
            return (lane >> 2) * 32 + ((2 * ((lane >> 1) & 1) + (r & 1)) * 2 + (lane & 1)) * 4 + (r >> 1);
        }
        return (lane & (kSplit ? 15 : 31)) * 4 + v % kRows;
    };
    auto init = [&](float2 (&X)[kN2], int c) {
#pragma unroll
        for (int v = 0; v < Shape::kVals; ++v) {
            const int i = row_of(v);
            const bool is_v = kSplit ? lane >= 16 : v >= kRows;
            float x = 0.0f;
            if (c < k && i < k) x = is_v ? (i == c ? 1.0f : 0.0f) : C[(size_t)c * k + i];
            if (v & 1) X[v / 2].y = x;
            else X[v / 2].x = x;
        }
    };
#pragma unroll
    for (int j = 0; j < kS; ++j) {
        const bool have = gw * kS + j < npairs;
        init(P[j], have ? col_of(j, 0) : k);
        init(Q[j], have ? col_of(j, 1) : k);
    }
    // this lane's part of x . y, in the order of the sums: four rows from the first to the last (two such sums for 8 rows)
    auto dot4 = [&](const float2 (&X)[kN2], const float2 (&Y)[kN2], float &ta, float &tb) {
        if (kLen == 256) {
            float2 t = mul2(X[1], Y[1]);
            t = fma2(X[0], Y[0], t);
            t = fma2(X[2], Y[2], t);
            t = fma2(X[3], Y[3], t);
            ta = t.x;
            tb = t.y;
        } else {
            float t = __fmul_rn(X[0].y, Y[0].y);
            t = __fmaf_rn(X[0].x, Y[0].x, t);
            t = __fmaf_rn(X[1].x, Y[1].x, t);
            ta = __fmaf_rn(X[1].y, Y[1].y, t);
            tb = 0.0f;
        }
    };
    // squared norm of a column, the same value in every lane
    auto norm2 = [&](const float2 (&X)[kN2]) {
        float ta, tb;
        dot4(X, X, ta, tb);
        if (kLen == 64) {
#pragma unroll
            for (int d = 8; d > 0; d >>= 1) ta += __shfl_xor_sync(kFullMask, ta, d);
            return __shfl_sync(kFullMask, ta, 0);
        }
        if (kLen == 256) {
            const float o = __shfl_xor_sync(kFullMask, ta + tb, 2);      // the lower half's sum, in the lanes of the upper half
            ta = (o + ta) + tb;
        } else {
            ta += __shfl_xor_sync(kFullMask, ta, 2);
        }
        ta += __shfl_xor_sync(kFullMask, ta, 1);
        float a = 0.0f;
#pragma unroll
        for (int d = 0; d < 8; ++d) a += __shfl_sync(kFullMask, ta, 4 * d + 2);
        return a;
    };
    const float tol = sqrtf((float)kLen) * 5.9604645e-08f, tol2 = tol * tol;
    auto rotate = [&](float2 (&X)[kN2], float2 (&Y)[kN2], float c, float s) {
        const float2 c2 = make_float2(c, c), s2 = make_float2(s, s), n2 = make_float2(-s, -s);
#pragma unroll
        for (int u = 0; u < kN2; ++u) {
            const float2 x = X[u], y = Y[u];
            X[u] = fma2(c2, x, mul2(n2, y));
            Y[u] = kLen == 128 ? fma2(c2, y, mul2(s2, x)) : fma2(s2, x, mul2(c2, y));
        }
    };
    auto put = [&](unsigned to, const float2 (&X)[kN2]) {
#pragma unroll
        for (int u = 0; u < kQ; ++u)
            asm volatile("st.shared.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(to + u * 512), "f"(X[2 * u].x), "f"(X[2 * u].y), "f"(X[2 * u + 1].x),
                         "f"(X[2 * u + 1].y)
                         : "memory");
    };
    auto put_remote = [&](unsigned to, const float2 (&X)[kN2], unsigned bar) {
#pragma unroll
        for (int u = 0; u < kQ; ++u) st_async_f4(to + u * 512, X[2 * u].x, X[2 * u].y, X[2 * u + 1].x, X[2 * u + 1].y, bar);
    };
    auto take = [&](unsigned at, float2 (&X)[kN2]) {
#pragma unroll
        for (int u = 0; u < kQ; ++u)
            asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(X[2 * u].x), "=f"(X[2 * u].y), "=f"(X[2 * u + 1].x), "=f"(X[2 * u + 1].y)
                         : "r"(at + u * 512) : "memory");
    };

    unsigned it = 0;                                          // rounds so far
    int vote = 1, sp_last = 0;                                // bit 0: a pair above kJacobiLastSweepCos in the last sweep, bit 1: a wait ran out
    bool failed = false;                                      // a wait ran out: stop sending and waiting, finish quickly
    unsigned failed_at = 0;                                   // ... in this round
    const int own_slot = w * kS + own;
    for (int sweep = 0;; ++sweep) {
        // exact squared norms (in between they are carried along through the rotations), into every CTA, with the votes
        const int sp = sp_last = sweep & 1;
        if (works) {
            float a_own = 0.0f, b_own = 0.0f;
#pragma unroll
            for (int j = 0; j < kS; ++j) {
                const float a = norm2(P[j]), b = norm2(Q[j]);
                if (own == j) { a_own = a; b_own = b; }
                if (gw * kS + j < npairs && lane < ctas) {
                    float *dst = kCluster ? cluster.map_shared_rank(nall, lane) : nall;
                    dst[sp * kRingMaxK + col_of(j, 0)] = a;
                    dst[sp * kRingMaxK + col_of(j, 1)] = b;
                }
            }
            if (leader) {
                norms[(it & 1) * 2 * spc + own_slot] = a_own;
                norms[(it & 1) * 2 * spc + spc + own_slot] = b_own;
            }
        }
        if (kCluster) {
            if (tid < ctas) cluster.map_shared_rank(votes, tid)[sp * 16 + cr] = vote;
            cluster.sync();
            vote = 0;
            for (int d = 0; d < ctas; ++d) vote |= votes[sp * 16 + d];
        } else {
            __syncthreads();
        }
        if (!(vote & 1) || (vote & 2) || sweep == kJacobiMaxSweeps) break;
        float seen = 0.0f;                                    // 1: this lane's slot met a pair above the bound of the last sweep
        // The sums of the pairs that stay inside the warp are begun in front of the round's barrier, while the columns of the others are on their
        // way (256 columns 1084 -> 1023 us), at 128 columns what only the end of a sweep wants comes last (375 -> 366 at rank 100), and rounds are unrolled where that helps: two
        // at 256 columns (1008), four at 64 (216 -> 199), none at 128 (two 413 -> 459).  Not so: columns that leave rotated and sent
        // before the others (128 columns 418 -> 447), what comes in taken from shared memory before the vote on the waits (462).
        constexpr int kUnroll = kLen == 64 ? 4 : kLen == 256 ? 2 : 1;
        float inner_a[2], inner_b[2];
        dot4(P[1], Q[1], inner_a[0], inner_b[0]);
        dot4(P[2], Q[2], inner_a[1], inner_b[1]);
#pragma unroll kUnroll
        for (int r = 0; r < rounds; ++r, ++it) {
            const unsigned par = it & 1, phase = (it >> 1) & 1;
            if (works) {
                const float alpha = lds1(norm_at + par * norm_par), beta = lds1(norm_at + par * norm_par + spc * 4);
                // ---- dot products: slot j's ends up in the eight (four) lanes that work out its angle ----
                float g;
                {
                    float ta[kS], tb[kS];
                    ta[1] = inner_a[0];
                    tb[1] = inner_b[0];
                    ta[2] = inner_a[1];
                    tb[2] = inner_b[1];
                    dot4(P[0], Q[0], ta[0], tb[0]);
                    dot4(P[3], Q[3], ta[3], tb[3]);
                    float g2[2], o[2];
                    if (kLen == 256) {
                        // slots 0 and 1 add the lower half's two sums first (in either order), slots 2 and 3 the upper half's:
                        // the lanes of the other half finish
#pragma unroll
                        for (int j = 0; j < 2; ++j) o[j] = __shfl_xor_sync(kFullMask, hi ? ta[j + 2] + tb[j + 2] : ta[j] + tb[j], 2);
                        g2[0] = (o[0] + (hi ? ta[0] : ta[2])) + (hi ? tb[0] : tb[2]);
                        g2[1] = (o[1] + (hi ? tb[1] : tb[3])) + (hi ? ta[1] : ta[3]);
                    } else {
#pragma unroll
                        for (int j = 0; j < 2; ++j) o[j] = __shfl_xor_sync(kFullMask, hi ? ta[j] : ta[j + 2], kLen == 128 ? 2 : 8);
#pragma unroll
                        for (int j = 0; j < 2; ++j) g2[j] = (hi ? ta[j + 2] : ta[j]) + o[j];
                    }
                    g = (odd ? g2[1] : g2[0]) + __shfl_xor_sync(kFullMask, odd ? g2[0] : g2[1], kLen == 64 ? 4 : 1);
                    if (kLen == 64) {
                        g += __shfl_xor_sync(kFullMask, g, 2);
                        g += __shfl_xor_sync(kFullMask, g, 1);
                    } else {
                        g += __shfl_xor_sync(kFullMask, g, 4);
                        g += __shfl_xor_sync(kFullMask, g, 8);
                        g += __shfl_xor_sync(kFullMask, g, 16);
                    }
                }
                const bool turn = on && alpha > 0.0f && beta > 0.0f && g * g > tol2 * alpha * beta;
                const unsigned turns = __ballot_sync(kFullMask, turn);
                // (lanes without a rotation take harmless values: a division by zero would send the warp down its slow path)
                const float num = turn ? beta - alpha : 1.0f, den = turn ? 2.0f * g : 1.0f;
                float t, c;
                if (kLen == 64) {
                    const float zeta = num / den;
                    t = fabsf(zeta) > 1.0e8f ? 0.5f / zeta : copysignf(1.0f, zeta) / (fabsf(zeta) + sqrtf(1.0f + zeta * zeta));
                    c = rsqrt_ftz(1.0f + t * t);
                } else {
                    // tangent, cosine and sine to a few units in the last place: what they leave of the pair's product is far below
                    // the tolerance.  (What the roots and the second quotient take is a normal number whatever zeta is.)
                    const float zeta = __fdividef(num, den), small = __fdividef(0.5f, zeta);
                    const float wz = fmaf(zeta, zeta, 1.0f);
                    t = div_ftz(copysignf(1.0f, zeta), fabsf(zeta) + wz * rsqrt_ftz(wz));
                    t = fabsf(zeta) > 1.0e8f ? small : t;
                    c = rsqrt_ftz(fmaf(t, t, 1.0f));
                }
                const float sn = c * t;
                float cj[kS], sj[kS];
#pragma unroll
                for (int j = 0; j < kS; ++j) {
                    cj[j] = __shfl_sync(kFullMask, c, lane_of(j));
                    sj[j] = __shfl_sync(kFullMask, sn, lane_of(j));
                }
                const float pn = turn ? fmaxf(alpha - t * g, 0.0f) : alpha, qn = turn ? beta + t * g : beta;
                if (kLen != 128) seen = turn && g * g > kJacobiLastSweepCos * kJacobiLastSweepCos * alpha * beta ? 1.0f : seen;
                constexpr unsigned kAll = 1u << lane_of(0) | 1u << lane_of(1) | 1u << lane_of(2) | 1u << lane_of(3);
                if ((turns & kAll) == kAll) {
                    rotate(P[0], Q[0], cj[0], sj[0]);
                    rotate(P[3], Q[3], cj[3], sj[3]);
                    rotate(P[1], Q[1], cj[1], sj[1]);
                    rotate(P[2], Q[2], cj[2], sj[2]);
                } else {
#pragma unroll
                    for (int j = 0; j < kS; ++j)
                        if (turns >> lane_of(j) & 1) rotate(P[j], Q[j], cj[j], sj[j]);
                }
                const unsigned to_norm = (par ^ 1) * norm_par;
                st1_if(np_to + to_norm, pn, np_local);
                st1_if(nq_to + to_norm, qn, nq_local);
                if (is_end) {
                    if (is_top) {                             // the ring turns: Q of the last slot comes back as its P
#pragma unroll
                        for (int j = 0; j + 1 < kS; ++j)
                            if (top_j == j) {
#pragma unroll
                                for (int u = 0; u < kN2; ++u) P[j + 1][u] = Q[j][u];
                            }
                    }
                    if (is_bot) {                             // ... and at the bottom around the column that stays
#pragma unroll
                        for (int u = 0; u < kN2; ++u) {
                            const float2 x = P[0][u];
                            P[0][u] = P[1][u];
                            P[1][u] = x;
                        }
                    }
                }
                if (kCluster && rem_dn) {
                    if (!failed) {
                        put_remote(dn_to + par * box_par, P[0], dn_bar + par * 8);
                        st1_async_if(np_to + to_norm, pn, dn_bar + par * 8, np_remote);
                    }
                } else {
                    put(dn_to + par * box_par, P[0]);
                }
                if (kCluster && rem_up) {
                    if (!failed) {
                        put_remote(up_to + par * box_par, Q[kS - 1], up_bar + par * 8);
                        st1_async_if(nq_to + to_norm, qn, up_bar + par * 8, nq_remote);
                    }
                } else {
                    put(up_to + par * box_par, Q[kS - 1]);
                }
                if (kLen == 128) seen = turn && g * g > kJacobiLastSweepCos * kJacobiLastSweepCos * alpha * beta ? 1.0f : seen;
                // everything moves one slot on
#pragma unroll
                for (int j = 0; j + 1 < kS; ++j)
#pragma unroll
                    for (int u = 0; u < kN2; ++u) P[j][u] = P[j + 1][u];
#pragma unroll
                for (int j = kS - 1; j > 0; --j)
#pragma unroll
                    for (int u = 0; u < kN2; ++u) Q[j][u] = Q[j - 1][u];
            }
            dot4(P[1], Q[1], inner_a[0], inner_b[0]);
            dot4(P[2], Q[2], inner_a[1], inner_b[1]);
            __syncthreads();
            if (works) {
                if (kCluster) {
                    // (uniform over the warp: a lane that gives up takes the others with it)
                    if (rem_up && !failed) {
                        failed = __any_sync(kFullMask, !mbar_wait_bounded(&mbar[par], phase, status));
                        if (lane == 0 && !failed) mbar_expect_tx(&mbar[par], kTx);
                    }
                    if (rem_dn && !failed) {
                        failed = __any_sync(kFullMask, !mbar_wait_bounded(&mbar[2 + par], phase, status));
                        if (lane == 0 && !failed) mbar_expect_tx(&mbar[2 + par], kTx);
                    }
                    if (failed && failed_at == 0) failed_at = it + 1;
                }
                take(box_at + par * box_par, P[kS - 1]);
                take(box_at + par * box_par + kCol * 4, Q[0]);
            }
        }
        vote = __syncthreads_or(leader && seen > 0.0f) ? 1 : 0;
        if (kCluster) vote |= __syncthreads_or(failed) ? 2 : 0;
    }

    // ---- singular values, order, output ----
    float *sv = nall + sp_last * kRingMaxK;
    for (int i = tid; i < kp; i += blockDim.x) sv[i] = sqrtf(sv[i]);
    __syncthreads();
    if (works) {
        auto out = [&](const float2 (&X)[kN2], int c) {
            if (c >= k) return;                               // (the padding column of an odd k)
            const float s = sv[c];
            int rk = 0;
            for (int i = lane; i < k; i += 32) {
                const float si = sv[i];
                rk += (si > s || (si == s && i < c)) ? 1 : 0;
            }
            rk = __reduce_add_sync(kFullMask, rk);
            if (lane == 0) S[rk] = s;
#pragma unroll
            for (int v = 0; v < Shape::kVals; ++v) {
                const int i = row_of(v);
                const bool is_v = kSplit ? lane >= 16 : v >= kRows;
                const float x = (v & 1) ? X[v / 2].y : X[v / 2].x;
                if (i >= k) continue;
                const size_t o = (size_t)rk * k + i;
                if (is_v) {
                    Vcol[o] = x;
                } else {
                    Ucol[o] = s > 0.0f ? x / s : 0.0f;
                    if (!kWithV) Vcol[o] = s > 0.0f ? x / (s * s) : 0.0f;
                }
            }
        };
#pragma unroll
        for (int j = 0; j < kS; ++j)
            if (gw * kS + j < npairs) {
                out(P[j], col_of(j, 0));
                out(Q[j], col_of(j, 1));
            }
    }
    if (kCluster) {
        // A warp that gave up: the neighbour may have sent the round that was waited for all the same, and the one behind it (not more, since
        // it got nothing back).  These stores land, or do not come, before this CTA's shared memory goes away.
        if (failed) {
            for (unsigned i = failed_at - 1; i <= failed_at; ++i) {
                if (rem_up) mbar_wait_bounded(&mbar[i & 1], (i >> 1) & 1, status);
                if (rem_dn) mbar_wait_bounded(&mbar[2 + (i & 1)], (i >> 1) & 1, status);
            }
        }
        cluster.sync();                                       // nobody leaves while a neighbour could still store into it
    }
}

typedef void (*RingJacobiFn)(const float *, int, float *, float *, float *, unsigned *);
struct RingLaunch {
    RingJacobiFn fn;
    int ctas, warps;                                          // warps per CTA
    size_t smem;
};
// The instance and the split for a core of k columns (up to 64 the right factor is always accumulated).
RingLaunch ring_jacobi_launch(int k, bool with_v) {
    const int all = ring_warps(k);
    if (k <= 64) return {ring_jacobi_kernel<64, true, false>, 1, all, ring_smem_bytes<64, true>(all)};
    RingLaunch r;
    r.ctas = (all + kRingWarps - 1) / kRingWarps;
    r.warps = (all + r.ctas - 1) / r.ctas;
    if (k <= 128) {
        r.fn = with_v ? ring_jacobi_kernel<128, true, true> : ring_jacobi_kernel<128, false, true>;
        r.smem = with_v ? ring_smem_bytes<128, true>(r.warps) : ring_smem_bytes<128, false>(r.warps);
    } else {
        r.fn = with_v ? ring_jacobi_kernel<256, true, true> : ring_jacobi_kernel<256, false, true>;
        r.smem = with_v ? ring_smem_bytes<256, true>(r.warps) : ring_smem_bytes<256, false>(r.warps);
    }
    return r;
}
void ring_jacobi_config(cudaLaunchConfig_t *cfg, cudaLaunchAttribute (&attr)[2], const RingLaunch &r, cudaStream_t st) {
    cfg->gridDim = dim3(r.ctas, 1, 1);
    cfg->blockDim = dim3(32 * r.warps, 1, 1);
    cfg->dynamicSmemBytes = r.smem;
    cfg->stream = st;
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = r.ctas;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg->attrs = attr;
    cfg->numAttrs = 2;
}

}  // namespace
}  // namespace bsq

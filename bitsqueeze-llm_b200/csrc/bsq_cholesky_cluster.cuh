// The Cholesky factor and its inverse of bsq_cholesky.cuh by a cluster of CTAs, one for every 32 columns, 32 < k <= 256 (sm_100a).
//
// Same blocks, same sums in the same order, so the same bits; what differs is where they are made.  One CTA that factors is bound by
// its own multiply-adds above 200 columns (53 us at 256, of which the chain of pivots is 14), and a small matrix waits for the CTA that
// makes the inverse, which learns of every block row through global memory.  Here CTA c keeps block column c:
//   * CTA J walks the pivots of its diagonal block; every eight of them go to the CTAs behind it by bulk copies into their shared memory,
//     which count off on mbarriers there.  CTA c makes block (J, c) of the factor behind them, and its own diagonal block behind that,
//     so that CTA J + 1 starts its pivots about 1500 clocks after CTA J has finished.
//   * Block (J, c) goes on to the CTAs behind c, which take its product with their own block of row J from the blocks above their diagonal.
//   * When its pivots are done, CTA c makes block row c of the inverse, T_cJ = -(sum_L T_cL R_LJ) T_JJ from left to right: all that it needs
//     from others are the blocks of R, which they send it as well, and the inverses of their diagonal blocks.  So it goes on beside the
//     pivots, and behind the last of them are left the inverse of one diagonal block and one product.  (By columns every T_cJ would wait for
//     another CTA's: 63 us at 256 columns instead of 32.)
// Every barrier is used once per launch; waits are bounded and nobody leaves a barrier out because one ran out.
// Factor and inverse 32 us at 256 columns (71 us by one CTA and those of the inverse), 20 at 128 (31.5), 11.2 at 64 (14.4), 10.7 at 48 (15.3): per
// 32 columns the chain of pivots, 1.75 us, and as much again until the next CTA's can begin.  It is the better one where other matrices
// fill the device as well: eight compress calls of 4096 x 14336 at rank 256 side by side 9.89 ms, by a kernel of one CTA and one of seven 10.01,
// six of 8192 x 4096 5.16 and 5.28.
#pragma once

#include "bsq_cholesky.cuh"

#include <cooperative_groups.h>

namespace bsq {
namespace {

constexpr int kCcMaxBlocks = kCholeskyBlockedMaxK / kCB;
constexpr int kCcPairs = 3;                                // pairs of warps for what can wait while a column is made
constexpr int kCcDia = kCBB + 3 * kCB;                     // a row of zeros, the block, room for reads that run on, 1 / diagonal
struct CcBars {
    uint64_t dia[kCcMaxBlocks][kCB / kCholStep];           // rows of R_JJ from CTA J
    uint64_t blk[kCcMaxBlocks * (kCcMaxBlocks - 1) / 2];   // R_JA from CTA A, at cc_pair(J, A)
    uint64_t tjj[kCcMaxBlocks];                            // T_JJ from CTA J
    int failed;
};
__host__ __device__ constexpr int cc_pair(int J, int A) { return A * (A - 1) / 2 + J; }
// Offsets in floats, the same in every CTA of a launch.  col: blocks (0 .. c, c) of the factor, behind them the sums of the inverse's
// blocks (c, J); rblk: what comes of the other columns; dia: R_JJ for J <= c, T_JJ for the others; tjj: T_cc; tij: T_cJ^T.
struct CcLayout {
    int col, rblk, dia, tjj, tij, red, bars, total;
    __host__ __device__ constexpr explicit CcLayout(int nb)
        : col(0), rblk(nb * kCBB), dia(rblk + nb * (nb - 1) / 2 * kCBB), tjj(dia + nb * kCcDia), tij(tjj + kCBB), red(tij + kCB * kCTs),
          bars(red + kCB), total(bars + (int)(sizeof(CcBars) + 15) / 16 * 4) {}
};
__host__ __device__ constexpr size_t cholesky_cluster_smem_bytes(int k) { return (size_t)CcLayout(chol_blocks(k)).total * sizeof(float); }

// shared memory of this CTA -> that of another one of the cluster, counted in bytes on an mbarrier there
__device__ __forceinline__ void cluster_copy(unsigned dst, unsigned src, unsigned bytes, unsigned bar) {
    asm volatile("cp.async.bulk.shared::cluster.shared::cta.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst), "r"(src), "r"(bytes),
                 "r"(bar)
                 : "memory");
}
__device__ __forceinline__ void cc_wait(uint64_t *bar, CcBars *bars, unsigned *status) {
    for (unsigned i = 0; i < kMbarSpinLimit; ++i) {
        unsigned ok;
        asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], 0;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                     : "=r"(ok)
                     : "r"(smem_u32(bar))
                     : "memory");
        if (ok) return;
        if ((i & 1023u) == 1023u && *reinterpret_cast<volatile int *>(&bars->failed)) return;       // (one wait that ran out is enough)
    }
    *reinterpret_cast<volatile int *>(&bars->failed) = 1;
    if (status) atomicOr(status, kStatusBarrierTimeout);
}

// Named barriers: 1 - 4 eight pivots are done, 5 block (J, c) is done, 6 - 9 eight rows of it, 10 step J is over for block (J + 1, c), 11 the
// diagonal block is complete, 12 all pivots are done.
constexpr int kCcRowDone = 5, kCcStepOver = 10, kCcDiagonal = 11, kCcPivots = 12;
constexpr int kCcUpdaters = 64 * kCcPairs;

__global__ void __launch_bounds__(kCholThreads, 1) cholesky_cluster_kernel(const float *G, int k, float *R, float *T, unsigned *status) {
    chain_begin();
    namespace cg = cooperative_groups;
    cg::cluster_group cluster = cg::this_cluster();
    const int c = (int)cluster.block_rank(), nb = (int)cluster.num_blocks();
    const CcLayout at(nb);
    float *sm = chol_smem();
    CcBars *bars = reinterpret_cast<CcBars *>(sm + at.bars);
    float *col = sm + at.col;                              // block (I, c) at I
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int col0 = c * kCB;
    if (tid == 0) {
        for (int J = 0; J < nb; ++J) {
            for (int g = 0; g < kCB / kCholStep; ++g) {
                mbar_init(&bars->dia[J][g], 1);
                if (J < c) mbar_expect_tx(&bars->dia[J][g], (kCholStep * kCB + kCholStep) * sizeof(float));
            }
            mbar_init(&bars->tjj[J], 1);
            if (T && J > c) mbar_expect_tx(&bars->tjj[J], kCBB * sizeof(float));
            for (int A = J + 1; A < nb; ++A) {
                mbar_init(&bars->blk[cc_pair(J, A)], 1);
                if (A < c || (T && J >= c && A > c)) mbar_expect_tx(&bars->blk[cc_pair(J, A)], kCBB * sizeof(float));
            }
        }
        bars->failed = 0;
        mbar_fence_init();
    }
    // load, padded with an identity (what lies below the diagonal of the diagonal block is never used)
    for (int e = tid; e < (c + 1) * (kCBB / 4); e += kCholThreads) {
        const int u = e % (kCBB / 4), i = e / (kCBB / 4) * kCB + (u >> 3), j = col0 + 4 * (u & 7);
        float *dst = col + (size_t)4 * e;
        if ((k & 3) == 0 && i < k && j < k) {
            copy16_async(dst, G + (size_t)i * k + j);
        } else {
#pragma unroll
            for (int q = 0; q < 4; ++q) dst[q] = (i < k && j + q < k) ? G[(size_t)i * k + j + q] : (i == j + q ? 1.0f : 0.0f);
        }
    }
    float md = tid < k ? fmaxf(G[(size_t)tid * k + tid], 0.0f) : 0.0f;
    for (int d = 16; d > 0; d >>= 1) md = fmaxf(md, __shfl_xor_sync(0xffffffffu, md, d));
    if (lane == 0) sm[at.red + warp] = md;
    // the last block's pivots end with the matrix, by whole steps: what follows is the identity as the pivots would leave it
    const int steps = c == nb - 1 ? (k - col0 + kCholStep - 1) / kCholStep : kCB / kCholStep;
    float *dia = sm + at.dia + c * kCcDia + kCB, *dinv = dia + kCBB + kCB;
    if (tid < kCB) {
        dia[tid - kCB] = 0.0f;
        dinv[tid] = 1.0f;
    }
    for (int e = kCholStep * steps * kCB + tid; e < kCBB; e += kCholThreads) dia[e] = e / kCB == e % kCB ? 1.0f : 0.0f;
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
    float m = 0.0f;
#pragma unroll
    for (int w = 0; w < kCholeskyBlockedMaxK / 32; ++w) m = fmaxf(m, sm[at.red + w]);
    const float shift = m > 0.0f ? m * 1.0e-5f : 0.0f, half = 0.5f * shift;
    if (tid < kCB && col0 + tid < k) col[(size_t)c * kCBB + tid * (kCB + 1)] += shift;
    __syncthreads();
    cluster.sync();                                        // every CTA runs, its mbarriers ready, before anybody copies into its shared memory
    // the same place in CTA `to`, a lane per CTA
    const auto put_remote = [&](int to, int offset, int floats, uint64_t *bar) {
        const unsigned here = smem_u32(sm + offset);
        cluster_copy(cluster_addr(here, to), here, floats * sizeof(float), cluster_addr(smem_u32(bar), to));
    };
    const int wi = (warp & 3) ? (warp >> 2) * 3 + (warp & 3) - 1 : -1;              // warps off the pivots' scheduler

    if (warp == 0) {
        if (c > 0) bar_sync(kCcDiagonal, 96);
        const int at_dia = at.dia + c * kCcDia + kCB;
        if (half >= 1.17549435e-38f) factor_diagonal<true>(at.col + c * kCBB, at_dia, at_dia + kCBB + kCB, half, 64, steps);
        else factor_diagonal<false>(at.col + c * kCBB, at_dia, at_dia + kCBB + kCB, half, 64, steps);
        bar_arrive(kCcPivots, 64);
    } else if (warp == 4) {
        // the pivots' rows as they come: to the CTAs behind this one, and out
        for (int g = 0; g < steps; ++g) {
            bar_sync(1 + g, 64);
            if (c + 1 < nb) {                              // the next CTA waits for them: stores, which are there sooner than copies
                const unsigned bar = cluster_addr(smem_u32(&bars->dia[c][g]), c + 1);
                const unsigned rows = smem_u32(dia + g * kCholStep * kCB) + lane * 16, there = cluster_addr(rows, c + 1);
                const float4 x = lds4(rows), y = lds4(rows + 512);
                st_async_f4(there, x.x, x.y, x.z, x.w, bar);
                st_async_f4(there + 512, y.x, y.y, y.z, y.w, bar);
                if (lane < kCholStep / 4) {
                    const unsigned inv = smem_u32(dinv + g * kCholStep) + lane * 16;
                    const float4 z = lds4(inv);
                    st_async_f4(cluster_addr(inv, c + 1), z.x, z.y, z.z, z.w, bar);
                }
            }
            fence_proxy_async_smem();
            if (lane > c + 1 && lane < nb) {
                put_remote(lane, at.dia + c * kCcDia + kCB + g * kCholStep * kCB, kCholStep * kCB, &bars->dia[c][g]);
                put_remote(lane, at.dia + c * kCcDia + 2 * kCB + kCBB + g * kCholStep, kCholStep, &bars->dia[c][g]);
            }
        }
        for (int i = 0; i < kCB; ++i)
            if (col0 + i < k && col0 + lane < k) R[(size_t)(col0 + i) * k + col0 + lane] = lane < i ? 0.0f : dia[i * kCB + lane];
    } else if (warp == 8) {
        // zeros below the diagonal blocks; block (J, c) of R out; the inverse of the diagonal block
        for (int i = col0 + kCB; i < k; ++i)
            if (col0 + lane < k) {
                R[(size_t)i * k + col0 + lane] = 0.0f;
                if (T) T[(size_t)i * k + col0 + lane] = 0.0f;
            }
        for (int J = 0; J < c; ++J) {
            bar_sync(kCcRowDone, 64 + kCcUpdaters);
            if (J + 1 < c) bar_arrive(kCcStepOver, 64 + kCcUpdaters + 64);
            const float *src = col + (size_t)J * kCBB + lane;
            if (col0 + lane < k)
#pragma unroll 8
                for (int i = 0; i < kCB; ++i) R[(size_t)(J * kCB + i) * k + col0 + lane] = src[i * kCB];
        }
        bar_sync(kCcPivots, 64);
        if (T) {
            float t[kCB];
            invert_diagonal(dia, dinv[lane], t, lane);
            const bool in = col0 + lane < k;
#pragma unroll
            for (int i = 0; i < kCB; ++i) {
                if (!in || col0 + i >= k) t[i] = 0.0f;
                sm[at.tjj + i * kCB + lane] = t[i];
            }
            fence_proxy_async_smem();
            __syncwarp();
            if (lane < c) {
                const unsigned there = smem_u32(sm + at.dia + c * kCcDia + kCB);
                cluster_copy(cluster_addr(there, lane), smem_u32(sm + at.tjj), kCBB * sizeof(float), cluster_addr(smem_u32(&bars->tjj[c]), lane));
            }
#pragma unroll
            for (int i = 0; i < kCB; ++i) {
                if (in && col0 + i < k) T[(size_t)(col0 + i) * k + col0 + lane] = t[i];
                sm[at.tij + lane * kCTs + i] = t[i];
            }
        }
    } else if (warp == 1) {
        // ---- block (J, c), behind the pivots of CTA J ----
        for (int J = 0; J < c; ++J) {
            if (J > 0) bar_sync(kCcStepOver, 64 + kCcUpdaters + 64);
            const int at_dia = at.dia + J * kCcDia + kCB;
            block_row<1>(at.col + J * kCBB + lane, at_dia, at_dia + kCBB + kCB, true, [&](int g) { cc_wait(&bars->dia[J][g], bars, status); });
            bar_arrive(kCcRowDone, 64 + kCcUpdaters);
            fence_proxy_async_smem();
            __syncwarp();
            if (lane < nb && (lane > c || (T && lane <= J))) {
                const unsigned slot = smem_u32(sm + at.rblk + cc_pair(J, c) * kCBB), bar = smem_u32(&bars->blk[cc_pair(J, c)]);
                cluster_copy(cluster_addr(slot, lane), smem_u32(col + (size_t)J * kCBB), kCBB * sizeof(float), cluster_addr(bar, lane));
            }
        }
    } else if (warp == 2 || warp == 3) {
        // ---- the diagonal block, eight rows behind ----
        const int t = (warp - 2) * 32 + lane;
        float *O = col + (size_t)c * kCBB;
        float2 acc[4][2];
        tile_load_wide(acc, O, t);
        for (int J = 0; J < c; ++J) {
            const float *RA = col + (size_t)J * kCBB;
#pragma unroll 1
            for (int j0 = 0; j0 < kCB; j0 += kCholStep) {
                bar_sync(6 + j0 / kCholStep, 32 + 64);
                block_mac_wide<kCB, kCB, kCholStep>(acc, RA + j0 * kCB, RA + j0 * kCB, t);
            }
            if (J + 1 < c) bar_arrive(kCcStepOver, 64 + kCcUpdaters + 64);
        }
        if (c > 0) {
            tile_store_wide(acc, O, t);
            bar_arrive(kCcDiagonal, 96);
        }
    } else {
        // ---- G_Ac -= R_JA^T R_Jc for the blocks in between ----
        const int pair = (wi - 3) >> 1, t = ((wi - 3) & 1) * 32 + lane;
        for (int J = 0; J < c; ++J) {
            bar_sync(kCcRowDone, 64 + kCcUpdaters);
            if (pair > 0 && J + 1 < c) bar_arrive(kCcStepOver, 64 + kCcUpdaters + 64);
            for (int A = J + 1 + pair; A < c; A += kCcPairs) {
                cc_wait(&bars->blk[cc_pair(J, A)], bars, status);
                float *O = col + (size_t)A * kCBB;
                float2 acc[4][2];
                tile_load_wide(acc, O, t);
                block_mac_wide<kCB, kCB, kCB>(acc, sm + at.rblk + cc_pair(J, A) * kCBB, col + (size_t)J * kCBB, t);
                tile_store_wide(acc, O, t);
                if (A == J + 1) bar_arrive(kCcStepOver, 64 + kCcUpdaters + 64);       // (pair 0)
            }
        }
    }
    if (T) {
        __syncthreads();
        // ---- row c of the inverse ----
        float *tij = sm + at.tij;
        for (int J = c; J < nb; ++J) {
            if (J > c) {
                // T_cJ^T = T_JJ^T (-S_J^T), four elements of a column per thread of eight warps
                cc_wait(&bars->tjj[J], bars, status);
                if (warp < 8) {
                    const float *B = col + (size_t)J * kCBB + lane;
                    const unsigned at_t = smem_u32(sm + at.dia + J * kCcDia + kCB + 4 * warp);
                    float o[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
                    for (int l = 0; l < kCB; ++l) {
                        const float4 t = lds4(at_t + l * kCB * 4);
                        const float b = B[l * kCB];
                        o[0] = fmaf(t.x, b, o[0]);
                        o[1] = fmaf(t.y, b, o[1]);
                        o[2] = fmaf(t.z, b, o[2]);
                        o[3] = fmaf(t.w, b, o[3]);
                    }
#pragma unroll
                    for (int q = 0; q < 4; ++q) tij[(4 * warp + q) * kCTs + lane] = o[q];
                }
                __syncthreads();
                for (int r = warp; r < kCB; r += kCholWarps)
                    if (J * kCB + lane < k) T[(size_t)(col0 + r) * k + J * kCB + lane] = tij[lane * kCTs + r];
            }
            for (int C = J + 1 + warp / 2; C < nb; C += kCholWarps / 2) {
                cc_wait(&bars->blk[cc_pair(J, C)], bars, status);
                const int t = (warp & 1) * 32 + lane;
                float2 acc[4][2] = {};
                float *S = col + (size_t)C * kCBB;
                if (J > c) tile_load_wide(acc, S, t);
                block_mac_wide<kCB, kCTs, kCB>(acc, sm + at.rblk + cc_pair(J, C) * kCBB, tij, t);
                tile_store_wide(acc, S, t);
            }
            __syncthreads();                               // the sums of the next column are whole, tij may be overwritten
        }
    }
    __syncthreads();                                       // every warp's waits are behind it (without T nothing else is between the roles and here)
    if (tid == 0 && bars->failed) {
        // a wait ran out: what may still be on its way into this CTA's shared memory has to land before it goes away
        bars->failed = 0;
        for (int J = 0; J < c; ++J) {
            for (int g = 0; g < kCB / kCholStep; ++g) cc_wait(&bars->dia[J][g], bars, status);
            for (int A = J + 1; A < c; ++A) cc_wait(&bars->blk[cc_pair(J, A)], bars, status);
        }
        for (int J = c; T && J < nb; ++J) {
            if (J > c) cc_wait(&bars->tjj[J], bars, status);
            for (int A = J + 1; A < nb; ++A) cc_wait(&bars->blk[cc_pair(J, A)], bars, status);
        }
    }
    cluster.sync();                                        // nobody leaves while its blocks are read, or announcements come
}

// Launch configuration: one cluster, behind the kernel before as launch_chained has it.
inline void cholesky_cluster_config(cudaLaunchConfig_t *cfg, cudaLaunchAttribute (&attr)[2], int k, cudaStream_t st) {
    *cfg = cudaLaunchConfig_t{};
    cfg->gridDim = chol_blocks(k);
    cfg->blockDim = kCholThreads;
    cfg->dynamicSmemBytes = cholesky_cluster_smem_bytes(k);
    cfg->stream = st;
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = chol_blocks(k);
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg->attrs = attr;
    cfg->numAttrs = 2;
}

}  // namespace
}  // namespace bsq

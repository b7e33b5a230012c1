// The prompt path's GEMM for blocks of more than 64 tokens: C[tokens][rows] = X . W^T on pairs of SMs.
//
// Up to 64 tokens a GEMM of the prompt path is bound by the weight stream and prefill_gemm_umma_kernel does one 128-row
// tile per CTA.  Beyond that the same weights serve several tiles of tokens and the tensor cores (hi + lo operands: 4
// FLOP per weight and token) and the path from L2 into shared memory bound it.  A pair of CTAs (one cluster, one
// tcgen05.mma.cta_group::2 of M 256 x N 256 x K 16 at a time) works on 256 weight rows x 128 tokens: each CTA stages 128
// of the weight rows, the even one the hi and the odd one the lo rows of the activations, so per 64 inputs an SM fetches
// 32 KiB for 512 clocks of MMA (a single CTA with N 256: 48 KiB).  The first 128 columns of an accumulator are W . hi,
// the others W . lo.  256 tokens a pair (hi and lo one after the other into one accumulator, 48 KiB per 1024 clocks) was
// not faster: 5.9 against 5.2 ms for 1023 tokens of the Llama-3.2-1B shape, 95 against 87 ms for 3000 of the Llama-3-8B
// shape.  Before (blocks of 64 tokens, the weights streamed once for each): 15.0 and 259 ms.
//
// The tensor cores add to the accumulator with truncation, so the error of a sum grows with the number of steps: after
// kPairChunk stages (1024 inputs) the MMAs go on in the other accumulator while the epilogue warps add the finished one to
// FP32 registers, rounding to nearest.  With whole rows of K in one accumulator the logits of the 3000-token prompt were
// 2.6e-5 off the 64-bit ones (the CTA kernel with its ranges of K: 1.7e-5).
//
// Two accumulators of 256 columns fill tensor memory: the epilogue of one chunk overlaps the MMAs of the next.  Roles per
// CTA as in prefill_gemm_umma_kernel (warp 0 copies, warp 1 MMA issue -- in the even CTA only --, warps 2..9 epilogue).
// Barriers: "full" lies in the even CTA and counts both CTAs' bytes; "empty" and "accumulator full" lie in each CTA and
// are arrived on by multicast commits; "accumulator empty" lies in the even CTA and is arrived on by both CTAs'
// epilogue warps.  Copies are plain tensor copies of this GPU's own memory without multicast.  Waits are bounded; every
// path reaches the common exit, where the pair meets before tensor memory is freed.
#pragma once
#include "prefill.cuh"

namespace lpp {

constexpr int kPairM = 256;                 // weight rows of a pair
constexpr int kPairSub = 128 * 128;         // 128 rows x 64 inputs: 16 KiB
constexpr int kPairTokens = 128;            // tokens of an item
constexpr int kPairStage = 2 * kPairSub;    // weights, activations
constexpr int kPairStages = 6;
constexpr int kPairSmemBytes = 1024 /*barriers*/ + 1024 /*alignment slack*/ + 192 * 1024;
constexpr int kPairCols = 512;              // tensor memory columns: two accumulators of 256
constexpr int kPairChunk = 16;              // stages that go into one accumulator

template <typename T>
__host__ __device__ constexpr uint32_t pair_idesc() {  // as umma_idesc, M = 256, N = 256
    return (1u << 4) | (std::is_same<T, __nv_bfloat16>::value ? (1u << 7) | (1u << 10) : 0u) | ((uint32_t)(256 >> 3) << 17) | ((uint32_t)(256 >> 4) << 24);
}

__device__ __forceinline__ uint32_t cluster_rank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ uint32_t cluster_addr(uint32_t smem_addr, uint32_t rank) {  // the same place in the CTA `rank` of the cluster
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(smem_addr), "r"(rank));
    return r;
}
__device__ __forceinline__ void pair_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ void pair_alloc(uint32_t* smem_dst, uint32_t cols) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(smem_dst)), "r"(cols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void pair_dealloc(uint32_t taddr, uint32_t cols) {
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(cols) : "memory");
}
__device__ __forceinline__ void pair_commit(uint64_t* bar) {  // arrives on this barrier of both CTAs
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(smem_u32(bar)),
                 "h"((uint16_t)3)
                 : "memory");
}
__device__ __forceinline__ void pair_mma(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(d_tmem), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
}
// Tensor copies into this CTA whose bytes count on a barrier of the even CTA.
__device__ __forceinline__ void pair_load_3d(uint32_t smem_dst, const CUtensorMap* map, int x, int y, int z, uint32_t bar_cluster_addr) {
    asm volatile("cp.async.bulk.tensor.3d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];" ::"r"(
                     smem_dst),
                 "l"(map), "r"(x), "r"(y), "r"(z), "r"(bar_cluster_addr)
                 : "memory");
}
__device__ __forceinline__ void pair_load_4d(uint32_t smem_dst, const CUtensorMap* map, int x, int y, int z, int w, uint32_t bar_cluster_addr) {
    asm volatile("cp.async.bulk.tensor.4d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5}], [%6];" ::"r"(
                     smem_dst),
                 "l"(map), "r"(x), "r"(y), "r"(z), "r"(w), "r"(bar_cluster_addr)
                 : "memory");
}
// 32 lanes x 16 consecutive 32-bit columns (see tc_ld32)
__device__ __forceinline__ void tc_ld16(uint32_t taddr, float (&v)[16]) {
    uint32_t r[16];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]),
          "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr)
        : "memory");
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(r[i]);
}
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t bar_cluster_addr) {
    asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(bar_cluster_addr) : "memory");
}

template <typename T, int EPI>
static __global__ void __launch_bounds__(kUmmaThreads, 1) prefill_gemm_pair_kernel(const __grid_constant__ CUtensorMap w_map,
                                                                                   const __grid_constant__ CUtensorMap x_map,
                                                                                   const PrefillGemmArgs a) {
    constexpr int kStages = kPairStages, kStage = kPairStage;
    extern __shared__ __align__(128) unsigned char smem[];
    uint64_t* full = reinterpret_cast<uint64_t*>(smem);  // [kStages], the even CTA's are used
    uint64_t* empty = full + kStages;                    // [kStages]
    uint64_t* acc_full = empty + kStages;                // [2]
    uint64_t* acc_empty = acc_full + 2;                  // [2], the even CTA's are used
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_empty + 2);
    int* s_fail = reinterpret_cast<int*>(tmem_slot + 1);  // set by a role whose wait ran out
    const uint32_t ring = (smem_u32(smem) + 1024u + 1023u) & ~1023u;
    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
    const int rank = (int)cluster_rank(), unit = blockIdx.x >> 1, n_units = gridDim.x >> 1;
    const int row_tiles = (a.n_rows + kPairM - 1) / kPairM, tok_tiles = (a.n_tokens + kPairTokens - 1) / kPairTokens;
    const int n_kc = a.K / 64, S = a.splits;
    const int n_items = row_tiles * tok_tiles * S;
    pdl_launch_dependents();
    if (tid == 0) {
        *s_fail = 0;
        for (int i = 0; i < kStages; ++i) {
            mbar_init(&full[i], 1);
            mbar_init(&empty[i], 1);
        }
        for (int i = 0; i < 2; ++i) {
            mbar_init(&acc_full[i], 1);
            mbar_init(&acc_empty[i], 2 * kUmmaEpiWarps);
        }
        mbar_fence_init();
    }
    if (warp == 1) pair_alloc(tmem_slot, kPairCols);
    tc_fence_before();
    __syncthreads();
    pair_sync();  // both CTAs' barriers are initialised before anything signals them
    tc_fence_after();
    const uint32_t tmem = *reinterpret_cast<volatile uint32_t*>(tmem_slot);

    if (warp == 0) {
        // ---------------- producer: this CTA's weight rows and its half of the activation rows
        if (lane == 0) {
            int slot = 0, pass = 0;
            bool ok = true, waited = false;
            int early = 0;  // stages whose weights are already in flight
            auto full_at = [&](int sl) { return cluster_addr(smem_u32(&full[sl]), 0); };
            auto load_w = [&](int sl, int kc, int wrow) { pair_load_3d(ring + (uint32_t)sl * kStage, &w_map, 0, wrow, kc, full_at(sl)); };
            auto load_x = [&](int sl, int kc, int tok0) {
                pair_load_4d(ring + (uint32_t)sl * kStage + kPairSub, &x_map, 0, tok0, rank, kc, full_at(sl));  // hi rows or lo rows
            };
            auto expect = [&](int sl) {
                if (rank == 0) mbar_arrive_expect_tx(&full[sl], 2 * kStage);
            };
            for (int item = unit; item < n_items && ok; item += n_units) {
                const int tile = item / S, split = item - tile * S;
                const int kc0 = (int)((long long)split * n_kc / S), kc1 = (int)((long long)(split + 1) * n_kc / S);
                const int row_tile = tile / tok_tiles, tok0 = (tile - row_tile * tok_tiles) * kPairTokens;
                const int wrow = a.row0 + row_tile * kPairM + rank * 128;
                if (!waited) {
                    early = min(kc1 - kc0, kStages);
                    for (int i = 0; i < early; ++i) {
                        expect(i);
                        load_w(i, kc0 + i, wrow);
                    }
                    pdl_wait();
                    waited = true;
                }
                for (int kc = kc0; kc < kc1; ++kc) {
                    if (early > 0) {
                        --early;  // first pass of the first item: only the activations are missing
                    } else {
                        if (pass > 0 && !mbar_wait_bounded(&empty[slot], (uint32_t)(pass - 1) & 1u, a.st)) {
                            *s_fail = 1;
                            ok = false;
                            break;
                        }
                        expect(slot);
                        load_w(slot, kc, wrow);
                    }
                    load_x(slot, kc, tok0);
                    if (++slot == kStages) {
                        slot = 0;
                        ++pass;
                    }
                }
            }
            if (!waited) pdl_wait();
        }
    } else if (warp == 1) {
        // ---------------- MMA issue for the pair
        if (rank == 0) {
            int slot = 0, it = 0;
            uint32_t par = 0;
            bool ok = true;
            for (int item = unit; item < n_items && ok; item += n_units) {
                const int split = item % S;
                const int kc0 = (int)((long long)split * n_kc / S), kc1 = (int)((long long)(split + 1) * n_kc / S);
                for (int k0 = kc0; k0 < kc1 && ok; k0 += kPairChunk, ++it) {
                    const int b = it & 1, use = it >> 1, k1 = min(k0 + kPairChunk, kc1);
                    if (use > 0 && !mbar_wait_bounded(&acc_empty[b], (uint32_t)(use - 1) & 1u, a.st)) {
                        *s_fail = 1;
                        ok = false;
                        break;
                    }
                    tc_fence_after();
                    const uint32_t d_tmem = tmem + (uint32_t)(b * 256);
                    for (int kc = k0; kc < k1; ++kc) {
                        if (!mbar_wait_bounded(&full[slot], par, a.st)) {
                            *s_fail = 1;
                            ok = false;
                            break;
                        }
                        tc_fence_after();
                        const uint32_t wt = ring + (uint32_t)slot * kStage, xt = wt + kPairSub;
                        if (elect_one()) {
#pragma unroll
                            for (int ks = 0; ks < 4; ++ks)  // 16 inputs = 32 bytes along the swizzled row per step
                                pair_mma(d_tmem, umma_desc(wt + ks * 32), umma_desc(xt + ks * 32), pair_idesc<T>(), (kc > k0 || ks > 0) ? 1u : 0u);
                            pair_commit(&empty[slot]);  // arrives in both CTAs once the MMAs issued so far have read this stage
                        }
                        __syncwarp();
                        if (++slot == kStages) {
                            slot = 0;
                            par ^= 1u;
                        }
                    }
                    if (ok && elect_one()) pair_commit(&acc_full[b]);
                    __syncwarp();
                }
            }
        }
    } else {
        // ---------------- epilogue: tensor-memory lanes 32 * (warp % 4) .. + 31 = rows of this CTA's half of the tile,
        // and one half of the tokens, 32 at a time
        const int quarter = warp & 3, half = (warp - 2) >> 2;
        constexpr int kCols = kPairTokens / 2;  // tokens of this thread
        int it = 0;
        bool ok = true;
        for (int item = unit; item < n_items && ok; item += n_units) {
            const int tile = item / S, split = item - tile * S;
            const int row_tile = tile / tok_tiles, tok0 = (tile - row_tile * tok_tiles) * kPairTokens + half * kCols;
            const int kc0 = (int)((long long)split * n_kc / S), kc1 = (int)((long long)(split + 1) * n_kc / S);
            float sum[kCols / 32][32];
            for (int k0 = kc0; k0 < kc1; k0 += kPairChunk, ++it) {
                const int b = it & 1, use = it >> 1;
                if (!__all_sync(0xffffffffu, mbar_wait_bounded(&acc_full[b], (uint32_t)use & 1u, a.st))) {
                    *s_fail = 1;
                    ok = false;
                    break;
                }
                tc_fence_after();
                const uint32_t taddr = tmem + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(b * 256 + half * kCols);
#pragma unroll
                for (int c = 0; c < kCols; c += 16) {  // 16 at a time: the sums leave few registers
                    float v[16];
                    tc_ld16(taddr + c, v);
                    float vlo[16];
                    tc_ld16(taddr + kPairTokens + c, vlo);
#pragma unroll
                    for (int i = 0; i < 16; ++i) v[i] += vlo[i];
#pragma unroll
                    for (int i = 0; i < 16; ++i) {
                        float& to = sum[c / 32][c % 32 + i];
                        to = k0 > kc0 ? to + v[i] : v[i];
                    }
                }
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive_cluster(cluster_addr(smem_u32(&acc_empty[b]), 0));  // it may be filled again
            }
            if (!ok) break;
            const int row = row_tile * kPairM + rank * 128 + quarter * 32 + lane;
#pragma unroll
            for (int c = 0; c < kCols / 32; ++c)
                if (tok0 + c * 32 < a.n_tokens) umma_epilogue<T, EPI>(a, split, 0, row, tok0 + c * 32, sum[c], lane);
        }
    }
    // ---------------- common exit
    __syncwarp();
    tc_fence_before();
    __syncthreads();
    // A wait that ran out has set the status word (mbar_wait_bounded) and this CTA's flag.  Copies may then still be in
    // flight towards its shared memory: give them a bounded time to land before the pair leaves.
    if (tid == 0 && *reinterpret_cast<volatile int*>(s_fail) != 0) {
        const long long t0 = clock64();
        while (clock64() - t0 < (1 << 17)) __nanosleep(1000);
    }
    __syncthreads();
    pair_sync();  // nothing of this pair signals or reads the other CTA any more
    tc_fence_after();
    if (warp == 1) pair_dealloc(tmem, kPairCols);
}

}  // namespace lpp

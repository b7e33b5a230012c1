// Causal attention of a prompt block over the K/V cache on the fifth-generation tensor cores, head sizes 64 and 128
// (src/model.cpp:178-199; FP16 operands, FP32 accumulation).
//
// The query heads that share a key/value head are one matrix: a row tile of 128 rows is 128 / gqa neighbouring tokens with all
// their heads.  Per tile of 128 keys one tcgen05.mma chain forms the scores S = Q . K^T (tensor memory, two buffers), sixteen
// warps turn them into probabilities (four threads a row, 32 keys each) which go to shared memory as FP16 in the swizzled layout
// of an MMA operand, and a second chain forms P . V with V as it lies in the cache (keys along K, so the operand is "MN-major").
// P . V of a tile starts from zero and is added to FP32 registers, rescaled by the running maximum, while the tensor cores
// work on the next tile: no correction pass over tensor memory, and no long chain of the accumulator's truncating additions.
// Exponentials are taken to base 2 with the scale folded into one multiply-add.
//
// Bound by the exponentials (16384 a tile: 1024 clocks of the special-function units against 1024 (HS 128) or 512 clocks of
// MMA) and the hand-overs around them.  Where the row tiles do not fill the GPU (short blocks behind a long cache) a cluster of
// up to eight CTAs shares the keys of a row tile and puts the results together through distributed shared memory.  Long row
// tiles come first in the grid, so that the last wave is made of short ones.
// 1000 tokens of the Llama-3-8B shape behind 0 to 2000 others: 64 us a launch, 1023 tokens of the Llama-3.2-1B shape 25 us, 47
// tokens of the TinyLlama shape behind 1100 11 us.  Before (a CTA of gqa warps per 16 tokens, mma.sync): 149, 39 and 36 us.
//
// Warp 0 copies keys and values (tensor memory accelerator, this GPU's own memory, no multicast), warp 1 issues the MMAs,
// warps 2..17 are the softmax (eight warps left the special-function units idle while they waited: 70 against 64 us below).  Rows of the last key tile beyond the last visible position hold whatever the cache holds
// there: their scores are masked and the value rows are zeroed in shared memory, so that nothing of them gets through.
// Waits are bounded; every path reaches the common exit.
#pragma once
#include "attention.cuh"
#include "latent_attention.cuh"
#include "prefill_pair.cuh"

namespace lpp {

constexpr int kFaRows = 128, kFaKeys = 128;
constexpr int kFaSub = 128 * 128;  // bytes of 128 rows x 64 columns
constexpr int kFaMaxCluster = 8;
constexpr int kFaSoftWarps = 16, kFaParts = kFaSoftWarps / 4;  // threads that share a row
constexpr int kFaThreads = (2 + kFaSoftWarps) * 32;
template <int HS>
constexpr int fa_smem() {
    return 1024 /*barriers*/ + 1024 /*alignment slack*/ + 5 * (HS / 64) * kFaSub /*Q, 2 x K, 2 x V*/ + 2 * kFaSub /*P*/;
}

struct PrefillAttnArgs {
    const float* q;     // [tokens][q_rows]
    __half* out;        // hi and lo plane [cap][q_rows]
    StepState* st;
    int n_tokens, start_pos, gqa, kv_heads, q_rows, cap;
    int row0, seq_len;  // cache row of this layer's first position, positions of a head
    int cluster;        // CTAs that share the keys of a row tile
};

__device__ __forceinline__ float ex2(float x) {
    float r;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}
// Operand tile whose rows run along K (128-byte rows of 64 MN elements, swizzled): 1024 bytes between groups of eight K rows,
// kFaSub between blocks of 64 MN elements.
__device__ __forceinline__ uint64_t fa_desc_mn(uint32_t smem_addr) {
    return (uint64_t)((smem_addr & 0x3ffffu) >> 4) | ((uint64_t)(kFaSub >> 4) << 16) | ((uint64_t)(1024 >> 4) << 32) | (1ull << 46) | (2ull << 61);
}
__host__ __device__ constexpr uint32_t fa_idesc(int n, bool b_mn_major) {  // as umma_idesc, FP16, M = 128
    return (1u << 4) | (b_mn_major ? 1u << 16 : 0u) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);
}
__device__ __forceinline__ void fence_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

template <int HS>
static __global__ void __launch_bounds__(kFaThreads, 1) prefill_attention_umma_kernel(const __grid_constant__ CUtensorMap k_map,
                                                                                                   const __grid_constant__ CUtensorMap v_map,
                                                                                                   const PrefillAttnArgs a) {
    constexpr int kPieces = HS / 64, kTile = kPieces * kFaSub, kCols = HS / kFaParts;  // kCols: output columns of a softmax thread
    extern __shared__ __align__(128) unsigned char smem[];
    __shared__ float s_max[2][kFaParts][kFaRows], s_l[kFaParts][kFaRows], s_m[kFaRows], s_w[kFaRows][kFaMaxCluster];
    uint64_t* k_full = reinterpret_cast<uint64_t*>(smem);  // pairs, by tile parity
    uint64_t *k_empty = k_full + 2, *v_full = k_full + 4, *v_empty = k_full + 6, *s_full = k_full + 8, *s_free = k_full + 10, *pv_full = k_full + 12,
             *pv_free = k_full + 14, *q_ready = k_full + 16, *p_ready = k_full + 17,
             *max_ready = k_full + 18;  // [4]: by quarter of the rows
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(k_full + 22);
    int* s_fail = reinterpret_cast<int*>(tmem_slot + 1);
    const uint32_t base = (smem_u32(smem) + 1024u + 1023u) & ~1023u;
    const uint32_t sq = base, sk = sq + kTile, sv = sk + 2 * kTile, sp = sv + 2 * kTile;
    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
    const int rank = a.cluster > 1 ? (int)cluster_rank() : 0, work = blockIdx.x / a.cluster;
    const int kvh = work % a.kv_heads, tile_tokens = kFaRows / a.gqa;
    const int row_tile = (a.n_tokens + tile_tokens - 1) / tile_tokens - 1 - work / a.kv_heads;
    const int t0 = row_tile * tile_tokens, tokens = min(tile_tokens, a.n_tokens - t0);
    const int t_max = a.start_pos + t0 + tokens;  // positions visible to the last token of the tile
    const int n_tiles = (t_max + kFaKeys - 1) / kFaKeys;
    const int kb = rank * n_tiles / a.cluster, n_here = (rank + 1) * n_tiles / a.cluster - kb;
    if (tid == 0) {
        *s_fail = 0;
        for (int i = 0; i < 2; ++i) {
            mbar_init(&k_full[i], 1);
            mbar_init(&k_empty[i], 1);
            mbar_init(&v_full[i], 1);
            mbar_init(&v_empty[i], 1);
            mbar_init(&s_full[i], 1);
            mbar_init(&s_free[i], kFaSoftWarps);
            mbar_init(&pv_full[i], 1);
            mbar_init(&pv_free[i], kFaSoftWarps);
        }
        mbar_init(q_ready, kFaSoftWarps);
        mbar_init(p_ready, kFaSoftWarps);
        for (int i = 0; i < 4; ++i) mbar_init(&max_ready[i], kFaParts);
        mbar_fence_init();
    }
    if (warp == 1) {
        tc_alloc(tmem_slot, 512);  // S: columns 0, 128; P . V: columns 256, 384
        tc_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *reinterpret_cast<volatile uint32_t*>(tmem_slot);
    pdl_launch_dependents();  // tensor memory is ours: what comes next cannot take it first

    if (warp == 0) {
        // ---------------- producer
        if (lane == 0) {
            const int row = a.row0 + kvh * a.seq_len + kb * kFaKeys;
            bool waited = false;
            for (int it = 0; it < n_here; ++it) {
                const int b = it & 1;
                // rows before this block do not depend on the kernels before: a block starts behind a plain copy
                if (!waited && (kb + it + 1) * kFaKeys > a.start_pos) {
                    pdl_wait();
                    waited = true;
                }
                const uint32_t par = (uint32_t)((it >> 1) - 1) & 1u;
                if (it >= 2 && !mbar_wait_bounded(&k_empty[b], par, a.st)) {
                    *s_fail = 1;
                    break;
                }
                mbar_arrive_expect_tx(&k_full[b], kTile);
                tma_load_3d(sk + b * kTile, &k_map, 0, row + it * kFaKeys, 0, smem_u32(&k_full[b]));
                if (it >= 2 && !mbar_wait_bounded(&v_empty[b], par, a.st)) {
                    *s_fail = 1;
                    break;
                }
                mbar_arrive_expect_tx(&v_full[b], kTile);
                tma_load_3d(sv + b * kTile, &v_map, 0, row + it * kFaKeys, 0, smem_u32(&v_full[b]));
            }
        }
    } else if (warp == 1) {
        // ---------------- MMA issue
        auto scores = [&](int it) -> bool {
            const int b = it & 1;
            if (!mbar_wait_bounded(&k_full[b], (uint32_t)(it >> 1) & 1u, a.st)) return false;
            if (it >= 2 && !mbar_wait_bounded(&s_free[b], (uint32_t)((it >> 1) - 1) & 1u, a.st)) return false;
            tc_fence_after();
            if (elect_one()) {
#pragma unroll
                for (int ks = 0; ks < HS / 16; ++ks) {
                    const uint32_t off = (uint32_t)((ks >> 2) * kFaSub + (ks & 3) * 32);
                    tc_mma_f16(tmem + b * 128, umma_desc(sq + off), umma_desc(sk + b * kTile + off), fa_idesc(kFaKeys, false), ks > 0 ? 1u : 0u);
                }
                tc_commit(&k_empty[b]);
                tc_commit(&s_full[b]);
            }
            __syncwarp();
            return true;
        };
        bool ok = n_here == 0 || (mbar_wait_bounded(q_ready, 0, a.st) && scores(0));
        for (int it = 0; it < n_here && ok; ++it) {
            const int b = it & 1;
            ok = (it + 1 >= n_here || scores(it + 1)) && mbar_wait_bounded(&v_full[b], (uint32_t)(it >> 1) & 1u, a.st);
            if (!ok) break;
            const int valid = t_max - (kb + it) * kFaKeys;
            if (valid < kFaKeys) {  // the last tile: values beyond the last visible position
                for (int i = lane; i < (kFaKeys - valid) * 8 * kPieces; i += 32) {
                    const int piece = i & 7, r = valid + (i >> 3) % (kFaKeys - valid), sub = (i >> 3) / (kFaKeys - valid);
                    asm volatile("st.shared.v4.b32 [%0], {%1, %1, %1, %1};" ::"r"(sv + b * kTile + sub * kFaSub + r * 128 + piece * 16), "r"(0) : "memory");
                }
                fence_async_smem();
                __syncwarp();
            }
            ok = mbar_wait_bounded(p_ready, (uint32_t)it & 1u, a.st) && (it < 2 || mbar_wait_bounded(&pv_free[b], (uint32_t)((it >> 1) - 1) & 1u, a.st));
            if (!ok) break;
            tc_fence_after();
            if (elect_one()) {
#pragma unroll
                for (int ks = 0; ks < kFaKeys / 16; ++ks)
                    tc_mma_f16(tmem + 256 + b * 128, umma_desc(sp + (uint32_t)((ks >> 2) * kFaSub + (ks & 3) * 32)), fa_desc_mn(sv + b * kTile + ks * 2048),
                               fa_idesc(HS, true), ks > 0 ? 1u : 0u);
                tc_commit(&v_empty[b]);
                tc_commit(&pv_full[b]);
            }
            __syncwarp();
        }
        if (!ok) *s_fail = 1;
    } else {
        // ---------------- softmax: row of the tile, one part of the keys of a tile and of the output columns
        const int quarter = warp & 3, part = (warp - 2) >> 2, row = quarter * 32 + lane;
        pdl_wait();
        {  // queries as FP16 operand rows
            constexpr int kChunks = HS / 8;
            for (int i = tid - 64; i < kFaRows * kChunks; i += kFaSoftWarps * 32) {
                const int r = i / kChunks, c = i % kChunks, t = r / a.gqa;
                float4 x = make_float4(0.f, 0.f, 0.f, 0.f), y = x;
                if (t < tokens) {
                    const float4* src = reinterpret_cast<const float4*>(a.q + (size_t)(t0 + t) * a.q_rows + (size_t)(kvh * a.gqa + (r - t * a.gqa)) * HS) + 2 * c;
                    x = src[0];
                    y = src[1];
                }
                asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(sq + (uint32_t)((c >> 3) * kFaSub + r * 128 + (((c & 7) ^ (r & 7)) << 4))),
                             "r"(pack_half2(x.x, x.y)), "r"(pack_half2(x.z, x.w)), "r"(pack_half2(y.x, y.y)), "r"(pack_half2(y.z, y.w))
                             : "memory");
            }
            fence_async_smem();
            __syncwarp();
            if (lane == 0) mbar_arrive(q_ready);
        }
        const float rate = __fdiv_rn(1.0f, __fsqrt_rn((float)HS)) * 1.4426950408889634f;  // exp(s / sqrt(HS)) = 2^(s rate)
        const int token = row / a.gqa, lim = a.start_pos + t0 + min(token, tokens - 1);   // (rows beyond the tile: zero queries, not stored)
        const uint32_t lanes = (uint32_t)(quarter * 32) << 16;
        const uint32_t p_row = sp + (uint32_t)((part >> 1) * kFaSub + row * 128), p_chunk = (part & 1) * 4;
        float m = -INFINITY, l = 0.f, f_before = 0.f;
        float o[kCols];
#pragma unroll
        for (int i = 0; i < kCols; ++i) o[i] = 0.f;
        auto add_values = [&](int it) -> bool {  // o = o * (rescaling) + P . V of tile `it`
            const int b = it & 1;
            if (!__all_sync(0xffffffffu, mbar_wait_bounded(&pv_full[b], (uint32_t)(it >> 1) & 1u, a.st))) return false;
            tc_fence_after();
            const uint32_t at = tmem + lanes + 256 + b * 128 + part * kCols;
            float v[kCols];
            if constexpr (kCols == 32)
                tc_ld32(at, v);
            else
                tc_ld16(at, v);
#pragma unroll
            for (int i = 0; i < kCols; ++i) o[i] = fmaf(o[i], f_before, v[i]);
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&pv_free[b]);
            return true;
        };
        bool ok = true;
        for (int it = 0; it < n_here && ok; ++it) {
            const int b = it & 1, p0 = (kb + it) * kFaKeys + part * 32;
            if (!__all_sync(0xffffffffu, mbar_wait_bounded(&s_full[b], (uint32_t)(it >> 1) & 1u, a.st))) {
                ok = false;
                break;
            }
            tc_fence_after();
            float s[32];
            tc_ld32(tmem + lanes + b * 128 + part * 32, s);
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&s_free[b]);
            if (p0 + 31 > a.start_pos + t0) {  // positions that the tile's first token does not see
#pragma unroll
                for (int i = 0; i < 32; ++i) s[i] = p0 + i <= lim ? s[i] : -INFINITY;
            }
            float mx[4] = {s[0], s[1], s[2], s[3]};
#pragma unroll
            for (int i = 4; i < 32; ++i) mx[i & 3] = fmaxf(mx[i & 3], s[i]);
            s_max[b][part][row] = fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3]));
            __syncwarp();
            if (lane == 0) mbar_arrive(&max_ready[quarter]);  // the warps of these rows
            if (!__all_sync(0xffffffffu, mbar_wait_bounded(&max_ready[quarter], (uint32_t)it & 1u, a.st))) {
                ok = false;
                break;
            }
            float top = s_max[b][0][row];
#pragma unroll
            for (int i = 1; i < kFaParts; ++i) top = fmaxf(top, s_max[b][i][row]);
            const float m_new = fmaxf(m, top * rate);
            const float u = m_new == -INFINITY ? 0.f : m_new;  // nothing visible yet
            const float f = ex2(m - u);
            m = m_new;
            uint32_t p[16];
            float sum0 = 0.f, sum1 = 0.f;
#pragma unroll
            for (int i = 0; i < 16; ++i) {
                const float e0 = ex2(fmaf(s[2 * i], rate, -u)), e1 = ex2(fmaf(s[2 * i + 1], rate, -u));
                sum0 += e0;
                sum1 += e1;
                p[i] = pack_half2(e0, e1);
            }
            l = fmaf(l, f, sum0 + sum1);
            // the probabilities of the tile before have been read when its product is there
            if (it > 0 && !__all_sync(0xffffffffu, mbar_wait_bounded(&pv_full[b ^ 1], (uint32_t)((it - 1) >> 1) & 1u, a.st))) {
                ok = false;
                break;
            }
#pragma unroll
            for (int c = 0; c < 4; ++c)
                asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(p_row + (uint32_t)(((p_chunk + c) ^ (row & 7)) << 4)), "r"(p[4 * c]), "r"(p[4 * c + 1]),
                             "r"(p[4 * c + 2]), "r"(p[4 * c + 3])
                             : "memory");
            fence_async_smem();
            __syncwarp();
            if (lane == 0) mbar_arrive(p_ready);
            if (it > 0) ok = add_values(it - 1);
            f_before = f;
        }
        if (ok && n_here > 0) ok = add_values(n_here - 1);
        if (!ok) *s_fail = 1;
        s_l[part][row] = l;
        if (part == 0) s_m[row] = m;
        if (a.cluster == 1) {
            asm volatile("bar.sync %0, %1;" ::"r"(1 + quarter), "n"(32 * kFaParts) : "memory");  // (every warp gets here)
            float total = s_l[0][row];
#pragma unroll
            for (int i = 1; i < kFaParts; ++i) total += s_l[i][row];
            if (token < tokens) {
                __half* dst = a.out + (size_t)(t0 + token) * a.q_rows + (size_t)(kvh * a.gqa + (row - token * a.gqa)) * HS + part * kCols;
#pragma unroll
                for (int c = 0; c < kCols; c += 8) {
                    __align__(16) __half hi[8], lo[8];
#pragma unroll
                    for (int i = 0; i < 8; ++i) split_half(__fdiv_rn(o[c + i], total), hi[i], lo[i]);
                    *reinterpret_cast<uint4*>(dst + c) = *reinterpret_cast<const uint4*>(hi);
                    *reinterpret_cast<uint4*>(dst + (size_t)a.cap * a.q_rows + c) = *reinterpret_cast<const uint4*>(lo);
                }
            }
        } else {  // unnormalised, over the keys and values (every copy has landed and been read)
            float* os = reinterpret_cast<float*>(smem + (sk - smem_u32(smem))) + row * (HS + 4) + part * kCols;
#pragma unroll
            for (int c = 0; c < kCols; c += 4) *reinterpret_cast<float4*>(os + c) = make_float4(o[c], o[c + 1], o[c + 2], o[c + 3]);
        }
    }
    if (a.cluster > 1) {
        __syncwarp();
        pair_sync();  // of the whole cluster: every CTA's results are there
        // this CTA's share of the rows.  Weights of the CTAs first, eight lanes per row: 2^(m_c - max m) / sum
        const int share = kFaRows / a.cluster, r0 = rank * share, rows_here = min(share, tokens * a.gqa - r0);
        for (int i = tid; i < share * kFaMaxCluster; i += kFaThreads) {  // (whole warps: share is a multiple of 16)
            const int r = r0 + i / kFaMaxCluster, c = i % kFaMaxCluster;
            float mc = -INFINITY, lc = 0.f;
            if (c < a.cluster) {
                float lp[kFaParts];
                mc = cluster_load(cluster_map(smem_u32(&s_m[r]), c));
#pragma unroll
                for (int k = 0; k < kFaParts; ++k) lp[k] = cluster_load(cluster_map(smem_u32(&s_l[k][r]), c));
#pragma unroll
                for (int k = 0; k < kFaParts; ++k) lc += lp[k];
            }
            float top = mc;
#pragma unroll
            for (int d = kFaMaxCluster / 2; d > 0; d >>= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, d));
            const float e = mc == -INFINITY ? 0.f : ex2(mc - top);
            float sum = e * lc;
#pragma unroll
            for (int d = kFaMaxCluster / 2; d > 0; d >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, d);
            s_w[r][c] = __fdiv_rn(e, sum);
        }
        __syncthreads();
        for (int i = tid; i < rows_here * (HS / 4); i += kFaThreads) {
            const int r = r0 + i / (HS / 4), col = (i % (HS / 4)) * 4, t = r / a.gqa;
            const uint32_t at = sk + (uint32_t)(r * (HS + 4) + col) * 4;
            float y[4] = {};
            float4 x[kFaMaxCluster];
#pragma unroll
            for (int c = 0; c < kFaMaxCluster; ++c)
                if (c < a.cluster) x[c] = cluster_load4(cluster_map(at, c));
#pragma unroll
            for (int c = 0; c < kFaMaxCluster; ++c) {
                const float w = c < a.cluster ? s_w[r][c] : 0.f;
                if (w != 0.f) {
                    y[0] = fmaf(w, x[c].x, y[0]);
                    y[1] = fmaf(w, x[c].y, y[1]);
                    y[2] = fmaf(w, x[c].z, y[2]);
                    y[3] = fmaf(w, x[c].w, y[3]);
                }
            }
            __half* dst = a.out + (size_t)(t0 + t) * a.q_rows + (size_t)(kvh * a.gqa + (r - t * a.gqa)) * HS + col;
            __align__(8) __half hi[4], lo[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) split_half(y[k], hi[k], lo[k]);
            *reinterpret_cast<uint2*>(dst) = *reinterpret_cast<const uint2*>(hi);
            *reinterpret_cast<uint2*>(dst + (size_t)a.cap * a.q_rows) = *reinterpret_cast<const uint2*>(lo);
        }
        __syncwarp();
        pair_sync();  // every CTA's shared memory stays until all have read it
    }
    // ---------------- common exit
    __syncwarp();
    tc_fence_before();
    __syncthreads();
    // after a wait that ran out, copies may still be in flight: give them a bounded time to land
    if (tid == 0 && *reinterpret_cast<volatile int*>(s_fail) != 0) {
        const long long c0 = clock64();
        while (clock64() - c0 < (1 << 17)) __nanosleep(1000);
    }
    __syncthreads();
    if (warp == 1) tc_dealloc(tmem, 512);
}

}  // namespace lpp

// Attention over shared rows (latent_attention.cuh) of a prompt block on the fifth-generation tensor cores.
//
// A row tile is 128 query rows: neighbouring tokens with all heads of a group.  A CTA holds them as one operand (up to 640
// columns, 160 KiB), and keys and values pass through a ring of 64 rows x 64 columns (8 KiB) that the tensor memory
// accelerator fills: first the pieces whose scores S = Q . K^T add up, then, once the probabilities are there, the pieces of
// the value part again (the same cache rows; a tile of keys does not fit beside the queries, and re-reading a half of it costs
// less than the smaller row tile would).  A CTA takes up to 256 value columns, so wider rows are shared by two CTAs that both
// form the scores.  Sixteen warps are the softmax, four threads a row.  P . V of a tile starts from zero in tensor memory and is
// added to FP32 registers, rescaled by the running maximum, while the scores of the next tile are formed: the tensor cores add with
// truncation, and results of a whole window in one accumulator came out too small (3000 alike rows: by 1.9e-5, now 1.5e-7).
//
// Bound by the MMAs, 52 of 64 keys a tile at the widest (about 150 clocks each where 32 are arithmetic), and the hand-overs between
// them and the softmax.  1023 tokens of the rutenex-1b shape (16 heads, rows of 512 + 64, window 1024): 71 us a launch (64 with results
// that stay in tensor memory, mma.sync 170), rutenex-300m (rows of 256 + 32, window 512) 34 us (29).  mma.sync tiles of 32 rows
// (latent_attn_mma_kernel) fetch every key four times as often; they remain for blocks whose row tiles leave most of the GPU idle,
// because there a cluster shares the keys (prefill_row_attention in engine.cu draws the line).
// Rows outside the tile's span of keys are masked, and as values zeroed in shared memory.  Waits are bounded; every path
// reaches the common exit.
#pragma once
#include "latent_attention.cuh"
#include "prefill_attention.cuh"

namespace lpp {

constexpr int kRaRows = 128, kRaKeys = 64;
constexpr int kRaPiece = kRaKeys * 128;       // a ring slot: 64 keys x 64 columns
constexpr int kRaQueryPiece = kRaRows * 128;  // 128 query rows x 64 columns
constexpr int kRaMaxSlots = 16, kRaMinSlots = 5;
constexpr int kRaMaxPieces = 4;               // value columns of a CTA / 64
constexpr int kRaStatic = 7 * 1024;           // static shared memory and what the driver keeps, at most
__host__ __device__ constexpr int ra_pieces(int cols) { return (cols + 63) / 64; }
constexpr int ra_fixed(int row_width) { return 1024 /*barriers*/ + 1024 /*alignment slack*/ + ra_pieces(row_width) * kRaQueryPiece + kRaRows * 128 /*P*/; }

struct RowAttnArgs {
    LatentAttnArgs a;
    int slots;    // of the ring
    int halves;   // CTAs that share the value columns of a row tile
    int pieces;   // 64-column pieces of values of a CTA
};

__device__ __forceinline__ void tma_load_2d(uint32_t smem_dst, const CUtensorMap* map, int x, int y, uint32_t bar_addr) {
    asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(smem_dst), "l"(map),
                 "r"(x), "r"(y), "r"(bar_addr)
                 : "memory");
}
// grid: groups x halves x row tiles, the last tokens first.  q_map: queries as (columns, heads, tokens), boxes of 64 columns x
// a group's heads x the tile's tokens; c_map: the layer's cache as (columns, rows), boxes of 64 x 64.
template <bool SKV>
static __global__ void __launch_bounds__(kFaThreads, 1) row_attention_umma_kernel(const __grid_constant__ CUtensorMap q_map,
                                                                                  const __grid_constant__ CUtensorMap c_map, const RowAttnArgs ra) {
    const LatentAttnArgs& a = ra.a;
    extern __shared__ __align__(128) unsigned char smem[];
    __shared__ float s_max[2][kFaParts][kRaRows], s_l[kFaParts][kRaRows];
    uint64_t* full = reinterpret_cast<uint64_t*>(smem);
    uint64_t *empty = full + kRaMaxSlots, *s_full = empty + kRaMaxSlots, *s_free = s_full + 2, *q_full = s_free + 2, *p_ready = q_full + 1,
             *pv_done = p_ready + 1, *max_ready = pv_done + 1;  // [4]: by quarter of the rows
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(max_ready + 4);
    int* s_fail = reinterpret_cast<int*>(tmem_slot + 1);
    const int row_pieces = ra_pieces(a.row_width), S = ra.slots, P = ra.pieces;
    const uint32_t base_addr = (smem_u32(smem) + 1024u + 1023u) & ~1023u;
    const uint32_t sq = base_addr, sp = sq + row_pieces * kRaQueryPiece, ring = sp + kRaRows * 128;
    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
    const int groups = a.all_heads / a.heads, group = blockIdx.x % groups, half = blockIdx.x / groups % ra.halves;
    const int tile_tokens = kRaRows / a.heads;
    const int t0 = ((a.n_tokens + tile_tokens - 1) / tile_tokens - 1 - (int)blockIdx.x / (groups * ra.halves)) * tile_tokens;
    const int tokens = min(tile_tokens, a.n_tokens - t0), base = a.start_pos;
    const int k_begin = a.window > 0 ? max(0, base + t0 - a.window + 1) : 0, k_end = base + t0 + tokens;
    const int n_tiles = base >= 0 && k_end <= a.seq_len ? (k_end - k_begin + kRaKeys - 1) / kRaKeys : 0;
    if (tid == 0) {
        *s_fail = 0;
        for (int i = 0; i < S; ++i) {
            mbar_init(&full[i], 1);
            mbar_init(&empty[i], 1);
        }
        for (int i = 0; i < 2; ++i) {
            mbar_init(&s_full[i], 1);
            mbar_init(&s_free[i], kFaSoftWarps);
        }
        mbar_init(q_full, 1);
        mbar_init(p_ready, kFaSoftWarps);
        mbar_init(pv_done, 1);
        for (int i = 0; i < 4; ++i) mbar_init(&max_ready[i], kFaParts);
        mbar_fence_init();
    }
    if (warp == 1) {
        tc_alloc(tmem_slot, 512);  // results: columns 0..255; S: 256, 320
        tc_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *reinterpret_cast<volatile uint32_t*>(tmem_slot);
    pdl_launch_dependents();  // tensor memory is ours: what comes next cannot take it first
    StepState* st = const_cast<StepState*>(a.st);

    if (warp == 0) {
        // ---------------- producer
        if (lane == 0 && n_tiles > 0) {
            pdl_wait();
            const int row = group * a.seq_len + k_begin;
            int slot = 0, pass = 0;
            auto load = [&](int tile, int piece) -> bool {
                if (pass > 0 && !mbar_wait_bounded(&empty[slot], (uint32_t)(pass - 1) & 1u, st)) return false;
                mbar_arrive_expect_tx(&full[slot], kRaPiece);
                tma_load_2d(ring + slot * kRaPiece, &c_map, piece * 64, row + tile * kRaKeys, smem_u32(&full[slot]));
                if (++slot == S) {
                    slot = 0;
                    ++pass;
                }
                return true;
            };
            // the queries, as many rows as there are whole tokens in a tile
            mbar_arrive_expect_tx(q_full, (uint32_t)(row_pieces * a.heads * tile_tokens * 128));
            for (int p = 0; p < row_pieces; ++p) tma_load_3d(sq + p * kRaQueryPiece, &q_map, p * 64, group * a.heads, t0, smem_u32(q_full));
            bool ok = true;
            for (int it = -1; it < n_tiles && ok; ++it) {  // in the order that the MMAs take them
                for (int p = 0; p < row_pieces && ok && it + 1 < n_tiles; ++p) ok = load(it + 1, p);
                for (int p = 0; p < P && ok && it >= 0; ++p) ok = load(it, half * P + p);
            }
            if (!ok) *s_fail = 1;
        }
    } else if (warp == 1) {
        // ---------------- MMA issue
        int slot = 0;
        uint32_t par = 0;
        auto taken = [&]() {
            if (elect_one()) tc_commit(&empty[slot]);
            __syncwarp();
            if (++slot == S) {
                slot = 0;
                par ^= 1u;
            }
        };
        auto scores = [&](int it) -> bool {
            const int b = it & 1;
            if (it >= 2 && !mbar_wait_bounded(&s_free[b], (uint32_t)((it >> 1) - 1) & 1u, st)) return false;
            for (int p = 0; p < row_pieces; ++p) {
                if (!mbar_wait_bounded(&full[slot], par, st)) return false;
                tc_fence_after();
                if (elect_one()) {
#pragma unroll
                    for (int ks = 0; ks < 4; ++ks)
                        tc_mma_f16(tmem + 256 + b * kRaKeys, umma_desc(sq + p * kRaQueryPiece + ks * 32), umma_desc(ring + slot * kRaPiece + ks * 32),
                                   fa_idesc(kRaKeys, false), p > 0 || ks > 0 ? 1u : 0u);
                }
                taken();
            }
            if (elect_one()) tc_commit(&s_full[b]);
            __syncwarp();
            return true;
        };
        bool ok = n_tiles == 0 || (mbar_wait_bounded(q_full, 0, st) && scores(0));
        for (int it = 0; it < n_tiles && ok; ++it) {
            ok = (it + 1 >= n_tiles || scores(it + 1)) && mbar_wait_bounded(p_ready, (uint32_t)it & 1u, st);
            const int valid = k_end - k_begin - it * kRaKeys;
            for (int p = 0; p < P && ok; ++p) {
                ok = mbar_wait_bounded(&full[slot], par, st);
                if (!ok) break;
                if (valid < kRaKeys) {  // the last tile: values beyond the tile's last position
                    for (int i = lane; i < (kRaKeys - valid) * 8; i += 32)
                        asm volatile("st.shared.v4.b32 [%0], {%1, %1, %1, %1};" ::"r"(ring + slot * kRaPiece + valid * 128 + i * 16), "r"(0) : "memory");
                    fence_async_smem();
                    __syncwarp();
                }
                tc_fence_after();
                if (elect_one()) {
#pragma unroll
                    for (int ks = 0; ks < kRaKeys / 16; ++ks)
                        tc_mma_f16(tmem + p * 64, umma_desc(sp + ks * 32), fa_desc_mn(ring + slot * kRaPiece + ks * 2048), fa_idesc(64, true),
                                   ks > 0 ? 1u : 0u);
                }
                taken();
            }
            if (ok && elect_one()) tc_commit(pv_done);
            __syncwarp();
        }
        if (!ok) *s_fail = 1;
    } else {
        // ---------------- softmax: row of the tile, sixteen of the keys of a tile and a quarter of the results
        const int quarter = warp & 3, part = (warp - 2) >> 2, row = quarter * 32 + lane;
        const int token = row / a.heads, last = base + t0 + min(token, tokens - 1), first = a.window > 0 ? last - a.window + 1 : 0;
        const int all_from = a.window > 0 ? base + t0 + tokens - a.window : 0, all_to = base + t0;  // what every row of the tile sees
        const uint32_t lanes = (uint32_t)(quarter * 32) << 16, results = tmem + lanes + (uint32_t)(part * P * 16);
        const uint32_t p_row = sp + (uint32_t)(row * 128);
        pdl_wait();  // (gates, and what still reads the finished rows of the layer before)
        constexpr float kLog2e = 1.4426950408889634f;
        const float rate = a.scale * kLog2e;
        float m = -INFINITY, l = 0.f, f_before = 0.f;
        float o[kRaMaxPieces][16];
#pragma unroll
        for (int c = 0; c < kRaMaxPieces; ++c)
#pragma unroll
            for (int i = 0; i < 16; ++i) o[c][i] = 0.f;
        auto products_done = [&](int it) -> bool { return __all_sync(0xffffffffu, mbar_wait_bounded(pv_done, (uint32_t)it & 1u, st)); };
        auto add_values = [&]() {  // o = o * (rescaling) + P . V of the tile whose products are done
            tc_fence_after();
#pragma unroll
            for (int c = 0; c < kRaMaxPieces; ++c) {
                if (c >= P) break;
                float v[16];
                tc_ld16(results + c * 16, v);
#pragma unroll
                for (int i = 0; i < 16; ++i) o[c][i] = fmaf(o[c][i], f_before, v[i]);
            }
            tc_fence_before();
        };
        bool ok = true;
        for (int it = 0; it < n_tiles && ok; ++it) {
            const int b = it & 1, p0 = k_begin + it * kRaKeys + part * 16;
            ok = __all_sync(0xffffffffu, mbar_wait_bounded(&s_full[b], (uint32_t)(it >> 1) & 1u, st));
            if (!ok) break;
            tc_fence_after();
            float s[16];
            tc_ld16(tmem + lanes + 256 + b * kRaKeys + part * 16, s);
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&s_free[b]);
            if (SKV && a.softcap > 0.f) {
#pragma unroll
                for (int i = 0; i < 16; ++i) s[i] = capped_score(a, s[i] * a.scale) * kLog2e;
            } else {
#pragma unroll
                for (int i = 0; i < 16; ++i) s[i] *= rate;
            }
            if (p0 + 15 > all_to || p0 < all_from) {
#pragma unroll
                for (int i = 0; i < 16; ++i) s[i] = p0 + i <= last && p0 + i >= first ? s[i] : -INFINITY;
            }
            float mx[4] = {s[0], s[1], s[2], s[3]};
#pragma unroll
            for (int i = 4; i < 16; ++i) mx[i & 3] = fmaxf(mx[i & 3], s[i]);
            s_max[b][part][row] = fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3]));
            __syncwarp();
            if (lane == 0) mbar_arrive(&max_ready[quarter]);  // the warps of these rows
            ok = __all_sync(0xffffffffu, mbar_wait_bounded(&max_ready[quarter], (uint32_t)it & 1u, st));
            if (!ok) break;
            float top = s_max[b][0][row];
#pragma unroll
            for (int i = 1; i < kFaParts; ++i) top = fmaxf(top, s_max[b][i][row]);
            const float m_new = fmaxf(m, top);
            const float u = m_new == -INFINITY ? 0.f : m_new;  // nothing visible yet
            const float f = ex2(m - u);
            m = m_new;
            uint32_t p[8];
            float sum0 = 0.f, sum1 = 0.f;
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const float e0 = ex2(s[2 * i] - u), e1 = ex2(s[2 * i + 1] - u);
                sum0 += e0;
                sum1 += e1;
                p[i] = pack_half2(e0, e1);
            }
            l = fmaf(l, f, sum0 + sum1);
            // the probabilities of the tile before have been read, and its results are there, when its products are done
            if (it > 0 && !products_done(it - 1)) {
                ok = false;
                break;
            }
#pragma unroll
            for (int c = 0; c < 2; ++c)
                asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(p_row + (uint32_t)(((part * 2 + c) ^ (row & 7)) << 4)), "r"(p[4 * c]),
                             "r"(p[4 * c + 1]), "r"(p[4 * c + 2]), "r"(p[4 * c + 3])
                             : "memory");
            fence_async_smem();
            if (it > 0) add_values();  // (the next products replace them)
            f_before = f;
            __syncwarp();
            if (lane == 0) mbar_arrive(p_ready);
        }
        if (ok && n_tiles > 0) {
            ok = products_done(n_tiles - 1);
            if (ok) add_values();
        }
        if (!ok) *s_fail = 1;
        s_l[part][row] = l;
        asm volatile("bar.sync %0, %1;" ::"r"(1 + quarter), "n"(32 * kFaParts) : "memory");  // (every warp gets here)
        if (n_tiles > 0) {  // (also after a wait that ran out: the warps of these rows meet once more below)
            float total = s_l[0][row];
#pragma unroll
            for (int i = 1; i < kFaParts; ++i) total += s_l[i][row];
            // finished rows over the operands (every copy has landed and been read), so that a warp stores whole pieces of a row
            const int pitch = P * 64 + 4;
            float* rows = reinterpret_cast<float*>(smem + (sq - smem_u32(smem)));
            float* mine = rows + row * pitch + part * P * 16;
#pragma unroll
            for (int c = 0; c < kRaMaxPieces; ++c) {
                if (c >= P) break;
#pragma unroll
                for (int i = 0; i < 16; i += 4)
                    *reinterpret_cast<float4*>(mine + c * 16 + i) =
                        make_float4(__fdiv_rn(o[c][i], total), __fdiv_rn(o[c][i + 1], total), __fdiv_rn(o[c][i + 2], total), __fdiv_rn(o[c][i + 3], total));
            }
            asm volatile("bar.sync %0, %1;" ::"r"(1 + quarter), "n"(32 * kFaParts) : "memory");  // rows of this quarter
            for (int r = part; r < 32; r += kFaParts) {
                const int t = (quarter * 32 + r) / a.heads;
                if (t >= tokens) break;
                for (int c = 4 * lane; c < P * 64; c += 128) {
                    const float4 v = *reinterpret_cast<const float4*>(rows + (quarter * 32 + r) * pitch + c);
                    float y[4] = {v.x, v.y, v.z, v.w};
                    latent_planes4<SKV>(a, t0 + t, group * a.heads + quarter * 32 + r - t * a.heads, half * P * 64 + c, y);
                }
            }
        }
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

// The batched prompt path of engines with FP32 weights and an FP32 cache (the reference's own architecture on one GPU).
//
// The same arithmetic as the decode step, operation by operation and in the same order, only that every weight row is used
// for a block of tokens: a prompt's cache rows and logits are bit for bit those of the token-by-token loop, which streams
// all weights and pays a step's launches and host round trip for every token.  Bound by FP32 FMAs for large shapes, by the
// launches for small ones.
#pragma once
#include "attention.cuh"
#include "mamba.cuh"
#include "prefill.cuh"

namespace lpp {

// RMSNorm of a block's rows, the embedding rows in layer 0 (also written out as the residual stream).  The sum of squares is
// formed as the GEMV prologue forms it with its 256 threads (stage_input): neighbouring inputs strided over the threads one
// by one for an embedding row, four by four otherwise.  grid: rows; with a row list, block i takes row rows[i].
constexpr int kF32NormThreads = 256;
struct PrefillF32NormArgs {
    float* x;            // [tokens][D]
    const int* tokens;   // layer 0
    const float* emb;    // layer 0: [vocab][D], else nullptr
    float emb_scale;
    int vocab;
    const int* rows;
    const float* norm_w;
    float norm_eps;
    float* out;          // [rows][D]
    int D;
    StepState* st;
};
static __global__ void __launch_bounds__(kF32NormThreads) prefill_f32_norm_kernel(const PrefillF32NormArgs a) {
    __shared__ float red[kF32NormThreads / 32];
    pdl_launch_dependents();
    pdl_wait();
    const int tid = threadIdx.x, D = a.D;
    const int t = a.rows ? *reinterpret_cast<const volatile int*>(a.rows + blockIdx.x) : (int)blockIdx.x;
    float* x = a.x + (size_t)t * D;
    float* out = a.out + (size_t)blockIdx.x * D;
    float ss = 0.f;
    if (a.emb) {
        int tok = *reinterpret_cast<const volatile int*>(a.tokens + t);
        if (tok < 0 || tok >= a.vocab) {
            if (tid == 0) atomicOr(&a.st->status, kStatusBadToken);
            tok = 0;
        }
        const float* row = a.emb + (size_t)tok * D;
        for (int k = tid; k < D; k += kF32NormThreads) {
            const float v = __ldg(row + k) * a.emb_scale;
            ss = fmaf(v, v, ss);
            x[k] = v;
        }
        __syncthreads();  // the row is read back below in another split
    } else {
        for (int i = tid; i < (D >> 2); i += kF32NormThreads) {
            const float4 v = __ldcg(reinterpret_cast<const float4*>(x) + i);
            ss = fmaf(v.x, v.x, fmaf(v.y, v.y, fmaf(v.z, v.z, fmaf(v.w, v.w, ss))));
        }
    }
    ss = warp_sum(ss);
    if ((tid & 31) == 0) red[tid >> 5] = ss;
    __syncthreads();
    float tot = 0.f;
#pragma unroll
    for (int w = 0; w < kF32NormThreads / 32; ++w) tot += red[w];
    const float scale = __fdiv_rn(1.0f, __fsqrt_rn(__fadd_rn(__fdiv_rn(tot, (float)D), a.norm_eps)));
    for (int i = tid; i < (D >> 2); i += kF32NormThreads) {
        const float4 v = __ldcg(reinterpret_cast<const float4*>(x) + i), w = __ldg(reinterpret_cast<const float4*>(a.norm_w) + i);
        reinterpret_cast<float4*>(out)[i] = make_float4(__fmul_rn(__fmul_rn(v.x, scale), w.x), __fmul_rn(__fmul_rn(v.y, scale), w.y),
                                                        __fmul_rn(__fmul_rn(v.z, scale), w.z), __fmul_rn(__fmul_rn(v.w, scale), w.w));
    }
}

// W . x for a block of tokens.  A warp takes four weight rows and eight tokens: lane l forms the partial sums of inputs 4 l,
// 4 l + 128, ... as dot_rows does (two FMA chains, added at the end of every chunk of kc inputs), 128 FMAs for 12 vector
// loads; the 32 results are then added up over the lanes in the tree of warp_sum, which for 32 values at once takes 31
// shuffles instead of 160 and leaves lane 8 i + j with row i of token j.  Neighbouring warps of a CTA share rows or tokens,
// so most loads hit L1.  CHUNKS: K has more than one chunk.
constexpr int kF32Threads = 256, kF32Rows = 16, kF32Tokens = 16;  // a CTA's warps: four row groups x two token groups
struct PrefillF32Args {
    const float* w;      // [n_rows][K]
    const float* x;      // [tokens][K]
    int n_rows, K, kc, n_tokens;
    float* out;          // kPfResid: [tokens][out_pitch] += ; kPfSwiglu: [tokens][out_pitch], column row / 2; kPfStore: [tokens][out_pitch]
    int out_pitch, act;
    PrefillGemmArgs qkv; // kPfQkv: what pf_qkv_store takes
};
template <int EPI, bool CHUNKS>
static __global__ void __launch_bounds__(kF32Threads) prefill_f32_gemm_kernel(const PrefillF32Args a) {
    pdl_launch_dependents();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, K = a.K;
    const int row0 = blockIdx.x * kF32Rows + (warp & 3) * 4, tok0 = blockIdx.y * kF32Tokens + (warp >> 2) * 8;
    const float4 *w[4], *x[8];  // rows and tokens beyond the end repeat the last one and are not stored
#pragma unroll
    for (int i = 0; i < 4; ++i) w[i] = reinterpret_cast<const float4*>(a.w + (size_t)min(row0 + i, a.n_rows - 1) * K);
#pragma unroll
    for (int j = 0; j < 8; ++j) x[j] = reinterpret_cast<const float4*>(a.x + (size_t)min(tok0 + j, a.n_tokens - 1) * K);
    pdl_wait();
    float sum[4][8];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 8; ++j) sum[i][j] = 0.f;
    for (int k0 = 0; k0 < K; k0 += a.kc) {
        float p[4][8], q[4][8];
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 8; ++j) p[i][j] = q[i][j] = 0.f;
        const int end = min(k0 + a.kc, K) >> 2;
        for (int v = (k0 >> 2) + lane; v < end; v += 32) {
            float4 wv[4], xv[8];
#pragma unroll
            for (int i = 0; i < 4; ++i) wv[i] = __ldg(w[i] + v);
#pragma unroll
            for (int j = 0; j < 8; ++j) xv[j] = x[j][v];
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    p[i][j] = fmaf(wv[i].x, xv[j].x, p[i][j]);
                    q[i][j] = fmaf(wv[i].y, xv[j].y, q[i][j]);
                    p[i][j] = fmaf(wv[i].z, xv[j].z, p[i][j]);
                    q[i][j] = fmaf(wv[i].w, xv[j].w, q[i][j]);
                }
        }
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 8; ++j) sum[i][j] += p[i][j] + q[i][j];
        if (!CHUNKS) break;
    }
    // warp_sum of all 32: at every level a lane keeps the half of the values whose number has its bit set or clear
    float v[32];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 8; ++j) v[8 * i + j] = sum[i][j];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const bool up = lane & o;
#pragma unroll
        for (int n = 0; n < 32; ++n)
            if (n < o) {
                const float keep = up ? v[n + o] : v[n], send = up ? v[n] : v[n + o];
                v[n] = keep + __shfl_xor_sync(0xffffffffu, send, o);
            }
    }
    const float s = v[0], other = __shfl_xor_sync(0xffffffffu, s, 8);  // the row pair's other value
    const int row = row0 + (lane >> 3), t = tok0 + (lane & 7);
    if (row >= a.n_rows || t >= a.n_tokens) return;
    if constexpr (EPI == kPfStore) {
        a.out[(size_t)t * a.out_pitch + row] = s;
    } else if constexpr (EPI == kPfResid) {
        float* p = a.out + (size_t)t * a.out_pitch + row;
        *p = s + *p;  // x += W.xb (src/model.cpp:232, 239)
    } else if constexpr (EPI == kPfSwiglu) {
        // rows interleaved (gate, up): hb = (h1*sigmoid(h1))*h3 (src/ops.cpp:78-87)
        if ((row & 1) == 0) {
            const float sig = __fdiv_rn(1.0f, 1.0f + expf(-act_gate_arg(a.act, s)));
            a.out[(size_t)t * a.out_pitch + (row >> 1)] = __fmul_rn(__fmul_rn(s, sig), other);
        }
    } else {
        pf_qkv_store(a.qkv, row, t, s, other);
    }
}

// The same products for rows short enough that a tile of weight rows and of tokens fits shared memory.  KS (4 or 8) lanes share four
// rows x four tokens: lane c forms, one after the other, the partial sums that lanes c, c + KS, .. of the step's warp have (two FMA
// chains, here one pair: fma.rn.f32x2 rounds both halves like fmaf) and adds them up in the order in which warp_sum's tree takes
// them (lanes 16, 8, 4 apart); the last two or three levels are shuffles.  The kernel above needs 12 global vector loads and the
// transposing tree for a warp's 32 outputs, on one CTA an SM.  Bound by the instructions issued; a warp has 8 vector loads from shared
// memory and 32 pair FMAs for 16 rows x 8 tokens x 16 inputs.  201 tokens of the stories15M shape, us a launch above -> here: gate|up 30.1 ->
// 16.9, q|k|v 21.1 -> 12.4, output and down projection 13.6 -> 8.6.  (Lanes as tokens, weights read as broadcasts: 18.5, 15.6, 16.6: a vector
// load from shared memory keeps its pipe for four clocks also where all lanes read the same address.)
constexpr int kTileTokens = 32, kTileWarps = 8;  // four warps side by side cover the tokens, 8 each
template <int KS>
constexpr int kTileRows = 2 * 64 / KS;  // of a CTA: two warps of 4 (32 / KS / 2) rows each
__host__ __device__ inline int f32_tile_pitch(int K) { return ((K >> 2) | 1) << 2; }  // odd number of 16-byte pieces: no bank conflicts
__host__ __device__ inline size_t f32_tile_smem(int K, int rows) { return (size_t)(rows + kTileTokens) * f32_tile_pitch(K) * 4; }
template <int EPI, int KS>
static __global__ void __launch_bounds__(kTileWarps * 32, 2) prefill_f32_tile_kernel(const PrefillF32Args a) {
    extern __shared__ __align__(128) unsigned char smem[];
    constexpr int kRows = kTileRows<KS>, kGroups = 32 / KS / 2;  // row groups of a warp
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, K = a.K, nv = K >> 2, pitch = f32_tile_pitch(K) >> 2;
    uint4* ws = reinterpret_cast<uint4*>(smem);
    uint4* xs = ws + (size_t)kRows * pitch;
    const int row0 = blockIdx.x * kRows, tok0 = blockIdx.y * kTileTokens;
    pdl_launch_dependents();
    // A warp fetches row after row.  Rows and tokens beyond the end are neither fetched nor stored: what lies in their place only
    // reaches their own sums (to repeat the last token made every CTA read that row 32 times: 33 tokens 384 us, 64 tokens 280).
    for (int r = warp; r < min(kRows, a.n_rows - row0); r += kTileWarps) {
        const uint4* src = reinterpret_cast<const uint4*>(a.w + (size_t)(row0 + r) * K);
        for (int v = lane; v < nv; v += 32) cp_async_16(ws + r * pitch + v, src + v, true);  // constants: ahead of the dependency wait
    }
    pdl_wait();
    for (int r = warp; r < min(kTileTokens, a.n_tokens - tok0); r += kTileWarps) {
        const uint4* src = reinterpret_cast<const uint4*>(a.x + (size_t)(tok0 + r) * K);
        for (int v = lane; v < nv; v += 32) cp_async_16(xs + r * pitch + v, src + v, true);
    }
    cp_async_commit();
    cp_async_wait<0>();
    __syncthreads();
    const int c = lane % KS, group = lane / KS;
    const int r0 = ((warp >> 2) * kGroups + group % kGroups) * 4, t0 = (warp & 3) * 8 + (group / kGroups) * 4;  // within the tile
    uint32_t wa[4], xa[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        wa[i] = smem_u32(ws + (r0 + i) * pitch);
        xa[i] = smem_u32(xs + (t0 + i) * pitch);
    }
    auto lds = [](uint32_t at) -> ulonglong2 {
        ulonglong2 v;
        asm volatile("ld.shared.v2.u64 {%0, %1}, [%2];" : "=l"(v.x), "=l"(v.y) : "r"(at));
        return v;
    };
    // Partial sums of lane l of the step's warp, as pairs of tokens.  (A chain that starts with a product instead of a sum with +0, and p + q
    // without the sum with +0 it goes into there, differ from the step's in the sign of a zero only: the last line makes up for that.)
    auto chain = [&](int l, f32x2 (&s)[4][2]) {
        f32x2 pq[4][4];
        auto step = [&](uint32_t v, bool first) {
            ulonglong2 wv[4], xv[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                wv[i] = lds(wa[i] + v);
                xv[i] = lds(xa[i] + v);
            }
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) pq[i][j] = first ? mul2(wv[i].x, xv[j].x) : fma2(wv[i].x, xv[j].x, pq[i][j]);
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) pq[i][j] = fma2(wv[i].y, xv[j].y, pq[i][j]);
        };
        const uint32_t end = 16u * (uint32_t)nv;
        uint32_t v = 16u * (uint32_t)l;
        if (v < end) {
            step(v, true);
#pragma unroll 1
            for (v += 512u; v < end; v += 512u) step(v, false);
        } else {
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) pq[i][j] = 0ull;
        }
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 2; ++j) s[i][j] = pack_f2(pair_sum(pq[i][2 * j]), pair_sum(pq[i][2 * j + 1]));
    };
    auto add = [](f32x2 (&s)[4][2], const f32x2 (&o)[4][2]) {
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 2; ++j) s[i][j] = add2(s[i][j], o[i][j]);
    };
    f32x2 total[4][2];
#pragma unroll
    for (int b = 0; b < 8 / KS; ++b) {  // KS 4: lanes c, then c + 4
        f32x2 s8[4][2], s16[4][2], s[4][2];
        chain(c + 4 * b, s8);
        chain(c + 4 * b + 16, s);
        add(s8, s);
        chain(c + 4 * b + 8, s16);
        chain(c + 4 * b + 24, s);
        add(s16, s);
        add(s8, s16);
        if (b == 0) {
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 2; ++j) total[i][j] = s8[i][j];
        } else {
            add(total, s8);
        }
    }
    float sum[4];  // lane c goes on with token c of the four
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const float2 two = unpack_f2(total[i][j >> 1]);
            float v = j & 1 ? two.y : two.x;
            if constexpr (KS == 8) v += __shfl_xor_sync(0xffffffffu, v, 4);
            v += __shfl_xor_sync(0xffffffffu, v, 2);
            v += __shfl_xor_sync(0xffffffffu, v, 1);
            if (j == 0 || c == j) sum[i] = v + 0.f;
        }
    if (c >= 4) return;
    const int row = row0 + r0, t = tok0 + t0 + c;
    if (t >= a.n_tokens) return;
    if constexpr (EPI == kPfStore) {
#pragma unroll
        for (int i = 0; i < 4; ++i)
            if (row + i < a.n_rows) a.out[(size_t)t * a.out_pitch + row + i] = sum[i];
    } else if constexpr (EPI == kPfResid) {
        float* p = a.out + (size_t)t * a.out_pitch + row;
        float old[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) old[i] = row + i < a.n_rows ? p[i] : 0.f;
#pragma unroll
        for (int i = 0; i < 4; ++i)
            if (row + i < a.n_rows) p[i] = sum[i] + old[i];  // x += W.xb (src/model.cpp:232, 239)
    } else if constexpr (EPI == kPfSwiglu) {
        // rows interleaved (gate, up): hb = (h1*sigmoid(h1))*h3 (src/ops.cpp:78-87)
#pragma unroll
        for (int i = 0; i < 4; i += 2)
            if (row + i < a.n_rows) {
                const float sig = __fdiv_rn(1.0f, 1.0f + expf(-act_gate_arg(a.act, sum[i])));
                a.out[(size_t)t * a.out_pitch + ((row + i) >> 1)] = __fmul_rn(__fmul_rn(sum[i], sig), sum[i + 1]);
            }
    } else {
#pragma unroll
        for (int i = 0; i < 4; ++i) pf_qkv_store(a.qkv, row + i, t, sum[i], sum[i ^ 1]);
    }
}

// The decode attention of attn_decode_kernel for a block of tokens: token t attends to positions 0 .. start_pos + t with the
// splits that a step at its position uses (a.n_splits: at least as many as the last token's); rows before block_pos are complete before the block's first kernel starts.  grid: (splits of the last token, kv heads, tokens x head batches)
// Bound by the latency of its stages, so CTAs an SM count: as many as fit without spills to speak of.  800 tokens, whole prompts in us with the
// compiler's own choice / with one CTA but three up to dpl * gb = 8 / with these: head size 128, 8 heads of 1024 7747 / 8713 / 7716; 64
// with two query heads a KV head 3972 / 3882 / 3139; 32 with four 4100 / 5253 / 4098; 48 with two 1480 / 2055 / 1476; 16 heads of 16 2275 / 2628 /
// 2310; 64 with one (three CTAs spill 144 bytes, 5571) 5478.
constexpr int f32_attn_ctas(int dpl, int gb) { return dpl * gb <= 4 ? 4 : dpl * gb <= 8 && dpl < 8 ? 3 : dpl * gb <= 16 ? 2 : 1; }
template <int DPL, int GB>
static __global__ void __launch_bounds__(kAttnKernelThreads, f32_attn_ctas(DPL, GB)) prefill_f32_attn_kernel(AttnArgs a, int start_pos, int block_pos, int n_z, int q_rows,
                                                                                      int part_row) {
    __shared__ float s_scratch[(kAttnKernelThreads / 32) * GB * (DPL * 8 + 2)];
    __shared__ int s_last;
    pdl_launch_dependents();
    const int t = blockIdx.z / n_z, hz = blockIdx.z - t * n_z, T = start_pos + t + 1;
    const int n_eff = attn_effective_splits(T, a.n_splits, a.min_chunk);
    if ((int)blockIdx.x >= n_eff) return;
    a.q += (size_t)t * q_rows;
    a.out += (size_t)t * q_rows;
    a.part += (size_t)t * part_row;
    a.counters += (size_t)t * gridDim.y * n_z;
    attn_item<float, DPL, GB, kAttnKernelThreads>(a, blockIdx.x, blockIdx.y, hz, n_z, T, n_eff, s_scratch, &s_last, threadIdx.x, 0, block_pos);
}

}  // namespace lpp

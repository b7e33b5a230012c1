// The batched prompt path of engines with FP32 weights and an FP32 cache (the reference's own architecture on one GPU).
//
// The same arithmetic as the decode step, operation by operation and in the same order, only that every weight row is used
// for a block of tokens: a prompt's cache rows and logits are bit for bit those of the token-by-token loop, which streams
// all weights and pays a step's launches and host round trip for every token.  Bound by FP32 FMAs for large shapes, by the
// launches for small ones.  201 tokens of the stories15M shape: 20.9 ms token by token, 0.77 ms here.
#pragma once
#include "attention.cuh"
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

// The decode attention of attn_decode_kernel for a block of tokens: token t attends to positions 0 .. start_pos + t with the
// splits that a step at its position uses; rows before block_pos are complete before the block's first kernel starts.  grid: (splits of the last token, kv heads, tokens x head batches)
template <int DPL, int GB>
static __global__ void __launch_bounds__(kAttnKernelThreads) prefill_f32_attn_kernel(AttnArgs a, int start_pos, int block_pos, int n_z, int q_rows,
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

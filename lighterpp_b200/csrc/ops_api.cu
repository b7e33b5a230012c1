// C-ABI entry points for the stand-alone operators: one per host wrapper of the reference's
// src/kernels.cuh:24-36, same argument meaning, device pointers in and out, nothing synchronised
// (like the reference wrappers, callers order work through the stream).
#include <cuda_runtime.h>
#include <cuda_fp16.h>
#include <stddef.h>

#include <algorithm>

#include "../../include/lpp_b200.h"
#include "common.cuh"
#include "gemv.cuh"
#include "ops.cuh"
#include "sampler.cuh"
#include "sampler_exact.cuh"

using namespace lpp;

namespace {

inline lpp_status chk() { return cudaGetLastError() == cudaSuccess ? LPP_OK : LPP_ERR_CUDA; }
inline cudaStream_t S(void* s) { return (cudaStream_t)s; }
inline int blocks(long long n, int t) { return (int)std::max<long long>(1, (n + t - 1) / t); }

// Launches an operator kernel.  It may start while the kernel before it in the stream ends (it waits for it in op_begin):
// 18 operators of a layer one after the other take about a microsecond less each.  A stream that is being captured gets a plain
// launch, because what comes before it in the graph need not be a kernel.
template <typename... KArgs, typename... Args>
lpp_status launch_op(void (*kernel)(KArgs...), dim3 grid, int threads, size_t smem, cudaStream_t s, Args... args) {
    cudaStreamCaptureStatus capturing = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(s, &capturing) != cudaSuccess) {
        (void)cudaGetLastError();
        capturing = cudaStreamCaptureStatusActive;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute attr = {};
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = capturing == cudaStreamCaptureStatusNone ? 1 : 0;
    cudaLaunchKernelEx(&cfg, kernel, ((KArgs)args)...);
    return chk();
}

// Any-shape fallback for the stand-alone GEMV: one warp per row, scalar loads.
template <typename WT>
__global__ void gemv_generic_kernel(float* out, const float* x, const WT* w, int n, int d) {
    op_begin();
    const int row = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    const int lane = threadIdx.x & 31;
    if (row >= n) return;
    const WT* r = w + (size_t)row * d;
    float acc = 0.f;
    for (int k = lane; k < d; k += 32) {
        float wv;
        if constexpr (sizeof(WT) == 2)
            wv = __half2float(r[k]);
        else
            wv = r[k];
        acc = fmaf(wv, x[k], acc);
    }
    acc = warp_sum(acc);
    if (lane == 0) out[row] = acc;
}

template <typename WT>
lpp_status op_gemv_t(float* out, const float* x, const void* w, int n, int d, cudaStream_t s) {
    const int vec = 16 / (int)sizeof(WT);
    const size_t smem = (size_t)d * 4;
    // the vector kernel stages x and reads the rows with 16-byte loads: anything else (an offset sub-vector, say) takes the
    // scalar kernel
    if ((d % vec) || (((uintptr_t)w) & 15) || (((uintptr_t)x) & 15) || smem > 200 * 1024)
        return launch_op(gemv_generic_kernel<WT>, dim3(blocks(n, 8)), 256, 0, s, out, x, (const WT*)w, n, d);
    if (smem > 48 * 1024 &&
        cudaFuncSetAttribute(op_gemv_kernel<WT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess)
        return LPP_ERR_CUDA;
    int dev = 0, sms = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    // two CTAs per SM; as many warps on a row as leave every warp something to do in one round, and a row of less than a
    // batch per warp to one
    const int warps = kOpGemvThreads / 32, ctas = 2 * sms;
    int split = 1;
    while (split < warps && (long long)n * split * 2 <= (long long)ctas * warps && d / vec >= split * 2 * 32 * kOpGemvU) split *= 2;
    const int grid = std::min(ctas, blocks((long long)n * split, warps));
    return launch_op(op_gemv_kernel<WT>, dim3(grid), kOpGemvThreads, smem, s, out, x, (const WT*)w, n, d, split);
}

// ---- scratch layout of the stand-alone samplers: step state, per-block partials, ticket counter and barrier
//      words, then what the exact-order kernel adds (block sums, entry counts, entry lists).
//      `cap_blocks` sizes the areas: the blocks of this call (stream-ordered scratch) or of the largest
//      vocabulary the fixed array takes.
struct SampleScratch {
    size_t state, part, counters, sums, counts, entries, total;
};
constexpr SampleScratch sample_scratch_layout(int cap_blocks, bool exact) {
    SampleScratch L = {};
    size_t o = 0;
    L.state = o;
    o += (sizeof(StepState) + 255) & ~(size_t)255;
    L.part = o;
    o += ((size_t)cap_blocks * 12 + 255) & ~(size_t)255;
    L.counters = o;  // [0] ticket counter of the tree kernel; from +256: barrier counter and exit ticket of the exact kernel
    o += 512;
    if (exact) {
        L.sums = o;
        o += ((size_t)cap_blocks * sizeof(double) + 255) & ~(size_t)255;
        L.counts = o;
        o += ((size_t)kExactLists * cap_blocks * sizeof(int) + 255) & ~(size_t)255;
        L.entries = o;
        o += (size_t)kExactLists * cap_blocks * kExactMaxEntries * sizeof(ExactEntry);
    }
    L.total = o;
    return L;
}

// Writes the step-state header the sampler reads, copies the history device-to-device and zeroes
// the counters -- everything in the scratch that has to start clean.
__global__ void __launch_bounds__(256) sample_setup_kernel(StepState* st, unsigned int* counters, float temperature, float penalty, float r,
                                                           const int* history, int history_len) {
    op_begin();
    if (threadIdx.x == 0) {
        st->token = 0;
        st->pos = 0;
        st->history_len = history_len;
        st->history_window = 0;
        st->history_count = 0;
        st->step_idx = 0;
        st->advance = 0;
        st->temperature = temperature;
        st->penalty = penalty;
        st->r = r;
        st->out_token = -1;
        st->status = 0;
        st->wait_cycles = 0;
        st->tp_wait_cycles = 0;
    }
    if (threadIdx.x < 128) counters[threadIdx.x] = 0u;  // ticket counter, barrier counter, exit ticket
    for (int i = threadIdx.x; i < history_len; i += blockDim.x) st->history[i] = history[i];
}

// What a call on a vocabulary of this size launches.
struct SamplePlan {
    int blocks;
    bool exact;  // the exact-order kernel (ids equal to the reference's sequential CPU sample()) needs all its blocks co-resident
};
lpp_status sample_plan(int vocab_size, SamplePlan* p) {
    int dev = 0, sms = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return LPP_ERR_CUDA;
    p->blocks = (vocab_size + kSampleChunk - 1) / kSampleChunk;
    p->exact = p->blocks <= sms;
    return p->blocks > kSampleMaxBlocks ? LPP_ERR_TOO_LARGE : LPP_OK;
}

// Runs the sampler on logits with its scratch at `scratch` (laid out by sample_scratch_layout for at least the blocks of this
// vocabulary): two launches, everything that a call needs travels as kernel arguments.  (Header and counters as copies and a
// memset, the token as another copy: four more operations of the stream between the launches.)
lpp_status run_sampler(char* scratch, const SampleScratch& L, const SamplePlan& plan, float* d_logits, int vocab_size, float temperature, float penalty,
                       const int* d_history, int history_len, float r, int* d_token, cudaStream_t s) {
    const int nb = plan.blocks;
    const bool use_hist = penalty > 1.0f && d_history && history_len > 0;
    const lpp_status st = launch_op(sample_setup_kernel, dim3(1), 256, 0, s, (StepState*)(scratch + L.state), (unsigned int*)(scratch + L.counters),
                                    temperature, penalty, r, use_hist ? d_history : nullptr, use_hist ? history_len : 0);
    if (st != LPP_OK) return st;
    SampleArgs a = {};
    a.logits = d_logits;
    a.vocab = vocab_size;
    a.st = (StepState*)(scratch + L.state);
    a.part_max = (float*)(scratch + L.part);
    a.part_idx = (int*)(scratch + L.part + (size_t)nb * 4);
    a.part_sum = (float*)(scratch + L.part + (size_t)nb * 8);
    a.counter = (unsigned int*)(scratch + L.counters);
    a.token_out = d_token;
    if (!plan.exact) return launch_op(sample_kernel, dim3(nb), kSampleThreads, 0, s, a);
    SampleExactArgs ea = {};
    ea.base = a;
    ea.sync = (unsigned int*)(scratch + L.counters + 256);
    ea.block_sum = (double*)(scratch + L.sums);
    ea.entry_count = (int*)(scratch + L.counts);
    ea.entries = (ExactEntry*)(scratch + L.entries);
    return launch_op(sample_exact_kernel, dim3(nb), kSampleThreads, 0, s, ea);
}

// ---- scratch for lpp_op_sample_static: lives in the library image, one copy per GPU that loads it
constexpr int kStaticSampleMaxVocab = 262144;  // 128 blocks of kSampleChunk logits
constexpr int kStaticSampleBlocks = kStaticSampleMaxVocab / kSampleChunk;
constexpr SampleScratch kStaticLayout = sample_scratch_layout(kStaticSampleBlocks, true);
static __device__ __align__(256) unsigned char g_sample_scratch[kStaticLayout.total];
// Device addresses of g_sample_scratch, one per CUDA device, filled in on first use.  In host code
// the name g_sample_scratch is only a handle for cudaGetSymbolAddress, never a pointer to pass on.
static unsigned char* g_sample_scratch_addr[64];

}  // namespace

void lpp_internal_set_error(const char* msg);  // engine.cu: text behind lpp_last_error()

extern "C" {

lpp_status lpp_op_convert_f32_to_f16(void* d_dst, const float* d_src, int64_t n, void* stream) {
    if (!d_dst || !d_src || n < 0) return LPP_ERR_INVALID_ARG;
    if (n == 0) return LPP_OK;
    return launch_op(convert_f32_to_f16_kernel, dim3(std::min(blocks(n, 256), 148 * 16)), 256, 0, S(stream), (__half*)d_dst, d_src, (long long)n);
}

lpp_status lpp_op_gemv(float* d_out, const float* d_x, const void* d_w, int n, int d, int w_dtype, void* stream) {
    if (!d_out || !d_x || !d_w || n <= 0 || d <= 0) return LPP_ERR_INVALID_ARG;
    if (w_dtype == LPP_F16) return op_gemv_t<__half>(d_out, d_x, d_w, n, d, S(stream));
    if (w_dtype == LPP_F32) return op_gemv_t<float>(d_out, d_x, d_w, n, d, S(stream));
    return LPP_ERR_INVALID_ARG;
}

lpp_status lpp_op_rmsnorm(float* d_out, const float* d_x, const float* d_w, int n, void* stream) {
    if (!d_out || !d_x || !d_w || n <= 0) return LPP_ERR_INVALID_ARG;
    return launch_op(rmsnorm_kernel, dim3(1), kOpNormThreads, 0, S(stream), d_out, d_x, d_w, n);
}

lpp_status lpp_op_rope(float* d_q, float* d_k, int pos, int dim, int kv_dim, int head_size, float rope_base,
                       void* stream) {
    if (!d_q || !d_k || dim <= 0 || (dim & 1) || head_size <= 0 || (head_size & 1)) return LPP_ERR_INVALID_ARG;
    return launch_op(rope_kernel, dim3(blocks(dim / 2, 256)), 256, 0, S(stream), d_q, d_k, pos, dim, kv_dim, head_size, rope_base);
}

lpp_status lpp_op_swiglu(float* d_hb, const float* d_h1, const float* d_h3, int size, void* stream) {
    if (!d_hb || !d_h1 || !d_h3 || size <= 0) return LPP_ERR_INVALID_ARG;
    return launch_op(swiglu_kernel, dim3(blocks(size, 256)), 256, 0, S(stream), d_hb, d_h1, d_h3, size);
}

lpp_status lpp_op_softmax_multihead(float* d_out, const float* d_x, int n_heads, int seq_len, int att_stride,
                                    void* stream) {
    if (!d_out || !d_x || n_heads <= 0 || seq_len <= 0) return LPP_ERR_INVALID_ARG;
    return launch_op(softmax_multihead_kernel, dim3(n_heads), 256, 0, S(stream), d_out, d_x, seq_len, att_stride);
}

lpp_status lpp_op_scale_multihead(float* d_att, float scale, int n_heads, int seq_len, int att_stride, void* stream) {
    if (!d_att || n_heads <= 0 || seq_len <= 0) return LPP_ERR_INVALID_ARG;
    return launch_op(scale_multihead_kernel, dim3(blocks(seq_len, 256), n_heads), 256, 0, S(stream), d_att, scale, seq_len, att_stride);
}

lpp_status lpp_op_aggregation_multihead(float* d_out, const void* d_v_f16, const float* d_att, int n_heads,
                                        int seq_len, int head_size, int gqa_factor, int att_stride, void* stream) {
    if (!d_out || !d_v_f16 || !d_att || n_heads <= 0 || seq_len <= 0 || head_size <= 0 || head_size > 128 ||
        gqa_factor <= 0)
        return LPP_ERR_INVALID_ARG;
    const __half* v = (const __half*)d_v_f16;
    if (head_size % 8 || ((uintptr_t)v & 15))
        return launch_op(aggregation_any_kernel, dim3(n_heads), 128, 0, S(stream), d_out, v, d_att, seq_len, head_size, gqa_factor, att_stride);
    return launch_op(aggregation_kernel, dim3(n_heads * kAggCtas), kAggThreads, 0, S(stream), d_out, v, d_att, seq_len, head_size, gqa_factor,
                     att_stride);
}

lpp_status lpp_op_residual_add(float* d_out, const float* d_a, const float* d_b, int n, void* stream) {
    if (!d_out || !d_a || !d_b || n <= 0) return LPP_ERR_INVALID_ARG;
    return launch_op(residual_add_kernel, dim3(blocks(n, 256)), 256, 0, S(stream), d_out, d_a, d_b, n);
}

lpp_status lpp_op_scatter_kv(void* d_kc_f16, void* d_vc_f16, const float* d_k, const float* d_v, int layer, int pos,
                             int n_kv_heads, int head_size, int seq_len, void* stream) {
    if (!d_kc_f16 || !d_vc_f16 || !d_k || !d_v || layer < 0 || pos < 0 || pos >= seq_len || n_kv_heads <= 0 ||
        head_size <= 0)
        return LPP_ERR_INVALID_ARG;
    return launch_op(scatter_kv_kernel, dim3(blocks(n_kv_heads * head_size, 256)), 256, 0, S(stream), (__half*)d_kc_f16, (__half*)d_vc_f16, d_k,
                     d_v, layer, pos, n_kv_heads, head_size, seq_len);
}

lpp_status lpp_op_multihead_gemv(float* d_out, const float* d_q, const void* d_k_cache_f16, int layer, int pos,
                                 int n_heads, int n_kv_heads, int head_size, int seq_len, void* stream) {
    if (!d_out || !d_q || !d_k_cache_f16 || layer < 0 || pos < 0 || pos >= seq_len || n_heads <= 0 ||
        n_kv_heads <= 0 || n_heads % n_kv_heads)
        return LPP_ERR_INVALID_ARG;
    const __half* kc = (const __half*)d_k_cache_f16;
    auto dot = [&](auto kernel, int lanes) {  // lanes of a cache row
        const int rows = kDotThreads / lanes * kDotRows;
        return launch_op(kernel, dim3(blocks(pos + 1, rows), n_heads), kDotThreads, 0, S(stream), d_out, d_q, kc, layer, pos, n_heads, n_kv_heads,
                         seq_len);
    };
    if (((uintptr_t)kc & 15) == 0) {
        switch (head_size) {
            case 16: return dot(multihead_gemv_kernel<2>, 2);
            case 32: return dot(multihead_gemv_kernel<4>, 4);
            case 64: return dot(multihead_gemv_kernel<8>, 8);
            case 128: return dot(multihead_gemv_kernel<16>, 16);
            case 256: return dot(multihead_gemv_kernel<32>, 32);
        }
    }
    return launch_op(multihead_gemv_any_kernel, dim3(blocks(pos + 1, 4), n_heads), 128, 0, S(stream), d_out, d_q, kc, layer, pos, n_heads,
                     n_kv_heads, head_size, seq_len);
}

lpp_status lpp_op_rope_scatter(float* d_q, const float* d_k, const float* d_v, void* d_kc_f16, void* d_vc_f16,
                               int layer, int pos, int dim, int n_kv_heads, int head_size, int seq_len,
                               float rope_base, void* stream) {
    if (!d_q || !d_k || !d_v || !d_kc_f16 || !d_vc_f16 || layer < 0 || pos < 0 || pos >= seq_len || dim <= 0 ||
        (dim & 1) || (head_size & 1) || head_size <= 0)
        return LPP_ERR_INVALID_ARG;
    return launch_op(rope_scatter_kernel, dim3(blocks(dim / 2, 256)), 256, 0, S(stream), d_q, d_k, d_v, (__half*)d_kc_f16, (__half*)d_vc_f16,
                     layer, pos, dim, n_kv_heads, head_size, seq_len, rope_base);
}

int64_t lpp_op_sample_scratch_bytes(int vocab_size) {
    SamplePlan p = {};
    if (vocab_size <= 0 || sample_plan(vocab_size, &p) != LPP_OK) return -1;
    return (int64_t)sample_scratch_layout(p.blocks, p.exact).total;
}

lpp_status lpp_op_sample_on(void* scratch, int64_t scratch_bytes, float* d_logits, int vocab_size, float temperature, float penalty,
                            const int* d_history, int history_len, float r, int* d_sampled_token, void* stream) {
    if (!scratch || ((uintptr_t)scratch & 255) || !d_logits || !d_sampled_token || vocab_size <= 0 || history_len < 0 || history_len > kHistoryMax)
        return LPP_ERR_INVALID_ARG;
    SamplePlan p = {};
    const lpp_status st = sample_plan(vocab_size, &p);
    if (st != LPP_OK) return st;
    const SampleScratch L = sample_scratch_layout(p.blocks, p.exact);
    if (scratch_bytes < (int64_t)L.total) return LPP_ERR_INVALID_ARG;
    return run_sampler((char*)scratch, L, p, d_logits, vocab_size, temperature, penalty, d_history, history_len, r, d_sampled_token, S(stream));
}

lpp_status lpp_op_sample(float* d_logits, int vocab_size, float temperature, float penalty, const int* d_history,
                         int history_len, float r, int* d_sampled_token, void* stream) {
    if (!d_logits || !d_sampled_token || vocab_size <= 0 || history_len < 0 || history_len > kHistoryMax)
        return LPP_ERR_INVALID_ARG;
    cudaStream_t s = S(stream);
    SamplePlan p = {};
    lpp_status st = sample_plan(vocab_size, &p);
    if (st != LPP_OK) return st;
    const SampleScratch L = sample_scratch_layout(p.blocks, p.exact);  // stream-ordered scratch, sized for this call
    char* scratch = nullptr;
    if (cudaMallocAsync((void**)&scratch, L.total, s) != cudaSuccess) return LPP_ERR_CUDA;
    st = run_sampler(scratch, L, p, d_logits, vocab_size, temperature, penalty, d_history, history_len, r, d_sampled_token, s);
    cudaFreeAsync(scratch, s);
    return st != LPP_OK ? st : chk();
}

lpp_status lpp_op_sample_static(float* d_logits, int vocab_size, float temperature, float penalty,
                                const int* d_history, int history_len, float r, int* d_sampled_token, void* stream) {
    if (!d_logits || !d_sampled_token || vocab_size <= 0 || history_len < 0) {
        lpp_internal_set_error("lpp_op_sample_static: null pointer or non-positive size");
        return LPP_ERR_INVALID_ARG;
    }
    if (vocab_size > kStaticSampleMaxVocab || history_len > kHistoryMax) {
        lpp_internal_set_error("lpp_op_sample_static: vocab_size > 262144 or history_len > 4096 exceeds the built-in "
                               "scratch; use lpp_op_sample, which sizes its scratch per call");
        return LPP_ERR_TOO_LARGE;
    }
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) {
        lpp_internal_set_error("lpp_op_sample_static: no current CUDA device");
        return LPP_ERR_CUDA;
    }
    if (!g_sample_scratch_addr[dev]) {
        // one-time set-up for this device (it must be the current one): resolve where the symbol lives
        unsigned char* p = nullptr;
        const cudaError_t ge = cudaGetSymbolAddress((void**)&p, g_sample_scratch);
        if (ge != cudaSuccess || !p) {
            lpp_internal_set_error(cudaGetErrorString(ge));
            return LPP_ERR_CUDA;
        }
        g_sample_scratch_addr[dev] = p;
    }
    unsigned char* scratch = g_sample_scratch_addr[dev];
    cudaStream_t s = S(stream);
    SamplePlan p = {};
    const lpp_status st = sample_plan(vocab_size, &p);  // the same choice of kernel as lpp_op_sample
    if (st != LPP_OK) return st;
    return run_sampler((char*)scratch, kStaticLayout, p, d_logits, vocab_size, temperature, penalty, d_history, history_len, r, d_sampled_token, s);
}

}  // extern "C"

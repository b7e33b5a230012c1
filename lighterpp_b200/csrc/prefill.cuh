// Batched prompt path ("prefill"): the K/V cache rows of a block of prompt positions in one pass over
// the weights, instead of one pass per token.
//
// The reference feeds a prompt through forward() token by token (src/main.cpp:163-179): every prompt token
// streams all weights once.  Here the layer's matrices are streamed ONCE for the whole block of tokens: the
// four projections become small GEMMs  C[tokens][rows] = X[tokens][K] . W[rows][K]^T  that are still bound by
// the weight stream (2 FLOP per weight byte and token: far below the tensor cores' ridge for 64 tokens), so the
// kernels are organised around that stream like the decode GEMV -- a producer thread, a ring of shared-memory
// stages, mbarrier hand-over -- only that a stage is a pair of tiles fetched by the tensor memory accelerator
// (cp.async.bulk.tensor with the 128-byte swizzle, one copy per operand and stage: 128 weight rows x 128 inputs
// through a 3-D map, the matching 64 tokens x 128 inputs of the activations, hi and lo plane, through a 4-D map;
// the weight tiles of the first ring pass are requested before the dependency wait) and the arithmetic runs on
// the tensor cores: prefill_gemm_umma_kernel issues tcgen05.mma reading both operands from shared memory through
// matrix descriptors, FP32 accumulators in tensor memory, epilogue warps that read them back with tcgen05.ld.
// (An earlier kernel that consumed the same ring with ldmatrix + mma.sync.m16n8k16 in eight warps measured 1.17 ms
// against 0.83 ms for a 64-token pass of the Llama-3.2-1B shape and was removed.)
// Matrices whose row tiles do not fill the GPU (QKV, o_proj, down) are also cut along K so that every SM streams
// a share; partial sums are added in a fixed order by the next kernel (the norm kernel for the residual
// projections, prefill_qkv_finish_kernel for QKV).  Activations reach the MMAs as hi + lo FP16 pairs (see
// split_half); everything between the GEMMs (residual stream, RMSNorm, RoPE, softmax) stays FP32, following
// src/ops.cpp like the decode path.  The causal attention of the block is a tensor-core
// flash attention over the cache (prefill_attention.cuh; other head sizes: prefill_attention_kernel).
//
// Tensor maps cover this GPU's own memory only, and no copy is a multicast one.
#pragma once
#include <cuda.h>

#include "common.cuh"

namespace lpp {

constexpr int kPfTile = 64;          // tokens of an item of the CTA kernel (rows of its activation tiles)
constexpr int kPfMaxTokens = 1024;   // most tokens of a block
constexpr int kPfKc = 128;           // inputs per stage: two 64-wide (128-byte) swizzled sub-tiles per operand
constexpr int kPfMaxSplits = 8;
constexpr int kPfRingBytes = 192 * 1024;
constexpr int kPfSmemBytes = 1024 /*barriers*/ + 1024 /*alignment slack*/ + kPfRingBytes;

enum PfEpi : int {
    kPfQkv = 0,
    kPfResid = 1,
    kPfSwiglu = 2,
    kPfStore = 3,         // logits, or partial sums for a finishing kernel
    kPfLatentQuery = 4,   // latent attention: a head's query in the latent space -> FP16 query rows
    kPfLatentValue = 5    // latent attention: a head's value times its gate -> hi + lo operand
};

// An activation x is handed to the tensor cores as two numbers of the weights' 16-bit type, hi = round(x) and
// lo = round(x - hi): the MMA accumulates W.hi + W.lo in FP32, which keeps about 22 bits of x with FP16 (17 with BF16),
// so the batched pass carries FP32 activations through 16-bit-operand MMAs like the token loop carries them through its
// FP32 arithmetic.  Every activation buffer holds the hi plane [cap][cols] (cap: the tokens the buffers have room
// for) followed by the lo plane; one
// 4-D tensor map covers both.
template <typename T>
__device__ __forceinline__ void split_pair(float x, T& hi, T& lo) {
    hi = from_float<T>(x);
    lo = from_float<T>(x - to_float(hi));
}
__device__ __forceinline__ void split_half(float x, __half& hi, __half& lo) { split_pair(x, hi, lo); }

struct PrefillGemmArgs {
    int n_rows, K;        // rows of the weight matrix, inputs per row
    int row0;             // first row of this layer's matrix inside the tensor map (layers are stacked)
    int n_tokens;         // valid tokens
    int cap;              // token rows of a plane of the activation buffers
    int part_tokens;      // token rows of one range of K in part and out
    int start_pos;        // position of token 0
    int tile;             // tokens of an item: kPfTile (this file's kernel) or kPairTokens (prefill_pair.cuh)
    int box_tokens;       // this file's kernel: token rows of an activation tile, a multiple of 16 up to kPfTile
    int splits;           // K is cut into this many ranges: work item = (row tile, token tile, range)
    StepState* st;
    // kPfResid: x[t][row] += c (x: [tokens][n_rows] FP32) when splits == 1; else the partial sums go to
    // part[split][t][row] and the next kernel (prefill_norm_kernel) adds them to x in split order
    float* x;
    float* part;
    int x_pitch;          // row pitch of x and part (kPfResid)
    // kPfSwiglu: hb[t][row/2] = act(gate) * up   (rows interleaved gate, up; hb: hi and lo plane [cap][hb_pitch])
    void* hb;
    int hb_pitch;
    int act;
    // kPfStore: out[split][t][row], rows of out_pitch floats
    float* out;
    int out_pitch;
    // Grouped weights (heads): `groups` matrices of n_rows rows each, group_stride rows apart in the tensor map; group g
    // multiplies the K inputs that start at 64-input piece g * group_pieces of the activations.  0 = one matrix.
    int groups, group_stride, group_pieces;
    // kPfLatentQuery: query rows (token * groups + group) of lat_pitch FP16 elements
    __half* lat_query;
    int lat_pitch;
    // kPfLatentValue: column group * n_valid + row of hb (rows below n_valid), times gate[t][group]
    const float* gate;
    int n_valid;
    // kPfQkv: partial sums like kPfResid, also of one range; prefill_qkv_finish_kernel: rows are q | k | v; RoPE on q and k, q -> FP32 [tokens][q_rows], k/v -> cache at start_pos + t
    float* q;
    int q_rows, kv_rows, head_size, seq_len;
    const float2* rope;   // [seq_len][head_size/2]
    void* k_cache;        // this layer: [kv_heads][seq_len][head_size], FP16 (FP32 weights: FP32)
    void* v_cache;
};

__device__ __forceinline__ void tma_load_3d(uint32_t smem_dst, const CUtensorMap* map, int x, int y, int z, uint32_t bar_addr) {
    asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];" ::"r"(
                     smem_dst),
                 "l"(map), "r"(x), "r"(y), "r"(z), "r"(bar_addr)
                 : "memory");
}
__device__ __forceinline__ void tma_load_4d(uint32_t smem_dst, const CUtensorMap* map, int x, int y, int z, int w, uint32_t bar_addr) {
    asm volatile("cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5}], [%6];" ::"r"(
                     smem_dst),
                 "l"(map), "r"(x), "r"(y), "r"(z), "r"(w), "r"(bar_addr)
                 : "memory");
}

__device__ __forceinline__ void mma_f16_16816(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
                 : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void ldmatrix_x4(uint32_t addr, uint32_t& r0, uint32_t& r1, uint32_t& r2, uint32_t& r3) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3) : "r"(addr));
}
// One value of the QKV rows of the FP32 path: row `row` (and its pair partner `other`, the value of row ^ 1), token t: rotation of q and k
// pairs, q -> FP32 rows, k / v -> cache rows at the reference index.
__device__ __forceinline__ void pf_qkv_store(const PrefillGemmArgs& a, int row, int t, float v, float other) {
    const int pos = a.start_pos + t;
    if (row >= a.n_rows || t >= a.n_tokens) return;
    if (pos < 0 || pos >= a.seq_len) {
        atomicOr(&a.st->status, kStatusBadPos);
        return;
    }
    const int hs = a.head_size;
    float r = v;
    if (row < a.q_rows + a.kv_rows) {
        // adjacent-pair rotation with the table entry for (pos, (row % hs)/2) (src/ops.cpp:34-54)
        const float2 cs = __ldg(a.rope + (size_t)pos * (hs >> 1) + ((row % hs) >> 1));
        r = (row & 1) ? __fadd_rn(__fmul_rn(other, cs.y), __fmul_rn(v, cs.x))   // v1' = v0*sin + v1*cos
                      : __fsub_rn(__fmul_rn(v, cs.x), __fmul_rn(other, cs.y));  // v0' = v0*cos - v1*sin
    }
    if (row < a.q_rows) {
        a.q[(size_t)t * a.q_rows + row] = r;
    } else {
        const bool is_k = row < a.q_rows + a.kv_rows;
        const int rr = row - a.q_rows - (is_k ? 0 : a.kv_rows);
        const int h = rr / hs, off = rr % hs;
        // cache index within the layer: h*(seq_len*hs) + pos*hs + off (src/scatter_kv.cu:15-16)
        const size_t idx = (size_t)h * ((size_t)a.seq_len * hs) + (size_t)pos * hs + off;
        reinterpret_cast<float*>(is_k ? a.k_cache : a.v_cache)[idx] = r;
    }
}

// ---- the GEMM on the fifth-generation tensor cores (tcgen05), accumulators in tensor memory
//
// A work item is (tile of 128 weight rows, K range).  Per stage the tensor memory accelerator delivers the two
// 128-row x 64-input weight sub-tiles and, per 64-input piece, the 64 hi rows followed by the 64 lo rows of the
// activations, all in the 128-byte swizzled K-major layout that the MMA reads straight from shared memory through
// matrix descriptors: one elected thread issues eight 128 x 128 x 16 MMAs per stage (D[128 rows][hi tokens | lo
// tokens] += W . X^T) into one of two 128-column accumulators in tensor memory, commits the stage back to the
// producer, and after the last stage of the item commits the accumulator to the eight epilogue warps; these read
// their 32 lanes (rows) x 32 token columns of both halves with tcgen05.ld, add them, release the accumulator and
// run the epilogue from registers while the next item's MMAs already fill the other accumulator.  Warp roles: 0
// producer, 1 MMA issue and tensor-memory allocation, 2..9 epilogue (a warp may only read the tensor-memory lanes
// of its quarter, warp index modulo 4; two warps share a quarter and take 32 tokens each).  An epilogue thread owns
// one weight row and walks its tokens, so what depends on the row alone is computed once.
// Every CTA reads all activations of its K range through L2, which for 128 weight rows x 64 tokens weighs as much as the weights:
// the token rows of a tile follow the block (16, 32, 48 or 64; hi and lo rows are one N of twice that), and smaller tiles leave
// room for more stages.  Whole prompts with 64-token tiles for all / now: 8 tokens, 8B 4.19 / 3.77 ms; 16 tokens, TinyLlama 1.250 /
// 1.177; 4 tokens, 1B 1.020 / 0.987; 30 tokens, rutenex-1b 1.289 / 1.254.  (Fewer weight rows an item where 128 leave SMs
// idle, 80 or 112: within 1.5 % either way at 64 tokens, not kept: the activations are read the more often.)
// Every wait is bounded; every path, also a failed one, reaches the common exit, which lets copies in flight land
// (bounded) and frees the tensor memory.
constexpr int kUmmaM = 128;
constexpr int kUmmaSubW = kUmmaM * 128;                            // 16 KiB
constexpr int kUmmaMaxStages = 4;                                  // tiles of 16 tokens: 40 KiB a stage
constexpr int kUmmaEpiWarps = 8;                                   // two per tensor-memory lane quarter: 32 tokens each
constexpr int kUmmaThreads = (2 + kUmmaEpiWarps) * 32;
constexpr int kUmmaN = 2 * kPfTile;                                // MMA N: the 64 hi rows and the 64 lo rows of the activation tile
constexpr int kUmmaAccCols = kUmmaN;                               // FP32 columns of one accumulator: W.hi | W.lo
constexpr int kUmmaTmemCols = 2 * kUmmaAccCols;                    // power of two >= 32
// Instruction descriptor: D = F32 (bits 4-5 = 1), A and B of the same 16-bit type (bits 7-9 and 10-12: 0 = FP16,
// 1 = BF16), both K-major (bits 15, 16 = 0), N / 8 in bits 17-22, M / 16 in bits 24-28.
template <typename T>
__host__ __device__ constexpr uint32_t umma_idesc(int n = kUmmaN) {
    return (1u << 4) | (std::is_same<T, __nv_bfloat16>::value ? (1u << 7) | (1u << 10) : 0u) | ((uint32_t)(n >> 3) << 17) |
           ((uint32_t)(kUmmaM >> 4) << 24);
}

// Shared-memory matrix descriptor of a K-major operand tile with the 128-byte swizzle: start address / 16 in bits
// 0-13, leading byte offset (unused for swizzled K-major, set to 1) in bits 16-29, stride between 8-row groups
// (1024 bytes) / 16 in bits 32-45, descriptor version 1 in bits 46-47, layout type 2 (128-byte swizzle) in bits 61-63.
__device__ __forceinline__ uint64_t umma_desc(uint32_t smem_addr) {
    return (uint64_t)((smem_addr & 0x3ffffu) >> 4) | (1ull << 16) | ((uint64_t)(1024 >> 4) << 32) | (1ull << 46) | (2ull << 61);
}
__device__ __forceinline__ void tc_alloc(uint32_t* smem_dst, uint32_t cols) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(smem_dst)), "r"(cols) : "memory");
}
__device__ __forceinline__ void tc_relinquish() {
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tc_dealloc(uint32_t taddr, uint32_t cols) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(cols) : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_commit(uint64_t* bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}
// True in one thread of a converged warp, the same one every time.  The MMA and commit instructions take their operands from
// the warp's uniform registers; behind a branch on the lane number the compiler has to assume several threads.
__device__ __forceinline__ bool elect_one() {
    uint32_t p;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(p));
    return p != 0;
}
__device__ __forceinline__ void tc_mma_f16(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(d_tmem), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
}
// 32 lanes x 32 consecutive 32-bit columns: thread i of the warp receives lane (quarter base + i), columns c .. c+31
__device__ __forceinline__ void tc_ld32(uint32_t taddr, float (&v)[32]) {
    uint32_t r[32];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
        "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
          "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
          "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr)
        : "memory");
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(r[i]);
}

// Epilogue of one thread: weight row `row`, tokens t0 .. t0+31 with the sums v[0..31].  Lanes are consecutive rows,
// so for a fixed token a warp's stores are contiguous; the partner row (row ^ 1) of the rotation and SwiGLU pairs
// is the neighbouring lane.
template <typename T, int EPI>
__device__ __forceinline__ void umma_epilogue(const PrefillGemmArgs& a, int split, int group, int row, int t0, const float (&v)[32],
                                              int lane) {
    const bool row_ok = row < a.n_rows;
    const int nt = min(32, a.n_tokens - t0);  // valid tokens of this half (may be <= 0)
    if constexpr (EPI == kPfResid) {
        if (a.splits > 1) {
            float* p = a.part + ((size_t)split * a.part_tokens + t0) * a.x_pitch + row;
#pragma unroll
            for (int i = 0; i < 32; ++i)
                if (row_ok && i < nt) p[(size_t)i * a.x_pitch] = v[i];
        } else {
            float* p = a.x + (size_t)t0 * a.x_pitch + row;
#pragma unroll
            for (int i0 = 0; i0 < 32; i0 += 8) {  // eight loads in flight: the pair kernel has no registers for more
                float old[8];
#pragma unroll
                for (int i = 0; i < 8; ++i) old[i] = (row_ok && i0 + i < nt) ? p[(size_t)(i0 + i) * a.x_pitch] : 0.f;
#pragma unroll
                for (int i = 0; i < 8; ++i)
                    if (row_ok && i0 + i < nt) p[(size_t)(i0 + i) * a.x_pitch] = old[i] + v[i0 + i];  // x += W.xb (src/model.cpp:232, 239)
            }
        }
    } else if constexpr (EPI == kPfStore) {
        float* p = a.out + ((size_t)split * a.part_tokens + t0) * a.out_pitch + row;
#pragma unroll
        for (int i = 0; i < 32; ++i)
            if (row_ok && i < nt) p[(size_t)i * a.out_pitch] = v[i];
    } else if constexpr (EPI == kPfLatentQuery) {
        __half* p = a.lat_query + ((size_t)t0 * a.groups + group) * a.lat_pitch + row;
#pragma unroll
        for (int i = 0; i < 32; ++i)
            if (row_ok && i < nt) p[(size_t)i * a.groups * a.lat_pitch] = __float2half_rn(v[i]);
    } else if constexpr (EPI == kPfLatentValue) {
        T* p = reinterpret_cast<T*>(a.hb) + (size_t)t0 * a.hb_pitch + (size_t)group * a.n_valid + row;
        const float* gate = a.gate + (size_t)t0 * a.groups + group;
        float gt[32];  // requested together: one round trip, not one per token
#pragma unroll
        for (int i = 0; i < 32; ++i) gt[i] = i < nt ? gate[(size_t)i * a.groups] : 0.f;
#pragma unroll
        for (int i = 0; i < 32; ++i)
            if (row < a.n_valid && i < nt) {
                T hi, lo;
                split_pair(v[i] * gt[i], hi, lo);
                p[(size_t)i * a.hb_pitch] = hi;
                p[(size_t)(a.cap + i) * a.hb_pitch] = lo;
            }
    } else if constexpr (EPI == kPfSwiglu) {
        // rows interleaved (gate_i, up_i): the even lane finishes tokens 0..15 of the pair, the odd lane tokens 16..31;
        // each sends the partner the half it does not finish itself.  hb = (h1*sigmoid(h1))*h3 (src/ops.cpp:78-87)
        // with the fast exponential and division (relative error ~1e-6, far below the 16-bit weights' own rounding), or
        // the tanh form of GELU in place of h1*sigmoid(h1).
        const bool even = (lane & 1) == 0;
        T* hb = reinterpret_cast<T*>(a.hb) + (size_t)(t0 + (even ? 0 : 16)) * a.hb_pitch + (row >> 1);
        const int nt_mine = nt - (even ? 0 : 16);
#pragma unroll
        for (int k = 0; k < 16; ++k) {
            const float keep = even ? v[k] : v[k + 16], send = even ? v[k + 16] : v[k];
            const float recv = __shfl_xor_sync(0xffffffffu, send, 1);
            const float g = even ? keep : recv, u = even ? recv : keep;
            const float r = __fdividef(g, 1.0f + __expf(-act_gate_arg(a.act, g))) * u;
            T hi, lo;
            split_pair(r, hi, lo);
            if (row_ok && k < nt_mine) {
                hb[(size_t)k * a.hb_pitch] = hi;
                hb[(size_t)(a.cap + k) * a.hb_pitch] = lo;
            }
        }
    } else {  // kPfQkv: partial sums (also of one range: the rotation's table and the cache rows want another layout), finished
              // by prefill_qkv_finish_kernel
        float* p = a.part + ((size_t)split * a.part_tokens + t0) * a.n_rows + row;
#pragma unroll
        for (int i = 0; i < 32; ++i)
            if (row_ok && i < nt) p[(size_t)i * a.n_rows] = v[i];
    }
}

#ifdef LPP_TIMING_AIDS
// timing aid: global-timer stamps [cta][slot] of the last gate|up launch
__device__ unsigned long long g_pf_trace[160][48];
#define PF_STAMP(k)                                                                      \
    do {                                                                                 \
        if (EPI == kPfSwiglu && (k) < 48) {                                              \
            unsigned long long t_;                                                       \
            asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t_));                       \
            g_pf_trace[blockIdx.x][k] = t_;                                              \
        }                                                                                \
    } while (0)
#else
#define PF_STAMP(k) \
    do {            \
    } while (0)
#endif

// BOX: token rows of an activation tile, 0 = a.box_tokens (whole tiles of 64 keep their sizes as constants).
template <typename T, int EPI, int BOX>
static __global__ void __launch_bounds__(kUmmaThreads, 1) prefill_gemm_umma_kernel(const __grid_constant__ CUtensorMap w_map,
                                                                                   const __grid_constant__ CUtensorMap x_map,
                                                                                   const PrefillGemmArgs a) {
    constexpr int kMaxStages = kUmmaMaxStages;
    const int box_tokens = BOX ? BOX : a.box_tokens, kSubX = box_tokens * 128, kStage = 2 * kUmmaSubW + 4 * kSubX;
    const int kStages = min(kMaxStages, kPfRingBytes / kStage);
    extern __shared__ __align__(128) unsigned char smem[];
    uint64_t* full = reinterpret_cast<uint64_t*>(smem);  // [kMaxStages]
    uint64_t* empty = full + kMaxStages;                 // [kMaxStages]
    uint64_t* acc_full = empty + kMaxStages;             // [2]
    uint64_t* acc_empty = acc_full + 2;                  // [2]
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_empty + 2);
    int* s_fail = reinterpret_cast<int*>(tmem_slot + 1);  // set by a role whose wait ran out
    const uint32_t ring = (smem_u32(smem) + 1024u + 1023u) & ~1023u;
    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
    const int unit = blockIdx.x, n_units = gridDim.x;
    const int group_tiles = (a.n_rows + kUmmaM - 1) / kUmmaM;  // row tiles of one matrix
    const int n_tiles = group_tiles * max(1, a.groups);        // items along the rows
    const int n_kc = (a.K + kPfKc - 1) / kPfKc;
    const int S = a.splits, tok_tiles = (a.n_tokens + kPfTile - 1) / kPfTile;
    const int n_items = n_tiles * tok_tiles * S;  // item = (row tile, token tile, K range)
    pdl_launch_dependents();
    if (tid == 0) {
        *s_fail = 0;
        for (int i = 0; i < kStages; ++i) {
            mbar_init(&full[i], 1);
            mbar_init(&empty[i], 1);
        }
        for (int i = 0; i < 2; ++i) {
            mbar_init(&acc_full[i], 1);
            mbar_init(&acc_empty[i], kUmmaEpiWarps);
        }
        mbar_fence_init();
    }
    if (warp == 1) {
        tc_alloc(tmem_slot, kUmmaTmemCols);
        tc_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *reinterpret_cast<volatile uint32_t*>(tmem_slot);

    if (warp == 0) {
        // ---------------- producer
        if (lane == 0) {
            PF_STAMP(0);
            // The weight sub-tiles of the first ring pass do not depend on the previous kernel: they are requested
            // before the dependency wait, the activation sub-tiles of the same stages right after it.
            int slot = 0, pass = 0;
            bool ok = true, waited = false;
            int early = 0;  // stages whose weights are already in flight
            // one copy per operand and stage: both 64-input weight sub-tiles / the four activation sub-tiles (hi, lo)
            auto load_w = [&](uint32_t dst, int kc, int wrow, int sl) { tma_load_3d(dst, &w_map, 0, wrow, 2 * kc, smem_u32(&full[sl])); };
            auto load_x = [&](uint32_t dst, int tok0, int piece, int sl) { tma_load_4d(dst, &x_map, 0, tok0, 0, piece, smem_u32(&full[sl])); };
            auto expect = [&](int sl) { mbar_arrive_expect_tx(&full[sl], kStage); };
            for (int item = unit; item < n_items && ok; item += n_units) {
                const int unsplit = item / S, split = item - unsplit * S, tile = unsplit / tok_tiles;
                const int tok0 = (unsplit - tile * tok_tiles) * kPfTile;
                const int kc0 = (split * n_kc) / S, kc1 = ((split + 1) * n_kc) / S;
                const int group = tile / group_tiles, piece0 = group * a.group_pieces;
                const int wrow = a.row0 + group * a.group_stride + (tile - group * group_tiles) * kUmmaM;
                if (!waited) {
                    early = min(kc1 - kc0, kStages);
                    for (int i = 0; i < early; ++i) {
                        const uint32_t dst = ring + (uint32_t)i * kStage;
                        expect(i);
                        load_w(dst, kc0 + i, wrow, i);
                    }
                    pdl_wait();
                    PF_STAMP(1);
                    waited = true;
                }
                for (int kc = kc0; kc < kc1; ++kc) {
                    const uint32_t dst = ring + (uint32_t)slot * kStage;
                    if (early > 0) {
                        --early;  // first pass of the first item: only the activations are missing
                    } else {
                        if (pass > 0 && !mbar_wait_bounded(&empty[slot], (uint32_t)(pass - 1) & 1u, a.st)) {
                            *s_fail = 1;
                            ok = false;
                            break;
                        }
                        expect(slot);
                        load_w(dst, kc, wrow, slot);
                    }
                    PF_STAMP(2 + kc - kc0);
                    load_x(dst + 2 * kUmmaSubW, tok0, piece0 + 2 * kc, slot);
                    if (++slot == kStages) {
                        slot = 0;
                        ++pass;
                    }
                }
            }
            if (!waited) pdl_wait();
        }
    } else if (warp == 1) {
        // ---------------- MMA issue
        {
            const uint32_t idesc = umma_idesc<T>(2 * box_tokens);
            int slot = 0;
            uint32_t par = 0;
            bool ok = true;
            int it = 0;
            for (int item = unit; item < n_items && ok; item += n_units, ++it) {
                const int split = item % S;
                const int kc0 = (split * n_kc) / S, kc1 = ((split + 1) * n_kc) / S;
                const int b = it & 1, use = it >> 1;
                if (use > 0 && !mbar_wait_bounded(&acc_empty[b], (uint32_t)(use - 1) & 1u, a.st)) {
                    *s_fail = 1;
                    break;
                }
                tc_fence_after();
                const uint32_t d_tmem = tmem + (uint32_t)(b * kUmmaAccCols);
                for (int kc = kc0; kc < kc1; ++kc) {
                    if (!mbar_wait_bounded(&full[slot], par, a.st)) {
                        *s_fail = 1;
                        ok = false;
                        break;
                    }
                    tc_fence_after();
                    PF_STAMP(18 + kc - kc0);
                    const uint32_t st = ring + (uint32_t)slot * kStage;
                    if (elect_one()) {
#pragma unroll
                        for (int sub = 0; sub < 2; ++sub) {
                            // the activation sub-tile holds the hi rows followed by the lo rows: one MMA covers both
                            const uint32_t wt = st + sub * kUmmaSubW, xt = st + 2 * kUmmaSubW + sub * 2 * kSubX;
#pragma unroll
                            for (int ks = 0; ks < 4; ++ks) {  // 16 inputs = 32 bytes along the swizzled row per step
                                const uint32_t acc = (kc > kc0 || sub > 0 || ks > 0) ? 1u : 0u;
                                tc_mma_f16(d_tmem, umma_desc(wt + ks * 32), umma_desc(xt + ks * 32), idesc, acc);
                            }
                        }
                        tc_commit(&empty[slot]);  // arrives once the MMAs issued so far have read this stage
                    }
                    __syncwarp();
                    if (++slot == kStages) {
                        slot = 0;
                        par ^= 1u;
                    }
                }
                if (ok && elect_one()) tc_commit(&acc_full[b]);
                __syncwarp();
            }
        }
    } else {
        // ---------------- epilogue: this warp owns tensor-memory lanes 32 * (warp % 4) .. + 31 = rows of the tile,
        // and the first or second 32 columns (tokens) of the accumulator
        const int quarter = warp & 3, half = (warp - 2) >> 2;
        int it = 0;
        for (int item = unit; item < n_items; item += n_units, ++it) {
            const int unsplit = item / S, split = item - unsplit * S, tile = unsplit / tok_tiles;
            const int b = it & 1, use = it >> 1;
            if (!__all_sync(0xffffffffu, mbar_wait_bounded(&acc_full[b], (uint32_t)use & 1u, a.st))) {
                *s_fail = 1;
                break;
            }
            tc_fence_after();
            if (tid == 64) PF_STAMP(34);
            float v[32], vlo[32];
            const uint32_t taddr = tmem + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(b * kUmmaAccCols);
            tc_ld32(taddr + half * 32, v);                     // W.hi of this warp's 32 tokens
            tc_ld32(taddr + box_tokens + half * 32, vlo);  // W.lo
#pragma unroll
            for (int i = 0; i < 32; ++i) v[i] += vlo[i];
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&acc_empty[b]);
            if (tid == 64) PF_STAMP(35);
            const int group = tile / group_tiles;
            umma_epilogue<T, EPI>(a, split, group, (tile - group * group_tiles) * kUmmaM + quarter * 32 + lane,
                                  (unsplit - tile * tok_tiles) * kPfTile + half * 32, v, lane);
            if (tid == 64) PF_STAMP(36);
        }
    }
    // ---------------- common exit
    __syncwarp();
    tc_fence_before();
    __syncthreads();
    // A wait that ran out has set the status word (mbar_wait_bounded) and this CTA's flag.  Copies may then still be in
    // flight towards its shared memory: give them a bounded time to land before the CTA leaves (a tile copy takes a
    // few microseconds; nobody reads the tiles any more).
    if (tid == 0 && *reinterpret_cast<volatile int*>(s_fail) != 0) {
        const long long t0 = clock64();
        while (clock64() - t0 < (1 << 17)) __nanosleep(1000);
    }
    __syncthreads();
    if (warp == 1) tc_dealloc(tmem, kUmmaTmemCols);
}

// N tokens' sums of the partial sums of rows row .. row + 3, tokens t0 .. (clamped to the block: no branches, so the loads of
// a range of K are in flight together), in range order.
template <int N>
__device__ __forceinline__ void prefill_sums(const float* part, int part_tokens, int n_rows, int splits, int n_tokens, int t0, int row, float4 (&v)[N]) {
    const float4* p[N];
#pragma unroll
    for (int i = 0; i < N; ++i) {
        p[i] = reinterpret_cast<const float4*>(part + (size_t)min(max(t0 + i, 0), n_tokens - 1) * n_rows + row);
        v[i] = *p[i];
    }
#pragma unroll 2
    for (int s = 1; s < splits; ++s)
#pragma unroll
        for (int i = 0; i < N; ++i) {
            const float4 w = p[i][(size_t)s * part_tokens * n_rows / 4];
            v[i].x += w.x; v[i].y += w.y; v[i].z += w.z; v[i].w += w.w;
        }
}

// Finishes a QKV GEMM: adds the partial sums of the rows in range order and applies the QKV epilogue (rotation of q and k
// pairs, q -> FP32 rows, k/v -> cache rows at the reference index).  A thread takes four rows (two pairs; there are always whole
// quads: q rows come in multiples of 64, k and v rows are even and equally many) of kFinishTokens tokens, so that 64 bytes per
// range of K are in flight and the rotation's table is there before the sums are.  Bound by the traffic through L2.  One pair of
// one token per thread took 17 us for 1023 tokens of 3072 rows and 40 us for 1000 tokens of 6144 rows (one range).  Few tokens are
// bound by the latency of their up to eight ranges instead: TOKENS 1, all ranges in flight.  Whole prompts with four tokens a thread /
// with one: 47 tokens of the TinyLlama shape 1169 / 1116 us, 33 of the Llama-3.2-1B shape 1031 / 1000, 64 of it 1042 / 1002.
// grid: (ceil(tokens / TOKENS), ceil(rows / 1024)).
constexpr int kFinishTokens = 4;
template <int TOKENS>
static __global__ void __launch_bounds__(256) prefill_qkv_finish_kernel(const PrefillGemmArgs a) {
    pdl_launch_dependents();
    const int t0 = blockIdx.x * TOKENS, row = 4 * ((int)blockIdx.y * 256 + (int)threadIdx.x), hs = a.head_size;
    const bool mine = row < a.n_rows;
    float2 cs[TOKENS][2];
    size_t at[2] = {0, 0};  // in the cache: position 0 of the pair's row
    const bool is_q = row < a.q_rows;
    if (mine) {  // constants: ahead of the dependency wait
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            const int r = row + 2 * j;
            const bool turned = r < a.q_rows + a.kv_rows;
            const int rr = is_q ? r : r - a.q_rows - (turned ? 0 : a.kv_rows);  // within q, k or v
            const int h = rr / hs, off = rr - h * hs;
            at[j] = (size_t)h * ((size_t)a.seq_len * hs) + off;  // h*(seq_len*hs) + pos*hs + off (src/scatter_kv.cu:15-16)
#pragma unroll
            for (int i = 0; i < TOKENS; ++i) {
                const int pos = a.start_pos + t0 + i;
                // adjacent-pair rotation with the table entry for (pos, (row % hs)/2) (src/ops.cpp:34-54)
                cs[i][j] = turned && pos >= 0 && pos < a.seq_len ? __ldg(a.rope + (size_t)pos * (hs >> 1) + (off >> 1)) : make_float2(1.f, 0.f);
            }
        }
    }
    pdl_wait();
    if (!mine) return;
    float4 v[TOKENS];
    if constexpr (TOKENS == 1) {
        float4 p[kPfMaxSplits];
        const float4* at0 = reinterpret_cast<const float4*>(a.part + (size_t)t0 * a.n_rows + row);
#pragma unroll
        for (int s = 0; s < kPfMaxSplits; ++s)
            if (s < a.splits) p[s] = at0[(size_t)s * a.part_tokens * a.n_rows / 4];
        v[0] = p[0];
#pragma unroll
        for (int s = 1; s < kPfMaxSplits; ++s)  // in range order
            if (s < a.splits) {
                v[0].x += p[s].x; v[0].y += p[s].y; v[0].z += p[s].z; v[0].w += p[s].w;
            }
    } else {
        prefill_sums<TOKENS>(a.part, a.part_tokens, a.n_rows, a.splits, a.n_tokens, t0, row, v);
    }
#pragma unroll
    for (int i = 0; i < TOKENS; ++i) {
        const int t = t0 + i, pos = a.start_pos + t;
        if (t >= a.n_tokens) break;
        if (pos < 0 || pos >= a.seq_len) {
            atomicOr(&a.st->status, kStatusBadPos);
            break;
        }
        auto turn = [&](float x, float y, int j) -> float2 {
            if (row + 2 * j >= a.q_rows + a.kv_rows) return make_float2(x, y);  // v
            const float2 c = cs[i][j];
            return make_float2(__fsub_rn(__fmul_rn(x, c.x), __fmul_rn(y, c.y)), __fadd_rn(__fmul_rn(x, c.y), __fmul_rn(y, c.x)));
        };
        const float2 p0 = turn(v[i].x, v[i].y, 0), p1 = turn(v[i].z, v[i].w, 1);
        if (is_q) {
            *reinterpret_cast<float4*>(a.q + (size_t)t * a.q_rows + row) = make_float4(p0.x, p0.y, p1.x, p1.y);
        } else {
            auto put = [&](float2 p, int j) {
                __half* dst = reinterpret_cast<__half*>(row + 2 * j < a.q_rows + a.kv_rows ? a.k_cache : a.v_cache) + at[j] + (size_t)pos * hs;
                *reinterpret_cast<uint32_t*>(dst) = pack_half2(p.x, p.y);
            };
            put(p0, 0);
            put(p1, 1);
        }
    }
}

// Rows of the residual stream -> normalised rows (hi + lo MMA operands): RMSNorm, or LayerNorm when a bias is given.
// Layer 0 takes the embedding rows of the prompt tokens, times their factor, and also writes them out as the FP32 residual
// stream.  With a row list, block i takes row rows[i] (the positions whose logits are wanted).  D is the row pitch; the
// statistics cover the first norm_n inputs, the rest is zero padding with zero weights.  grid: rows; prefill_norm_threads
// threads.  Without partial sums there are many rows: a thread has four pieces of four floats, few enough threads and registers
// that the rows of a block are all resident at once (one or two pieces on 512 threads, two or three rows an SM: 13 us for 1023
// rows of 2048 and 22 us for 1000 of 4096; now 6 and 11).  With partial sums of a few rows the latency counts: one
// or two pieces a thread, all ranges in flight (47 rows of 2048 with 8 ranges: 4.5 us, four pieces a thread 8.3), one row an SM.  Many
// rows become waves that way: half the threads and registers for four rows an SM instead (64 registers, 88 bytes of spills; 517 rows of 2048 with partial sums: 12.3 -> 7.9
// us), from 384 rows of 512 threads on (whole prompts of the TinyLlama shape, few / many rows' kernel: 200 tokens 1878 / 1946 us, 350
// 2127 / 2169, 400 2554 / 2501; kolatar-300m, rows of 256 threads: 400 tokens 2739 / 2788, 900 4080 / 3938).
enum PfNormMode : int { kNormPlain = 0, kNormFewParts = 1, kNormManyParts = 2 };
constexpr int kPfNormManyThreads = 384 * 512;
template <int MODE>
struct PfNorm {
    static constexpr int kPer = MODE == kNormFewParts ? 2 : 4, kMaxThreads = MODE == kNormFewParts ? 512 : 256;
    static constexpr int kResident = MODE == kNormPlain ? 5 : MODE == kNormManyParts ? 4 : 1;
};
static int prefill_norm_threads(int D, int mode) {
    const int per = mode == kNormPlain ? PfNorm<kNormPlain>::kPer : mode == kNormManyParts ? 2 : 1, pieces = (D / 4 + per - 1) / per;
    return std::min(mode == kNormFewParts ? PfNorm<kNormFewParts>::kMaxThreads : PfNorm<kNormPlain>::kMaxThreads, std::max(64, (pieces + 31) / 32 * 32));
}
struct PrefillNormArgs {
    float* x;            // [tokens][D]
    const int* tokens;   // with emb
    const void* emb;     // [vocab][D], nullptr = the rows of x
    float emb_scale;     // factor of the embedding rows
    const float* add;    // [D] added to every row first (nullptr = nothing)
    int vocab;
    const int* rows;     // nullptr = block i takes row i
    const float* norm_w;
    const float* norm_b; // nullptr = RMSNorm
    float norm_eps;
    int norm_n;
    void* out;           // [2 planes][cap][D]
    int D;
    const float* part;   // [splits][part_tokens][D], added to x in order when splits > 1
    int cap, part_tokens;
    int splits;
    StepState* st;
};
__device__ __forceinline__ float norm_block_sum(float v, float* red, int tid) {
    v = warp_sum(v);
    if ((tid & 31) == 0) red[tid >> 5] = v;
    __syncthreads();
    return warp_sum((tid & 31) < (int)(blockDim.x >> 5) ? red[tid & 31] : 0.f);
}
// Partial sums, where there are any, are added first.  Only the weights (emb, norm_w, norm_b) are loaded as read-only data: a load of what
// the preceding kernel produced must not become an invariant one, which the compiler may move above the dependency wait.
template <typename T, int MODE>
static __global__ void __launch_bounds__(PfNorm<MODE>::kMaxThreads, PfNorm<MODE>::kResident) prefill_norm_kernel(const PrefillNormArgs a) {
    constexpr int kPfNormPer = PfNorm<MODE>::kPer;
    constexpr bool PARTS = MODE != kNormPlain;
    __shared__ float red[2][PfNorm<MODE>::kMaxThreads / 32];
    pdl_launch_dependents();
    const int tid = threadIdx.x, D = a.D, nt = blockDim.x;
    const int nv4 = D >> 2;  // D is a multiple of 8
    float4 v[kPfNormPer];
    pdl_wait();
    const int t = a.rows ? *reinterpret_cast<const volatile int*>(a.rows + blockIdx.x) : (int)blockIdx.x;
    float4* xr = reinterpret_cast<float4*>(a.x + (size_t)t * D);
    int tok = 0;
    if (a.emb) {
        tok = *reinterpret_cast<const volatile int*>(a.tokens + t);
        if (tok < 0 || tok >= a.vocab) {
            if (tid == 0) atomicOr(&a.st->status, kStatusBadToken);
            tok = 0;
        }
    }
    auto load = [&](int i) -> float4 {  // the embedding, or the residual stream
        if (!a.emb) return xr[i];
        const uint2 h = __ldg(reinterpret_cast<const uint2*>(reinterpret_cast<const T*>(a.emb) + (size_t)tok * D + 4 * (size_t)i));
        const float2 lo = unpack2<T>(h.x), hi = unpack2<T>(h.y);
        return make_float4(lo.x * a.emb_scale, lo.y * a.emb_scale, hi.x * a.emb_scale, hi.y * a.emb_scale);
    };
    auto part = [&](int s, int i) -> float4 { return reinterpret_cast<const float4*>(a.part + ((size_t)s * a.part_tokens + t) * D)[i]; };
    auto plus = [](float4& x, const float4& y) { x.x += y.x; x.y += y.y; x.z += y.z; x.w += y.w; };
    const bool store = a.emb || a.add || PARTS;  // the residual stream as the next residual GEMM reads it
    const bool ln = a.norm_b != nullptr;
    const float n = (float)a.norm_n;
    float ss = 0.f;  // RMSNorm: sum of squares; LayerNorm: sum
    auto first = [&](int i, float4& x) {
        if (a.add) plus(x, __ldg(reinterpret_cast<const float4*>(a.add) + i));
        if (store) xr[i] = x;
        ss = ln ? ss + ((x.x + x.y) + (x.z + x.w)) : fmaf(x.x, x.x, fmaf(x.y, x.y, fmaf(x.z, x.z, fmaf(x.w, x.w, ss))));
    };
#pragma unroll
    for (int k = 0; k < kPfNormPer; ++k)
        if (tid + k * nt < nv4) v[k] = load(tid + k * nt);
    if constexpr (PARTS) {
#pragma unroll
        for (int k = 0; k < kPfNormPer; ++k) {
            if (tid + k * nt >= nv4) continue;
            float4 p[kPfMaxSplits];
#pragma unroll
            for (int s = 0; s < kPfMaxSplits; ++s)
                if (s < a.splits) p[s] = part(s, tid + k * nt);
#pragma unroll
            for (int s = 0; s < kPfMaxSplits; ++s)  // in range order
                if (s < a.splits) plus(v[k], p[s]);
        }
    }
#pragma unroll
    for (int k = 0; k < kPfNormPer; ++k)
        if (tid + k * nt < nv4) first(tid + k * nt, v[k]);
    // rows wider than what the threads keep: the rest without register caching
    for (int i = tid + kPfNormPer * nt; i < nv4; i += nt) {
        float4 x = load(i);
        if constexpr (PARTS)
            for (int s = 0; s < a.splits; ++s) plus(x, part(s, i));
        first(i, x);
    }
    float tot = norm_block_sum(ss, red[0], tid), mean = 0.f;
    if (ln) {
        mean = __fdiv_rn(tot, n);
        float q = 0.f;
        auto second = [&](int i, const float4& x) {
            const float d[4] = {x.x - mean, x.y - mean, x.z - mean, x.w - mean};
#pragma unroll
            for (int c = 0; c < 4; ++c)
                if (4 * i + c < a.norm_n) q = fmaf(d[c], d[c], q);
        };
#pragma unroll
        for (int k = 0; k < kPfNormPer; ++k)
            if (tid + k * nt < nv4) second(tid + k * nt, v[k]);
        for (int i = tid + kPfNormPer * nt; i < nv4; i += nt) second(i, xr[i]);
        tot = norm_block_sum(q, red[1], tid);
    }
    const float scale = __fdiv_rn(1.0f, __fsqrt_rn(__fadd_rn(__fdiv_rn(tot, n), a.norm_eps)));
    T* out = reinterpret_cast<T*>(a.out) + (size_t)blockIdx.x * D;
    auto emit = [&](int i, const float4& xv) {
        const float4 wv = __ldg(reinterpret_cast<const float4*>(a.norm_w) + i);
        float y[4];
        if (ln) {
            const float4 b = __ldg(reinterpret_cast<const float4*>(a.norm_b) + i);
            y[0] = fmaf(__fmul_rn(xv.x - mean, scale), wv.x, b.x);
            y[1] = fmaf(__fmul_rn(xv.y - mean, scale), wv.y, b.y);
            y[2] = fmaf(__fmul_rn(xv.z - mean, scale), wv.z, b.z);
            y[3] = fmaf(__fmul_rn(xv.w - mean, scale), wv.w, b.w);
        } else {
            y[0] = __fmul_rn(__fmul_rn(xv.x, scale), wv.x);
            y[1] = __fmul_rn(__fmul_rn(xv.y, scale), wv.y);
            y[2] = __fmul_rn(__fmul_rn(xv.z, scale), wv.z);
            y[3] = __fmul_rn(__fmul_rn(xv.w, scale), wv.w);
        }
        __align__(8) T hi[4], lo[4];
#pragma unroll
        for (int c = 0; c < 4; ++c) split_pair(y[c], hi[c], lo[c]);
        *reinterpret_cast<uint2*>(out + 4 * (size_t)i) = *reinterpret_cast<const uint2*>(hi);
        *reinterpret_cast<uint2*>(out + (size_t)a.cap * D + 4 * (size_t)i) = *reinterpret_cast<const uint2*>(lo);
    };
#pragma unroll
    for (int k = 0; k < kPfNormPer; ++k)
        if (tid + k * nt < nv4) emit(tid + k * nt, v[k]);
    for (int i = tid + kPfNormPer * nt; i < nv4; i += nt) emit(i, xr[i]);  // re-read what this thread wrote
}

// Causal attention of the prompt block: query token t (position start_pos + t) over cache rows 0..start_pos + t,
// scores scaled after the dot product, softmax, weighted sum of V (src/model.cpp:178-199); one warp per query head,
// lanes over positions with an online softmax, FP32 throughout.  grid: (tokens, kv heads), block: gqa warps.
static __global__ void __launch_bounds__(256) prefill_attention_kernel(const float* q, const __half* k_cache, const __half* v_cache,
                                                                       __half* out, int n_tokens, int start_pos, int seq_len,
                                                                       int head_size, int gqa, int q_rows, int cap) {
    extern __shared__ float sm[];  // [gqa][head_size] query rows, then [gqa warps][32 lanes][head_size] is too much: V sums go through registers
    pdl_launch_dependents();
    pdl_wait();
    const int t = blockIdx.x, kvh = blockIdx.y;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int h = kvh * gqa + warp;
    const int hs = head_size;
    float* qs = sm + warp * hs;
    for (int d = lane; d < hs; d += 32) qs[d] = q[(size_t)t * q_rows + (size_t)h * hs + d];
    __syncwarp();
    const int T = start_pos + t + 1;
    const float scale = __fdiv_rn(1.0f, __fsqrt_rn((float)hs));
    const __half* kb = k_cache + (size_t)kvh * seq_len * hs;
    const __half* vb = v_cache + (size_t)kvh * seq_len * hs;
    // one position's score: the K row in 16-byte pieces, all requested before the first is used
    auto score = [&](int p) -> float {
        const uint4* kr = reinterpret_cast<const uint4*>(kb + (size_t)p * hs);
        float s = 0.f;
        for (int d0 = 0; d0 < hs / 8; d0 += 8) {
            uint4 u[8];
#pragma unroll
            for (int i = 0; i < 8; ++i)
                if (d0 + i < hs / 8) u[i] = __ldcg(kr + d0 + i);
#pragma unroll
            for (int i = 0; i < 8; ++i)
                if (d0 + i < hs / 8) {
                    const float* qq = qs + 8 * (d0 + i);
                    float2 f;
                    f = half2_bits_to_float2(u[i].x); s = fmaf(qq[0], f.x, s); s = fmaf(qq[1], f.y, s);
                    f = half2_bits_to_float2(u[i].y); s = fmaf(qq[2], f.x, s); s = fmaf(qq[3], f.y, s);
                    f = half2_bits_to_float2(u[i].z); s = fmaf(qq[4], f.x, s); s = fmaf(qq[5], f.y, s);
                    f = half2_bits_to_float2(u[i].w); s = fmaf(qq[6], f.x, s); s = fmaf(qq[7], f.y, s);
                }
        }
        return s * scale;
    };
    // pass 1: scores of this lane's positions, maximum
    float m = -INFINITY;
    for (int p = lane; p < T; p += 32) m = fmaxf(m, score(p));
    m = warp_max(m);
    // pass 2: every lane owns head dims lane, lane + 32, ...; positions in order, eight V rows in flight
    float l = 0.f;
    float acc[4] = {0.f, 0.f, 0.f, 0.f};  // head_size <= 128
    for (int p0 = 0; p0 < T; p0 += 32) {
        const int p = p0 + lane;
        const float e = (p < T) ? __expf(score(p) - m) : 0.f;
        l += e;
        const int cnt = min(32, T - p0);
        for (int i0 = 0; i0 < cnt; i0 += 8) {
            __half vv[8][4];
#pragma unroll
            for (int i = 0; i < 8; ++i)
#pragma unroll
                for (int c = 0; c < 4; ++c)
                    if (i0 + i < cnt && lane + 32 * c < hs) vv[i][c] = vb[(size_t)(p0 + i0 + i) * hs + lane + 32 * c];
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const float ei = __shfl_sync(0xffffffffu, e, (i0 + i) & 31);
#pragma unroll
                for (int c = 0; c < 4; ++c)
                    if (i0 + i < cnt && lane + 32 * c < hs) acc[c] = fmaf(ei, __half2float(vv[i][c]), acc[c]);
            }
        }
    }
    l = warp_sum(l);
#pragma unroll
    for (int c = 0; c < 4; ++c)
        if (lane + 32 * c < hs) {
            __half hi, lo;
            split_half(__fdiv_rn(acc[c], l), hi, lo);
            out[(size_t)t * q_rows + (size_t)h * hs + lane + 32 * c] = hi;
            out[(size_t)(cap + t) * q_rows + (size_t)h * hs + lane + 32 * c] = lo;
        }
}

__device__ __forceinline__ void ldmatrix_x4_trans(uint32_t (&r)[4], uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(addr));
}

}  // namespace lpp

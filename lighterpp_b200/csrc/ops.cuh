// Standalone operator kernels behind the reference's per-op host wrappers (src/kernels.cuh:24-36).
// The decode step itself does not launch these -- it uses the fused kernels in gemv.cuh,
// attention.cuh and sampler.cuh -- but host code that calls the operators one by one (the
// reference's own runtests.cpp, or a partially ported model.cpp) gets the same results from them.
// All are element-wise or small reductions over L2-resident activations, a few microseconds each, so the hand-over from one
// to the next weighs as much as they do: they are launched with programmatic dependent launch (launch_op in ops_api.cu),
// wait for the kernel before them first thing and let the next one launch at once.
#pragma once
#include "common.cuh"

namespace lpp {

// First statement of every operator kernel: nothing of the kernel before may be touched ahead of it.
__device__ __forceinline__ void op_begin() {
    pdl_launch_dependents();
    pdl_wait();
}

// src/matmul.cu:150-161
static __global__ void convert_f32_to_f16_kernel(__half* dst, const float* src, long long n) {
    op_begin();
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const long long stride = (long long)gridDim.x * blockDim.x;
    for (long long k = i; k < n; k += stride) dst[k] = __float2half_rn(src[k]);
}
static __global__ void convert_f16_to_f32_kernel(float* dst, const __half* src, long long n) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const long long stride = (long long)gridDim.x * blockDim.x;
    for (long long k = i; k < n; k += stride) dst[k] = __half2float(src[k]);
}

// Strided 2-D repack with optional type conversion: dst[r*dst_row + c*dst_col] = source element (r, c), where source
// row r starts at src + ((r / group) * group_stride + r % group) * src_pitch (strides in elements).  Used to build the
// engine's fused weight layouts from full tensors (row and column slices, gate/up interleave, per-head sections,
// transposes).
template <typename DT, typename ST>
static __global__ void repack_kernel(DT* dst, long long dst_row, long long dst_col, const ST* src, long long src_pitch, int group,
                                     long long group_stride, int rows, int cols) {
    const long long total = (long long)rows * cols;
    const long long stride = (long long)gridDim.x * blockDim.x;
    for (long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x; k < total; k += stride) {
        const long long r = k / cols, c = k % cols;
        const ST v = src[((r / group) * group_stride + r % group) * src_pitch + c];
        DT o;
        if constexpr (std::is_same<DT, ST>::value)
            o = v;
        else
            o = from_float<DT>(to_float(v));
        dst[r * dst_row + c * dst_col] = o;
    }
}

// src/RMSNorm.cu:11-71 -- one CTA; out = x * rsqrt(mean(x^2) + 1e-5) * w (src/ops.cpp:20-32).  Bound by the latency of its
// two passes over the row: 1024 threads, the first kOpNormKeep values of each stay in registers and the weights are fetched
// together with them.
constexpr int kOpNormThreads = 1024, kOpNormKeep = 8;
static __global__ void __launch_bounds__(kOpNormThreads) rmsnorm_kernel(float* out, const float* x, const float* w, int n) {
    __shared__ float red[kOpNormThreads / 32];
    op_begin();
    const int tid = threadIdx.x;
    float v[kOpNormKeep], wv[kOpNormKeep];
#pragma unroll
    for (int k = 0; k < kOpNormKeep; ++k) {
        const int i = tid + k * kOpNormThreads;
        v[k] = i < n ? x[i] : 0.f;
        wv[k] = i < n ? w[i] : 0.f;
    }
    float ss = 0.f;
#pragma unroll
    for (int k = 0; k < kOpNormKeep; ++k) ss = fmaf(v[k], v[k], ss);
    for (int i = tid + kOpNormKeep * kOpNormThreads; i < n; i += kOpNormThreads) ss = fmaf(x[i], x[i], ss);
    ss = warp_sum(ss);
    if ((tid & 31) == 0) red[tid >> 5] = ss;
    __syncthreads();
    const float tot = warp_sum(red[tid & 31]);
    const float scale = __fdiv_rn(1.0f, __fsqrt_rn(__fadd_rn(__fdiv_rn(tot, (float)n), 1e-5f)));
#pragma unroll
    for (int k = 0; k < kOpNormKeep; ++k) {
        const int i = tid + k * kOpNormThreads;
        if (i < n) out[i] = __fmul_rn(__fmul_rn(v[k], scale), wv[k]);
    }
    for (int i = tid + kOpNormKeep * kOpNormThreads; i < n; i += kOpNormThreads) out[i] = __fmul_rn(__fmul_rn(x[i], scale), w[i]);
}

// (cos, sin) of pos / base^((2j)/hs) with the device's accurate powf/cosf/sinf.  The step path uses
// a host-built table instead (bit-identical to libm); this is for the stand-alone wrapper only.
__device__ __forceinline__ float2 rope_cos_sin(int pos, int j, int head_size, float rope_base) {
    const float freq = __fdiv_rn(1.0f, powf(rope_base, (float)(2 * j) / (float)head_size));
    const float val = (float)pos * freq;
    return make_float2(cosf(val), sinf(val));
}

// src/rope.cu:7-38 (in place, adjacent pairs, k rotated for i < kv_dim)
static __global__ void rope_kernel(float* q, float* k, int pos, int dim, int kv_dim, int head_size, float rope_base) {
    op_begin();
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    const int i = 2 * p;
    if (i >= dim) return;
    const float2 cs = rope_cos_sin(pos, (i % head_size) >> 1, head_size, rope_base);
    const float q0 = q[i], q1 = q[i + 1];
    q[i] = __fsub_rn(__fmul_rn(q0, cs.x), __fmul_rn(q1, cs.y));
    q[i + 1] = __fadd_rn(__fmul_rn(q0, cs.y), __fmul_rn(q1, cs.x));
    if (i < kv_dim) {
        const float k0 = k[i], k1 = k[i + 1];
        k[i] = __fsub_rn(__fmul_rn(k0, cs.x), __fmul_rn(k1, cs.y));
        k[i + 1] = __fadd_rn(__fmul_rn(k0, cs.y), __fmul_rn(k1, cs.x));
    }
}

// src/scatter_kv.cu:6-26
static __global__ void scatter_kv_kernel(__half* kc, __half* vc, const float* k, const float* v, int layer, int pos,
                                  int n_kv_heads, int head_size, int seq_len) {
    op_begin();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int kv_dim = n_kv_heads * head_size;
    if (i >= kv_dim) return;
    const int h = i / head_size, off = i % head_size;
    const size_t idx = (size_t)layer * ((size_t)kv_dim * seq_len) + (size_t)h * ((size_t)seq_len * head_size) +
                       (size_t)pos * head_size + off;
    kc[idx] = __float2half_rn(k[i]);
    vc[idx] = __float2half_rn(v[i]);
}

// rope + scatter in one launch: q rotated in place; k rotated and written with v to the FP16 cache.
static __global__ void rope_scatter_kernel(float* q, const float* k, const float* v, __half* kc, __half* vc, int layer,
                                    int pos, int dim, int n_kv_heads, int head_size, int seq_len,
                                    float rope_base) {
    op_begin();
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    const int i = 2 * p;
    if (i >= dim) return;
    const int kv_dim = n_kv_heads * head_size;
    const float2 cs = rope_cos_sin(pos, (i % head_size) >> 1, head_size, rope_base);
    const float q0 = q[i], q1 = q[i + 1];
    q[i] = __fsub_rn(__fmul_rn(q0, cs.x), __fmul_rn(q1, cs.y));
    q[i + 1] = __fadd_rn(__fmul_rn(q0, cs.y), __fmul_rn(q1, cs.x));
    if (i < kv_dim) {
        const float k0 = k[i], k1 = k[i + 1];
        const float r0 = __fsub_rn(__fmul_rn(k0, cs.x), __fmul_rn(k1, cs.y));
        const float r1 = __fadd_rn(__fmul_rn(k0, cs.y), __fmul_rn(k1, cs.x));
        const int h = i / head_size, off = i % head_size;
        const size_t idx = (size_t)layer * ((size_t)kv_dim * seq_len) +
                           (size_t)h * ((size_t)seq_len * head_size) + (size_t)pos * head_size + off;
        *reinterpret_cast<__half2*>(kc + idx) = __floats2half2_rn(r0, r1);
        *reinterpret_cast<__half2*>(vc + idx) = __floats2half2_rn(v[i], v[i + 1]);
    }
}

// src/swiglu.cu:6-33
static __global__ void swiglu_kernel(float* hb, const float* h1, const float* h3, int size) {
    op_begin();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= size) return;
    const float val = h1[i];
    const float sig = __fdiv_rn(1.0f, 1.0f + expf(-val));
    hb[i] = __fmul_rn(__fmul_rn(val, sig), h3[i]);
}

// src/residual.cu:5-31
static __global__ void residual_add_kernel(float* out, const float* a, const float* b, int n) {
    op_begin();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) out[i] = a[i] + b[i];
}

// src/scale.cu:6-21
static __global__ void scale_multihead_kernel(float* att, float scale, int seq_len, int att_stride) {
    op_begin();
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t < seq_len) att[(size_t)blockIdx.y * att_stride + t] *= scale;
}

// src/softmax.cu:5-125 -- one CTA per head, max / exp / sum / divide (src/ops.cpp:56-75)
static __global__ void __launch_bounds__(256) softmax_multihead_kernel(float* out, const float* x, int seq_len,
                                                                int att_stride) {
    op_begin();
    __shared__ float red[8];
    const float* xi = x + (size_t)blockIdx.x * att_stride;
    float* oi = out + (size_t)blockIdx.x * att_stride;
    float m = -INFINITY;
    for (int t = threadIdx.x; t < seq_len; t += 256) m = fmaxf(m, xi[t]);
    m = warp_max(m);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = m;
    __syncthreads();
    m = red[0];
    for (int k = 1; k < 8; ++k) m = fmaxf(m, red[k]);
    __syncthreads();
    float s = 0.f;
    for (int t = threadIdx.x; t < seq_len; t += 256) {
        const float e = expf(xi[t] - m);
        oi[t] = e;
        s += e;
    }
    s = warp_sum(s);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
    __syncthreads();
    float tot = 0.f;
    for (int k = 0; k < 8; ++k) tot += red[k];
    for (int t = threadIdx.x; t < seq_len; t += 256) oi[t] = __fdiv_rn(oi[t], tot);
}

// src/multihead_gemv.cu:6-68 -- att[h][t] = q_h . K[kv(h)][t] (unscaled).  G lanes share a cache row, 8 elements (16 bytes)
// each: head sizes 16 to 256 that are powers of two, cache rows on 16-byte boundaries.  A lane keeps its piece of the query
// in registers and has the loads of kDotRows rows in flight; the sums go through log2(G) shuffles.  Bound by L2 latency.
// One warp per row with 2-byte loads (multihead_gemv_any_kernel) took 10.5 us for 32 heads of 128 and 1501 positions.
constexpr int kDotThreads = 256, kDotRows = 4;
template <int G>
static __global__ void __launch_bounds__(kDotThreads) multihead_gemv_kernel(float* att, const float* q, const __half* kc, int layer, int pos,
                                                                            int n_heads, int n_kv_heads, int seq_len) {
    op_begin();
    constexpr int hs = 8 * G, kStep = kDotThreads / G;
    const int h = blockIdx.y, kvh = h / (n_heads / n_kv_heads), piece = threadIdx.x % G;
    const int t0 = blockIdx.x * (kStep * kDotRows) + threadIdx.x / G;
    const uint4* kr = reinterpret_cast<const uint4*>(kc + ((size_t)layer * n_kv_heads + kvh) * ((size_t)seq_len * hs)) + piece;
    uint4 u[kDotRows];
#pragma unroll
    for (int r = 0; r < kDotRows; ++r) {
        const int t = t0 + r * kStep;
        u[r] = t <= pos ? kr[(size_t)t * G] : make_uint4(0, 0, 0, 0);
    }
    float qv[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) qv[i] = q[(size_t)h * hs + piece * 8 + i];
#pragma unroll
    for (int r = 0; r < kDotRows; ++r) {
        const int t = t0 + r * kStep;
        const float2 a = half2_bits_to_float2(u[r].x), b = half2_bits_to_float2(u[r].y);
        const float2 c = half2_bits_to_float2(u[r].z), d = half2_bits_to_float2(u[r].w);
        float s = fmaf(qv[3], b.y, fmaf(qv[2], b.x, fmaf(qv[1], a.y, qv[0] * a.x)));
        s += fmaf(qv[7], d.y, fmaf(qv[6], d.x, fmaf(qv[5], c.y, qv[4] * c.x)));
#pragma unroll
        for (int o = G / 2; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        if (piece == 0 && t <= pos) att[(size_t)h * seq_len + t] = s;
    }
}
// Any head size and alignment: one warp per (h, t).
static __global__ void __launch_bounds__(128) multihead_gemv_any_kernel(float* att, const float* q, const __half* kc, int layer, int pos,
                                                                        int n_heads, int n_kv_heads, int head_size, int seq_len) {
    op_begin();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int t = blockIdx.x * 4 + warp, h = blockIdx.y;
    if (t > pos) return;
    const int kvh = h / (n_heads / n_kv_heads);
    const __half* kr = kc + (size_t)layer * ((size_t)n_kv_heads * head_size * seq_len) +
                       (size_t)kvh * ((size_t)seq_len * head_size) + (size_t)t * head_size;
    const float* qh = q + (size_t)h * head_size;
    float s = 0.f;
    for (int d = lane; d < head_size; d += 32) s = fmaf(qh[d], __half2float(kr[d]), s);
    s = warp_sum(s);
    if (lane == 0) att[(size_t)h * seq_len + t] = s;
}

// src/aggregation.cu:6-31 -- out[h][i] = sum_t V[kv(h)][t][i] * att[h][t]; V points at the layer.  Bound by the latency of a
// serial walk over the positions unless many walk at once: a cluster of kAggCtas CTAs per head, each takes a contiguous part
// of the positions, its threads (position, 16-byte piece of the row) with kAggRows loads in flight; the partial sums meet in
// shared memory and then in the first CTA, both in a fixed order.  Head sizes that are multiples of 8, up to 128, rows on
// 16-byte boundaries.  One CTA of four warps per head with 2-byte loads (aggregation_any_kernel) took 125 us for 32 heads of
// 128 and 1501 positions.
constexpr int kAggThreads = 256, kAggCtas = 8, kAggRows = 4;
static __global__ void __launch_bounds__(kAggThreads) __cluster_dims__(kAggCtas, 1, 1)
    aggregation_kernel(float* out, const __half* v, const float* att, int seq_len, int head_size, int gqa_factor, int att_stride) {
    __shared__ float part[kAggThreads * 8];  // [position row][head_size]
    __shared__ float sums[kAggCtas][128];    // of the first CTA: what every CTA of the cluster found
    // The first CTA has to run before its shared memory is written: everybody reports, and waits only ahead of the store.
    asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");
    op_begin();
    const int rank = blockIdx.x % kAggCtas, h = blockIdx.x / kAggCtas, tid = threadIdx.x;
    const int pieces = head_size >> 3, rows = kAggThreads / pieces;
    const int row = tid / pieces, piece = tid - row * pieces;
    const int per = (seq_len + kAggCtas - 1) / kAggCtas, t_end = min(seq_len, (rank + 1) * per);
    // cache stride per kv head is att_stride (= allocated seq_len) rows, as in the reference call
    const uint4* vb = reinterpret_cast<const uint4*>(v + (size_t)(h / gqa_factor) * ((size_t)att_stride * head_size)) + piece;
    const float* ah = att + (size_t)h * att_stride;
    float acc[8] = {};
    if (row < rows)
        for (int t0 = rank * per + row; t0 < t_end; t0 += rows * kAggRows) {
            uint4 u[kAggRows];
            float w[kAggRows];
#pragma unroll
            for (int r = 0; r < kAggRows; ++r) {
                const int t = t0 + r * rows;
                u[r] = t < t_end ? vb[(size_t)t * pieces] : make_uint4(0, 0, 0, 0);
                w[r] = t < t_end ? ah[t] : 0.f;
            }
#pragma unroll
            for (int r = 0; r < kAggRows; ++r) {
                const uint32_t bits[4] = {u[r].x, u[r].y, u[r].z, u[r].w};
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const float2 f = half2_bits_to_float2(bits[i]);
                    acc[2 * i] = fmaf(f.x, w[r], acc[2 * i]);
                    acc[2 * i + 1] = fmaf(f.y, w[r], acc[2 * i + 1]);
                }
            }
        }
    if (row < rows) {
#pragma unroll
        for (int i = 0; i < 8; ++i) part[row * head_size + piece * 8 + i] = acc[i];
    }
    __syncthreads();
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");  // all CTAs of the cluster have started
    if (tid < head_size) {
        float s = 0.f;
        for (int r = 0; r < rows; ++r) s += part[r * head_size + tid];
        uint32_t to;  // sums[rank][tid] of the cluster's first CTA
        asm volatile("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(to) : "r"(smem_u32(&sums[rank][tid])));
        asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(to), "f"(s) : "memory");
    }
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    if (rank == 0 && tid < head_size) {
        float s = 0.f;
#pragma unroll
        for (int c = 0; c < kAggCtas; ++c) s += sums[c][tid];
        out[(size_t)h * head_size + tid] = s;
    }
}
// Other head sizes and alignments.
static __global__ void __launch_bounds__(128) aggregation_any_kernel(float* out, const __half* v, const float* att, int seq_len,
                                                                     int head_size, int gqa_factor, int att_stride) {
    // 4 warps split the positions, lanes split the head dimension; fixed-order merge
    __shared__ float part[4][128];
    op_begin();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int h = blockIdx.x, kvh = h / gqa_factor;
    const __half* vb = v + (size_t)kvh * ((size_t)att_stride * head_size);
    const float* ah = att + (size_t)h * att_stride;
    for (int d0 = 0; d0 < head_size; d0 += 32) {
        const int d = d0 + lane;
        float acc = 0.f;
        if (d < head_size)
            for (int t = warp; t < seq_len; t += 4) acc = fmaf(__half2float(vb[(size_t)t * head_size + d]), ah[t], acc);
        if (d < 128) part[warp][d] = acc;
    }
    __syncthreads();
    for (int d = threadIdx.x; d < head_size; d += 128)
        out[(size_t)h * head_size + d] = part[0][d] + part[1][d] + part[2][d] + part[3][d];
}

// src/matmul.cu:14-148 -- out[n] = W[n][d] . x for rows of whole 16-byte vectors.  Bound by the weight stream: every warp
// walks its rows in batches of kOpGemvU 16-byte loads a lane, the next batch requested before the current one is used, also
// across the end of a row and before the input is staged in shared memory.  `split` warps of a CTA share a row where there
// are fewer rows than warps (split > 1: one round, so that a single exchange through shared memory ends it).
// A warp on two rows at a time that waited for the input first, and for its loads at the end of every row, streamed
// 117 MB in 27 us and a layer's seven matrices (436 MB) in 114 us.
constexpr int kOpGemvThreads = 512, kOpGemvU = 4;
template <typename WT>
static __global__ void __launch_bounds__(kOpGemvThreads, 2) op_gemv_kernel(float* out, const float* x, const WT* w, int n, int d, int split) {
    extern __shared__ __align__(128) unsigned char op_smem[];
    __shared__ float part[kOpGemvThreads / 32];
    op_begin();
    constexpr int kVec = 16 / (int)sizeof(WT), kWarps = kOpGemvThreads / 32;
    const int tid = threadIdx.x, lane = tid & 31, sub = (tid >> 5) % split;
    const int nvec = d / kVec, step = gridDim.x * (kWarps / split);
    const int first = blockIdx.x * (kWarps / split) + (tid >> 5) / split;
    // vectors v0 .. v1 of a row, 32 * kOpGemvU at a time
    const int v0 = (int)((long long)nvec * sub / split), v1 = (int)((long long)nvec * (sub + 1) / split);
    const uint4* wv = reinterpret_cast<const uint4*>(w);
    int lrow = first, lv = v0;  // what is requested next
    auto load = [&](uint4 (&u)[kOpGemvU]) {
#pragma unroll
        for (int i = 0; i < kOpGemvU; ++i) {
            const int v = lv + i * 32 + lane;
            if (lrow < n && v < v1) u[i] = ldg_stream_u4(wv + (size_t)lrow * nvec + v);
        }
        lv += 32 * kOpGemvU;
        if (lv >= v1) {
            lv = v0;
            lrow += step;
        }
    };
    uint4 a[kOpGemvU], b[kOpGemvU];
    load(a);
    // the input as planes of four floats per vector, so that a warp's 16-byte reads meet no bank twice
    float4* xs = reinterpret_cast<float4*>(op_smem);
    const float4* x4 = reinterpret_cast<const float4*>(x);
    constexpr int kPlanes = kVec / 4;
    for (int i = tid; i < nvec * kPlanes; i += kOpGemvThreads) xs[(i % kPlanes) * nvec + i / kPlanes] = x4[i];
    __syncthreads();
    int row = first, v = v0;
    float s0 = 0.f, s1 = 0.f;
    auto use = [&](const uint4 (&u)[kOpGemvU]) {
#pragma unroll
        for (int i = 0; i < kOpGemvU; ++i) {
            const int k = v + i * 32 + lane;
            if (k >= v1) continue;
            if constexpr (sizeof(WT) == 2) {
                const float4 lo = xs[k], hi = xs[nvec + k];
                float2 p;
                p = unpack2<WT>(u[i].x); s0 = fmaf(p.x, lo.x, s0); s1 = fmaf(p.y, lo.y, s1);
                p = unpack2<WT>(u[i].y); s0 = fmaf(p.x, lo.z, s0); s1 = fmaf(p.y, lo.w, s1);
                p = unpack2<WT>(u[i].z); s0 = fmaf(p.x, hi.x, s0); s1 = fmaf(p.y, hi.y, s1);
                p = unpack2<WT>(u[i].w); s0 = fmaf(p.x, hi.z, s0); s1 = fmaf(p.y, hi.w, s1);
            } else {
                const float4 f = xs[k];
                s0 = fmaf(__uint_as_float(u[i].x), f.x, s0); s1 = fmaf(__uint_as_float(u[i].y), f.y, s1);
                s0 = fmaf(__uint_as_float(u[i].z), f.z, s0); s1 = fmaf(__uint_as_float(u[i].w), f.w, s1);
            }
        }
        v += 32 * kOpGemvU;
        if (v >= v1) {
            const float s = warp_sum(s0 + s1);
            if (split > 1)
                part[tid >> 5] = s;  // the same value from every lane
            else if (lane == 0)
                out[row] = s;
            s0 = s1 = 0.f;
            v = v0;
            row += step;
        }
    };
    while (row < n) {
        load(b);
        use(a);
        if (row >= n) break;
        load(a);
        use(b);
    }
    if (split > 1) {
        __syncthreads();
        const int r = blockIdx.x * (kWarps / split) + tid;
        if (tid < kWarps / split && r < n) {
            float s = 0.f;
            for (int i = 0; i < split; ++i) s += part[tid * split + i];
            out[r] = s;
        }
    }
}

}  // namespace lpp

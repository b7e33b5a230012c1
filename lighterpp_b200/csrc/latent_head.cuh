// Latent attention of one token after its input projection, a cluster of CTAs per head: the query in the latent space, the attention over
// the window, and the values, in one launch (latent.cuh has the scheme; its query GEMV, attention and value GEMV are the same as three
// launches for engines and sizes that do not fit here).
//
// Why: each of the three moves a few hundred KB and is bound by a launch, its dependency wait and a round trip or two (rutenex-300m: 3.0 + 3.8 +
// 3.9 us back to back); per head they depend on nothing of the other heads.  The CTAs of a head share its work: rows of W_uk, keys
// of the window, rows of W_uv.  What they owe each other, the query (rank floats) and the unnormalised results (rank floats a CTA),
// is written straight into everybody's shared memory, and a hardware cluster barrier follows: two exchanges, and a meeting at the start
// (a CTA has to run before it is written to), where three kernel boundaries were.  Weights and the cache rows of earlier positions are requested before the dependency wait.  Every head reads the shared cache rows by
// itself (16 heads: 4.7 MB from L2 at the 300m shape), in exchange for as many SMs; query, scores and probabilities stay FP32.
// Measured, 33 tokens of rutenex-300m at 700: 21.75 -> 20.1 ms, 18.9 with the SM's memory split as the GEMVs have it.  What is left is latency:
// launch and dependency wait, the three barriers, and code that is fetched once a launch (loops are kept short; 98 registers of
// prefetched weights instead of shared memory: 0.3 ms more at position 3).
#pragma once
#include "latent.cuh"
#include "prefill.cuh"

namespace lpp {

constexpr int kLhThreads = 256, kLhMaxCtas = 8, kLhMaxRank = 2048;
// Shared memory beside which a GEMV's CTA finds room on an SM.  A CTA with more waits for the input GEMV's CTA to leave and clusters then
// for whole groups of free SMs (rutenex-1b, 208 KB, of which 150 are cache rows: a token at 3 771 us instead of 695, at 700 906 instead of 762).
constexpr size_t kLhSmemBytes = 80 * 1024;

struct LatentHeadArgs {
    LatentArgs lat;
    StepState* st;
    const __nv_bfloat16* w_uk;  // [heads * rank_pitch][dim_pitch]
    const __nv_bfloat16* w_uv;  // [heads * vdim_rows][val_pitch]
    float* out;                 // [heads * vdim]
    int val_pitch, seq_len, rows_cap;  // rows_cap: keys a CTA takes at most
    int early;                  // position and cache may be read before the dependency wait
    float scale;
};
// Cache rows in shared memory: an odd number of 16-byte pieces, so that rows lie on different banks.
__host__ __device__ inline int latent_head_row_bytes(int row_width) { return row_width * 2 + 16; }
__host__ __device__ inline size_t latent_head_smem(int row_width, int rank_pitch, int dim_pitch, int vdim_rows, int val_pitch, int rows_cap, int ctas) {
    return (size_t)rows_cap * latent_head_row_bytes(row_width) +
           4 * ((size_t)row_width + dim_pitch + 2 * (size_t)((rows_cap + 3) / 4 * 4) + (size_t)ctas * rank_pitch + 2 * kLhMaxCtas + 8 * kLhThreads + val_pitch + 16) +
           2 * ((size_t)((rank_pitch + ctas - 1) / ctas) * dim_pitch + (size_t)((vdim_rows + ctas - 1) / ctas) * val_pitch);
}

__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
// *p of CTA `rank` of the cluster <- v
__device__ __forceinline__ void cluster_store(const float* p, int rank, float v) {
    uint32_t to;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(to) : "r"(smem_u32(p)), "r"(rank));
    asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(to), "f"(v) : "memory");
}
// Eight 16-bit elements times eight floats from shared memory, on top of s.
template <typename T>
__device__ __forceinline__ float dot8(const uint4& u, const float* x, float s) {
    const float4 a = *reinterpret_cast<const float4*>(x), b = *reinterpret_cast<const float4*>(x + 4);
    float2 f;
    f = unpack2<T>(u.x); s = fmaf(f.x, a.x, s); s = fmaf(f.y, a.y, s);
    f = unpack2<T>(u.y); s = fmaf(f.x, a.z, s); s = fmaf(f.y, a.w, s);
    f = unpack2<T>(u.z); s = fmaf(f.x, b.x, s); s = fmaf(f.y, b.y, s);
    f = unpack2<T>(u.w); s = fmaf(f.x, b.z, s); s = fmaf(f.y, b.w, s);
    return s;
}

static __global__ void __launch_bounds__(kLhThreads) latent_head_kernel(const LatentHeadArgs a) {
    extern __shared__ __align__(16) unsigned char lh_smem[];
    typedef __nv_bfloat16 T;
    const LatentArgs& L = a.lat;
    uint32_t C, rank;
    asm volatile("mov.u32 %0, %%cluster_nctaid.x;" : "=r"(C));
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
    // a CTA has to run before its shared memory is written: everybody reports now and waits ahead of the first such store
    asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");
    pdl_launch_dependents();
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, h = (int)(blockIdx.x / C);
    const int row_bytes = latent_head_row_bytes(L.row_width), RP = L.rank_pitch, nv = L.row_width >> 3;
    unsigned char* rows = lh_smem;                                                    // [rows_cap]
    float* ql = reinterpret_cast<float*>(rows + (size_t)a.rows_cap * row_bytes);      // [row_width]: the query
    float* qp = ql + L.row_width;                                                     // [dim_pitch]: its plain part
    float* sc = qp + L.dim_pitch;                                                     // [rows_cap]: scores
    float* pr = sc + (a.rows_cap + 3) / 4 * 4;                                        // [rows_cap]: probabilities
    float* recv = pr + (a.rows_cap + 3) / 4 * 4;                                      // [C][rank_pitch]: everybody's results
    float* ml = recv + (size_t)C * RP;                                                // [C] maxima, [C] sums
    float* pv = ml + 2 * kLhMaxCtas;                                                  // [key groups][rank_pitch]
    float* olat = pv + 8 * kLhThreads;                                                // [val_pitch]
    float* red = olat + a.val_pitch;
    if (!a.early) pdl_wait();
    const int pos = a.st->pos;
    const bool ok = pos >= 0 && pos < a.seq_len;
    const int first = L.window > 0 ? max(0, pos - L.window + 1) : 0, n_keys = ok ? pos - first + 1 : 0;
    const int chunk = min((n_keys + (int)C - 1) / (int)C, a.rows_cap), k0 = first + (int)rank * chunk, nk = max(0, min(chunk, n_keys - (int)rank * chunk));
    const __half* cache = reinterpret_cast<const __half*>(L.cache);
    const bool owner = nk > 0 && pos < k0 + nk && pos >= k0;  // of the present position's row
    const int n_fixed = nk - (owner ? 1 : 0);              // rows of earlier positions
    unsigned char* present = rows + (size_t)n_fixed * row_bytes;
#pragma unroll 1
    for (int i = warp; i < n_fixed; i += kLhThreads / 32)
        for (int v = lane; v < nv; v += 32) cp_async_16(rows + (size_t)i * row_bytes + v * 16, cache + (size_t)(k0 + i) * L.row_width + v * 8, true);
    // this CTA's rows of both matrices
    const int vk = L.dim_pitch >> 3, RS = (RP + (int)C - 1) / (int)C, ra = (int)rank * RS, rn = max(0, min(RS, RP - ra));
    const int vv = a.val_pitch >> 3, VS = (L.vdim_rows + (int)C - 1) / (int)C, va = (int)rank * VS, vn = max(0, min(VS, L.vdim_rows - va));
    uint4* wk = reinterpret_cast<uint4*>(red + 16);  // [RS][dim_pitch]
    uint4* wv = wk + (size_t)RS * vk;                // [VS][val_pitch]
    const uint4* wk_src = reinterpret_cast<const uint4*>(a.w_uk + ((size_t)h * RP + ra) * L.dim_pitch);
    const uint4* wv_src = reinterpret_cast<const uint4*>(a.w_uv + ((size_t)h * L.vdim_rows + va) * a.val_pitch);
#pragma unroll 1
    for (int i = tid; i < rn * vk; i += kLhThreads) cp_async_16(wk + i, wk_src + i, true);
#pragma unroll 1
    for (int i = tid; i < vn * vv; i += kLhThreads) cp_async_16(wv + i, wv_src + i, true);
    cp_async_commit();
    if (owner)
#pragma unroll 1
        for (int k = tid; k < L.rank; k += kLhThreads) pv[k] = __ldg(L.norm_w + k);
    if (a.early) pdl_wait();
    const float gate = __ldcg(L.gate + h);
    const unsigned short* qrot = reinterpret_cast<const unsigned short*>(L.query) + (size_t)h * L.row_width;
    const unsigned short* krot = reinterpret_cast<const unsigned short*>(L.cache) + (size_t)pos * L.row_width;
    if (tid < L.dim_pitch) qp[tid] = __ldcg(L.q_plain + (size_t)h * L.dim_pitch + tid);
#pragma unroll 1
    for (int i = tid + kLhThreads; i < L.dim_pitch; i += kLhThreads) qp[i] = __ldcg(L.q_plain + (size_t)h * L.dim_pitch + i);
#pragma unroll 1
    for (int i = RP + tid; i < L.row_width; i += kLhThreads) {
        ql[i] = __half2float(__ushort_as_half(__ldcg(qrot + i)));
        if (owner) reinterpret_cast<unsigned short*>(present)[i] = __ldcg(krot + i);
    }
    float ss = 0.f;
    if (owner)
#pragma unroll 1
        for (int k = tid; k < L.rank; k += kLhThreads) {
            const float v = __ldcg(L.latent + k);
            olat[k] = v;
            ss = fmaf(v, v, ss);
        }
    cp_async_wait<0>();
    __syncthreads();
    cluster_wait();
    // ---- the query in the latent space: this CTA's columns, eight lanes each, to everybody
    const int l8 = tid & 7;
#pragma unroll 1
    for (int row = tid >> 3; row < (rn + 3) / 4 * 4; row += kLhThreads / 8) {  // whole warps
        float s = 0.f;
#pragma unroll 1
        for (int v = l8; v < vk; v += 8) s = dot8<T>(wk[min(row, rn - 1) * vk + v], qp + v * 8, s);
        s += __shfl_xor_sync(0xffffffffu, s, 4);
        s += __shfl_xor_sync(0xffffffffu, s, 2);
        s += __shfl_xor_sync(0xffffffffu, s, 1);
        if (row < rn && l8 < (int)C) cluster_store(ql + ra + row, l8, s);
    }
    // ---- the present position's row: the latent normed, its rotated part from the cache; the first head leaves the latent there
    if (owner) {
        ss = warp_sum(ss);
        if (lane == 0) red[warp] = ss;
        __syncthreads();
        float tot = 0.f;
#pragma unroll
        for (int w = 0; w < kLhThreads / 32; ++w) tot += red[w];
        const float scale = __fdiv_rn(1.0f, __fsqrt_rn(__fadd_rn(__fdiv_rn(tot, (float)L.rank), L.norm_eps)));
        __half* there = reinterpret_cast<__half*>(L.cache) + (size_t)pos * L.row_width;
#pragma unroll 1
        for (int k = tid; k < RP; k += kLhThreads) {
            const __half y = __float2half_rn(k < L.rank ? __fmul_rn(__fmul_rn(olat[k], scale), pv[k]) : 0.f);
            reinterpret_cast<__half*>(present)[k] = y;
            if (h == 0 && k < L.rank) there[k] = y;
        }
    }
    cluster_arrive();
    cluster_wait();
    // ---- scores: eight lanes a key
#pragma unroll 1
    for (int kb = 0; kb < nk; kb += kLhThreads / 8) {
        const int key = kb + (tid >> 3);
        const uint4* r = reinterpret_cast<const uint4*>(rows + (size_t)min(key, nk - 1) * row_bytes);
        float s = 0.f;
#pragma unroll 5
        for (int v = l8; v < nv; v += 8) s = dot8<__half>(r[v], ql + v * 8, s);
        s += __shfl_xor_sync(0xffffffffu, s, 4);
        s += __shfl_xor_sync(0xffffffffu, s, 2);
        s += __shfl_xor_sync(0xffffffffu, s, 1);
        if (l8 == 0 && key < nk) sc[key] = s * a.scale;
    }
    __syncthreads();
    float m = -INFINITY;  // every warp for itself
    for (int k = lane; k < nk; k += 32) m = fmaxf(m, sc[k]);
    m = warp_max(m);
    for (int k = tid; k < nk; k += kLhThreads) pr[k] = __expf(sc[k] - m);
    __syncthreads();
    // ---- weighted sum: eight columns a thread, the keys dealt to as many groups as there are threads for
    const int V = RP >> 3, KG = kLhThreads / V, vi = tid % V, kg = tid / V;
    if (kg < KG) {
        float o[8] = {};
#pragma unroll 8
        for (int k = kg; k < nk; k += KG) {
            const uint4 u = *reinterpret_cast<const uint4*>(rows + (size_t)k * row_bytes + vi * 16);
            const float p = pr[k];
            const float2 f0 = half2_bits_to_float2(u.x), f1 = half2_bits_to_float2(u.y), f2 = half2_bits_to_float2(u.z), f3 = half2_bits_to_float2(u.w);
            o[0] = fmaf(p, f0.x, o[0]); o[1] = fmaf(p, f0.y, o[1]); o[2] = fmaf(p, f1.x, o[2]); o[3] = fmaf(p, f1.y, o[3]);
            o[4] = fmaf(p, f2.x, o[4]); o[5] = fmaf(p, f2.y, o[5]); o[6] = fmaf(p, f3.x, o[6]); o[7] = fmaf(p, f3.y, o[7]);
        }
        float4* d = reinterpret_cast<float4*>(pv + (size_t)kg * RP + vi * 8);
        d[0] = make_float4(o[0], o[1], o[2], o[3]);
        d[1] = make_float4(o[4], o[5], o[6], o[7]);
    }
    if (warp == 0) {
        float l = 0.f;
        for (int k = lane; k < nk; k += 32) l += pr[k];
        l = warp_sum(l);
        if (lane < (int)C) {
            cluster_store(ml + rank, lane, m);
            cluster_store(ml + kLhMaxCtas + rank, lane, l);
        }
    }
    __syncthreads();
    for (int c = tid; c < RP; c += kLhThreads) {
        float s = 0.f;
        for (int g = 0; g < KG; ++g) s += pv[(size_t)g * RP + c];
        for (int t = 0; t < (int)C; ++t) cluster_store(recv + (size_t)rank * RP + c, t, s);
    }
    cluster_arrive();
    cluster_wait();
    // ---- everybody puts the parts together, then its rows of the values
    float mm = -INFINITY, w[kLhMaxCtas], sum = 0.f;
#pragma unroll
    for (int t = 0; t < kLhMaxCtas; ++t)
        if (t < (int)C) mm = fmaxf(mm, ml[t]);
#pragma unroll
    for (int t = 0; t < kLhMaxCtas; ++t) {
        w[t] = t < (int)C && ml[t] != -INFINITY ? __expf(ml[t] - mm) : 0.f;
        if (t < (int)C) sum = fmaf(w[t], ml[kLhMaxCtas + t], sum);
    }
    const float inv = sum > 0.f ? __fdiv_rn(1.f, sum) : 0.f;
    for (int c = tid; c < a.val_pitch; c += kLhThreads) {
        float s = 0.f;
        if (c < RP)
#pragma unroll
            for (int t = 0; t < kLhMaxCtas; ++t)
                if (t < (int)C) s = fmaf(w[t], recv[(size_t)t * RP + c], s);
        olat[c] = s * inv;
    }
    __syncthreads();
#pragma unroll 1
    for (int row = warp; row < vn; row += kLhThreads / 32) {
        float s = 0.f;
#pragma unroll 1
        for (int v = lane; v < vv; v += 32) s = dot8<T>(wv[row * vv + v], olat + v * 8, s);
        s = warp_sum(s);
        if (lane == 0 && va + row < L.vdim) a.out[(size_t)h * L.vdim + va + row] = s * gate;
    }
}

}  // namespace lpp

// Exact-order sampler: repetition penalty -> temperature -> softmax -> categorical draw with the
// SAME floating-point results as the reference's sequential CPU code (src/model.cpp:256-303 with
// softmax() of src/ops.cpp:56-75), computed in parallel.
//
// The reference sums 128K probabilities one after the other in FP32, twice (the softmax denominator
// and the running CDF).  Those sums carry ~1e-5 of rounding drift, more than the width of one
// token's probability in a flat 128K distribution, so any re-associated (tree) sum picks a
// neighbouring token in a large share of draws.  Re-association is avoided here by emulating the
// sequential rounding exactly:
//
//   While the running sum s stays inside one binade [2^E, 2^(E+1)) with ulp u, fl(s + x) equals
//   s + q*u where q = x/u rounded to nearest; only an exact tie depends on s, and then only on the
//   parity of s/u.  So each element acts on the integer S = s/u as a map
//   "S -> S + d[parity of S]", and maps compose associatively: a run of elements collapses, with a
//   parallel scan, into one pair (D0, D1).
//
//   Where the sum may change binade one map does not do.  Every thread classifies its four consecutive
//   elements from an approximate (double) prefix sum: if the prefix before and after the quad is safely
//   inside one binade the quad is "plain" and contributes a map; near a power of two it is a "window"
//   whose elements are added one by one with real FP32 additions; and where many quads of a block lie
//   near one (a confident distribution: the sum sits at 1 + a little for the whole rest of the
//   vocabulary) they are "dual" and contribute the maps of both binades, of which the walk takes the one
//   that the exact sum is in.  Blocks publish a short list of entries (runs of maps and windows); one warp
//   then walks all entries in order.  A map entry is applied only after checking that s really is in its
//   binade and stays in it; a run that leaves it is done over by the whole block (resolve_range: parallel
//   scan up to the element that leaves the binade, one real addition, and on from there), so the result
//   never depends on the approximate prefix being accurate -- only the speed does.
//
//   Latency-bound: ceil(V/2048) blocks, a few microseconds per dependent stage.  A token of the
//   Llama-3.2-1B shape whose distribution is confident (0.998 on one token): 3.35 ms with windows of
//   whole blocks added one by one by one warp, of which this kernel took 2.7 ms; 0.66 ms now.
//   128256 logits with 64 history entries, calls behind one another on one box: 43.5 us with maps of 64-bit words,
//   carries and offsets found warp after warp, checks inside the walk's chain and the history searched per entry;
//   32.6 us with 32-bit maps made by two additions, carries scanned by every warp, checks after the walk and
//   counts; 31.2 us with the registers of one CTA an SM.
//
// exp() is exp_repro (common.cuh): IEEE double arithmetic only, identical on host and device; it
// differs from libm's expf in the last bit for about 0.06 % of arguments, which is the only source
// of disagreement with the reference left (none in 3000 test draws at 32K-128K vocabularies).
//
// One launch, ceil(V/2048) co-resident blocks, bounded grid barriers between the stages (max, sum,
// CDF); vocabularies that need more blocks than the GPU has SMs use the tree sampler of sampler.cuh.
#pragma once
#include "common.cuh"
#include "sampler.cuh"

namespace lpp {

constexpr int kExactMaxEntries = 48;  // per block and list; a block that needs more becomes one kEntrySeq entry
constexpr int kExactLists = 2;        // of the denominator's sum and of the running distribution
constexpr double kExactEps = 1.0 / 4096.0;  // safety margin of the binade prediction (speed only)
// Quads near a power of two become dual runs when a block has more of them than this.  A window is the cheaper form where
// the sum passes a power of two within a quad or two (flat distributions: some ten windows per vocabulary, nearly each of
// which would leave its binade inside a dual run and be done over); a block that stays near one has hundreds.
constexpr int kExactDualMin = 16;

enum : int { kEntryMap = 0, kEntrySeq = 1, kEntryQuad = 2, kEntryDual = 3 };
constexpr int kExactListCap = 512;  // entries the walking block stages in shared memory per round

struct ExactEntry {
    int kind;  // kEntryMap: elements [lo, hi) as the map d[0..1] of binade e; kEntryDual: also as the map d[2..3] of binade
               // e + 1; kEntryQuad: add the four floats in d, elements lo..lo+3, one by one; kEntrySeq: elements [lo, hi)
               // through resolve_range
    int lo, hi;
    int e;
    unsigned int d[4];
};

struct SampleExactArgs {
    SampleArgs base;
    unsigned int* sync;      // [0] grid-barrier counter, [1] exit ticket; zero between launches
    double* block_sum;       // [n_blocks] approximate sum of exp per block
    int* entry_count;        // [kExactLists][n_blocks]
    ExactEntry* entries;     // [kExactLists][n_blocks][kExactMaxEntries]
};

// ---- the integer map of one element -------------------------------------------------------------

// Increments of a valid run are at most 2^23 (it ends inside its binade or on the next power of two); larger ones only have
// to stay larger, so sums saturate here and a map is two 32-bit words.
constexpr unsigned int kMapCap = 0x3fffffffu;
struct Map2 {
    unsigned int d0, d1;  // increment of S when S is even / odd
};
__device__ __forceinline__ Map2 map_identity() { return Map2{0u, 0u}; }
// b after a
__device__ __forceinline__ Map2 map_compose(Map2 a, Map2 b) {
    Map2 c;
    c.d0 = min(a.d0 + ((a.d0 & 1u) ? b.d1 : b.d0), kMapCap);
    c.d1 = min(a.d1 + ((a.d1 & 1u) ? b.d0 : b.d1), kMapCap);
    return c;
}
// Map of adding x (a non-negative float) to a sum in binade E (ulp 2^(E-23)); requires x < 2^E.  The two additions are
// those to the binade's first even and first odd S: S + x/u stays below 2^24 + 1, and where it passes 2^24 (S = 2^23 + 1,
// x = 2^E - u/2) the coarser rounding there gives 2^24 as the tie in this binade does.
__device__ __forceinline__ Map2 map_of(float x, int E) {
    const unsigned int b = (unsigned int)(E + 127) << 23;
    return Map2{__float_as_uint(__fadd_rn(__uint_as_float(b), x)) - b, __float_as_uint(__fadd_rn(__uint_as_float(b + 1u), x)) - (b + 1u)};
}

__device__ __forceinline__ int binade_of(double v) {  // floor(log2(v)) for v > 0 (normal doubles)
    return (int)((__double_as_longlong(v) >> 52) & 0x7ff) - 1023;
}

// The float that S ulps of binade E are (S in [2^23, 2^24]).
__device__ __forceinline__ float float_of_ulps(unsigned int S, int E) {
    return (S >= (1u << 24)) ? __uint_as_float((unsigned int)(E + 128) << 23)
                               : __uint_as_float(((unsigned int)(E + 127) << 23) | (S & 0x7fffffu));
}

// ---- grid barrier for this kernel (all blocks co-resident; bounded wait) -------------------------
// The block's writes are ordered by its own barrier and thread 0's release; a fence of every thread on top of that cost a microsecond a stage.

__device__ __forceinline__ bool sampler_grid_barrier(unsigned int* counter, unsigned int target, StepState* st,
                                                     int* s_flag, int tid) {
    __syncthreads();
    if (tid == 0) {
        asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(counter) : "memory");
        bool ok = true;
        unsigned int v;
        asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(counter) : "memory");
        if (v < target) {
            const long long t0 = clock64();
            long long limit = 1 << 17;  // the engine's limit is fetched from global memory only after ~65 us
            bool fetched = false;
            while (true) {
                asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(counter) : "memory");
                if (v >= target) break;
                if (clock64() - t0 > limit) {
                    if (!fetched) {
                        limit = wait_limit(st);
                        fetched = true;
                        continue;
                    }
                    atomicOr(&st->status, kStatusBarrierTimeout);
                    ok = false;
                    break;
                }
            }
        }
        *s_flag = ok ? 1 : 0;
    }
    __syncthreads();
    return *s_flag != 0;
}

// Inclusive segmented scan of per-thread maps over the block: `start` marks the first thread of a
// run.  Returns the composition of the maps of the run's threads up to and including this one.
__device__ __forceinline__ Map2 block_segscan(Map2 v, bool start, Map2* s_warp_map, int* s_warp_flag, int tid) {
    const int lane = tid & 31, warp = tid >> 5;
    int f = start ? 1 : 0;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        Map2 u;
        u.d0 = __shfl_up_sync(0xffffffffu, v.d0, o);
        u.d1 = __shfl_up_sync(0xffffffffu, v.d1, o);
        const int fu = __shfl_up_sync(0xffffffffu, f, o);
        if (lane >= o) {
            if (!f) v = map_compose(u, v);
            f |= fu;
        }
    }
    // v = composition from the last start at or before this lane within the warp; f = a start exists
    if (lane == 31) {
        s_warp_map[warp] = v;
        s_warp_flag[warp] = f;
    }
    __syncthreads();
    // the maps of the warps are scanned in the same way by every warp; one that is carried into this warp is prepended
    constexpr int kWarps = kSampleThreads / 32;
    Map2 c = map_identity();
    int fc = 1;
    if (lane < kWarps) {
        c = s_warp_map[lane];
        fc = s_warp_flag[lane];
    }
#pragma unroll
    for (int o = 1; o < kWarps; o <<= 1) {
        Map2 u;
        u.d0 = __shfl_up_sync(0xffffffffu, c.d0, o);
        u.d1 = __shfl_up_sync(0xffffffffu, c.d1, o);
        const int fu = __shfl_up_sync(0xffffffffu, fc, o);
        if (lane >= o) {
            if (!fc) c = map_compose(u, c);
            fc |= fu;
        }
    }
    Map2 carry;
    carry.d0 = __shfl_sync(0xffffffffu, c.d0, (warp - 1) & 31);
    carry.d1 = __shfl_sync(0xffffffffu, c.d1, (warp - 1) & 31);
    if (!f && warp > 0) v = map_compose(carry, v);
    __syncthreads();
    return v;
}

// Inclusive block scan of doubles (one value per thread).
__device__ __forceinline__ double block_scan_double(double v, double* s_warp, int tid) {
    const int lane = tid & 31, warp = tid >> 5;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const double u = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= o) v += u;
    }
    if (lane == 31) s_warp[warp] = v;
    __syncthreads();
    double off = 0.0;
    for (int w = 0; w < warp; ++w) off += s_warp[w];
    __syncthreads();
    return v + off;
}

// Sum of one double per thread over the block, returned to every thread.
__device__ __forceinline__ double block_sum_double(double v, double* s_warp, int tid) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if ((tid & 31) == 0) s_warp[tid >> 5] = v;
    __syncthreads();
    double t = 0.0;
#pragma unroll
    for (int w = 0; w < kSampleThreads / 32; ++w) t += s_warp[w];
    __syncthreads();
    return t;
}

// Stage helper: every thread owns four consecutive values x[0..3] (element indices base+4*tid+k,
// zero past the end).  Given the approximate prefix `pre` (double, exclusive) before the quad, the
// block writes its entry list for the sequential sum of these values.
static __device__ __noinline__ void emit_entries(const float (&x)[4], double pre, int first_elem, int n_valid_quads,
                                             ExactEntry* out, int* out_count, Map2* s_wm, int* s_wf, int* s_i,
                                             int tid) {
    const int lane = tid & 31;
    const bool valid = tid < n_valid_quads;
    const double post = pre + (double)x[0] + (double)x[1] + (double)x[2] + (double)x[3];
    // plain: the sum is provably inside one binade before, during and after this quad; near: inside one or the next
    bool plain = false, near = false;
    int E = 0;
    if (valid && pre > 0.0) {
        const int e0 = binade_of(pre * (1.0 - kExactEps)), e1 = binade_of(post * (1.0 + kExactEps));
        E = e0;
        const float lim = __uint_as_float((unsigned int)((e0 > -120 && e0 < 120 ? e0 : 0) + 127) << 23);  // 2^e0
        const bool fits = e0 > -120 && e0 < 119 && x[0] < lim && x[1] < lim && x[2] < lim && x[3] < lim;
        plain = fits && e0 == e1;
        near = fits && e1 == e0 + 1;
    }
    const bool use_dual = __syncthreads_count(near) > kExactDualMin;
    const bool dual = near && use_dual;
    const bool mapped = plain || dual;
    const bool zero = valid && post == 0.0;  // nothing but zeros so far: no entry
    // runs: maximal sequences of threads of one class (mapped runs also share E)
    const int cls = !valid ? 5000 : zero ? 4000 : plain ? E : dual ? 1000 + E : 3000;  // binades lie in (-120, 119): no clash
    const int prev = __shfl_up_sync(0xffffffffu, cls, 1);
    __shared__ int s_cls_last[kSampleThreads / 32], s_cls_first[kSampleThreads / 32];
    if (lane == 31) s_cls_last[tid >> 5] = cls;
    __syncthreads();
    const int before = (tid == 0) ? 6000 : (lane == 0 ? s_cls_last[(tid >> 5) - 1] : prev);
    // a quad without a map is an entry of its own: it travels with its four values
    const bool start = valid && !zero && (cls != before || !mapped);
    Map2 mp = map_identity(), mp2 = map_identity();
    if (mapped) {
#pragma unroll
        for (int k = 0; k < 4; ++k) mp = map_compose(mp, map_of(x[k], E));
    }
    const Map2 run = block_segscan(mp, start, s_wm, s_wf, tid);
    Map2 run2 = map_identity();
    if (use_dual) {  // the same for the whole block
        if (dual) {
#pragma unroll
            for (int k = 0; k < 4; ++k) mp2 = map_compose(mp2, map_of(x[k], E + 1));
        }
        run2 = block_segscan(mp2, start, s_wm, s_wf, tid);
    }
    // entry index = number of run starts up to and including this thread, minus one
    const unsigned int starts = __ballot_sync(0xffffffffu, start);
    if (lane == 0) s_i[tid >> 5] = __popc(starts);
    if (lane == 0) s_cls_first[tid >> 5] = cls;
    __syncthreads();
    const int warp_starts = (lane < kSampleThreads / 32) ? s_i[lane] : 0;
    const int off = __reduce_add_sync(0xffffffffu, lane < (tid >> 5) ? warp_starts : 0);
    const int total = __reduce_add_sync(0xffffffffu, warp_starts);
    const int idx = off + __popc(starts & (0xffffffffu >> (31 - lane))) - 1;
    const bool overflow = total > kExactMaxEntries;
    // is this thread the last of its run?
    const int nxt_cls = __shfl_down_sync(0xffffffffu, cls, 1);
    const int after = (tid == kSampleThreads - 1) ? 6000 : (lane == 31 ? s_cls_first[(tid >> 5) + 1] : nxt_cls);
    const bool last = valid && !zero && (cls != after || !mapped);
    if (!overflow) {
        if (start) {
            out[idx].kind = plain ? kEntryMap : dual ? kEntryDual : kEntryQuad;
            out[idx].lo = first_elem + 4 * tid;
            out[idx].e = E;
        }
        if (last) {
            out[idx].hi = first_elem + 4 * tid + 4;
            uint4 d;
            if (mapped)
                d = make_uint4(run.d0, run.d1, run2.d0, run2.d1);
            else  // a window carries its values, sparing the walker a memory round trip
                d = make_uint4(__float_as_uint(x[0]), __float_as_uint(x[1]), __float_as_uint(x[2]), __float_as_uint(x[3]));
            *reinterpret_cast<uint4*>(out[idx].d) = d;
        }
        if (tid == 0) *out_count = total;
    } else if (tid == 0) {
        out[0].kind = kEntrySeq;
        out[0].lo = first_elem;
        out[0].hi = first_elem + 4 * n_valid_quads;
        out[0].e = 0;
        *reinterpret_cast<uint4*>(out[0].d) = make_uint4(0u, 0u, 0u, 0u);
        *out_count = 1;
    }
    __syncthreads();
}

// State of the walk over all entries (shared memory).
struct WalkState {
    float s;       // exact running sum
    int found;     // >= 0: first element whose running sum exceeds r
    int resolved;  // runs that were done over
};
struct ResolveScratch {
    float s;
    int brk, cross, found;
    Map2 last_map[kSampleThreads / 32];
};

// Adds elements [lo, hi) of x to w->s in order, exactly, by the whole block: while the sum stays in one binade E the
// elements are maps and a block scan gives the sum before and after each; the first element that leaves the binade (or is
// no map of it: x >= 2^E, or the sum is zero) is added with one FP32 addition, and the scan starts over behind it.  Sums
// close to the subnormals go element by element.  With `stop`, ends at the first element after which the sum exceeds r.
// Every pass leaves a binade for good or ends the range, so a range costs a few passes of about 1.5 us.  A sum that is no
// number ends it at once: nothing changes it any more.
static __device__ __noinline__ void resolve_range(const float* x, int lo, int hi, bool stop, float r, WalkState* w, ResolveScratch* z, Map2* s_wm,
                                                  int* s_wf, int tid) {
    const int lane = tid & 31, warp = tid >> 5;
    constexpr int kNone = 0x7fffffff;
    for (int c0 = lo; c0 < hi; c0 += kSampleChunk) {
        const int end = min(hi - c0, kSampleChunk), i0 = 4 * tid;  // chunk-relative elements i0 .. i0 + 3 are this thread's
        float y[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) y[k] = (i0 + k < end) ? __ldcg(x + c0 + i0 + k) : 0.f;
        int from = 0;
        while (from < end) {
            const float s = w->s;
            if (!(s < INFINITY)) return;
            const unsigned int bits = __float_as_uint(s);
            const int E = (int)((bits >> 23) & 0xffu) - 127;
            const bool scan = s > 0.f && E > -120 && E < 119;
            __syncthreads();
            if (s > 0.f && !scan) {
                if (warp == 0) {
                    float sum = s;
                    int at = from;
                    bool hit = false;
                    while (at < end && !hit && sum < 0x1p-118f) {
                        const float v = (at + lane < end) ? __ldcg(x + c0 + at + lane) : 0.f;
                        const int m = min(32, end - at);
                        for (int j = 0; j < m && !hit; ++j, ++at) {
                            sum = __fadd_rn(sum, __shfl_sync(0xffffffffu, v, j));
                            hit = stop && r < sum;
                        }
                    }
                    if (lane == 0) {
                        w->s = sum;
                        if (hit) w->found = c0 + at - 1;
                        z->brk = at;
                    }
                }
                __syncthreads();
                if (w->found >= 0) return;
                from = z->brk;
                __syncthreads();
                continue;
            }
            if (tid == 0) z->brk = z->cross = z->found = kNone;
            __syncthreads();
            // the first element that is no map
            const float lim = scan ? __uint_as_float((unsigned int)(E + 127) << 23) : 0.f;
#pragma unroll
            for (int k = 3; k >= 0; --k)
                if (i0 + k >= from && i0 + k < end && (scan ? !(y[k] < lim) : y[k] != 0.f)) atomicMin(&z->brk, i0 + k);
            __syncthreads();
            const int brk = min(z->brk, end);
            // maps of the elements before it
            Map2 m[4], mp = map_identity();
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                m[k] = (scan && i0 + k >= from && i0 + k < brk) ? map_of(y[k], E) : map_identity();
                mp = map_compose(mp, m[k]);
            }
            const Map2 incl = block_segscan(mp, tid == 0, s_wm, s_wf, tid);
            Map2 ex;  // everything before this thread's elements
            ex.d0 = __shfl_up_sync(0xffffffffu, incl.d0, 1);
            ex.d1 = __shfl_up_sync(0xffffffffu, incl.d1, 1);
            if (lane == 31) z->last_map[warp] = incl;
            __syncthreads();
            if (lane == 0) ex = (warp == 0) ? map_identity() : z->last_map[warp - 1];
            const unsigned int S0 = (bits & 0x7fffffu) | 0x800000u;
            unsigned int S = S0 + ((S0 & 1u) ? ex.d1 : ex.d0), before[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                before[k] = S;
                S += (S & 1u) ? m[k].d1 : m[k].d0;
                if (scan && i0 + k >= from && i0 + k < brk) {
                    if (S > (1u << 24))
                        atomicMin(&z->cross, i0 + k);
                    else if (stop && r < float_of_ulps(S, E))
                        atomicMin(&z->found, i0 + k);
                }
            }
            __syncthreads();
            const int cross = min(z->cross, brk), found = z->found;
            if (found < cross) {
                if (tid == 0) w->found = c0 + found;
                __syncthreads();
                return;
            }
            // the element at `cross` is added on its own; at the end of the range there is none
            if (cross < end) {
#pragma unroll
                for (int k = 0; k < 4; ++k)
                    if (i0 + k == cross) z->s = __fadd_rn(scan ? float_of_ulps(before[k], E) : s, y[k]);
            } else if (tid == kSampleThreads - 1) {
                z->s = scan ? float_of_ulps(S, E) : s;
            }
            __syncthreads();
            if (tid == 0) {
                w->s = z->s;
                if (stop && cross < end && r < z->s) w->found = c0 + cross;
            }
            __syncthreads();
            if (w->found >= 0) return;
            from = cross + 1;
        }
    }
}

// Whole-block walk.  The blocks' entry lists are concatenated in block order (a prefix sum of the
// counts gives every entry its place), staged into shared memory kExactListCap at a time, and
// applied by warp 0.  Leaves the final state in *out (shared memory).
static __device__ __noinline__ void walk_all(const ExactEntry* entries, const int* counts, int n_blocks, const float* x,
                                         int n_total, bool stop, float r, ExactEntry* s_list, int* s_pref, int* s_i, Map2* s_wm, int* s_wf,
                                         ResolveScratch* z, WalkState* out, int tid) {
    static_assert(kSampleMaxBlocks <= kSampleThreads, "one thread per block's count");
    const int lane = tid & 31;
    __shared__ int s_ctl[2];                              // first entry that was not applied, first crossing entry
    __shared__ unsigned int s_before[kExactListCap + 1];  // bit pattern of the sum before every staged entry
    // inclusive prefix of the counts: thread t owns block t
    int c = (tid < n_blocks) ? __ldcg(counts + tid) : 0;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int u = __shfl_up_sync(0xffffffffu, c, o);
        if (lane >= o) c += u;
    }
    if (lane == 31) s_i[tid >> 5] = c;
    if (tid == 0) {
        out->s = 0.f;
        out->found = -1;
        out->resolved = 0;
        s_pref[0] = 0;
    }
    __syncthreads();
    int off = 0;
    for (int w = 0; w < (tid >> 5); ++w) off += s_i[w];
    s_pref[tid + 1] = c + off;
    __syncthreads();
    const int tot = s_pref[n_blocks];
    for (int base = 0; base < tot; base += kExactListCap) {
        const int m = min(kExactListCap, tot - base);
        for (int j = tid; j < m; j += kSampleThreads) {
            const int g = base + j;
            int lo = 0, hi = n_blocks;  // s_pref[lo] <= g < s_pref[hi]: entry g belongs to block lo
            while (hi - lo > 1) {
                const int mid = (lo + hi) >> 1;
                if (s_pref[mid] <= g)
                    lo = mid;
                else
                    hi = mid;
            }
            const uint4* src = reinterpret_cast<const uint4*>(entries + (size_t)lo * kExactMaxEntries + (g - s_pref[lo]));
            uint4* dst = reinterpret_cast<uint4*>(s_list + j);
            uint4 v0 = __ldcg(src);
            const uint4 v1 = __ldcg(src + 1);
            v0.w = (v0.w + 128u) << 23;  // the binade as the bit pattern of its end
            dst[0] = v0;
            dst[1] = v1;
        }
        __syncthreads();
        for (int i0 = 0; i0 < m;) {
            // pass 1 (warp 0, every lane the same): apply the entries from i0 on speculatively without a branch or a check,
            // keeping the sum before every entry.  A map moves the sum by an integer number of ulps inside one binade (or
            // exactly onto the next power of two), which on the bit pattern of a positive float is a plain integer addition.
            // The chain from sum to sum bounds the walk: with the checks inside it took 70 clocks an entry, 3.3 us for the
            // list of a 128 K vocabulary.
            if (tid < 32) {
                unsigned int bits = __float_as_uint(out->s);
#pragma unroll 4
                for (int i = i0; i < m; ++i) {
                    const int4 h = *reinterpret_cast<const int4*>(&s_list[i]);  // kind, lo, hi, end of the binade
                    const uint4 d = *reinterpret_cast<const uint4*>(s_list[i].d);
                    s_before[i] = bits;
                    // as a map: of the entry's binade, or of the next one (none there unless the entry is dual)
                    const bool next = bits >= (unsigned int)h.w, odd = bits & 1u;
                    const unsigned int even_d = next ? d.z : d.x, odd_d = next ? d.w : d.y;
                    const unsigned int nb = bits + (odd ? odd_d : even_d);
                    // as four values
                    float q = __uint_as_float(bits);
                    q = __fadd_rn(q, __uint_as_float(d.x));
                    q = __fadd_rn(q, __uint_as_float(d.y));
                    q = __fadd_rn(q, __uint_as_float(d.z));
                    q = __fadd_rn(q, __uint_as_float(d.w));
                    bits = (h.x == kEntryQuad) ? __float_as_uint(q) : nb;
                }
                s_before[m] = bits;
                if (lane == 0) s_ctl[0] = s_ctl[1] = 0x7fffffff;
            }
            __syncthreads();
            // pass 2: the first entry whose map does not hold at the sum before it, so that everything before it is exact,
            // and the first entry after which the running sum exceeds r (sums never decrease)
            for (int i = i0 + tid - lane; i < m; i += kSampleThreads) {
                int bad = 0x7fffffff, cross = 0x7fffffff;
                if (i + lane < m) {
                    const int kind = s_list[i + lane].kind;
                    const unsigned int end = (unsigned int)s_list[i + lane].e, in = s_before[i + lane], after = s_before[i + lane + 1];
                    const unsigned int from = (kind == kEntryDual && in >= end) ? end : end - 0x800000u;
                    const bool holds = in - from < 0x800000u && after - in <= 0x800000u && after - from <= 0x800000u;
                    if (kind == kEntrySeq || (kind != kEntryQuad && !holds)) bad = i + lane;
                    if (stop && r < __uint_as_float(after)) cross = i + lane;
                }
                bad = __reduce_min_sync(0xffffffffu, bad);
                cross = __reduce_min_sync(0xffffffffu, cross);
                if (lane == 0 && bad != 0x7fffffff) atomicMin(&s_ctl[0], bad);
                if (lane == 0 && cross != 0x7fffffff) atomicMin(&s_ctl[1], cross);
            }
            __syncthreads();
            const int good = min(m, s_ctl[0]);  // entries [i0, good) were applied exactly
            const int redo = stop ? min(s_ctl[1], good) : good;  // entry to look at element by element, m = none
            if (tid == 0) {
                out->s = __uint_as_float(s_before[redo]);
                if (redo == good && good < m) ++out->resolved;
            }
            __syncthreads();
            if (redo == m) break;
            resolve_range(x, s_list[redo].lo, min(s_list[redo].hi, n_total), stop, r, out, z, s_wm, s_wf, tid);
            if (out->found >= 0 || !(out->s < INFINITY)) return;
            i0 = redo + 1;
        }
    }
}

// One CTA an SM is all that ever runs: said in the bounds, since without it ptxas goes for two with 64 registers and 128 bytes of spills instead
// of 97 and none (stories15M, a token drawn 117.6 us / 108.8, greedy 89.1 / 88.4; 128256 logits 32.6 us / 31.2).
static __global__ void __launch_bounds__(kSampleThreads, 1) sample_exact_kernel(const SampleExactArgs ea) {
    const SampleArgs& a = ea.base;
    __shared__ float s_val[kSampleChunk];
    __shared__ MaxIdx s_mi[kSampleThreads / 32];
    __shared__ double s_d[kSampleThreads / 32];
    __shared__ Map2 s_wm[kSampleThreads / 32];
    __shared__ int s_wf[kSampleThreads / 32];
    __shared__ int s_i[kSampleThreads / 32];
    __shared__ int s_flag;
    __shared__ __align__(16) ExactEntry s_list[kExactListCap];
    __shared__ int s_pref[kSampleThreads + 1];
    __shared__ WalkState s_walk;
    __shared__ ResolveScratch s_res;
    __shared__ int s_cnt[kSampleChunk];  // occurrences in the history

    pdl_launch_dependents();
    pdl_wait();
    StepState* st = a.st;
    const int tid = threadIdx.x;
    const int nb = gridDim.x;
    const int base = blockIdx.x * kSampleChunk;
    const int n = min(kSampleChunk, a.vocab - base);
    const int n_quads = (n + 3) >> 2;
    const float temperature = st->temperature;
    const float penalty = st->penalty;
    const int hist_len = min(st->history_len, kHistoryMax);
    const bool greedy = (temperature == 0.0f);
    unsigned int bar = 0;  // barriers passed so far
    // ---- stage 0: penalty, temperature, block maximum (element i of the block lives in s_val[i])
    const int h0 = st->history[tid];  // in bounds whatever the length
    for (int i = tid; i < kSampleChunk; i += kSampleThreads) {
        s_val[i] = (i < n) ? __ldcg(a.logits + base + i) : 0.f;
        s_cnt[i] = 0;
    }
    __syncthreads();
    const bool penalised = penalty > 1.0f && hist_len > 0;
    if (penalised) count_history(st->history, h0, hist_len, base, n, s_cnt, tid);
    MaxIdx best = {-INFINITY, 0x7fffffff};
    for (int i = tid; i < n; i += kSampleThreads) {
        float v = s_val[i];
        if (penalised) v = penalise(v, s_cnt[i], penalty);
        if (!greedy) v = __fdiv_rn(v, temperature);
        s_val[i] = v;
        best = better(best, MaxIdx{v, base + i});
    }
    best = block_argmax(best, s_mi, tid);
    if (tid == 0) {
        __stcg(a.part_max + blockIdx.x, best.v);
        __stcg(a.part_idx + blockIdx.x, best.i);
    }
    bool alive = sampler_grid_barrier(&ea.sync[0], ++bar * nb, st, &s_flag, tid);

    // ---- global maximum (every block reduces the partials itself)
    MaxIdx g = {-INFINITY, 0x7fffffff};
    for (int b = tid; b < nb; b += kSampleThreads) g = better(g, MaxIdx{__ldcg(a.part_max + b), __ldcg(a.part_idx + b)});
    g = block_argmax(g, s_mi, tid);
    int token = g.i;

    if (!greedy && alive) {
        // ---- stage 1: e = exp(v - max) (kept in s_val and written to global), approximate block sums
        float x[4];
        double loc = 0.0;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const int i = 4 * tid + k;
            x[k] = (i < n) ? exp_repro(s_val[i] - g.v) : 0.f;
            if (i < n) a.logits[base + i] = x[k];
            loc += (double)x[k];
        }
        const double incl = block_scan_double(loc, s_d, tid);
        if (tid == kSampleThreads - 1) ea.block_sum[blockIdx.x] = incl;
        alive = sampler_grid_barrier(&ea.sync[0], ++bar * nb, st, &s_flag, tid);

        // ---- stage 2: entry list of the sequential sum of e
        // approximate sum of e over the blocks before this one (loads in parallel, then a block reduction)
        double mine = 0.0;
        for (int b = tid; b < (int)blockIdx.x; b += kSampleThreads) mine += __ldcg(ea.block_sum + b);
        const double before_blocks = block_sum_double(mine, s_d, tid);
        if (alive) {
            emit_entries(x, before_blocks + (incl - loc), base, n_quads, ea.entries + (size_t)blockIdx.x * kExactMaxEntries,
                         ea.entry_count + blockIdx.x, s_wm, s_wf, s_i, tid);
        }
        alive = alive && sampler_grid_barrier(&ea.sync[0], ++bar * nb, st, &s_flag, tid);

        // ---- stage 3: every block walks the entries itself: the exact softmax denominator (handing it out from one block
        // would cost another grid barrier).  Runs that were done over read the e of other blocks, which these replace below:
        // all blocks have come to the same end and wait for each other then.
        float denom = 1.f;
        if (alive) {
            walk_all(ea.entries, ea.entry_count, nb, a.logits, a.vocab, false, 0.f, s_list, s_pref, s_i, s_wm, s_wf, &s_res, &s_walk, tid);
            denom = s_walk.s;
            if (s_walk.resolved > 0) alive = sampler_grid_barrier(&ea.sync[0], ++bar * nb, st, &s_flag, tid);
        }

        // ---- stage 4: p = e / sum (IEEE division), entry list of the running CDF
        double locp = 0.0;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const int i = 4 * tid + k;
            x[k] = (i < n) ? __fdiv_rn(x[k], denom) : 0.f;
            if (i < n) a.logits[base + i] = x[k];  // like the reference, the logits end up as probabilities
            locp += (double)x[k];
        }
        const double inclp = block_scan_double(locp, s_d, tid);
        // approximate prefix of p before this block = (approximate prefix of e) / denominator
        const double pre_p = before_blocks / (double)denom + (inclp - locp);
        ExactEntry* cdf_entries = ea.entries + (size_t)nb * kExactMaxEntries;  // other blocks may still walk the first list
        int* cdf_count = ea.entry_count + nb;
        if (alive) {
            emit_entries(x, pre_p, base, n_quads, cdf_entries + (size_t)blockIdx.x * kExactMaxEntries, cdf_count + blockIdx.x, s_wm, s_wf, s_i, tid);
        }
        alive = alive && sampler_grid_barrier(&ea.sync[0], ++bar * nb, st, &s_flag, tid);

        // ---- stage 5: block 0 finds the first index whose running sum exceeds r
        if (alive && blockIdx.x == 0) {
            const float r = st->advance ? a.r_values[st->step_idx] : st->r;
            walk_all(cdf_entries, cdf_count, nb, a.logits, a.vocab, true, r, s_list, s_pref, s_i, s_wm, s_wf, &s_res, &s_walk, tid);
            token = (s_walk.found >= 0) ? s_walk.found : a.vocab - 1;
        }
    }

    // ---- exit ticket: the last block to get here publishes the result and resets the counters
    __syncthreads();
    if (blockIdx.x == 0 && tid == 0) {
        st->out_token = token;
        if (a.token_out) *a.token_out = token;
        if (st->advance) {
            const int k = st->step_idx;
            a.out_tokens[k] = token;
            st->token = token;
            st->pos = st->pos + 1;
            st->step_idx = k + 1;
            const int w = st->history_window;
            if (w > 0) {
                st->history[st->history_count % w] = token;
                st->history_count = st->history_count + 1;
                st->history_len = min(st->history_count, w);
            }
        }
    }
    __syncthreads();
    if (tid == 0) {
        const unsigned int ticket = atomicAdd(&ea.sync[1], 1u);
        s_flag = (ticket == (unsigned int)nb - 1);
    }
    __syncthreads();
    if (s_flag) {
        if (tid == 0) {
            ea.sync[0] = 0u;
            ea.sync[1] = 0u;
        }
        for (int i = tid; i < a.zero_n; i += kSampleThreads) a.zero[i] = 0u;
        if (a.bump && tid == 0) *a.bump = *a.bump + 1u;
    }
}

}  // namespace lpp

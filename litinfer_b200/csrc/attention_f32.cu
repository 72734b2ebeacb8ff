// Causal grouped-query attention of a ragged batch over the paged cache in float32: the 32-bit path's kernel for heads of up
// to 128 elements (a multiple of 4) on pages of a multiple of 16 keys.
//
// The general kernel (attention_generic.cu) walks a token's keys one by one, a warp a head: every key costs a reduction
// over the warp and a round trip to memory, and a group's query heads read the same keys once each (3 tokens of 12 heads on
// 2 key/value heads at 700 keys: 912 us).  Here the keys are taken in units of 32 at absolute positions (32 u .. 32 u + 31).
// A warp computes a unit for up to eight query heads of one key/value head: keys and values come through shared memory
// (16-byte copies, rows 16 bytes further apart than they are long), a lane a key for the scores, a lane every 32nd element
// for the values.  The units' results (maximum, denominator, weighted values) are merged in ascending order with a running
// maximum, so that a token's output does not depend on how many warps or blocks shared its units out: a block of four
// warps alone where there are many tokens, a cluster of up to eight blocks a token where there are few.  A round's merge takes
// its factors for all units at once (a lane a unit, the running maximum by a scan), then one multiply-add a unit and output.
// Scores, exponentials (full precision), sums and weighted values are float.
//
// All of AttentionOptions but several maps a query row (attention.cu sends those to the general kernel).
#define LI_PDL_KIND 4
#include "attention_options.h"
#include "common.cuh"

#include <cooperative_groups.h>

namespace {

namespace cg = cooperative_groups;

constexpr int kWarps = 4, kThreads = kWarps * 32;
constexpr int kUnit = 32, kHeads = 8, kMaxDim = 128, kQ = kMaxDim / 32;

// Per warp: keys [32][dh + 4] (later the unit's weighted values [heads][dh]), values [dh][36], probabilities [8][32], then the
// unit's maxima and denominators [2][8].
__host__ __device__ constexpr int warp_floats(int dh) { return kUnit * (dh + 4) + dh * 36 + kHeads * kUnit + 2 * kHeads; }
__host__ __device__ constexpr int shared_floats(int dh) { return kHeads * dh + kWarps * warp_floats(dh); }

__device__ __forceinline__ void copy16(float* dst, const float* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}

// NH: query heads a block computes (the last block of a key/value head may have fewer of its own; the rest it computes from
// zeros and leaves out).
template <int NH>
__global__ void __launch_bounds__(kThreads)
attention_f32_kernel(const float* __restrict__ qkv, float* __restrict__ out, const float* __restrict__ kcache, const float* __restrict__ vcache,
                     const int* __restrict__ block_table, int max_blocks, const int* __restrict__ seq_of_token, const int* __restrict__ positions,
                     int nh, int nkv, int dh, int page_size, int num_pages, float scale, int window, int csize, AttentionOptions opt) {
    extern __shared__ float4 raw[];
    float* q_sm = reinterpret_cast<float*>(raw);                           // [NH][dh]
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    float* mine = q_sm + kHeads * dh + warp * warp_floats(dh);
    float* k_sm = mine;
    float* v_sm = k_sm + kUnit * (dh + 4);
    float* p_sm = v_sm + dh * 36;
    float* ml_sm = p_sm + kHeads * kUnit;
    const int t = (int)blockIdx.x, rank = (int)blockIdx.z;
    const int G = nh / nkv, groups = (G + NH - 1) / NH;
    const int kvh = (int)blockIdx.y / groups, h0 = kvh * G + ((int)blockIdx.y % groups) * NH;
    const int heads = min(NH, kvh * G + G - h0);

    // (launched as a dependent, and lets the next one come: the o product asks for its weights meanwhile)
    pdl_launch_dependents();
    const int s = seq_of_token[t], p = positions[t];
    const int lo = first_seen_key(p, window, opt.chunk);
    const int keep_first = window > 0 ? opt.keep_first : 0;
    const int kept = keep_first < lo ? keep_first : lo;                    // kept first keys behind the window: 0 .. kept - 1
    const int kept_units = (kept + kUnit - 1) / kUnit, first_unit = lo / kUnit;
    const int units = kept_units + p / kUnit - first_unit + 1;
    const int* bt = block_table + (size_t)s * max_blocks;
    const int quads = dh >> 2;

    pdl_wait();
    const size_t row = opt.q_ld > 0 ? opt.q_ld : (nh + 2 * nkv) * dh;
    for (int e = tid; e < NH * dh; e += kThreads) q_sm[e] = e < heads * dh ? qkv[t * row + (size_t)h0 * dh + e] : 0.0f;
    __syncthreads();

    // the merge: item (head, 32 elements), shared out over the warps of all blocks of the cluster; a lane an element
    const int gwarp = rank * kWarps + warp, stride = kWarps * csize;
    float O[kHeads], L[kHeads], Mx[kHeads];
#pragma unroll
    for (int j = 0; j < kHeads; ++j) O[j] = L[j] = 0.0f, Mx[j] = -INFINITY;

    for (int base = 0; base < units; base += stride) {
        const int u = base + gwarp;
        if (u < units) {
            // kept units see keys below `kept`, the others keys from lo to p
            const bool is_kept = u < kept_units;
            const int key0 = (is_kept ? u : first_unit + u - kept_units) * kUnit;
            const int from = is_kept ? 0 : lo, to = is_kept ? kept - 1 : p;
            // two pieces of 16 keys, each within a page
#pragma unroll
            for (int half = 0; half < 2; ++half) {
                const int key = key0 + 16 * half;
                if (key <= to) {
                    int page = bt[key / page_size];
                    if (page < 0 || page >= num_pages) page = 0;           // host-validated; keep the read inside the cache
                    const float* kp = kcache + (((size_t)page * nkv + kvh) * page_size + key % page_size) * dh;
                    for (int c = lane; c < quads; c += 32) {
#pragma unroll
                        for (int r = 0; r < 16; ++r) copy16(k_sm + (16 * half + r) * (dh + 4) + 4 * c, kp + (size_t)r * dh + 4 * c);
                    }
                }
            }
            asm volatile("cp.async.commit_group;" ::: "memory");
#pragma unroll
            for (int half = 0; half < 2; ++half) {
                const int key = key0 + 16 * half;
                if (key <= to) {
                    int page = bt[key / page_size];
                    if (page < 0 || page >= num_pages) page = 0;
                    const float* vp = vcache + ((size_t)page * nkv + kvh) * dh * page_size + key % page_size + 4 * (lane & 3);
#pragma unroll 4
                    for (int d = lane >> 2; d < dh; d += 8) copy16(v_sm + d * 36 + 16 * half + 4 * (lane & 3), vp + (size_t)d * page_size);
                }
            }
            asm volatile("cp.async.commit_group;" ::: "memory");
            asm volatile("cp.async.wait_group 1;" ::: "memory");
            __syncwarp();
            // scores: this lane's key against every head
            const int key = key0 + lane;
            const bool seen = key >= from && key <= to;
            float4 sc[NH];                                                 // four chains a key, added in pairs
#pragma unroll
            for (int h = 0; h < NH; ++h) sc[h] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            const float4* kr = reinterpret_cast<const float4*>(k_sm + lane * (dh + 4));
#pragma unroll 4
            for (int c = 0; c < quads; ++c) {
                const float4 k4 = kr[c];
#pragma unroll
                for (int h = 0; h < NH; ++h) {
                    const float4 q4 = *reinterpret_cast<const float4*>(q_sm + h * dh + 4 * c);
                    sc[h].x = fmaf(q4.x, k4.x, sc[h].x);
                    sc[h].y = fmaf(q4.y, k4.y, sc[h].y);
                    sc[h].z = fmaf(q4.z, k4.z, sc[h].z);
                    sc[h].w = fmaf(q4.w, k4.w, sc[h].w);
                }
            }
            float m[NH], l[NH];
#pragma unroll
            for (int h = 0; h < NH; ++h) {
                float v = ((sc[h].x + sc[h].y) + (sc[h].z + sc[h].w)) * scale;
                if (opt.softcap > 0.0f) v = opt.softcap * tanhf(v / opt.softcap);
                if (opt.slopes && h < heads) v -= opt.slopes[h0 + h] * (float)(p - key);
                v = seen ? v : -INFINITY;
                m[h] = warp_max(v);
                // (a score of minus infinity has no weight, also where the unit has no other; NaN stays NaN)
                const float e = seen && v != -INFINITY ? expf(v - m[h]) : 0.0f;
                l[h] = warp_sum(e);
                p_sm[h * kUnit + lane] = e;
            }
            asm volatile("cp.async.wait_group 0;" ::: "memory");
            __syncwarp();
            float acc[NH][kQ];
#pragma unroll
            for (int h = 0; h < NH; ++h)
#pragma unroll
                for (int i = 0; i < kQ; ++i) acc[h][i] = 0.0f;
            const int quads_seen = (min(kUnit, to - key0 + 1) + 3) >> 2;
#pragma unroll 2
            for (int j = 0; j < quads_seen; ++j) {
                // keys that are not seen: whatever lies in their place (no finite number perhaps) is left out
                const int left = to - key0 - 4 * j, skip = from - key0 - 4 * j;
                float4 v4[kQ];
#pragma unroll
                for (int i = 0; i < kQ; ++i) {
                    const int d = lane + 32 * i;
                    v4[i] = d < dh ? *reinterpret_cast<const float4*>(v_sm + d * 36 + 4 * j) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                    if (skip > 0) v4[i].x = 0.0f;
                    if (left < 1 || skip > 1) v4[i].y = 0.0f;
                    if (left < 2 || skip > 2) v4[i].z = 0.0f;
                    if (left < 3 || skip > 3) v4[i].w = 0.0f;
                }
#pragma unroll
                for (int h = 0; h < NH; ++h) {
                    const float4 e4 = *reinterpret_cast<const float4*>(p_sm + h * kUnit + 4 * j);
#pragma unroll
                    for (int i = 0; i < kQ; ++i) {
                        acc[h][i] = fmaf(e4.x, v4[i].x, acc[h][i]);
                        acc[h][i] = fmaf(e4.y, v4[i].y, acc[h][i]);
                        acc[h][i] = fmaf(e4.z, v4[i].z, acc[h][i]);
                        acc[h][i] = fmaf(e4.w, v4[i].w, acc[h][i]);
                    }
                }
            }
#pragma unroll
            for (int h = 0; h < NH; ++h) {
#pragma unroll
                for (int i = 0; i < kQ; ++i)
                    if (lane + 32 * i < dh) k_sm[h * dh + lane + 32 * i] = acc[h][i];
                if (lane == 0) ml_sm[h] = m[h], ml_sm[kHeads + h] = l[h];
            }
        }
        // merge this round's units (at most 32) in ascending order
        if (csize > 1) cg::this_cluster().sync();
        else __syncthreads();
        const int here = min(stride, units - base);
        auto results = [&](int x) -> const float* {
            float* r = q_sm + kHeads * dh + (x % kWarps) * warp_floats(dh);
            return csize > 1 ? cg::this_cluster().map_shared_rank(r, x / kWarps) : r;
        };
#pragma unroll
        for (int j = 0; j < kHeads; ++j) {
            const int item = gwarp + j * stride;
            if (item >= heads * kQ) continue;                              // (uniform)
            const int h = item / kQ, d = lane + 32 * (item % kQ);
            // a lane a unit: its maximum and denominator, the running maximum up to it, and the two factors of its merge
            float mu = -INFINITY, lu = 0.0f;
            if (lane < here) {
                const float* ml = results(lane) + kUnit * (dh + 4) + dh * 36 + kHeads * kUnit;
                mu = ml[h], lu = ml[kHeads + h];
            }
            float run = mu;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const float v = __shfl_up_sync(0xffffffffu, run, o);
                if (lane >= o) run = fmaxf(run, v);
            }
            run = fmaxf(run, Mx[j]);
            float before = __shfl_up_sync(0xffffffffu, run, 1);
            if (lane == 0) before = Mx[j];
            const float fo = before == -INFINITY ? 0.0f : expf(before - run), fu = mu == -INFINITY ? 0.0f : expf(mu - run);
            for (int x0 = 0; x0 < here; x0 += 8) {
                float v[8];
#pragma unroll
                for (int x = 0; x < 8; ++x) v[x] = (x0 + x < here && d < dh) ? results(x0 + x)[h * dh + d] : 0.0f;
#pragma unroll
                for (int x = 0; x < 8; ++x) {
                    if (x0 + x < here) {
                        const float a = __shfl_sync(0xffffffffu, fo, x0 + x), b = __shfl_sync(0xffffffffu, fu, x0 + x);
                        O[j] = O[j] * a + v[x] * b;
                        L[j] = L[j] * a + __shfl_sync(0xffffffffu, lu, x0 + x) * b;
                    }
                }
            }
            Mx[j] = __shfl_sync(0xffffffffu, run, here - 1);
        }
        if (csize > 1) cg::this_cluster().sync();
        else __syncthreads();
    }
    const float* gate = opt.gate ? (const float*)opt.gate + (size_t)t * opt.gate_ld : nullptr;
#pragma unroll
    for (int j = 0; j < kHeads; ++j) {
        const int item = gwarp + j * stride;
        if (item >= heads * kQ) continue;
        const int h = h0 + item / kQ, d = lane + 32 * (item % kQ);
        if (opt.sinks) {
            const float sk = opt.sinks[h], mn = fmaxf(Mx[j], sk), fo = expf(Mx[j] - mn);
            L[j] = L[j] * fo + expf(sk - mn);
            O[j] *= fo;
        }
        // (keys, but no score above minus infinity: undefined)
        float inv = L[j] > 0.0f ? 1.0f / L[j] : Mx[j] == -INFINITY && p >= 0 && !opt.sinks ? NAN : 0.0f;
        if (gate && !opt.gate_elements) inv *= 1.0f / (1.0f + expf(-gate[h]));
        if (d < dh) {
            float r = O[j] * inv;
            if (gate && opt.gate_elements) r *= 1.0f / (1.0f + expf(-gate[(size_t)h * dh + d]));
            out[(size_t)t * nh * dh + (size_t)h * dh + d] = r;
        }
    }
}

// Blocks of a cluster that share a token's units and the outputs of its merge (1, 2, 4 or 8), for `pairs` (token, key/value head,
// part of its heads): as many as one wave of blocks has room for, however short the contexts are (a token of 12 heads on 2 at
// 8 keys, one unit: 9.1 us with eight, whose warps share the merge, 12.6 with one).  (Eight below 128 pairs, one from there on: a
// prompt of 16 tokens of 28 heads on 4 took four waves of clusters, 44.4 us against 21.4 of the general kernel.)
int attention_f32_cluster(long long pairs, int dh) {
    const long long room = 148LL * (dh > 64 ? 1 : 2);                        // blocks at once, by shared memory and registers
    int c = 8;
    while (c > 1 && pairs * c > room) c /= 2;
    return c;
}

// heads a block: a key/value head's group in equal parts of at most eight
int heads_of(int nh, int nkv) {
    const int G = nh / nkv;
    return ceil_div(G, ceil_div(G, kHeads));
}

template <int NH>
int launch(const void* qkv, void* out, const void* kcache, const void* vcache, const int* block_table, int max_blocks, const int* seq_of_token,
           const int* positions, int T, int nh, int nkv, int dh, int page_size, int num_pages, float scale, int window, const AttentionOptions& opt,
           cudaStream_t stream) {
    const int groups = ceil_div(nh / nkv, NH);
    const int csize = attention_f32_cluster((long long)T * nkv * groups, dh);
    static LiOncePerDevice raised;
    cudaError_t e = li_raise_shared(raised, (const void*)attention_f32_kernel<NH>, shared_floats(kMaxDim) * sizeof(float));
    if (e != cudaSuccess) return li_fail("attention (float32): cannot raise shared memory: %s", cudaGetErrorString(e));
    li_launch_pdl(attention_f32_kernel<NH>, dim3(T, nkv * groups, csize), dim3(kThreads), shared_floats(dh) * sizeof(float), stream, dim3(1, 1, csize),
                  (const float*)qkv, (float*)out, (const float*)kcache, (const float*)vcache, block_table, max_blocks, seq_of_token, positions, nh, nkv, dh,
                  page_size, num_pages, scale, window, csize, opt);
    return li_check_launch("attention (float32)");
}

}  // namespace

bool li_attention_f32_accepts(const void* qkv, const void* kcache, const void* vcache, int nh, int nkv, int dh, int page_size, const AttentionOptions& opt) {
    return opt.maps == 1 && dh % 4 == 0 && dh <= kMaxDim && page_size % 16 == 0 && nkv * ceil_div(nh / nkv, heads_of(nh, nkv)) <= 65535 &&
           (uintptr_t)kcache % 16 == 0 && (uintptr_t)vcache % 16 == 0 && (uintptr_t)qkv % 4 == 0;
}

// For tests of the rule.
LI_EXPORT int li_attention_f32_blocks(int T, int nh, int nkv, int dh) {
    return attention_f32_cluster((long long)T * nkv * ceil_div(nh / nkv, heads_of(nh, nkv)), dh);
}

int li_attention_f32(const void* qkv, void* out, const void* kcache, const void* vcache, const int* block_table, int max_blocks, const int* seq_of_token,
                     const int* positions, int T, int nh, int nkv, int dh, int page_size, int num_pages, float scale, int window,
                     const AttentionOptions& opt, cudaStream_t stream) {
#define LI_CASE(N)                                                                                                                                  \
    case N:                                                                                                                                         \
        return launch<N>(qkv, out, kcache, vcache, block_table, max_blocks, seq_of_token, positions, T, nh, nkv, dh, page_size, num_pages, scale, window, \
                         opt, stream);
    switch (heads_of(nh, nkv)) { LI_CASE(1) LI_CASE(2) LI_CASE(3) LI_CASE(4) LI_CASE(5) LI_CASE(6) LI_CASE(7) LI_CASE(8) }
#undef LI_CASE
    return li_fail("attention (float32): %d heads on %d key/value heads", nh, nkv);
}

// Choosing the next token on the device: argmax, and temperature / top-k /
// top-p sampling, one block per logits row.
//
// Candidates as LitInfer's sampler keeps them (src/llaisys/models/qwen2.cpp:890-920):
// z = logits / temperature; the top_k largest if 0 < k < V; softmax over
// those; the shortest prefix, in descending order, whose cumulative
// probability reaches top_p if 0 < p < 1.  Instead of sorting, two thresholds
// over the order-preserving integer image of a float decide who stays:
//   t_k = smallest t with  #{z_i > t} < k                  (the k-th largest value)
//   t_p = smallest t with  sum_{z_i > t} prob_i < top_p    (a token stays iff the
//         probability mass of strictly larger candidates is below top_p)
// t_k comes from radix selection (three passes over the row with a histogram
// in shared memory); the values at or above it are gathered into shared
// memory in a fixed order, and t_p and the draw are found there.  Rows whose
// candidates do not fit (a flat distribution with top_p alone) and small
// vocabularies take bisection over the whole row, 32 passes a threshold.
// Equal values stay or go together.  The draw is Gumbel-max over the
// candidates, argmax(z_i + g_i), g_i = -log(-log(u_i)), with u_i a hash of
// (seed, index of the output token, i): exact sampling from the candidates'
// softmax that depends on nothing outside the request.  The first maximum wins
// ties (src/ops/argmax/op.cpp:28-33).  All sums are in a fixed order.
//
// Large vocabularies with a small top_k (sample_topk_kernel, the usual options): a cluster of blocks a row, one pass.  Each
// thread keeps the maximum of its elements; the k-th largest of a block's thread maxima is a bound below the row's
// k-th largest value, and only the few threads whose maximum reaches it are looked through again, by their whole warp.
// The candidates, the sums over them (the same order, so the same bits) and the draw are those of the general way,
// by which the cluster's first block does whatever row this leaves (NaN, too many equal values, other options).  64 rows
// of 151,936, top-k 50 and top-p 0.8: 20 us (two blocks a row); six passes by one block a row and 32 block-wide sums for
// the second threshold took 136 us.
#include "common.cuh"

#include <cooperative_groups.h>

namespace {

constexpr int kThreads = 1024;

__device__ __forceinline__ unsigned long long splitmix64(unsigned long long x) {
    x += 0x9E3779B97F4A7C15ull;
    x = (x ^ (x >> 30)) * 0xBF58476D1CE4E5B9ull;
    x = (x ^ (x >> 27)) * 0x94D049BB133111EBull;
    return x ^ (x >> 31);
}

__device__ __forceinline__ float gumbel(unsigned long long key, int token) {
    const unsigned long long bits = splitmix64(key ^ ((unsigned long long)token * 0xD1342543DE82EF95ull)) >> 41;   // 23 bits
    const float u = ((float)bits + 0.5f) * (1.0f / 8388608.0f);                                                    // in (0, 1), exact
    return -logf(-logf(u));
}

__device__ __forceinline__ unsigned sortable(float f) {
    const unsigned b = __float_as_uint(f);
    return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}

struct Best {
    float v;
    int i;
};

__device__ __forceinline__ Best better(Best a, Best b) {
    if (b.v > a.v || (b.v == a.v && b.i < a.i)) return b;
    return a;
}

__device__ Best block_best(Best x, Best* scratch /* 32 */) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = (blockDim.x + 31) >> 5;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        Best y;
        y.v = __shfl_xor_sync(0xffffffffu, x.v, o);
        y.i = __shfl_xor_sync(0xffffffffu, x.i, o);
        x = better(x, y);
    }
    __syncthreads();
    if (lane == 0) scratch[warp] = x;
    __syncthreads();
    Best r = (lane < nwarps) ? scratch[lane] : Best{-INFINITY, 0x7fffffff};
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        Best y;
        y.v = __shfl_xor_sync(0xffffffffu, r.v, o);
        y.i = __shfl_xor_sync(0xffffffffu, r.i, o);
        r = better(r, y);
    }
    return r;
}

// f(i, row[i]) for this thread's elements i = threadIdx.x, + blockDim.x, ... in ascending order, eight loads in flight:
// the row comes from L2, and one load at a time would wait out its latency each time
template <typename F>
__device__ __forceinline__ void for_each_element(const float* __restrict__ row, int V, F f) {
    constexpr int U = 8;
    int i = threadIdx.x;
    for (; i + (U - 1) * (int)blockDim.x < V; i += U * blockDim.x) {
        float v[U];
#pragma unroll
        for (int u = 0; u < U; ++u) v[u] = row[i + u * blockDim.x];
#pragma unroll
        for (int u = 0; u < U; ++u) f(i + u * (int)blockDim.x, v[u]);
    }
    for (; i < V; i += blockDim.x) f(i, row[i]);
}

__device__ Best row_argmax(const float* row, int V, Best* scratch) {
    Best b{-INFINITY, 0x7fffffff};
    // eight loads in flight per thread: the row comes from L2 and one load at a time would wait out its latency each time
    constexpr int U = 8;
    int i = threadIdx.x;
    for (; i + (U - 1) * (int)blockDim.x < V; i += U * blockDim.x) {
        float v[U];
#pragma unroll
        for (int u = 0; u < U; ++u) v[u] = row[i + u * blockDim.x];
#pragma unroll
        for (int u = 0; u < U; ++u)
            if (v[u] > b.v) b = Best{v[u], i + u * (int)blockDim.x};      // ascending index per thread: the first maximum stays
    }
    for (; i < V; i += blockDim.x) {
        const float v = row[i];
        if (v > b.v) b = Best{v, i};
    }
    b = block_best(b, scratch);
    if (b.i == 0x7fffffff) b.i = 0;             // a row of NaN or -inf
    return b;
}

__global__ void __launch_bounds__(kThreads) argmax_kernel(const float* __restrict__ logits, int* __restrict__ out, int V) {
    __shared__ Best scratch[32];
    pdl_launch_dependents();
    pdl_wait();
    const Best b = row_argmax(logits + (size_t)blockIdx.x * V, V, scratch);
    if (threadIdx.x == 0) out[blockIdx.x] = b.i;
}

// Few rows of a large vocabulary (decode): one CTA a row would read its 600 KB alone while the rest of the GPU waits.  A row
// is cut into kChunks pieces; the CTA that finishes a row last (a counter per row) picks the best of the pieces, the
// first maximum again: pieces are compared in ascending order of their indices.
constexpr int kChunks = 16;
constexpr int kChunkRows = 1024;                 // rows the static scratch below holds
__device__ Best g_chunk_best[kChunkRows * kChunks];
__device__ unsigned g_chunk_done[kChunkRows];    // zero between launches

__global__ void __launch_bounds__(256) argmax_chunks_kernel(const float* __restrict__ logits, int* __restrict__ out, int V) {
    __shared__ Best scratch[32];
    __shared__ int is_last;
    pdl_launch_dependents();
    pdl_wait();
    const int row = blockIdx.y, chunk = blockIdx.x;
    const int per = (((V + kChunks - 1) / kChunks) + 3) & ~3;
    const int lo = chunk * per, hi = min(V, lo + per);
    Best b{-INFINITY, 0x7fffffff};
    if (lo < hi) {
        b = row_argmax(logits + (size_t)row * V + lo, hi - lo, scratch);
        // a chunk without a finite maximum (all NaN or -inf) must not win with a made-up index
        if (!(b.v > -INFINITY)) b = Best{-INFINITY, 0x7fffffff};
        else b.i += lo;
    }
    if (threadIdx.x == 0) {
        g_chunk_best[row * kChunks + chunk] = b;
        __threadfence();
        is_last = atomicAdd(&g_chunk_done[row], 1u) == (unsigned)(kChunks - 1);
    }
    __syncthreads();
    if (!is_last || threadIdx.x != 0) return;
    __threadfence();
    Best r{-INFINITY, 0x7fffffff};
    for (int c = 0; c < kChunks; ++c) {
        const volatile Best* p = &g_chunk_best[row * kChunks + c];
        r = better(r, Best{p->v, p->i});
    }
    out[row] = r.i == 0x7fffffff ? 0 : r.i;      // a row of NaN or -inf
    g_chunk_done[row] = 0;                       // ready for the next launch on this stream
}

// The thresholds by bisection with a pass over the whole row per step (64 passes for top-k and top-p): for small
// vocabularies, and where the selection below cannot be used.
__device__ void sample_row_by_bisection(const float* __restrict__ row, int V, float temperature, int top_k, float top_p,
                                        unsigned long long seed, unsigned long long index, Best top, int* __restrict__ out_token,
                                        Best* scratch, float* fscratch) {
    const float zmax = top.v / temperature;
    unsigned keep_from = 0;                       // candidates: sortable(z_i) >= keep_from

    if (top_k > 0 && top_k < V) {
        unsigned lo = 0, hi = 0xFFFFFFFFu;
        while (lo < hi) {
            const unsigned mid = lo + ((hi - lo) >> 1);
            float cnt = 0.0f;                     // counts below 2^24 are exact in float
            for_each_element(row, V, [&](int, float x) { cnt += (sortable(x / temperature) > mid) ? 1.0f : 0.0f; });
            cnt = block_sum(cnt, fscratch);
            if (cnt < (float)top_k) hi = mid; else lo = mid + 1;
        }
        keep_from = lo;
    }
    if (top_p > 0.0f && top_p < 1.0f) {
        float z = 0.0f;
        for_each_element(row, V, [&](int, float x) {
            const float zi = x / temperature;
            if (sortable(zi) >= keep_from) z += expf(zi - zmax);
        });
        z = block_sum(z, fscratch);
        const float target = top_p * z;           // compare unnormalised masses with top_p * Z
        unsigned lo = keep_from, hi = 0xFFFFFFFFu;
        while (lo < hi) {
            const unsigned mid = lo + ((hi - lo) >> 1);
            float mass = 0.0f;
            for_each_element(row, V, [&](int, float x) {
                const float zi = x / temperature;
                if (sortable(zi) > mid) mass += expf(zi - zmax);
            });
            mass = block_sum(mass, fscratch);
            if (mass < target) hi = mid; else lo = mid + 1;
        }
        if (lo > keep_from) keep_from = lo;
    }
    const unsigned long long key = splitmix64(seed ^ splitmix64(index));
    Best b{-INFINITY, 0x7fffffff};
    for_each_element(row, V, [&](int i, float x) {
        const float zi = x / temperature;
        if (sortable(zi) >= keep_from) {
            const float v = zi + gumbel(key, i);
            if (v > b.v) b = Best{v, i};
        }
    });
    b = block_best(b, scratch);
    if (threadIdx.x == 0) *out_token = (b.i == 0x7fffffff) ? top.i : b.i;
}

// Temperature alone (no top-k, no top-p): the draw is one reduction, argmax(z_i + g_i) over the whole row, and is cut into
// pieces over many CTAs like argmax_chunks_kernel.  Rows with other options are left to sample_kernel (`handled` says which).
constexpr int kDrawChunks = 64;                  // the draw costs a hash and two logarithms per token: more, smaller pieces
__device__ Best g_draw_best[kChunkRows * kDrawChunks];
__device__ unsigned g_draw_done[kChunkRows];     // zero between launches

__global__ void __launch_bounds__(256) sample_temperature_chunks_kernel(const float* __restrict__ logits, const int* __restrict__ params,
                                                                        int* __restrict__ out, int V) {
    __shared__ Best scratch[32];
    __shared__ int is_last;
    pdl_launch_dependents();
    pdl_wait();
    const int row = blockIdx.y, chunk = blockIdx.x;
    const int* pr = params + row * 6;
    const float temperature = __int_as_float(pr[0]);
    const int top_k = pr[1];
    const float top_p = __int_as_float(pr[2]);
    const bool plain = temperature > 0.0f && !(top_k > 0 && top_k < V) && top_k != 1 && !(top_p > 0.0f && top_p < 1.0f);
    if (!plain) return;                                  // the whole grid row agrees
    const unsigned long long seed = (unsigned long long)(unsigned)pr[3] | ((unsigned long long)(unsigned)pr[4] << 32);
    const unsigned long long key = splitmix64(seed ^ splitmix64((unsigned long long)(long long)pr[5]));
    const int per = (((V + kDrawChunks - 1) / kDrawChunks) + 3) & ~3;
    const int lo = chunk * per, hi = min(V, lo + per);
    Best b{-INFINITY, 0x7fffffff};
    if (lo < hi) {
        for_each_element(logits + (size_t)row * V + lo, hi - lo, [&](int i, float x) {
            const float v = x / temperature + gumbel(key, lo + i);
            if (v > b.v) b = Best{v, lo + i};
        });
        b = block_best(b, scratch);
    }
    if (threadIdx.x == 0) {
        g_draw_best[row * kDrawChunks + chunk] = b;
        __threadfence();
        is_last = atomicAdd(&g_draw_done[row], 1u) == (unsigned)(kDrawChunks - 1);
    }
    __syncthreads();
    if (!is_last || threadIdx.x != 0) return;
    __threadfence();
    Best r{-INFINITY, 0x7fffffff};
    for (int c = 0; c < kDrawChunks; ++c) {
        const volatile Best* p = &g_draw_best[row * kDrawChunks + c];
        r = better(r, Best{p->v, p->i});
    }
    if (r.i != 0x7fffffff) out[row] = r.i;               // else (nothing finite) sample_kernel's answer stands: the first maximum
    g_draw_done[row] = 0;
}

__device__ __forceinline__ float unsortable(unsigned k) { return __uint_as_float((k & 0x80000000u) ? (k & 0x7FFFFFFFu) : ~k); }

// Large vocabularies.  The same candidates and the same draw with few passes over the row: the k-th largest value by
// radix selection on the sortable image of z (three passes: 11, 11 and 10 bits, a histogram in shared memory each), the
// candidates (at most kCand of them) gathered into shared memory in a fixed order, and top-p and the draw done there.
// With top-p alone the kCand largest are gathered first: if they hold at least top_p of the mass, the cut lies among them
// (a token below them has at least that mass above it); if not (a very flat distribution), the bisection above runs.
constexpr int kCand = 4096;

struct SelectShared {
    unsigned hist[2048];
    unsigned ckey[kCand];
    int cidx[kCand];
    unsigned scan[kThreads];
    unsigned warp_total[32];
    unsigned prefix, need;
};

// One round of the selection: among the keys that match `prefix` under `mask`, the digit (`bits` bits at `shift`) that
// holds the need-th largest; prefix and need are updated in shared memory.  extra(i, z, key) is called for every element.
template <typename Extra>
__device__ void select_round(const float* __restrict__ row, int V, float temperature, unsigned mask, int shift, int bits, SelectShared& sh,
                             Extra extra) {
    const int nb = 1 << bits;
    for (int i = threadIdx.x; i < nb; i += blockDim.x) sh.hist[i] = 0;
    __syncthreads();
    const unsigned prefix = sh.prefix;
    for_each_element(row, V, [&](int i, float x) {
        const float z = x / temperature;
        const unsigned key = sortable(z);
        extra(i, z, key);
        if ((key & mask) == prefix) atomicAdd(&sh.hist[(key >> shift) & (unsigned)(nb - 1)], 1u);       // integer counts: any order
    });
    __syncthreads();
    if (threadIdx.x < 32) {
        // lane l takes the digits nb - 1 - (per * l) downwards
        const int per = nb / 32, lane = threadIdx.x;
        unsigned mine = 0;
        for (int j = 0; j < per; ++j) mine += sh.hist[nb - 1 - (lane * per + j)];
        unsigned incl = mine;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned y = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += y;
        }
        const unsigned before = incl - mine, need = sh.need;
        if (before < need && need <= incl) {
            unsigned run = before;
            for (int j = 0; j < per; ++j) {
                const int d = nb - 1 - (lane * per + j);
                const unsigned c = sh.hist[d];
                if (run + c >= need) {
                    sh.prefix = prefix | ((unsigned)d << shift);
                    sh.need = need - run;
                    break;
                }
                run += c;
            }
        }
    }
    __syncthreads();
}

__device__ unsigned block_exclusive_scan(unsigned v, SelectShared& sh, unsigned* total) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    unsigned incl = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned y = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += y;
    }
    if (lane == 31) sh.warp_total[warp] = incl;
    __syncthreads();
    if (warp == 0) {
        const unsigned w = lane < (int)(blockDim.x >> 5) ? sh.warp_total[lane] : 0u;
        unsigned wi = w;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned y = __shfl_up_sync(0xffffffffu, wi, o);
            if (lane >= o) wi += y;
        }
        sh.warp_total[lane] = wi - w;                   // exclusive
        if (lane == 31) sh.scan[0] = wi;                // the total
    }
    __syncthreads();
    *total = sh.scan[0];
    const unsigned r = sh.warp_total[warp] + incl - v;
    __syncthreads();
    return r;
}

struct GeneralShared {
    Best scratch[32];
    float fscratch[32];
    SelectShared select;
};

// A row by one block, whatever its options.  chunked_plain: rows with temperature alone are drawn by
// sample_temperature_chunks_kernel, launched behind; here they only get the first maximum as a stand-in (which stays if the
// row has nothing finite).
__device__ __noinline__ void sample_row(const float* __restrict__ row, const int* __restrict__ pr, int* __restrict__ out, int V, int chunked_plain, GeneralShared& gs) {
    Best* scratch = gs.scratch;
    float* fscratch = gs.fscratch;
    SelectShared& sh = gs.select;
    const float temperature = __int_as_float(pr[0]);
    const int top_k = pr[1];
    const float top_p = __int_as_float(pr[2]);
    const unsigned long long seed = (unsigned long long)(unsigned)pr[3] | ((unsigned long long)(unsigned)pr[4] << 32);
    const unsigned long long index = (unsigned long long)(long long)pr[5];

    const bool use_k = top_k > 0 && top_k < V, use_p = top_p > 0.0f && top_p < 1.0f;
    if (chunked_plain && temperature > 0.0f && top_k != 1 && !use_k && !use_p) {
        if (threadIdx.x == 0) *out = 0;                // stands only if the row has nothing finite (what the first maximum would give)
        return;
    }
    const Best top = row_argmax(row, V, scratch);
    if (temperature <= 0.0f || top_k == 1) {
        if (threadIdx.x == 0) *out = top.i;
        return;
    }
    if (V <= kCand || !(use_k || use_p) || (use_k && top_k > kCand)) {
        sample_row_by_bisection(row, V, temperature, top_k, top_p, seed, index, top, out, scratch, fscratch);
        return;
    }
    const float zmax = top.v / temperature;
    // the k-th largest key (top-k), or the kCand-th largest (top-p alone)
    if (threadIdx.x == 0) {
        sh.prefix = 0;
        sh.need = use_k ? (unsigned)top_k : (unsigned)kCand;
    }
    __syncthreads();
    float zsum = 0.0f;                                   // over the whole row, for top-p alone: sum of exp(z - zmax) in a fixed order
    select_round(row, V, temperature, 0u, 21, 11, sh, [&](int, float z, unsigned) { zsum += expf(z - zmax); });
    select_round(row, V, temperature, 0xFFE00000u, 10, 11, sh, [](int, float, unsigned) {});
    select_round(row, V, temperature, 0xFFFFFC00u, 0, 10, sh, [](int, float, unsigned) {});
    const unsigned kth = sh.prefix;
    // candidates: keys >= the k-th largest (top-k: equal values stay together), keys > the kCand-th largest (top-p alone)
    const unsigned low = use_k ? kth : kth + 1u;          // kth < 0xFFFFFFFF: it is the key of a finite or infinite float, never all ones
    unsigned mine = 0;
    for_each_element(row, V, [&](int, float x) { mine += sortable(x / temperature) >= low ? 1u : 0u; });
    unsigned total = 0;
    unsigned at = block_exclusive_scan(mine, sh, &total);
    if (total > (unsigned)kCand || total == 0) {          // more equal values than fit, or nothing finite: the slow way decides
        sample_row_by_bisection(row, V, temperature, top_k, top_p, seed, index, top, out, scratch, fscratch);
        return;
    }
    for_each_element(row, V, [&](int i, float x) {
        const unsigned key = sortable(x / temperature);
        if (key >= low) {
            sh.ckey[at] = key;
            sh.cidx[at] = i;
            ++at;
        }
    });
    __syncthreads();
    const int C = (int)total;
    unsigned keep_from = low;
    if (use_p) {
        float zc = 0.0f;
        for (int j = threadIdx.x; j < C; j += blockDim.x) zc += expf(unsortable(sh.ckey[j]) - zmax);
        zc = block_sum(zc, fscratch);
        float target;
        if (use_k) {
            target = top_p * zc;                          // the mass after top-k
        } else {
            const float zall = block_sum(zsum, fscratch);
            target = top_p * zall;
            if (!(zc >= target)) {                        // the gathered tokens hold less than top_p of the mass: the cut is below them
                sample_row_by_bisection(row, V, temperature, top_k, top_p, seed, index, top, out, scratch, fscratch);
                return;
            }
        }
        unsigned lo = low, hi = 0xFFFFFFFFu;
        while (lo < hi) {
            const unsigned mid = lo + ((hi - lo) >> 1);
            float mass = 0.0f;
            for (int j = threadIdx.x; j < C; j += blockDim.x) {
                const unsigned key = sh.ckey[j];
                if (key > mid) mass += expf(unsortable(key) - zmax);
            }
            mass = block_sum(mass, fscratch);
            if (mass < target) hi = mid; else lo = mid + 1;
        }
        if (lo > keep_from) keep_from = lo;
    }
    const unsigned long long key = splitmix64(seed ^ splitmix64(index));
    Best b{-INFINITY, 0x7fffffff};
    for (int j = threadIdx.x; j < C; j += blockDim.x) {
        const unsigned kj = sh.ckey[j];
        if (kj >= keep_from) {
            const int i = sh.cidx[j];
            const float v = unsortable(kj) + gumbel(key, i);
            if (v > b.v || (v == b.v && i < b.i)) b = Best{v, i};
        }
    }
    b = block_best(b, scratch);
    if (threadIdx.x == 0) *out = (b.i == 0x7fffffff) ? top.i : b.i;
}

// The rows that sample_topk_kernel looks at: a vocabulary that leaves most threads of its blocks something, and a top_k whose
// candidates are few.  A block's bound, the top_k-th largest of its threads' maxima, is reached by a little more than top_k
// of its elements, and the largest of the blocks' bounds by as many of every other block's: about blocks x top_k
// candidates, of which there is room for 1,024.  Each is ranked against all: beyond an element in forty of the row the general
// way is as fast, and a large top_k of a small vocabulary is not worth its cut at top_p.  Measured, general way / this one,
// us: 16,384 x 8 rows, top_k 50, top_p 0.8 35.2 / 27.7, top_k 128 21.8 / 65; 32,000 x 33 rows, top_k 256, top_p 0.9 49 / 59;
// 151,936 x 8 rows, top_k 128 121 / 65, top_k 256 (2,300 candidates, so both ways one after the other) 134 / 150.
constexpr int kFastK = 256, kFastCand = 1024, kFastVocab = 16384;
__device__ __forceinline__ bool fast_options(float temperature, int top_k, int V, int blocks) {
    return temperature > 0.0f && top_k > 1 && top_k <= kFastK && V >= kFastVocab && top_k <= V / 160 && blocks * top_k <= min(V / 40, kFastCand);
}

struct FastShared {
    unsigned key[kFastCand], okey[kFastCand];
    int idx[kFastCand], oidx[kFastCand];
    float e[kFastCand];
    float x[kFastCand];
    unsigned count, keep, keep_from;
    float bound;                                          // this block's bound below the k-th largest (NaN: the row has one)
    float fscratch[32];
    Best scratch[32];
};

// A row by the cluster's blocks in one pass if its options are such and the pass settles it, else by the first block alone
// (sample_row), in the same launch.  A caller that knows of no such row does not launch it (li_sample_rows): its blocks
// are in the way of the kernels around them (8 rows of 151,936 with temperature alone: 12.6 us without, 18.2 with).
// leave: rows that the pass does not settle get -1 instead.
template <bool kVec>
__global__ void __launch_bounds__(kThreads) sample_topk_kernel(const float* __restrict__ logits, const int* __restrict__ params, int* __restrict__ out, int V,
                                                               int chunked_plain, int leave) {
    namespace cg = cooperative_groups;
    __shared__ union Shared {
        FastShared fast;
        GeneralShared general;
        __device__ Shared() {}
    } shared;
    FastShared& sh = shared.fast;
    cg::cluster_group cluster = cg::this_cluster();
    pdl_launch_dependents();
    pdl_wait();
    const int blocks = (int)gridDim.x, rank = (int)blockIdx.x, r = (int)blockIdx.y;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int* pr = params + r * 6;
    const float temperature = __int_as_float(pr[0]);
    const int top_k = pr[1];
    const float top_p = __int_as_float(pr[2]);
    const float* row = logits + (size_t)r * V;
    auto otherwise = [&]() {                              // (called by the whole first block, once no other block looks at its memory)
        if (leave) {
            if (tid == 0) out[r] = -1;
            return;
        }
        __syncthreads();
        sample_row(row, pr, out + r, V, chunked_plain, shared.general);
    };
    if (!fast_options(temperature, top_k, V, blocks)) {           // (the whole cluster agrees)
        if (rank == 0) otherwise();
        return;
    }
    const int per = ((V + blocks - 1) / blocks + 3) & ~3;
    const int lo = min(V, rank * per), hi = min(V, lo + per);
    // a thread's elements: four in a row at 4 (tid + 1024 j)
    auto load4 = [&](int i) {
        float4 v = make_float4(-INFINITY, -INFINITY, -INFINITY, -INFINITY);
        if constexpr (kVec) {
            if (i < hi) v = __ldcg(reinterpret_cast<const float4*>(row + i));
        } else {
            if (i < hi) v.x = __ldcg(row + i);
            if (i + 1 < hi) v.y = __ldcg(row + i + 1);
            if (i + 2 < hi) v.z = __ldcg(row + i + 2);
            if (i + 3 < hi) v.w = __ldcg(row + i + 3);
        }
        return v;
    };
    if (tid == 0) sh.count = 0, sh.keep = 0, sh.keep_from = 0xFFFFFFFFu;
    float mx = -INFINITY;
    bool odd = false;
    constexpr int U = 8;
    for (int i0 = lo + 4 * tid; i0 < hi; i0 += U * 4 * kThreads) {
        float4 v[U];
#pragma unroll
        for (int u = 0; u < U; ++u) v[u] = load4(i0 + u * 4 * kThreads);
#pragma unroll
        for (int u = 0; u < U; ++u) {
            mx = fmaxf(mx, fmaxf(fmaxf(v[u].x, v[u].y), fmaxf(v[u].z, v[u].w)));
            odd |= (v[u].x != v[u].x) | (v[u].y != v[u].y) | (v[u].z != v[u].z) | (v[u].w != v[u].w);
        }
    }
    // the top_k-th largest of the block's thread maxima
    const unsigned mkey = sortable(mx);
    unsigned a = 0, b = 0xFFFFFFFFu;
    while (a < b) {
        const unsigned mid = a + ((b - a) >> 1);
        if (__syncthreads_count(mkey > mid) < top_k) b = mid;
        else a = mid + 1;
    }
    const bool any_odd = __syncthreads_or(odd);
    if (tid == 0) sh.bound = any_odd ? __int_as_float(0x7fc00000) : unsortable(a);
    cluster.sync();
    float bound = -INFINITY;
    bool give_up = false;
    for (int k = 0; k < blocks; ++k) {
        const float o = *cluster.map_shared_rank(&sh.bound, k);
        give_up |= o != o;
        bound = fmaxf(bound, o);
    }
    // Candidates are chosen by z = x / temperature, which may round different x together: elements a few units in the last
    // place below the bound are looked at too.  (Where z overflows or becomes so small that more falls together, or the bound
    // says nothing, the general kernel decides.)
    const float zb = fabsf(bound / temperature);
    give_up |= !(fabsf(bound) < INFINITY) || !(zb < 1e30f) || (bound != 0.0f && zb < 1e-30f) || (bound == 0.0f && !(temperature < 1e30f));
    const float from = bound - fabsf(bound) * 1e-6f;
    if (!give_up) {
        FastShared* first = cluster.map_shared_rank(&sh, 0);
        unsigned flagged = __ballot_sync(0xffffffffu, mx >= from);
        while (flagged) {
            const int l = __ffs(flagged) - 1;
            flagged &= flagged - 1;
            const int t = (tid & ~31) + l;
            for (int i = lo + 4 * t + lane * 4 * kThreads; i < hi; i += 32 * 4 * kThreads) {
                const float4 v = load4(i);
                const float x[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
                for (int q = 0; q < 4; ++q)
                    if (x[q] >= from && i + q < hi) {
                        const unsigned at = atomicAdd(&first->count, 1u);
                        if (at < (unsigned)kFastCand) first->x[at] = x[q], first->idx[at] = i + q;
                    }
            }
        }
    }
    cluster.sync();
    if (rank != 0) return;
    const int n = (int)sh.count;
    if (give_up || n > kFastCand || n < top_k) {          // (uniform)
        otherwise();
        return;
    }
    const unsigned key = tid < n ? sortable(sh.x[tid] / temperature) : 0u;
    const int idx = tid < n ? sh.idx[tid] : 0;
    sh.key[tid] = key;
    __syncthreads();
    int above = 0;
    for (int j = 0; j < n; ++j) above += sh.key[j] > key ? 1 : 0;
    const bool stays = tid < n && above < top_k;          // the k-th largest and what equals it stay together
    __syncthreads();
    sh.idx[tid] = stays ? idx : -1;
    __syncthreads();
    // in the order of the general kernel: by the element's place modulo 1024, then by the element
    if (stays) {
        int before = 0;
        for (int j = 0; j < n; ++j) {
            const int o = sh.idx[j];
            before += (o >= 0 && ((o & (kThreads - 1)) < (idx & (kThreads - 1)) || ((o & (kThreads - 1)) == (idx & (kThreads - 1)) && o < idx))) ? 1 : 0;
        }
        sh.okey[before] = key;
        sh.oidx[before] = idx;
    }
    const int C = __syncthreads_count(stays);
    const unsigned mine = tid < C ? sh.okey[tid] : 0u;
    // the largest of all: z of the row's maximum
    if (tid < C) atomicMax(&sh.keep, mine);
    __syncthreads();
    const float zmax = unsortable(sh.keep);
    unsigned keep_from = 0;
    if (top_p > 0.0f && top_p < 1.0f) {
        const float e = tid < C ? expf(unsortable(mine) - zmax) : 0.0f;
        sh.e[tid] = e;
        const float target = top_p * block_sum(e, sh.fscratch);      // (its barriers also publish sh.e)
        // The smallest threshold whose mass above it is below the target is one of the candidates' keys: a warp a key, its
        // sum in the order of block_sum.
        for (int j = warp; j < C; j += kThreads / 32) {
            const unsigned t = sh.okey[j];
            float part = 0.0f;
            for (int g = 0; 32 * g < C; ++g) {
                const int q = 32 * g + lane;
                const float v = warp_sum(q < C && sh.okey[q] > t ? sh.e[q] : 0.0f);
                if (lane == g) part = v;
            }
            const float mass = warp_sum(part);
            if (lane == 0 && mass < target) atomicMin(&sh.keep_from, t);
        }
        __syncthreads();
        keep_from = sh.keep_from;
    }
    const unsigned long long seed = (unsigned long long)(unsigned)pr[3] | ((unsigned long long)(unsigned)pr[4] << 32);
    const unsigned long long hash = splitmix64(seed ^ splitmix64((unsigned long long)(long long)pr[5]));
    Best best{-INFINITY, 0x7fffffff};
    if (tid < C && mine >= keep_from) {
        const float v = unsortable(mine) + gumbel(hash, sh.oidx[tid]);
        if (v > best.v) best = Best{v, sh.oidx[tid]};
    }
    best = block_best(best, sh.scratch);
    if (tid == 0) sh.count = best.i == 0x7fffffff;
    __syncthreads();
    if (sh.count) otherwise();                            // no candidate has a number
    else if (tid == 0) out[r] = best.i;
}

__global__ void __launch_bounds__(kThreads) sample_kernel(const float* __restrict__ logits, const int* __restrict__ params,
                                                          int* __restrict__ out, int V, int chunked_plain) {
    __shared__ GeneralShared sh;
    pdl_launch_dependents();
    pdl_wait();
    sample_row(logits + (size_t)blockIdx.x * V, params + blockIdx.x * 6, out + blockIdx.x, V, chunked_plain, sh);
}

int g_leave = 0;

}  // namespace

// 1: rows that the one pass of sample_topk_kernel does not settle get -1.  For tests.
LI_EXPORT void li_sample_leave_rows(int on) { g_leave = on; }

LI_EXPORT int li_argmax(const float* logits, int* out, int R, int V, cudaStream_t stream) {
    LI_REQUIRE(R >= 0 && V > 0, "argmax: bad sizes R=%d V=%d", R, V);
    if (R == 0) return 0;
    if (R <= 64 && R <= kChunkRows && V >= 16384) {
        li_launch_pdl(argmax_chunks_kernel, dim3(kChunks, R), dim3(256), 0, stream, logits, out, V);
        return li_check_launch("argmax (chunks)");
    }
    li_launch_pdl(argmax_kernel, dim3(R), dim3(kThreads), 0, stream, logits, out, V);
    return li_check_launch("argmax");
}

// rows, what the caller knows of them: bit 0 whether some row may have a top_k of 2 to 256 (else its kernel is not launched), bit 1
// that none has temperature as its only option (else a row of a large vocabulary is drawn by a kernel of its own, 5 us that
// the launch costs where there is no such row).
LI_EXPORT int li_sample_rows(const float* logits, const int* params, int* out, int R, int V, int rows, cudaStream_t stream) {
    const bool small_top_k = rows & 1, none_alone = rows & 2;
    LI_REQUIRE(R >= 0 && V > 0, "sample: bad sizes R=%d V=%d", R, V);
    LI_REQUIRE(V < (1 << 24), "sample: vocabulary %d is too large", V);
    if (R == 0) return 0;
    // few rows of a large vocabulary: rows with temperature alone are drawn over many CTAs by a second kernel
    const int chunked_plain = (R <= 64 && R <= kChunkRows && V >= 16384) ? 1 : 0;
    // rows with a small top-k: two to eight blocks a row, as many as there is room for at once, a block a multiprocessor (15 clusters
    // of eight, 33 of four, 74 of two; 16 rows in clusters of eight: 24 us, of four 15)
    if (R <= 64 && V >= kFastVocab && small_top_k) {
        const int blocks = R > 32 ? 2 : R > 15 ? 4 : 8;
        if (V % 4 == 0 && (uintptr_t)logits % 16 == 0)
            li_launch_pdl(sample_topk_kernel<true>, dim3(blocks, R), dim3(kThreads), 0, stream, dim3(blocks, 1, 1), logits, params, out, V, chunked_plain, g_leave);
        else
            li_launch_pdl(sample_topk_kernel<false>, dim3(blocks, R), dim3(kThreads), 0, stream, dim3(blocks, 1, 1), logits, params, out, V, chunked_plain, g_leave);
    } else {
        li_launch_pdl(sample_kernel, dim3(R), dim3(kThreads), 0, stream, logits, params, out, V, chunked_plain);
    }
    if (int rc = li_check_launch("sample")) return rc;
    if (chunked_plain && !none_alone) {
        li_launch_pdl(sample_temperature_chunks_kernel, dim3(kDrawChunks, R), dim3(256), 0, stream, logits, params, out, V);
        return li_check_launch("sample (temperature, chunks)");
    }
    return 0;
}

LI_EXPORT int li_sample(const float* logits, const int* params, int* out, int R, int V, cudaStream_t stream) {
    return li_sample_rows(logits, params, out, R, V, 1, stream);
}

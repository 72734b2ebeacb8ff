// The two chunk passes of li_decay_scan and li_ssm_scan (recurrent.cu) as products of small matrices, for chunks of up to 64 tokens,
// keys (state sizes) of up to 128 and values in tiles of 128 columns.
//
// Walked token by token, a chunk's outputs cost a reduction over a warp a token and eight columns, and its tokens come through shared
// memory sixteen at a time (777 tokens, 12 heads of 128: 35 us from zeros, 53 us with outputs; 48 heads of 64 with a state of 128:
// 62 and 87).  With w(t, s) the product of the decays behind s up to t (and the step size of s), the same values are
//     end state   U[c, i] = sum over s of w(n - 1, s) v_s[c] k_s[i]
//     outputs     o_t[c]  = w(t, start) sum over i of q_t[i] S[c, i]  +  sum over s <= t of w(t, s) (q_t . k_s) v_s[c]
// that is products of a chunk's rows with each other, with the state it starts from and with its values, all in float with packed
// multiply-adds.  A block of 256 threads takes a chunk of a head's 128 value columns (two heads of 64, which share B and C); 8 x 8
// outputs a thread for the end state, 4 x 8 for the outputs (the two passes: 18 and 40 us, 24 and 58), operands along the summed index so that pairs of it are the packed
// pairs.  What bounds them is shared-memory reads (a 16-byte read of a warp takes four cycles, whatever the lanes share).
// w comes from sums of logarithms in double, or from powers of the head's one decay.
#include "common.cuh"

#include <type_traits>

namespace {

constexpr int kTokens = 64, kCols = 128, kThreads = 256, kDim = 128;
constexpr int kRow = kDim + 4, kPiece = 32, kPieceRow = kPiece + 4, kTokRow = kTokens + 4;      // floats a row: a multiple of four, odd in fours

// x / (1 + e^-x).  The quotient by the fast reciprocal and one step of Newton's method (within two units in the last place of the exact
// quotient): with the division the activations of a chunk's rows took longer than its products.
__device__ __forceinline__ float silu_f(float x) {
    const float d = 1.0f + fminf(expf(-x), 1e37f);
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(d));
    return x * fmaf(r, fmaf(-d, r, 1.0f), r);
}
__device__ __forceinline__ float softplus_f(float x) { return fmaxf(x, 0.0f) + log1pf(expf(-fabsf(x))); }

__device__ __forceinline__ unsigned long long pack2(float lo, float hi) {
    unsigned long long r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ float2 unpack2(unsigned long long v) {
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
    return r;
}
__device__ __forceinline__ void fma2(unsigned long long& d, unsigned long long a, unsigned long long b) {
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(d) : "l"(a), "l"(b));
}
__device__ __forceinline__ ulonglong2 pair4(const float* p) { return *reinterpret_cast<const ulonglong2*>(p); }

// Where the rows of a launch lie.  Head h's keys, queries and values are columns k_off + h k_step .. of the row of a token (for the
// state-space form of its group); values and outputs of a tile lie side by side from column 128 tile on.
template <typename T>
struct Source {
    const T* rows;
    int stride, q_off, k_off, v_off, d, heads, dv;
    int per_group;                       // state space: heads that share keys and queries
    const T* dt_raw;
    int dt_stride;
    const float *dt_bias, *A_log, *skip, *decay;
};

template <typename T, bool kSsm>
struct Chunk {
    int q0, n, index;                    // first token, tokens, number
    int head, heads_here, col0, cols;    // first head, heads of the tile, first column among all heads', columns
    const T *q, *k, *v;                  // of the first token
    __device__ Chunk(const Source<T>& s, const int* __restrict__ seg) {
        const int4 sg = reinterpret_cast<const int4*>(seg)[blockIdx.z];
        q0 = sg.x, n = min(kTokens, sg.y - sg.x), index = sg.z;
        if constexpr (kSsm) {
            heads_here = kCols / s.dv;
            head = (int)blockIdx.y * heads_here;
            col0 = (int)blockIdx.y * kCols;
            cols = kCols;
        } else {
            heads_here = 1;
            head = (int)blockIdx.y;
            col0 = head * s.dv + (int)blockIdx.x * kCols;
            cols = min(kCols, s.dv - (int)blockIdx.x * kCols);
        }
        const int kh = kSsm ? head / s.per_group : head;
        const T* row = s.rows + (size_t)q0 * s.stride;
        q = row + s.q_off + kh * s.d;
        k = row + s.k_off + kh * s.d;
        v = row + s.v_off + col0;
    }
    static __device__ bool wide(const T* p, int stride) { return ((uintptr_t)p & 15) == 0 && stride * sizeof(T) % 16 == 0; }
};

// Eight neighbouring elements of a token's row, `left` of them there, as floats; 16 bytes at a time where the rows allow.
constexpr int kVec = 8;
template <typename T, bool kSsm>
__device__ __forceinline__ void load8(float (&x)[kVec], const T* p, int left, bool wide) {
    if (wide && left >= kVec) {
        constexpr int kPieces = kVec * sizeof(T) / 16;
        uint4 raw[kPieces];
#pragma unroll
        for (int i = 0; i < kPieces; ++i) raw[i] = __ldg(reinterpret_cast<const uint4*>(p) + i);
        const T* e = reinterpret_cast<const T*>(raw);
#pragma unroll
        for (int i = 0; i < kVec; ++i) x[i] = to_float(e[i]);
    } else {
#pragma unroll
        for (int i = 0; i < kVec; ++i) x[i] = i < left ? to_float(p[i]) : 0.0f;
    }
}
template <bool kSsm>
__device__ __forceinline__ void activate(float (&x)[kVec], int left) {
    if constexpr (!kSsm) {
#pragma unroll
        for (int i = 0; i < kVec; ++i) x[i] = i < left ? silu_f(x[i]) : 0.0f;
    }
}
// Rows of 128 elements of a chunk's tokens, four pieces of eight a thread, all asked for before the first is used.
template <typename T, bool kSsm, typename Put>
__device__ __forceinline__ void stage_rows(const T* rows, int stride, int n, int width, bool wide, bool by_token, Put put) {
    constexpr int kEach = kTokens * kDim / kVec / kThreads;
    float x[kEach][kVec];
    auto place = [&](int r, int& t, int& i) {
        const int e = (int)threadIdx.x + kThreads * r;
        // (by_token: neighbouring lanes on neighbouring tokens, for the transposed form)
        t = by_token ? e % kTokens : e / (kDim / kVec);
        i = kVec * (by_token ? e / kTokens : e % (kDim / kVec));
    };
#pragma unroll
    for (int r = 0; r < kEach; ++r) {
        int t, i;
        place(r, t, i);
        load8<T, kSsm>(x[r], rows + (size_t)(t < n ? t : 0) * stride + i, t < n ? width - i : 0, wide);
    }
#pragma unroll
    for (int r = 0; r < kEach; ++r) {
        int t, i;
        place(r, t, i);
        activate<kSsm>(x[r], t < n ? width - i : 0);
        put(t, i, x[r]);
    }
}
__device__ __forceinline__ void put8(float* to, const float (&x)[kVec]) {
    *reinterpret_cast<float4*>(to) = make_float4(x[0], x[1], x[2], x[3]);
    *reinterpret_cast<float4*>(to + 4) = make_float4(x[4], x[5], x[6], x[7]);
}

// Per head of the tile: w(t, start) of every token, and what w(t, s) is made of.  Decay: powers of it.
struct Weights {
    float power[kTokens + 1];
    double log_sum[2][kTokens];          // of the decays up to a token
    float dt[2][kTokens];
};

template <typename T, bool kSsm>
__device__ __forceinline__ void make_weights(Weights& w, const Source<T>& s, const Chunk<T, kSsm>& c) {
    if constexpr (kSsm) {
        const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
        if (warp < c.heads_here) {
            const int h = c.head + warp;
            const float rate = expf(s.A_log[h]), bias = s.dt_bias[h];
            double a[2];
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const int t = 2 * lane + e;
                const float dt = t < c.n ? softplus_f(to_float(s.dt_raw[(size_t)(c.q0 + t) * s.dt_stride + h]) + bias) : 0.0f;
                w.dt[warp][t] = dt;
                const double x = (double)rate * (double)dt;
                a[e] = -(x > 1e30 ? 1e30 : x);             // (a decay to nothing: differences stay numbers)
            }
            double run = a[0] + a[1];
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const double before = __shfl_up_sync(0xffffffffu, run, o);
                if (lane >= o) run += before;
            }
            w.log_sum[warp][2 * lane] = run - a[1];
            w.log_sum[warp][2 * lane + 1] = run;
        }
    } else if (threadIdx.x <= kTokens) {
        w.power[threadIdx.x] = powf(s.decay[c.head], (float)(int)threadIdx.x);
    }
}
// w(t, s), s <= t < n; hh: which of the tile's heads
template <bool kSsm>
__device__ __forceinline__ float weight(const Weights& w, int hh, int t, int s) {
    if constexpr (kSsm) return expf((float)(w.log_sum[hh][t] - w.log_sum[hh][s])) * w.dt[hh][s];
    else return w.power[t - s];
}
template <bool kSsm>
__device__ __forceinline__ float weight_from_start(const Weights& w, int hh, int t) {
    if constexpr (kSsm) return expf((float)w.log_sum[hh][t]);
    else return w.power[t + 1];
}

template <typename T, bool kSsm>
__global__ void __launch_bounds__(kThreads, 2)
chunk_end_kernel(const Source<T> src, const int* __restrict__ seg, float* __restrict__ chunk_state, float* __restrict__ chunk_decay) {
    extern __shared__ float4 raw[];
    float* ks = reinterpret_cast<float*>(raw);             // [token][element]
    float* vs = ks + kTokens * kRow;                       // [token][column], weighted
    Weights& w = *reinterpret_cast<Weights*>(vs + kTokens * kRow);
    pdl_launch_dependents();
    pdl_wait();
    const Chunk<T, kSsm> c(src, seg);
    if (c.n <= 0) return;
    const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
    make_weights<T, kSsm>(w, src, c);
    stage_rows<T, kSsm>(c.k, src.stride, c.n, src.d, c.wide(c.k, src.stride), false, [&](int s, int i, const float (&x)[kVec]) { put8(ks + s * kRow + i, x); });
    __syncthreads();
    // (a weight a row and head; what lies behind the last token stays out of the sums)
    stage_rows<T, kSsm>(c.v, src.stride, c.n, c.cols, c.wide(c.v, src.stride), false, [&](int s, int j, const float (&x)[kVec]) {
        const float f = s < c.n ? weight<kSsm>(w, kSsm && j >= src.dv ? 1 : 0, c.n - 1, s) : 0.0f;
        float y[kVec];
#pragma unroll
        for (int i = 0; i < kVec; ++i) y[i] = x[i] * f;
        put8(vs + s * kRow + j, y);
    });
    if constexpr (kSsm)
        if (tid < c.heads_here) chunk_decay[(size_t)c.index * src.heads + c.head + tid] = weight_from_start<kSsm>(w, tid, c.n - 1);
    __syncthreads();
    // columns 4 ty .. and 64 + 4 ty .., elements 4 tx .. and 64 + 4 tx ..
    unsigned long long acc[8][4];
#pragma unroll
    for (int a = 0; a < 8; ++a)
#pragma unroll
        for (int b = 0; b < 4; ++b) acc[a][b] = 0ull;
#pragma unroll 2
    for (int s = 0; s < c.n; ++s) {
        const ulonglong2 k0 = pair4(ks + s * kRow + 4 * tx), k1 = pair4(ks + s * kRow + 64 + 4 * tx);
        const float4 v0 = *reinterpret_cast<const float4*>(vs + s * kRow + 4 * ty), v1 = *reinterpret_cast<const float4*>(vs + s * kRow + 64 + 4 * ty);
        const float v[8] = {v0.x, v0.y, v0.z, v0.w, v1.x, v1.y, v1.z, v1.w};
#pragma unroll
        for (int a = 0; a < 8; ++a) {
            const unsigned long long vv = pack2(v[a], v[a]);
            fma2(acc[a][0], vv, k0.x), fma2(acc[a][1], vv, k0.y), fma2(acc[a][2], vv, k1.x), fma2(acc[a][3], vv, k1.y);
        }
    }
    float* to = chunk_state + ((size_t)c.index * src.heads * src.dv + c.col0) * src.d;       // [column][element]
#pragma unroll
    for (int a = 0; a < 8; ++a) {
        const int j = (a >> 2) * 64 + 4 * ty + (a & 3);
#pragma unroll
        for (int half = 0; half < 2; ++half) {
            const int i = 64 * half + 4 * tx;
            const float2 x = unpack2(acc[a][2 * half]), y = unpack2(acc[a][2 * half + 1]);
            if (j < c.cols && i < src.d) *reinterpret_cast<float4*>(to + (size_t)j * src.d + i) = make_float4(x.x, x.y, y.x, y.y);
        }
    }
}

// Shared memory of the pass with outputs: queries (then values, transposed), keys (then pieces of the state), the weighted scores.
template <bool kSsm>
struct OutputSmem {
    static constexpr int kHeads = kSsm ? 2 : 1;
    float a[kCols * kTokRow];            // [token][element], later [column][token]
    float b[kTokens * kRow];             // [token][element], later [column][element of a piece]
    float p[kHeads][kTokens * kTokRow];  // [token][earlier token]
    Weights w;
};

template <typename T, bool kSsm>
__global__ void __launch_bounds__(kThreads, 2)
chunk_output_kernel(const Source<T> src, const int* __restrict__ seg, const float* __restrict__ chunk_state, float* __restrict__ out) {
    extern __shared__ float4 raw[];
    OutputSmem<kSsm>& sm = *reinterpret_cast<OutputSmem<kSsm>*>(raw);
    pdl_launch_dependents();
    pdl_wait();
    const Chunk<T, kSsm> c(src, seg);
    if (c.n <= 0) return;
    const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;          // tokens ty + 16 a, columns tx + 16 b
    make_weights<T, kSsm>(sm.w, src, c);
    stage_rows<T, kSsm>(c.q, src.stride, c.n, src.d, c.wide(c.q, src.stride), false, [&](int t, int i, const float (&x)[kVec]) { put8(sm.a + t * kRow + i, x); });
    stage_rows<T, kSsm>(c.k, src.stride, c.n, src.d, c.wide(c.k, src.stride), false, [&](int t, int i, const float (&x)[kVec]) { put8(sm.b + t * kRow + i, x); });
    // the state, 32 elements of every column at a time: asked for a piece ahead
    const float* state = chunk_state + ((size_t)c.index * src.heads * src.dv + c.col0) * src.d;
    float4 ahead[4];
    auto ask = [&](int piece) {
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            const int e = tid + kThreads * r, j = e >> 3, i = piece * kPiece + 4 * (e & 7);
            ahead[r] = j < c.cols && i < src.d ? __ldg(reinterpret_cast<const float4*>(state + (size_t)j * src.d + i)) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        }
    };
    ask(0);
    __syncthreads();
    // Blocks of sixteen tokens that the chunk has: the last chunk of a portion may have few (777 tokens of 48 heads of 64: 312 blocks, 24 of
    // them of nine tokens, for 296 places: 68 - 79 -> 58 us).
    auto with_blocks = [&](auto blocks) {
        constexpr int A = decltype(blocks)::value;
        {
            // scores of a token with the earlier ones, weighted: blocks of sixteen tokens on and below the diagonal
            unsigned long long acc[A][A];
#pragma unroll
            for (int a = 0; a < A; ++a)
#pragma unroll
                for (int b = 0; b < A; ++b) acc[a][b] = 0ull;
            const int quads = (src.d + 3) >> 2;
#pragma unroll 2
            for (int i = 0; i < quads; ++i) {
                ulonglong2 q[A];
#pragma unroll
                for (int a = 0; a < A; ++a) q[a] = pair4(sm.a + (ty + 16 * a) * kRow + 4 * i);
#pragma unroll
                for (int b = 0; b < A; ++b) {
                    const ulonglong2 k = pair4(sm.b + (tx + 16 * b) * kRow + 4 * i);
#pragma unroll
                    for (int a = b; a < A; ++a) fma2(acc[a][b], q[a].x, k.x), fma2(acc[a][b], q[a].y, k.y);
                }
            }
#pragma unroll
            for (int a = 0; a < A; ++a)
#pragma unroll
                for (int b = 0; b <= a; ++b) {
                    const int t = ty + 16 * a, s = tx + 16 * b;
                    const float2 x = unpack2(acc[a][b]);
#pragma unroll
                    for (int hh = 0; hh < OutputSmem<kSsm>::kHeads; ++hh)
                        if (hh < c.heads_here) sm.p[hh][t * kTokRow + s] = s <= t && t < c.n ? (x.x + x.y) * weight<kSsm>(sm.w, hh, t, s) : 0.0f;
                }
        }
        unsigned long long acc[A][8];
#pragma unroll
        for (int a = 0; a < A; ++a)
#pragma unroll
            for (int b = 0; b < 8; ++b) acc[a][b] = 0ull;
        // queries with the state the chunk starts from
        const int pieces = (src.d + kPiece - 1) / kPiece;
        for (int piece = 0; piece < pieces; ++piece) {
            __syncthreads();                                   // the keys, or the piece before, have been used up
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                const int e = tid + kThreads * r;
                *reinterpret_cast<float4*>(sm.b + (e >> 3) * kPieceRow + 4 * (e & 7)) = ahead[r];
            }
            __syncthreads();
            if (piece + 1 < pieces) ask(piece + 1);
#pragma unroll 2
            for (int i = 0; i < kPiece / 4; ++i) {
                ulonglong2 q[A];
#pragma unroll
                for (int a = 0; a < A; ++a) q[a] = pair4(sm.a + (ty + 16 * a) * kRow + piece * kPiece + 4 * i);
#pragma unroll
                for (int b = 0; b < 8; ++b) {
                    const ulonglong2 s = pair4(sm.b + (tx + 16 * b) * kPieceRow + 4 * i);
#pragma unroll
                    for (int a = 0; a < A; ++a) fma2(acc[a][b], q[a].x, s.x), fma2(acc[a][b], q[a].y, s.y);
                }
            }
        }
        const int second = kSsm ? src.dv : kCols;              // from this column on the tile's second head
#pragma unroll
        for (int a = 0; a < A; ++a)
#pragma unroll
            for (int b = 0; b < 8; ++b) {
                const float2 x = unpack2(acc[a][b]);
                const int t = ty + 16 * a, hh = tx + 16 * b >= second ? 1 : 0;
                acc[a][b] = pack2(t < c.n ? (x.x + x.y) * weight_from_start<kSsm>(sm.w, kSsm ? hh : 0, t) : 0.0f, 0.0f);
            }
        __syncthreads();                                       // the queries have been used up
        bool finite = true;
        stage_rows<T, kSsm>(c.v, src.stride, c.n, c.cols, c.wide(c.v, src.stride), true, [&](int t, int j, const float (&x)[kVec]) {
#pragma unroll
            for (int i = 0; i < kVec; ++i) {
                finite = finite && fabsf(x[i]) < INFINITY;
                sm.a[(j + i) * kTokRow + t] = x[i];
            }
        });
        // A value that is no finite number must not reach the tokens before it by way of a weight of zero: such a chunk is summed one
        // by one.
        const bool one_by_one = __syncthreads_or(!finite);
        // weighted scores with the values of the tokens
#pragma unroll
        for (int sb = 0; sb < A; ++sb) {
            if (16 * sb < c.n && !one_by_one) {
#pragma unroll 1
                for (int i = 0; i < 4; ++i) {
                    ulonglong2 p[A], p2[A];
#pragma unroll
                    for (int a = sb; a < A; ++a) {
                        p[a] = pair4(sm.p[0] + (ty + 16 * a) * kTokRow + 16 * sb + 4 * i);
                        if constexpr (kSsm) p2[a] = c.heads_here > 1 ? pair4(sm.p[1] + (ty + 16 * a) * kTokRow + 16 * sb + 4 * i) : p[a];
                    }
#pragma unroll
                    for (int b = 0; b < 8; ++b) {
                        const ulonglong2 v = pair4(sm.a + (tx + 16 * b) * kTokRow + 16 * sb + 4 * i);
#pragma unroll
                        for (int a = sb; a < A; ++a) {
                            const ulonglong2 x = kSsm && b >= 4 ? p2[a] : p[a];      // (two heads are of 64 columns)
                            fma2(acc[a][b], x.x, v.x), fma2(acc[a][b], x.y, v.y);
                        }
                    }
                }
            }
        }
#pragma unroll
        for (int a = 0; a < A; ++a) {
            const int t = ty + 16 * a;
            if (t >= c.n) continue;
            float* to = out + (size_t)(c.q0 + t) * src.heads * src.dv + c.col0;
#pragma unroll
            for (int b = 0; b < 8; ++b) {
                const int j = tx + 16 * b;
                const float2 x = unpack2(acc[a][b]);
                float y = x.x + x.y;
                if (one_by_one)
                    for (int i = 0; i <= t; ++i) y = fmaf(sm.p[kSsm && j >= second ? 1 : 0][t * kTokRow + i], sm.a[j * kTokRow + i], y);
                if constexpr (kSsm) y = fmaf(src.skip[c.head + (j >= second ? 1 : 0)], sm.a[j * kTokRow + t], y);
                if (j < c.cols) to[j] = y;
            }
        }
    };
    if (c.n > 32) with_blocks(std::integral_constant<int, 4>{});
    else if (c.n > 16) with_blocks(std::integral_constant<int, 2>{});
    else with_blocks(std::integral_constant<int, 1>{});
}

template <typename T, bool kSsm>
int launch(const Source<T>& src, const int* seg, int chunks, dim3 grid, int mode, float* chunk_state, float* chunk_decay, float* out, cudaStream_t stream) {
    const char* what = kSsm ? "state-space scan (chunks)" : "decay scan (chunks)";
    static LiOncePerDevice raised[2];
    const size_t end = (2 * kTokens * kRow) * sizeof(float) + sizeof(Weights);
    static_assert(sizeof(OutputSmem<kSsm>) <= 113 * 1024, "two blocks a multiprocessor");
    cudaError_t e = li_raise_shared(raised[0], (const void*)chunk_end_kernel<T, kSsm>, end);
    if (e == cudaSuccess) e = li_raise_shared(raised[1], (const void*)chunk_output_kernel<T, kSsm>, sizeof(OutputSmem<kSsm>));
    if (e != cudaSuccess) return li_fail("%s: cannot raise shared memory: %s", what, cudaGetErrorString(e));
    if (mode == 1) li_launch_pdl(chunk_end_kernel<T, kSsm>, grid, dim3(kThreads), end, stream, src, seg, chunk_state, chunk_decay);
    else li_launch_pdl(chunk_output_kernel<T, kSsm>, grid, dim3(kThreads), sizeof(OutputSmem<kSsm>), stream, src, seg, (const float*)chunk_state, out);
    return li_check_launch(what);
}

template <typename T>
int decay_chunks(const void* qkv, int stride, int q_off, int k_off, int v_off, const float* decay, float* out, int chunks, int heads, int d, int dv,
                 const int* seg, int mode, float* chunk_state, cudaStream_t stream) {
    const Source<T> src{(const T*)qkv, stride, q_off, k_off, v_off, d, heads, dv, 1, nullptr, 0, nullptr, nullptr, nullptr, decay};
    return launch<T, false>(src, seg, chunks, dim3(ceil_div(dv, kCols), heads, chunks), mode, chunk_state, nullptr, out, stream);
}
template <typename T>
int ssm_chunks(const void* xbc, int C, const void* dt_raw, int dt_stride, const float* dt_bias, const float* A_log, const float* D, float* y, int chunks,
               int heads, int P, int N, int groups, const int* seg, int mode, float* chunk_state, float* chunk_decay, cudaStream_t stream) {
    const int inner = heads * P;
    const Source<T> src{(const T*)xbc, C, inner + groups * N, inner, 0, N, heads, P, heads / groups, (const T*)dt_raw, dt_stride, dt_bias, A_log, D, nullptr};
    return launch<T, true>(src, seg, chunks, dim3(1, heads * P / kCols, chunks), mode, chunk_state, chunk_decay, y, stream);
}

}  // namespace

// Whether chunks of at most `length` tokens go this way: a tile of 128 value columns is a part of one head, or with the state-space form
// one head of 128 or two neighbours of 64 in one group; elements in fours.
LI_EXPORT int li_decay_chunks_accepts(int length, int d) { return length <= kTokens && d >= 4 && d <= kDim && d % 4 == 0; }
LI_EXPORT int li_ssm_chunks_accepts(int length, int heads, int P, int N, int groups) {
    return length <= kTokens && N >= 4 && N <= kDim && N % 4 == 0 && groups >= 1 && heads % groups == 0 &&
           (P == 128 || (P == 64 && heads % 2 == 0 && heads / groups % 2 == 0));
}

// mode 1: every chunk from a state of zeros, its end state to chunk_state; 2: its outputs from the state in chunk_state (recurrent.cu).
LI_EXPORT int li_decay_chunks(const void* qkv, int dtype, int stride, int q_off, int k_off, int v_off, const float* decay, float* out, int chunks, int heads,
                              int d, int dv, const int* seg, int mode, float* chunk_state, cudaStream_t stream) {
    LI_REQUIRE(dtype == LI_F32 || dtype == LI_BF16, "decay scan (chunks): unknown dtype %d", dtype);
    LI_REQUIRE(heads > 0 && dv > 0 && li_decay_chunks_accepts(kTokens, d) && (mode == 1 || mode == 2), "decay scan (chunks): %d heads of %d x %d, pass %d", heads, d, dv, mode);
    LI_REQUIRE(seg != nullptr && (uintptr_t)seg % 16 == 0 && chunk_state != nullptr && (uintptr_t)chunk_state % 16 == 0, "decay scan (chunks): needs the chunks and their states");
    if (chunks == 0) return 0;
    LI_REQUIRE(chunks > 0 && chunks <= 65535 && heads <= 65535, "decay scan (chunks): %d chunks or %d heads in one launch", chunks, heads);
    return dtype == LI_F32 ? decay_chunks<float>(qkv, stride, q_off, k_off, v_off, decay, out, chunks, heads, d, dv, seg, mode, chunk_state, stream)
                           : decay_chunks<bf16>(qkv, stride, q_off, k_off, v_off, decay, out, chunks, heads, d, dv, seg, mode, chunk_state, stream);
}

LI_EXPORT int li_ssm_chunks(const void* xbc, int dtype, int C, const void* dt_raw, int dt_stride, const float* dt_bias, const float* A_log, const float* D,
                            float* y, int chunks, int heads, int P, int N, int groups, const int* seg, int mode, float* chunk_state, float* chunk_decay,
                            cudaStream_t stream) {
    LI_REQUIRE(dtype == LI_F32 || dtype == LI_BF16, "state-space scan (chunks): unknown dtype %d", dtype);
    LI_REQUIRE(heads > 0 && li_ssm_chunks_accepts(kTokens, heads, P, N, groups) && (mode == 1 || mode == 2),
               "state-space scan (chunks): %d heads of %d in %d groups, state size %d, pass %d", heads, P, groups, N, mode);
    LI_REQUIRE(C == heads * P + 2 * groups * N, "state-space scan (chunks): %d channels for %d heads of %d and %d groups of %d", C, heads, P, groups, N);
    LI_REQUIRE(seg != nullptr && (uintptr_t)seg % 16 == 0 && chunk_state != nullptr && (uintptr_t)chunk_state % 16 == 0 && chunk_decay != nullptr,
               "state-space scan (chunks): needs the chunks, their states and their decays");
    if (chunks == 0) return 0;
    LI_REQUIRE(chunks > 0 && chunks <= 65535 && heads <= 65535, "state-space scan (chunks): %d chunks or %d heads in one launch", chunks, heads);
    return dtype == LI_F32 ? ssm_chunks<float>(xbc, C, dt_raw, dt_stride, dt_bias, A_log, D, y, chunks, heads, P, N, groups, seg, mode, chunk_state, chunk_decay, stream)
                           : ssm_chunks<bf16>(xbc, C, dt_raw, dt_stride, dt_bias, A_log, D, y, chunks, heads, P, N, groups, seg, mode, chunk_state, chunk_decay, stream);
}

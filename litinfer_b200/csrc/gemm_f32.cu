// out[M, N] = a[M, K] w[N, K]^T (+ bias[N]) in float32 on the CUDA cores: the matrix product of the true 32-bit path (no
// tensor-core mode that would round the operands; accumulation in float, bias added in float after the dot product, as in
// LitInfer's linear, src/ops/linear/cpu/linear_cpu.cpp:45-60).
//
// Every output is summed in one order that K alone decides, whatever M is and whichever of the two kernels below takes the
// product, so that the value of a row does not depend on how many other rows are in the batch:
//   chunk:   32 consecutive k, one chain of multiply-adds in ascending order;
//   half:    256 consecutive k, its chunks added in ascending order;
//   segment: 512 consecutive k, its two halves added;
//   total:   the segments added in ascending order, then the bias.
// That order leaves three places to cut the work: chunks over the warps of a block, segments over the blocks of a cluster
// (their sums meet through distributed shared memory: no workspace, no counters), rows and columns over the grid.  Its
// error is also smaller than that of one chain over all of k (1.5B shape, 28 layers: logits 1e-6 off against 64 bits, 6.4e-6
// with the chain).
//
// Measured against one 64 x 64 kernel for every size, single chain, scalar loads (us): 3 rows, N 17920, K 1536 21.4 (5.1 TB/s),
// N 1536, K 8960 16.7, N 151936 153 (6.1 TB/s; that kernel: 307 on average over a step's products).
//
// f32_stream_kernel, M <= 16: bound by reading w once.  A block takes 32 rows of w; whole segments of those rows come
// through two stages of 64 KB by TMA, a tile of 32 rows a chunk (128-byte swizzle: eight lanes on consecutive rows meet
// eight bank groups), asked for by a warp of its own.  Warp i multiplies chunks 2 i and 2 i + 1; a lane takes several rows
// and tokens (2 x 4, 4 x 4 or 4 x 8), since with one row a lane the reads of the activations from shared memory cost more
// than memory needs for w.  One block a multiprocessor walks over the tiles; where there are fewer tiles than
// multiprocessors the segments of a tile go to a cluster.
// f32_tile_kernel, M > 16 (and operands that are not 16-byte aligned): bound by the multiply-add pipes (packed multiply-adds
// from registers alone reach 57 to 62 TFLOP/s here), the latencies of two warps a scheduler, and by how the tiles fill the GPU.
// 128 columns by 32, 48, 64 or 80 rows a group of 128 threads, 4 x 8 to 10 x 8 outputs a thread, packed multiply-adds over pairs of
// columns, tiles of 16 k through registers into two transposed buffers.  The halves of a tile's segments are shared out over the
// groups of a block (one or two) and the blocks of a cluster; tile_plan chooses.  Against 64 (or 32) rows, whole segments and
// blocks of one group (us): 64 rows N 2048, K 1536 38.9 -> 27.1, N 17920 119 -> 96, N 1536, K 8960 125 -> 97; 128 rows N 1536, K 8960
// 182 -> 130; 192 rows N 1536, K 1536 50 -> 34.
#define LI_PDL_KIND 2
#include "tcgen05.cuh"

#include <algorithm>
#include <atomic>
#include <cooperative_groups.h>

namespace {

namespace cg = cooperative_groups;
using namespace tc;

constexpr int kChunk = 32, kSegment = 512, kChunks = kSegment / kChunk, kHalf = kSegment / 2;
constexpr int kMaxCluster = 8;

// ---------------------------------------------------------------------------------------------
// few rows
// ---------------------------------------------------------------------------------------------

constexpr int kRows = 32;                                  // rows of w a block
constexpr int kConsumers = 256, kThreadsS = kConsumers + 32;     // eight warps multiply, the ninth asks for the stages
constexpr int kStagesS = 2;

template <int MT>
struct __align__(1024) StreamSmem {
    static constexpr int XR = MT < 8 ? 8 : MT;             // rows of a tile of activations: whole patterns of the swizzle
    static constexpr int kSlots = MT < 16 ? 12 : 8;        // segments a block of a cluster may hold the sums of
    unsigned char w[kStagesS][kChunks][kRows * 128];       // a chunk: rows of 32 k, 128-byte swizzle
    unsigned char x[kStagesS][kChunks][XR * 128];
    float part[kChunks][(MT < 8 ? MT : 8) * kRows];        // at most eight tokens at a time
    float slot[kSlots][MT * kRows];
    unsigned long long full[kStagesS], empty[kStagesS];
};

// 16 bytes j of row r of a chunk's tile
__device__ __forceinline__ float4 swizzled(const unsigned char* tile, int r, int j) {
    return *reinterpret_cast<const float4*>(tile + r * 128 + ((j ^ (r & 7)) << 4));
}
__device__ __forceinline__ void consumers_sync() { asm volatile("bar.sync 1, 256;" ::: "memory"); }

template <int MT, int R, int T>
__global__ void __launch_bounds__(kThreadsS, 1)
f32_stream_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_x, const float* __restrict__ bias,
                  float* __restrict__ out, int M, int N, int K, int tiles, int csize, int* __restrict__ error_flag) {
    extern __shared__ unsigned char raw[];
    using Smem = StreamSmem<MT>;
    Smem& sm = *reinterpret_cast<Smem*>(((uintptr_t)raw + 1023) & ~(uintptr_t)1023);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int rank = (int)blockIdx.y;                      // place in the cluster
    const int nseg = (K + kSegment - 1) / kSegment;
    const int mine = (nseg - rank + csize - 1) / csize;    // segments rank, rank + csize, ...
    const int my_tiles = (tiles - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x;
    const int total = my_tiles * mine;                     // stages this block walks over

    if (tid == 0) {
        for (int s = 0; s < kStagesS; ++s) {
            mbar_init(&sm.full[s], 1);
            mbar_init(&sm.empty[s], kConsumers / 32);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    pdl_launch_dependents();

    if (warp == kConsumers / 32) {
        // Lanes 0 - 15 ask for a chunk of w each, lanes 16 - 31 for a chunk of a (what lies behind the last k, row or token
        // is filled with zeros).
        auto ask = [&](int i, bool weights, bool acts) {
            const int n0 = ((int)blockIdx.x + (i / mine) * (int)gridDim.x) * kRows, k0 = (rank + (i % mine) * csize) * kSegment + (lane & 15) * kChunk;
            const int s = i % kStagesS;
            if (weights && lane < 16) tma_load_2d(sm.w[s][lane], &map_w, k0, n0, &sm.full[s]);
            if (acts && lane >= 16) tma_load_2d(sm.x[s][lane - 16], &map_x, k0, 0, &sm.full[s]);
        };
        auto expect = [&](int i) {
            if (lane == 0) mbar_expect_tx(&sm.full[i % kStagesS], (unsigned)(kChunks * (kRows + Smem::XR) * 128));
            __syncwarp();
        };
        const int first = min(kStagesS, total);
        // the weights of the first stages do not depend on the kernel before
        for (int i = 0; i < first; ++i) expect(i), ask(i, true, false);
        pdl_wait();
        for (int i = 0; i < first; ++i) ask(i, false, true);
        bool ok = true;
        int issued = first;
        for (int i = first; i < total && ok; ++i) {
            ok = __all_sync(0xffffffffu, mbar_wait(&sm.empty[i % kStagesS], (i / kStagesS - 1) & 1));
            if (!ok) break;
            expect(i);
            ask(i, true, true);
            issued = i + 1;
        }
        if (!ok) {
            if (lane == 0) atomicExch(error_flag, 41);
            // the copies in flight still write to this block's shared memory
            for (int i = max(0, issued - kStagesS); i < issued; ++i) mbar_wait(&sm.full[i % kStagesS], (i / kStagesS) & 1);
        }
    } else {
        pdl_wait();
        // a lane: rows rl, rl + RL, ... (R of them), tokens tg T .. tg T + T - 1, one of the warp's two chunks
        constexpr int RL = kRows / R, TG = MT / T;
        static_assert(RL * TG == 16 && RL % 8 == 0, "two chunks a warp; eight lanes on consecutive rows");
        const int rl = lane % RL, tg = lane / RL % TG, chunk = 2 * warp + (lane >> 4);
        constexpr int kParts = MT > 8 ? MT / 8 : 1, TR = T / kParts, kPartTokens = MT / kParts;      // rounds of the sums over chunks
        float sum[kParts];
#pragma unroll
        for (int r = 0; r < kParts; ++r) sum[r] = 0.0f;
        bool ok = true;
        for (int i = 0; i < total; ++i) {
            const int s = i % kStagesS, n0 = ((int)blockIdx.x + (i / mine) * (int)gridDim.x) * kRows;
            // (a wait that ran out: the rest is computed from whatever is there, and the status says so)
            if (ok) {
                ok = mbar_wait(&sm.full[s], (i / kStagesS) & 1);
                if (!ok) atomicExch(error_flag, 42);
            }
            const unsigned char* wt = sm.w[s][chunk];
            const unsigned char* xt = sm.x[s][chunk];
            float acc[R][T];
#pragma unroll
            for (int a = 0; a < R; ++a)
#pragma unroll
                for (int m = 0; m < T; ++m) acc[a][m] = 0.0f;
#pragma unroll
            for (int j = 0; j < kChunk / 4; ++j) {
                float4 w4[R];
#pragma unroll
                for (int a = 0; a < R; ++a) w4[a] = swizzled(wt, rl + a * RL, j);
#pragma unroll
                for (int m = 0; m < T; ++m) {
                    const float4 x4 = swizzled(xt, tg * T + m, j);
#pragma unroll
                    for (int a = 0; a < R; ++a) {
                        acc[a][m] = fmaf(x4.x, w4[a].x, acc[a][m]);
                        acc[a][m] = fmaf(x4.y, w4[a].y, acc[a][m]);
                        acc[a][m] = fmaf(x4.z, w4[a].z, acc[a][m]);
                        acc[a][m] = fmaf(x4.w, w4[a].w, acc[a][m]);
                    }
                }
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(&sm.empty[s]);
            const bool last = i % mine == mine - 1;
#pragma unroll
            for (int r = 0; r < kParts; ++r) {
#pragma unroll
                for (int m = 0; m < TR; ++m)
#pragma unroll
                    for (int a = 0; a < R; ++a) sm.part[chunk][(tg * TR + m) * kRows + rl + a * RL] = acc[a][r * TR + m];
                consumers_sync();
                if (tid < kPartTokens * kRows) {
                    const int pm = tid / kRows, m = pm / TR * T + r * TR + pm % TR, n = n0 + (tid & (kRows - 1));
                    float v = 0.0f, second = 0.0f;
#pragma unroll
                    for (int c = 0; c < kChunks / 2; ++c) v += sm.part[c][tid], second += sm.part[kChunks / 2 + c][tid];
                    v += second;
                    if (csize == 1) {
                        sum[r] += v;
                        if (last) {
                            if (m < M && n < N) out[(size_t)m * N + n] = sum[r] + (bias ? bias[n] : 0.0f);
                            sum[r] = 0.0f;
                        }
                    } else {
                        sm.slot[i][m * kRows + (tid & (kRows - 1))] = v;
                    }
                }
                consumers_sync();                          // before the next partial sums
            }
        }
    }
    if (csize == 1) return;
    cg::cluster_group cluster = cg::this_cluster();
    cluster.sync();
    if (warp < kConsumers / 32) {
        const int n0 = (int)blockIdx.x * kRows;            // one tile a cluster
        for (int e = tid + rank * kConsumers; e < M * kRows; e += csize * kConsumers) {
            float v = 0.0f;
            for (int g = 0; g < nseg; ++g) v += *cluster.map_shared_rank(&sm.slot[g / csize][e], g % csize);
            const int m = e / kRows, n = n0 + (e & (kRows - 1));
            if (n < N) out[(size_t)m * N + n] = v + (bias ? bias[n] : 0.0f);
        }
    }
    cluster.sync();                                        // nobody leaves while its sums may be read
}

// ---------------------------------------------------------------------------------------------
// more rows
// ---------------------------------------------------------------------------------------------

constexpr int kBN = 128, kBK = 16, kThreadsT = 128;

// What a group of 128 threads works with.  TM rows a thread: TM / 4 times four (rows 32 h + 4 ty ..), then two where TM is not a
// multiple of four.
template <int TM>
struct __align__(16) GroupSmem {
    float w[2][kBK][kBN + 4];
    float a[2][kBK][8 * TM + 4];
    float4 sums[2 * TM][kThreadsT];                        // the sums of a half segment, per thread
};
template <int TM, int kGroups>
struct __align__(16) TileSmem {
    GroupSmem<TM> g[kGroups];
    float4 total[1][kGroups * kThreadsT];                  // running totals: all of a group's own (alone), or its share of the tile's
};
__device__ __forceinline__ unsigned long long pack2(float lo, float hi) {
    unsigned long long r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ void unpack2(unsigned long long v, float& lo, float& hi) { asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v)); }
// two multiply-adds in one instruction, each rounded as a single one
__device__ __forceinline__ void fma2(unsigned long long& d, unsigned long long a, unsigned long long b) {
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(d) : "l"(a), "l"(b));
}
__device__ __forceinline__ float4 add4(float4 a, float4 b) { return make_float4(a.x + b.x, a.y + b.y, a.z + b.z, a.w + b.w); }

template <int TM, int kGroups, bool kVec>
__global__ void __launch_bounds__(kGroups * kThreadsT, kGroups == 1 ? 2 : 1)
f32_tile_kernel(const float* __restrict__ A, const float* __restrict__ W, const float* __restrict__ bias, float* __restrict__ out, int M, int N, int K,
                bool wide_stores) {
    extern __shared__ float4 raw4[];
    TileSmem<TM, kGroups>& sm = *reinterpret_cast<TileSmem<TM, kGroups>*>(raw4);
    constexpr int BM = 8 * TM, kLoadsA = (BM + 31) / 32, kFours = TM / 4;
    static_assert(TM % 2 == 0 && kGroups <= 2, "rows in fours and a two");
    const int grp = (int)threadIdx.x / kThreadsT, tid = (int)threadIdx.x % kThreadsT, tx = tid & 15, ty = tid >> 4;      // columns 4 tx .. and 64 + 4 tx ..
    GroupSmem<TM>& gs = sm.g[grp];
    // tiles of rows run fastest, so that a tile of w is read by neighbours; all tiles along x, which has room for any N
    const int mt = (M + BM - 1) / BM;
    const int m0 = (int)blockIdx.x % mt * BM, n0 = (int)blockIdx.x / mt * kBN;
    // the half segments of a tile are shared out over the groups of a cluster's blocks: group v takes v, v + vr, ...
    const int csize = (int)gridDim.z, rank = (int)blockIdx.z, vr = csize * kGroups, v = rank * kGroups + grp;
    const int halves = (K + kHalf - 1) / kHalf;
    const int lr = tid >> 2, lk = (tid & 3) * 4;           // loads: rows lr + 32 r, four k from lk on
    auto group_sync = [&] {
        if constexpr (kGroups == 1) __syncthreads();
        else asm volatile("bar.sync %0, 128;" ::"r"(1 + grp) : "memory");
    };

    float4 pa[kLoadsA], pw[4];
    auto load4 = [&](const float* base, int row, int rows, int k) {
        float4 x = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        if (row < rows) {
            const float* p = base + (size_t)row * K + k;
            if constexpr (kVec) {
                if (k < K) x = __ldg(reinterpret_cast<const float4*>(p));
            } else {
                if (k < K) x.x = p[0];
                if (k + 1 < K) x.y = p[1];
                if (k + 2 < K) x.z = p[2];
                if (k + 3 < K) x.w = p[3];
            }
        }
        return x;
    };
    auto fetch = [&](int k0) {
#pragma unroll
        for (int r = 0; r < 4; ++r) pw[r] = load4(W, n0 + lr + 32 * r, N, k0 + lk);
#pragma unroll
        for (int r = 0; r < kLoadsA; ++r)
            if (lr + 32 * r < BM) pa[r] = load4(A, m0 + lr + 32 * r, M, k0 + lk);
    };
    auto put = [&](int b) {
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            gs.w[b][lk][lr + 32 * r] = pw[r].x, gs.w[b][lk + 1][lr + 32 * r] = pw[r].y;
            gs.w[b][lk + 2][lr + 32 * r] = pw[r].z, gs.w[b][lk + 3][lr + 32 * r] = pw[r].w;
        }
#pragma unroll
        for (int r = 0; r < kLoadsA; ++r) {
            if (lr + 32 * r < BM) {
                gs.a[b][lk][lr + 32 * r] = pa[r].x, gs.a[b][lk + 1][lr + 32 * r] = pa[r].y;
                gs.a[b][lk + 2][lr + 32 * r] = pa[r].z, gs.a[b][lk + 3][lr + 32 * r] = pa[r].w;
            }
        }
    };

    unsigned long long acc[TM][4];
    float seg[TM][8];
#pragma unroll
    for (int i = 0; i < TM; ++i) {
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = 0ull;
#pragma unroll
        for (int j = 0; j < 8; ++j) seg[i][j] = 0.0f;
    }
    // float4 q of a thread: its row q / 2, columns 4 tx .. (q even) or 64 + 4 tx .. (q odd)
    for (int q = v; q < 2 * TM; q += vr) sm.total[q / vr][threadIdx.x] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);

    const int waves = (halves + vr - 1) / vr;
    int buf = 0;
    pdl_launch_dependents();
    pdl_wait();
    if (v < halves) fetch(v * kHalf);
    for (int wave = 0; wave < waves; ++wave) {
        const int g = wave * vr + v;
        if (g < halves) {
            const int k_begin = g * kHalf, k_end = min(K, k_begin + kHalf);
            for (int k0 = k_begin; k0 < k_end; k0 += kBK) {
                put(buf);
                group_sync();                              // (two buffers: one barrier a tile)
                const int next = k0 + kBK < k_end ? k0 + kBK : (g + vr) * kHalf;
                if (next < K) fetch(next);
#pragma unroll
                for (int kk = 0; kk < kBK; ++kk) {
                    const ulonglong2 w01 = *reinterpret_cast<const ulonglong2*>(&gs.w[buf][kk][4 * tx]);
                    const ulonglong2 w23 = *reinterpret_cast<const ulonglong2*>(&gs.w[buf][kk][64 + 4 * tx]);
                    const unsigned long long w2[4] = {w01.x, w01.y, w23.x, w23.y};
#pragma unroll
                    for (int h = 0; h < kFours; ++h) {
                        const float4 a4 = *reinterpret_cast<const float4*>(&gs.a[buf][kk][32 * h + 4 * ty]);
                        const float av[4] = {a4.x, a4.y, a4.z, a4.w};
#pragma unroll
                        for (int i = 0; i < 4; ++i) {
                            const unsigned long long aa = pack2(av[i], av[i]);
#pragma unroll
                            for (int j = 0; j < 4; ++j) fma2(acc[4 * h + i][j], aa, w2[j]);
                        }
                    }
                    if constexpr (TM % 4 != 0) {
                        const float2 a2 = *reinterpret_cast<const float2*>(&gs.a[buf][kk][32 * kFours + 2 * ty]);
                        const float av[2] = {a2.x, a2.y};
#pragma unroll
                        for (int i = 0; i < 2; ++i) {
                            const unsigned long long aa = pack2(av[i], av[i]);
#pragma unroll
                            for (int j = 0; j < 4; ++j) fma2(acc[4 * kFours + i][j], aa, w2[j]);
                        }
                    }
                }
                buf ^= 1;
                if (((k0 + kBK) & (kChunk - 1)) == 0 || k0 + kBK >= k_end) {       // the end of a chunk
#pragma unroll
                    for (int i = 0; i < TM; ++i)
#pragma unroll
                        for (int j = 0; j < 4; ++j) {
                            float lo, hi;
                            unpack2(acc[i][j], lo, hi);
                            seg[i][2 * j] += lo, seg[i][2 * j + 1] += hi;
                            acc[i][j] = 0ull;
                        }
                }
            }
        }
        // alone: the first half of a segment waits in `sums` for the second; else every group's halves meet, two by two
        const bool pair = vr > 1 || ((g & 1) == 0 && g + 1 < halves);
#pragma unroll
        for (int q = 0; q < 2 * TM; ++q) {
            float* sg = &seg[q >> 1][4 * (q & 1)];
            const float4 x = make_float4(sg[0], sg[1], sg[2], sg[3]);
            if (pair) gs.sums[q][tid] = x;
            else sm.total[q][tid] = add4(sm.total[q][tid], (g & 1) ? add4(gs.sums[q][tid], x) : x);
            sg[0] = sg[1] = sg[2] = sg[3] = 0.0f;
        }
        if (vr > 1) {
            cg::cluster_group cluster = cg::this_cluster();
            if (csize > 1) cluster.sync();
            else __syncthreads();
            const int here = min(vr, halves - wave * vr);
            auto of = [&](int q, int r) {
                const float4* p = &sm.g[r % kGroups].sums[q][tid];
                return csize > 1 ? *cluster.map_shared_rank(p, r / kGroups) : *p;
            };
            for (int q = v; q < 2 * TM; q += vr) {
                float4 x = sm.total[q / vr][threadIdx.x];
                int r = 0;
                for (; r + 1 < here; r += 2) x = add4(x, add4(of(q, r), of(q, r + 1)));
                if (r < here) x = add4(x, of(q, r));
                sm.total[q / vr][threadIdx.x] = x;
            }
            if (csize > 1) cluster.sync();                 // before the next sums, and before anyone leaves
            else __syncthreads();
        }
    }
    for (int q = v; q < 2 * TM; q += vr) {
        const float4 x = sm.total[q / vr][threadIdx.x];
        const int i = q >> 1, row = i < 4 * kFours ? (i >> 2) * 32 + 4 * ty + (i & 3) : 32 * kFours + 2 * ty + (i - 4 * kFours);
        const int m = m0 + row, n = n0 + (q & 1) * 64 + 4 * tx;
        if (m >= M) continue;
        float r[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
        for (int j = 0; j < 4; ++j)
            if (bias && n + j < N) r[j] += bias[n + j];
        float* to = out + (size_t)m * N + n;
        if (wide_stores && n + 3 < N) {
            *reinterpret_cast<float4*>(to) = make_float4(r[0], r[1], r[2], r[3]);
        } else {
#pragma unroll
            for (int j = 0; j < 4; ++j)
                if (n + j < N) to[j] = r[j];
        }
    }
}

// Few rows: blocks of a cluster that share a tile's segments: 1, 2, 4 or 8 (clusters of three left multiprocessors idle: 3 rows,
// N 1536, K 8960 25.4 us against 16.7 with two), whichever has the least of waves of blocks x (segments a block takes one
// after the other + 1.5 for its start and its merge).
int stream_cluster(int tiles, int nseg, int slots) {
    int best = 1;
    double least = 0.0;
    for (int c = 1; c <= kMaxCluster && c <= nseg; c *= 2) {
        const int each = ceil_div(nseg, c);
        if (c > 1 && each > slots) continue;
        const double cost = ceil_div(tiles * c, li_multiprocessors()) * (each + 1.5);
        if (least == 0.0 || cost < least) least = cost, best = c;
    }
    return best;
}

// More rows: the shape of a launch.
struct TilePlan {
    int tm, groups, cluster;                               // rows a thread (tiles of 8 tm rows), groups a block, blocks that share a tile
};
TilePlan g_forced_tile{0, 0, 0};

template <int TM, int kGroups>
size_t tile_shared(int c) {
    return sizeof(TileSmem<TM, kGroups>) + (ceil_div(2 * TM, c * kGroups) - 1) * sizeof(float4) * kThreadsT * kGroups;
}

// How many clusters of c blocks the current device holds at once (asked once a size and device; two threads that ask at the same time
// both ask).
template <int TM, int kGroups>
int clusters_at_once(int c) {
    static std::atomic<int> known[16][kMaxCluster + 1];
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 16) return 1;
    int n = known[dev][c].load(std::memory_order_relaxed);
    if (n == 0) {
        static LiOncePerDevice raised;
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(1, 1, c);
        cfg.blockDim = dim3(kThreadsT * kGroups);
        cfg.dynamicSmemBytes = tile_shared<TM, kGroups>(c);
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = attr[0].val.clusterDim.y = 1;
        attr[0].val.clusterDim.z = c;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        if (li_raise_shared(raised, (const void*)f32_tile_kernel<TM, kGroups, true>, tile_shared<TM, kGroups>(1)) != cudaSuccess ||
            (c == 1 ? cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, f32_tile_kernel<TM, kGroups, true>, kThreadsT * kGroups, tile_shared<TM, kGroups>(1))
                    : cudaOccupancyMaxActiveClusters(&n, f32_tile_kernel<TM, kGroups, true>, &cfg)) != cudaSuccess || n < 1) {
            cudaGetLastError();
            n = 1;
        }
        if (c == 1) n *= li_multiprocessors();
        known[dev][c].store(n, std::memory_order_relaxed);
    }
    return n;
}

// What a launch should take, in microseconds: a half segment is 256 k of `step` cycles, the longer of the thread's multiply-adds and the
// reads of their operands; one, two or three groups on a multiprocessor take 2.4 (blocks that come when others have gone 1.8), 3.25 or
// 4.5 times that; a cluster's merge 1.5 us.  (145 rows: N 17920, K 1536 says 211, takes 209; N 1536, K 8960 150 and 150; N 1536, K 1536 32 and 31; 45 rows, N 1536, K
// 8960 80 and 83.)
template <int TM>
void consider(int M, int N, int K, bool vec, TilePlan& best, double& least) {
    const long long tiles = ceil_div_ll(M, 8 * TM) * ceil_div_ll(N, kBN);
    const int halves = ceil_div(K, kHalf), sms = li_multiprocessors();
    const double half = (TM * 8 > (TM + 8) * 4 ? TM * 8 : (TM + 8) * 4) * kHalf / 1920.0;
    const double times[4] = {0.0, 2.4, 3.25, 4.5};
    for (int groups = 1; groups <= (vec ? 2 : 1); ++groups)
        for (int c = 1; c <= kMaxCluster; c += (groups == 1 && c > 1) ? 2 : 1) {
            const int vr = c * groups;
            if (vr > 1 && vr > halves + 1) break;
            const int most = groups == 1 ? clusters_at_once<TM, 1>(c) : clusters_at_once<TM, 2>(c), alone = clusters_at_once<TM, 2>(c);
            const int dense = groups == 2 ? 2 : std::min(3, std::max(1, most * c / sms + (most * c % sms > sms / 2)));       // groups on a multiprocessor that is full
            auto round = [&](long long t) { return times[groups == 1 && t <= alone ? 1 : groups == 1 && t <= 2 * alone ? std::min(2, dense) : dense]; };
            const long long full = tiles / most, rest = tiles % most;
            const double each = (full * times[dense] + (rest == 0 ? 0.0 : full > 0 && c == 1 && groups == 1 && rest <= alone ? 1.8 : round(rest))) * (groups == 2 ? 1.05 : 1.0);
            const double us = 2.0 + ceil_div(halves, vr) * (each * half + (vr > 1 ? 1.5 * (full + (rest > 0)) : 0.0));
            if (least == 0.0 || us < least) least = us, best = TilePlan{TM, groups, c};
        }
}
TilePlan tile_plan(int M, int N, int K, bool vec) {
    if (g_forced_tile.tm > 0 && vec) return g_forced_tile;
    TilePlan best{8, 1, 1};
    double least = 0.0;
    consider<4>(M, N, K, vec, best, least);
    consider<8>(M, N, K, vec, best, least);
    if (vec) {
        consider<6>(M, N, K, vec, best, least);
        consider<10>(M, N, K, vec, best, least);
    }
    return best;
}

// Row-major [rows, K] float32 in tiles of box_rows x 32, 128-byte swizzle, zeros outside.
int make_map_f32(EncodeTiledFn encode, CUtensorMap* map, const float* base, int rows, int K, int box_rows) {
    const cuuint64_t dims[2] = {(cuuint64_t)K, (cuuint64_t)rows}, strides[1] = {(cuuint64_t)K * 4};
    const cuuint32_t box[2] = {kChunk, (cuuint32_t)box_rows}, ones[2] = {1, 1};
    const CUresult r = encode(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<float*>(base), dims, strides, box, ones, CU_TENSOR_MAP_INTERLEAVE_NONE,
                              CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    LI_REQUIRE(r == CUDA_SUCCESS, "linear (float32): cannot describe a %d x %d matrix (status %d)", rows, K, (int)r);
    return 0;
}

template <int MT, int R, int T>
int launch_stream(const float* a, const float* w, const float* bias, float* out, int M, int N, int K, cudaStream_t stream) {
    EncodeTiledFn encode = nullptr;
    int *err_host = nullptr, *err_dev = nullptr;
    if (int rc = setup(&encode, &err_host, &err_dev)) return rc;
    if (*err_host != 0)
        return li_fail("linear (float32): an earlier launch gave up waiting on a barrier (status %d); the results since then are invalid", *err_host);
    CUtensorMap map_w, map_x;
    if (int rc = make_map_f32(encode, &map_w, w, N, K, kRows)) return rc;
    if (int rc = make_map_f32(encode, &map_x, a, M, K, StreamSmem<MT>::XR)) return rc;
    const int tiles = ceil_div(N, kRows), nseg = ceil_div(K, kSegment), sms = li_multiprocessors();
    const int c = stream_cluster(tiles, nseg, StreamSmem<MT>::kSlots);
    const size_t smem = sizeof(StreamSmem<MT>) + 1024;
    static_assert(sizeof(StreamSmem<MT>) + 1024 <= 227 * 1024, "a block's shared memory");
    static LiOncePerDevice raised;
    cudaError_t e = li_raise_shared(raised, (const void*)f32_stream_kernel<MT, R, T>, smem);
    if (e != cudaSuccess) return li_fail("linear (float32): cannot raise shared memory to %zu: %s", smem, cudaGetErrorString(e));
    li_launch_pdl(f32_stream_kernel<MT, R, T>, dim3(c == 1 ? (tiles < sms ? tiles : sms) : tiles, c), dim3(kThreadsS), smem, stream, dim3(1, c, 1), map_w,
                  map_x, bias, out, M, N, K, tiles, c, err_dev);
    return li_check_launch("linear (float32, few rows)");
}

template <int TM, int kGroups, bool kVec>
int launch_tile(const float* a, const float* w, const float* bias, float* out, int M, int N, int K, int c, cudaStream_t stream) {
    const long long tiles = ceil_div_ll(M, 8 * TM) * ceil_div_ll(N, kBN);
    LI_REQUIRE(tiles <= 2147483647LL, "linear: M=%d, N=%d are too large for one launch", M, N);
    using Smem = TileSmem<TM, kGroups>;
    const size_t most = tile_shared<TM, kGroups>(1), smem = tile_shared<TM, kGroups>(c);
    static_assert(sizeof(Smem) + (2 * TM / kGroups - 1) * sizeof(float4) * kThreadsT * kGroups <= (kGroups == 1 ? 113 : 227) * 1024, "a block's shared memory");
    static LiOncePerDevice raised;
    cudaError_t e = li_raise_shared(raised, (const void*)f32_tile_kernel<TM, kGroups, kVec>, most);
    if (e != cudaSuccess) return li_fail("linear (float32): cannot raise shared memory to %zu: %s", most, cudaGetErrorString(e));
    li_launch_pdl(f32_tile_kernel<TM, kGroups, kVec>, dim3((unsigned)tiles, 1, c), dim3(kThreadsT * kGroups), smem, stream, dim3(1, 1, c), a, w, bias, out,
                  M, N, K, N % 4 == 0 && (uintptr_t)out % 16 == 0);
    return li_check_launch("linear (float32)");
}

template <bool kVec>
int tile_of(const float* a, const float* w, const float* bias, float* out, int M, int N, int K, cudaStream_t stream) {
    const TilePlan p = tile_plan(M, N, K, kVec);
    if constexpr (kVec) {
        if (p.groups == 2) {
            switch (p.tm) {
                case 4: return launch_tile<4, 2, true>(a, w, bias, out, M, N, K, p.cluster, stream);
                case 6: return launch_tile<6, 2, true>(a, w, bias, out, M, N, K, p.cluster, stream);
                case 8: return launch_tile<8, 2, true>(a, w, bias, out, M, N, K, p.cluster, stream);
                default: return launch_tile<10, 2, true>(a, w, bias, out, M, N, K, p.cluster, stream);
            }
        }
        if (p.tm == 6) return launch_tile<6, 1, true>(a, w, bias, out, M, N, K, p.cluster, stream);
        if (p.tm == 10) return launch_tile<10, 1, true>(a, w, bias, out, M, N, K, p.cluster, stream);
    }
    return p.tm == 4 ? launch_tile<4, 1, kVec>(a, w, bias, out, M, N, K, p.cluster, stream)
                     : launch_tile<8, 1, kVec>(a, w, bias, out, M, N, K, p.cluster, stream);
}

}  // namespace

// This shape for the aligned products of more than 16 rows (rows a thread 4, 6, 8 or 10; groups a block; blocks of a cluster), 0: by
// size.  Two blocks of a group pair the halves of a segment, so a cluster of groups of one is 1 or even.  For tests and measurements.
LI_EXPORT int li_linear_f32_force_tile(int tm, int groups, int cluster) {
    if (tm == 0) {
        g_forced_tile = TilePlan{0, 0, 0};
        return 0;
    }
    LI_REQUIRE((tm == 4 || tm == 6 || tm == 8 || tm == 10) && (groups == 1 || groups == 2) && cluster >= 1 && cluster <= kMaxCluster &&
                   (groups == 2 || cluster == 1 || cluster % 2 == 0), "linear (float32): no tile of %d rows a thread, %d groups, cluster %d", tm, groups, cluster);
    g_forced_tile = TilePlan{tm, groups, cluster};
    return 0;
}

int li_linear_f32(const float* a, const float* w, const float* bias, float* out, int M, int N, int K, cudaStream_t stream) {
    const bool vec = K % 4 == 0 && (uintptr_t)a % 16 == 0 && (uintptr_t)w % 16 == 0;
    if (!vec) return tile_of<false>(a, w, bias, out, M, N, K, stream);
    if (M <= 4) return launch_stream<4, 2, 4>(a, w, bias, out, M, N, K, stream);
    if (M <= 8) return launch_stream<8, 4, 4>(a, w, bias, out, M, N, K, stream);
    if (M <= 16) return launch_stream<16, 4, 8>(a, w, bias, out, M, N, K, stream);
    return tile_of<true>(a, w, bias, out, M, N, K, stream);
}

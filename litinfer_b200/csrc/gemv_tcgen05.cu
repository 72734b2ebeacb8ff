// out[M, N] = a[M, K] w[N, K]^T (+ bias) in bfloat16 for few rows of a (M <= 64:
// decode), with the roles of the operands swapped on the fifth-generation
// tensor cores: 128 weight rows are the M side of tcgen05.mma, the tokens its N
// side (16, 32 or 64 columns of tensor memory).  The kernel is bound by reading
// every weight once; TMA streams 16 KB weight tiles through a ring of shared
// memory stages with no registers involved, which keeps more bytes in flight per
// multiprocessor than loads into registers can.
//
// Grid (tiles of 128 weight rows, splits of k).  Warp 0: producer (TMA), warp 1:
// tensor-memory allocation and MMA issue, warps 2-5: epilogue.  The weight tiles of
// the first stages are requested before griddepcontrol.wait (weights do not depend
// on the kernel before), the activation tiles after it.  With several splits the
// CTAs of a tile form a cluster of up to eight: each leaves its float partial tile
// in its shared memory, and CTA r of the cluster takes the tokens r, r + size, ...,
// adds their sums in split order through distributed shared memory and does their
// epilogue.  What that costs is the trips through the cluster: sixteen loads are in
// flight at a time (64 tokens, N 1536, K 8960, eight splits: a load after the other
// 15.6 us, so 11.7; N 2048, K 1536 10.4 and 6.8).  The splits are a function of N
// and K: a token's result does not depend on how many others there are.
// Epilogue: bias, or the SwiGLU of gate and up rows interleaved in groups of 8
// (up * gate / (1 + exp(-gate)), src/ops/swiglu/op.cpp:17-23).
//
// K a multiple of 8; waits bounded as in the other tcgen05 kernel.
#define LI_PDL_KIND 2
#include "gemv_epilogue.cuh"
#include "row_scale.cuh"
#include "tcgen05.cuh"

#include <atomic>

namespace {

using namespace tc;

constexpr int BR = 128;                  // weight rows per CTA
constexpr int kThreads = 192;
constexpr int kTargetCtas = 148;
constexpr int kMaxCluster = 8;

// Stages: six (deep), or as many as two CTAs a multiprocessor leave room for.  Two are better where the CTAs come in several waves,
// since the next tile streams in while the other's epilogue runs (64 tokens, N 37888, K 3584: 61 -> 49 us).  Where every CTA of
// the launch has a multiprocessor to itself, four stages only keep less in flight (N 12288, K 18944: 102 us, with six 90).
constexpr int kDeep = 6;
template <int BT>
constexpr int kShallow = BT <= 16 ? 6 : BT <= 32 ? 5 : 4;

template <int BT, int kStages>
struct __align__(1024) Smem {
    unsigned char w[kStages][BR * BK * 2];
    unsigned char x[kStages][BT * BK * 2];
    unsigned long long full[kStages];
    unsigned long long empty[kStages];
    unsigned long long accum;
    unsigned tmem_base;
    float factor[64];                // per token: the reciprocal root of the norm before this product
    float squares[4][64];            // per epilogue warp and token: sums of squares of the new residual values
};

template <int N>
__device__ __forceinline__ void tmem_ld(unsigned taddr, float (&v)[N]);

template <>
__device__ __forceinline__ void tmem_ld<16>(unsigned taddr, float (&v)[16]) {
    unsigned r[16];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]),
          "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(r[i]);
}

template <>
__device__ __forceinline__ void tmem_ld<32>(unsigned taddr, float (&v)[32]) { tmem_ld_32x32(taddr, v); }

template <>
__device__ __forceinline__ void tmem_ld<64>(unsigned taddr, float (&v)[64]) {
    float a[32], b[32];
    tmem_ld_32x32(taddr, a);
    tmem_ld_32x32(taddr + 32, b);
#pragma unroll
    for (int i = 0; i < 32; ++i) {
        v[i] = a[i];
        v[32 + i] = b[i];
    }
}

// All threads of a cluster's CTAs, each warp by itself.
__device__ __forceinline__ void cluster_arrive_wait() {
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ unsigned peer_address(unsigned addr, unsigned rank) {
    unsigned r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
    return r;
}
__device__ __forceinline__ float peer_load(unsigned addr) {
    float v;
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(addr) : "memory");
    return v;
}

enum { kEpiNone = 0, kEpiSwiglu = 1, kEpiAddScaled = 2, kEpiGluClamped = 3, kEpiGeglu = 4, kEpiRope = 5 };     // (3 and 4: SwiGLU's layout, another activation)

// kSplit: k is split over the `csize` CTAs of a cluster (the grid's y).
// The sum into the residual stream is held to two CTAs a multiprocessor: without the bound its 33 to 64 tokens took 255
// registers, one CTA a multiprocessor, and clusters of five, six and eight, of which the GPU then holds 26, 22 and 15, no longer
// ran all at once (64 tokens, N 3584, K 8960, 28 clusters of five: 40.5 us, with the bound 22.3; N 2048, K 8960 35.9 and 20.1).
// The other forms stay below that number by themselves.
template <int BT, typename Tout, int kEpi, bool kSplit, int kStages>
__global__ void __launch_bounds__(kThreads, kEpi == kEpiAddScaled && BT >= 32 ? 2 : 0)
gemv_tcgen05_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_x,
                    const float* __restrict__ bias, Tout* __restrict__ out, int M, int N, int K, int csize, int* __restrict__ error_flag, const RowScale rs,
                    const AddScaled add, const RopeArgs rope) {
    constexpr int kSwiglu = kEpi == kEpiSwiglu ? LI_EPILOGUE_SWIGLU : kEpi == kEpiGluClamped ? LI_EPILOGUE_GLU_CLAMPED : kEpi == kEpiGeglu ? LI_EPILOGUE_GEGLU : 0;
    constexpr bool kAdd = kEpi == kEpiAddScaled;
    extern __shared__ unsigned char smem_raw[];
    Smem<BT, kStages>& sm = *reinterpret_cast<Smem<BT, kStages>*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int tile = blockIdx.x, split = blockIdx.y;
    const int n0 = tile * BR;
    const int nkb_total = (K + BK - 1) / BK;
    const int kb0 = (int)((long long)split * nkb_total / csize), kb1 = (int)((long long)(split + 1) * nkb_total / csize);
    const int nkb = kb1 - kb0;
    constexpr unsigned kStageBytes = BR * BK * 2 + BT * BK * 2;
    constexpr unsigned kCols = BT < 32 ? 32 : BT;
    constexpr int kMine = kSplit ? BT / 2 : BT;            // tokens a CTA finishes at most (a cluster has at least two)

    if (threadIdx.x == 0) {
        for (int s = 0; s < kStages; ++s) {
            mbar_init(&sm.full[s], 1);
            mbar_init(&sm.empty[s], 1);
        }
        mbar_init(&sm.accum, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    // (The other tcgen05 kernels take their tensor memory only after the kernel before them has finished, see
    // gemm_tcgen05.cu.  This one takes its 32 or 64 of the 512 columns at once: with the allocation behind the wait a decode
    // step of batch 8 went from 1.311 to 1.337 ms.  A CTA that holds them while it waits must not keep a CTA of the kernel
    // before from allocating, which may want all 512: every kernel with tensor memory lets its dependents go only after its
    // own allocation, so that by the time this kernel is there, each CTA before it has what it needs.)
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&sm.tmem_base)), "r"(kCols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const unsigned tmem_acc = sm.tmem_base;
    pdl_launch_dependents();

    if (warp == 0) {
        if (lane == 0) {
            // weights of the first stages at once; the activations once the kernel before has finished
            const int first = nkb < kStages ? nkb : kStages;
            for (int i = 0; i < first; ++i) {
                mbar_expect_tx(&sm.full[i], kStageBytes);
                tma_load_2d(sm.w[i], &map_w, (kb0 + i) * BK, n0, &sm.full[i]);
            }
            pdl_wait();
            for (int i = 0; i < first; ++i) tma_load_2d(sm.x[i], &map_x, (kb0 + i) * BK, 0, &sm.full[i]);
            bool ok = true;
            int issued = first;
            for (int i = first; i < nkb; ++i) {
                const int s = i % kStages;
                ok = mbar_wait(&sm.empty[s], ((i / kStages) & 1) ^ 1);
                if (!ok) break;
                mbar_expect_tx(&sm.full[s], kStageBytes);
                tma_load_2d(sm.w[s], &map_w, (kb0 + i) * BK, n0, &sm.full[s]);
                tma_load_2d(sm.x[s], &map_x, (kb0 + i) * BK, 0, &sm.full[s]);
                issued = i + 1;
            }
            if (!ok) {
                atomicExch(error_flag, 31);
                for (int i = (issued > kStages ? issued - kStages : 0); i < issued; ++i) mbar_wait(&sm.full[i % kStages], (i / kStages) & 1);
            }
        }
    } else if (warp == 1) {
        if (lane == 0) {
            const unsigned idesc = umma_idesc(BR, BT);
            bool ok = true;
            for (int i = 0; i < nkb && ok; ++i) {
                const int s = i % kStages;
                ok = mbar_wait(&sm.full[s], (i / kStages) & 1);
                if (!ok) break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const unsigned long long da = umma_desc(sm.w[s]), db = umma_desc(sm.x[s]);
#pragma unroll
                for (int k = 0; k < BK / 16; ++k)
                    umma_bf16(tmem_acc, da + (unsigned long long)(k * 2), db + (unsigned long long)(k * 2), idesc, (i | k) ? 1u : 0u);
                umma_commit(&sm.empty[s]);
            }
            if (ok) umma_commit(&sm.accum);
            else atomicExch(error_flag, 32);
        }
    } else {
        pdl_wait();
        const int quarter = warp & 3;
        const int r_in_tile = quarter * 32 + lane;
        const int row = n0 + r_in_tile;
        // while the weights stream: the tokens' factors from the partial sums of squares, and the old values of
        // the residual stream that the product will be added to (row_scale.cuh)
        if (rs.ssq) {
            // a warp takes every fourth token, eight tokens' loads in flight at once
            row_scales_of_warp<8>(rs, M, warp - 2, 4, lane, sm.factor);
            asm volatile("bar.sync 1, 128;" ::: "memory");
        }
        // the tokens this CTA finishes: all of them, or every csize-th of a cluster's
        const int rank = kSplit ? split : 0, step = kSplit ? csize : 1;
        float xold[kAdd ? kMine : 1];
        auto load_old = [&]() {
            if constexpr (kAdd) {
#pragma unroll
                for (int i = 0; i < kMine; ++i) {
                    const int j = rank + i * step;
                    xold[i] = (j < M && row < N) ? __ldcg(add.x32 + (size_t)j * N + row) : 0.0f;
                }
            }
        };
        // The rotation's angles and the tokens' places in the cache, of this CTA's tokens: worked out while the weights stream.  (In
        // the epilogue itself, a token after the other, each of them a load and a sine: 61 tokens, N 4608, K 3584 22.2 us.)
        float2* rot = reinterpret_cast<float2*>(&sm + 1);
        const int tokens_here = rank < M ? (M - rank + step - 1) / step : 0;
        int* place = reinterpret_cast<int*>(rot + tokens_here * (BR / 2));
        if constexpr (kEpi == kEpiRope) {
            const int t = (int)threadIdx.x - 64;
            if (rope.denom != nullptr && tile < rope.nh + rope.nkv)
                for (int e = t; e < tokens_here * (BR / 2); e += 128) {
                    float sn, cs;
                    sincosf((float)rope.positions[rank + e / (BR / 2) * step] / rope.denom[e % (BR / 2)], &sn, &cs);
                    rot[e] = make_float2(cs, sn);
                }
            if (rope.write)
                for (int e = t; e < tokens_here; e += 128) place[e] = rope.slot_mapping[rank + e * step];
        }
        // (32 tokens with a split: asked for when the partial tile has left its registers, else some of them spill)
        if constexpr (!kSplit || BT != 32) load_old();
        const bool ok = mbar_wait(&sm.accum, 0);
        if (!ok && lane == 0) atomicExch(error_flag, 33);
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        float v[BT];
        tmem_ld<BT>(tmem_acc + ((unsigned)(quarter * 32) << 16), v);
        const bool write = ok;
        if constexpr (kSplit) {
            // (every load into the stages has been multiplied: their room holds the partial tile [token][row] now)
            float* mine = reinterpret_cast<float*>(sm.w[0]) + r_in_tile;
#pragma unroll
            for (int j = 0; j < BT; ++j)
                if (j < M) mine[j * BR] = v[j];
            if constexpr (BT == 32) load_old();
            cluster_arrive_wait();
            // sixteen loads in flight, of four tokens and four CTAs: without branches around them (tokens that are not there read
            // the last one's place), since a load that waits for the one before costs a trip through the cluster each
            constexpr int kTok = 4, kPeers = 4;
            const unsigned own = smem_u32(mine);
#pragma unroll
            for (int i0 = 0; i0 < kMine; i0 += kTok) {
                float t[kTok] = {};
                if (rank + i0 * step < M) {
#pragma unroll 1
                    for (int r0 = 0; r0 < csize; r0 += kPeers) {
                        float x[kPeers][kTok];
#pragma unroll
                        for (int q = 0; q < kPeers; ++q) {
                            const unsigned src = peer_address(own, (unsigned)min(r0 + q, csize - 1));
#pragma unroll
                            for (int i = 0; i < kTok; ++i) x[q][i] = peer_load(src + (unsigned)min(rank + (i0 + i) * step, M - 1) * (BR * 4));
                        }
#pragma unroll
                        for (int q = 0; q < kPeers; ++q)
#pragma unroll
                            for (int i = 0; i < kTok; ++i)
                                if (r0 + q < csize) t[i] += x[q][i];
                    }
                }
#pragma unroll
                for (int i = 0; i < kTok; ++i) v[i0 + i] = t[i];
            }
        }
        if (write && rs.ssq) {
#pragma unroll
            for (int i = 0; i < kMine; ++i)
                if (rank + i * step < M) v[i] *= sm.factor[rank + i * step];
        }
        if (write) {
            if constexpr (kAdd) {
                // into the residual stream, and on to the next product as bfloat16(norm_weight * x) with the sums of x^2
                const float b = (bias && row < N) ? bias[row] : 0.0f;
                const float nw = row < N ? add.norm_weight[row] : 0.0f;
                constexpr int kTok = 4;                                    // tokens whose squares are added up side by side
#pragma unroll
                for (int i0 = 0; i0 < kMine; i0 += kTok) {
                    if (rank + i0 * step < M) {                            // uniform
                        float sq[kTok];
#pragma unroll
                        for (int i = 0; i < kTok; ++i) {
                            const int j = rank + (i0 + i) * step;
                            const float x = j < M && row < N ? xold[i0 + i] + (v[i0 + i] + b) : 0.0f;
                            if (j < M && row < N) {
                                __stcg(add.x32 + (size_t)j * N + row, x);
                                add.hprime[(size_t)j * N + row] = __float2bfloat16_rn(nw * x);
                            }
                            sq[i] = x * x;
                        }
#pragma unroll
                        for (int o = 16; o > 0; o >>= 1)
#pragma unroll
                            for (int i = 0; i < kTok; ++i) sq[i] += __shfl_xor_sync(0xffffffffu, sq[i], o);
#pragma unroll
                        for (int i = 0; i < kTok; ++i)
                            if (lane == 0 && rank + (i0 + i) * step < M) sm.squares[quarter][rank + (i0 + i) * step] = sq[i];
                    }
                }
                asm volatile("bar.sync 1, 128;" ::: "memory");
                const int j = rank + ((int)threadIdx.x - 64) * step;
                if (j < M) add.ssq_out[(size_t)j * gridDim.x + tile] = ((sm.squares[0][j] + sm.squares[1][j]) + sm.squares[2][j]) + sm.squares[3][j];
            } else if constexpr (kEpi == kEpiRope) {
                // the tile is one head: rotation, then q into its row, k and v (transposed) into the paged cache (rope.cu)
                const int head = tile, d = r_in_tile;
                const float b = bias ? bias[row] : 0.0f;
                const bool rotate = rope.denom != nullptr && head < rope.nh + rope.nkv;
                float* both = reinterpret_cast<float*>(sm.x[0]) + d;       // the other half of a pair is 64 rows, two warps, away
#pragma unroll
                for (int i = 0; i < kMine; ++i) {
                    v[i] += b;
                    // q and k are rounded to bfloat16 by the projection before they are rotated, as in the unfused path
                    both[i * BR] = rotate ? __bfloat162float(__float2bfloat16_rn(v[i])) : v[i];
                }
                asm volatile("bar.sync 1, 128;" ::: "memory");
                const size_t ld = (size_t)(rope.nh + 2 * rope.nkv) * BR;
#pragma unroll 4
                for (int i = 0; i < tokens_here; ++i) {
                    const int j = rank + i * step;
                    float y = both[i * BR];
                    if (rotate) {
                        const float2 cs = rot[i * (BR / 2) + (d & 63)];
                        const float other = d < 64 ? both[i * BR + 64] : both[i * BR - 64];
                        y = d < 64 ? y * cs.x - other * cs.y : y * cs.x + other * cs.y;
                    }
                    const bf16 r = __float2bfloat16_rn(y);
                    if (head >= rope.nh + 2 * rope.nkv) {
                        rope.extra_out[((size_t)j * rope.extra + (head - rope.nh - 2 * rope.nkv)) * BR + d] = r;
                    } else if (head < rope.nh) {
                        reinterpret_cast<bf16*>(out)[j * ld + (size_t)head * BR + d] = r;
                    } else if (rope.write) {
                        const int slot = place[i];
                        const int page = slot / rope.page_size, off = slot - page * rope.page_size;
                        if (slot < 0 || page >= rope.num_pages) continue;      // validated on the host; never write outside the cache
                        if (head < rope.nh + rope.nkv)
                            rope.kcache[(((size_t)page * rope.nkv + (head - rope.nh)) * rope.page_size + off) * BR + d] = r;
                        else
                            rope.vcache[((size_t)page * rope.nkv + (head - rope.nh - rope.nkv)) * BR * rope.page_size + (size_t)d * rope.page_size + off] = r;
                    }
                }
            } else if constexpr (kSwiglu == 0) {
                const float b = (bias && row < N) ? bias[row] : 0.0f;
#pragma unroll
                for (int i = 0; i < kMine; ++i) {
                    const int j = rank + i * step;
                    if (j < M && row < N) out[(size_t)j * N + row] = from_float<Tout>(v[i] + b);
                }
            } else {
                // rows come as 8 gate, 8 up, ...: lanes 0-7 and 16-23 hold gates, the lane 8 further on the matching up
                const int half_n = N >> 1;
                const int col = (row >> 4) * 8 + (row & 7);
#pragma unroll
                for (int i = 0; i < kMine; ++i) {
                    const int j = rank + i * step;
                    const float up = __shfl_down_sync(0xffffffffu, v[i], 8);
                    if (j < M && (lane & 8) == 0 && row + 8 < N) {
                        const float gate = v[i];
                        out[(size_t)j * half_n + col] = from_float<Tout>(glu_of<Tout, kSwiglu>(gate, up, bias));
                    }
                }
            }
        }
    }
    if constexpr (kSplit) {
        __syncwarp();
        if (warp < 2) cluster_arrive_wait();               // (the epilogue warps met there for the partial tiles)
        cluster_arrive_wait();                             // nobody leaves while its partial tile may be read
    }
    __syncwarp();
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 1) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_acc), "r"(kCols) : "memory");
    }
}

// Shared memory of a CTA that finishes `tokens` tokens: the stages, and the rotation's angles and places in the cache.
template <int BT, int kEpi, int kStages>
constexpr size_t shared_bytes(int tokens) { return sizeof(Smem<BT, kStages>) + 1024 + (kEpi == kEpiRope ? tokens * (BR / 2 * sizeof(float2) + sizeof(int)) : 0); }

int g_forced_ksplit = 0;          // > 0: this many splits of k whatever the shape (measurements)

// Splits of k: a function of N and K alone, never of the number of tokens.  One cluster a tile; the sums are read four CTAs at a time,
// and two CTAs a multiprocessor hold 30 clusters of eight and 66 of four.  Measured (us; 1, 8, 32, 64 tokens): N 3584, K 18944, five
// splits 26.1 27.1 29.2 33.8, four 27.1 27.1 28.2 29.7, eight 24.0 25.6 26.1 28.7; N 3584, K 3584, five 8.4 9.1 10.8 13.4, four 8.0 8.2
// 9.3 10.4, eight 7.8 8.6 8.6 10.2; N 4608, K 3584 four 9.8 9.8 10.9 12.1, eight 13.2 14.3 15.0 18.0; N 7168, K 5120 two 16.9 17.4 18.4
// 20.5, four 15.4 15.9 16.9 18.4; N 5120, K 5120 two 15.6 16.0 17.6 19.3, three 13.1 13.1 14.3 16.0.  (N 1536, K 8960 with twelve, three
// clusters of four that met in a workspace, 10.4 10.7, with eight 9.2 9.8.)
int choose_ksplit(int N, int K) {
    const int tiles = ceil_div(N, BR), nkb = ceil_div(K, BK), by_work = nkb / 2 > 0 ? nkb / 2 : 1;      // at least two k-blocks a CTA
    int ks = g_forced_ksplit;
    if (ks <= 0) ks = tiles <= 18 || (tiles <= 28 && nkb >= 112) ? 8 : tiles <= 37 ? 4 : tiles <= 49 ? 3 : tiles <= 60 ? 4 : tiles <= 74 ? 2 : 1;
    if (ks > by_work) ks = by_work;
    return ks < kMaxCluster ? ks : kMaxCluster;
}
int token_tile(int M) { return M <= 16 ? 16 : M <= 32 ? 32 : 64; }

// How many clusters of `csize` CTAs of a kernel the current device holds at once (asked once a size and device; a size that is asked
// by two threads at the same time is asked twice).
template <int BT, typename Tout, int kEpi, int kStages>
int clusters_at_once(int csize) {
    static std::atomic<int> known[16][9];
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 16) return 0;
    int n = known[dev][csize].load(std::memory_order_relaxed);
    if (n == 0) {
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(1, csize);
        cfg.blockDim = dim3(kThreads);
        cfg.dynamicSmemBytes = shared_bytes<BT, kEpi, kStages>(ceil_div(BT, csize));
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = attr[0].val.clusterDim.z = 1;
        attr[0].val.clusterDim.y = csize;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        if (cudaOccupancyMaxActiveClusters(&n, gemv_tcgen05_kernel<BT, Tout, kEpi, true, kStages>, &cfg) != cudaSuccess) {
            cudaGetLastError();
            n = 0;
        }
        known[dev][csize].store(n, std::memory_order_relaxed);
    }
    return n;
}

template <int BT, typename Tout, int kEpi, int kStages>
int raise_shared() {
    static LiOncePerDevice raised[2];
    const size_t smem = shared_bytes<BT, kEpi, kStages>(BT);
    cudaError_t e = li_raise_shared(raised[0], (const void*)gemv_tcgen05_kernel<BT, Tout, kEpi, false, kStages>, smem);
    if (e == cudaSuccess) e = li_raise_shared(raised[1], (const void*)gemv_tcgen05_kernel<BT, Tout, kEpi, true, kStages>, smem);
    if (e != cudaSuccess) return li_fail("linear (tcgen05 gemv): cannot raise shared memory to %zu: %s", smem, cudaGetErrorString(e));
    return 0;
}

// Deep where the launch is one wave of CTAs with a multiprocessor each: without a split as many tiles as there are
// multiprocessors at most, with one as many clusters as the device holds of that kernel at once.  (Clusters that do not all
// fit must come two CTAs a multiprocessor: 64 tokens, N 3584, K 8960, 28 clusters of five: 19.1 us, deep 32.2.)
template <int BT, typename Tout, int kEpi>
int choose_deep(int tiles, int ksplit, bool* deep) {
    *deep = false;
    if (kShallow<BT> == kDeep) return 0;
    if (ksplit == 1) {
        *deep = tiles <= kTargetCtas;
        return 0;
    }
    if (int rc = raise_shared<BT, Tout, kEpi, kDeep>()) return rc;
    *deep = (long long)tiles * ksplit <= (long long)clusters_at_once<BT, Tout, kEpi, kDeep>(ksplit) * ksplit;
    return 0;
}

template <int BT, typename Tout, int kEpi, int kStages>
int launch_stages(const CUtensorMap& map_w, const CUtensorMap& map_x, const float* bias, void* out, int M, int N, int K, int tiles, int ksplit,
                  int* err_dev, const RowScale& rs, const AddScaled& add, const RopeArgs& rope, cudaStream_t stream) {
    if (int rc = raise_shared<BT, Tout, kEpi, kStages>()) return rc;
    const size_t smem = shared_bytes<BT, kEpi, kStages>(ceil_div(M, ksplit));
    if (ksplit == 1)
        li_launch_pdl(gemv_tcgen05_kernel<BT, Tout, kEpi, false, kStages>, dim3(tiles, 1), dim3(kThreads), smem, stream, map_w, map_x, bias, (Tout*)out, M, N, K,
                      1, err_dev, rs, add, rope);
    else
        li_launch_pdl(gemv_tcgen05_kernel<BT, Tout, kEpi, true, kStages>, dim3(tiles, ksplit), dim3(kThreads), smem, stream, dim3(1, ksplit, 1), map_w, map_x,
                      bias, (Tout*)out, M, N, K, ksplit, err_dev, rs, add, rope);
    return li_check_launch("linear (tcgen05 gemv)");
}

template <int BT, typename Tout, int kEpi>
int launch(const void* a, const void* w, const float* bias, void* out, int M, int N, int K, cudaStream_t stream, const RowScale& rs,
           const AddScaled& add, const RopeArgs& rope) {
    EncodeTiledFn encode = nullptr;
    int *err_host = nullptr, *err_dev = nullptr;
    if (int rc = setup(&encode, &err_host, &err_dev)) return rc;
    if (*err_host != 0)
        return li_fail("linear (tcgen05 gemv): an earlier launch gave up waiting on a barrier (status %d); the results since then are invalid", *err_host);
    const int tiles = ceil_div(N, BR);
    const int ksplit = choose_ksplit(N, K);
    CUtensorMap map_w, map_x;
    if (int rc = make_map(&map_w, w, N, K, BR)) return rc;
    if (int rc = make_map(&map_x, a, M, K, BT)) return rc;
    bool deep = false;
    if (int rc = choose_deep<BT, Tout, kEpi>(tiles, ksplit, &deep)) return rc;
    return deep ? launch_stages<BT, Tout, kEpi, kDeep>(map_w, map_x, bias, out, M, N, K, tiles, ksplit, err_dev, rs, add, rope, stream)
                : launch_stages<BT, Tout, kEpi, kShallow<BT>>(map_w, map_x, bias, out, M, N, K, tiles, ksplit, err_dev, rs, add, rope, stream);
}

template <typename Tout, int kEpi>
int launch_bt(const void* a, const void* w, const float* bias, void* out, int M, int N, int K, cudaStream_t stream, const RowScale& rs,
              const AddScaled& add = AddScaled{}, const RopeArgs& rope = RopeArgs{}) {
    if (M <= 16) return launch<16, Tout, kEpi>(a, w, bias, out, M, N, K, stream, rs, add, rope);
    if (M <= 32) return launch<32, Tout, kEpi>(a, w, bias, out, M, N, K, stream, rs, add, rope);
    return launch<64, Tout, kEpi>(a, w, bias, out, M, N, K, stream, rs, add, rope);
}

}  // namespace

// 0: splits of k by shape; n > 0: n splits, as far as there are k-blocks for them and a cluster holds them
// (li_gemv_tcgen05_plan says how many it became).  For measurements.
LI_EXPORT void li_gemv_tcgen05_force_ksplit(int n) { g_forced_ksplit = n; }

// How a product of M <= 64 rows is cut: the splits of k, and how many of them form a cluster; with `deep` (needs a device)
// whether its plain form takes the deep pipeline.  For tests.
LI_EXPORT int li_gemv_tcgen05_plan(int M, int N, int K, int* splits, int* cluster, int* deep) {
    LI_REQUIRE(M >= 1 && M <= 64 && N >= 1 && K >= 8 && splits && cluster, "linear (tcgen05 gemv): no plan for M=%d N=%d K=%d", M, N, K);
    *splits = choose_ksplit(N, K);
    *cluster = *splits;
    if (deep) {
        bool d = false;
        const int tiles = ceil_div(N, BR);
        if (int rc = token_tile(M) == 16 ? choose_deep<16, bf16, kEpiNone>(tiles, *splits, &d)
                     : token_tile(M) == 32 ? choose_deep<32, bf16, kEpiNone>(tiles, *splits, &d) : choose_deep<64, bf16, kEpiNone>(tiles, *splits, &d))
            return rc;
        *deep = d;
    }
    return 0;
}

bool li_gemv_tcgen05_accepts(const void* a, const void* w, int M, int N, int K) {
    return M >= 1 && M <= 64 && N >= 1 && K >= 8 && K % 8 == 0 && ((uintptr_t)a % 16 == 0) && ((uintptr_t)w % 16 == 0);
}

int li_linear_gemv_tcgen05(const void* a, const void* w, const float* bias, void* out, int dtype_out, int M, int N, int K,
                           int epilogue, cudaStream_t stream, const RowScale& rs) {
    LI_REQUIRE(li_gemv_tcgen05_accepts(a, w, M, N, K), "linear (tcgen05 gemv): refuses M=%d N=%d K=%d (M <= 64, K a multiple of 8, 16-byte aligned operands)", M, N, K);
    if (li_epilogue_is_gated(epilogue)) {
        LI_REQUIRE(N % 16 == 0 && li_epilogue_bias_ok(epilogue, bias) && dtype_out == LI_BF16,
                   "linear (tcgen05 gemv): the swiglu epilogue needs N a multiple of 16, no bias and bfloat16 output");
        return epilogue == LI_EPILOGUE_GLU_CLAMPED ? launch_bt<bf16, kEpiGluClamped>(a, w, bias, out, M, N, K, stream, rs)
               : epilogue == LI_EPILOGUE_GEGLU     ? launch_bt<bf16, kEpiGeglu>(a, w, bias, out, M, N, K, stream, rs)
                                                   : launch_bt<bf16, kEpiSwiglu>(a, w, bias, out, M, N, K, stream, rs);
    }
    if (dtype_out == LI_BF16) return launch_bt<bf16, kEpiNone>(a, w, bias, out, M, N, K, stream, rs);
    if (dtype_out == LI_F32) return launch_bt<float, kEpiNone>(a, w, bias, out, M, N, K, stream, rs);
    return li_fail("linear (tcgen05 gemv): unsupported output dtype %d", dtype_out);
}

// The fused q|k|v projection with rotary encoding and cache write in its epilogue: heads of 128 (rotated whole or not at all),
// a tile a head.  Against the register-fed kernel's (li_linear_gemv_rope) where its rows are long: rope.cu says from where.
bool li_gemv_tcgen05_rope_accepts(const void* a, const void* w, int M, int N, int K, int nh, int nkv, int dh, int rotary_dim) {
    return li_gemv_tcgen05_accepts(a, w, M, N, K) && dh == BR && (rotary_dim == dh || rotary_dim == 0) && N == (nh + 2 * nkv) * dh;
}

int li_linear_gemv_tcgen05_rope(const void* a, const void* w, const float* bias, void* out, int M, int N, int K, const RopeArgs& rope, const RowScale& rs,
                                cudaStream_t stream) {
    return launch_bt<bf16, kEpiRope>(a, w, bias, out, M, N + rope.extra * BR, K, stream, rs, AddScaled{}, rope);
}

// x32 += a w^T (+ bias), hprime = bfloat16(norm_weight * x32), ssq_out[token, tile] = sums of squares (row_scale.cuh).
int li_gemv_tcgen05_tiles(int N) { return ceil_div(N, BR); }

int li_linear_gemv_tcgen05_add_scaled(const void* a, const void* w, const float* bias, int M, int N, int K, const AddScaled& add,
                                      cudaStream_t stream) {
    LI_REQUIRE(li_gemv_tcgen05_accepts(a, w, M, N, K), "linear + add (tcgen05 gemv): refuses M=%d N=%d K=%d", M, N, K);
    return launch_bt<bf16, kEpiAddScaled>(a, w, bias, add.hprime, M, N, K, stream, RowScale{}, add);
}

// out[M, N] = a[M, K] w[N, K]^T for products of many tiles (a prefill step's): a persistent form of the tcgen05 GEMM in
// which the epilogue of one tile runs while the tensor cores work on the next.
//
// With k = 1536 a tile's main loop is only 24 k-blocks long; filling the pipeline and, above all, the epilogue (SwiGLU and
// the stores of a 256 x 256 tile) then cost as much as the products, and a kernel that does one tile per CTA cannot
// overlap them.  Here one pair of CTAs per pair of multiprocessors (a cluster of two, tcgen05.mma cta_group::2) walks over
// tiles of 256 x 256: each CTA brings its own 128 rows of a and half of the 256 rows of w per k-block (32 KB a stage, six
// stages) and keeps the accumulator of its rows, 256 columns of tensor memory.  The other 256 columns hold the tile before:
// the four epilogue warps of each CTA read it, apply bias or SwiGLU and store, while the first CTA's issuer already
// multiplies the next tile; the producers run ahead through the ring of stages without regard to tile boundaries.
// Products in groups (a mixture's experts): every 256 rows of a belong to one group, which a table on the device names; the
// groups' matrices lie one below the other in the tensor map of w, a tile adds group * N to its row there, and tiles of no group
// are passed over by every role alike.
// Tiles are taken in the order (row pair fastest, then columns), so that the pairs at work at one time share few tiles of w.
//
// Barriers: full / empty per stage as in gemm_tcgen05.cu (both CTAs' loads are counted on the first CTA's full barrier; the
// commit that frees a stage arrives in both); acc_full per accumulator (commit to both CTAs); acc_empty per accumulator in
// the first CTA, on which the epilogue warps of both CTAs arrive.  Every wait is bounded; a wait that runs out raises the
// status word of the tcgen05 kernels, and every role leaves its loops and meets the others at the final barriers.
#define LI_PDL_KIND 1
#include "gemm_epilogue.cuh"
#include "rope_epilogue.cuh"
#include "tcgen05.cuh"

#include <algorithm>

namespace {

using namespace tc;

constexpr int kRows = 128;          // rows of a per CTA
constexpr int BN = 256;             // columns of a tile
constexpr int kStages = 6;
constexpr int kThreads = 192;
constexpr int kBytesA = kRows * BK * 2, kBytesB = (BN / 2) * BK * 2;

__host__ __device__ constexpr int cdiv(int a, int b) { return (a + b - 1) / b; }

struct __align__(1024) Smem {
    unsigned char a[kStages][kBytesA];
    unsigned char b[kStages][kBytesB];
    unsigned long long full[kStages];
    unsigned long long empty[kStages];
    unsigned long long acc_full[2];
    unsigned long long acc_empty[2];
    unsigned tmem_base;
};

template <typename Tout, int kSwiglu>
__global__ void __launch_bounds__(kThreads, 1)
gemm_tcgen05_persistent_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_w,
                               const float* __restrict__ bias, Tout* __restrict__ out, int M, int N, int K, int* __restrict__ error_flag,
                               const int* __restrict__ tile_group) {
    extern __shared__ unsigned char smem_raw[];
    Smem& sm = *reinterpret_cast<Smem*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const unsigned rank = cluster_cta_rank();
    const int pair = blockIdx.x >> 1, npairs = gridDim.x >> 1;
    const int row_pairs = (cdiv(M, kRows) + 1) >> 1, col_tiles = cdiv(N, BN);
    const int total = row_pairs * col_tiles;
    const int nkb = cdiv(K, BK);
    constexpr unsigned kCols = 512;

    if (threadIdx.x == 0) {
        for (int s = 0; s < kStages; ++s) {
            mbar_init(&sm.full[s], 1);
            mbar_init(&sm.empty[s], 1);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(&sm.acc_full[b], 1);
            mbar_init(&sm.acc_empty[b], 8);          // four epilogue warps in each of the two CTAs
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    // Tensor memory is taken only once the kernel before this one has finished: a CTA that waits for that kernel must not
    // hold what a CTA of it may still ask for (gemm_tcgen05.cu has the story).  Nothing here could start before that anyway.
    // The kernel behind this one is let go once this CTA holds its columns.
    pdl_wait();
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&sm.tmem_base)), "r"(kCols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    pdl_launch_dependents();
    cluster_sync_all();                               // the other CTA's barriers are set up before anything arrives on them
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const unsigned tmem_acc = sm.tmem_base;

    if (warp == 0) {
        if (lane == 0) {
            bool ok = true;
            int it = 0;                               // k-blocks loaded so far, over all tiles
            for (int t = pair; t < total && ok; t += npairs) {
                const int group = tile_group ? tile_group[t % row_pairs] : 0;
                if (group < 0) continue;
                const int m0 = ((t % row_pairs) * 2 + (int)rank) * kRows, n0 = (t / row_pairs) * BN;
                for (int kb = 0; kb < nkb; ++kb, ++it) {
                    const int s = it % kStages;
                    ok = mbar_wait(&sm.empty[s], ((it / kStages) & 1) ^ 1);
                    if (!ok) break;
                    if (rank == 0) mbar_expect_tx(&sm.full[s], 2 * (kBytesA + kBytesB));
                    tma_load_2d_pair(sm.a[s], &map_a, kb * BK, m0, &sm.full[s]);
                    tma_load_2d_pair(sm.b[s], &map_w, kb * BK, group * N + n0 + (int)rank * (BN / 2), &sm.full[s]);
                }
            }
            if (!ok) atomicExch(error_flag, 21);
        }
    } else if (warp == 1) {
        if (lane == 0 && rank == 0) {                 // the first CTA issues the products of both
            constexpr unsigned idesc = umma_idesc(2 * kRows, BN);
            bool ok = true;
            int it = 0, ti = 0;
            for (int t = pair; t < total && ok; t += npairs) {
                if (tile_group && tile_group[t % row_pairs] < 0) continue;
                const unsigned acc = tmem_acc + (unsigned)((ti & 1) * BN);
                ok = mbar_wait(&sm.acc_empty[ti & 1], ((ti >> 1) & 1) ^ 1);     // both epilogues are done with this accumulator
                if (!ok) break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                for (int kb = 0; kb < nkb; ++kb, ++it) {
                    const int s = it % kStages;
                    ok = mbar_wait(&sm.full[s], (it / kStages) & 1);
                    if (!ok) break;
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    const unsigned long long da = umma_desc(sm.a[s]), db = umma_desc(sm.b[s]);
#pragma unroll
                    for (int k = 0; k < BK / 16; ++k)
                        umma_bf16_pair(acc, da + (unsigned long long)(k * 2), db + (unsigned long long)(k * 2), idesc, (kb | k) ? 1u : 0u);
                    umma_commit_pair(&sm.empty[s]);
                }
                if (ok) umma_commit_pair(&sm.acc_full[ti & 1]);
                ++ti;
            }
            if (!ok) atomicExch(error_flag, 22);
        }
    } else {
        // epilogue: warp w may read the tensor-memory lanes 32 (w % 4) .. 32 (w % 4) + 31
        const int quarter = warp & 3;
        bool ok = true;
        int ti = 0;
        for (int t = pair; t < total && ok; t += npairs) {
            if (tile_group && tile_group[t % row_pairs] < 0) continue;
            const int m0 = ((t % row_pairs) * 2 + (int)rank) * kRows, n0 = (t / row_pairs) * BN;
            ok = mbar_wait(&sm.acc_full[ti & 1], (ti >> 1) & 1);
            if (!ok) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const unsigned acc = tmem_acc + ((unsigned)(quarter * 32) << 16) + (unsigned)((ti & 1) * BN);
#pragma unroll 1
            for (int c = 0; c < BN; c += 32) {
                float v[32];
                tmem_ld_32x32(acc + (unsigned)c, v);
                gemm_store_piece<Tout, kSwiglu>(m0 + quarter * 32 + lane, n0 + c, v, bias, out, M, N);
            }
            // this warp has read its lanes of the accumulator: one arrival on the first CTA's barrier
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive_remote(&sm.acc_empty[ti & 1], 0);
            ++ti;
        }
        if (!ok && lane == 0) atomicExch(error_flag, 23);
    }
    __syncwarp();
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    cluster_sync_all();                               // neither CTA frees tensor memory or leaves while the other may still use it
    if (warp == 1) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_acc), "r"(kCols) : "memory");
    }
}

template <typename Tout, int kSwiglu>
int launch(const void* a, const void* w, const float* bias, void* out, int M, int N, int K, cudaStream_t stream, const int* tile_group = nullptr, int G = 1) {
    EncodeTiledFn encode = nullptr;
    int *err_host = nullptr, *err_dev = nullptr;
    if (int rc = setup(&encode, &err_host, &err_dev)) return rc;
    if (*err_host != 0)
        return li_fail("linear (tcgen05, persistent): an earlier launch gave up waiting on a barrier (status %d); the results since then are invalid", *err_host);
    CUtensorMap map_a, map_w;
    if (int rc = make_map(&map_a, a, M, K, kRows)) return rc;
    if (int rc = make_map(&map_w, w, G * N, K, BN / 2)) return rc;
    const size_t smem = sizeof(Smem) + 1024;
    static LiOncePerDevice raised;
    cudaError_t e = li_raise_shared(raised, (const void*)gemm_tcgen05_persistent_kernel<Tout, kSwiglu>, smem);
    if (e != cudaSuccess) return li_fail("linear (tcgen05, persistent): cannot raise shared memory to %zu: %s", smem, cudaGetErrorString(e));
    const int total = ((ceil_div(M, kRows) + 1) / 2) * ceil_div(N, BN);
    int pairs = li_multiprocessors() / 2;
    if (pairs > total) pairs = total;
    li_launch_pdl(gemm_tcgen05_persistent_kernel<Tout, kSwiglu>, dim3(2 * pairs), dim3(kThreads), smem, stream, dim3(2, 1, 1), map_a, map_w, bias,
                  (Tout*)out, M, N, K, err_dev, tile_group);
    return li_check_launch("linear (tcgen05, persistent)");
}

}  // namespace

// Worth it when a pair of multiprocessors gets more than one tile (measured against 256 x 256 tiles of one CTA each: gate|up of
// K 1536 and 512 rows, 140 tiles: 29 us against 33 us; 2,048 rows: 94 us against 138 us; K 5120, N 27648: 640 rows 149 against
// 184 us, 2,048 rows 385 against 428 us; K 13824, N 5120, 2,048 rows 224 against 300 us), except where the single CTAs fill one
// wave (up to 148 tiles: a pair then takes two of its tiles in the time a CTA takes one of its own) and k is so long that the
// epilogue hardly counts: 2,048 rows, N 4096, 128 tiles, K 4160 66.6 against 68.6 us, K 8192 111.0 against 107.8, K 13824 183.0
// against 175.9; 150 tiles, K 13824 228 against 300.
bool li_tcgen05_persistent_wanted(int M, int N, int K) {
    const long long total = (long long)((ceil_div(M, kRows) + 1) / 2) * ceil_div(N, BN);
    return total >= 120 && (total > 148 || ceil_div(K, BK) < 128);
}

// The same, for tests of the rule.
LI_EXPORT int li_tcgen05_takes_persistent(int M, int N, int K) { return li_tcgen05_persistent_wanted(M, N, K) ? 1 : 0; }

int li_linear_tcgen05_persistent(const void* a, const void* w, const float* bias, void* out, int dtype_out, int M, int N, int K, int epilogue,
                                 cudaStream_t stream) {
    if (li_epilogue_is_gated(epilogue)) {
        LI_REQUIRE(N % 16 == 0 && li_epilogue_bias_ok(epilogue, bias) && dtype_out == LI_BF16,
                   "linear (tcgen05, persistent): the swiglu epilogue needs N a multiple of 16, no bias and bfloat16 output");
        return epilogue == LI_EPILOGUE_GLU_CLAMPED ? launch<bf16, 2>(a, w, bias, out, M, N, K, stream)
               : epilogue == LI_EPILOGUE_GEGLU     ? launch<bf16, 3>(a, w, bias, out, M, N, K, stream)
                                                   : launch<bf16, 1>(a, w, bias, out, M, N, K, stream);
    }
    if (dtype_out == LI_BF16) return launch<bf16, 0>(a, w, bias, out, M, N, K, stream);
    if (dtype_out == LI_F32) return launch<float, 0>(a, w, bias, out, M, N, K, stream);
    return li_fail("linear (tcgen05, persistent): unsupported output dtype %d", dtype_out);
}

// Products in groups on pairs of CTAs: a [M, K] with M a multiple of 256, every 256 rows of one group (tile_group[M / 256], -1:
// none); w [G, N, K]; out [M, N] bfloat16, or [M, N / 2] with a gated epilogue.
int li_linear_tcgen05_grouped_pairs(const void* a, const void* w, void* out, int M, int N, int K, int G, const int* tile_group, int epilogue,
                                    const float* glu_params, cudaStream_t stream) {
    LI_REQUIRE(M % (2 * kRows) == 0 && G >= 1 && tile_group != nullptr, "grouped linear (tcgen05, pairs): rows %d must be whole tiles of 256 with a table of their groups", M);
    LI_REQUIRE(K >= 8 && K % 8 == 0 && ((uintptr_t)a % 16 == 0) && ((uintptr_t)w % 16 == 0), "grouped linear (tcgen05, pairs): refuses K=%d or unaligned operands", K);
    LI_REQUIRE((long long)G * N < (1LL << 31), "grouped linear (tcgen05, pairs): %d matrices of %d rows are too many", G, N);
    const bool gated = li_epilogue_is_gated(epilogue);
    LI_REQUIRE(!gated || N % 16 == 0, "grouped linear (tcgen05, pairs): a gated epilogue needs N a multiple of 16, got %d", N);
    if (epilogue == LI_EPILOGUE_GLU_CLAMPED) return launch<bf16, 2>(a, w, glu_params, out, M, N, K, stream, tile_group, G);
    if (epilogue == LI_EPILOGUE_GEGLU) return launch<bf16, 3>(a, w, nullptr, out, M, N, K, stream, tile_group, G);
    if (gated) return launch<bf16, 1>(a, w, nullptr, out, M, N, K, stream, tile_group, G);
    return launch<bf16, 0>(a, w, nullptr, out, M, N, K, stream, tile_group, G);
}

// ---------------------------------------------------------------------------------------------
// tokens as columns
// ---------------------------------------------------------------------------------------------
// out[M, N] = a[M, K] w[N, K]^T in bfloat16 on the fifth-generation tensor cores with the roles of the operands swapped: 256 rows of
// w are the M side of tcgen05.mma, the tokens its N side.  For steps of a few hundred tokens: the N side comes in steps of 32, so
// that 544 tokens are two tiles of 288 and not three of 256 (where the tokens are the M side, 29 % of the work is padding), and a
// tile of up to 512 tokens reads its rows of w once.
//
// Persistent like the kernel above: one pair of CTAs per pair of multiprocessors (cta_group::2) walks over tiles of 256
// rows of w by up to 512 tokens; each CTA brings its own 128 rows of w and half of the tokens' rows per k-block, through a ring of as
// many stages as fit.  Up to 256 tokens two accumulators take turns and the epilogue of a tile runs while the next is multiplied;
// wider tiles (two products of up to 256 columns a k-step) have one accumulator, and their epilogue shows.  What bounds the main loop
// is the tensor pipe, and up to 256 tokens the loop of the one thread that issues its products: the width is chosen by the time that
// they take in whole waves of pairs (plan_of).
// The epilogue's thread has one row of w and 32 tokens: neighbouring lanes exchange values so that stores are pairs of columns.
// With rotary encoding a tile of rows is loaded in pieces of 16 so that the two halves of a rotation pair lie 16 lanes apart.
//
// Barriers as above; every wait is bounded.

namespace {
namespace columns {

constexpr int kRows = 128;                       // rows of w per CTA
constexpr int kEpilogueWarps = 8, kThreads = 64 + 32 * kEpilogueWarps;
constexpr int kMaxStages = 8;
constexpr int kRingBytes = 216 * 1024;
constexpr int kBytesW = kRows * BK * 2;
constexpr int kRope = 4;                         // epilogue: 0 none, 1 to 3 gated (glu_of), 4 rotation and cache

__host__ __device__ constexpr int stage_bytes(int tokens) { return kBytesW + tokens / 2 * BK * 2; }
__host__ __device__ constexpr int stages_of(int tokens) { return kRingBytes / stage_bytes(tokens) < kMaxStages ? kRingBytes / stage_bytes(tokens) : kMaxStages; }

struct Barriers {
    unsigned long long full[kMaxStages];
    unsigned long long empty[kMaxStages];
    unsigned long long acc_full[2];
    unsigned long long acc_empty[2];
    unsigned long long peer_alloc;
    unsigned tmem_base;
};

// A head's 128 rows of w as rows 0 - 15 and 64 - 79, 16 - 31 and 80 - 95, ...: the map has the dimensions k, row of a piece, half, piece,
// head.
__device__ __forceinline__ void tma_load_head_pair(void* dst, const CUtensorMap* map, int k0, int head, unsigned long long* bar) {
    asm volatile(
        "cp.async.bulk.tensor.5d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %5, %5, %5, %4}], [%2];"
        ::"r"(smem_u32(dst)), "l"(map), "r"(smem_u32(bar) & 0xFEFFFFFFu), "r"(k0), "r"(head), "r"(0)
        : "memory");
}

// Two neighbouring lanes hold columns f and f + 1 (f even) of two tokens: the even lane gets the first token's pair, the odd one the
// second's.
__device__ __forceinline__ unsigned pair_up(float first, float second, bool odd) {
    const float got = __shfl_xor_sync(0xffffffffu, odd ? first : second, 1);
    const __nv_bfloat162 h = odd ? __floats2bfloat162_rn(got, second) : __floats2bfloat162_rn(first, got);
    return *reinterpret_cast<const unsigned*>(&h);
}

// 32 tokens (tok0 ..) of row `row` of w.
template <typename Tout>
__device__ __forceinline__ void store_plain(float (&v)[32], int row, int tok0, int lane, const float* __restrict__ bias, Tout* __restrict__ out, int M, int N) {
    const float b = bias && row < N ? bias[row] : 0.0f;
    if constexpr (sizeof(Tout) == 2) {
        if (N % 2 == 0 && ((uintptr_t)out & 3) == 0) {         // the same for all
            const bool odd = lane & 1;
#pragma unroll
            for (int i = 0; i < 32; i += 2) {
                const unsigned u = pair_up(v[i] + b, v[i + 1] + b, odd);
                const int tok = tok0 + i + odd;
                if (tok < M && row < N) *reinterpret_cast<unsigned*>(out + (size_t)tok * N + (row & ~1)) = u;
            }
            return;
        }
    }
#pragma unroll
    for (int i = 0; i < 32; ++i)
        if (tok0 + i < M && row < N) out[(size_t)(tok0 + i) * N + row] = from_float<Tout>(v[i] + b);
}

// Rows of w come as 8 gate, 8 up: of two tokens the gate's lane takes the first, the up's lane the second.
template <typename Tout, int kGlu>
__device__ __forceinline__ void store_gated(float (&v)[32], int row, int tok0, int lane, const float* __restrict__ params, Tout* __restrict__ out, int M, int N) {
    const bool is_up = lane & 8, odd = lane & 1;
    const int half = N >> 1, col = (row >> 4) * 8 + (row & 7);
#pragma unroll
    for (int i = 0; i < 32; i += 4) {
        float r[2];
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            const float first = v[i + 2 * q], second = v[i + 2 * q + 1];
            const float got = __shfl_xor_sync(0xffffffffu, is_up ? first : second, 8);
            r[q] = is_up ? glu_of<Tout, kGlu>(got, second, params) : glu_of<Tout, kGlu>(first, got, params);
        }
        // r[0]: token i (+ 1 in an up's lane), r[1]: token i + 2 (+ 1)
        const unsigned u = pair_up(r[0], r[1], odd);
        const int tok = tok0 + i + 2 * odd + is_up;
        if (tok < M && row < N) *reinterpret_cast<unsigned*>(out + (size_t)tok * half + (col & ~1)) = u;
    }
}

// One head.  d: this lane's element of it; its partner in the rotation is 16 lanes away.
__device__ __forceinline__ void store_rope(float (&v)[32], int head, int d, int tok0, int lane, const float* __restrict__ bias, bf16* __restrict__ out, int M, int N,
                                           const RopeEpilogue& re) {
    const float b = bias ? bias[head * 128 + d] : 0.0f;
    const bool odd = lane & 1, second_half = d >= 64;
    // lane i looks token i's place in the cache up
    int page = -1, off = 0, slot = -1;
    if (head >= re.nh && re.write && tok0 + lane < M) {
        slot = re.slot_mapping[tok0 + lane];
        page = slot / re.page_size;
        off = slot - page * re.page_size;
        if (slot < 0 || page >= re.num_pages) page = -1;       // validated on the host; never write outside the cache
    }
    if (head < re.nh + re.nkv) {
        // (all asked for before the first store, behind which none of them could go: a load after the other took 50 us for 2,048 tokens,
        // N 2048, K 1536)
        const float2* cs = reinterpret_cast<const float2*>(re.cos_sin) + (d & 63);
        float2 t[32];
#pragma unroll
        for (int i = 0; i < 32; ++i) t[i] = __ldg(cs + (size_t)min(tok0 + i, M - 1) * 64);
        bf16* kbase = re.kcache + (size_t)(head - re.nh) * re.page_size * 128;
#pragma unroll
        for (int i = 0; i < 32; i += 2) {
            float y[2];
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                // q and k are rounded to bfloat16 by the projection before they are rotated, as in the unfused path
                const float x = __bfloat162float(__float2bfloat16_rn(v[i + q] + b));
                const float other = __shfl_xor_sync(0xffffffffu, x, 16);
                y[q] = second_half ? x * t[i + q].x + other * t[i + q].y : x * t[i + q].x - other * t[i + q].y;
            }
            const unsigned u = pair_up(y[0], y[1], odd);
            const int p = __shfl_sync(0xffffffffu, page, i + odd), o = __shfl_sync(0xffffffffu, off, i + odd);
            const int tok = tok0 + i + odd;
            if (head < re.nh) {
                if (tok < M) *reinterpret_cast<unsigned*>(out + (size_t)tok * N + (size_t)head * 128 + (d & ~1)) = u;
            } else if (p >= 0) {
                *reinterpret_cast<unsigned*>(kbase + (size_t)p * re.nkv * re.page_size * 128 + (size_t)o * 128 + (d & ~1)) = u;
            }
        }
    } else {
        // values are cached transposed: a lane's tokens lie one behind the other where their places do
        bf16* vbase = re.vcache + (size_t)(head - re.nh - re.nkv) * 128 * re.page_size + (size_t)d * re.page_size;
        const int before = __shfl_up_sync(0xffffffffu, slot, 1);
        const unsigned follows = __ballot_sync(0xffffffffu, page >= 0 && slot == before + 1);
#pragma unroll
        for (int i = 0; i < 32; i += 8) {
            const int p = __shfl_sync(0xffffffffu, page, i), o = __shfl_sync(0xffffffffu, off, i);
            if (p >= 0 && o % 8 == 0 && ((follows >> (i + 1)) & 0x7fu) == 0x7fu) {       // the same for the warp
                unsigned u[4];
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    const __nv_bfloat162 h = __floats2bfloat162_rn(v[i + 2 * q] + b, v[i + 2 * q + 1] + b);
                    u[q] = *reinterpret_cast<const unsigned*>(&h);
                }
                *reinterpret_cast<uint4*>(vbase + (size_t)p * re.nkv * 128 * re.page_size + o) = make_uint4(u[0], u[1], u[2], u[3]);
            } else {
#pragma unroll
                for (int q = 0; q < 8; ++q) {
                    const int pq = __shfl_sync(0xffffffffu, page, i + q), oq = __shfl_sync(0xffffffffu, off, i + q);
                    if (pq >= 0) vbase[(size_t)pq * re.nkv * 128 * re.page_size + oq] = __float2bfloat16_rn(v[i + q] + b);
                }
            }
        }
    }
}

// A tile's tokens are the columns of one product, or (kWide) of two side by side: `sub` and `sub2` (or 0) of them, multiples of 32 up to
// 256.
template <typename Tout, int kEpi, bool kWide>
__global__ void __launch_bounds__(kThreads, 1)
gemm_tcgen05_tokens_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_x, const __grid_constant__ CUtensorMap map_x2,
                           const float* __restrict__ bias, Tout* __restrict__ out, int M, int N, int K, int sub, int sub2, int* __restrict__ error_flag, const RopeEpilogue rope) {
    extern __shared__ unsigned char smem_raw[];
    __shared__ Barriers br;
    unsigned char* ring = reinterpret_cast<unsigned char*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const unsigned rank = cluster_cta_rank();
    const int pair = blockIdx.x >> 1, npairs = gridDim.x >> 1;
    const int width = sub + sub2, token_tiles = cdiv(M, width), total = token_tiles * cdiv(N, 2 * kRows);
    const int nkb = cdiv(K, BK), bytes = stage_bytes(width), stages = stages_of(width);
    constexpr int buffers = kWide ? 1 : 2;                // accumulators, 256 columns apart
    constexpr unsigned kCols = 512;

    if (threadIdx.x == 0) {
        for (int s = 0; s < stages; ++s) {
            mbar_init(&br.full[s], 1);
            mbar_init(&br.empty[s], 1);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(&br.acc_full[b], 1);
            mbar_init(&br.acc_empty[b], 2 * kEpilogueWarps);
        }
        mbar_init(&br.peer_alloc, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    cluster_sync_all();                                    // the other CTA's barriers are set up before anything arrives on them

    // Tensor memory is taken only once the kernel before this one has finished, and the kernel behind this one let go only once it is
    // held (gemm_tcgen05.cu has the story).  The warps that read the accumulator meet warp 1 at a named barrier.
    auto meet_tensor_memory = [&]() {
        asm volatile("bar.sync 3, %0;" ::"n"(32 + 32 * kEpilogueWarps) : "memory");
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        return br.tmem_base;
    };

    if (warp == 0) {
        if (lane == 0) {
            // (no division in here: it once made the loop of this one thread the longest of all, 540 ns a k-block whatever the width)
            int row = 0, m0 = 0;
            auto tile_at = [&](int t) {
                row = t / token_tiles * 2 * kRows + (int)rank * kRows;
                m0 = t % token_tiles * width;
            };
            auto load_w = [&](int kb, int s) {
                if constexpr (kEpi == kRope) tma_load_head_pair(ring + s * bytes, &map_w, kb * BK, row / kRows, &br.full[s]);
                else tma_load_2d_pair(ring + s * bytes, &map_w, kb * BK, row, &br.full[s]);
            };
            auto load_x = [&](int kb, int s) {
                unsigned char* to = ring + s * bytes + kBytesW;
                tma_load_2d_pair(to, &map_x, kb * BK, m0 + (int)rank * (sub / 2), &br.full[s]);
                if constexpr (kWide) tma_load_2d_pair(to + sub / 2 * BK * 2, &map_x2, kb * BK, m0 + sub + (int)rank * (sub2 / 2), &br.full[s]);
            };
            tile_at(pair);
            // the weights of the first stages do not depend on the kernel before
            const int first = nkb < stages ? nkb : stages;
            for (int kb = 0; kb < first; ++kb) {
                if (rank == 0) mbar_expect_tx(&br.full[kb], 2 * bytes);
                load_w(kb, kb);
            }
            pdl_wait();
            for (int kb = 0; kb < first; ++kb) load_x(kb, kb);
            bool ok = true;
            int issued = first, kb = first, s = first == stages ? 0 : first;
            unsigned phase = first == stages ? 0u : 1u;    // of the wait for stage s: the first round does not wait
            for (int t = pair; t < total && ok; t += npairs, kb = 0) {
                tile_at(t);
                for (; kb < nkb; ++kb, ++issued) {
                    ok = mbar_wait(&br.empty[s], phase);
                    if (!ok) break;
                    if (rank == 0) mbar_expect_tx(&br.full[s], 2 * bytes);
                    load_w(kb, s);
                    load_x(kb, s);
                    if (++s == stages) s = 0, phase ^= 1;
                }
            }
            if (!ok) {
                atomicExch(error_flag, 51);
                // the copies already issued must land before the CTA may leave (only the first CTA can tell)
                if (rank == 0)
                    for (int i = (issued > stages ? issued - stages : 0); i < issued; ++i) mbar_wait(&br.full[i % stages], (i / stages) & 1);
            }
        }
    } else if (warp == 1) {
        pdl_wait();
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&br.tmem_base)), "r"(kCols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
        pdl_launch_dependents();
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        const unsigned tmem_acc = meet_tensor_memory();
        if (lane == 0 && rank == 1) mbar_arrive_remote(&br.peer_alloc, 0);
        if (lane == 0 && rank == 0) {                      // the first CTA issues the products of both
            const unsigned idesc = umma_idesc(2 * kRows, sub), idesc2 = umma_idesc(2 * kRows, sub2);
            bool ok = mbar_wait(&br.peer_alloc, 0);        // the products write the second CTA's tensor memory too
            // descriptors count in units of 16 bytes
            const unsigned long long first = umma_desc(ring), second = (unsigned long long)(sub / 2 * BK * 2 / 16), step = (unsigned long long)(bytes / 16);
            unsigned long long da = first;
            int s = 0, b = 0;
            unsigned phase = 0, acc_phase = 1;
            for (int t = pair; t < total && ok; t += npairs) {
                const unsigned acc = tmem_acc + (unsigned)(b * 256);
                ok = mbar_wait(&br.acc_empty[b], acc_phase);       // both epilogues are done with this accumulator
                if (!ok) break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                unsigned accumulate = 0;
                for (int kb = 0; kb < nkb; ++kb) {
                    ok = mbar_wait(&br.full[s], phase);
                    if (!ok) break;
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    const unsigned long long db = da + (unsigned long long)(kBytesW / 16);
#pragma unroll
                    for (int k = 0; k < BK / 16; ++k) {
                        umma_bf16_pair(acc, da + (unsigned long long)(k * 2), db + (unsigned long long)(k * 2), idesc, accumulate);
                        if constexpr (kWide)
                            umma_bf16_pair(acc + (unsigned)sub, da + (unsigned long long)(k * 2), db + second + (unsigned long long)(k * 2), idesc2, accumulate);
                        accumulate = 1;
                    }
                    umma_commit_pair(&br.empty[s]);
                    da += step;
                    if (++s == stages) s = 0, phase ^= 1, da = first;
                }
                if (ok) umma_commit_pair(&br.acc_full[b]);
                if (++b == buffers) b = 0, acc_phase ^= 1;
            }
            if (!ok) atomicExch(error_flag, 52);
        }
    } else {
        // epilogue: warp w may read the tensor-memory lanes 32 (w % 4) .. 32 (w % 4) + 31; two warps share them, every other 32 tokens each
        const unsigned tmem_acc = meet_tensor_memory();
        pdl_wait();
        const int quarter = warp & 3, part = (warp - 2) >> 2;
        bool ok = true;
        int b = 0;
        unsigned phase = 0;
        for (int t = pair; t < total && ok; t += npairs) {
            const int m0 = t % token_tiles * width, row0 = t / token_tiles * 2 * kRows + (int)rank * kRows;
            ok = mbar_wait(&br.acc_full[b], phase);
            if (!ok) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const unsigned acc = tmem_acc + ((unsigned)(quarter * 32) << 16) + (unsigned)(b * 256);
#pragma unroll 1
            for (int c = 32 * part; c < width && m0 + c < M; c += 64) {
                float v[32];
                tmem_ld_32x32(acc + (unsigned)c, v);
                if constexpr (kEpi == kRope) {
                    if (row0 < N)                          // (a tile of two heads may have but one)
                        store_rope(v, row0 / 128, (lane & 15) + 16 * quarter + (lane & 16) * 4, m0 + c, lane, bias, reinterpret_cast<bf16*>(out), M, N, rope);
                } else if constexpr (kEpi != 0) {
                    store_gated<Tout, kEpi>(v, row0 + quarter * 32 + lane, m0 + c, lane, bias, out, M, N);
                } else {
                    store_plain<Tout>(v, row0 + quarter * 32 + lane, m0 + c, lane, bias, out, M, N);
                }
            }
            // this warp has read its part of the accumulator: one arrival on the first CTA's barrier
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive_remote(&br.acc_empty[b], 0);
            if (++b == buffers) b = 0, phase ^= 1;
        }
        if (!ok && lane == 0) atomicExch(error_flag, 53);
    }
    __syncwarp();
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    cluster_sync_all();                                    // neither CTA frees tensor memory or leaves while the other may still use it
    if (warp == 1) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(br.tmem_base), "r"(kCols) : "memory");
    }
}

// How the tokens are cut, and what it should take in microseconds.
struct Plan {
    int width = 0;
    double us = 0.0;
};
int g_forced_width = 0;

// A k-block takes 345 ns up to 256 tokens, whatever their number (where the GPU is busy for several waves, 385 with 256), in two products
// 95 ns and one more a token each (several waves: 8 % more); beside that the start, and the epilogue of the last tile, or of every tile where nothing hides it.
// (640 tokens, N 7168, K 5120 says 47 us, takes 44; N 27648 134 and 139; N 5120, K 13824 82 and 78; 2,048 tokens, N 1536, K 1536 14.3 and 14.1.)
double plan_us(int M, int N, int K, int width) {
    const int tiles = cdiv(M, width) * cdiv(N, 2 * kRows), waves = cdiv(tiles, li_multiprocessors() / 2), nkb = cdiv(K, BK);
    const double block = width > 256 ? (190.0 + width) * (waves > 2 ? 1.08 : 1.0) : waves <= 2 || width <= 192 ? 345.0 : 345.0 + (width - 192) * 0.65;
    return waves * nkb * block * 1e-3 + 4.5 + (width > 256 ? waves : 1) * width * (0.25 / 32);
}
Plan plan_of(int M, int N, int K) {
    Plan best;
    for (int width = 32; width <= 512 && width - 32 < M; width += 32) {
        const double us = plan_us(M, N, K, width);
        if (best.width == 0 || us < best.us) best = Plan{width, us};
    }
    if (g_forced_width > 0) best = Plan{g_forced_width, 0.0};
    return best;
}

int make_head_map(EncodeTiledFn encode, CUtensorMap* map, const void* base, int heads, int K) {
    const cuuint64_t row = (cuuint64_t)K * 2;
    const cuuint64_t dims[5] = {(cuuint64_t)K, 16, 2, 4, (cuuint64_t)heads}, strides[4] = {row, 64 * row, 16 * row, 128 * row};
    const cuuint32_t box[5] = {(cuuint32_t)BK, 16, 2, 4, 1}, ones[5] = {1, 1, 1, 1, 1};
    const CUresult r = encode(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 5, const_cast<void*>(base), dims, strides, box, ones, CU_TENSOR_MAP_INTERLEAVE_NONE,
                              CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    LI_REQUIRE(r == CUDA_SUCCESS, "linear (tcgen05, tokens as columns): cannot describe %d heads of %d columns (status %d)", heads, K, (int)r);
    return 0;
}

template <typename Tout, int kEpi, bool kWide>
int launch_width(const void* a, const void* w, const float* bias, void* out, int M, int N, int K, int width, cudaStream_t stream, const RopeEpilogue& rope) {
    EncodeTiledFn encode = nullptr;
    int *err_host = nullptr, *err_dev = nullptr;
    if (int rc = setup(&encode, &err_host, &err_dev)) return rc;
    if (*err_host != 0)
        return li_fail("linear (tcgen05, tokens as columns): an earlier launch gave up waiting on a barrier (status %d); the results since then are invalid", *err_host);
    CUtensorMap map_w, map_x, map_x2;
    const int sub = kWide ? cdiv(width, 64) * 32 : width, sub2 = width - sub;
    if (int rc = kEpi == kRope ? make_head_map(encode, &map_w, w, N / kRows, K) : make_map(&map_w, w, N, K, kRows)) return rc;
    if (int rc = make_map(&map_x, a, M, K, sub / 2)) return rc;
    if (int rc = make_map(&map_x2, a, M, K, kWide ? sub2 / 2 : sub / 2)) return rc;
    const size_t smem = kRingBytes + 1024;
    static LiOncePerDevice raised;
    cudaError_t e = li_raise_shared(raised, (const void*)gemm_tcgen05_tokens_kernel<Tout, kEpi, kWide>, smem);
    if (e != cudaSuccess) return li_fail("linear (tcgen05, tokens as columns): cannot raise shared memory to %zu: %s", smem, cudaGetErrorString(e));
    const long long total = (long long)cdiv(M, width) * cdiv(N, 2 * kRows);
    LI_REQUIRE(total < (1 << 30), "linear (tcgen05, tokens as columns): M=%d, N=%d are too large for one launch", M, N);
    int pairs = li_multiprocessors() / 2;
    if (pairs > total) pairs = (int)total;
    li_launch_pdl(gemm_tcgen05_tokens_kernel<Tout, kEpi, kWide>, dim3(2 * pairs), dim3(kThreads), smem, stream, dim3(2, 1, 1), map_w, map_x, map_x2, bias,
                  (Tout*)out, M, N, K, sub, sub2, err_dev, rope);
    return li_check_launch("linear (tcgen05, tokens as columns)");
}

template <typename Tout, int kEpi>
int launch(const void* a, const void* w, const float* bias, void* out, int M, int N, int K, cudaStream_t stream, const RopeEpilogue& rope = RopeEpilogue{}) {
    const int width = plan_of(M, N, K).width;
    return width > 256 ? launch_width<Tout, kEpi, true>(a, w, bias, out, M, N, K, width, stream, rope)
                       : launch_width<Tout, kEpi, false>(a, w, bias, out, M, N, K, width, stream, rope);
}

}  // namespace columns
}  // namespace

// 0: the width of a tile of tokens by shape; else this many (32 to 512 in steps of 32).  For tests and measurements.
LI_EXPORT int li_tcgen05_tokens_force_width(int width) {
    LI_REQUIRE(width >= 0 && width <= 512 && width % 32 == 0, "linear (tcgen05, tokens as columns): no tiles of %d tokens", width);
    columns::g_forced_width = width;
    return 0;
}

// Whether a product has its tokens as columns, rather than in pairs of CTAs on 256 tokens by 256 (where N is a multiple of 192, by 192)
// rows of w, whose tiles take 388 (361) ns a k-block in whole waves, and seven microseconds beside that (four on the persistent
// kernel).  Fewer tiles than half a wave are split along k there.  Measured, those / tokens as columns (us): 640 tokens N 7168, K 5120
// 67.2 / 44.2, N 27648 150 / 139, N 5120 35.7 / 32.5; 320 tokens N 37888, K 3584 92 / 72; 1,536 tokens N 3584, K 18944 198 / 152;
// 2,048 tokens N 7168, K 5120 118 / 103; but N 17920, K 1536 79 / 82.  With rotation every tile's epilogue takes 14 us there, here
// all together 12 more (640 tokens, N 7168, K 5120 80 / 62; 2,048 tokens, N 2048, K 1536 20.9 / 25).
bool li_tcgen05_tokens_wanted(int M, int N, int K, bool rope) {
    const int pairs = li_multiprocessors() / 2, rows = cdiv(M, 256), nkb = cdiv(K, BK);
    if (M <= (nkb < 48 ? 256 : 128) || 2 * rows * cdiv(N, 256) < pairs) return false;      // (a short k and one tile of tokens: nothing to gain)
    const double us = columns::plan_of(M, N, K).us;
    const int waves = cdiv(rows * cdiv(N, 256), pairs);
    double other = waves * nkb * 0.388;
    if (rope) return us + 12.0 < 0.95 * (other + waves * 14.0);
    if (N % 192 == 0) other = std::min(other, cdiv(rows * cdiv(N, 192), pairs) * nkb * 0.361);
    return us < 0.95 * (other + (li_tcgen05_persistent_wanted(M, N, K) ? 4.0 : 7.0));
}

// The same, for tests of the rule.
LI_EXPORT int li_tcgen05_takes_tokens(int M, int N, int K) { return li_tcgen05_tokens_wanted(M, N, K, false) ? 1 : 0; }

int li_linear_tcgen05_tokens(const void* a, const void* w, const float* bias, void* out, int dtype_out, int M, int N, int K, int epilogue, cudaStream_t stream) {
    if (li_epilogue_is_gated(epilogue)) {
        LI_REQUIRE(N % 16 == 0 && li_epilogue_bias_ok(epilogue, bias) && dtype_out == LI_BF16 && ((uintptr_t)out & 3) == 0,
                   "linear (tcgen05, tokens as columns): the swiglu epilogue needs N a multiple of 16, no bias and bfloat16 output");
        return epilogue == LI_EPILOGUE_GLU_CLAMPED ? columns::launch<bf16, 2>(a, w, bias, out, M, N, K, stream)
               : epilogue == LI_EPILOGUE_GEGLU     ? columns::launch<bf16, 3>(a, w, bias, out, M, N, K, stream)
                                                   : columns::launch<bf16, 1>(a, w, bias, out, M, N, K, stream);
    }
    if (dtype_out == LI_BF16) return columns::launch<bf16, 0>(a, w, bias, out, M, N, K, stream);
    if (dtype_out == LI_F32) return columns::launch<float, 0>(a, w, bias, out, M, N, K, stream);
    return li_fail("linear (tcgen05, tokens as columns): unsupported output dtype %d", dtype_out);
}

int li_linear_tcgen05_tokens_rope(const void* a, const void* w, const float* bias, void* out, int M, int N, int K, const RopeEpilogue& rope, cudaStream_t stream) {
    return columns::launch<bf16, columns::kRope>(a, w, bias, out, M, N, K, stream, rope);
}

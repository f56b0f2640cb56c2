// The routed experts' two products on the 5th-generation tensor cores, bfloat16, over lists of (row, choice) pairs that
// are padded to tiles of 128 for every expert (moe.cu, align).
//
//   gather    the listed rows, one after another (a tile's operand is then a box that TMA can fetch).  Tiles are padded, rows are not: a
//             box goes on into the next expert's rows, and what comes of those is not stored, so the rows take as much memory as
//             there are pairs, however many experts share them
//   up        per tile and 256 rows of the expert's W (128 gate rows and their 128 up rows where the activation has a gate): tcgen05.mma
//             M = 128, N = 256, the activation in the epilogue, rows of bfloat16 in the same order
//   down      the same product over the inner numbers, times the pair's weight, to the pair's row of a 32-bit buffer
//
// A persistent kernel, one CTA per SM: a TMA warp, a warp that issues the products, eight epilogue warps (two for every
// quarter of the tensor-memory lanes, each half of the columns), a ring of four stages of 64 k, two accumulators so that a
// tile's epilogue runs under the next tile's products.  The tiles of one slice of W follow one another, so an expert's
// slice comes from memory once.  With few pairs the experts' weights' way from memory bounds it, with many the products
// themselves and the last wave of tiles.
//
// Measured (B200, 16 experts of 2,048 x 2,304 with relu^2, the best two of each of 2,048 rows): up 242 -> 58 us, down
// 238 -> 64 against tiles of 64 x 64 on mma.sync (37 GFLOP each: 0.65 PFLOP/s with the padded rows' share), the gather 6; a prompt of 2,048
// tokens of Nuvivik 3.95 -> 2.57 ms.  Few pairs, bound by the weights: 17 sequences' decode step 1.09 -> 0.97 ms, 64 sequences' 1.44
// -> 1.33, a prompt of 33 tokens 0.98 -> 0.86.
#include "common.cuh"
#include "expert_act.cuh"
#include "mma_utils.cuh"
#include "tcgen05_one.cuh"

namespace hos {

constexpr int XM = 128, XN = 256, XK = 64;              // rows of a tile, rows of W, numbers of k in a stage
constexpr int kXThreads = 320, kXStages = 4;
constexpr int kXABytes = XM * XK * 2, kXBBytes = XN * XK * 2, kXStageBytes = kXABytes + kXBBytes;
constexpr int kXSmem = kXStages * kXStageBytes + 256 + 1024;
constexpr long long kXWaitCycles = 1ll << 31;

enum GroupedStep : int { kGroupedUp = 0, kGroupedGatedUp = 1, kGroupedDown = 2 };

__device__ int g_moe_grouped_error = 0;
__device__ int* g_moe_grouped_error_host = nullptr;     // a word in pinned host memory, if the host gave one

__device__ __forceinline__ void grouped_give_up() {
    atomicExch(&g_moe_grouped_error, 1);
    int* w = g_moe_grouped_error_host;
    if (w != nullptr) {
        atomicExch_system(w, kGiveUpMoeGrouped);
        __threadfence_system();
    }
}

// A warp per list place.
__global__ void __launch_bounds__(256)
moe_gather_kernel(const bf16* __restrict__ h, const int* __restrict__ listed, const int* __restrict__ tile_expert,
                  const int* __restrict__ tile_row, bf16* __restrict__ rows, int D, int top) {
    pdl_enter();
    const int place = blockIdx.x * 8 + (threadIdx.x >> 5);
    if (tile_expert[place / XM] < 0) return;
    const int id = listed[place];
    if (id < 0) return;
    const uint4* from = reinterpret_cast<const uint4*>(h + (size_t)(id / top) * D);
    const int tile = place / XM;
    uint4* to = reinterpret_cast<uint4*>(rows + ((size_t)(tile_row != nullptr ? tile_row[tile] : tile * XM) + place % XM) * D);
#pragma unroll 4
    for (int i = threadIdx.x & 31; i < D / 8; i += 32) to[i] = from[i];
}

struct GroupedArgs {
    const int* listed;
    const int* tile_expert;
    const int* tile_row;        // where a tile's rows begin (null: at 128 times its number)
    const float* weight;        // by pair: on the expert's input (up) or its output (down), or null
    void* out;
    int max_tiles, N, K;        // N: numbers of an output row
    float limit, alpha, up_shift;
    long long wait_cycles;      // the limit of every wait
    int stop_tile;              // for tests of the give-up path: the CTA's tile at which an epilogue warp takes its wait as run out (-1: none)
};

template <int STEP>
__global__ void __launch_bounds__(kXThreads, 1)
moe_grouped_kernel(const __grid_constant__ CUtensorMap map_a,      // list places, boxes of [128 rows x 64]
                   const __grid_constant__ CUtensorMap map_w,      // all experts' rows, boxes of [128 rows x 64]
                   GroupedArgs p) {
    constexpr bool GATED = STEP == kGroupedGatedUp;
    constexpr int COLS = GATED ? XN / 2 : XN;           // output numbers of a tile
    extern __shared__ unsigned char smem_unaligned[];
    unsigned char* stages = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_unaligned) + 1023) & ~(uintptr_t)1023);
    uint64_t* bars = reinterpret_cast<uint64_t*>(stages + kXStages * kXStageBytes);
    uint64_t* full = bars;                      // [kXStages] TMA -> products
    uint64_t* empty = full + kXStages;          // [kXStages] products -> TMA
    uint64_t* acc_full = empty + kXStages;      // [2] products -> epilogue
    uint64_t* acc_empty = acc_full + 2;         // [2] epilogue -> products
    uint32_t* tmem_base_smem = reinterpret_cast<uint32_t*>(acc_empty + 2);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        for (int s = 0; s < kXStages; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); }
        for (int a = 0; a < 2; ++a) { mbar_init(&acc_full[a], 1); mbar_init(&acc_empty[a], 8); }
        mbar_fence_init();
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_base_smem)), "r"(2 * XN) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    const uint32_t tmem_base = *tmem_base_smem;
    pdl_enter();
    int used = 0;                               // the real tiles stand first
    for (int t0 = 0; t0 < p.max_tiles; t0 += kXThreads) {
        const int t = t0 + threadIdx.x;
        used += __syncthreads_count(t < p.max_tiles && p.tile_expert[t] >= 0);
    }
    const int n_tiles = (p.N + COLS - 1) / COLS, total = used * n_tiles, k_blocks = (p.K + XK - 1) / XK;
    const int rows_per_expert = (GATED ? 2 : 1) * p.N;
    auto first_row = [&](int mt) { return p.tile_row != nullptr ? p.tile_row[mt] : mt * XM; };
    bool ok = true;                             // false: a wait of this thread (in the epilogue: of its warp) ran out
    auto wait = [&](uint64_t* bar, uint32_t parity) { return mbar_wait_cycles(bar, parity, p.wait_cycles); };

    if (warp == 0) {
        if (lane == 0) {
            int it = 0;
            for (int tile = blockIdx.x; tile < total && ok; tile += gridDim.x) {
                const int mt = tile % used, n0 = tile / used * COLS, row0 = first_row(mt);
                const int w0 = p.tile_expert[mt] * rows_per_expert + n0, w1 = w0 + (GATED ? p.N : XN / 2);
                for (int kb = 0; kb < k_blocks; ++kb, ++it) {
                    const int s = it % kXStages;
                    if (it >= kXStages && !wait(&empty[s], ((it / kXStages) - 1) & 1)) { ok = false; break; }
                    unsigned char* a_dst = stages + s * kXStageBytes;
                    mbar_expect_tx(&full[s], kXStageBytes);
                    tc_tma_2d(a_dst, &map_a, kb * XK, row0, &full[s]);
                    tc_tma_2d(a_dst + kXABytes, &map_w, kb * XK, w0, &full[s]);
                    tc_tma_2d(a_dst + kXABytes + kXBBytes / 2, &map_w, kb * XK, w1, &full[s]);
                }
            }
            if (!ok) grouped_give_up();
        }
        __syncwarp();
    } else if (warp == 1) {
        if (lane == 0) {
            constexpr uint32_t idesc = tc_idesc(XM, XN, 0);
            int it = 0, local = 0;
            for (int tile = blockIdx.x; tile < total && ok; tile += gridDim.x, ++local) {
                const int acc = local & 1;
                if (local >= 2 && !wait(&acc_empty[acc], ((local >> 1) - 1) & 1)) { ok = false; break; }
                tc_fence_after_sync();
                for (int kb = 0; kb < k_blocks; ++kb, ++it) {
                    const int s = it % kXStages;
                    if (!wait(&full[s], (it / kXStages) & 1)) { ok = false; break; }
                    tc_fence_after_sync();
                    const uint32_t a_addr = smem_u32(stages + s * kXStageBytes);
                    const uint64_t a_desc = desc_kmajor(a_addr), b_desc = desc_kmajor(a_addr + kXABytes);
#pragma unroll
                    for (int k = 0; k < XK / 16; ++k)
                        tc_mma(tmem_base + acc * XN, a_desc + 2 * k, b_desc + 2 * k, idesc, (kb > 0 || k > 0) ? 1u : 0u);
                    tc_commit(&empty[s]);
                }
                if (ok) tc_commit(&acc_full[acc]);
            }
            if (!ok) grouped_give_up();
        }
        __syncwarp();
    } else {
        const int quarter = warp & 3, half = (warp - 2) >> 2, r = quarter * 32 + lane;
        int local = 0;
        for (int tile = blockIdx.x; tile < total; tile += gridDim.x, ++local) {
            const int mt = tile % used, n_first = tile / used * COLS;
            const int id = p.listed[mt * XM + r];
            const size_t row = STEP == kGroupedDown ? (size_t)max(id, 0) : (size_t)first_row(mt) + r;      // of the output
            const float wt = id >= 0 && p.weight != nullptr ? p.weight[id] : 1.f;
            const int acc = local & 1;
            ok = __all_sync(0xffffffffu, wait(&acc_full[acc], (local >> 1) & 1)) && !(local == p.stop_tile && warp == 2);
            if (!ok) break;
            tc_fence_after_sync();
            const uint32_t t_lane = tmem_base + ((uint32_t)(quarter * 32) << 16) + acc * XN;
#pragma unroll 1
            for (int c0 = half * (COLS / 2); c0 < (half + 1) * (COLS / 2); c0 += 32) {
                if (n_first + c0 >= p.N) break;
                uint32_t v[32], u[32];
                tc_ld32(t_lane + c0, v);
                if (GATED) tc_ld32(t_lane + XN / 2 + c0, u);
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                if (id >= 0) {
                    const int n0 = n_first + c0, left = p.N - n0;                // N is a multiple of 8
                    if (STEP == kGroupedDown) {
                        float4* dst = reinterpret_cast<float4*>((float*)p.out + row * p.N + n0);
#pragma unroll
                        for (int q = 0; q < 8; ++q)
                            if (4 * q < left)
                                dst[q] = make_float4(__uint_as_float(v[4 * q]) * wt, __uint_as_float(v[4 * q + 1]) * wt,
                                                     __uint_as_float(v[4 * q + 2]) * wt, __uint_as_float(v[4 * q + 3]) * wt);
                    } else {
                        constexpr int ACT = GATED ? kGatedSwish : kReluSquare;
                        uint4* dst = reinterpret_cast<uint4*>((bf16*)p.out + row * p.N + n0);
#pragma unroll
                        for (int q = 0; q < 4; ++q) {
                            uint32_t w[4];
#pragma unroll
                            for (int i = 0; i < 4; ++i) {
                                float y[2];
#pragma unroll
                                for (int e = 0; e < 2; ++e) {
                                    const int j = 8 * q + 2 * i + e;
                                    y[e] = expert_act<ACT>(__uint_as_float(v[j]) * wt, __uint_as_float(GATED ? u[j] : v[j]) * wt, p.limit,
                                                           p.alpha, p.up_shift);
                                }
                                w[i] = pack_bf16(y[0], y[1]);
                            }
                            if (8 * q < left) dst[q] = make_uint4(w[0], w[1], w[2], w[3]);
                        }
                    }
                }
                __syncwarp();
            }
            tc_fence_before_sync();
            __syncwarp();
            if (lane == 0) mbar_arrive(&acc_empty[acc]);
        }
        if (!ok && lane == 0) grouped_give_up();
    }
    tc_fence_before_sync();
    if (__syncthreads_or(!ok)) let_work_under_way_end();
    if (warp == 1)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(2 * XN) : "memory");
}

template <int STEP>
int launch_grouped(const void* rows, long long n_rows, const void* W, long long w_rows, const GroupedArgs& p, cudaStream_t stream) {
    CUtensorMap ma, mw;
    int rc;
    if ((rc = tc_make_map(&ma, rows, n_rows, p.K, p.K, XM))) return rc;
    if ((rc = tc_make_map(&mw, W, w_rows, p.K, p.K, XN / 2))) return rc;
    if (cudaFuncSetAttribute(moe_grouped_kernel<STEP>, cudaFuncAttributeMaxDynamicSharedMemorySize, kXSmem) != cudaSuccess)
        HOS_REFUSE("moe_grouped: cannot get %d bytes of shared memory", kXSmem);
    constexpr int COLS = STEP == kGroupedGatedUp ? XN / 2 : XN;
    const long long tiles = (long long)p.max_tiles * ((p.N + COLS - 1) / COLS);
    launch_pdl(moe_grouped_kernel<STEP>, dim3((unsigned)(tiles < sm_count_cached() ? tiles : sm_count_cached())), dim3(kXThreads), kXSmem, stream,
               ma, mw, p);
    return check_launch("moe_grouped");
}

}  // namespace hos

using namespace hos;

extern "C" int hos_moe_grouped_set_error_word(int* word) {
    if (cudaMemcpyToSymbol(g_moe_grouped_error_host, &word, sizeof(word)) != cudaSuccess)
        HOS_REFUSE("moe_grouped: cannot set the error word: %s", cudaGetErrorString(cudaGetLastError()));
    return 0;
}

// Both products of `max_tiles` listed tiles of 128.  rows [n_rows][D] and y [n_rows][F] bfloat16 are scratch: tile t's rows begin at
// tile_row[t] (null: at 128 t), so n_rows is the number of pairs (or 128 max_tiles).  pair_out [pairs][D] 32-bit by pair id.
// W_up: [experts][2F or F][D], W_down: [experts][D][F].  in_weight or out_weight (by pair, or null).  wait_cycles, stop_tile:
// for tests of what happens when a wait runs out (GroupedArgs); 0 and -1 otherwise.
extern "C" int hos_moe_grouped(const void* h, const void* W_up, const void* W_down, const int* listed, const int* tile_expert,
                               const int* tile_row, void* rows, void* y, float* pair_out, int n_rows, int max_tiles, int n_experts,
                               int D, int F, int top, float limit, float alpha, float up_shift, const float* in_weight, const float* out_weight, int act, long long wait_cycles, int stop_tile,
                               cudaStream_t stream) {
    if (max_tiles <= 0) return 0;
    if (n_rows <= 0 || (tile_row == nullptr && n_rows < (long long)max_tiles * XM))
        HOS_REFUSE("moe_grouped: %d rows do not hold %d tiles", n_rows, max_tiles);
    if (D <= 0 || F <= 0 || D % 8 || F % 8 || top <= 0 || n_experts <= 0 ||
        (((uintptr_t)h | (uintptr_t)W_up | (uintptr_t)W_down | (uintptr_t)rows | (uintptr_t)y | (uintptr_t)pair_out) & 15))
        HOS_REFUSE("moe_grouped: rows of %d and %d numbers must be multiples of 8, and the operands 16-byte aligned", D, F);
    const long long wide = D > F ? D : F;
    if (2 * wide * n_experts + XN > (1ll << 31) - 1 || max_tiles * (wide / 128 + 1) > (1ll << 30) || (long long)max_tiles * XM > (1ll << 30))
        HOS_REFUSE("moe_grouped: %d experts and %d tiles are more than one launch takes", n_experts, max_tiles);
    launch_pdl(moe_gather_kernel, dim3((unsigned)max_tiles * (XM / 8)), dim3(256), 0, stream, (const bf16*)h, listed, tile_expert, tile_row, (bf16*)rows,
               D, top);
    int rc = check_launch("moe_grouped (gather)");
    if (rc) return rc;
    if (wait_cycles <= 0) wait_cycles = kXWaitCycles;
    GroupedArgs up = {listed, tile_expert, tile_row, in_weight, y, max_tiles, F, D, limit, alpha, up_shift, wait_cycles, stop_tile};
    if (act == kGatedSwish) rc = launch_grouped<kGroupedGatedUp>(rows, n_rows, W_up, 2ll * n_experts * F, up, stream);
    else if (act == kReluSquare) rc = launch_grouped<kGroupedUp>(rows, n_rows, W_up, (long long)n_experts * F, up, stream);
    else HOS_REFUSE("moe_grouped: unknown activation %d", act);
    if (rc) return rc;
    GroupedArgs down = {listed, tile_expert, tile_row, out_weight, pair_out, max_tiles, D, F, 0.f, 0.f, 0.f, wait_cycles, stop_tile};
    return launch_grouped<kGroupedDown>(y, n_rows, W_down, (long long)n_experts * D, down, stream);
}

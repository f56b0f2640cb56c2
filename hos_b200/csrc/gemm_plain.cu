// Plain matrix product on the CUDA cores: out[m, n] = sum_k A[m, k] * W[n, k], with
// 32-bit FMA accumulation whatever the storage types are.  It is the 32-bit path's
// product where rows are not whole 16-byte pieces (elsewhere gemm_f32_kernel is; no tensor-core
// mode of reduced precision exists in that path), the reference that the tensor-core
// product is checked against, and the product for sizes the tensor-core kernel refuses.
// Any M, N, K.
//
// Epilogues: none; soft-cap (logits); gated (W holds gate rows then up rows,
// out = act(gate) * up), so that the 2F-wide intermediate is never written; bias (out = act(x + bias[n]), or
// act(x) without a bias, act none, the erf-form or the tanh-form GELU).
#include "common.cuh"

namespace hos {

constexpr int BM = 64, BN = 64, BK = 16;

enum Epilogue : int { kEpiNone = 0, kEpiSoftcap = 1, kEpiGated = 2, kEpiBias = 3 };

// What the epilogues make of a sum (and, gated, of the up row's).
template <int EPI>
__device__ __forceinline__ float plain_epilogue(float v, float up, const float* bias, int n, float cap, int act) {
    if (EPI == kEpiSoftcap) v = softcap_precise(v, cap);
    if (EPI == kEpiBias) {
        if (bias != nullptr) v += bias[n];
        if (act == 1) v = gelu_erf(v);
        else if (act == 2) v = gelu_tanh(v);
    }
    if (EPI == kEpiGated) {
        if (act == 2) return clamped_swish(v, up, cap);              // the clamp's limit rides in `cap`
        v = (act == 0 ? gelu_tanh(v) : v / (1.f + expf(-v))) * up;
    }
    return v;
}

template <typename TA, typename TW, typename TO, int EPI>
__global__ void __launch_bounds__(256)
gemm_plain_kernel(const TA* __restrict__ A, const TW* __restrict__ W, TO* __restrict__ out,
                  int M, int N, int K, int lda, int ldw, int ldo, float cap, int act, int gate_rows,
                  const float* __restrict__ bias) {
    __shared__ float As[BK][BM + 4];
    __shared__ float Ws[BK][BN + 4];
    __shared__ float Us[EPI == kEpiGated ? BK : 1][BN + 4];
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
    const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
    float acc[4][4] = {};
    float acc_u[EPI == kEpiGated ? 4 : 1][4] = {};
    for (int k0 = 0; k0 < K; k0 += BK) {
        // 64 rows x 16 k per operand: 1024 elements, 4 per thread
        for (int e = threadIdx.x; e < BM * BK; e += 256) {
            const int r = e >> 4, kk = e & 15;
            const int m = m0 + r, k = k0 + kk;
            As[kk][r] = (m < M && k < K) ? to_float(A[(size_t)m * lda + k]) : 0.f;
            const int n = n0 + r;
            Ws[kk][r] = (n < N && k < K) ? to_float(W[(size_t)n * ldw + k]) : 0.f;
            if (EPI == kEpiGated)
                Us[kk][r] = (n < N && k < K) ? to_float(W[(size_t)(gate_rows + n) * ldw + k]) : 0.f;
        }
        __syncthreads();
#pragma unroll
        for (int kk = 0; kk < BK; ++kk) {
            float a[4], w[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) a[i] = As[kk][ty * 4 + i];
#pragma unroll
            for (int j = 0; j < 4; ++j) w[j] = Ws[kk][tx * 4 + j];
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(a[i], w[j], acc[i][j]);
            if (EPI == kEpiGated) {
                float u[4];
#pragma unroll
                for (int j = 0; j < 4; ++j) u[j] = Us[kk][tx * 4 + j];
#pragma unroll
                for (int i = 0; i < 4; ++i)
#pragma unroll
                    for (int j = 0; j < 4; ++j) acc_u[i][j] = fmaf(a[i], u[j], acc_u[i][j]);
            }
        }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int m = m0 + ty * 4 + i;
        if (m >= M) continue;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int n = n0 + tx * 4 + j;
            if (n >= N) continue;
            const float v = plain_epilogue<EPI>(acc[i][j], EPI == kEpiGated ? acc_u[i][j] : 0.f, bias, n, cap, act);
            out[(size_t)m * ldo + n] = from_float<TO>(v);
        }
    }
}

template <typename TA, typename TW, typename TO>
static int launch_plain(const void* A, const void* W, void* out, int M, int N, int K, int lda,
                        int ldw, int ldo, int epi, float cap, int act, const float* bias, cudaStream_t stream) {
    dim3 grid((N + BN - 1) / BN, (M + BM - 1) / BM);
    if (grid.y > 65535) HOS_REFUSE("gemm_plain: %d rows are more than one launch takes", M);
    switch (epi) {
    case kEpiNone:
        gemm_plain_kernel<TA, TW, TO, kEpiNone><<<grid, 256, 0, stream>>>(
            (const TA*)A, (const TW*)W, (TO*)out, M, N, K, lda, ldw, ldo, cap, act, 0, bias);
        break;
    case kEpiSoftcap:
        gemm_plain_kernel<TA, TW, TO, kEpiSoftcap><<<grid, 256, 0, stream>>>(
            (const TA*)A, (const TW*)W, (TO*)out, M, N, K, lda, ldw, ldo, cap, act, 0, bias);
        break;
    case kEpiGated:
        gemm_plain_kernel<TA, TW, TO, kEpiGated><<<grid, 256, 0, stream>>>(
            (const TA*)A, (const TW*)W, (TO*)out, M, N, K, lda, ldw, ldo, cap, act, N, bias);
        break;
    case kEpiBias:
        gemm_plain_kernel<TA, TW, TO, kEpiBias><<<grid, 256, 0, stream>>>(
            (const TA*)A, (const TW*)W, (TO*)out, M, N, K, lda, ldw, ldo, cap, act, 0, bias);
        break;
    default:
        HOS_REFUSE("gemm_plain: unknown epilogue %d", epi);
    }
    return check_launch("gemm_plain");
}

// ---- 32-bit rows of whole 16-byte pieces ---------------------------------------------------------------------------
// What bounds it: at Gemma-2 2B's sizes one row costs 2.0 GFMA and a step reads 10.4 GB of weights, so up to about 30 rows
// the weights' way from memory bounds a step and above that the FMA lanes do.  A CTA of four warps takes BM rows x 64 rows
// of W; both operands lie in shared memory as they lie in global memory (k runs along a row, 32 k of a row are 128
// bytes whose 16-byte pieces are permuted by the row number, so that the reads of a warp hit every bank once), brought in
// by cp.async through a ring of stages.  A thread's accumulators are pairs, the even and the odd k of a sum: then one
// fma.rn.f32x2 takes two neighbours of a row of A and two of a row of W as they were read, and nothing is transposed
// or duplicated.  What a thread reads from shared memory costs as much time as what it multiplies at 8 x 8 sums a thread,
// and more with fewer sums, so the four warps split a stage's k instead of the tile: with tiles of 16 rows a thread still
// holds 8 x 4 sums, with tiles of 32 rows 8 x 8.  Where few rows leave too few tiles for the GPU's SMs, the CTAs of a cluster
// share one tile by k and add their sums through distributed shared memory, each a slice of the rows, in the order of the
// ranks; where there are tiles enough, one CTA walks over the same parts of k and adds their sums in the same order (f32_walks).
// In what order a sum is added up hangs on N and K alone: a row's results are the same bits whatever rows stand
// beside it (padding, another batch), so k is always cut for one tile of rows, and there are no tiles of more rows, whose
// warps would have to share k differently.
// Measured (B200): the gated product of 2 x 9,216 rows of W, K 2,304: 48 us at 16 rows (3.6 TB/s of weights), 79 at 32, 285 at 121, 2,178 at
// 1,000 (39 TFLOP/s); the tiles above take 510, 509, 621 and 3,476.  The logits' error against 64 bits of a float32 prompt went from 9.1e-6 to
// 3.7e-6 (sums of several parts, not a long one).
constexpr int kF32Threads = 128, kF32Cols = 64, kF32Depth = 32;

struct F32Gemm {
    const float* A;
    const float* W;
    float* out;
    const float* bias;
    int M, N, K, lda, ldw, ldo, act, splits;
    float cap;
};

// 16 bytes to shared memory, zeros where `there` is false (`from` is then any readable address).
__device__ __forceinline__ void copy16_or_zero(uint32_t to, const float* from, bool there) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(to), "l"(from), "r"(there ? 16 : 0) : "memory");
}
__device__ __forceinline__ void fma_pair(unsigned long long& acc, unsigned long long a, unsigned long long w) {
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(a), "l"(w));
}
__device__ __forceinline__ float pair_sum(unsigned long long v) {
    return __uint_as_float((uint32_t)v) + __uint_as_float((uint32_t)(v >> 32));
}

// A tile of BM rows: how a warp's lanes share it.
template <int BM>
struct F32Tile {
    static constexpr int WK = kF32Threads / 32;                      // the warps split k
    static constexpr int LC = BM <= 16 ? 16 : 8, LR = 32 / LC;       // lanes along the columns, along the rows
    static constexpr int RM = BM / LR, RN = kF32Cols / LC;         // sums of a thread
    static constexpr int STAGE = (BM + kF32Cols) * kF32Depth;        // numbers of a stage
    static constexpr int STAGES = 6;
    static constexpr int LD = kF32Cols + 1;                          // a row of the sums' tiles, which take the stages' place ...
    static constexpr int SMEM = STAGES * STAGE * 4;
    static constexpr int WALK_SMEM = SMEM + WK * BM * LD * 4;        // ... but for a CTA that goes on after adding them up
    static_assert(WK * BM * LD <= STAGES * STAGE && RM * LR == BM && RM <= 8, "tile");
};

template <int BM, int EPI, bool WALK>
__global__ void __launch_bounds__(kF32Threads, BM <= 16 ? 3 : 2) gemm_f32_kernel(F32Gemm p) {
    using T = F32Tile<BM>;
    constexpr int STAGE = T::STAGE, STAGES = T::STAGES, RM = T::RM, RN = T::RN, LD = T::LD;
    extern __shared__ __align__(128) float smem[];
    const int lane = threadIdx.x & 31, kg = threadIdx.x >> 5;
    const int tx = lane % T::LC, ty = lane / T::LC;                  // columns tx + LC j, rows ty + LR i
    constexpr int COLS = EPI == kEpiGated ? kF32Cols / 2 : kF32Cols;
    const int rank = !WALK && p.splits > 1 ? blockIdx.x % p.splits : 0;          // a cluster is `splits` CTAs along x
    const int tile = WALK ? blockIdx.x : blockIdx.x / p.splits, mt = (p.M + BM - 1) / BM;            // tiles of rows side by side: they share W in L2
    const int n0 = tile / mt * COLS, m0 = tile % mt * BM;
    const int blocks = (p.K + kF32Depth - 1) / kF32Depth;
    auto part_begin = [&](int part) { return (int)((long long)blocks * part / p.splits); };
    const int first = WALK ? 0 : part_begin(rank), last = WALK ? blocks : part_begin(rank + 1);

    // This thread's pieces of a stage: 8 pieces a row, so 16 rows a round of the block; piece and row parity are fixed.
    const int piece = threadIdx.x & 7, row0 = threadIdx.x >> 3;
    const uint32_t base = (uint32_t)__cvta_generic_to_shared(smem);
    const uint32_t to0 = base + (row0 * kF32Depth + ((piece ^ (row0 & 7)) << 2)) * 4;    // 16 rows on: the same place
    auto load = [&](int stage, int block) {
        const int k = block * kF32Depth + piece * 4;
        const bool inside = k < p.K;                                 // K is a multiple of 4: a piece is whole or absent
        const uint32_t to = to0 + stage * STAGE * 4;
#pragma unroll
        for (int i = 0; i < BM / 16; ++i) {
            const int m = m0 + row0 + 16 * i;
            const bool there = inside && m < p.M;
            copy16_or_zero(to + 16 * i * kF32Depth * 4, there ? p.A + (size_t)m * p.lda + k : p.A, there);
        }
#pragma unroll
        for (int i = 0; i < kF32Cols / 16; ++i) {
            const int r = row0 + 16 * i;
            int n = n0 + r;
            bool there = inside && n < p.N;
            if (EPI == kEpiGated) {                                  // 32 gate rows, then their 32 up rows
                n = n0 + (r & 31);
                there = inside && n < p.N;
                if (r >= 32) n += p.N;
            }
            copy16_or_zero(to + (BM + 16 * i) * kF32Depth * 4, there ? p.W + (size_t)n * p.ldw + k : p.W, there);
        }
    };

    unsigned long long acc[RM][RN] = {};
#pragma unroll
    for (int s = 0; s < STAGES - 1; ++s) {
        if (first + s < last) load(s, first + s);
        asm volatile("cp.async.commit_group;" ::: "memory");
    }
    float* sums = WALK ? smem + STAGES * STAGE : smem;               // a tile for each warp along k
    auto keep_sums = [&] {
#pragma unroll
        for (int i = 0; i < RM; ++i)
#pragma unroll
            for (int j = 0; j < RN; ++j) sums[(kg * BM + ty + T::LR * i) * LD + tx + T::LC * j] = pair_sum(acc[i][j]);
    };
    constexpr int OUTS = WALK ? BM * COLS / kF32Threads : 1;         // results of a thread
    float v_out[OUTS] = {}, up_out[OUTS] = {};
    int stage = 0, part = 0;
    for (int block = first; block < last; ++block) {
        asm volatile("cp.async.wait_group %0;" ::"n"(STAGES - 2) : "memory");
        __syncthreads();                                             // this stage is there, and the one before it is read
        const int ahead = block + STAGES - 1;
        if (ahead < last) load(stage == 0 ? STAGES - 1 : stage - 1, ahead);
        asm volatile("cp.async.commit_group;" ::: "memory");
        const float* a_at = smem + stage * STAGE + ty * kF32Depth;
        const float* w_at = smem + stage * STAGE + (BM + tx) * kF32Depth;
#pragma unroll 2
        for (int u = 0; u < kF32Depth / 4 / T::WK; ++u) {
            const int c = u * T::WK + kg;
            ulonglong2 a[RM];
#pragma unroll
            for (int i = 0; i < RM; ++i)
                a[i] = *reinterpret_cast<const ulonglong2*>(a_at + T::LR * i * kF32Depth +
                                                            ((c ^ ((ty + T::LR * i) & 7)) << 2));
#pragma unroll
            for (int j = 0; j < RN; ++j) {
                const ulonglong2 w = *reinterpret_cast<const ulonglong2*>(w_at + T::LC * j * kF32Depth + ((c ^ (tx & 7)) << 2));
#pragma unroll
                for (int i = 0; i < RM; ++i) {
                    fma_pair(acc[i][j], a[i].x, w.x);
                    fma_pair(acc[i][j], a[i].y, w.y);
                }
            }
        }
        stage = stage == STAGES - 1 ? 0 : stage + 1;
        if (WALK && block + 1 == part_begin(part + 1)) {             // the end of a part: its sums join the results
            keep_sums();
            __syncthreads();                                         // they are read before the next block's barrier
#pragma unroll
            for (int o = 0; o < OUTS; ++o) {
                const int e = threadIdx.x + o * kF32Threads, at = e / COLS * LD + e % COLS;
#pragma unroll
                for (int g = 0; g < T::WK; ++g) {
                    v_out[o] += sums[g * BM * LD + at];
                    if (EPI == kEpiGated) up_out[o] += sums[g * BM * LD + at + 32];
                }
            }
#pragma unroll
            for (int i = 0; i < RM; ++i)
#pragma unroll
                for (int j = 0; j < RN; ++j) acc[i][j] = 0;
            ++part;
        }
    }
    if constexpr (WALK) {
#pragma unroll
        for (int o = 0; o < OUTS; ++o) {
            const int e = threadIdx.x + o * kF32Threads, m = m0 + e / COLS, n = n0 + e % COLS;
            if (m < p.M && n < p.N) p.out[(size_t)m * p.ldo + n] = plain_epilogue<EPI>(v_out[o], up_out[o], p.bias, n, p.cap, p.act);
        }
        return;
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();

    // The sums to shared memory, the cluster's added, the rows' slices stored.
    keep_sums();
    if (p.splits > 1) {
        asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
        asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    } else {
        __syncthreads();
    }
    const int rows = (min(BM, p.M - m0) + p.splits - 1) / p.splits, lo = rank * rows;
    for (int e = threadIdx.x; e < rows * COLS; e += kF32Threads) {
        const int r = lo + e / COLS, c = e % COLS;
        if (r >= BM || m0 + r >= p.M || n0 + c >= p.N) continue;
        float v = 0.f, up = 0.f;
        for (int s = 0; s < p.splits; ++s) {
            uint32_t at = base + (r * LD + c) * 4;
            if (p.splits > 1) asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(at) : "r"(at), "r"(s));
#pragma unroll
            for (int g = 0; g < T::WK; ++g) {                        // an address of this CTA's own is one of the cluster's too
                float x;
                asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(x) : "r"(at + g * BM * LD * 4) : "memory");
                v += x;
                if (EPI == kEpiGated) {
                    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(x) : "r"(at + (g * BM * LD + 32) * 4) : "memory");
                    up += x;
                }
            }
        }
        p.out[(size_t)(m0 + r) * p.ldo + n0 + c] = plain_epilogue<EPI>(v, up, p.bias, n0 + c, p.cap, p.act);
    }
    if (p.splits > 1) {                                              // no CTA leaves while its sums are being read
        asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
        asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    }
}

template <int BM, int EPI>
cudaLaunchConfig_t f32_config(long long tiles, int splits, cudaLaunchAttribute* attr, cudaStream_t stream) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(tiles * splits));
    cfg.blockDim = kF32Threads;
    cfg.dynamicSmemBytes = F32Tile<BM>::SMEM;
    cfg.stream = stream;
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = splits;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = splits > 1 ? 1 : 0;
    return cfg;
}

constexpr int kF32MaxSplits = 8;

// How many clusters of 1 .. 8 CTAs of this kernel the GPU holds at once (asked once per kernel), or null on an error.
template <int BM, int EPI>
const int* f32_clusters() {
    struct Counts {
        int n[kF32MaxSplits + 1];
        bool ok;
    };
    static const Counts counts = [] {
        Counts c = {};
        c.ok = cudaFuncSetAttribute(gemm_f32_kernel<BM, EPI, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, F32Tile<BM>::SMEM) == cudaSuccess;
        int per_sm = 0;
        c.ok = c.ok && cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, gemm_f32_kernel<BM, EPI, false>, kF32Threads, F32Tile<BM>::SMEM) == cudaSuccess;
        c.n[1] = per_sm * sm_count_cached();
        for (int s = 2; s <= kF32MaxSplits && c.ok; ++s) {
            cudaLaunchAttribute attr[1];
            cudaLaunchConfig_t cfg = f32_config<BM, EPI>(1024, s, attr, 0);
            if (cudaOccupancyMaxActiveClusters(&c.n[s], gemm_f32_kernel<BM, EPI, false>, &cfg) != cudaSuccess) c.n[s] = 0;
        }
        cudaGetLastError();                                          // a size that does not fit is none to choose, not an error
        c.ok = c.ok && c.n[1] > 0;
        return c;
    }();
    return counts.ok ? counts.n : nullptr;
}

// In how many parts k is cut, for one tile of rows (so not by M: see above).  A CTA's time is its blocks of 32 k, plus about four blocks' worth for filling the ring and
// adding up; an SM's time is that of its CTAs together, but a single CTA does not fill it; clusters that do not fit at
// once wait for a whole one.
inline int f32_splits(const int* clusters, int tiles, int K) {
    const int blocks = (K + kF32Depth - 1) / kF32Depth, sms = sm_count_cached();
    int best = 1;
    float best_cost = 0.f;
    for (int s = 1; s <= kF32MaxSplits; ++s) {
        if (s > 1 && blocks < 4 * s) break;
        if (clusters[s] <= 0) continue;
        const int full = tiles / clusters[s], rest = tiles % clusters[s];
        auto per_sm = [&](int n) { return n == 0 ? 0.f : fmaxf(1.5f, (float)((n * s + sms - 1) / sms)); };
        const float cost = (full * per_sm(clusters[s]) + per_sm(rest)) * (float)((blocks + s - 1) / s + 4);
        if (s == 1 || cost < best_cost) best = s, best_cost = cost;
    }
    return best;
}

// Whether one CTA had better walk over a tile's parts of k, one after another, than a cluster share them (the bits are the same).
// A cluster fills and empties its rings for every part, about 5.5 blocks' worth, but gives few tiles to many SMs; a CTA that walks
// fills its ring once, and adding up a part costs it about a block.  A lone CTA takes 0.65 of what two on an SM take.
// Measured, cluster / walk in us, for rows of K 2,304 to 4,096 results: 121 rows 89 / 85, 160 rows 109 / 125, 512 rows 312 / 274, 4,096
// rows 2,397 / 2,092; K 1,024 to 1,024: 64 rows 14 / 30, 160 rows 29 / 30, 300 rows 48 / 46, 2,048 rows 264 / 149 (the tiles above 244);
// K 9,216 to 2,304: 300 rows 433 / 467, 512 rows 683 / 604.
inline bool f32_walks(const int* clusters, long long tiles, int splits, int K) {
    const int blocks = (K + kF32Depth - 1) / kF32Depth, sms = sm_count_cached();
    auto per_sm = [&](long long ctas) { return ctas == 0 ? 0.f : fmaxf(1.3f, (float)((ctas + sms - 1) / sms)); };
    auto rounds = [&](int slots, int ctas) {
        return (float)(tiles / slots) * per_sm((long long)slots * ctas) + per_sm(tiles % slots * ctas);
    };
    return rounds(clusters[1], 1) * (float)(blocks + 4 + splits) < rounds(clusters[splits], splits) * ((float)blocks / splits + 5.5f);
}

template <int EPI>
bool f32_walk_ready() {
    static const bool ok = cudaFuncSetAttribute(gemm_f32_kernel<32, EPI, true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                F32Tile<32>::WALK_SMEM) == cudaSuccess;
    return ok;
}

template <int BM, int EPI>
int launch_f32(F32Gemm p, cudaStream_t stream) {
    const int cols = EPI == kEpiGated ? kF32Cols / 2 : kF32Cols;
    const int nt = (p.N + cols - 1) / cols, mt = (p.M + BM - 1) / BM;
    const int* clusters = f32_clusters<32, EPI>();       // the larger tiles' for both heights: the same cut of k
    if (clusters == nullptr || f32_clusters<BM, EPI>() == nullptr) HOS_REFUSE("gemm_f32: the kernel does not fit on this GPU");
    p.splits = f32_splits(clusters, nt, p.K);
    if constexpr (BM == 32) {
        if (p.splits > 1 && f32_walks(clusters, (long long)nt * mt, p.splits, p.K)) {
            if (!f32_walk_ready<EPI>()) HOS_REFUSE("gemm_f32: the kernel does not fit on this GPU");
            gemm_f32_kernel<32, EPI, true><<<(unsigned)((long long)nt * mt), kF32Threads, F32Tile<32>::WALK_SMEM, stream>>>(p);
            return check_launch("gemm_f32");
        }
    }
    cudaLaunchAttribute attr[1];
    cudaLaunchConfig_t cfg = f32_config<BM, EPI>((long long)nt * mt, p.splits, attr, stream);
    cudaLaunchKernelEx(&cfg, gemm_f32_kernel<BM, EPI, false>, p);
    return check_launch("gemm_f32");
}

template <int EPI>
int launch_f32_rows(const F32Gemm& p, cudaStream_t stream) {
    return p.M <= 16 ? launch_f32<16, EPI>(p, stream) : launch_f32<32, EPI>(p, stream);
}

// Whether rows are whole 16-byte pieces and the launch's counts fit.
inline bool f32_can_take(const void* A, const void* W, long long M, long long N, int K, int lda, int ldw) {
    const long long tiles = (M / 16 + 1) * (N / 32 + 1);
    return (((uintptr_t)A | (uintptr_t)W) & 15) == 0 && ((K | lda | ldw) & 3) == 0 && tiles <= (1LL << 31) / (2 * kF32MaxSplits) && N <= (1LL << 28);
}

}  // namespace hos

using namespace hos;

// out[M, N] = A[M, K] . W[N, K]^T.  For the gated epilogue W has 2N rows (gate, then up); for the bias epilogue `bias` has N
// numbers or is null, and act 1 is the erf-form GELU, 2 the tanh form (0: none).
// Leading dimensions are in elements.
extern "C" int hos_gemm_plain(const void* A, int a_dtype, const void* W, int w_dtype, void* out,
                              int out_dtype, int M, int N, int K, int lda, int ldw, int ldo,
                              int epilogue, float cap, int act, const float* bias, cudaStream_t stream) {
    if (M <= 0 || N <= 0) return 0;
    if (K <= 0) HOS_REFUSE("gemm_plain: K must be positive");
    if (a_dtype == kF32 && w_dtype == kF32 && out_dtype == kF32 && f32_can_take(A, W, M, N, K, lda, ldw)) {
        F32Gemm p = {(const float*)A, (const float*)W, (float*)out, bias, M, N, K, lda, ldw, ldo, act, 1, cap};
        switch (epilogue) {
        case kEpiNone: return launch_f32_rows<kEpiNone>(p, stream);
        case kEpiSoftcap: return launch_f32_rows<kEpiSoftcap>(p, stream);
        case kEpiGated: return launch_f32_rows<kEpiGated>(p, stream);
        case kEpiBias: return launch_f32_rows<kEpiBias>(p, stream);
        default: HOS_REFUSE("gemm_plain: unknown epilogue %d", epilogue);
        }
    }
#define HOS_CASE(da, dw, dout, TA, TW, TO)                                         \
    if (a_dtype == da && w_dtype == dw && out_dtype == dout)                       \
        return launch_plain<TA, TW, TO>(A, W, out, M, N, K, lda, ldw, ldo, epilogue, cap, act, bias, stream);
    HOS_CASE(kF32, kF32, kF32, float, float, float)
    HOS_CASE(kBF16, kBF16, kBF16, bf16, bf16, bf16)
    HOS_CASE(kBF16, kBF16, kF32, bf16, bf16, float)
    HOS_CASE(kBF16, kF32, kBF16, bf16, float, bf16)
    HOS_CASE(kBF16, kF32, kF32, bf16, float, float)
    HOS_CASE(kF32, kBF16, kF32, float, bf16, float)
#undef HOS_CASE
    HOS_REFUSE("gemm_plain: no kernel for dtypes A=%d W=%d out=%d", a_dtype, w_dtype, out_dtype);
}

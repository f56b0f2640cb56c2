// Attention of whole prompts from position 0 over latent rows on the 5th-generation tensor cores, bfloat16.
//
// With many queries the absorbed form (latent_attention.cu) pays for its small cache in arithmetic: every (query, key) pair
// costs a head rank + rot + rank products, against dim + rot + vdim where keys and values are formed first.  Here the step's
// own latents are expanded once, by one product over all heads (the ordinary tcgen05 product, 32-bit results), and
// latent_expand_kernel writes what the attention reads.  Nothing that the absorbed form holds in 32 bits is rounded to 16 here:
//   a key's unrotated part [W_uk_h c]   two bfloat16 terms (16 bits of mantissa), as the absorbed query has there
//   a query's rotated part              two terms
//   a query's unrotated part, a key's rotated part (the cache's own row)   bfloat16 as projected or stored: exact
//   a value W_uv_h c, the weights       two terms
//
// The kernel is the walk of attention_prefill_tc.cu: one CTA takes 128 consecutive queries of one sequence and one head and
// walks over tiles of 64 keys; S = Q K^T from four products of 64 numbers (q k_hi, q k_lo, r_hi r_key, r_lo r_key) into tensor
// memory (two buffers), eight softmax warps (two threads per row), O += P_hi V_hi + P_lo V_hi + P_hi V_lo.
// Sizes up to 64 + 64 numbers a key and 128 a value fit: smaller ones are padded with zeros as they are written.
//
// Measured (B200, 16 heads, 64 + 64 and 128 numbers, rank 512, a window of 1,024 of 2,048 tokens): product 19 us, expansion 12,
// walk 57 (50 with the values as one term; what bounds it: 256 CTAs of up to 18 tiles on 148 SMs, one at a time, 1.4 us a tile); the
// absorbed form took 117 + 943 + 38 us with its products before and after.  Nuvivik's prompt of 2,048 tokens 9.50 -> 3.95 ms, of 4,000
// 19.3 -> 7.1, of 512 2.36 -> 1.67, of 64 1.03 -> 0.97.
#include "common.cuh"
#include "latent_rot.cuh"
#include "mma_utils.cuh"
#include "tcgen05_one.cuh"

namespace hos {

constexpr int LQ = 128, LK = 64;                        // queries of a CTA, keys of a tile
constexpr int LDIM = 64, LVDIM = 128;                   // numbers of a key's two parts, of a value, as laid out
constexpr int kLqCols = 3 * LDIM, kLkCols = 2 * LDIM, kLvCols = 2 * LVDIM;    // [q | r_hi | r_lo], [k_hi | k_lo], [v_hi | v_lo]
constexpr int kLqBlock = LQ * 128, kLkBlock = LK * 128; // a column block of 64 numbers of the queries, of a tile
constexpr int kLqBytes = 3 * kLqBlock, kLkBytes = 3 * kLkBlock, kLvTerm = LVDIM / 64 * kLkBlock, kLvBytes = 2 * kLvTerm;
constexpr int kLStages = 2, kLpBytes = 2 * LQ * 128;    // the weights' two terms
constexpr int kLSmem = kLqBytes + kLStages * (kLkBytes + kLvBytes) + 2 * kLpBytes + 2 * LQ * 4 + 160 + 976;
constexpr int kLThreads = 320;
constexpr int kLColS = 0, kLColO = 2 * LK, kLTmemCols = 256;
constexpr long long kLWaitCycles = 1ll << 31;
static_assert(kLSmem <= 232448 && kLColO + LVDIM <= kLTmemCols, "what an SM has");

__device__ int g_latent_prompt_error = 0;
__device__ int* g_latent_prompt_error_host = nullptr;   // a word in pinned host memory, if the host gave one

__device__ __forceinline__ void latent_give_up() {
    atomicExch(&g_latent_prompt_error, 1);
    int* w = g_latent_prompt_error_host;
    if (w != nullptr) {
        atomicExch_system(w, kGiveUpLatentPrompt);
        __threadfence_system();
    }
}

// ---- what the attention reads -------------------------------------------------------------------------------------
struct LatentExpand {
    const bf16* q;              // row n, head h at q + n * ldq + h * (dq + P): unrotated, then rotated numbers
    const float* kv;            // row n: the heads' W_uk_h c (dq each), then the heads' W_uv_h c (vd each)
    long long ldq;
    int H, dq, P, vd;
    LatentRot rot;
    const int* token_pos;
    const int* token_seq;
    bf16* q_out;                // [n][H][192]
    bf16* k_out;                // [n][H][128]
    bf16* v_out;                // [n][H][256]
    bf16* out;                  // the attention's output [n][H * vd]: zeros in padding rows, which the walk does not visit
};

__device__ __forceinline__ void split4(const float (&x)[4], uint2& hi, uint2& lo) {
    hi = make_uint2(pack_bf16(x[0], x[1]), pack_bf16(x[2], x[3]));
    lo = make_uint2(pack_bf16(x[0] - __uint_as_float(hi.x << 16), x[1] - __uint_as_float(hi.x & 0xffff0000u)),
                    pack_bf16(x[2] - __uint_as_float(hi.y << 16), x[3] - __uint_as_float(hi.y & 0xffff0000u)));
}

// A block per row, four numbers per thread and turn.
__global__ void __launch_bounds__(256) latent_expand_kernel(LatentExpand a) {
    pdl_enter();
    __shared__ float2 sincos_tab[LDIM / 2];
    const int n = blockIdx.x, H = a.H;
    bf16* v_out = a.v_out + (size_t)n * H * kLvCols;
    if (a.token_seq[n] < 0) {   // padding: nobody's key, but its values may lie in a tile with weight 0
        uint4* out = reinterpret_cast<uint4*>(a.out + (size_t)n * H * a.vd);
        for (int i = threadIdx.x; i < H * a.vd / 8; i += blockDim.x) out[i] = make_uint4(0u, 0u, 0u, 0u);
        for (int i = threadIdx.x; i < H * kLvCols / 4; i += blockDim.x) reinterpret_cast<uint2*>(v_out)[i] = make_uint2(0u, 0u);
        return;
    }
    const float pos = (float)a.token_pos[n];
    for (int i = threadIdx.x; i < a.rot.rot_dims >> 1; i += blockDim.x) {
        float s, c;
        sincosf(pos * a.rot.inv_freq[i], &s, &c);
        sincos_tab[i] = make_float2(s, c);
    }
    __syncthreads();
    const bf16* q = a.q + (size_t)n * a.ldq;
    const float* kv = a.kv + (size_t)n * H * (a.dq + a.vd);
    bf16* q_out = a.q_out + (size_t)n * H * kLqCols;
    bf16* k_out = a.k_out + (size_t)n * H * kLkCols;
    for (int i = threadIdx.x; i < H * LDIM / 4; i += blockDim.x) {
        const int h = i / (LDIM / 4), c = i % (LDIM / 4) * 4;
        const bf16* qh = q + (size_t)h * (a.dq + a.P);
        uint2 plain = make_uint2(0u, 0u), hi = plain, lo = plain, k_hi = plain, k_lo = plain;
        if (c < a.dq) {         // dq, P and vd are multiples of 8
            plain = *reinterpret_cast<const uint2*>(qh + c);
            const float4 k = *reinterpret_cast<const float4*>(kv + (size_t)h * a.dq + c);
            const float x[4] = {k.x, k.y, k.z, k.w};
            split4(x, k_hi, k_lo);
        }
        if (c < a.P) {
            float x[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) x[u] = rotated(qh + a.dq, c + u, sincos_tab, a.rot);
            split4(x, hi, lo);
        }
        *reinterpret_cast<uint2*>(q_out + h * kLqCols + c) = plain;
        *reinterpret_cast<uint2*>(q_out + h * kLqCols + LDIM + c) = hi;
        *reinterpret_cast<uint2*>(q_out + h * kLqCols + 2 * LDIM + c) = lo;
        *reinterpret_cast<uint2*>(k_out + h * kLkCols + c) = k_hi;
        *reinterpret_cast<uint2*>(k_out + h * kLkCols + LDIM + c) = k_lo;
    }
    const float* v = kv + (size_t)H * a.dq;
    for (int i = threadIdx.x; i < H * LVDIM / 4; i += blockDim.x) {
        const int h = i / (LVDIM / 4), c = i % (LVDIM / 4) * 4;
        uint2 hi = make_uint2(0u, 0u), lo = hi;
        if (c < a.vd) {
            const float4 t = *reinterpret_cast<const float4*>(v + (size_t)h * a.vd + c);
            const float x[4] = {t.x, t.y, t.z, t.w};
            split4(x, hi, lo);
        }
        *reinterpret_cast<uint2*>(v_out + h * kLvCols + c) = hi;
        *reinterpret_cast<uint2*>(v_out + h * kLvCols + LVDIM + c) = lo;
    }
}

// ---- the walk --------------------------------------------------------------------------------------------------------
struct LatentPrompt {
    bf16* out;                  // row n, head h at out + n * H * vd + h * vd
    const float* sink;
    const int* cu_seqlens;
    const int* token_seq;
    int n_seqs, n_rows, H, vd, rank, window;
    float scale;
    long long wait_cycles;      // the limit of every wait
    int stop_tile;              // for tests of the give-up path: the tile at which a softmax warp takes its wait as run out (-1: none)
};

__global__ void __launch_bounds__(kLThreads, 1)
latent_prompt_kernel(const __grid_constant__ CUtensorMap map_q,      // queries, boxes of [128 rows x 64 columns]
                     const __grid_constant__ CUtensorMap map_k,      // keys' unrotated parts, boxes of [64 x 64]
                     const __grid_constant__ CUtensorMap map_r,      // latent rows (their rotated part), boxes of [64 x 64]
                     const __grid_constant__ CUtensorMap map_v,      // values, boxes of [64 x 64]
                     LatentPrompt a) {
    pdl_launch_dependents();
    extern __shared__ unsigned char smem_unaligned[];
    unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_unaligned) + 1023) & ~(uintptr_t)1023);
    unsigned char* q_s = smem;
    unsigned char* k_s = q_s + kLqBytes;                         // [stage]: k_hi, k_lo, rotated part
    unsigned char* v_s = k_s + kLStages * kLkBytes;              // [stage]
    unsigned char* p_s = v_s + kLStages * kLvBytes;              // [buffer]: high terms, low terms
    float* xchg = reinterpret_cast<float*>(p_s + 2 * kLpBytes);  // [2 halves][128 rows]
    uint64_t* bars = reinterpret_cast<uint64_t*>(xchg + 2 * LQ);
    uint64_t* q_full = bars;                 // 1
    uint64_t* k_full = bars + 1;             // [2] keys of a stage have landed
    uint64_t* k_empty = bars + 3;            // [2] S of that stage has been computed: its keys may be replaced
    uint64_t* s_full = bars + 5;             // [2]
    uint64_t* s_empty = bars + 7;            // [2]
    uint64_t* p_full = bars + 9;             // [2] one per P buffer
    uint64_t* pv_done = bars + 11;           // [2] one per P buffer
    uint64_t* v_full = bars + 13;            // [2] values of a stage have landed
    uint64_t* v_empty = bars + 15;           // [2] P V of that stage is done: its values may be replaced
    uint32_t* tmem_base_smem = reinterpret_cast<uint32_t*>(bars + 17);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

    // long blocks first, the heads as the fast index (as in attention_prefill_tc.cu); the step's arrays of places are
    // written at its head, long before the kernel before this one
    int seq = 0, tile = blockIdx.y, row0 = 0, len = 0, nt = 0;
    for (; seq < a.n_seqs; ++seq) {
        row0 = a.cu_seqlens[seq];
        len = a.cu_seqlens[seq + 1] - row0;
        if (len > 0 && (row0 >= a.n_rows || a.token_seq[row0] < 0)) len = 0;               // padding
        nt = (len + LQ - 1) / LQ;
        if (tile < nt) break;
        tile -= nt;
    }
    if (seq >= a.n_seqs) return;
    const int q0 = (nt - 1 - tile) * LQ, head = blockIdx.x;      // positions are rows within the sequence
    const int last_q = min(len - 1, q0 + LQ - 1);
    const int kt_lo = (a.window > 0 ? max(0, q0 + 1 - a.window) : 0) / LK, kt_hi = last_q / LK;
    const int n_tiles = kt_hi - kt_lo + 1;

    if (threadIdx.x == 0) {
        mbar_init(q_full, 1);
        for (int s = 0; s < 2; ++s) {
            mbar_init(&k_full[s], 1); mbar_init(&k_empty[s], 1);
            mbar_init(&v_full[s], 1); mbar_init(&v_empty[s], 1);
            mbar_init(&s_full[s], 1); mbar_init(&s_empty[s], 8);
            mbar_init(&p_full[s], 8); mbar_init(&pv_done[s], 1);
        }
        mbar_fence_init();
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_base_smem)),
                     "r"(kLTmemCols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    const uint32_t tmem_base = *tmem_base_smem;
    bool ok = true;             // false: a wait of this thread (in the softmax warps: of its warp) ran out
    auto wait = [&](uint64_t* bar, uint32_t parity) { return mbar_wait_cycles(bar, parity, a.wait_cycles); };

    if (warp == 0) {
        // ---------------- TMA producer ----------------
        if (lane == 0) {
            pdl_wait();
            mbar_expect_tx(q_full, kLqBytes);
            for (int c = 0; c < 3; ++c) tc_tma_2d(q_s + c * kLqBlock, &map_q, head * kLqCols + 64 * c, row0 + q0, q_full);
            for (int j = 0; j < n_tiles && ok; ++j) {
                const int s = j % kLStages, krow = row0 + (kt_lo + j) * LK;
                unsigned char* kd = k_s + s * kLkBytes;
                unsigned char* vd = v_s + s * kLvBytes;
                if (j >= kLStages && !wait(&k_empty[s], ((j / kLStages) - 1) & 1)) { ok = false; break; }
                mbar_expect_tx(&k_full[s], kLkBytes);
                tc_tma_2d(kd, &map_k, head * kLkCols, krow, &k_full[s]);
                tc_tma_2d(kd + kLkBlock, &map_k, head * kLkCols + 64, krow, &k_full[s]);
                tc_tma_2d(kd + 2 * kLkBlock, &map_r, a.rank, krow, &k_full[s]);
                if (j >= kLStages && !wait(&v_empty[s], ((j / kLStages) - 1) & 1)) { ok = false; break; }
                mbar_expect_tx(&v_full[s], kLvBytes);
                for (int c = 0; c < kLvCols / 64; ++c)
                    tc_tma_2d(vd + c * kLkBlock, &map_v, head * kLvCols + 64 * c, krow, &v_full[s]);
            }
            if (!ok) latent_give_up();
        }
        __syncwarp();
    } else if (warp == 1) {
        // ---------------- MMA issuer ----------------
        if (lane == 0) {
            constexpr uint32_t idesc_s = tc_idesc(LQ, LK, 0);        // S = Q K^T: both K-major
            constexpr uint32_t idesc_o = tc_idesc(LQ, LVDIM, 1);     // O = P V: V is MN-major
            ok = wait(q_full, 0);
            tc_fence_after_sync();
            auto issue_s = [&](int j) -> bool {
                const int s = j % kLStages, sb = j & 1;
                if (!wait(&k_full[s], (j / kLStages) & 1)) return false;
                if (j >= 2 && !wait(&s_empty[sb], ((j >> 1) - 1) & 1)) return false;
                tc_fence_after_sync();
                const uint32_t k_addr = smem_u32(k_s + s * kLkBytes), q_addr = smem_u32(q_s);
#pragma unroll
                for (int b = 0; b < 4; ++b) {                        // q k_hi, q k_lo, r_hi r_key, r_lo r_key
                    const int qb = b < 2 ? 0 : b - 1, kb = b < 2 ? b : 2;
#pragma unroll
                    for (int kk = 0; kk < 4; ++kk)
                        tc_mma(tmem_base + kLColS + sb * LK, desc_kmajor(q_addr + qb * kLqBlock) + 2 * kk,
                               desc_kmajor(k_addr + kb * kLkBlock) + 2 * kk, idesc_s, b + kk > 0 ? 1u : 0u);
                }
                tc_commit(&s_full[sb]);
                tc_commit(&k_empty[s]);
                return true;
            };
            if (ok) ok = issue_s(0);
            for (int j = 0; j < n_tiles && ok; ++j) {
                if (j + 1 < n_tiles && !issue_s(j + 1)) { ok = false; break; }      // the next S runs under this tile's softmax
                const int pb = j & 1, s = j % kLStages;
                if (!wait(&p_full[pb], (j >> 1) & 1)) { ok = false; break; }
                if (!wait(&v_full[s], (j / kLStages) & 1)) { ok = false; break; }
                tc_fence_after_sync();
                const uint32_t v_addr = smem_u32(v_s + s * kLvBytes), p_addr = smem_u32(p_s + pb * kLpBytes);
#pragma unroll
                for (int term = 0; term < 3; ++term)                 // P_hi V_hi, P_lo V_hi, P_hi V_lo
#pragma unroll
                    for (int ks = 0; ks < LK / 16; ++ks)
                        tc_mma(tmem_base + kLColO, desc_kmajor(p_addr + (term == 1 ? LQ * 128 : 0)) + 2 * ks,
                               desc_mnmajor(v_addr + (term == 2 ? kLvTerm : 0) + ks * 16 * 128, kLkBlock), idesc_o, (j > 0 || term > 0 || ks > 0) ? 1u : 0u);
                tc_commit(&v_empty[s]);
                tc_commit(&pv_done[pb]);      // this P buffer has been read, O holds tile j
            }
            if (!ok) latent_give_up();
        }
        __syncwarp();
    } else {
        // ---------------- softmax, correction, epilogue: two threads per query row ----------------
        const int quarter = warp & 3;
        const int half = (warp - 2) >> 2;                        // which 32 of the tile's 64 keys
        const int r = quarter * 32 + lane;                       // row of the tile = lane of tensor memory
        const uint32_t t_lane = tmem_base + ((uint32_t)(quarter * 32) << 16);
        const int qpos = q0 + r;
        const float c2 = a.scale * 1.4426950408889634f;          // weights are exp2(s c2 - m c2), the maximum over raw s
        const float slack = 8.f / a.scale;                       // the running maximum is raised when exceeded by e^8
        float m_ref = -INFINITY, l_run = 0.f;                    // l_run: this thread's keys only
        // The eight warps meet at barriers, twice a tile and twice at the end, so none of them leaves on its own: a warp whose
        // wait ran out waits for nothing and computes nothing any more, but comes to every barrier that is left.  The others'
        // waits for what it then does not hand on run out in turn, once for each, so the block ends.
        auto warp_wait = [&](uint64_t* bar, uint32_t parity) { return __all_sync(0xffffffffu, wait(bar, parity)) != 0; };
        for (int j = 0; j < n_tiles; ++j) {
            const int sb = j & 1, pb = j & 1;
            const int kt0 = (kt_lo + j) * LK, k0 = kt0 + 32 * half;
            float m_half = -INFINITY;
            float sc[32];
            if (ok) ok = warp_wait(&s_full[sb], (j >> 1) & 1);
            if (ok) {
                tc_fence_after_sync();
                {
                    uint32_t v0[32];
                    tc_ld32(t_lane + kLColS + sb * LK + 32 * half, v0);
                    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                    for (int i = 0; i < 32; ++i) sc[i] = __uint_as_float(v0[i]);
                }
                tc_fence_before_sync();
                __syncwarp();
                if (lane == 0) mbar_arrive(&s_empty[sb]);
                const bool whole = kt0 + LK - 1 <= q0 && (a.window <= 0 || kt0 > q0 + LQ - 1 - a.window);
                if (!whole) {
#pragma unroll
                    for (int i = 0; i < 32; ++i) {
                        const int key = k0 + i;
                        sc[i] = key <= qpos && (a.window <= 0 || key > qpos - a.window) ? sc[i] : -INFINITY;
                    }
                }
#pragma unroll
                for (int i = 0; i < 32; ++i) m_half = fmaxf(m_half, sc[i]);
            }
            xchg[half * LQ + r] = m_half;
            asm volatile("bar.sync 1, 256;" ::: "memory");
            const float m_tile = fmaxf(m_half, xchg[(half ^ 1) * LQ + r]);
            asm volatile("bar.sync 1, 256;" ::: "memory");       // both have read before the next tile writes
            if (!ok) continue;
            float factor = 1.f;
            if (m_tile > m_ref + slack || (m_ref == -INFINITY && m_tile > -INFINITY)) {
                factor = m_ref == -INFINITY ? 0.f : ex2_approx((m_ref - m_tile) * c2);
                m_ref = m_tile;
            }
            const float m_use2 = (m_ref == -INFINITY ? 0.f : m_ref) * c2;
            float psum = 0.f;
            uint32_t hi[16], lo[16];
#pragma unroll
            for (int i = 0; i < 32; i += 2) {
                const float w0 = ex2_approx(fmaf(sc[i], c2, -m_use2)), w1 = ex2_approx(fmaf(sc[i + 1], c2, -m_use2));
                psum += w0 + w1;
                hi[i / 2] = pack_bf16(w0, w1);
                lo[i / 2] = pack_bf16(w0 - __uint_as_float(hi[i / 2] << 16), w1 - __uint_as_float(hi[i / 2] & 0xffff0000u));
            }
            l_run = l_run * factor + psum;
            if (j >= 2) ok = warp_wait(&pv_done[pb], ((j >> 1) - 1) & 1);
            if (j == a.stop_tile && warp == 2) ok = false;
            if (!ok) continue;
            if (j > 0 && __any_sync(0xffffffffu, factor != 1.f)) {
                // O is touched only between products: wait for the one of the tile before
                ok = warp_wait(&pv_done[pb ^ 1], ((j - 1) >> 1) & 1);
                if (!ok) continue;
                tc_fence_after_sync();
#pragma unroll 1
                for (int c = half * (LVDIM / 2); c < (half + 1) * (LVDIM / 2); c += 32) {
                    uint32_t o[32];
                    tc_ld32(t_lane + kLColO + c, o);
                    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                    for (int i = 0; i < 32; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * factor);
                    tc_st32(t_lane + kLColO + c, o);
                }
                asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
            }
            // this thread's 32 keys of row r: pieces 4 half .. 4 half + 3 of 16 bytes, piece c at c ^ (r & 7)
            unsigned char* prow = p_s + (size_t)pb * kLpBytes + (size_t)r * 128;
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                const int at = ((4 * half + c) ^ (r & 7)) << 4;
                *reinterpret_cast<uint4*>(prow + at) = make_uint4(hi[4 * c], hi[4 * c + 1], hi[4 * c + 2], hi[4 * c + 3]);
                *reinterpret_cast<uint4*>(prow + LQ * 128 + at) = make_uint4(lo[4 * c], lo[4 * c + 1], lo[4 * c + 2], lo[4 * c + 3]);
            }
            if (kt0 + LK > len) {
                // the tile's rows beyond the sequence are another's, whose values must not matter (0 times infinity)
                const int s = j % kLStages, vr = (int)(threadIdx.x - 64) >> 2, part = threadIdx.x & 3;
                ok = warp_wait(&v_full[s], (j / kLStages) & 1);
                if (!ok) continue;
                if (kt0 + vr >= len)
                    for (int c = part * 8; c < part * 8 + 8; ++c)
                        *reinterpret_cast<uint4*>(v_s + s * kLvBytes + (c >> 3) * kLkBlock + vr * 128 + (c & 7) * 16) = make_uint4(0u, 0u, 0u, 0u);
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");     // generic writes -> visible to the tensor core
            tc_fence_before_sync();
            __syncwarp();
            if (lane == 0) mbar_arrive(&p_full[pb]);
        }
        // ---- epilogue: O / l -> bfloat16; each thread half of its row ----
        if (ok) ok = warp_wait(&pv_done[(n_tiles - 1) & 1], ((n_tiles - 1) >> 1) & 1);
        tc_fence_after_sync();
        asm volatile("bar.sync 1, 256;" ::: "memory");      // every reader of xchg's maxima is done
        xchg[half * LQ + r] = l_run;
        asm volatile("bar.sync 1, 256;" ::: "memory");
        if (ok) {
            float l_row = l_run + xchg[(half ^ 1) * LQ + r];
            if (a.sink != nullptr) l_row += expf(a.sink[head] - m_ref * a.scale);
            const float inv = l_row > 0.f ? 1.f / l_row : 0.f;
            bf16* orow = a.out + (size_t)(row0 + q0 + r) * a.H * a.vd + (size_t)head * a.vd;
#pragma unroll 1
            for (int c = half * (LVDIM / 2); c < (half + 1) * (LVDIM / 2); c += 32) {
                uint32_t o[32];
                tc_ld32(t_lane + kLColO + c, o);
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                if (q0 + r < len) {
#pragma unroll
                    for (int q4 = 0; q4 < 4; ++q4)
                        if (c + 8 * q4 < a.vd)                   // a multiple of 8
                            *reinterpret_cast<uint4*>(orow + c + 8 * q4) = make_uint4(
                                pack_bf16(__uint_as_float(o[8 * q4]) * inv, __uint_as_float(o[8 * q4 + 1]) * inv),
                                pack_bf16(__uint_as_float(o[8 * q4 + 2]) * inv, __uint_as_float(o[8 * q4 + 3]) * inv),
                                pack_bf16(__uint_as_float(o[8 * q4 + 4]) * inv, __uint_as_float(o[8 * q4 + 5]) * inv),
                                pack_bf16(__uint_as_float(o[8 * q4 + 6]) * inv, __uint_as_float(o[8 * q4 + 7]) * inv));
                }
            }
        }
        if (!ok && lane == 0) latent_give_up();
    }
    tc_fence_before_sync();
    if (__syncthreads_or(!ok)) let_work_under_way_end();
    if (warp == 1)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(kLTmemCols) : "memory");
}

}  // namespace hos

using namespace hos;

// The host's word for waits that ran out; null takes it away.
extern "C" int hos_latent_prompt_set_error_word(int* word) {
    if (cudaMemcpyToSymbol(g_latent_prompt_error_host, &word, sizeof(word)) != cudaSuccess)
        HOS_REFUSE("latent_prompt: cannot set the error word: %s", cudaGetErrorString(cudaGetLastError()));
    return 0;
}

// Rows 0 .. n_rows - 1 of a step whose sequences all start at position 0 (sequence s has the rows cu_seqlens[s] ..).
// q: row n, head h at q + n * ldq + h * (dq + P); kv: 32-bit [n_rows][H * dq + H * vd], the latents expanded; kc: the latent
// rows [n_rows][rank + P].  q_ws [n_rows][H][192], k_ws [n_rows][H][128] and v_ws [n_rows][H][256] bfloat16: scratch.  out [n_rows][H * vd], zeros
// in padding rows (token_seq < 0).
// n_q_tiles: at least the sum over the sequences of ceil(rows / 128).  wait_cycles, stop_tile: for tests of what happens when a
// wait runs out (LatentPrompt); 0 and -1 otherwise.
extern "C" int hos_latent_prompt(const void* q, long long ldq, const float* kv, const void* kc, const float* inv_freq, int rot_dims,
                                 int style, const float* sink, const int* token_pos, const int* token_seq, const int* cu_seqlens,
                                 int n_seqs, int n_q_tiles, int n_rows, int H, int dq, int P, int vd, int rank, float scale, int window,
                                 void* q_ws, void* k_ws, void* v_ws, void* out, long long wait_cycles, int stop_tile,
                                 cudaStream_t stream) {
    if (n_rows <= 0 || n_seqs <= 0 || n_q_tiles <= 0) return 0;
    if (H <= 0 || dq <= 0 || dq > LDIM || P <= 0 || P > LDIM || vd <= 0 || vd > LVDIM || ((dq | P | vd | rank) & 7) || (ldq & 3))
        HOS_REFUSE("latent_prompt: keys of %d + %d and values of %d numbers (rank %d) are not multiples of 8 up to %d, %d and %d",
                   dq, P, vd, rank, LDIM, LDIM, LVDIM);
    if (!(scale > 0.f)) HOS_REFUSE("latent_prompt: the scale must be positive");
    if (n_q_tiles > 65535) HOS_REFUSE("latent_prompt: %d blocks of queries are more than one launch takes", n_q_tiles);
    if (((uintptr_t)q & 7) || (((uintptr_t)kv | (uintptr_t)kc | (uintptr_t)q_ws | (uintptr_t)k_ws | (uintptr_t)v_ws | (uintptr_t)out) & 15))
        HOS_REFUSE("latent_prompt: rows must be 16-byte aligned");
    CUtensorMap mq, mk, mr, mv;
    int rc;
    if ((rc = tc_make_map(&mq, q_ws, n_rows, H * kLqCols, H * kLqCols, LQ))) return rc;
    if ((rc = tc_make_map(&mk, k_ws, n_rows, H * kLkCols, H * kLkCols, LK))) return rc;
    if ((rc = tc_make_map(&mr, kc, n_rows, rank + P, rank + P, LK))) return rc;
    if ((rc = tc_make_map(&mv, v_ws, n_rows, H * kLvCols, H * kLvCols, LK))) return rc;
    if (cudaFuncSetAttribute(latent_prompt_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kLSmem) != cudaSuccess)
        HOS_REFUSE("latent_prompt: cannot get %d bytes of shared memory", kLSmem);
    LatentExpand e = {(const bf16*)q, kv, ldq, H, dq, P, vd, {inv_freq, inv_freq != nullptr ? rot_dims : 0, style}, token_pos, token_seq,
                      (bf16*)q_ws, (bf16*)k_ws, (bf16*)v_ws, (bf16*)out};
    launch_pdl(latent_expand_kernel, dim3(n_rows), dim3(256), 0, stream, e);
    if ((rc = check_launch("latent_prompt (expansion)"))) return rc;
    LatentPrompt a = {(bf16*)out, sink, cu_seqlens, token_seq, n_seqs, n_rows, H, vd, rank, window, scale,
                      wait_cycles > 0 ? wait_cycles : kLWaitCycles, stop_tile};
    launch_pdl(latent_prompt_kernel, dim3(H, n_q_tiles), dim3(kLThreads), kLSmem, stream, mq, mk, mr, mv, a);
    return check_launch("latent_prompt");
}

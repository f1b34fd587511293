// Quantized-weight linear for prompts (more than 128 tokens): the streaming kernel's pipeline (gemm_stream.cuh) on
// CTA pairs, with an accumulator of up to 384 tokens, so that a weight is dequantised once for all of a prompt's
// tokens.
//
// What bounds it: tensor arithmetic, and next to it the copies into shared memory.  A 64-k block of 256 features x
// 304 tokens is 606 cycles of each SM's tensor core; dequantising an SM's 8192 weights is about 250 cycles of its issue
// slots, spread over sixteen warps.
//   * a pair of CTAs (cta_group::2) computes 256 features x up to 384 tokens: each CTA dequantises its own 128
//     features into its own tensor memory (the UMMA's A operand: columns 384 ..) and brings HALF of the activation
//     rows.  With one CTA per tile each SM fetched and stored all rows: 148 SMs x 44 KB per 0.5 us block is more than L2
//     delivers, and the stores and the UMMA's reads together were more than shared memory takes (301 tokens,
//     4096 x 12288: 0.50 us per block);
//   * sixteen dequantise warps in two teams: team t takes the k blocks j with j % 2 == t, so that one team's
//     shared-memory reads and conversions run while the other's TMEM stores and barrier arrivals are under way;
//   * the k range is cut into 1 .. 4 slices that run as one thread-block cluster of 2 .. 8 CTAs, summed through
//     distributed shared memory in slice order (no workspace, the same bits every run);
//   * token tiles are the launch's second dimension, equal in width (a multiple of sixteen tokens);
//   * barriers as in gemm_prefill_pair.cuh: one "full" barrier per k block (activation bytes, dequantise warps, on the
//     leader also the other CTA's forward) and one "done" barrier that the leader's commit signals in both CTAs.
// Measured (B200, one linear in a CUDA graph of distinct weights; the prefill kernel's tiles before -> this): FP4 6144 / 4096 /
// 24576 x 4096 and 4096 x 12288 at 301 tokens 40 -> 22, 41 -> 19, 108 -> 66, 119 -> 34 us; at 1024 tokens 66 -> 37, 48 -> 30,
// 157 -> 156 (the pair tile again), 136 -> 74 us.  The four calls of a Llama-3.1-8B layer at 301 tokens: 328 -> 155 us.
#pragma once

#include "gemm_prefill_pair.cuh"
#include "gemm_stream.cuh"

namespace b200
{

constexpr int SW_TEAMS = 2;                              // teams of SK_DQ_WARPS dequantise warps
constexpr int SW_DQ_WARPS = SW_TEAMS * SK_DQ_WARPS;
constexpr int SW_THREADS = 32 * (SW_DQ_WARPS + 3);       // + activation TMA warp, MMA warp, weight TMA warp
constexpr int SW_A_STAGES = 4;                           // A stages in TMEM
constexpr int SW_RING = 8;                               // k blocks in flight at most: barrier slots, activation stages
constexpr int SW_X_MIN_STAGES = 6;                       // activation stages in shared memory at the widest tile
constexpr int SW_MAX_SPLIT = 4;                          // k slices: clusters of up to eight CTAs
constexpr int SW_MAX_TOKENS = 384;                       // accumulator columns
constexpr int SW_A_COLS = SK_BK / 2;                     // TMEM columns of one A stage
constexpr int SW_RUNS = 4;                               // 64-byte runs per raw weight stage
constexpr int SW_RAW_STAGES = 2;
constexpr int SW_X_RING_BYTES = SW_X_MIN_STAGES * SW_MAX_TOKENS / 2 * SK_BK * 2;    // 144 KB of [tokens / 2][64 k] tiles
__host__ __device__ constexpr int sw_smem_bytes(int wt)
{
    return SK_HEADER_BYTES + SW_X_RING_BYTES + SW_RAW_STAGES * sk_raw_bytes(wt, SW_RUNS) + 1024;
}
static_assert(SW_MAX_TOKENS + SW_A_STAGES * SW_A_COLS <= 512, "accumulator and A stages share the 512 TMEM columns");
static_assert(SW_MAX_TOKENS * SK_BM * 4 <= SW_X_RING_BYTES + SW_RAW_STAGES * sk_raw_bytes(DT_E4M3, SW_RUNS),
    "the partial tile reuses the activation stages and the raw ring");

struct StreamWideParams
{
    StreamParams s;
    unsigned int tile_tokens;    // tokens per token tile: chunks * chunk
    unsigned int chunk, chunks;  // tokens per UMMA (a multiple of sixteen), UMMAs per tile
    unsigned int x_stages;       // activation stages in the ring
    unsigned int keep_weights;   // 1: several token tiles read the weights, they are worth keeping in L2
};

// D[tmem of both CTAs] (+)= A[tmem of both CTAs: 128 rows each] * B[smem of both CTAs: N/2 rows each]; BF16, FP32 accumulate.
__device__ __forceinline__ void umma_bf16_ts_pair(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc, uint32_t accumulate)
{
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], [%1], %2, %3, p;\n\t}" ::"r"(d_tmem),
        "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(accumulate)
        : "memory");
}
// umma_commit_pair for a pair that is part of a larger cluster: `mask` names the pair's two CTAs.
__device__ __forceinline__ void umma_commit_pair_mask(uint64_t* bar, uint16_t mask)
{
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(smem_u32(bar)),
                 "h"(mask)
                 : "memory");
}

template <int WT, bool SCALED>
__global__ void __launch_bounds__(SW_THREADS, 1) gemm_wq_stream_wide_kernel(const __grid_constant__ CUtensorMap tmX, const __grid_constant__ StreamWMaps tmW,
    const StreamWideParams wp)
{
    namespace cg = cooperative_groups;
    const StreamParams& p = wp.s;
    constexpr int RAW_W_BYTES = sk_raw_w_bytes(SW_RUNS);
    constexpr int RAW_BYTES = sk_raw_bytes(WT, SW_RUNS);
    constexpr int KB_PER_RAW = sk_kb_per_raw(WT, SW_RUNS);
    extern __shared__ unsigned char sw_smem_raw[];
    // the aligned base lies at the same offset in every CTA of the cluster, so peers map each other's tiles
    unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(sw_smem_raw) + 1023) & ~(uintptr_t)1023);
    uint64_t* full = reinterpret_cast<uint64_t*>(smem);    // [8] k block kb % 8: my activations and weights (leader: the pair's)
    uint64_t* done = full + SW_RING;                       // [8] its UMMAs are complete
    uint64_t* raw_full = done + SW_RING;
    uint64_t* raw_empty = raw_full + SW_RAW_STAGES;
    uint64_t* acc_full = raw_empty + SW_RAW_STAGES;
    uint32_t* tmem_base_slot = reinterpret_cast<uint32_t*>(acc_full + 1);
    volatile unsigned int* abort_flag = reinterpret_cast<volatile unsigned int*>(tmem_base_slot + 1);
    unsigned char* xs = smem + SK_HEADER_BYTES;
    unsigned char* raws = xs + SW_X_RING_BYTES;

    cg::cluster_group cluster = cg::this_cluster();
    const unsigned int S = p.split;
    const unsigned int cta = cluster_cta_rank(), rank = cta >> 1, half_cta = cta & 1u;    // k slice, half of the pair
    const unsigned int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    unsigned int si = 0;
    if (p.n_seg > 1 && blockIdx.z >= p.seg[1].tile0) { si = 1; }
    if (p.n_seg > 2 && blockIdx.z >= p.seg[2].tile0) { si = 2; }
    const PrefillSeg& g = p.seg[si];
    const unsigned int n0 = (blockIdx.z - g.tile0) * (2 * SK_BM) + half_cta * SK_BM;    // my CTA's features
    const unsigned int m0 = blockIdx.y * wp.tile_tokens;
    const unsigned int live = min(wp.tile_tokens, p.M - m0);    // live tokens of this tile
    // tokens of the tile's one or two UMMAs (N: a multiple of sixteen); each CTA brings half of either
    const unsigned int live0 = (min(live, wp.chunk) + 15u) & ~15u, live1 = live > wp.chunk ? (live - wp.chunk + 15u) & ~15u : 0u;
    const unsigned int pitch = wp.tile_tokens / 2 * SK_BK * 2;    // bytes of an activation stage
    const unsigned int units = p.K / SK_SLICE_ELEMS;
    const unsigned int kb_begin = (unsigned int)(((unsigned long long)units * rank) / S) * (SK_SLICE_ELEMS / SK_BK);
    const unsigned int kb_end = (unsigned int)(((unsigned long long)units * (rank + 1)) / S) * (SK_SLICE_ELEMS / SK_BK);
    const unsigned int nkb = kb_end - kb_begin;    // a multiple of four
    const unsigned int n_raw = (nkb + KB_PER_RAW - 1) / KB_PER_RAW;

    if (threadIdx.x == 0)
    {
        for (int s = 0; s < SW_RING; s++)
        {
            mbar_init(full + s, 1 + SK_DQ_WARPS + (half_cta == 0 ? 1 : 0));
            mbar_init(done + s, 1);
        }
        for (int s = 0; s < SW_RAW_STAGES; s++)
        {
            mbar_init(raw_full + s, 1);
            mbar_init(raw_empty + s, SW_DQ_WARPS);
        }
        mbar_init(acc_full, 1);
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == SW_DQ_WARPS + 1) { tmem_alloc_pair(tmem_base_slot, 512); }
    tc_fence_before();
    __syncthreads();
    cluster_sync_all();    // both CTAs' barriers exist before any remote arrive or commit
    tc_fence_after();
    const uint32_t tmem_base = *tmem_base_slot;
    const uint32_t tmem_a = tmem_base + SW_MAX_TOKENS;
    pdl_launch_dependents();

    if (warp == SW_DQ_WARPS + 2)
    {
        // =========================== TMA lane: quantised weights ===========================
        if (lane == 0)
        {
            const uint64_t pol = l2_policy_evict_first();
            auto load = [&](void* dst, const CUtensorMap* map, int row, int run, uint64_t* bar) {
                if (wp.keep_weights) { tma_load_3d(dst, map, 0, row, run, bar); }
                else { tma_load_3d_hint(dst, map, 0, row, run, bar, pol); }
            };
            bool ok = true;
            unsigned int issued = 0;
            for (unsigned int r = 0; r < n_raw; r++)
            {
                const unsigned int s = r % SW_RAW_STAGES;
                if (r >= SW_RAW_STAGES && (*abort_flag != 0 || !mbar_wait_bounded(raw_empty + s, ((r / SW_RAW_STAGES) - 1) & 1u)))
                {
                    ok = false;
                    atomicMax(p.status, (unsigned int)ST_TIMEOUT_EMPTY);
                    *abort_flag = 1;
                    break;
                }
                unsigned char* dst = raws + s * RAW_BYTES;
                const unsigned int kb0 = kb_begin + r * KB_PER_RAW;
                mbar_expect_tx(raw_full + s, RAW_BYTES);
                load(dst, &tmW.w[si], (int)n0, (int)(WT == DT_FP4 ? kb0 / 2 : kb0), raw_full + s);
                if (WT == DT_FP4) { load(dst + RAW_W_BYTES, &tmW.s[si], (int)n0, (int)(kb0 / 4), raw_full + s); }
                mbar_arrive(raw_full + s);
                issued = r + 1;
            }
            if (!ok)
            {
                const unsigned int first = issued > SW_RAW_STAGES ? issued - SW_RAW_STAGES : 0;
                for (unsigned int r = first; r < issued; r++) { mbar_wait_bounded(raw_full + (r % SW_RAW_STAGES), (r / SW_RAW_STAGES) & 1u); }
            }
        }
    }
    else if (warp == SW_DQ_WARPS)
    {
        // =========================== TMA lane: activations ===========================
        if (lane == 0)
        {
            pdl_wait();    // the activations are the previous kernel's output
            bool ok = true;
            unsigned int issued = 0;
            const unsigned int box = wp.chunk / 2 * SK_BK * 2;    // bytes; a tile's second half may lie past the last token
            for (unsigned int j = 0; j < nkb; j++)
            {
                const unsigned int s = j % wp.x_stages, before = j - wp.x_stages;
                if (j >= wp.x_stages && (*abort_flag != 0 || !mbar_wait_bounded(done + before % SW_RING, (before / SW_RING) & 1u)))
                {
                    ok = false;
                    atomicMax(p.status, (unsigned int)ST_TIMEOUT_EMPTY);
                    *abort_flag = 1;
                    break;
                }
                uint64_t* bar = full + j % SW_RING;
                mbar_expect_tx(bar, live1 != 0 ? 2 * box : box);
                tma_load_2d(xs + s * pitch, &tmX, (int)((kb_begin + j) * SK_BK), (int)(m0 + half_cta * (live0 / 2)), bar);
                if (live1 != 0) { tma_load_2d(xs + s * pitch + box, &tmX, (int)((kb_begin + j) * SK_BK), (int)(m0 + wp.chunk + half_cta * (live1 / 2)), bar); }
                mbar_arrive(bar);
                issued = j + 1;
            }
            if (!ok)
            {
                // The barriers also count the dequantise warps, which may have given up too: the copies land within
                // microseconds, 100 us per barrier is ample.
                const unsigned int first = issued > wp.x_stages ? issued - wp.x_stages : 0;
                for (unsigned int j = first; j < issued; j++)
                {
                    const unsigned long long t0 = global_timer_ns();
                    while (!mbar_try_wait(full + j % SW_RING, (j / SW_RING) & 1u) && global_timer_ns() - t0 < 100000ull) {}
                }
            }
        }
    }
    else if (warp == SW_DQ_WARPS + 1)
    {
        if (half_cta != 0)
        {
            // =========================== second CTA: forward "block full" to the leader ===========================
            if (lane == 0)
            {
                const uint32_t peer = map_to_cta(full, cta - 1);
                for (unsigned int j = 0; j < nkb; j++)
                {
                    if (*abort_flag != 0 || !mbar_wait_bounded(full + j % SW_RING, (j / SW_RING) & 1u))
                    {
                        atomicMax(p.status, (unsigned int)ST_TIMEOUT_FULL);
                        *abort_flag = 1;
                        break;
                    }
                    mbar_arrive_cluster(peer + (j % SW_RING) * 8);
                }
            }
        }
        else
        {
            // =========================== leader: UMMA warp ===========================
            bool ok = true;
            const uint32_t idesc0 = umma_idesc_bf16(2 * SK_BM, live0), idesc1 = umma_idesc_bf16(2 * SK_BM, live1);
            const uint16_t mask = (uint16_t)(3u << cta);
            unsigned int xstage = 0;
            for (unsigned int j = 0; j < nkb && ok; j++)
            {
                if (*abort_flag != 0 || !mbar_wait_bounded(full + j % SW_RING, (j / SW_RING) & 1u))
                {
                    ok = false;
                    if (lane == 0)
                    {
                        atomicMax(p.status, (unsigned int)ST_TIMEOUT_FULL);
                        *abort_flag = 1;
                    }
                    break;
                }
                tc_fence_after();
                const uint32_t b_addr = smem_u32(xs + xstage * pitch), b_addr1 = b_addr + wp.chunk / 2 * SK_BK * 2;
                const uint32_t a_tmem = tmem_a + (j % SW_A_STAGES) * SW_A_COLS;
                if (elect_one())
                {
#pragma unroll
                    for (int k = 0; k < SK_BK / 16; k++)
                    {
                        // 16 k of A = 8 TMEM columns; of B = 32 bytes further along the 128-byte swizzle row
                        const uint32_t accumulate = (j | (unsigned int)k) != 0 ? 1u : 0u;
                        umma_bf16_ts_pair(tmem_base, a_tmem + k * 8, umma_desc_kmajor_sw128(b_addr + k * 32), idesc0, accumulate);
                        if (live1 != 0) { umma_bf16_ts_pair(tmem_base + wp.chunk, a_tmem + k * 8, umma_desc_kmajor_sw128(b_addr1 + k * 32), idesc1, accumulate); }
                    }
                    umma_commit_pair_mask(done + j % SW_RING, mask);
                }
                __syncwarp();
                if (++xstage == wp.x_stages) { xstage = 0; }
            }
            __syncwarp();
            // also on the abort path: it completes once the UMMAs in flight no longer read either CTA's memory
            if (elect_one()) { umma_commit_pair_mask(acc_full, mask); }
        }
    }
    else
    {
        // =========================== dequantise (warps 0 .. 15) ===========================
        // thread = (output feature, k half) of its team's k blocks: TMEM lane 32 (warp & 3) + lane, columns 16 half ..
        const unsigned int row = (warp & 3u) * 32 + lane;
        const unsigned int half = (warp >> 2) & 1u;
        const unsigned int team = warp >> 3;
        const uint32_t lane_field = ((warp & 3u) * 32u) << 16;
        const uint32_t sw64 = (row >> 1) & 3u;    // the TMA's 64-byte swizzle: 16-byte chunk index ^= row bits 1-2
        bool ok = true;
        for (unsigned int j = team; j < nkb; j += SW_TEAMS)
        {
            const unsigned int r = j / KB_PER_RAW, jr = j % KB_PER_RAW;
            const unsigned int rs = r % SW_RAW_STAGES;
            if (ok && jr < SW_TEAMS && (*abort_flag != 0 || !mbar_wait_bounded(raw_full + rs, (r / SW_RAW_STAGES) & 1u)))
            {
                ok = false;
                if (*abort_flag == 0)
                {
                    atomicMax(p.status, (unsigned int)ST_TIMEOUT_FULL);
                    *abort_flag = 1;
                }
            }
            const unsigned int s = j % SW_A_STAGES;
            uint64_t* const before = done + (j - SW_A_STAGES) % SW_RING;    // the block that used the A stage last
            const uint32_t epar = ((j - SW_A_STAGES) / SW_RING) & 1u;
            const bool stage_free = (j < SW_A_STAGES) || mbar_try_wait(before, epar);    // asked early, needed late
            uint32_t out[16];
            if (ok)
            {
                const uint32_t raw = smem_u32(raws + rs * RAW_BYTES);
                if (WT == DT_FP4)
                {
                    // run jr / 2 holds 128 k of the row; my 32 k of the block are one 16-byte chunk
                    const uint4 v = sk_lds128(raw + (jr >> 1) * (SK_BM * 64) + row * 64 + ((((jr & 1u) * 2 + half) ^ sw64) << 4));
                    const uint32_t sc = sk_lds16(raw + RAW_W_BYTES + (jr >> 2) * (SK_BM * 16) + row * 16 + (jr & 3u) * 4 + half * 2);
                    uint32_t lo[8], hi[8];
                    dequant_fp4x16_natural(make_uint2(v.x, v.y), sc & 0xFFu, lo);
                    dequant_fp4x16_natural(make_uint2(v.z, v.w), sc >> 8, hi);
#pragma unroll
                    for (int q = 0; q < 8; q++)
                    {
                        out[q] = lo[q];
                        out[8 + q] = hi[q];
                    }
                }
                else
                {
                    const uint32_t base = raw + jr * (SK_BM * 64) + row * 64;
                    const uint4 a = sk_lds128(base + (((2 * half) ^ sw64) << 4)), b = sk_lds128(base + (((2 * half + 1) ^ sw64) << 4));
                    const uint32_t w[8] = { a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w };
#pragma unroll
                    for (int q = 0; q < 8; q++) { dequant_fp8x4<WT, SCALED>(w[q], g.w_scale, out[2 * q], out[2 * q + 1]); }
                }
            }
            // my last block of this raw stage has been read into registers
            if (ok && (jr + SW_TEAMS >= KB_PER_RAW || j + SW_TEAMS >= nkb))
            {
                __syncwarp();
                if (lane == 0) { mbar_arrive(raw_empty + rs); }
            }
            if (ok && !stage_free && (*abort_flag != 0 || !mbar_wait_bounded(before, epar)))
            {
                ok = false;
                if (*abort_flag == 0)
                {
                    atomicMax(p.status, (unsigned int)ST_TIMEOUT_EMPTY);
                    *abort_flag = 1;
                }
            }
            if (ok)
            {
                tc_fence_after();    // the UMMAs that read this stage last have completed (the empty barrier said so)
                tmem_st_32x16(tmem_a + lane_field + s * SW_A_COLS + half * 16, out);
                tmem_st_wait();
                tc_fence_before();
                __syncwarp();
                if (lane == 0) { mbar_arrive(full + j % SW_RING); }
            }
        }
    }

    // ---- the slices' partial tiles: TMEM -> this CTA's shared memory ----
    float* part = reinterpret_cast<float*>(xs);    // [tokens][128 features]; the activation stages and the raw ring are idle now
    if (warp < SW_DQ_WARPS)
    {
        pdl_wait();    // Y (and beta * Y) belong to the stream's order
        if (!mbar_wait_bounded(acc_full, 0))
        {
            atomicMax(p.status, (unsigned int)ST_TIMEOUT_FULL);
            *abort_flag = 1;
        }
        const bool good = *abort_flag == 0 && nkb > 0;
        tc_fence_after();
        const unsigned int f = (warp & 3u) * 32 + lane;
        for (unsigned int c0 = (warp >> 2) * 16; c0 < live; c0 += 16 * (SW_DQ_WARPS / 4))
        {
            uint32_t r[16];
            if (good)
            {
                tmem_ld_32x16(tmem_base + (((warp & 3u) * 32u) << 16) + c0, r);
                tmem_ld_wait();
            }
#pragma unroll
            for (int q = 0; q < 16; q++) { part[(c0 + q) * SK_BM + f] = good ? __uint_as_float(r[q]) : 0.f; }
        }
    }
    tc_fence_before();
    cluster_sync_all();

    // ---- sum the slices in slice order; the pair of slice `rank` finishes tokens rank, rank + S, ...; a thread takes four features ----
    if (warp < SW_DQ_WARPS && *abort_flag == 0)
    {
        const unsigned int f = lane * 4, n = n0 + f;
        // four elements of Y at once where they lie side by side.  With an old Y to add, as in a residual, they were taken one by one,
        // two bytes to an access: E4M3 4096 x 4096 at 129 / 301 / 1021 tokens 15.8 / 20.2 / 38.1 -> 14.2 / 18.1 / 32.4 us (14.1 /
        // 17.4 / 29.4 without one), FP4 16.2 / 20.9 / 39.5 -> 14.6 / 18.6 / 33.7.
        const bool whole = g.ldy_n == 1 && n + 4 <= g.N && p.out_f32 != 1u && (g.ldy_m % 4) == 0 && (reinterpret_cast<uintptr_t>(g.Y) & 7u) == 0;
        const float* peer[SW_MAX_SPLIT];
#pragma unroll
        for (int r = 0; r < SW_MAX_SPLIT; r++) { peer[r] = (unsigned int)r < S ? cluster.map_shared_rank(part, 2 * r + half_cta) : part; }
        // All slices' loads of a token are under way before the first is added.  (Two and four tokens per turn were slower, by
        // 2 and by 8 % at 301 tokens: the tiles of a cluster are read by all its CTAs at once.)
        // Without an old Y the turn has none of its instructions: with both in one loop, 301 tokens through a layer's linears took 1 us
        // more, 1021 tokens through 4096 x 4096 (E5M2) 28.5 for 27.6 us.
        auto rows = [&](auto old_y) {
            constexpr bool ADD = decltype(old_y)::value;
            for (unsigned int t = rank + S * warp; t < live; t += S * SW_DQ_WARPS)
            {
                float4 v[SW_MAX_SPLIT];
                uint2 y_old = make_uint2(0u, 0u);
                if (ADD && whole) { y_old = *reinterpret_cast<const uint2*>(g.Y + (long long)(m0 + t) * g.ldy_m + n); }
#pragma unroll
                for (int r = 0; r < SW_MAX_SPLIT; r++)
                {
                    if ((unsigned int)r < S) { v[r] = *reinterpret_cast<const float4*>(peer[r] + t * SK_BM + f); }
                }
                float4 sum = v[0];
#pragma unroll
                for (int r = 1; r < SW_MAX_SPLIT; r++)
                {
                    if ((unsigned int)r < S)
                    {
                        sum.x += v[r].x;
                        sum.y += v[r].y;
                        sum.z += v[r].z;
                        sum.w += v[r].w;
                    }
                }
                float o[4] = { g.alpha * (sum.x * g.post_scale), g.alpha * (sum.y * g.post_scale), g.alpha * (sum.z * g.post_scale), g.alpha * (sum.w * g.post_scale) };
                const long long yi = (long long)(m0 + t) * g.ldy_m + (long long)n * g.ldy_n;
                if (whole)
                {
                    if (ADD)
                    {
                        const float old[4] = { __uint_as_float(y_old.x << 16), __uint_as_float(y_old.x & 0xFFFF0000u), __uint_as_float(y_old.y << 16), __uint_as_float(y_old.y & 0xFFFF0000u) };
#pragma unroll
                        for (int q = 0; q < 4; q++) { o[q] = (p.out_f32 == 2u ? __bfloat162float(__float2bfloat16_rn(o[q])) : o[q]) + g.beta * old[q]; }
                    }
                    *reinterpret_cast<uint2*>(g.Y + yi) = make_uint2(pack_bf16x2(o[0], o[1]), pack_bf16x2(o[2], o[3]));
                    continue;
                }
#pragma unroll
                for (int q = 0; q < 4; q++)
                {
                    if (n + q >= g.N) { continue; }
                    float y_new = o[q];
                    if (p.out_f32 == 1u)
                    {
                        float* y = reinterpret_cast<float*>(g.Y) + yi + q * g.ldy_n;
                        if (ADD) { y_new += g.beta * *y; }
                        *y = y_new;
                    }
                    else
                    {
                        uint16_t* y = g.Y + yi + q * g.ldy_n;
                        if (ADD) { y_new = (p.out_f32 == 2u ? __bfloat162float(__float2bfloat16_rn(y_new)) : y_new) + g.beta * bf16_bits_to_float(*y); }
                        *y = __bfloat16_as_ushort(__float2bfloat16_rn(y_new));
                    }
                }
            }
        };
        if (g.beta != 0.f) { rows(std::true_type{}); }
        else { rows(std::false_type{}); }
    }
    // nobody leaves while a peer may still read its partial tile
    cluster_sync_all();
    tc_fence_after();
    if (warp == SW_DQ_WARPS + 1) { tmem_dealloc_pair(tmem_base, 512); }
}

// ---- host side -----------------------------------------------------------------------------------------
static void sw_configure(cudaLaunchConfig_t* cfg, cudaLaunchAttribute* attr, int w_type, dim3 grid, unsigned int split, cudaStream_t stream, bool pdl)
{
    memset(cfg, 0, sizeof(*cfg));
    cfg->gridDim = grid;
    cfg->blockDim = dim3(SW_THREADS);
    cfg->dynamicSmemBytes = sw_smem_bytes(w_type);
    cfg->stream = stream;
    int na = 0;
    attr[na].id = cudaLaunchAttributeClusterDimension;
    attr[na].val.clusterDim.x = 2 * split;
    attr[na].val.clusterDim.y = 1;
    attr[na].val.clusterDim.z = 1;
    na++;
    if (pdl)
    {
        attr[na].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[na].val.programmaticStreamSerializationAllowed = 1;
        na++;
    }
    cfg->attrs = attr;
    cfg->numAttrs = na;
}

template <int WT, bool SCALED>
static bool sw_prepare(int device)
{
    static std::atomic<bool> attr_set[64];
    if (!attr_set[device].load(std::memory_order_acquire))
    {
        if (cudaFuncSetAttribute(gemm_wq_stream_wide_kernel<WT, SCALED>, cudaFuncAttributeMaxDynamicSharedMemorySize, sw_smem_bytes(WT)) != cudaSuccess) { return false; }
        attr_set[device].store(true, std::memory_order_release);
    }
    return true;
}

// How many clusters of 2 x `split` CTAs the device holds at once (one CTA per SM): what the GPCs leave of 148.  A fact of
// the device, the same for every form of the kernel; asked for once.
static int sw_resident_clusters(unsigned int split, int device)
{
    static std::atomic<int> known[64][SW_MAX_SPLIT + 1];
    int n = known[device][split].load(std::memory_order_acquire);
    if (n == 0)
    {
        cudaLaunchConfig_t cfg;
        cudaLaunchAttribute attr[2];
        sw_configure(&cfg, attr, DT_FP4, dim3(2 * split, 1, 1), split, nullptr, false);
        if (!sw_prepare<DT_FP4, false>(device) || cudaOccupancyMaxActiveClusters(&n, gemm_wq_stream_wide_kernel<DT_FP4, false>, &cfg) != cudaSuccess || n < 1)
        {
            cudaGetLastError();
            return 1;
        }
        known[device][split].store(n, std::memory_order_release);
    }
    return n;
}

struct StreamWidePlan
{
    unsigned int split, token_tiles, chunk, chunks;
    float us;
};

// Token tiles and k slices: the smallest waves x (k blocks per CTA x time per block + the rest of a CTA's life).  Fitted to
// N x K of 1024 x 2048 ... 24576 x 4096, 4096 x 12288, all three weight types, 129 ... 2048 tokens: a 64-k block takes
// 0.30 us (dequantising) up to 272 tokens and 1.1 ns per token above (the UMMAs), launch, first loads and the last barriers
// 5.5 us, reading and adding the accumulator 18 ns per token whatever the slices.
static StreamWidePlan sw_plan(unsigned int pair_tiles, unsigned int M, unsigned int K, int device)
{
    StreamWidePlan best = { 0, 0, 0, 0, 1e30f };
    const unsigned int units = K / SK_SLICE_ELEMS, z0 = (M + SW_MAX_TOKENS - 1) / SW_MAX_TOKENS;
    for (unsigned int z = z0; z <= z0 + z0 / 2 + 1; z++)
    {
        const unsigned int tokens = (M + z - 1) / z;
        const unsigned int chunks = tokens > 256 ? 2 : 1;
        const unsigned int chunk = ((tokens + chunks - 1) / chunks + 15) / 16 * 16;
        const unsigned int width = chunk * chunks, tiles = (M + width - 1) / width;
        for (unsigned int s = 1; s <= (unsigned)SW_MAX_SPLIT && s <= units; s++)
        {
            const unsigned int resident = (unsigned int)sw_resident_clusters(s, device);
            const unsigned int waves = (pair_tiles * tiles + resident - 1) / resident;
            const float block = fmaxf(0.30f, 0.0011f * (float)width);
            const float us = (float)waves * ((float)((units + s - 1) / s * (SK_SLICE_ELEMS / SK_BK)) * block + 5.5f + 0.018f * (float)width);
            if (us < best.us) { best = { s, tiles, chunk, chunks, us }; }
        }
    }
    return best;
}

// Is this kernel the faster one at more than kStreamNarrowTokens tokens?  Against it stands only the 256 features x 512
// tokens pair tile of gemm_prefill_pair.cuh (0.73 us per k block, 3.5 us besides), which dequantises a weight once per 512
// tokens and overlaps nothing less; where that tile has too few tiles to fill the device, its other shapes took 1.2 to 5
// times as long as this kernel (4096 x 12288 at 129 / 301 / 1024 tokens: 123 / 119 / 136 us against 28 / 34 / 75;
// 24576 x 4096 at 301: 108 against 67).  At equal estimates the pair tile measured a few percent faster (2048 tokens:
// 4096 x 12288 143 against 148 us), hence 0.93.
static bool sw_preferred(unsigned int pair_tiles, unsigned int n_total, unsigned int M, unsigned int K, int device, int sm_count)
{
    if (pf_pick_variant(0, n_total, M, K, sm_count) != PFV_PAIR_T512) { return true; }
    const unsigned int tiles = (M + 511) / 512 * ((n_total + 255) / 256), slots = (unsigned)sm_count / 2;
    const float other = (float)((tiles + slots - 1) / slots) * ((float)(K / SK_BK) * 0.73f + 3.5f);
    return sw_plan(pair_tiles, M, K, device).us < 0.93f * other;
}

template <int WT, bool SCALED>
static int launch_stream_wide_t(const void* X, unsigned int ldx, const StreamParams& sp_in, int device, cudaStream_t stream, bool pdl)
{
    StreamWideParams wp;
    memset(&wp, 0, sizeof(wp));
    wp.s = sp_in;
    StreamParams& sp = wp.s;
    unsigned int feature_tiles = 0;
    for (unsigned int j = 0; j < sp.n_seg; j++)
    {
        sp.seg[j].tile0 = feature_tiles;
        feature_tiles += (sp.seg[j].N + 2 * SK_BM - 1) / (2 * SK_BM);
    }
    if (!sw_prepare<WT, SCALED>(device))
    {
        report_launch("gemm_wq_bf16");
        return 1;
    }
    const StreamWidePlan plan = sw_plan(feature_tiles, sp.M, sp.K, device);
    if (feature_tiles == 0 || feature_tiles > 65535u || plan.token_tiles > 65535u || plan.split == 0) { return -2; }
    sp.split = plan.split;
    wp.chunk = plan.chunk;
    wp.chunks = plan.chunks;
    wp.tile_tokens = plan.chunk * plan.chunks;
    wp.x_stages = (unsigned int)SW_X_RING_BYTES / (wp.tile_tokens / 2 * SK_BK * 2);
    wp.x_stages = wp.x_stages > (unsigned)SW_RING ? (unsigned)SW_RING : wp.x_stages;
    wp.keep_weights = plan.token_tiles > 1 ? 1 : 0;
    CUtensorMap tmX;
    StreamWMaps tmW;
    memset(&tmW, 0, sizeof(tmW));
    bool ok = make_map_2d(&tmX, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, X, sp.K, sp.M, (unsigned long long)ldx * 2, SK_BK, wp.chunk / 2, true);
    const unsigned long long kbytes = (WT == DT_FP4) ? sp.K / 2 : sp.K;
    for (unsigned int j = 0; j < sp.n_seg && ok; j++)
    {
        const PrefillSeg& g = sp.seg[j];
        const unsigned long long ldw_bytes = (WT == DT_FP4) ? g.ldw / 2 : g.ldw;
        ok = make_map(&tmW.w[j], CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, g.W, 64, g.N, kbytes / 64, ldw_bytes, SK_BM, SW_RUNS, false, true);
        if (ok && WT == DT_FP4) { ok = make_map(&tmW.s[j], CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, g.blk, 16, g.N, sp.K / 256, g.ldw / 16, SK_BM, SW_RUNS / 2, false); }
    }
    if (!ok) { return -2; }
    cudaLaunchConfig_t cfg;
    cudaLaunchAttribute attr[2];
    sw_configure(&cfg, attr, WT, dim3(2 * sp.split, plan.token_tiles, feature_tiles), sp.split, stream, pdl);
    count_launch();
    if (cudaLaunchKernelEx(&cfg, gemm_wq_stream_wide_kernel<WT, SCALED>, tmX, tmW, wp) != cudaSuccess)
    {
        report_launch("gemm_wq_bf16");
        return 1;
    }
    return 0;
}

// One launch for up to PF_MAX_GROUP linears that share X; arguments as launch_stream.  -2: not taken.
static int launch_stream_wide(int w_type, const GemvParams* items, unsigned int count, int device, cudaStream_t stream, bool pdl)
{
    StreamParams sp;
    bool scaled = false;
    if (!stream_params(w_type, items, count, &sp, &scaled)) { return -2; }
    const void* X = items[0].X;
    const unsigned int ldx = items[0].ldx;
    if (w_type == DT_FP4) { return launch_stream_wide_t<DT_FP4, false>(X, ldx, sp, device, stream, pdl); }
    if (!scaled)
    {
        return w_type == DT_E5M2 ? launch_stream_wide_t<DT_E5M2, false>(X, ldx, sp, device, stream, pdl)
                                 : launch_stream_wide_t<DT_E4M3, false>(X, ldx, sp, device, stream, pdl);
    }
    return w_type == DT_E5M2 ? launch_stream_wide_t<DT_E5M2, true>(X, ldx, sp, device, stream, pdl)
                             : launch_stream_wide_t<DT_E4M3, true>(X, ldx, sp, device, stream, pdl);
}

}    // namespace b200

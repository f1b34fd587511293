// W8A8 linear for two dozen tokens and more: E4M3 weights x E4M3 activations (tcgen05.mma
// kind::f8f6f4), a CTA per 128 output features and k slice.
//
// At these sizes the weights are the work: 4096 x 4096 is 16 MB, 2.6 us of HBM, whatever the 64 tokens cost.  The CTA pairs of
// gemm_w8a8_pair.cuh (256 features per pair, the whole k range) put that linear on 32 of 148 SMs.  Here:
//   * a tile is 128 features x 64 or 128 tokens; up to four k slices run as ONE cluster, so that the CTAs that fit the GPU at
//     once share the k range, and the next kernel's weights are already on their way (programmatic launch) while the quantiser of
//     its activations runs: weights and activations have a copying lane each, and only the latter waits for the stream;
//   * a stage is one 128-k block of both operands as they lie in memory (128-byte swizzle), 16 KB of weights; four stages and two
//     CTAs per SM (64 tokens), or six and one (128 tokens), keep 96 to 128 KB of weights in flight per SM;
//   * the result does not depend on how many CTAs share the k range: k is always cut into WS_SLICES slices, each summed from zero
//     in tensor-memory columns of its own, and the slices are added as (s0 + s1) + (s2 + s3), inside a CTA or through
//     distributed shared memory.  A group of linears therefore gives the bits of the separate calls.
// Measured (dynamic scale, quantiser included, a chain of distinct weights; pairs -> slices, us): 4096 x 4096 at 33 / 64 tokens
// 16.3 -> 11.1, 16.7 -> 13.1; 24576 x 4096 28.6 -> 24.5, 28.7 -> 25.1; 4096 x 12288 31.8 -> 18.6, 33.5 -> 20.8, at 256 tokens
// 43.7 -> 31.4; the four calls of a Qwen3-8B layer at 64 tokens 124 -> 78.
// Every wait is bounded; a CTA whose wait ran out raises the status word, still meets its cluster, frees its columns and returns.
#pragma once

#include "gemm_w8a8_pair.cuh"

namespace b200
{

constexpr int WS_SLICES = 4;
constexpr int WS_WARPS = 8;    // 0 weights, 1 activations, 2 MMA; all eight read the accumulators afterwards
constexpr int WS_THREADS = 32 * WS_WARPS;
__host__ __device__ constexpr int ws_stages(int bn) { return bn == 64 ? 4 : 6; }
__host__ __device__ constexpr int ws_stage_bytes(int bn) { return WP_TILE_BYTES + bn * WP_BK; }
__host__ __device__ constexpr int ws_smem_bytes(int bn) { return SK_HEADER_BYTES + ws_stages(bn) * ws_stage_bytes(bn) + 1024; }

template <int BN>
__global__ void __launch_bounds__(WS_THREADS, BN == 64 ? 2 : 1)
    gemm_w8a8_split_kernel(const __grid_constant__ CUtensorMap tmX, const __grid_constant__ StreamWMaps tmW, const NativeParams p, const unsigned int split)
{
    namespace cg = cooperative_groups;
    constexpr int NS = ws_stages(BN);
    constexpr int STAGE = ws_stage_bytes(BN);
    constexpr int TMEM_COLS = WS_SLICES * BN;
    static_assert(TMEM_COLS <= 512 && (TMEM_COLS & (TMEM_COLS - 1)) == 0, "an allocation is a power of two");
    static_assert(BN * SK_BM * 4 <= NS * STAGE, "the partial tile reuses the stages");
    static_assert(NS <= 8, "barrier arrays hold eight stages");
    extern __shared__ unsigned char ws_smem_raw[];
    unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(ws_smem_raw) + 1023) & ~(uintptr_t)1023);
    uint64_t* full = reinterpret_cast<uint64_t*>(smem);    // [8]: both operands of the stage have landed
    uint64_t* empty = full + 8;                            // [8]: its UMMAs are complete
    uint64_t* acc_full = empty + 8;
    uint32_t* tmem_base_slot = reinterpret_cast<uint32_t*>(acc_full + 1);
    volatile unsigned int* abort_flag = reinterpret_cast<volatile unsigned int*>(tmem_base_slot + 1);
    unsigned char* stages = smem + SK_HEADER_BYTES;

    cg::cluster_group cluster = cg::this_cluster();
    const unsigned int rank = split > 1 ? cluster.block_rank() : 0u;
    const unsigned int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    unsigned int si = 0;
    if (p.n_seg > 1 && blockIdx.y >= p.seg[1].tile0) { si = 1; }
    if (p.n_seg > 2 && blockIdx.y >= p.seg[2].tile0) { si = 2; }
    const PrefillSeg& g = p.seg[si];
    const unsigned int n0 = (blockIdx.y - g.tile0) * SK_BM;
    const unsigned int m0 = blockIdx.z * BN;
    const unsigned int tile_tokens = min((unsigned int)BN, p.M - m0);
    const unsigned int own = WS_SLICES / split;    // slices of this CTA
    auto slice_begin = [&](unsigned int s) { return (unsigned int)(((unsigned long long)p.nkb * s) / WS_SLICES); };
    const unsigned int kb_begin = slice_begin(rank * own), kb_end = slice_begin((rank + 1) * own);

    if (threadIdx.x == 0)
    {
        for (int s = 0; s < NS; s++)
        {
            mbar_init(full + s, 2);
            mbar_init(empty + s, 1);
        }
        mbar_init(acc_full, 1);
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 2) { tmem_alloc(tmem_base_slot, TMEM_COLS); }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_base_slot;
    pdl_launch_dependents();

    if (warp < 2)
    {
        // =========================== TMA lanes: warp 0 the weights, warp 1 the activations ===========================
        if (lane == 0)
        {
            if (warp == 1) { pdl_wait(); }    // the activations are the quantiser's output
            const uint64_t pol = l2_policy_evict_first();
            unsigned int issued = kb_begin;
            bool ok = true;
            for (unsigned int kb = kb_begin; kb < kb_end; kb++)
            {
                const unsigned int i = kb - kb_begin, s = i % NS;
                if (i == (unsigned int)NS) { pdl_wait(); }    // from here on the ring waits for products: see the MMA warp
                if (i >= (unsigned int)NS && (*abort_flag != 0 || !mbar_wait_bounded(empty + s, ((i / NS) - 1u) & 1u)))
                {
                    ok = false;
                    atomicMax(p.status, (unsigned int)ST_TIMEOUT_EMPTY);
                    *abort_flag = 1;
                    break;
                }
                unsigned char* st = stages + s * STAGE;
                if (warp == 0)
                {
                    mbar_expect_tx(full + s, WP_TILE_BYTES);
                    // several token tiles read a weight tile: it stays in L2 then
                    if (gridDim.z == 1) { tma_load_2d_hint(st, &tmW.w[si], (int)(kb * WP_BK), (int)n0, full + s, pol); }
                    else { tma_load_2d(st, &tmW.w[si], (int)(kb * WP_BK), (int)n0, full + s); }
                }
                else
                {
                    mbar_expect_tx(full + s, BN * WP_BK);
                    tma_load_2d(st + WP_TILE_BYTES, &tmX, (int)(kb * WP_BK), (int)m0, full + s);
                }
                mbar_arrive(full + s);
                issued = kb + 1;
            }
            if (!ok)
            {
                // wait (bounded) for the copies in flight before the CTA may leave
                const unsigned int n = issued - kb_begin, first = n > (unsigned int)NS ? n - NS : 0;
                for (unsigned int i = first; i < n; i++)
                {
                    const unsigned long long t0 = global_timer_ns();
                    while (!mbar_try_wait(full + (i % NS), (i / NS) & 1u) && global_timer_ns() - t0 < 100000ull) {}
                }
            }
        }
        __syncwarp();
    }
    else if (warp == 2)
    {
        // =========================== MMA warp ===========================
        pdl_wait();    // the first stage needs the activations: the limit on the waits below does not count the kernels before this one
        bool ok = true;
        const uint32_t idesc = umma_idesc_f8(false, false, SK_BM, (tile_tokens + 15u) & ~15u);
        for (unsigned int l = 0; l < own && ok; l++)
        {
            const unsigned int b = slice_begin(rank * own + l), e = slice_begin(rank * own + l + 1);
            for (unsigned int kb = b; kb < e && ok; kb++)
            {
                const unsigned int i = kb - kb_begin, s = i % NS;
                if (*abort_flag != 0 || !mbar_wait_bounded(full + s, (i / NS) & 1u))
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
                const uint32_t a_addr = smem_u32(stages + s * STAGE), b_addr = a_addr + WP_TILE_BYTES;
                if (elect_one())
                {
#pragma unroll
                    for (int k = 0; k < WP_BK / 32; k++)
                    {
                        umma_f8(tmem_base + l * BN, umma_desc_kmajor_sw128(a_addr + k * 32), umma_desc_kmajor_sw128(b_addr + k * 32), idesc,
                            kb != b || k != 0 ? 1u : 0u);
                    }
                    umma_commit(empty + s);
                }
                __syncwarp();
            }
        }
        __syncwarp();
        if (elect_one()) { umma_commit(acc_full); }    // also after an abort: no UMMA reads the stages any more once it completes
        __syncwarp();
    }

    // ---- this CTA's slices: TMEM -> shared memory [tokens][128 features] (the stages are idle once acc_full has completed) ----
    float* part = reinterpret_cast<float*>(stages);
    pdl_wait();    // Y, and the activations' multiplier, belong to the stream's order
    if (!mbar_wait_bounded(acc_full, 0))
    {
        atomicMax(p.status, (unsigned int)ST_TIMEOUT_FULL);
        *abort_flag = 1;
    }
    const bool good = *abort_flag == 0;
    tc_fence_after();
    {
        const unsigned int quarter = warp & 3u, f = quarter * 32 + lane;
        for (unsigned int c = (warp >> 2) * (BN / 2); c < ((warp >> 2) + 1) * (BN / 2) && c < tile_tokens; c += 16)
        {
            float sum[2][16];    // s0 + s1 (or the only one), s2 + s3
#pragma unroll
            for (unsigned int l = 0; l < (unsigned int)WS_SLICES; l++)
            {
                if (l >= own) { break; }
                uint32_t r[16];
                const bool any = good && slice_begin(rank * own + l) < slice_begin(rank * own + l + 1);
                if (any)
                {
                    tmem_ld_32x16(tmem_base + ((quarter * 32u) << 16) + l * BN + c, r);
                    tmem_ld_wait();
                }
#pragma unroll
                for (int q = 0; q < 16; q++)
                {
                    const float v = any ? __uint_as_float(r[q]) : 0.f;
                    sum[l >> 1][q] = (l & 1u) ? sum[l >> 1][q] + v : v;
                }
            }
#pragma unroll
            for (int q = 0; q < 16; q++) { part[(c + q) * SK_BM + f] = own > 2 ? sum[0][q] + sum[1][q] : sum[0][q]; }
        }
    }
    tc_fence_before();
    if (split > 1) { cluster.sync(); }
    else { __syncthreads(); }

    // ---- the cluster's sums, in the same order; CTA `rank` finishes tokens rank, rank + split, ...: a warp per token, four features per lane ----
    if (*abort_flag == 0)
    {
        const float4* peer[WS_SLICES];
#pragma unroll
        for (int r = 0; r < WS_SLICES; r++)
        {
            peer[r] = reinterpret_cast<const float4*>(split > 1 && (unsigned int)r < split ? cluster.map_shared_rank(part, r) : part);
        }
        const float act_inv = p.inv_scale != nullptr ? *p.inv_scale : p.act_inv;
        const unsigned int n = n0 + 4 * lane;
        const bool wide = (p.out_f32 == 0u || p.out_f32 == 2u) && g.beta == 0.f && g.ldy_n == 1 && (g.ldy_m & 3) == 0
            && (reinterpret_cast<uintptr_t>(g.Y) & 7u) == 0 && n + 3 < g.N;
        for (unsigned int t = rank + split * warp; t < tile_tokens; t += split * WS_WARPS)
        {
            float4 v = peer[0][t * (SK_BM / 4) + lane];
            if (split > 1)
            {
                const float4 w = peer[1][t * (SK_BM / 4) + lane];
                v = make_float4(v.x + w.x, v.y + w.y, v.z + w.z, v.w + w.w);
            }
            if (split > 2)
            {
                const float4 a = peer[2][t * (SK_BM / 4) + lane], b = peer[3][t * (SK_BM / 4) + lane];
                v = make_float4(v.x + (a.x + b.x), v.y + (a.y + b.y), v.z + (a.z + b.z), v.w + (a.w + b.w));
            }
            const float s[4] = { v.x, v.y, v.z, v.w };
            const long long row = (long long)(m0 + t) * g.ldy_m;
            if (wide)
            {
                uint32_t o[2];
#pragma unroll
                for (int q = 0; q < 2; q++)
                {
                    const uint32_t lo = __bfloat16_as_ushort(__float2bfloat16_rn(g.alpha * ((s[2 * q] * act_inv) * g.post_scale)));
                    const uint32_t hi = __bfloat16_as_ushort(__float2bfloat16_rn(g.alpha * ((s[2 * q + 1] * act_inv) * g.post_scale)));
                    o[q] = lo | (hi << 16);
                }
                *reinterpret_cast<uint2*>(g.Y + row + n) = make_uint2(o[0], o[1]);
                continue;
            }
#pragma unroll
            for (int q = 0; q < 4; q++)
            {
                if (n + q >= g.N) { continue; }
                const long long yi = row + (long long)(n + q) * g.ldy_n;
                float o = g.alpha * ((s[q] * act_inv) * g.post_scale);
                if (p.out_f32 == 1u)
                {
                    float* y = reinterpret_cast<float*>(g.Y) + yi;
                    if (g.beta != 0.f) { o += g.beta * *y; }
                    *y = o;
                }
                else if (p.out_f32 == 3u) { reinterpret_cast<uint8_t*>(g.Y)[yi] = float_to_e4m3(__bfloat162float(__float2bfloat16_rn(o)), 1.0f); }
                else
                {
                    uint16_t* y = g.Y + yi;
                    if (g.beta != 0.f) { o = (p.out_f32 == 2u ? __bfloat162float(__float2bfloat16_rn(o)) : o) + g.beta * bf16_bits_to_float(*y); }
                    *y = __bfloat16_as_ushort(__float2bfloat16_rn(o));
                }
            }
        }
    }
    // nobody leaves while a peer may still read its partial tile
    if (split > 1) { cluster.sync(); }
    else { __syncthreads(); }
    tc_fence_after();
    if (warp == 2) { tmem_dealloc(tmem_base, TMEM_COLS); }
}

template <int BN>
static int launch_w8a8_split_bn(const CUtensorMap& tmX, const StreamWMaps& tmW, const NativeParams& np, unsigned int split, int device, cudaStream_t stream,
    bool pdl)
{
    auto kernel = gemm_w8a8_split_kernel<BN>;
    static std::atomic<bool> attr_set[64];
    if (!attr_set[device].load(std::memory_order_acquire))
    {
        if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, ws_smem_bytes(BN)) != cudaSuccess)
        {
            report_launch("gemm_w8a8_bf16");
            return 1;
        }
        attr_set[device].store(true, std::memory_order_release);
    }
    cudaLaunchConfig_t cfg;
    memset(&cfg, 0, sizeof(cfg));
    cfg.gridDim = dim3(split, np.tiles, (np.M + BN - 1) / BN);
    cfg.blockDim = dim3(WS_THREADS);
    cfg.dynamicSmemBytes = ws_smem_bytes(BN);
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    int na = 0;
    if (split > 1)
    {
        attr[na].id = cudaLaunchAttributeClusterDimension;
        attr[na].val.clusterDim.x = split;
        attr[na].val.clusterDim.y = attr[na].val.clusterDim.z = 1;
        na++;
    }
    if (pdl)
    {
        attr[na].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[na].val.programmaticStreamSerializationAllowed = 1;
        na++;
    }
    cfg.attrs = attr;
    cfg.numAttrs = na;
    count_launch();
    if (cudaLaunchKernelEx(&cfg, kernel, tmX, tmW, np, split) != cudaSuccess)
    {
        report_launch("gemm_w8a8_bf16");
        return 1;
    }
    return 0;
}

// The launch behind the quantiser.  np as for launch_w8a8_pair, with `tiles` and every member's tile0 in tiles of 128 features.
// pdl: the launch before it on the stream is the quantiser, or the caller allows its calls to overlap.  -2: not taken.
static int launch_w8a8_split(const NativeParams& np, const W8A8Member* mem, const uint8_t* Q, unsigned int ldq, int device, int sm_count, cudaStream_t stream,
    bool pdl)
{
    const unsigned int bn = np.M <= 64 ? 64u : 128u;
    const unsigned int token_tiles = (np.M + bn - 1) / bn;
    if (np.tiles == 0 || np.tiles > 65535u || token_tiles > 65535u) { return -2; }
    CUtensorMap tmX;
    StreamWMaps tmW;
    memset(&tmW, 0, sizeof(tmW));
    bool ok = make_map_2d(&tmX, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, Q, np.K, np.M, ldq, WP_BK, bn, true);
    for (unsigned int j = 0; j < (unsigned int)PF_MAX_GROUP && ok; j++)
    {
        const W8A8Member& m = mem[j < np.n_seg ? j : 0];
        ok = make_map_2d(&tmW.w[j], CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, m.W, np.K, m.N_out, m.ldw, WP_BK, SK_BM, true);
    }
    if (!ok) { return -2; }
    // as many CTAs per tile as fit the GPU at once, a tenth left for SMs whose cluster slots do not divide evenly
    const unsigned long long slots = (bn == 64 ? 2ull : 1ull) * (unsigned)sm_count * 9ull / 10ull;
    unsigned int split = 1;
    while (2 * split <= (unsigned int)WS_SLICES && 2ull * split * np.tiles * token_tiles <= slots && 2 * split <= np.nkb) { split *= 2; }
    return bn == 64 ? launch_w8a8_split_bn<64>(tmX, tmW, np, split, device, stream, pdl) : launch_w8a8_split_bn<128>(tmX, tmW, np, split, device, stream, pdl);
}

}    // namespace b200

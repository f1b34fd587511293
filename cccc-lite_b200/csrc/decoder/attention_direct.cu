// BF16 attention of few query rows (decoding), HBM-bound: keys and values go from global memory straight into the
// fragments of mma.m16n8k16, no shared memory in between.
//
// A warp holds up to 8 (or 16) query rows and walks 16-key tiles.  Scores: a lane reads 32 bytes of key row lane / 4, the
// four lanes of a row 64 consecutive elements; the order of the elements inside the product is permuted, alike for
// the queries.  Values: lane (g, t) reads the columns g * DV / 8 ... of the rows 2t, 2t + 1, 2t + 8, 2t + 9, so that a warp
// reads whole rows and a register pair becomes a fragment with one byte permute; which columns a fragment's n stands
// for is permuted in turn, and undone when the result is stored.  The next tile's keys are requested as soon as the scores
// are out, its values as soon as the value product is.  Softmax weights enter the value product as the sum of two BF16 numbers.
// Decoding steps (one token per sequence) are fused: the CTA whose split holds the new position brings its key to unit
// RMS, mixes its value and appends both (and takes them from shared memory itself); every CTA brings its own queries to unit RMS.
// The splits of a unit are one cluster: each CTA stores its statistics and its share of everyone's outputs into the others' shared
// memory, one barrier, and the shares are summed where they lie.  (Partial results through global memory, summed by the last CTA
// to arrive at a counter, took four more round trips to L2 of a chain that is all latency at a few hundred rows: 8 sequences
// of 250 rows, 4 kv heads, 17 us behind the projections, now 8.4.)
#include <atomic>
#include <cooperative_groups.h>
#include <type_traits>

#include "attention_mma.cuh"

namespace b200
{

__device__ __forceinline__ void ldg32(const void* p, uint32_t (&r)[8], bool ok)
{
#pragma unroll
    for (int i = 0; i < 8; i++) { r[i] = 0u; }
    if (ok)
    {
        asm volatile("ld.global.v8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                     : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                     : "l"(p)
                     : "memory");
    }
}
__device__ __forceinline__ void ldg16(const void* p, uint32_t (&r)[4], bool ok)
{
#pragma unroll
    for (int i = 0; i < 4; i++) { r[i] = 0u; }
    if (ok) { asm volatile("ld.global.v4.b32 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "l"(p) : "memory"); }
}

// rows 8-15 of the fragment do not exist: their inputs and results are zero
__device__ __forceinline__ void mma_bf16_top(float& c0, float& c1, uint32_t a0, uint32_t a2, uint32_t b0, uint32_t b1)
{
    [[maybe_unused]] float d2, d3;
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%5}, {%7,%8}, {%0,%1,%9,%9};"
        : "+f"(c0), "+f"(c1), "=f"(d2), "=f"(d3)
        : "r"(a0), "r"(0u), "r"(a2), "r"(b0), "r"(b1), "f"(0.f));
}

constexpr unsigned int kDirectSplits = 16;    // one cluster

template <int DK, int DV, int RT>
struct DirectMeet
{
    float om[AS_WARPS][RT * DV];
    float ml[AS_WARPS][RT][2];                 // a warp's maximum (log2) and sum of every row
    float recv_ml[kDirectSplits][RT][2];       // a split's
    float recv[RT * DV + kDirectSplits];       // [split][outputs that this CTA finishes]
    __nv_bfloat16 kn[DK], vn[DV];              // the new row (fused)
};

// grid (splits, Hkv * row_tiles, entries), clusters along x
template <int DK, int DV, int NR>    // NR: row groups of eight (1 or 2)
__global__ void __launch_bounds__(32 * AS_WARPS, NR == 1 && DK + DV < 256 ? 3 : 2) attention_direct_kernel(const AttnParams p)
{
    constexpr int RT = 8 * NR, KB = DK / 64, C = DV / 8, VR = C / 2;    // VR: registers of a value row per lane
    __shared__ __align__(16) DirectMeet<DK, DV, RT> meet;
    cooperative_groups::cluster_group cluster = cooperative_groups::this_cluster();
    grid_dependency_launch();
    grid_dependency_wait();
    const unsigned int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    const unsigned int split = blockIdx.x, kvh = blockIdx.y % p.Hkv, rt = blockIdx.y / p.Hkv, e = p.e0 + blockIdx.z;
    const unsigned int n = (unsigned int)p.n[e], start = (unsigned int)p.start[e], pos = (unsigned int)p.pos[e], r0 = rt * RT;
    const unsigned int rows = n * p.G;
    if (r0 >= rows) { return; }    // the whole cluster
    asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");    // met before the first store into a peer
    const __nv_bfloat16* qkvg = (const __nv_bfloat16*)p.qkvg;
    const size_t seq = ((size_t)p.slot[e] * p.Hkv + kvh) * p.T_max;
    __nv_bfloat16* K = (__nv_bfloat16*)p.k_cache + seq * p.k_ld;
    __nv_bfloat16* V = (__nv_bfloat16*)p.v_cache + seq * p.v_ld;
    const unsigned int last_row = min(r0 + RT - 1u, rows - 1);
    const unsigned int T = min(pos + last_row / p.G + 1, p.T_max);
    const unsigned int first_lim = pos + r0 / p.G + 1, last_low = first_key(p, e, pos + last_row / p.G + 1);
    const unsigned int begin = first_key(p, e, first_lim) / 16;
    const unsigned int tiles = (T + 15) / 16, per = (tiles - begin + p.splits - 1) / p.splits;
    const unsigned int tile0 = min(begin + split * per, tiles), tile1 = min(tile0 + per, tiles);

    const bool owner = p.fused && pos < p.T_max && pos / 16 >= tile0 && pos / 16 < tile1;
    uint32_t k[2][KB][8], v[4][VR];
    auto load_k = [&](unsigned int tile, unsigned int skip) {
#pragma unroll
        for (int i = 0; i < 2; i++)
        {
            const unsigned int key = tile * 16 + i * 8 + g;
#pragma unroll
            for (int b = 0; b < KB; b++)
            {
                const unsigned int d = b * 64 + t * 16;
                ldg32(K + (size_t)key * p.k_ld + d, k[i][b], tile < tile1 && key < T && d < p.k_ld && key != skip);
            }
        }
    };
    auto load_v = [&](unsigned int tile, unsigned int skip) {
#pragma unroll
        for (int i = 0; i < 4; i++)
        {
            const unsigned int key = tile * 16 + 2 * t + (i & 1) + (i >> 1) * 8, d = g * C;
            const bool ok = tile < tile1 && key < T && d < p.v_ld && key != skip;
            if constexpr (VR == 8) { ldg32(V + (size_t)key * p.v_ld + d, v[i], ok); }
            else { ldg16(V + (size_t)key * p.v_ld + d, v[i], ok); }
        }
    };
    // Two tiles ahead of the registers, whole lines on their way to L2.
    auto prefetch = [&](unsigned int tile) {
        if (tile < tile1)
        {
            const unsigned int kl = p.k_ld * 32, vl = p.v_ld * 32;    // bytes of a tile
            const char* kp = reinterpret_cast<const char*>(K + (size_t)tile * 16 * p.k_ld) + lane * 128;
            const char* vp = reinterpret_cast<const char*>(V + (size_t)tile * 16 * p.v_ld) + lane * 128;
            if (lane * 128 < kl && (tile + 1) * 16 <= T) { asm volatile("prefetch.global.L2 [%0];" ::"l"(kp)); }
            if (lane * 128 < vl && (tile + 1) * 16 <= T) { asm volatile("prefetch.global.L2 [%0];" ::"l"(vp)); }
        }
    };
    // the step's own row is in the cache only after the append below: a first tile takes it from shared memory
    load_k(tile0 + warp, owner ? pos : 0xFFFFFFFFu);
    load_v(tile0 + warp, owner ? pos : 0xFFFFFFFFu);
    prefetch(tile0 + warp + AS_WARPS);
    prefetch(tile0 + warp + 2 * AS_WARPS);
    const bool wide_q = (p.dim % 16) == 0 && (p.q_ld % 16) == 0;
    auto q_row = [&](unsigned int r) { return qkvg + (size_t)(start + r / p.G) * p.ld + (size_t)(kvh * p.G + r % p.G) * p.q_ld; };
    uint32_t raw[NR][KB][8];
#pragma unroll
    for (int h = 0; h < NR; h++)
    {
        const unsigned int r = r0 + g + 8 * h;
#pragma unroll
        for (int b = 0; b < KB; b++) { ldg32(q_row(r < rows ? r : 0) + b * 64 + t * 16, raw[h][b], wide_q && r < rows && b * 64 + t * 16 < p.dim); }
    }
    // (every row tile of the unit writes the same values)
    if (owner)
    {
        const __nv_bfloat16* x = qkvg + (size_t)start * p.ld;
        if (warp == 0)
        {
            const __nv_bfloat16* src = x + p.k_off + (size_t)kvh * p.dim;
            float inv = 1.f;
            if (p.qk_norm)
            {
                float sq = 0.f;
                for (unsigned int d = lane; d < p.dim; d += 32)
                {
                    const float v = __bfloat162float(src[d]);
                    sq += v * v;
                }
                inv = 1.0f / sqrtf(warp_sum(sq) / (float)p.dim + p.eps);
            }
            for (unsigned int d = lane; d < DK; d += 32)
            {
                const __nv_bfloat16 x = __float2bfloat16_rn(d < p.dim ? __bfloat162float(src[d]) * inv : 0.f);
                meet.kn[d] = x;
                if (d < p.dim) { K[(size_t)pos * p.k_ld + d] = x; }
            }
        }
        else if (warp == 1)
        {
            const __nv_bfloat16* src = x + p.v_off + (size_t)kvh * p.vdim;
            __nv_bfloat16* first = p.v_mix ? (__nv_bfloat16*)p.v_first + (size_t)start * p.v_first_ld + (size_t)kvh * p.vdim : nullptr;
            for (unsigned int d = lane; d < DV; d += 32)
            {
                float v = d < p.vdim ? __bfloat162float(src[d]) : 0.f;
                if (d < p.vdim && p.v_mix == 1) { first[d] = src[d]; }
                else if (d < p.vdim && p.v_mix == 2) { v = (1.0f - p.lambda) * v + p.lambda * __bfloat162float(first[d]); }
                const __nv_bfloat16 x = __float2bfloat16_rn(v);
                meet.vn[d] = x;
                if (d < p.vdim) { V[(size_t)pos * p.v_ld + d] = x; }
            }
        }
        __syncthreads();
    }

    if (owner && tile0 + warp == pos / 16)
    {
        const unsigned int at = pos % 16;
#pragma unroll
        for (int i = 0; i < 2; i++)
        {
            if (at == i * 8 + g)
            {
#pragma unroll
                for (int b = 0; b < KB; b++)
                {
#pragma unroll
                    for (int x = 0; x < 8; x++) { k[i][b][x] = reinterpret_cast<const uint32_t*>(meet.kn + b * 64 + t * 16)[x]; }
                }
            }
        }
#pragma unroll
        for (int i = 0; i < 4; i++)
        {
            if (at == 2 * t + (i & 1) + (i >> 1) * 8)
            {
#pragma unroll
                for (int x = 0; x < VR; x++) { v[i][x] = reinterpret_cast<const uint32_t*>(meet.vn + g * C)[x]; }
            }
        }
    }

    // queries: the same permuted element order as the keys
    uint32_t q[NR][KB][8];
    unsigned int low[NR], lim[NR];
#pragma unroll
    for (int h = 0; h < NR; h++)
    {
        const unsigned int r = r0 + g + 8 * h;
        const bool ok = r < rows;
        const __nv_bfloat16* src = q_row(ok ? r : 0);
        low[h] = first_key(p, e, pos + r / p.G + 1);
        lim[h] = min(pos + r / p.G + 1, T);
        float f[KB][16], sq = 0.f;
#pragma unroll
        for (int b = 0; b < KB; b++)
        {
            const unsigned int d0 = b * 64 + t * 16;
            if (wide_q)
            {
#pragma unroll
                for (int j = 0; j < 8; j++)
                {
                    f[b][2 * j] = __uint_as_float(raw[h][b][j] << 16);
                    f[b][2 * j + 1] = __uint_as_float(raw[h][b][j] & 0xFFFF0000u);
                }
            }
            else
            {
#pragma unroll
                for (int j = 0; j < 16; j++) { f[b][j] = ok && d0 + j < p.dim ? __bfloat162float(src[d0 + j]) : 0.f; }
            }
#pragma unroll
            for (int j = 0; j < 16; j++) { sq += f[b][j] * f[b][j]; }
        }
        float inv = 1.f;
        if (p.fused && p.qk_norm)
        {
            sq += __shfl_xor_sync(0xFFFFFFFFu, sq, 1);
            sq += __shfl_xor_sync(0xFFFFFFFFu, sq, 2);
            inv = 1.0f / sqrtf(sq / (float)p.dim + p.eps);
        }
#pragma unroll
        for (int b = 0; b < KB; b++)
        {
#pragma unroll
            for (int j = 0; j < 8; j++) { q[h][b][j] = pack_bf16x2(f[b][2 * j] * inv, f[b][2 * j + 1] * inv); }
        }
    }

    float o[C][2 * NR], m[NR], l[NR];
#pragma unroll
    for (int h = 0; h < NR; h++)
    {
        m[h] = -INFINITY;
        l[h] = 0.f;
    }
#pragma unroll
    for (int j = 0; j < C; j++)
    {
#pragma unroll
        for (int i = 0; i < 2 * NR; i++) { o[j][i] = 0.f; }
    }
    const float scale2 = p.scale * 1.44269504088896341f;
    for (unsigned int tile = tile0 + warp; tile < tile1; tile += AS_WARPS)
    {
        float s[2][2 * NR];
#pragma unroll
        for (int i = 0; i < 2; i++)
        {
#pragma unroll
            for (int j = 0; j < 2 * NR; j++) { s[i][j] = 0.f; }
#pragma unroll
            for (int b = 0; b < KB; b++)
            {
#pragma unroll
                for (int x = 0; x < 4; x++)
                {
                    if constexpr (NR == 1) { mma_bf16_top(s[i][0], s[i][1], q[0][b][2 * x], q[0][b][2 * x + 1], k[i][b][2 * x], k[i][b][2 * x + 1]); }
                    else
                    {
                        mma_bf16_16816(s[i], q[0][b][2 * x], q[NR - 1][b][2 * x], q[0][b][2 * x + 1], q[NR - 1][b][2 * x + 1], k[i][b][2 * x],
                            k[i][b][2 * x + 1]);
                    }
                }
            }
        }
        load_k(tile + AS_WARPS, 0xFFFFFFFFu);
        prefetch(tile + 3 * AS_WARPS);
        const bool masked = (tile + 1) * 16 > first_lim || tile * 16 < last_low;
        uint32_t hi[2 * NR], lo[2 * NR];    // [key half][row group]
#pragma unroll
        for (int h = 0; h < NR; h++)
        {
            float mx = -INFINITY;
#pragma unroll
            for (int i = 0; i < 2; i++)
            {
#pragma unroll
                for (int j = 0; j < 2; j++)
                {
                    float& z = s[i][2 * h + j];
                    z *= scale2;
                    const unsigned int key = tile * 16 + i * 8 + 2 * t + j;
                    if (masked && (key < low[h] || key >= lim[h])) { z = -INFINITY; }
                    mx = fmaxf(mx, z);
                }
            }
            mx = fmaxf(mx, __shfl_xor_sync(0xFFFFFFFFu, mx, 1));
            mx = fmaxf(mx, __shfl_xor_sync(0xFFFFFFFFu, mx, 2));
            const float mn = fmaxf(m[h], mx), base = mn == -INFINITY ? 0.f : mn;
            if (__any_sync(0xFFFFFFFFu, mn > m[h]))
            {
                const float c = exp2f(m[h] - base);
                m[h] = mn;
                l[h] *= c;
#pragma unroll
                for (int j = 0; j < C; j++)
                {
                    o[j][2 * h] *= c;
                    o[j][2 * h + 1] *= c;
                }
            }
#pragma unroll
            for (int i = 0; i < 2; i++)
            {
                const float p0 = exp2f(s[i][2 * h] - base), p1 = exp2f(s[i][2 * h + 1] - base);
                l[h] += p0 + p1;
                const uint32_t u = pack_bf16x2(p0, p1);
                hi[i * NR + h] = u;
                lo[i * NR + h] = pack_bf16x2(p0 - __uint_as_float(u << 16), p1 - __uint_as_float(u & 0xFFFF0000u));
            }
        }
#pragma unroll
        for (int j = 0; j < C; j++)
        {
            const uint32_t sel = (j & 1) ? 0x7632u : 0x5410u;
            const uint32_t b0 = prmt(v[0][j / 2], v[1][j / 2], sel), b1 = prmt(v[2][j / 2], v[3][j / 2], sel);
            if constexpr (NR == 1)
            {
                mma_bf16_top(o[j][0], o[j][1], hi[0], hi[1], b0, b1);
                mma_bf16_top(o[j][0], o[j][1], lo[0], lo[1], b0, b1);
            }
            else
            {
                mma_bf16_16816(o[j], hi[0], hi[NR - 1], hi[NR], hi[2 * NR - 1], b0, b1);
                mma_bf16_16816(o[j], lo[0], lo[NR - 1], lo[NR], lo[2 * NR - 1], b0, b1);
            }
        }
        load_v(tile + AS_WARPS, 0xFFFFFFFFu);
    }
    // n index 2t (+ 1) of fragment j is column (2t (+ 1)) * C + j
#pragma unroll
    for (int h = 0; h < NR; h++)
    {
        l[h] += __shfl_xor_sync(0xFFFFFFFFu, l[h], 1);
        l[h] += __shfl_xor_sync(0xFFFFFFFFu, l[h], 2);
        float* dst = meet.om[warp] + (g + 8 * h) * DV + 2 * t * C;
#pragma unroll
        for (int j = 0; j < C; j++)
        {
            dst[j] = o[j][2 * h];
            dst[C + j] = o[j][2 * h + 1];
        }
        if (t == 0)
        {
            meet.ml[warp][g + 8 * h][0] = m[h];
            meet.ml[warp][g + 8 * h][1] = l[h];
        }
    }
    __syncthreads();

    // ---- warps -> CTA -> the CTA of the cluster that finishes the output ----
    const unsigned int tid = threadIdx.x, S = p.splits, live = min((unsigned int)RT, rows - r0), outputs = live * p.vdim, share = (outputs + S - 1) / S;
    auto top = [](const float (*ml)[RT][2], unsigned int n, unsigned int r) {
        float m = -INFINITY;
        for (unsigned int i = 0; i < n; i++) { m = fmaxf(m, ml[i][r][0]); }
        return m;
    };
    asm volatile("barrier.cluster.wait.aligned;" ::: "memory");    // every CTA of the cluster runs
    for (unsigned int i = tid; i < live * S; i += 32 * AS_WARPS)
    {
        const unsigned int r = i % live;
        const float mr = top(meet.ml, AS_WARPS, r), base = mr == -INFINITY ? 0.f : mr;
        float lr = 0.f;
#pragma unroll
        for (int w = 0; w < AS_WARPS; w++) { lr += exp2f(meet.ml[w][r][0] - base) * meet.ml[w][r][1]; }
        float* to = cluster.map_shared_rank(&meet.recv_ml[split][r][0], i / live);
        to[0] = mr;
        to[1] = lr;
    }
    for (unsigned int j = tid; j < outputs; j += 32 * AS_WARPS)
    {
        const unsigned int r = j / p.vdim, d = j % p.vdim, to = j / share;
        const float mr = top(meet.ml, AS_WARPS, r), base = mr == -INFINITY ? 0.f : mr;
        float x = 0.f;
#pragma unroll
        for (int w = 0; w < AS_WARPS; w++) { x += exp2f(meet.ml[w][r][0] - base) * meet.om[w][r * DV + d]; }
        *cluster.map_shared_rank(&meet.recv[split * share + (j - to * share)], to) = x;
    }
    cluster.sync();
    const unsigned int first = split * share, count = first < outputs ? min(share, outputs - first) : 0u;
    for (unsigned int i = tid; i < count; i += 32 * AS_WARPS)
    {
        const unsigned int r = (first + i) / p.vdim, d = (first + i) % p.vdim;
        // (a row all of whose scores are minus infinity has weights of zero: with a sink its output is zero)
        const float mr = top(meet.recv_ml, S, r), base = mr == -INFINITY ? 0.f : mr;
        float lr = 0.f, x = 0.f;
        for (unsigned int c = 0; c < S; c++)
        {
            const float w = exp2f(meet.recv_ml[c][r][0] - base);
            lr += w * meet.recv_ml[c][r][1];
            x += w * meet.recv[c * share + i];
        }
        if (p.sink != nullptr) { lr += exp2f(p.sink[kvh * p.G + (r0 + r) % p.G] * 1.44269504088896341f - base); }
        attention_store(p, qkvg, start, kvh, r0 + r, d, x / lr);
    }
}

// Clusters of S CTAs that the device holds at once, less what the previous kernel's CTAs, which leave one after the other, may cut up:
// one in twenty (32 clusters of eight where 33 fit ran in two rounds behind an append), a quarter of the sizes between eight and
// sixteen (16 clusters of thirteen where 17 fit did).  The GPCs differ in size, so this is asked for, once for each kernel and size.
template <int DK, int DV, int NR>
static unsigned int direct_clusters(unsigned int S, int device)
{
    static std::atomic<int> known[64][kDirectSplits + 1];
    int n = known[device][S].load(std::memory_order_acquire);
    if (n == 0)
    {
        auto kernel = attention_direct_kernel<DK, DV, NR>;
        cudaLaunchConfig_t cfg;
        memset(&cfg, 0, sizeof(cfg));
        cfg.gridDim = dim3(S);
        cfg.blockDim = dim3(32 * AS_WARPS);
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = S;
        attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        if ((S > 8 && cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess)
            || cudaOccupancyMaxActiveClusters(&n, kernel, &cfg) != cudaSuccess)
        {
            cudaGetLastError();
            n = 0;
        }
        known[device][S].store(n > 0 ? n : -1, std::memory_order_release);
    }
    return n <= 0 ? 0u : (unsigned int)(S == 1 ? n : S > 8 && S < 16 ? n * 3 / 4 : n * 19 / 20);
}

// Splits of a unit, from a model fitted to the like kernel of the quantised models (attn_splits of decode_ops.cu, with its
// measurements): clusters run in rounds on the slots of the GPU; a round of n CTAs takes 4 ns and the larger of 14 ns (a CTA's own
// pace) and 0.08 n ns (HBM) per row of a split, and 5 us, and 5 more for a second one; a cluster takes 0.15 us per member to meet.
// Measured (16384 rows, us, split counts; with slots counted as eight GPCs of equal size and no clusters of more than eight past one
// CTA per SM / now): 4 sequences of 4 tokens, 8 kv heads of 128, 1 query head each 8: 91.5 / 7: 59.1; 32 sequences of 4 tokens, 4 kv heads
// of 64 2: 140 / 3: 102; 4 sequences of one token, the same heads 8: 32.0 / 16: 23.1; the other way, where nothing cuts the places up, 4
// sequences of one token, 8 kv heads of 128, 8 query heads each 8: 52.9 / 7: 57.8.  Over 290 shapes of 256 to 16384 rows the
// model's choice among 1 to 8 and 16 takes 1.008 times the best one's time, before 1.028.
template <class Clusters>
static unsigned int direct_splits(unsigned long long units, unsigned int len, Clusters clusters)
{
    unsigned int best = 1;
    float least = INFINITY;
    for (unsigned int S = 1; S <= kDirectSplits; S++)
    {
        if (S > 1 && len / S < 64u) { break; }
        if (S > 8 && S < 16 && len / S < 256u) { continue; }    // 1024 rows, 8 units: 11 splits 7.6 us, 8 6.8
        const unsigned long long slots = (unsigned long long)clusters(S) * S;
        if (slots == 0 || (S > 8 && units * S > slots)) { continue; }
        const float rows = (float)((len + S - 1) / S);
        auto round = [&](unsigned long long n) { return n == 0 ? 0.f : rows * (4.f + fmaxf(14.f, 0.08f * (float)n)) + 5000.f; };
        const float cost = (float)(units * S / slots) * round(slots) + round(units * S % slots) + 150.f * (float)S + (units * S > slots ? 5000.f : 0.f);
        if (cost < least)
        {
            least = cost;
            best = S;
        }
    }
    return best;
}

template <int DK, int DV, int NR>
static int run_direct(AttnParams p, unsigned int entries, unsigned int max_len, int device, cudaStream_t stream, bool pdl)
{
    p.splits = direct_splits((unsigned long long)entries * p.Hkv * p.row_tiles, max_len, [&](unsigned int S) { return direct_clusters<DK, DV, NR>(S, device); });
    const dim3 grid(p.splits, p.Hkv * p.row_tiles, entries);
    return launch_cluster("attention_direct", attention_direct_kernel<DK, DV, NR>, grid, dim3(32 * AS_WARPS), 0, p.splits, stream, pdl, p);
}

int launch_attention_direct(const AttnParams& p0, unsigned int entries, unsigned int max_n, unsigned int max_len, cudaStream_t stream, bool pdl)
{
    AttnParams p = p0;
    auto low = [](const void* q) { return (reinterpret_cast<uintptr_t>(q) & 31u) != 0; };
    if (p.dim > 128 || p.vdim > 128 || (p.k_ld % 16) || (p.v_ld % 16) || low(p.k_cache) || low(p.v_cache) || low(p.qkvg) || (p.ld % 16) || entries > 65535u) { return -1; }
    const unsigned int nr = max_n * p.G <= 8 ? 1 : 2;
    p.row_tiles = (max_n * p.G + 8 * nr - 1) / (8 * nr);
    if ((unsigned long long)p.Hkv * p.row_tiles > 65535ull) { return -1; }
    const DecoderDevice* dev = decoder_device();
    if (!dev) { return 1; }
    if (p.window != 0 && max_len > p.window + max_n) { max_len = p.window + max_n; }
    auto run = [&](auto dk, auto dv) {
        constexpr int DK = decltype(dk)::value, DV = decltype(dv)::value;
        return nr == 1 ? run_direct<DK, DV, 1>(p, entries, max_len, dev->device, stream, pdl) : run_direct<DK, DV, 2>(p, entries, max_len, dev->device, stream, pdl);
    };
    using C64 = std::integral_constant<int, 64>;
    using C128 = std::integral_constant<int, 128>;
    if (p.dim <= 64) { return p.vdim <= 64 ? run(C64(), C64()) : run(C64(), C128()); }
    return p.vdim <= 64 ? run(C128(), C64()) : run(C128(), C128());
}

}    // namespace b200

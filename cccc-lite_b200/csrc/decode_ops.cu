// C-ABI of the non-GEMM ops of a decode layer: RMSNorm (with the residual add that precedes it),
// RoPE, embedding gather, SwiGLU, and attention of one new token per sequence over a BF16 KV cache
// with the q/k norms, RoPE and the cache append folded into its prologue.
#include "common.cuh"
#include "attn_decode.cuh"
#include "../../include/cccc_cuda_b200.h"

#include <atomic>

namespace cg = cooperative_groups;

namespace b200
{

// ---- RMSNorm ------------------------------------------------------------------------------------
// One CTA per row.  With a residual: s = bf16(x + r) is stored (the reference's add tensor,
// R1 = X + O_out) and normalised.  Shared memory: the row as floats + 256 partial sums.
__global__ void __launch_bounds__(kTeam) rms_norm_bf16_kernel(const uint16_t* __restrict__ X, const uint16_t* __restrict__ R,
    uint16_t* __restrict__ S, uint16_t* __restrict__ Y, const uint16_t* __restrict__ scale, unsigned int inner, float eps)
{
    extern __shared__ __align__(16) float rn_smem[];
    float* xs = rn_smem;
    float* part = rn_smem + inner;
    const unsigned int tid = threadIdx.x;
    const size_t row = (size_t)blockIdx.x * inner;
    pdl_launch_dependents();
    pdl_wait();
    for (unsigned int i = tid; i < inner; i += kTeam)
    {
        float v = bf16_bits_to_float(X[row + i]);
        if (R != nullptr)
        {
            v = bf16_round(__fadd_rn(v, bf16_bits_to_float(R[row + i])));
            if (S != nullptr) { S[row + i] = bf16_bits(v); }
        }
        xs[i] = v;
    }
    team_sync();
    team_sum_squares(xs, part, 1, inner, tid);
    const float invstd = rms_invstd(part[0], inner, eps);
    for (unsigned int i = tid; i < inner; i += kTeam)
    {
        Y[row + i] = bf16_bits(rms_apply(xs[i], invstd, scale ? bf16_bits_to_float(scale[i]) : 1.f));
    }
}

// The same with a row's elements in eights, for rows that start on 16 bytes.  Bound by its latencies: in a decode step it stands
// between two linears with a block to a token.  The row and its scale are under way together, before anything is summed, and stay in
// registers; the sums of squares keep the order of team_sum_squares (thread t the elements t, t + 256, ..: through shared memory), and
// every warp adds the 256 sums by itself, in the halving tree's order, so that two barriers are left of six.  4 rows of 4096 columns
// 2.7 -> 1.9 us, with a residual 3.7 -> 2.3; 1024 rows 7.1 -> 5.2 and 9.1 -> 7.0 (17 MB to move, 2.6 us).
template <int C>    // eights per thread
__global__ void __launch_bounds__(kTeam) rms_norm_bf16_wide_kernel(const uint16_t* __restrict__ X, const uint16_t* __restrict__ R,
    uint16_t* __restrict__ S, uint16_t* __restrict__ Y, const uint16_t* __restrict__ scale, unsigned int inner, float eps)
{
    __shared__ __align__(16) float xs[C * kTeam * 8];
    __shared__ float part[kTeam];
    const unsigned int tid = threadIdx.x, lane = tid & 31u;
    const size_t row = (size_t)blockIdx.x * inner;
    pdl_launch_dependents();
    pdl_wait();
    uint4 xv[C], rv[C], wv[C];
#pragma unroll
    for (int c = 0; c < C; c++)
    {
        const unsigned int i = (c * kTeam + tid) * 8;
        xv[c] = rv[c] = make_uint4(0u, 0u, 0u, 0u);
        wv[c] = make_uint4(0x3F803F80u, 0x3F803F80u, 0x3F803F80u, 0x3F803F80u);
        if (i < inner)
        {
            xv[c] = *reinterpret_cast<const uint4*>(X + row + i);
            if (R != nullptr) { rv[c] = *reinterpret_cast<const uint4*>(R + row + i); }
            if (scale != nullptr) { wv[c] = *reinterpret_cast<const uint4*>(scale + i); }
        }
    }
    float v[C][8];
#pragma unroll
    for (int c = 0; c < C; c++)
    {
        const unsigned int i = (c * kTeam + tid) * 8;
        const uint32_t x[4] = { xv[c].x, xv[c].y, xv[c].z, xv[c].w }, r[4] = { rv[c].x, rv[c].y, rv[c].z, rv[c].w };
#pragma unroll
        for (int j = 0; j < 4; j++)
        {
            v[c][2 * j] = __uint_as_float(x[j] << 16);
            v[c][2 * j + 1] = __uint_as_float(x[j] & 0xFFFF0000u);
            if (R != nullptr)
            {
                v[c][2 * j] = bf16_round(__fadd_rn(v[c][2 * j], __uint_as_float(r[j] << 16)));
                v[c][2 * j + 1] = bf16_round(__fadd_rn(v[c][2 * j + 1], __uint_as_float(r[j] & 0xFFFF0000u)));
            }
        }
        if (i < inner)
        {
            if (R != nullptr && S != nullptr)
            {
                uint32_t s[4];
#pragma unroll
                for (int j = 0; j < 4; j++) { s[j] = bf16_bits(v[c][2 * j]) | ((uint32_t)bf16_bits(v[c][2 * j + 1]) << 16); }
                *reinterpret_cast<uint4*>(S + row + i) = make_uint4(s[0], s[1], s[2], s[3]);
            }
            *reinterpret_cast<float4*>(xs + i) = make_float4(v[c][0], v[c][1], v[c][2], v[c][3]);
            *reinterpret_cast<float4*>(xs + i + 4) = make_float4(v[c][4], v[c][5], v[c][6], v[c][7]);
        }
    }
    __syncthreads();
    float s = 0.f;
#pragma unroll
    for (int j = 0; j < 8 * C; j++)
    {
        const unsigned int i = tid + j * kTeam;
        if (i < inner) { s = __fmaf_rn(xs[i], xs[i], s); }
    }
    part[tid] = s;
    __syncthreads();
    float q[8];
#pragma unroll
    for (int j = 0; j < 8; j++) { q[j] = part[lane + 32 * j]; }
#pragma unroll
    for (int j = 0; j < 4; j++) { q[j] += q[j + 4]; }
    q[0] += q[2];
    q[1] += q[3];
    s = q[0] + q[1];
#pragma unroll
    for (int k = 16; k > 0; k >>= 1) { s += __shfl_down_sync(0xFFFFFFFFu, s, k); }
    const float invstd = rms_invstd(__shfl_sync(0xFFFFFFFFu, s, 0), inner, eps);
#pragma unroll
    for (int c = 0; c < C; c++)
    {
        const unsigned int i = (c * kTeam + tid) * 8;
        const uint32_t w[4] = { wv[c].x, wv[c].y, wv[c].z, wv[c].w };
        uint32_t y[4];
#pragma unroll
        for (int j = 0; j < 4; j++)
        {
            y[j] = bf16_bits(rms_apply(v[c][2 * j], invstd, __uint_as_float(w[j] << 16)))
                | ((uint32_t)bf16_bits(rms_apply(v[c][2 * j + 1], invstd, __uint_as_float(w[j] & 0xFFFF0000u))) << 16);
        }
        if (i < inner) { *reinterpret_cast<uint4*>(Y + row + i) = make_uint4(y[0], y[1], y[2], y[3]); }
    }
}

// ---- RoPE (standalone) ---------------------------------------------------------------------------
__global__ void __launch_bounds__(256) rope_bf16_kernel(const uint16_t* __restrict__ X, uint16_t* __restrict__ Y,
    const uint16_t* __restrict__ cos_tab, const uint16_t* __restrict__ sin_tab, unsigned int D, unsigned int T, unsigned long long total,
    unsigned int pos_offset)
{
    const unsigned int half = D / 2;
    pdl_launch_dependents();
    pdl_wait();
    for (unsigned long long idx = (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x; idx < total;
         idx += (unsigned long long)gridDim.x * blockDim.x)
    {
        const unsigned int i = (unsigned int)(idx % half);
        const unsigned long long bt = idx / half;
        const unsigned int t = (unsigned int)(bt % T);
        const size_t base = (size_t)bt * D;
        const size_t tab = (size_t)(t + pos_offset) * half + i;
        float yl, yr;
        rope_pair(bf16_bits_to_float(X[base + i]), bf16_bits_to_float(X[base + half + i]), bf16_bits_to_float(cos_tab[tab]),
            bf16_bits_to_float(sin_tab[tab]), yl, yr);
        Y[base + i] = bf16_bits(yl);
        Y[base + half + i] = bf16_bits(yr);
    }
}

// ---- embedding gather ----------------------------------------------------------------------------
__global__ void __launch_bounds__(256) embed_bf16_kernel(const int* __restrict__ ids, const uint16_t* __restrict__ W,
    uint16_t* __restrict__ Y, unsigned int D, unsigned int vocab)
{
    pdl_launch_dependents();
    pdl_wait();
    const int id = ids[blockIdx.x];
    const bool ok = id >= 0 && (unsigned int)id < vocab;
    const uint16_t* src = W + (size_t)(ok ? id : 0) * D;
    uint16_t* dst = Y + (size_t)blockIdx.x * D;
    if ((D % 8) == 0 && ((reinterpret_cast<uintptr_t>(src) | reinterpret_cast<uintptr_t>(dst)) & 15u) == 0)
    {
        for (unsigned int i = threadIdx.x; i < D / 8; i += blockDim.x)
        {
            reinterpret_cast<uint4*>(dst)[i] = ok ? reinterpret_cast<const uint4*>(src)[i] : make_uint4(0, 0, 0, 0);
        }
    }
    else
    {
        for (unsigned int i = threadIdx.x; i < D; i += blockDim.x) { dst[i] = ok ? src[i] : (uint16_t)0; }
    }
}

// ---- SwiGLU ----------------------------------------------------------------------------------------
__global__ void __launch_bounds__(256) swiglu_bf16_kernel(const uint16_t* __restrict__ G, const uint16_t* __restrict__ U,
    uint16_t* __restrict__ O, unsigned int cols, unsigned int ldg, unsigned int ldu, unsigned int ldo)
{
    pdl_launch_dependents();
    pdl_wait();
    const size_t row = blockIdx.y;
    for (unsigned int i = blockIdx.x * blockDim.x + threadIdx.x; i < cols; i += gridDim.x * blockDim.x)
    {
        O[row * ldo + i] = bf16_bits(swiglu_one(bf16_bits_to_float(G[row * ldg + i]), bf16_bits_to_float(U[row * ldu + i])));
    }
}

// Eight elements a thread, from rows that start on 16 bytes: a prompt's.  Bound by the sigmoids' instructions and by HBM (38 MB in
// 6 us at 6144 columns x 1024 rows); the one-element form above is bound by its two-byte accesses and its blocks' starts.  6144
// columns x 256 / 1024 rows 6.8 / 25.8 -> 4.6 / 10.1 us.
__global__ void __launch_bounds__(256) swiglu_bf16_wide_kernel(const uint16_t* __restrict__ G, const uint16_t* __restrict__ U,
    uint16_t* __restrict__ O, unsigned int cols, unsigned int ldg, unsigned int ldu, unsigned int ldo)
{
    pdl_launch_dependents();
    pdl_wait();
    const size_t row = blockIdx.y;
    const unsigned int i = (blockIdx.x * blockDim.x + threadIdx.x) * 8;
    if (i >= cols) { return; }
    const uint4 g = *reinterpret_cast<const uint4*>(G + row * ldg + i), u = *reinterpret_cast<const uint4*>(U + row * ldu + i);
    const uint32_t gw[4] = { g.x, g.y, g.z, g.w }, uw[4] = { u.x, u.y, u.z, u.w };
    uint32_t ow[4];
#pragma unroll
    for (int j = 0; j < 4; j++)
    {
        const uint32_t lo = bf16_bits(swiglu_one(__uint_as_float(gw[j] << 16), __uint_as_float(uw[j] << 16)));
        const uint32_t hi = bf16_bits(swiglu_one(__uint_as_float(gw[j] & 0xFFFF0000u), __uint_as_float(uw[j] & 0xFFFF0000u)));
        ow[j] = lo | (hi << 16);
    }
    *reinterpret_cast<uint4*>(O + row * ldo + i) = make_uint4(ow[0], ow[1], ow[2], ow[3]);
}

// ---- q/k norm, RoPE and cache append of many tokens ----------------------------------------------------
// One warp per (token, head); heads 0 .. H-1 are queries, then Hkv keys, then Hkv values.  Lane l holds the elements l, l + 32,
// ..: a rotation's two elements meet in one lane, and the squares are added in the order of team_sum_squares, so that a row
// has the bits that the decode kernel's prologue gives it.  Bound by HBM: a prompt's projections are read once, its queries and
// cache rows written once.
template <int HD>
__global__ void __launch_bounds__(256) attn_append_kernel(const AttnDecodeParams p)
{
    constexpr int N = HD / 32, HALF = N / 2;
    const unsigned int lane = threadIdx.x & 31u, head = blockIdx.y * 8 + (threadIdx.x >> 5);
    const unsigned int b = blockIdx.x;
    pdl_launch_dependents();
    pdl_wait();
    if (head >= p.H + 2 * p.Hkv) { return; }
    const int pos_i = p.pos[b];
    const unsigned int pos = pos_i < 0 ? 0u : (unsigned int)pos_i;
    const bool is_q = head < p.H, is_v = head >= p.H + p.Hkv;
    const unsigned int kvh = is_v ? head - p.H - p.Hkv : head - p.H;
    const uint16_t* src = is_q ? p.q + (size_t)b * p.ldq + (size_t)head * HD : (is_v ? p.v + (size_t)b * p.ldv : p.k + (size_t)b * p.ldk) + (size_t)kvh * HD;
    uint16_t* dst;
    if (is_q) { dst = p.out + (size_t)b * p.ldo + (size_t)head * HD; }
    else
    {
        if (pos >= p.T_max) { return; }
        dst = (is_v ? p.v_cache : p.k_cache) + (attn_cache_row(p, b, kvh) + pos) * HD;
    }
    if (is_v)
    {
#pragma unroll
        for (int i = 0; i < N; i++) { dst[lane + 32 * i] = src[lane + 32 * i]; }
        return;
    }
    float x[N];
#pragma unroll
    for (int i = 0; i < N; i++) { x[i] = bf16_bits_to_float(src[lane + 32 * i]); }
    const uint16_t* w = is_q ? p.q_norm : p.k_norm;
    if (w != nullptr)
    {
        float sq[N];
#pragma unroll
        for (int i = 0; i < N; i++) { sq[i] = __fmul_rn(x[i], x[i]); }
#pragma unroll
        for (int h = N / 2; h > 0; h >>= 1)
        {
#pragma unroll
            for (int i = 0; i < h; i++) { sq[i] += sq[i + h]; }
        }
        float sum = sq[0];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) { sum += __shfl_down_sync(0xFFFFFFFFu, sum, o); }
        const float invstd = rms_invstd(__shfl_sync(0xFFFFFFFFu, sum, 0), HD, p.eps);
#pragma unroll
        for (int i = 0; i < N; i++) { x[i] = rms_apply(x[i], invstd, bf16_bits_to_float(w[lane + 32 * i])); }
    }
    const uint16_t *c = p.cos_tab + (size_t)pos * (HD / 2), *s = p.sin_tab + (size_t)pos * (HD / 2);
#pragma unroll
    for (int i = 0; i < HALF; i++)
    {
        float yl, yr;
        rope_pair(x[i], x[i + HALF], bf16_bits_to_float(c[lane + 32 * i]), bf16_bits_to_float(s[lane + 32 * i]), yl, yr);
        dst[lane + 32 * i] = bf16_bits(yl);
        dst[lane + 32 * (i + HALF)] = bf16_bits(yr);
    }
}

struct DeviceFacts
{
    std::atomic<int> ready{ 0 };
    int sm_count = 0, max_smem = 0, sm_smem = 0, device = 0;
};
static DeviceFacts g_facts[64];
static const DeviceFacts* device_facts()
{
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) { return nullptr; }
    DeviceFacts& f = g_facts[dev];
    if (f.ready.load(std::memory_order_acquire) == 0)
    {
        int a = 0, b = 0, c = 0;
        if (cudaDeviceGetAttribute(&a, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess
            || cudaDeviceGetAttribute(&b, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) != cudaSuccess
            || cudaDeviceGetAttribute(&c, cudaDevAttrMaxSharedMemoryPerMultiprocessor, dev) != cudaSuccess)
        {
            return nullptr;
        }
        f.sm_count = a;    // two threads may both write the same values: harmless
        f.max_smem = b;
        f.sm_smem = c;
        f.device = dev;
        f.ready.store(1, std::memory_order_release);
    }
    return &f;
}

// Splits of a (sequence, kv head), from a model fitted to measurements (4096 rows, 8 kv heads): the clusters run in rounds on the
// slots of the GPU, up to three CTAs per SM - as many as their shared memory, which grows with the rows of a split, leaves room for -
// in eight GPCs of whole clusters; a round of n CTAs takes 4 ns and the larger of 14 ns (a CTA's own pace) and 0.08 n ns (HBM) per row
// of a split, and 5 us; a cluster takes 0.15 us per member to meet.  Hence as many splits as still run in one round, and more rounds
// only where one would leave slots empty for long.  Measured (us, split counts): 8 sequences 4: 35.5, 6: 30.4 (384 CTAs), 7: 45.7; 16
// sequences 2: 59.0, 3: 50.8, 4: 71.3; 32 sequences 1: 103.9, 2: 125.2, 3: 97.7, 5: 121.1; one sequence 8: 15.4, 16: 12.6.  Long
// caches, 32768 rows, as three CTAs per SM would have it / as their shared memory does: 16 sequences of 4 heads per kv head 3:
// 582 / 6: 345; of 8 heads 8 sequences 6: 281 / 8: 192, 16 sequences 3: 536 / 6: 420.
// smem(S): bytes that a CTA of S splits asks for.
template <class Smem>
static unsigned int attn_splits(unsigned long long units, unsigned int T_max, const DeviceFacts& dev, Smem smem)
{
    unsigned int best = 8;    // (its scores always fit: see attn_served)
    float least = INFINITY;
    for (unsigned int S = 1; S <= (unsigned int)AD_MAX_SPLITS; S = S < 8 ? S + 1 : S + 8)
    {
        if (S > 1 && T_max / S < 64u) { break; }
        if (smem(S) > (size_t)dev.max_smem) { continue; }
        const unsigned long long room = (size_t)dev.sm_smem / (smem(S) + 1024), per_sm = room < 3 ? room : 3;    // 1 KB of a CTA's is the system's
        const unsigned long long slots = (per_sm * ((unsigned)dev.sm_count / 8) / S) * S * 8;
        const float rows = (float)((T_max + S - 1) / S);
        if (slots == 0) { continue; }
        if (S > 8 && units * S > slots) { break; }
        auto round = [&](unsigned long long n) { return n == 0 ? 0.f : rows * (4.f + fmaxf(14.f, 0.08f * (float)n)) + 5000.f; };
        const float cost = (float)(units * S / slots) * round(slots) + round(units * S % slots) + 150.f * (float)S;
        if (cost < least)
        {
            least = cost;
            best = S;
        }
    }
    return best;
}

// Caches that this entry point serves: up to what sixteen splits hold whose scores are floats, in 32s of rows, beside (3 G + 5) HD + 260 G
// + 256 + max(2048 G, 8192) floats.  This kernel holds BF16 scores and would go on for twice the rows; callers take their own path
// from there on and rely on being told.
template <int G, int HD>
static bool attn_served(unsigned int T_max, int max_smem)
{
    constexpr size_t fixed = (3 * G + 5) * HD + 260 * G + 256 + (G < 4 ? 8192 : 2048 * G);
    const size_t rows = ((size_t)T_max + 15) / 16;
    return (fixed + G * ((rows + 31) / 32 * 32)) * sizeof(float) <= (size_t)max_smem;
}

template <int G, int HD>
static int launch_attn(const AttnDecodeParams& p, const DeviceFacts& dev, cudaStream_t stream, bool pdl)
{
    const int max_smem = dev.max_smem;
    if (!attn_served<G, HD>(p.T_max, max_smem)) { return -1; }
    auto kernel = attn_decode_kernel<G, HD>;
    auto row_cap = [&](unsigned int splits) { return ((p.T_max + splits * AD_TILE - 1) / (splits * AD_TILE)) * AD_TILE; };
    auto smem = [&](unsigned int splits) { return sizeof(AttnDecodeSmem<G, HD>) + (size_t)G * ad_score_row(row_cap(splits)) * 2; };
    unsigned int S = attn_splits((unsigned long long)p.B * p.Hkv, p.T_max, dev, smem);
    // (the same value from every thread)
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, max_smem) != cudaSuccess
        || (S > 8 && cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess))
    {
        return report_launch("attn_decode_bf16") ? 1 : 1;
    }
    cudaLaunchConfig_t cfg;
    memset(&cfg, 0, sizeof(cfg));
    cfg.gridDim = dim3(S, p.Hkv, p.B);
    cfg.blockDim = dim3(AD_THREADS);
    cfg.dynamicSmemBytes = smem(S);
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = S;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = pdl ? 2 : 1;
    // Can a cluster of more than eight be scheduled?  That depends on the device and on what its CTAs ask for: asked for once up to the
    // largest request that can, and down to the smallest that cannot.
    static std::atomic<unsigned int> can[64], cannot[64];    // bytes; 0: not known
    if (S > 8 && cfg.dynamicSmemBytes > can[dev.device].load(std::memory_order_relaxed))
    {
        const unsigned int no = cannot[dev.device].load(std::memory_order_relaxed);
        int n = 0;
        if ((no == 0 || cfg.dynamicSmemBytes < no) && cudaOccupancyMaxActiveClusters(&n, kernel, &cfg) == cudaSuccess && n > 0)
        {
            can[dev.device].store((unsigned int)cfg.dynamicSmemBytes, std::memory_order_relaxed);
        }
        else
        {
            cudaGetLastError();
            if (no == 0 || cfg.dynamicSmemBytes < no) { cannot[dev.device].store((unsigned int)cfg.dynamicSmemBytes, std::memory_order_relaxed); }
            S = 8;
            if (smem(S) > (size_t)max_smem) { return -1; }
            cfg.gridDim.x = attr[0].val.clusterDim.x = S;
            cfg.dynamicSmemBytes = smem(S);
        }
    }
    count_launch();
    if (cudaLaunchKernelEx(&cfg, kernel, p, row_cap(S)) != cudaSuccess) { return report_launch("attn_decode_bf16") ? 1 : 1; }
    return 0;
}

template <class K, class... Args>
static int launch_simple(const char* label, K kernel, dim3 grid, dim3 block, size_t smem, cudaStream_t stream, bool pdl, Args... args)
{
    cudaLaunchConfig_t cfg;
    memset(&cfg, 0, sizeof(cfg));
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = pdl ? 1 : 0;
    count_launch();
    if (cudaLaunchKernelEx(&cfg, kernel, args...) != cudaSuccess)
    {
        report_launch(label);
        return 1;
    }
    return 0;
}

}    // namespace b200

using namespace b200;

C_EXPORT int cuda_rms_norm_bf16(const void* X, const void* residual, void* sum_out, void* Y, const void* scale, unsigned int rows,
    unsigned int inner, float epsilon, void* stream, unsigned int flags)
{
    if (rows == 0 || inner == 0) { return 0; }
    if (!X || !Y) { return -1; }
    const size_t smem = ((size_t)inner + kTeam) * sizeof(float);
    const DeviceFacts* f = device_facts();
    if (!f) { return 1; }
    if (smem > (size_t)f->max_smem) { return -1; }
    const uintptr_t at = reinterpret_cast<uintptr_t>(X) | reinterpret_cast<uintptr_t>(residual) | reinterpret_cast<uintptr_t>(sum_out)
        | reinterpret_cast<uintptr_t>(Y) | reinterpret_cast<uintptr_t>(scale);
    // Rows of a few hundred columns, as a head's norms have, leave most of a team of eights without one: with more rows than SMs
    // the form of one element a thread is done first (128 columns, 300 rows: 2.0 against 2.2 us; 100 rows 1.7 against 1.5; of 512
    // columns, 300 rows 2.8 against 2.4).  Above 8192 columns a thread would hold too many eights.
    if ((at & 15u) == 0 && (inner & 7u) == 0 && inner <= 4 * 8 * kTeam && (inner >= 512 || rows <= 128))
    {
        auto run = [&](auto kernel) {
            return launch_simple("rms_norm_bf16", kernel, dim3(rows), dim3(kTeam), 0, (cudaStream_t)stream, (flags & 1u) != 0, (const uint16_t*)X,
                (const uint16_t*)residual, (uint16_t*)sum_out, (uint16_t*)Y, (const uint16_t*)scale, inner, epsilon);
        };
        if (inner <= 8 * kTeam) { return run(rms_norm_bf16_wide_kernel<1>); }
        if (inner <= 2 * 8 * kTeam) { return run(rms_norm_bf16_wide_kernel<2>); }
        return inner <= 3 * 8 * kTeam ? run(rms_norm_bf16_wide_kernel<3>) : run(rms_norm_bf16_wide_kernel<4>);
    }
    if (smem > 48 * 1024 && cudaFuncSetAttribute(rms_norm_bf16_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess)
    {
        return report_launch("rms_norm_bf16") ? 1 : 1;
    }
    return launch_simple("rms_norm_bf16", rms_norm_bf16_kernel, dim3(rows), dim3(kTeam), smem, (cudaStream_t)stream, (flags & 1u) != 0,
        (const uint16_t*)X, (const uint16_t*)residual, (uint16_t*)sum_out, (uint16_t*)Y, (const uint16_t*)scale, inner, epsilon);
}

C_EXPORT int cuda_rope_bf16(const void* X, void* Y, const void* cos_tab, const void* sin_tab, unsigned int D, unsigned int T,
    unsigned int B, unsigned int pos_offset, void* stream, unsigned int flags)
{
    const unsigned long long total = (unsigned long long)(D / 2) * T * B;
    if (total == 0) { return 0; }
    if (!X || !Y || !cos_tab || !sin_tab || (D & 1u)) { return -1; }
    const unsigned int grid = (unsigned int)((total + 255) / 256 < 4096 ? (total + 255) / 256 : 4096);
    return launch_simple("rope_bf16", rope_bf16_kernel, dim3(grid), dim3(256), 0, (cudaStream_t)stream, (flags & 1u) != 0, (const uint16_t*)X,
        (uint16_t*)Y, (const uint16_t*)cos_tab, (const uint16_t*)sin_tab, D, T, total, pos_offset);
}

C_EXPORT int cuda_embed_bf16(const void* ids, const void* W, void* Y, unsigned int D, unsigned int n_tokens, unsigned int vocab,
    void* stream, unsigned int flags)
{
    if (n_tokens == 0 || D == 0) { return 0; }
    if (!ids || !W || !Y) { return -1; }
    return launch_simple("embed_bf16", embed_bf16_kernel, dim3(n_tokens), dim3(256), 0, (cudaStream_t)stream, (flags & 1u) != 0, (const int*)ids,
        (const uint16_t*)W, (uint16_t*)Y, D, vocab);
}

C_EXPORT int cuda_swiglu_bf16(const void* gate, const void* up, void* out, unsigned int rows, unsigned int cols, unsigned int ld_gate,
    unsigned int ld_up, unsigned int ld_out, void* stream, unsigned int flags)
{
    if (rows == 0 || cols == 0) { return 0; }
    if (!gate || !up || !out || rows > 65535u) { return -1; }
    const unsigned int gx = (cols + 255) / 256 < 64 ? (cols + 255) / 256 : 64;
    const uintptr_t at = reinterpret_cast<uintptr_t>(gate) | reinterpret_cast<uintptr_t>(up) | reinterpret_cast<uintptr_t>(out);
    // Under three quarters of a million elements the one-element form's many short threads are done first (6144 columns of 64 rows
    // 1.9 against 3.2 us, of 1 row 1.1 against 1.6); from there on eight a thread are (128 rows 3.6 against 2.9).
    if ((unsigned long long)rows * cols >= 786432ull && ((cols | ld_gate | ld_up | ld_out) & 7u) == 0 && (at & 15u) == 0)
    {
        return launch_simple("swiglu_bf16", swiglu_bf16_wide_kernel, dim3((cols + 2047) / 2048, rows), dim3(256), 0, (cudaStream_t)stream,
            (flags & 1u) != 0, (const uint16_t*)gate, (const uint16_t*)up, (uint16_t*)out, cols, ld_gate, ld_up, ld_out);
    }
    return launch_simple("swiglu_bf16", swiglu_bf16_kernel, dim3(gx, rows), dim3(256), 0, (cudaStream_t)stream, (flags & 1u) != 0,
        (const uint16_t*)gate, (const uint16_t*)up, (uint16_t*)out, cols, ld_gate, ld_up, ld_out);
}

// The descriptor's checks and its kernel form.  0: ok, p is filled.
static int attn_params(const cuda_attn_decode* a, AttnDecodeParams* out)
{
    if (!a->q || !a->k || !a->v || !a->cos_tab || !a->sin_tab || !a->k_cache || !a->v_cache || !a->pos || !a->out) { return -1; }
    if (a->Hkv == 0 || (a->H % a->Hkv) != 0 || a->T_max == 0 || a->Hkv > 65535u) { return -1; }
    auto misaligned = [](const void* ptr) { return (reinterpret_cast<uintptr_t>(ptr) & 15u) != 0; };
    if ((a->ldq % 8) != 0 || (a->ldk % 8) != 0 || (a->ldv % 8) != 0 || misaligned(a->q) || misaligned(a->k) || misaligned(a->v)
        || misaligned(a->k_cache) || misaligned(a->v_cache) || misaligned(a->cos_tab) || misaligned(a->sin_tab)
        || (a->q_norm && misaligned(a->q_norm)) || (a->k_norm && misaligned(a->k_norm)))
    {
        return -1;
    }
    AttnDecodeParams& p = *out;
    p.q = (const uint16_t*)a->q;
    p.k = (const uint16_t*)a->k;
    p.v = (const uint16_t*)a->v;
    p.q_norm = (const uint16_t*)a->q_norm;
    p.k_norm = (const uint16_t*)a->k_norm;
    p.cos_tab = (const uint16_t*)a->cos_tab;
    p.sin_tab = (const uint16_t*)a->sin_tab;
    p.k_cache = (uint16_t*)a->k_cache;
    p.v_cache = (uint16_t*)a->v_cache;
    p.pos = (const int*)a->pos;
    p.slot = (const int*)a->slot;
    p.out = (uint16_t*)a->out;
    p.ldq = a->ldq;
    p.ldk = a->ldk;
    p.ldv = a->ldv;
    p.ldo = a->ldo;
    p.B = a->B;
    p.H = a->H;
    p.Hkv = a->Hkv;
    p.T_max = a->T_max;
    p.eps = a->epsilon;
    p.scale = 1.0f / sqrtf(a->dk > 0.f ? a->dk : (float)a->head_dim);
    return 0;
}

C_EXPORT int cuda_attn_append_bf16(const cuda_attn_decode* a, void* stream, unsigned int flags)
{
    if (!a) { return -1; }
    if (a->B == 0 || a->H == 0) { return 0; }
    AttnDecodeParams p;
    const int rc = attn_params(a, &p);
    if (rc != 0) { return rc; }
    const dim3 grid(a->B, (a->H + 2 * a->Hkv + 7) / 8);
    if (grid.y > 65535u) { return -1; }
    const bool pdl = (flags & 1u) != 0;
    if (a->head_dim == 128) { return launch_simple("attn_append_bf16", attn_append_kernel<128>, grid, dim3(256), 0, (cudaStream_t)stream, pdl, p); }
    if (a->head_dim == 64) { return launch_simple("attn_append_bf16", attn_append_kernel<64>, grid, dim3(256), 0, (cudaStream_t)stream, pdl, p); }
    return -1;
}

C_EXPORT int cuda_attn_decode_bf16(const cuda_attn_decode* a, void* stream, unsigned int flags)
{
    if (!a) { return -1; }
    if (a->B == 0 || a->H == 0) { return 0; }
    AttnDecodeParams p;
    const int rc = attn_params(a, &p);
    if (rc != 0 || a->B > 65535u) { return -1; }
    const DeviceFacts* f = device_facts();
    if (!f) { return 1; }
    const unsigned int G = a->H / a->Hkv;
    const bool pdl = (flags & 1u) != 0;
    cudaStream_t st = (cudaStream_t)stream;
    if (a->head_dim == 128)
    {
        switch (G)
        {
        case 1: return launch_attn<1, 128>(p, *f, st, pdl);
        case 2: return launch_attn<2, 128>(p, *f, st, pdl);
        case 4: return launch_attn<4, 128>(p, *f, st, pdl);
        case 8: return launch_attn<8, 128>(p, *f, st, pdl);
        default: return -1;
        }
    }
    if (a->head_dim == 64)
    {
        switch (G)
        {
        case 1: return launch_attn<1, 64>(p, *f, st, pdl);
        case 2: return launch_attn<2, 64>(p, *f, st, pdl);
        case 4: return launch_attn<4, 64>(p, *f, st, pdl);
        case 8: return launch_attn<8, 64>(p, *f, st, pdl);
        default: return -1;
        }
    }
    return -1;
}

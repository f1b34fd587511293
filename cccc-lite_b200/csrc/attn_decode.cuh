// BF16 decode attention (one new token per sequence).
//
// Bound by HBM at many rows and by its chain of dependent steps at few.  A CTA of four warps holds the G query heads of a kv
// head and walks a split of its rows; the splits of a (sequence, kv head) are one cluster.  A warp takes tiles of 16 rows by
// itself: keys and values go from global memory straight into the fragments of mma.m16n8k16 (the heads are rows 0 .. 7 of A),
// with the elements of a key, and the columns of a value, permuted so that every load is 16 bytes of a 32-byte sector that its
// neighbour completes, two tiles ahead in registers.  Roundings as the reference has them (MatrixEx.cpp:3056, 3091), and the
// decode program's form of it (attn_scores, attn_pv): scores to BF16, softmax weights - normalised - to BF16.  So the scores of
// a split wait in shared memory, where only the warp that made them reads them, until the cluster knows maximum and sum.
// Before the first product: one round trip brings projections, norms, rotation and the first tiles; a warp normalises and
// rotates a head; one barrier.  Between the products: every CTA sends its maximum and sum to all, one cluster barrier, with the
// first values under way.  Behind them: every CTA sends each its share of the outputs, one cluster barrier, and the shares are
// summed where they lie: nobody reads a peer's memory, so nobody has to wait for readers.
// Measured (32 query heads, 8 kv heads of 128, 4096 rows; before, with K and V through a cp.async ring of each thread's own
// pieces and eight barriers: now, us): 1 / 4 / 8 / 16 / 24 / 32 sequences 18.4 / 26.5 / 40.3 / 67.9 / 108.8 / 121.4 : 12.6 / 22.6 /
// 30.4 / 50.8 / 71.1 / 97.7 (0.85 of the HBM rate at 24 and 32); 250 rows, 4 kv heads, 4 sequences 10.9 : 6.5.
#pragma once

#include <cooperative_groups.h>

#include "decode_ops.cuh"

namespace b200
{

constexpr int AD_WARPS = 4;
constexpr int AD_THREADS = 32 * AD_WARPS;
constexpr int AD_TILE = 16;         // rows of a tile
constexpr int AD_MAX_SPLITS = 16;   // one cluster
constexpr int AD_AHEAD_BYTES = 48 * 1024;    // of keys and of values each, asked into L2 ahead of the previous kernel's end

__device__ __forceinline__ void ad_load16(uint32_t* r, const uint16_t* p, bool ok)
{
    const uint4 v = ok ? __ldcg(reinterpret_cast<const uint4*>(p)) : make_uint4(0u, 0u, 0u, 0u);
    r[0] = v.x;
    r[1] = v.y;
    r[2] = v.z;
    r[3] = v.w;
}
// D rows 0-7 += A rows 0-7 * B; rows 8-15 do not exist
__device__ __forceinline__ void ad_mma(float (&c)[2], uint32_t a0, uint32_t a2, uint32_t b0, uint32_t b1)
{
    [[maybe_unused]] float d2, d3;
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%5}, {%7,%8}, {%0,%1,%9,%9};"
        : "+f"(c[0]), "+f"(c[1]), "=f"(d2), "=f"(d3)
        : "r"(a0), "r"(0u), "r"(a2), "r"(b0), "r"(b1), "f"(0.f));
}
__device__ __forceinline__ uint32_t ad_pack(float lo, float hi)
{
    uint32_t r;
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
    return r;
}
// (m, l) += (m2, l2): maxima, and sums of exponentials relative to them
__device__ __forceinline__ void ad_merge(float& m, float& l, float m2, float l2)
{
    const float mn = fmaxf(m, m2), base = mn == -INFINITY ? 0.f : mn;
    l = l * __expf(m - base) + l2 * __expf(m2 - base);
    m = mn;
}

template <int G, int HD>
struct alignas(16) AttnDecodeSmem
{
    uint16_t q[8][HD];                    // rotated queries (rows past G: zeros)
    uint16_t kn[HD], vn[HD];              // the new token's row
    float ml[AD_WARPS][8][2];             // a warp's maximum and sum of exponentials
    float om[AD_WARPS][G][HD + 4];        // its outputs
    float recv_ml[AD_MAX_SPLITS][G][2];
    float recv[G * HD + AD_MAX_SPLITS];   // [split][outputs of this CTA]
    // behind it: scores [G][ad_score_row(row_cap)] as BF16
};
__host__ __device__ constexpr unsigned int ad_score_row(unsigned int row_cap) { return row_cap + 8; }    // heads start in different banks

template <int G, int HD>
__global__ void __launch_bounds__(AD_THREADS, 3) attn_decode_kernel(const AttnDecodeParams p, const unsigned int row_cap)
{
    namespace cg = cooperative_groups;
    constexpr int KP = HD / 32, VP = HD / 64;    // 16-byte pieces of a key row per lane; of a value row
    constexpr int N = HD / 32, HALF = N / 2;
    constexpr unsigned int STEP = AD_WARPS * AD_TILE;
    extern __shared__ __align__(16) unsigned char ad_smem[];
    AttnDecodeSmem<G, HD>& sm = *reinterpret_cast<AttnDecodeSmem<G, HD>*>(ad_smem);
    uint16_t* const scores = reinterpret_cast<uint16_t*>(ad_smem + sizeof(AttnDecodeSmem<G, HD>));
    cg::cluster_group cluster = cg::this_cluster();
    const unsigned int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    const unsigned int S = gridDim.x, rank = blockIdx.x, kvh = blockIdx.y, b = blockIdx.z;
    asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");    // met before the first store into a peer
    pdl_launch_dependents();

    // rows of this split: [t0, t1), whole tiles
    unsigned int pos, t0, t1;
    auto place = [&]() {
        const int pos_i = *reinterpret_cast<const volatile int*>(p.pos + b);
        pos = pos_i < 0 ? 0u : (unsigned int)pos_i;
        const unsigned int T = min(pos + 1u, p.T_max), per = ((T + S * AD_TILE - 1) / (S * AD_TILE)) * AD_TILE;
        t0 = min(rank * per, T);
        t1 = min(t0 + per, T);
    };
    if (p.slot == nullptr)
    {
        // Ahead of the previous kernel's end nothing is read but the position, and that only says how far to ask: an older one
        // does no harm.  (An older slot could lie anywhere: with slots nothing is asked for.)
        place();
        const unsigned int lines = min((t1 - t0) * (HD * 2 / 128), (unsigned int)AD_AHEAD_BYTES / 128);
        const size_t row = ((size_t)b * p.Hkv + kvh) * p.T_max + t0;
        for (unsigned int i = threadIdx.x; i < lines; i += AD_THREADS)
        {
            asm volatile("prefetch.global.L2 [%0];" ::"l"(reinterpret_cast<const char*>(p.k_cache + row * HD) + (size_t)i * 128));
            asm volatile("prefetch.global.L2 [%0];" ::"l"(reinterpret_cast<const char*>(p.v_cache + row * HD) + (size_t)i * 128));
        }
    }
    pdl_wait();
    place();
    const size_t row0 = attn_cache_row(p, b, kvh);
    const uint16_t *K = p.k_cache + row0 * HD, *V = p.v_cache + row0 * HD;
    const bool owner = pos >= t0 && pos < t1;    // this split appends the new row (and takes it from shared memory)

    using KTile = uint32_t[2][KP][4];
    using VTile = uint32_t[4][VP][4];
    auto load_k = [&](KTile& k, unsigned int r) {
#pragma unroll
        for (int i = 0; i < 2; i++)
        {
            const unsigned int key = r + i * 8 + g;
#pragma unroll
            for (int c = 0; c < KP; c++) { ad_load16(k[i][c], K + (size_t)key * HD + c * 32 + t * 8, key < t1 && key != pos); }
        }
    };
    auto load_v = [&](VTile& v, unsigned int r) {
#pragma unroll
        for (int i = 0; i < 4; i++)
        {
            const unsigned int key = r + 2 * t + (i & 1) + (i >> 1) * 8;
#pragma unroll
            for (int c = 0; c < VP; c++) { ad_load16(v[i][c], V + (size_t)key * HD + c * 64 + g * 8, key < t1 && key != pos); }
        }
    };
    // Whole lines of a later tile on their way to L2.
    auto ahead = [&](const uint16_t* rows, unsigned int r) {
        constexpr unsigned int LINES = HD * 2 / 128;    // of a row
        if (lane < AD_TILE * LINES && r + lane / LINES < t1)
        {
            asm volatile("prefetch.global.L2 [%0];" ::"l"(reinterpret_cast<const char*>(rows + (size_t)r * HD) + lane * 128));
        }
    };
    const unsigned int mine = t0 + warp * AD_TILE;    // this warp's first tile
    KTile ka, kb;
    load_k(ka, mine);
    load_k(kb, mine + STEP);
    ahead(K, mine + 2 * STEP);
    ahead(K, mine + 3 * STEP);
    ahead(V, mine);

    // ---- heads: warp w takes the query heads w and w + 4, then the owner's first two the new key and the new value ----
    auto head = [&](unsigned int job) -> const uint16_t* {    // nullptr: nothing to do
        const unsigned int h = job * AD_WARPS + warp;
        if (job < 2) { return h < (unsigned int)G ? p.q + (size_t)b * p.ldq + (size_t)(kvh * G + h) * HD : nullptr; }
        if (!owner || warp > 1) { return nullptr; }
        return (warp == 0 ? p.k + (size_t)b * p.ldk : p.v + (size_t)b * p.ldv) + (size_t)kvh * HD;
    };
    uint16_t raw[3][N];
    float cs[HALF], sn[HALF];
#pragma unroll
    for (int j = 0; j < 3; j++)
    {
        const uint16_t* src = head(j);
#pragma unroll
        for (int i = 0; i < N; i++) { raw[j][i] = src != nullptr ? __ldcg(src + lane + 32 * i) : (uint16_t)0; }
    }
#pragma unroll
    for (int i = 0; i < HALF; i++)
    {
        cs[i] = bf16_bits_to_float(__ldg(p.cos_tab + (size_t)pos * (HD / 2) + lane + 32 * i));
        sn[i] = bf16_bits_to_float(__ldg(p.sin_tab + (size_t)pos * (HD / 2) + lane + 32 * i));
    }
#pragma unroll 1
    for (int j = 0; j < 3; j++)
    {
        const bool is_q = j < 2, is_k = j == 2 && warp == 0;
        const unsigned int h = j * AD_WARPS + warp;
        if (head(j) == nullptr)
        {
#pragma unroll
            for (int i = 0; i < N; i++)
            {
                if (is_q) { sm.q[h][lane + 32 * i] = 0; }
            }
            continue;
        }
        float x[N];
#pragma unroll
        for (int i = 0; i < N; i++)
        {
            const uint16_t r = j == 0 ? raw[0][i] : (j == 1 ? raw[1][i] : raw[2][i]);
            x[i] = bf16_bits_to_float(r);
            if (!is_q && !is_k)
            {
                sm.vn[lane + 32 * i] = r;
                p.v_cache[(row0 + pos) * HD + lane + 32 * i] = r;
            }
        }
        if (!is_q && !is_k) { continue; }
        // lane l holds the elements l, l + 32, ..: a rotation's two elements meet in one lane, and the squares are added in the
        // order of the reference's kernel (team_sum_squares)
        const uint16_t* w = is_q ? p.q_norm : p.k_norm;
        if (w != nullptr)
        {
            float sq[N];
#pragma unroll
            for (int i = 0; i < N; i++) { sq[i] = __fmul_rn(x[i], x[i]); }
#pragma unroll
            for (int half = N / 2; half > 0; half >>= 1)
            {
#pragma unroll
                for (int i = 0; i < half; i++) { sq[i] += sq[i + half]; }
            }
            float sum = sq[0];
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) { sum += __shfl_down_sync(0xFFFFFFFFu, sum, o); }
            const float invstd = rms_invstd(__shfl_sync(0xFFFFFFFFu, sum, 0), HD, p.eps);
#pragma unroll
            for (int i = 0; i < N; i++) { x[i] = rms_apply(x[i], invstd, bf16_bits_to_float(__ldg(w + lane + 32 * i))); }
        }
        uint16_t* dst = is_q ? sm.q[h] : sm.kn;
        uint16_t* cache = is_k ? p.k_cache + (row0 + pos) * HD : nullptr;
#pragma unroll
        for (int i = 0; i < HALF; i++)
        {
            float yl, yr;
            rope_pair(x[i], x[i + HALF], cs[i], sn[i], yl, yr);
            const uint16_t bl = bf16_bits(yl), br = bf16_bits(yr);
            dst[lane + 32 * i] = bl;
            dst[lane + 32 * (i + HALF)] = br;
            if (cache != nullptr)
            {
                cache[lane + 32 * i] = bl;
                cache[lane + 32 * (i + HALF)] = br;
            }
        }
    }
    __syncthreads();
    uint32_t q[KP][4];
#pragma unroll
    for (int c = 0; c < KP; c++)
    {
        const uint4 x = *reinterpret_cast<const uint4*>(&sm.q[g][c * 32 + t * 8]);
        q[c][0] = x.x;
        q[c][1] = x.y;
        q[c][2] = x.z;
        q[c][3] = x.w;
    }

    // ---- scores ----
    const unsigned int srow = ad_score_row(row_cap);
    float m = -INFINITY, l = 0.f;    // of head g over the rows this lane sees
    auto score = [&](KTile& k, unsigned int r) {
        if (owner && pos - r < (unsigned int)AD_TILE)
        {
            const unsigned int at = pos - r;    // the new row, from shared memory
#pragma unroll
            for (int i = 0; i < 2; i++)
            {
                if (at == i * 8 + g)
                {
#pragma unroll
                    for (int c = 0; c < KP; c++)
                    {
#pragma unroll
                        for (int x = 0; x < 4; x++) { k[i][c][x] = reinterpret_cast<const uint32_t*>(sm.kn + c * 32 + t * 8)[x]; }
                    }
                }
            }
        }
        float s[2][2] = { { 0.f, 0.f }, { 0.f, 0.f } };    // [row half][rows 2t, 2t + 1] of head g
#pragma unroll
        for (int c = 0; c < KP; c++)
        {
#pragma unroll
            for (int x = 0; x < 4; x += 2)
            {
                ad_mma(s[0], q[c][x], q[c][x + 1], k[0][c][x], k[0][c][x + 1]);
                ad_mma(s[1], q[c][x], q[c][x + 1], k[1][c][x], k[1][c][x + 1]);
            }
        }
        load_k(k, r + 2 * STEP);
        ahead(K, r + 4 * STEP);
        float mn = m;
#pragma unroll
        for (int i = 0; i < 2; i++)
        {
#pragma unroll
            for (int j = 0; j < 2; j++)
            {
                s[i][j] = r + i * 8 + 2 * t + j < t1 ? bf16_round(__fmul_rn(p.scale, s[i][j])) : -INFINITY;
                mn = fmaxf(mn, s[i][j]);
            }
            if (g < (unsigned int)G) { *reinterpret_cast<uint32_t*>(scores + g * srow + (r - t0) + i * 8 + 2 * t) = ad_pack(s[i][0], s[i][1]); }
        }
        const float base = mn == -INFINITY ? 0.f : mn;
        l = l * __expf(m - base) + ((__expf(s[0][0] - base) + __expf(s[0][1] - base)) + (__expf(s[1][0] - base) + __expf(s[1][1] - base)));
        m = mn;
    };
    for (unsigned int r = mine; r < t1; r += 2 * STEP)
    {
        score(ka, r);
        if (r + STEP < t1) { score(kb, r + STEP); }
    }
    VTile va, vb;
    load_v(va, mine);
    load_v(vb, mine + STEP);
    ahead(V, mine + 2 * STEP);
    ahead(V, mine + 3 * STEP);
#pragma unroll
    for (int x = 1; x < 4; x <<= 1)
    {
        const float m2 = __shfl_xor_sync(0xFFFFFFFFu, m, x), l2 = __shfl_xor_sync(0xFFFFFFFFu, l, x);
        ad_merge(m, l, m2, l2);
    }
    if (t == 0)
    {
        sm.ml[warp][g][0] = m;
        sm.ml[warp][g][1] = l;
    }
    __syncthreads();
    asm volatile("barrier.cluster.wait.aligned;" ::: "memory");    // every CTA of the cluster runs
    for (unsigned int i = threadIdx.x; i < G * S; i += AD_THREADS)
    {
        const unsigned int h = i % G, to = i / G;
        m = sm.ml[0][h][0];
        l = sm.ml[0][h][1];
#pragma unroll
        for (int w = 1; w < AD_WARPS; w++) { ad_merge(m, l, sm.ml[w][h][0], sm.ml[w][h][1]); }
        float* dst = cluster.map_shared_rank(&sm.recv_ml[rank][h][0], to);
        dst[0] = m;
        dst[1] = l;
    }
    cluster.sync();
    m = -INFINITY;
    l = 0.f;
    if (g < (unsigned int)G)
    {
        for (unsigned int r = t; r < S; r += 4) { ad_merge(m, l, sm.recv_ml[r][g][0], sm.recv_ml[r][g][1]); }
    }
#pragma unroll
    for (int x = 1; x < 4; x <<= 1)
    {
        const float m2 = __shfl_xor_sync(0xFFFFFFFFu, m, x), l2 = __shfl_xor_sync(0xFFFFFFFFu, l, x);
        ad_merge(m, l, m2, l2);
    }
    const float inv = 1.0f / l;

    // ---- weights and values ----
    float o[VP * 8][2];
#pragma unroll
    for (int j = 0; j < VP * 8; j++) { o[j][0] = o[j][1] = 0.f; }
    auto value = [&](VTile& v, unsigned int r) {
        if (owner && pos - r < (unsigned int)AD_TILE)
        {
            const unsigned int at = pos - r;
#pragma unroll
            for (int i = 0; i < 4; i++)
            {
                if (at == 2 * t + (i & 1) + (i >> 1) * 8)
                {
#pragma unroll
                    for (int c = 0; c < VP; c++)
                    {
#pragma unroll
                        for (int x = 0; x < 4; x++) { v[i][c][x] = reinterpret_cast<const uint32_t*>(sm.vn + c * 64 + g * 8)[x]; }
                    }
                }
            }
        }
        uint32_t a[2] = { 0u, 0u };
        if (g < (unsigned int)G)
        {
#pragma unroll
            for (int i = 0; i < 2; i++)
            {
                const uint32_t z = *reinterpret_cast<const uint32_t*>(scores + g * srow + (r - t0) + i * 8 + 2 * t);
                a[i] = ad_pack(__fmul_rn(__expf(__uint_as_float(z << 16) - m), inv), __fmul_rn(__expf(__uint_as_float(z & 0xFFFF0000u) - m), inv));
            }
        }
#pragma unroll
        for (int c = 0; c < VP; c++)
        {
#pragma unroll
            for (int e = 0; e < 8; e++)    // n of fragment c * 8 + e is column (c * 8 + n) * 8 + e
            {
                const uint32_t sel = (e & 1) ? 0x7632u : 0x5410u;
                ad_mma(o[c * 8 + e], a[0], a[1], __byte_perm(v[0][c][e / 2], v[1][c][e / 2], sel), __byte_perm(v[2][c][e / 2], v[3][c][e / 2], sel));
            }
        }
        load_v(v, r + 2 * STEP);
        ahead(V, r + 4 * STEP);
    };
    for (unsigned int r = mine; r < t1; r += 2 * STEP)
    {
        value(va, r);
        if (r + STEP < t1) { value(vb, r + STEP); }
    }
    if (g < (unsigned int)G)
    {
#pragma unroll
        for (int c = 0; c < VP; c++)
        {
#pragma unroll
            for (int n = 0; n < 2; n++)
            {
                float* dst = &sm.om[warp][g][(c * 8 + 2 * t + n) * 8];
#pragma unroll
                for (int e = 0; e < 8; e += 4) { *reinterpret_cast<float4*>(dst + e) = make_float4(o[c * 8 + e][n], o[c * 8 + e + 1][n], o[c * 8 + e + 2][n], o[c * 8 + e + 3][n]); }
            }
        }
    }
    __syncthreads();

    // ---- warps -> CTA -> the CTA of the cluster that finishes the output ----
    constexpr unsigned int OUT = G * HD;
    const unsigned int share = (OUT + S - 1) / S;
    for (unsigned int i = threadIdx.x; i < OUT; i += AD_THREADS)
    {
        const unsigned int h = i / HD, d = i - h * HD, to = i / share;
        float sum = 0.f;
#pragma unroll
        for (int w = 0; w < AD_WARPS; w++) { sum += sm.om[w][h][d]; }
        *cluster.map_shared_rank(&sm.recv[rank * share + (i - to * share)], to) = sum;
    }
    cluster.sync();
    uint16_t* out = p.out + (size_t)b * p.ldo + (size_t)kvh * OUT;
    const unsigned int first = rank * share, count = first < OUT ? min(share, OUT - first) : 0u;
    for (unsigned int i = threadIdx.x; i < count; i += AD_THREADS)
    {
        float sum = 0.f;
        for (unsigned int r = 0; r < S; r++) { sum += sm.recv[r * share + i]; }
        out[first + i] = bf16_bits(sum);
    }
}

}    // namespace b200

// Linears of a few rows with BF16 weights (weight streaming, HBM-bound), and the linears of the float mode.
//
// The streaming kernel: eight warps, WK of which share 16 (or 2 x 16) output features and take the 64-wide k chunks in
// turn (all of them, or two where k is short).  A lane loads 32 bytes of weight row g and of row g + 8 straight into the A fragments
// of mma.m16n8k16 - the k order inside a chunk is permuted, identically for both operands, so that fragments are whole pieces of a
// row - and the rows of X are the eight B columns.  What bounds it is the stream of weights, and around it, in linears of a few
// microseconds, the chain from the previous kernel's end to the results: each chunk is requested a turn ahead into the registers of
// the chunk just used, the first ones of a dense member before the previous kernel of the stream has finished, a task's first ones
// while the sums of the task before it are made; what the results are added to is fetched before the products.  The warps' partial
// sums meet in shared memory.  At 8 rows, with two turns of two chunks, one CTA per task and no such prefetch, before: 2048 x 2048 3.9
// us, 5120 x 2048 8.4, 2048 x 6144 9.3, 32768 x 2048 27.5, gated 6144 x 2048 13.2; now 3.1, 7.4, 6.4, 24.6, 11.1.
#include "decoder_common.cuh"
#include "../gemv_decode.cuh"
#include "linear.cuh"

namespace b200
{

constexpr int LS_WARPS = 8;

struct LinearLaunch
{
    LinearMember m[LINEAR_MAX_MEMBERS];
    unsigned int count, blocks;
};

// 32 bytes of a weight row, read once
__device__ __forceinline__ void ldg_stream(const void* p, uint4& a, uint4& b)
{
    asm volatile("ld.global.nc.L1::no_allocate.L2::evict_first.v8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=r"(a.x), "=r"(a.y), "=r"(a.z), "=r"(a.w), "=r"(b.x), "=r"(b.y), "=r"(b.z), "=r"(b.w)
                 : "l"(p));
}

// What one CTA does at a time: C rows (from n0) of a CTA's share of the features of one group.
struct StreamTask
{
    unsigned int block, member, fc;    // fc: first feature of the CTA
    unsigned int group, row0, count, n0;
};

// NT: row groups of eight; RT: 16-feature tiles per warp; U: chunks per loop turn; WK: warps that share features; OCC: CTAs per SM.
// A warp adds up its chunks in k order and the warps' sums are added in warp order: the result depends on WK alone, and on no other
// choice below.
template <int NT, int RT, int U, int WK, int OCC>
__global__ void __launch_bounds__(32 * LS_WARPS, OCC) linear_stream_kernel(const __grid_constant__ LinearLaunch L)
{
    constexpr int R = 16 * RT, C = 8 * NT, NW = LS_WARPS, T = 32 * NW;
    constexpr int RED = NW * C * (R + 1);
    constexpr bool TWO = RED * 8 <= 24 * 1024;    // two places for the partial sums: one barrier per task instead of two
    constexpr int XD = U < 2 || (NT == 2 && U * RT > 2) || (NT == 4 && OCC == 2) ? 1 : 2;    // chunks of X in registers
    __shared__ float red_all[(TWO ? 2 : 1) * RED];
    const unsigned int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    const unsigned int wk = warp % WK, wf = warp / WK;
    grid_dependency_launch();
    bool waited = false;

    // The next task from `block` on (rows n0 ..) that has rows; false: none.  Which rows a group holds is the previous kernel's to say.
    auto find = [&](unsigned int block, StreamTask& k) {
        for (; block < L.blocks; block += gridDim.x)
        {
            unsigned int mi = 0;
            if (L.count > 1 && block >= L.m[1].block0) { mi = 1; }
            if (L.count > 2 && block >= L.m[2].block0) { mi = 2; }
            const LinearMember& m = L.m[mi];
            const unsigned int b = block - m.block0, fb = b % m.fblocks, slot = b / m.fblocks;
            k.block = block;
            k.member = mi;
            k.fc = fb * (activation_gated(m.activation) ? R / 2 : R) * (NW / WK);
            k.group = m.blocks > 1 ? slot : 0u;
            k.row0 = 0;
            k.count = m.rows;
            k.n0 = 0;
            if (m.group_offset != nullptr)
            {
                if (!waited)
                {
                    grid_dependency_wait();
                    waited = true;
                }
                const int id = m.active != nullptr ? m.active[slot] : (int)slot;
                if (id < 0) { continue; }
                k.group = (unsigned int)id;
                k.row0 = (unsigned int)m.group_offset[id];
                k.count = (unsigned int)m.group_offset[id + 1] - k.row0;
            }
            if (k.count != 0) { return true; }
        }
        return false;
    };
    const __nv_bfloat16* W = nullptr;
    unsigned int off[RT][2], chunks = 0;    // rows of the weights in 64 elements, of the task that is being loaded
    auto aim = [&](const StreamTask& k) {
        const LinearMember& m = L.m[k.member];
        const bool gated = activation_gated(m.activation);
        const unsigned int f0 = k.fc + wf * (gated ? R / 2 : R);
        W = (const __nv_bfloat16*)m.W + (size_t)k.group * m.group_rows * m.ldw + t * 16;
#pragma unroll
        for (int r = 0; r < RT; r++)
        {
#pragma unroll
            for (int h = 0; h < 2; h++)
            {
                unsigned int f = f0 + (gated ? 0 : r * 16) + g + h * 8;
                f = min(f, m.N - 1);    // rows past N: any valid row, the result is not stored
                off[r][h] = (f + (gated && r == 1 ? m.up_row : 0u)) * (m.ldw / 64);
            }
        }
        chunks = (m.K + 63) / 64;
    };
    // A chunk's weights are requested a whole turn before their use, into the registers of the chunk just used: of the next
    // task's where a task ends, so that the stream does not stop while sums are made.
    uint4 a[U][RT][2][2];
    auto load = [&](int u, unsigned int c) {
        if (c < chunks)
        {
#pragma unroll
            for (int r = 0; r < RT; r++)
            {
#pragma unroll
                for (int h = 0; h < 2; h++) { ldg_stream(W + ((size_t)off[r][h] + c) * 64, a[u][r][h][0], a[u][r][h][1]); }
            }
        }
    };
    StreamTask k;
    bool more = find(blockIdx.x, k);
    if (more)
    {
        aim(k);
#pragma unroll
        for (int u = 0; u < U; u++) { load(u, wk + u * WK); }
    }
    if (!waited) { grid_dependency_wait(); }
    waited = true;
    for (unsigned int turn_of_red = 0; more; turn_of_red ^= 1)
    {
        const LinearMember& m = L.m[k.member];
        float* red = red_all + (TWO ? turn_of_red * RED : 0);
        const bool gated = activation_gated(m.activation);
        const unsigned int xcol = m.blocks > 1 ? k.group * m.x_step : 0u, ycol = m.blocks > 1 ? k.group * m.y_step : 0u;
        const __nv_bfloat16* xr[NT];
        bool live[NT];
#pragma unroll
        for (int nt = 0; nt < NT; nt++)
        {
            const unsigned int n = k.n0 + nt * 8 + g;
            live[nt] = n < k.count;
            unsigned int r = k.row0 + (live[nt] ? n : 0u);
            if (m.x_row != nullptr) { r = (unsigned int)m.x_row[r]; }
            xr[nt] = (const __nv_bfloat16*)m.X + (size_t)r * m.ldx + xcol + t * 16;
        }
        const unsigned int here = chunks;
        uint4 x[XD][NT][2];
        auto load_x = [&](int d, unsigned int c) {
#pragma unroll
            for (int nt = 0; nt < NT; nt++)
            {
#pragma unroll
                for (int q = 0; q < 2; q++)
                {
                    x[d][nt][q] = make_uint4(0, 0, 0, 0);
                    if (live[nt] && c < here) { x[d][nt][q] = *reinterpret_cast<const uint4*>(xr[nt] + c * 64 + q * 8); }
                }
            }
        };
#pragma unroll
        for (int d = 0; d < XD; d++) { load_x(d, wk + d * WK); }
        // What the results are added to, fetched while the products are made; not in the forms of gated launches, which have no register
        // left and as good as never add.
        constexpr bool EARLY = RT == 1 || NT == 4;
        const unsigned int cols = min((unsigned int)C, k.count - k.n0);
        const unsigned int F = gated ? R / 2 : R, all = F * (NW / WK);    // output features of a warp, of the CTA
        float old = 0.f;
        const bool adds = EARLY && m.accumulate != 0 && threadIdx.x < cols * all && k.fc + threadIdx.x % all < m.N;
        if (adds) { old = ((const float*)m.Y)[(size_t)(k.row0 + k.n0 + threadIdx.x / all) * m.ldy + ycol + k.fc + threadIdx.x % all]; }
        // the task after this one
        StreamTask nk = k;
        bool again = true;
        if (k.n0 + C < k.count) { nk.n0 = k.n0 + C; }
        else { again = find(k.block + gridDim.x, nk); }

        float acc[RT][NT][4];
#pragma unroll
        for (int r = 0; r < RT; r++)
        {
#pragma unroll
            for (int nt = 0; nt < NT; nt++)
            {
#pragma unroll
                for (int j = 0; j < 4; j++) { acc[r][nt][j] = 0.f; }
            }
        }
        const unsigned int turns = (here + U * WK - 1) / (U * WK);    // the same for every warp
        for (unsigned int turn = 0; turn < turns; turn++)
        {
            const unsigned int c0 = wk + turn * (U * WK);
            const bool last = turn + 1 == turns;
            if (last && again) { aim(nk); }
            const unsigned int next = last ? wk : c0 + U * WK;
#pragma unroll
            for (int u = 0; u < U; u++)
            {
                if (c0 + u * WK < here)
                {
#pragma unroll
                    for (int nt = 0; nt < NT; nt++)
                    {
#pragma unroll
                        for (int q = 0; q < 2; q++)
                        {
                            const uint4 b = x[u % XD][nt][q];
#pragma unroll
                            for (int r = 0; r < RT; r++)
                            {
                                mma_bf16_16816(acc[r][nt], a[u][r][0][q].x, a[u][r][1][q].x, a[u][r][0][q].y, a[u][r][1][q].y, b.x, b.y);
                                mma_bf16_16816(acc[r][nt], a[u][r][0][q].z, a[u][r][1][q].z, a[u][r][0][q].w, a[u][r][1][q].w, b.z, b.w);
                            }
                        }
                    }
                }
                if (XD == 1) { load_x(0, c0 + (u + 1) * WK); }
                if (!last || again) { load(u, next + u * WK); }
                if (XD != 1) { load_x(u % XD, c0 + (u + XD) * WK); }
            }
        }
        if (!TWO) { __syncthreads(); }    // the last task's sums have been read
#pragma unroll
        for (int r = 0; r < RT; r++)
        {
#pragma unroll
            for (int nt = 0; nt < NT; nt++)
            {
#pragma unroll
                for (int j = 0; j < 4; j++) { red[(warp * C + nt * 8 + 2 * t + (j & 1)) * (R + 1) + r * 16 + g + 8 * (j >> 1)] = acc[r][nt][j]; }
            }
        }
        __syncthreads();
        for (unsigned int i = threadIdx.x; i < cols * all; i += T)
        {
            const unsigned int f = i % all, n = i / all, w0 = f / F * WK, fl = f % F;
            if (k.fc + f >= m.N) { continue; }
            float v = 0.f, up = 0.f;
#pragma unroll
            for (int w = 0; w < WK; w++) { v += red[((w0 + w) * C + n) * (R + 1) + fl]; }
            if (gated)
            {
#pragma unroll
                for (int w = 0; w < WK; w++) { up += red[((w0 + w) * C + n) * (R + 1) + (RT == 2 ? 16 : 0) + fl]; }
            }
            const unsigned int row = k.row0 + k.n0 + n;
            const float y = linear_activation<true>(m.activation, m.alpha * v, m.alpha * up, m.cap) * linear_row_factor<__nv_bfloat16>(m, row, k.group);
            if (adds && i == threadIdx.x) { ((float*)m.Y)[(size_t)row * m.ldy + ycol + k.fc + f] = old + y; }
            else { linear_store(m, row, ycol + k.fc + f, y); }
        }
        k = nk;
        more = again;
    }
}

// ---- the float mode: a plain tiled product in true float -------------------------------------------
constexpr int LF_F = 64, LF_R = 32, LF_K = 32;

template <bool GATED>
__global__ void __launch_bounds__(256) linear_f32_kernel(const LinearMember m)
{
    __shared__ float ws[GATED ? 2 : 1][LF_K][LF_F + 1];
    __shared__ float xs[LF_K][LF_R + 1];
    grid_dependency_launch();
    grid_dependency_wait();
    unsigned int group = 0, row0 = 0, count = m.rows;
    if (m.group_offset != nullptr)
    {
        group = blockIdx.z;
        row0 = (unsigned int)m.group_offset[group];
        count = (unsigned int)m.group_offset[group + 1] - row0;
    }
    const unsigned int f0 = blockIdx.x * LF_F, r0 = blockIdx.y * LF_R;
    if (r0 >= count) { return; }
    if (m.blocks > 1) { group = blockIdx.z; }
    const float* W = (const float*)m.W + (size_t)group * m.group_rows * m.ldw;
    const unsigned int xcol = m.blocks > 1 ? group * m.x_step : 0u, ycol = m.blocks > 1 ? group * m.y_step : 0u;
    const unsigned int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;    // 16 x 16 threads: 4 features x 2 rows each
    float acc[GATED ? 2 : 1][2][4] = {};
    for (unsigned int k0 = 0; k0 < m.K; k0 += LF_K)
    {
        for (unsigned int i = threadIdx.x; i < LF_F * LF_K; i += 256)
        {
            const unsigned int k = i % LF_K, f = i / LF_K;
            const bool ok = k0 + k < m.K && f0 + f < m.N;
            ws[0][k][f] = ok ? W[(size_t)(f0 + f) * m.ldw + k0 + k] : 0.f;
            if (GATED) { ws[GATED ? 1 : 0][k][f] = ok ? W[(size_t)(m.up_row + f0 + f) * m.ldw + k0 + k] : 0.f; }
        }
        for (unsigned int i = threadIdx.x; i < LF_R * LF_K; i += 256)
        {
            const unsigned int k = i % LF_K, r = i / LF_K;
            float v = 0.f;
            if (k0 + k < m.K && r0 + r < count)
            {
                unsigned int xr = row0 + r0 + r;
                if (m.x_row != nullptr) { xr = (unsigned int)m.x_row[xr]; }
                v = ((const float*)m.X)[(size_t)xr * m.ldx + xcol + k0 + k];
            }
            xs[k][r] = v;
        }
        __syncthreads();
#pragma unroll 8
        for (int k = 0; k < LF_K; k++)
        {
#pragma unroll
            for (int i = 0; i < 2; i++)
            {
                const float x = xs[k][ty + 16 * i];
#pragma unroll
                for (int j = 0; j < 4; j++)
                {
                    acc[0][i][j] = fmaf(ws[0][k][tx + 16 * j], x, acc[0][i][j]);
                    if (GATED) { acc[GATED ? 1 : 0][i][j] = fmaf(ws[GATED ? 1 : 0][k][tx + 16 * j], x, acc[GATED ? 1 : 0][i][j]); }
                }
            }
        }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < 2; i++)
    {
#pragma unroll
        for (int j = 0; j < 4; j++)
        {
            const unsigned int r = r0 + ty + 16 * i, f = f0 + tx + 16 * j;
            if (r < count && f < m.N)
            {
                const float y = linear_activation<false>(m.activation, m.alpha * acc[0][i][j], GATED ? m.alpha * acc[GATED ? 1 : 0][i][j] : 0.f, m.cap);
                linear_store(m, row0 + r, ycol + f, y * linear_row_factor<float>(m, row0 + r, group));
            }
        }
    }
}

template <int NT, int RT, int U, int WK, int OCC>
static int launch_stream_wk(LinearLaunch& L, unsigned int sm_count, unsigned int waves, cudaStream_t st, bool pdl)
{
    L.blocks = 0;
    for (unsigned int j = 0; j < L.count; j++)
    {
        LinearMember& m = L.m[j];
        const unsigned int F = (activation_gated(m.activation) ? 8 * RT : 16 * RT) * (LS_WARPS / WK);
        m.fblocks = (m.N + F - 1) / F;
        m.block0 = L.blocks;
        L.blocks += m.fblocks * m.slots;
    }
    const unsigned int places = sm_count * OCC;
    // The rows of X are read through L1, of which a kernel with much shared memory just before would otherwise leave little.
    static std::atomic<unsigned long long> done{ 0 };
    prefer_l1(linear_stream_kernel<NT, RT, U, WK, OCC>, done);
    const unsigned int grid = L.blocks > places && L.blocks / places < waves ? places : L.blocks;
    return launch_kernel("linear_stream", linear_stream_kernel<NT, RT, U, WK, OCC>, dim3(grid), dim3(32 * LS_WARPS), 0, st, pdl, L);
}

// Which form a launch takes (one linear in a CUDA graph of distinct weights, us; "few": a launch has no more tasks than there are SMs).
//   * Two warps over k up to 1024, eight beyond: the bits follow this alone.
//   * Few tasks: one CTA per SM with twice the chunks in flight, or four times (8 rows, one CTA / two: 2048 x 768 2.8 / 3.9, 8192 x 1024 4.8 / 5.9, gated 4096 x 512
//     3.4 / 4.4, 2048 x 6144 6.3 / 7.2; 16 rows: 8192 x 1024 7.0 / 7.6, gated 1024 x 4096 8.4 / 10.8).  Not where k is short enough to be under way whole with two: 512 x
//     8192 at 8 rows 3.4 / 3.3.
//   * More tasks, up to 8 rows, two warps over k: four chunks where a warp's chunks are whole fours, else two (32768 x 1024 14.3 / 14.9, 32768 x 768 12.0 / 11.8, the
//     down projections of 16 experts, k 768, 13.0 / 12.0).  Eight warps: a whole k of 2048 (four per warp), two chunks where k is longer (4096 x 12288 20.5 with
//     four, 18.1; 151936 x 4096 218, 202.5).
//   * CTAs that take task after task (up to so many rounds), or one for each task?  Taking the next task hides its first loads behind this one's sums, a CTA of its own
//     fits itself to what an SM gets done.  Up to 8 rows two warps over k gain in the second round (32768 x 1024: 14.0 against 14.8) and lose beyond (experts, 1024
//     tasks, k 1024: 26.1 against 24.8), dense tasks of eight warps gain nothing (5120 x 2048 at 1 row 7.3 against 6.0; 32768 x 2048 28.4 against 25.1), gated ones of eight
//     warps do up to four rounds (6144 x 2048 11.1 against 12.0), of two warps they lose (64 experts of 512, k 1024, at 32 tokens: 28.4 against 24.3).  More rows gain
//     at any number (32768 x 2048: 28.7 / 45.8 at 16 / 32 rows against 30.1 / 51.3).
//   * Registers: gated 9 to 16 rows hold one chunk on two CTAs per SM (two chunks spill: 12288 x 4096 at 9 / 16 rows 39.4 / 40.1 with one, 42.2 / 43.1 with two); 17 to 32 rows of
//     two warps that are not gated hold 16 features a warp on two CTAs (32 features on one: 32768 x 1024 at 32 rows 24.8 / 29.1, 2048 x 512, few, 6.0 / 10.2).
template <int NT, int RT>
static int launch_stream(LinearLaunch& L, cudaStream_t st, bool pdl)
{
    const DecoderDevice* dev = decoder_device();
    if (!dev) { return 1; }
    constexpr unsigned int EVERY = 0xFFFFFFFFu;
    const unsigned int sms = (unsigned int)dev->sm_count;
    unsigned int longest = 0;
    for (unsigned int j = 0; j < L.count; j++) { longest = L.m[j].K > longest ? L.m[j].K : longest; }
    // eight warps over few chunks would leave some without any; the members of a launch take one form
    const bool two = longest <= 1024;
    if constexpr (NT == 4 && RT == 1)
    {
        if (!two) { return launch_stream<4, 2>(L, st, pdl); }
    }
    unsigned int tasks = 0;
    for (unsigned int j = 0; j < L.count; j++)
    {
        const LinearMember& m = L.m[j];
        const unsigned int F = (activation_gated(m.activation) ? 8 * RT : 16 * RT) * (two ? LS_WARPS / 2 : 1);
        tasks += (m.N + F - 1) / F * m.slots;
    }
    const bool few = tasks <= sms;
    if constexpr (NT == 1 && RT == 1)
    {
        if (two)
        {
            const unsigned int own = ((longest + 63) / 64 + 1) / 2;    // chunks of a warp
            if (few && own > 4) { return launch_stream_wk<1, 1, 8, 2, 1>(L, sms, 1, st, pdl); }
            return own <= 4 || own % 4 == 0 ? launch_stream_wk<1, 1, 4, 2, 2>(L, sms, 2, st, pdl) : launch_stream_wk<1, 1, 2, 2, 2>(L, sms, 2, st, pdl);
        }
        if (few && longest >= 4096) { return launch_stream_wk<1, 1, 8, 8, 1>(L, sms, 1, st, pdl); }
        return longest > 2048 ? launch_stream_wk<1, 1, 2, 8, 2>(L, sms, 1, st, pdl) : launch_stream_wk<1, 1, 4, 8, 2>(L, sms, 1, st, pdl);
    }
    else if constexpr (NT == 1)
    {
        if (two) { return few ? launch_stream_wk<1, 2, 4, 2, 1>(L, sms, 1, st, pdl) : launch_stream_wk<1, 2, 2, 2, 2>(L, sms, 1, st, pdl); }
        return few && longest >= 4096 ? launch_stream_wk<1, 2, 4, 8, 1>(L, sms, 1, st, pdl) : launch_stream_wk<1, 2, 2, 8, 2>(L, sms, 4, st, pdl);
    }
    else if constexpr (NT == 2 && RT == 1)
    {
        if (two && few) { return launch_stream_wk<2, 1, 4, 2, 1>(L, sms, EVERY, st, pdl); }
        return two ? launch_stream_wk<2, 1, 2, 2, 2>(L, sms, EVERY, st, pdl) : launch_stream_wk<2, 1, 2, 8, 2>(L, sms, EVERY, st, pdl);
    }
    else if constexpr (NT == 2)
    {
        if (few) { return two ? launch_stream_wk<2, 2, 4, 2, 1>(L, sms, EVERY, st, pdl) : launch_stream_wk<2, 2, 4, 8, 1>(L, sms, EVERY, st, pdl); }
        return two ? launch_stream_wk<2, 2, 1, 2, 2>(L, sms, EVERY, st, pdl) : launch_stream_wk<2, 2, 1, 8, 2>(L, sms, EVERY, st, pdl);
    }
    else if constexpr (RT == 1)
    {
        return few ? launch_stream_wk<4, 1, 4, 2, 1>(L, sms, EVERY, st, pdl) : launch_stream_wk<4, 1, 2, 2, 2>(L, sms, EVERY, st, pdl);
    }
    else { return two ? launch_stream_wk<4, 2, 2, 2, 1>(L, sms, EVERY, st, pdl) : launch_stream_wk<4, 2, 2, 8, 1>(L, sms, EVERY, st, pdl); }
}

}    // namespace b200

using namespace b200;

C_EXPORT int cuda_b200_linear_rows(int dtype, unsigned int count, const cuda_b200_linear* members, void* stream, unsigned int flags, int kernel)
{
    if (count == 0) { return 0; }
    if (!members || count > LINEAR_MAX_MEMBERS || (dtype != DT_BF16 && dtype != DT_FLOAT)) { return -1; }
    LinearLaunch L;
    memset(&L, 0, sizeof(L));
    unsigned int most = 0, group_max[LINEAR_MAX_MEMBERS] = {};
    for (unsigned int j = 0; j < count; j++)
    {
        const cuda_b200_linear& a = members[j];
        if (a.rows == 0 || a.N == 0) { continue; }
        auto bad_align = [](const void* q) { return (reinterpret_cast<uintptr_t>(q) & 31u) != 0; };
        if (!a.W || !a.X || !a.Y || a.K == 0 || bad_align(a.W) || bad_align(a.X)) { return -1; }
        if (a.activation < B200_ACT_NONE || a.activation > B200_ACT_SOFTCAP || (a.out_type != DT_FLOAT && a.out_type != DT_BF16)) { return -1; }
        if (a.accumulate && a.out_type != DT_FLOAT) { return -1; }
        if (dtype == DT_FLOAT && a.out_type != DT_FLOAT) { return -1; }
        const unsigned int kp = (a.K + 63) / 64 * 64;
        if ((a.ldw % 64) || (a.ldx % 64) || a.ldw < kp || a.ldx < kp) { return -1; }
        if (a.group_offset && (a.groups == 0 || a.group_max == 0 || a.blocks > 1)) { return -1; }
        if (a.blocks > 1 && ((a.x_step % 8) || a.x_row)) { return -1; }
        if (a.activation == B200_ACT_SOFTCAP && !(a.cap > 0.f)) { return -1; }
        if (a.tail && (!a.Y_tail || a.accumulate || a.blocks > 1 || a.group_offset || a.activation != B200_ACT_NONE)) { return -1; }
        LinearMember& m = L.m[L.count++];
        m.W = a.W;
        m.X = a.X;
        m.Y = a.Y;
        m.row_scale = (const float*)a.row_scale;
        m.group_offset = (const int*)a.group_offset;
        m.x_row = (const int*)a.x_row;
        m.active = (const int*)a.active;
        m.rows = a.rows;
        m.N = a.N;
        m.K = a.K;
        m.ldw = a.ldw;
        m.ldx = a.ldx;
        m.ldy = a.ldy;
        m.groups = a.group_offset ? a.groups : 1;
        m.group_rows = a.group_rows;
        m.up_row = a.up_row;
        m.blocks = a.blocks > 1 ? a.blocks : 1;
        m.x_step = a.x_step;
        m.y_step = a.y_step;
        m.head_gate = a.head_gate;
        m.ld_gate = a.ld_gate;
        m.Y_tail = (float*)a.Y_tail;
        m.tail = a.tail ? a.tail : 0xFFFFFFFFu;
        m.ld_tail = a.ld_tail;
        m.cap = a.cap;
        m.slots = a.group_offset ? (a.active ? a.active_cap : a.groups) : m.blocks;
        m.out_type = a.out_type;
        m.activation = a.activation;
        m.accumulate = a.accumulate;
        m.alpha = a.alpha;
        if (m.slots == 0) { return -1; }
        group_max[L.count - 1] = a.group_max;
        const unsigned int rows = a.group_offset ? a.group_max : a.rows;
        most = rows > most ? rows : most;
    }
    if (L.count == 0) { return 0; }
    const bool pdl = (flags & 1u) != 0;
    cudaStream_t st = (cudaStream_t)stream;
    if (dtype == DT_FLOAT)
    {
        for (unsigned int j = 0; j < L.count; j++)
        {
            const LinearMember& m = L.m[j];
            const unsigned int rows = m.group_offset ? (most < m.rows ? most : m.rows) : m.rows;
            const dim3 grid((m.N + LF_F - 1) / LF_F, (rows + LF_R - 1) / LF_R, m.blocks > 1 ? m.blocks : m.groups);
            if (grid.y > 65535u || grid.z > 65535u) { return -1; }
            const int rc = activation_gated(m.activation) ? launch_kernel("linear_f32", linear_f32_kernel<true>, grid, dim3(256), 0, st, pdl, m)
                                                              : launch_kernel("linear_f32", linear_f32_kernel<false>, grid, dim3(256), 0, st, pdl, m);
            if (rc) { return rc; }
        }
        return 0;
    }
    // a dense linear of 17 to 32 rows with a tile for every SM (a head over a vocabulary): tiles stream weights as fast
    if (kernel == 0 && L.count == 1 && most > 16 && L.m[0].blocks == 1 && !L.m[0].group_offset && !L.m[0].x_row)
    {
        const DecoderDevice* dev = decoder_device();
        if (dev && L.m[0].N >= 256u * (unsigned int)dev->sm_count) { kernel = 2; }
    }
    if (kernel == 1 || (kernel == 0 && most <= 32))
    {
        // Members whose groups hold about as many rows share a launch: 8, 16 or 32 rows at a time.  A group with more rows
        // than that reads its weights again, so experts go by twice their mean.
        for (unsigned int width = 8; width <= 32; width *= 2)
        {
            LinearLaunch part;
            memset(&part, 0, sizeof(part));
            bool gated = false;
            for (unsigned int j = 0; j < L.count; j++)
            {
                const LinearMember& m = L.m[j];
                unsigned int rows = m.rows;
                if (m.group_offset)
                {
                    rows = 2 * ((m.rows + m.slots - 1) / m.slots);
                    if (rows > group_max[j]) { rows = group_max[j]; }
                }
                if (width < 32 ? rows > width : false) { continue; }
                if (width > 8 && rows <= width / 2) { continue; }
                part.m[part.count++] = m;
                gated = gated || activation_gated(m.activation);
            }
            if (part.count == 0) { continue; }
            int rc;
            if (width == 8) { rc = gated ? launch_stream<1, 2>(part, st, pdl) : launch_stream<1, 1>(part, st, pdl); }
            else if (width == 16) { rc = gated ? launch_stream<2, 2>(part, st, pdl) : launch_stream<2, 1>(part, st, pdl); }
            else { rc = gated ? launch_stream<4, 2>(part, st, pdl) : launch_stream<4, 1>(part, st, pdl); }
            if (rc) { return rc; }
        }
        return 0;
    }
    for (unsigned int j = 0; j < L.count; j++)
    {
        const int rc = launch_linear_tile(L.m[j], st, pdl);
        if (rc) { return rc; }
    }
    return 0;
}

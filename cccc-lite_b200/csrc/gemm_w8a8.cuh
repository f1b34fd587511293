// W8A8: E4M3 weights times E4M3 ACTIVATIONS (one scale for the whole activation tensor) with FP32 accumulation, the mode
// the reference selects with act_data_type = FP8_E4M3 (cccc/cublas_real.h:619-666: quantise the BF16 activations, static
// scale or dynamic absmax, then a cublasLt FP8 x FP8 matmul with both scales).  Here the quantised activations are one
// E4M3 row per token of the native-operand FP8 kernel (gemm_native.cuh, PIECES = 1): both operands go into
// tcgen05.mma kind::f8f6f4 as they are.  More tokens (24 and up) run with k slices (gemm_w8a8_split.cuh) or on CTA pairs
// (gemm_w8a8_pair.cuh).
#pragma once

#include "gemm_native.cuh"
#include "gemm_w8a8_pair.cuh"
#include "gemm_w8a8_split.cuh"

namespace b200
{

constexpr int W8A8_MAX_TOKENS = 32;    // what the streaming kernel takes (all SMs share the k range)

// Do k slices take what the streaming kernel would?  From 24 tokens on they are as fast or faster on every linear of a layer and on
// a head (dynamic, streaming / slices, us: 4096 x 4096 at 24 / 32 tokens 16.6 / 10.7, 17.7 / 11.0; 24576 x 4096 24.7 / 24.3,
// 25.5 / 23.8; 4096 x 12288 22.9 / 17.8, 24.3 / 18.4; 151936 x 4096 107.9 / 104.3, 109.9 / 105.8); at 17 tokens 24576 x 4096 takes
// 24.0 / 26.0, at 16 151936 x 4096 106.4 / 122.3.  Small tensors keep the quantiser that finds the maximum itself.
static inline bool w8a8_split_early(unsigned int M, unsigned int K) { return M >= 24 && (size_t)M * K > 16384; }

// More tokens: k slices, or CTA pairs?  Up to 64 the slices win on every linear of a layer (gemm_w8a8_split.cuh) and on 65536 features
// (K 4096: 57.1 against 52.4 us).  Above, where k is long and the tiles (128 features x 128 tokens, one CTA per SM) are few, the pairs
// leave the GPU idle; where they are many, the slices read a weight once per token tile and run in waves.  Measured (static scale,
// quantiser included, K = 8192, pairs' best form / slices, us):
//   up to 128 tokens, by tiles:  8 22.9 / 12.8,  32 23.4 / 14.9,  64 25.1 / 21.0,  80 27.0 / 28.2,  112 32.1 / 31.8,  148 37.7 / 36.6,
//     160 44.8 / 57.0,  224 52.6 / 59.5,  448 97.7 / 114.1;
//   129 tokens, by tiles (two per 128 features):  16 23.2 / 13.1,  64 23.7 / 19.1,  128 25.5 / 28.3,  160 27.2 / 42.2,  448 53.0 / 103.9;
//   256 tokens:  64 28.1 / 19.7,  128 30.3 / 28.9,  160 31.8 / 51.9.  (K = 12288 to 28672: the same sides, few tiles gain more.)
// Hence above 128 tokens as long as every tile gets two slices, which then run at once; up to 128 tokens to five quarters of a wave, which is behind
// what would be the best line, one wave.
// Shorter k: up to 128 tokens, where the tiles leave more than half of the SMs idle.  Dynamic scale, K = 4096, pairs / slices at 65 / 80 / 100 / 128 tokens:
//   256 features 15.5 / 11.5, 15.5 / 11.1, 16.4 / 12.8, 16.0 / 13.0;  1024 14.7 / 11.0, 15.0 / 11.5, 16.1 / 12.6, 16.6 / 13.6;
//   4096 15.2 / 13.7, 15.5 / 14.0, 15.8 / 13.4, 17.0 / 14.2;  6144 15.7 / 15.7, 16.1 / 16.0, 16.3 / 17.4, 17.5 / 18.3;
//   7168 15.9 / 16.5, 16.4 / 17.0, 18.1 / 17.7, 18.5 / 18.5;  8448 16.4 / 15.7, 17.5 / 16.0, 18.6 / 17.1, 19.1 / 17.9;  12288 18.9 / 19.6 at 65, 20.2 / 22.5 at 128.
// Between 4608 and 7168 features the pairs are up to 6 % ahead.  The line does not lie there because it would part a layer's q from its k and v, which then are two
// launches (q + k + v of 4096 + 512 + 512 features 23.1 at 65 tokens and 25.2 at 128; on pairs 15.5 and 17.2, in slices 15.2 and 17.9), and because a layer gains:
// the four calls of a Qwen3-8B layer 80.4 / 79.3, 81.4 / 79.9, 84.5 / 80.9, 88.5 / 85.0, of a Llama-3.1-8B layer 83.2 / 81.5, 85.2 / 83.5, 87.9 / 84.4, 92.1 / 89.0.
// Above 128 tokens 4096 features gain (20.8 / 17.8 at 256) less than q, k and v together lose (19.3 / 21.6 at 200), and at K = 2048 the pairs are ahead (4096
// features at 128 11.8 / 13.5).  A single tile keeps the pairs, which the tests hold; no layer has one beside a wider member but for a single kv head of 128.
// A feature's bits are the same in every matrix that takes the same kernel: from 24 to 64 tokens in all; to 128 tokens in all of 129 to 8448 features with K from 4096 to
// 8191 and of up to 20480 with K from 8192 (the tests hold both); to 256 in all of up to 4224 with K from 8192; otherwise (K below 4096, or more tokens) in all.
static inline bool w8a8_split_preferred(unsigned int M, unsigned int K, unsigned int N, int sm_count)
{
    if (M <= 64) { return true; }
    const unsigned long long tiles = (unsigned long long)((N + 127) / 128) * ((M + 127) / 128), sms = (unsigned)sm_count;
    if (K < 8192) { return K >= 4096 && M <= 128 && tiles >= 2 && 20 * tiles <= 9 * sms; }
    if (M > 256) { return false; }
    return M <= 128 ? 4 * tiles <= 5 * sms : 20 * tiles <= 9 * sms;
}

static inline int w8a8_launch_failed()
{
    report_launch("gemm_w8a8_bf16");
    return 1;
}

// Largest |x| over a [rows][cols] BF16 tensor (leading dimension ld) into *absmax (zero before), as the reference's
// absmax_bf16_kernel computes it (cccc-cuda/cuda_functions.cu:2611-2637): fmaxf over |x|, which skips NaN and keeps an
// infinity.  Non-negative floats order as their bits, so the device-wide step is an integer atomicMax.
static __global__ void __launch_bounds__(256) absmax_bf16_rows_kernel(const uint16_t* __restrict__ X, unsigned int ld, unsigned int cols,
    unsigned int rows, float* __restrict__ absmax)
{
    __shared__ unsigned int warp_max[8];
    const unsigned int tid = threadIdx.x;
    unsigned int m = 0;
    for (unsigned int r = blockIdx.y; r < rows; r += gridDim.y)
    {
        const uint16_t* x = X + (size_t)r * ld;
        for (unsigned int i = blockIdx.x * 256 + tid; i < cols; i += gridDim.x * 256)
        {
            const unsigned int b = x[i] & 0x7FFFu;
            if (b <= 0x7F80u) { m = max(m, b); }
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) { m = max(m, __shfl_xor_sync(0xFFFFFFFFu, m, o)); }
    if ((tid & 31u) == 0) { warp_max[tid >> 5] = m; }
    __syncthreads();
    if (tid == 0)
    {
#pragma unroll
        for (int w = 1; w < 8; w++) { m = max(m, warp_max[w]); }
        atomicMax(reinterpret_cast<unsigned int*>(absmax), m << 16);
    }
}

// The largest of n (at most W8A8_MAX_BLOCKS) non-negative floats, for every thread of a block of 256.
constexpr unsigned int W8A8_MAX_BLOCKS = 148;
__device__ __forceinline__ float block_maximum(const float* v, unsigned int n)
{
    __shared__ unsigned int of_warp[8];
    unsigned int m = threadIdx.x < n ? __float_as_uint(v[threadIdx.x]) : 0u;    // they order as their bits
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) { m = max(m, __shfl_xor_sync(0xFFFFFFFFu, m, o)); }
    if ((threadIdx.x & 31u) == 0) { of_warp[threadIdx.x >> 5] = m; }
    __syncthreads();
#pragma unroll
    for (int w = 0; w < 8; w++) { m = max(m, of_warp[w]); }
    return __uint_as_float(m);
}

// BF16 -> E4M3 with the reference's encoder (float_to_e4m3, cuda_functions.cu:2551-2580).  Dynamic (fwd_static == 0):
// scale = 448 / absmax, multiplier back = absmax / 448 (1 and 1 for an all-zero tensor), cuda_functions.cu:2640-2657;
// static: fwd_static = 1 / act_scale, multiplier back = inv_static = act_scale (cublas_real.h:627-632).
// Grid (column chunks, rows + padding rows): rows past `rows` are written as zeros.  inv_out[r] receives the multiplier
// back for each of the first n_inv rows (the linear reads one per token); pass n_inv = 1 for a single word.
static __global__ void __launch_bounds__(256) quantise_activations_kernel(const uint16_t* __restrict__ X, unsigned int ld, unsigned int cols,
    unsigned int rows, uint8_t* __restrict__ Q, unsigned int ldq, const float* __restrict__ absmax, unsigned int n_max, float fwd_static,
    float inv_static, float* __restrict__ inv_out, unsigned int n_inv, bool pdl, bool src_is_e4m3)
{
    if (pdl)
    {
        pdl_launch_dependents();
        pdl_wait();
    }
    if (src_is_e4m3)
    {
        // the activations are E4M3 already (ld in bytes): they are only moved into the padded rows the linear reads
        const unsigned int r = blockIdx.y, i = blockIdx.x * 256 + threadIdx.x;
        if (blockIdx.x == 0 && threadIdx.x == 0 && r < n_inv) { inv_out[r] = inv_static; }
        if (i < cols) { Q[(size_t)r * ldq + i] = r < rows ? reinterpret_cast<const uint8_t*>(X)[(size_t)r * ld + i] : (uint8_t)0; }
        return;
    }
    float fwd = fwd_static, inv = inv_static;
    if (fwd_static == 0.f)
    {
        float a;
        if (absmax && n_max == 1) { a = *absmax; }
        else if (absmax) { a = block_maximum(absmax, n_max); }
        else
        {
            // a small tensor: every block that quantises finds the largest magnitude itself (eight values per load; the
            // maximum does not depend on the order), which saves the memset and the absmax launch
            __shared__ unsigned int warp_max[8];
            unsigned int m = 0;
            if (blockIdx.y < rows)
            {
                const unsigned int per_row = cols / 8;
                for (unsigned int j = threadIdx.x; j < rows * per_row; j += 256)
                {
                    const uint4 v = *reinterpret_cast<const uint4*>(X + (size_t)(j / per_row) * ld + (size_t)(j % per_row) * 8);
                    const unsigned int w[4] = { v.x, v.y, v.z, v.w };
#pragma unroll
                    for (int q = 0; q < 4; q++)
                    {
                        const unsigned int lo = w[q] & 0x7FFFu, hi = (w[q] >> 16) & 0x7FFFu;
                        if (lo <= 0x7F80u) { m = max(m, lo); }
                        if (hi <= 0x7F80u) { m = max(m, hi); }
                    }
                }
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) { m = max(m, __shfl_xor_sync(0xFFFFFFFFu, m, o)); }
            if ((threadIdx.x & 31u) == 0) { warp_max[threadIdx.x >> 5] = m; }
            __syncthreads();
#pragma unroll
            for (int w = 0; w < 8; w++) { m = max(m, warp_max[w]); }
            a = __uint_as_float(m << 16);
        }
        fwd = (a > 0.f) ? (448.0f / a) : 1.0f;
        inv = (a > 0.f) ? (a / 448.0f) : 1.0f;
    }
    const unsigned int r = blockIdx.y, i = blockIdx.x * 256 + threadIdx.x;
    if (blockIdx.x == 0 && threadIdx.x == 0 && r < n_inv) { inv_out[r] = inv; }
    if (i >= cols) { return; }
    Q[(size_t)r * ldq + i] = r < rows ? float_to_e4m3(bf16_bits_to_float(X[(size_t)r * ld + i]), fwd) : (uint8_t)0;
}

// The same two steps, eight values per thread and access (16-byte loads; cols and ld multiples of 8, aligned bases).  The
// largest magnitudes of up to W8A8_MAX_BLOCKS blocks go side by side instead of into one word by atomicMax: nothing has to be
// cleared first, which took a memset of 1.5 us and a gap per call.
static __global__ void __launch_bounds__(1024) absmax_bf16_x8_kernel(const uint16_t* __restrict__ X, unsigned int ld, unsigned int cols, unsigned int rows,
    float* __restrict__ maxima, bool pdl)
{
    __shared__ unsigned int warp_max[32];
    pdl_launch_dependents();    // the quantiser
    if (pdl) { pdl_wait(); }
    const unsigned int per_row = cols / 8;
    const unsigned long long groups = (unsigned long long)rows * per_row, step = (unsigned long long)gridDim.x * 1024;
    unsigned int m = 0;
#pragma unroll 4
    for (unsigned long long j = (unsigned long long)blockIdx.x * 1024 + threadIdx.x; j < groups; j += step)
    {
        const uint4 v = *reinterpret_cast<const uint4*>(X + (size_t)(j / per_row) * ld + (size_t)(j % per_row) * 8);
        const unsigned int w[4] = { v.x, v.y, v.z, v.w };
#pragma unroll
        for (int q = 0; q < 4; q++)
        {
            const unsigned int lo = w[q] & 0x7FFFu, hi = (w[q] >> 16) & 0x7FFFu;
            if (lo <= 0x7F80u) { m = max(m, lo); }
            if (hi <= 0x7F80u) { m = max(m, hi); }
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) { m = max(m, __shfl_xor_sync(0xFFFFFFFFu, m, o)); }
    if ((threadIdx.x & 31u) == 0) { warp_max[threadIdx.x >> 5] = m; }
    __syncthreads();
    if (threadIdx.x == 0)
    {
#pragma unroll
        for (int w = 1; w < 32; w++) { m = max(m, warp_max[w]); }
        maxima[blockIdx.x] = __uint_as_float(m << 16);
    }
}

static __global__ void __launch_bounds__(256) quantise_activations_x8_kernel(const uint16_t* __restrict__ X, unsigned int ld, unsigned int cols,
    unsigned int rows, uint8_t* __restrict__ Q, const float* __restrict__ maxima, unsigned int n_max, float fwd_static, float inv_static,
    float* __restrict__ inv_out)
{
    pdl_launch_dependents();    // the linear: its weights do not depend on this
    pdl_wait();
    float fwd = fwd_static, inv = inv_static;
    if (fwd_static == 0.f)
    {
        const float a = block_maximum(maxima, n_max);
        fwd = (a > 0.f) ? (448.0f / a) : 1.0f;
        inv = (a > 0.f) ? (a / 448.0f) : 1.0f;
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) { *inv_out = inv; }
    const unsigned int per_row = cols / 8;
    const unsigned long long groups = (unsigned long long)rows * per_row;
    for (unsigned long long j = (unsigned long long)blockIdx.x * 256 + threadIdx.x; j < groups; j += (unsigned long long)gridDim.x * 256)
    {
        const size_t r = (size_t)(j / per_row), c = (size_t)(j % per_row) * 8;
        const uint4 v = *reinterpret_cast<const uint4*>(X + r * ld + c);
        const unsigned int w[4] = { v.x, v.y, v.z, v.w };
        unsigned int o[2] = { 0u, 0u };
#pragma unroll
        for (int q = 0; q < 4; q++)
        {
            const unsigned int lo = float_to_e4m3(bf16_bits_to_float((uint16_t)(w[q] & 0xFFFFu)), fwd);
            const unsigned int hi = float_to_e4m3(bf16_bits_to_float((uint16_t)(w[q] >> 16)), fwd);
            o[q >> 1] |= (lo | (hi << 8)) << (16 * (q & 1));
        }
        *reinterpret_cast<uint2*>(Q + r * cols + c) = make_uint2(o[0], o[1]);
    }
}

// The linear(s).  Returns the C-ABI code, -1 for what this path does not serve (K % 128 != 0, unaligned operands, more
// than three members, a workspace that is too small for the quantised activations).  pair_fh: form of the launch
// for many tokens (0: chosen here, 1 .. 3: of the pair kernels, 4: the k slices).
// x_is_e4m3: X holds E4M3 bytes (ldx in bytes) whose multiplier back is act_scale (> 0); y_e4m3: Y receives E4M3 bytes.
static int launch_w8a8(const GemvScratch* ws, const W8A8Member* mem, unsigned int count, const void* X, float act_scale, unsigned int M,
    unsigned int K, unsigned int ldx, cudaStream_t stream, unsigned int flags, bool x_is_e4m3 = false, bool y_e4m3 = false, unsigned int pair_fh = 0)
{
    if (count == 0 || count > (unsigned int)PF_MAX_GROUP || M == 0 || M > 65535u || act_scale < 0.f) { return -1; }
    if (pair_fh > 4) { pair_fh &= 3u; }
    const bool big = M > (unsigned int)W8A8_MAX_TOKENS || pair_fh == 4 || (pair_fh == 0 && w8a8_split_early(M, K));
    if (x_is_e4m3 && !(act_scale > 0.f)) { return -1; }
    const unsigned int bnp = big ? M : (M <= 16 ? 16u : 32u);    // rows the quantiser writes
    NativeParams np;
    memset(&np, 0, sizeof(np));
    np.n_seg = count;
    np.status = ws->status;
    np.M = M;
    np.K = K;
    np.out_f32 = y_e4m3 ? 3u : ((flags & 4u) ? 1u : ((flags & 8u) ? 2u : 0u));
    np.counters = ws->counters;
    np.nkb = K / NK_BK;
    for (unsigned int j = 0; j < count; j++)
    {
        if (!mem[j].W || !mem[j].Y || !native_supported(DT_E4M3, mem[j].N_out, 1u, K, mem[j].ldw, x_is_e4m3 ? 8u : ldx) || !sk_al16(mem[j].W)) { return -1; }
        PrefillSeg& g = np.seg[j];
        g.W = (const uint8_t*)mem[j].W;
        g.Y = (uint16_t*)mem[j].Y;
        g.N = mem[j].N_out;
        g.ldw = mem[j].ldw;
        g.ldy_m = mem[j].ldy_m;
        g.ldy_n = mem[j].ldy_n;
        g.alpha = mem[j].alpha;
        g.beta = mem[j].beta;
        g.w_scale = 1.0f;
        g.post_scale = mem[j].w_inv_scale;    // both scales multiply the FP32 sums, as cublasLt's scale pointers do
        g.tile0 = np.tiles;
        np.tiles += (mem[j].N_out + NK_BM - 1) / NK_BM;
    }
    const unsigned int grid = big ? 0u : nk_grid(np.tiles, np.nkb, 2ull * (unsigned)ws->sm_count);
    // scratch: [0, 1024): the multipliers back (one per token) and, at float 255, the absmax word; then the E4M3 rows; then partial tiles
    unsigned char* sc = reinterpret_cast<unsigned char*>(ws->partials);
    const size_t q_bytes = (((size_t)bnp * K) + 1023) & ~(size_t)1023;
    const size_t part_bytes = (size_t)2 * grid * M * NK_BM * sizeof(float);
    if (!sc || NK_SCALE_BYTES + q_bytes + part_bytes > ws->partial_bytes || grid > ws->n_counters || ((uintptr_t)sc & 255u) != 0) { return -1; }
    float* inv = reinterpret_cast<float*>(sc);
    float* absmax = inv + 255;
    uint8_t* Q = sc + NK_SCALE_BYTES;
    np.inv_scale = inv;
    np.partials = reinterpret_cast<float*>(Q + q_bytes);
    CUtensorMap tmX;
    StreamWMaps tmW;
    memset(&tmW, 0, sizeof(tmW));
    bool ok = big || make_map_2d(&tmX, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, Q, K, bnp, K, NK_BK, bnp, true);
    for (unsigned int j = 0; j < (unsigned int)PF_MAX_GROUP && ok && !big; j++)
    {
        const W8A8Member& m = mem[j < count ? j : 0];
        ok = make_map_2d(&tmW.w[j], CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, m.W, K, m.N_out, m.ldw, NK_BK, NK_BM, true);
    }
    if (!ok) { return -1; }
    const bool pdl = (flags & 1u) != 0;
    const bool dynamic = act_scale == 0.f && !x_is_e4m3;
    const bool eights = (K % 8) == 0 && (ldx % 8) == 0 && sk_al16(X);    // 16-byte loads of X
    // dynamic scale of a small tensor: the quantiser finds the maximum itself
    const bool self_absmax = dynamic && !big && (size_t)M * K <= 16384 && eights;
    // The linear behind the quantiser (`after`: that was the launch before it on the stream; it lets its successor start).
    // Every member takes the kernel that it would take alone, so that a group gives the bits of the separate calls; neighbours of a
    // kind share a launch.
    auto many_tokens = [&](const NativeParams& all, const uint8_t* q, unsigned int ldq, bool after) {
        auto slices = [&](unsigned int j) { return pair_fh == 4 || (pair_fh == 0 && w8a8_split_preferred(M, K, mem[j].N_out, ws->sm_count)); };
        for (unsigned int j = 0, end; j < count; j = end)
        {
            for (end = j + 1; end < count && slices(end) == slices(j);) { end++; }
            NativeParams n = all;
            n.n_seg = end - j;
            n.tiles = 0;
            for (unsigned int i = j; i < end; i++)
            {
                n.seg[i - j] = all.seg[i];
                n.seg[i - j].tile0 = n.tiles;
                n.tiles += (mem[i].N_out + NK_BM - 1) / NK_BM;
            }
            int r = slices(j) ? launch_w8a8_split(n, mem + j, q, ldq, ws->device, ws->sm_count, stream, after || pdl) : -2;
            if (r == -2) { r = launch_w8a8_pair(n, mem + j, q, ldq, ws->device, ws->sm_count, pair_fh, stream, after || pdl); }
            if (r != 0) { return r; }
        }
        return 0;
    };
    if (big && x_is_e4m3 && (ldx % 16) == 0 && sk_al16(X))
    {
        // E4M3 activations that TMA can read where they lie: no copy, the multiplier back goes with the launch
        np.inv_scale = nullptr;
        np.act_inv = act_scale;
        return many_tokens(np, (const uint8_t*)X, ldx, false);
    }
    cudaLaunchAttribute after[1];
    after[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    after[0].val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t qc;
    memset(&qc, 0, sizeof(qc));
    qc.stream = stream;
    qc.attrs = after;
    unsigned int n_max = 1;
    if (dynamic && !self_absmax && eights)
    {
        const unsigned long long blocks = ((unsigned long long)M * (K / 8) + 1023) / 1024;
        n_max = (unsigned int)(blocks < W8A8_MAX_BLOCKS ? blocks : W8A8_MAX_BLOCKS);
        absmax = inv + 64;    // behind the multipliers of up to 32 tokens
        qc.gridDim = dim3(n_max);
        qc.blockDim = dim3(1024);
        qc.numAttrs = pdl ? 1 : 0;
        count_launch();
        if (cudaLaunchKernelEx(&qc, absmax_bf16_x8_kernel, (const uint16_t*)X, ldx, K, M, absmax, pdl) != cudaSuccess) { return w8a8_launch_failed(); }
    }
    if (big && !x_is_e4m3 && eights)
    {
        // many tokens: eight values per thread, a grid that fills the GPU
        const unsigned long long blocks = ((unsigned long long)M * (K / 8) + 255) / 256, most = 8ull * (unsigned)ws->sm_count;
        qc.gridDim = dim3((unsigned int)(blocks < most ? blocks : most));
        qc.blockDim = dim3(256);
        qc.numAttrs = pdl || dynamic ? 1 : 0;    // behind the absmax kernel, which itself starts after whatever came before
        count_launch();
        if (cudaLaunchKernelEx(&qc, quantise_activations_x8_kernel, (const uint16_t*)X, ldx, K, M, Q, (const float*)absmax, n_max, dynamic ? 0.f : 1.0f / act_scale,
                dynamic ? 0.f : act_scale, inv)
            != cudaSuccess)
        {
            return w8a8_launch_failed();
        }
        return many_tokens(np, Q, K, true);
    }
    if (dynamic && !self_absmax && !eights)
    {
        if (cudaMemsetAsync(absmax, 0, sizeof(float), stream) != cudaSuccess) { return w8a8_launch_failed(); }
        unsigned int gx = (K + 255) / 256;
        if (gx > 64) { gx = 64; }
        count_launch();
        absmax_bf16_rows_kernel<<<dim3(gx, M), 256, 0, stream>>>((const uint16_t*)X, ldx, K, M, absmax);
    }
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg;
    memset(&cfg, 0, sizeof(cfg));
    cfg.stream = stream;
    cfg.attrs = attr;
    cfg.gridDim = dim3((K + 255) / 256, bnp);
    cfg.blockDim = dim3(256);
    const bool q_pdl = dynamic && !self_absmax ? eights : pdl;    // behind absmax_bf16_rows_kernel the quantiser is plainly ordered
    cfg.numAttrs = q_pdl ? 1 : 0;
    count_launch();
    if (cudaLaunchKernelEx(&cfg, quantise_activations_kernel, (const uint16_t*)X, ldx, K, M, Q, K, self_absmax ? (const float*)nullptr : (const float*)absmax, n_max,
            dynamic ? 0.f : 1.0f / act_scale, dynamic ? 0.f : act_scale, inv, big ? 1u : M, q_pdl, x_is_e4m3)
        != cudaSuccess)
    {
        return w8a8_launch_failed();
    }
    if (big) { return many_tokens(np, Q, K, q_pdl); }
    auto launch_linear = [&](auto kernel, int smem) -> int {
        static std::atomic<bool> attr_set[2][64];
        const int which = bnp == 16 ? 0 : 1;
        if (!attr_set[which][ws->device].load(std::memory_order_acquire))
        {
            if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess) { return w8a8_launch_failed(); }
            attr_set[which][ws->device].store(true, std::memory_order_release);
        }
        cfg.gridDim = dim3(grid);
        cfg.blockDim = dim3(NK_THREADS);
        cfg.dynamicSmemBytes = smem;
        cfg.numAttrs = 1;    // its weight prefetch does not depend on the quantiser before it
        count_launch();
        if (cudaLaunchKernelEx(&cfg, kernel, tmX, tmW, np) != cudaSuccess) { return w8a8_launch_failed(); }
        return 0;
    };
    return bnp == 16 ? launch_linear(gemm_wq_native_kernel<DT_E4M3, 16, false, 1>, nk_smem_bytes(16))
                     : launch_linear(gemm_wq_native_kernel<DT_E4M3, 32, false, 1>, nk_smem_bytes(32));
}

}    // namespace b200

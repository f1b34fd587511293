// A device for the CPU tests of the served quantised model: the CUDA runtime calls and the layer operations that its host code makes,
// on host memory, preloaded before the real libraries (tests/test_served_cpu.py).
//   * Fresh memory holds 0xA5 bytes.
//   * Work on the private (non-blocking) stream runs at once; work on the default stream as late as the runtime allows: when the
//     host waits for the device, or for a blocking copy.  Nothing orders the two.
//   * Linears, norms and attention leave the token's embedding as it is; the logits of a row whose first element is t are t
//     everywhere but at place t, where they are t + 1000 (as BF16 numbers).
#include <cublas_v2.h>
#include <cuda_runtime_api.h>

#include <cstdint>
#include <cstdlib>
#include <cstring>
#include <functional>
#include <vector>

#include "../include/cccc_b200_decoder.h"
#include "../include/cccc_cuda_b200.h"

namespace
{
using Work = std::function<void()>;
std::vector<Work> late;               // the default stream's
std::vector<Work>* recording = nullptr;
const cudaStream_t kStream = (cudaStream_t)0x10;
struct
{
    unsigned long long wild_rows, decode_calls, prompt_calls, bytes;
} seen;

int run(void* stream, Work w)
{
    if (recording) { recording->push_back(std::move(w)); }
    else if (stream) { w(); }
    else { late.push_back(std::move(w)); }
    return 0;
}
void drain()
{
    std::vector<Work> todo;
    todo.swap(late);
    for (auto& w : todo) { w(); }
}
float wide(uint16_t b)
{
    const uint32_t u = (uint32_t)b << 16;
    float f;
    std::memcpy(&f, &u, 4);
    return f;
}
uint16_t narrow(float f)
{
    uint32_t u;
    std::memcpy(&u, &f, 4);
    return (uint16_t)((u + 0x7FFFu + ((u >> 16) & 1u)) >> 16);
}
void look(const cuda_attn_decode& a, unsigned long long* calls)
{
    (*calls)++;
    for (unsigned int i = 0; i < a.B; i++)
    {
        const int pos = ((const int*)a.pos)[i], slot = ((const int*)a.slot)[i];
        seen.wild_rows += pos < 0 || pos >= (int)a.T_max || slot < 0 || slot >= 32;
    }
}
}    // namespace

// 0: (sequence, layer) pairs whose position or slot lay outside the cache; 1: decode attention calls; 2: prompt passes times layers;
// 3: device bytes asked for
C_EXPORT unsigned long long fake_seen(int what) { return ((unsigned long long*)&seen)[what]; }

extern "C" {
#define RT __attribute__((visibility("default"))) cudaError_t CUDARTAPI
RT cudaGetDeviceCount(int* n) { return *n = 1, cudaSuccess; }
RT cudaSetDevice(int) { return cudaSuccess; }
RT cudaGetLastError() { return cudaSuccess; }
RT cudaPeekAtLastError() { return cudaSuccess; }
RT cudaStreamCreateWithFlags(cudaStream_t* s, unsigned int) { return *s = kStream, cudaSuccess; }
RT cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
RT cudaStreamSynchronize(cudaStream_t s) { return s ? (void)0 : drain(), cudaSuccess; }
RT cudaDeviceSynchronize() { return drain(), cudaSuccess; }
RT cudaMallocHost(void** p, size_t n) { return *p = std::malloc(n), std::memset(*p, 0xA5, n), cudaSuccess; }
RT cudaMalloc(void** p, size_t n) { return seen.bytes += n, cudaMallocHost(p, n); }
RT cudaFree(void* p) { return std::free(p), cudaSuccess; }
RT cudaFreeHost(void* p) { return std::free(p), cudaSuccess; }
RT cudaMemset(void* p, int v, size_t n) { return late.push_back([=] { std::memset(p, v, n); }), cudaSuccess; }
RT cudaMemsetAsync(void* p, int v, size_t n, cudaStream_t s) { return run(s, [=] { std::memset(p, v, n); }), cudaSuccess; }
RT cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind) { return drain(), std::memcpy(d, s, n), cudaSuccess; }
RT cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t st) { return run(st, [=] { std::memcpy(d, s, n); }), cudaSuccess; }
#define BLAS __attribute__((visibility("default"))) cublasStatus_t CUBLASWINAPI
BLAS cublasCreate_v2(cublasHandle_t* h) { return *h = (cublasHandle_t)0x20, CUBLAS_STATUS_SUCCESS; }
BLAS cublasDestroy_v2(cublasHandle_t) { return CUBLAS_STATUS_SUCCESS; }
BLAS cublasSetMathMode(cublasHandle_t, cublasMath_t) { return CUBLAS_STATUS_SUCCESS; }
BLAS cublasSetStream_v2(cublasHandle_t, cudaStream_t) { return CUBLAS_STATUS_SUCCESS; }
RT cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { return recording = new std::vector<Work>, cudaSuccess; }
RT cudaStreamEndCapture(cudaStream_t, cudaGraph_t* g) { return *g = (cudaGraph_t)recording, recording = nullptr, cudaSuccess; }
RT cudaGraphInstantiate(cudaGraphExec_t* e, cudaGraph_t g, unsigned long long) { return *e = (cudaGraphExec_t)g, cudaSuccess; }
RT cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
RT cudaGraphExecDestroy(cudaGraphExec_t e) { return delete (std::vector<Work>*)e, cudaSuccess; }
RT cudaGraphLaunch(cudaGraphExec_t e, cudaStream_t)
{
    for (auto& w : *(std::vector<Work>*)e) { w(); }
    return cudaSuccess;
}
}

C_EXPORT int cuda_check_error(const char*) { return drain(), 0; }
C_EXPORT int cuda_b200_decoder_check(const char*) { return drain(), 0; }
C_EXPORT int cuda_b200_status(void* host, void* st) { return run(st, [=] { std::memset(host, 0, 4); }); }
C_EXPORT int cuda_embed_bf16(const void* ids, const void* W, void* Y, unsigned int D, unsigned int n, unsigned int vocab, void* st, unsigned int)
{
    return run(st, [=] {
        for (unsigned int i = 0; i < n; i++)
        {
            const unsigned int id = ((const unsigned int*)ids)[i];
            if (id < vocab) { std::memcpy((uint16_t*)Y + (size_t)i * D, (const uint16_t*)W + (size_t)id * D, D * 2); }
            else { std::memset((uint16_t*)Y + (size_t)i * D, 0, D * 2); }
        }
    });
}
C_EXPORT int cuda_rms_norm_bf16(const void* X, const void*, void*, void* Y, const void*, unsigned int rows, unsigned int inner, float, void* st, unsigned int)
{
    return run(st, [=] { std::memcpy(Y, X, (size_t)rows * inner * 2); });
}
C_EXPORT int cuda_gemm_wq_bf16(int, const void*, const void*, float, const void* X, void* Y, unsigned int N, unsigned int M, unsigned int, unsigned int,
    unsigned int ldx, unsigned int ldy, unsigned int, float, float beta, void* st, unsigned int)
{
    return beta != 0.f ? 0 : run(st, [=] {
        for (unsigned int m = 0; m < M; m++)
        {
            const float t = wide(((const uint16_t*)X)[(size_t)m * ldx]);
            for (unsigned int v = 0; v < N; v++) { ((uint16_t*)Y)[(size_t)m * ldy + v] = narrow(v == (unsigned int)t ? t + 1000.f : t); }
        }
    });
}
C_EXPORT int cuda_gemm_wq_bf16_group(int, unsigned int, const cuda_wq_linear*, const void*, unsigned int, unsigned int, unsigned int, void*, unsigned int)
{
    return 0;
}
C_EXPORT int cuda_swiglu_bf16(const void*, const void*, void*, unsigned int, unsigned int, unsigned int, unsigned int, unsigned int, void*, unsigned int)
{
    return 0;
}
C_EXPORT int cuda_attn_decode_bf16(const cuda_attn_decode* a, void* st, unsigned int)
{
    return run(st, [d = *a] { look(d, &seen.decode_calls); });
}
C_EXPORT int cuda_attn_append_bf16(const cuda_attn_decode* a, void* st, unsigned int)
{
    return run(st, [d = *a] { look(d, &seen.prompt_calls); });
}
C_EXPORT int cuda_b200_attention_rows(int, const cuda_b200_attention*, const cuda_b200_batch*, void*, unsigned int, int) { return 0; }
C_EXPORT int cuda_argmax_bf16(const void* x, unsigned int rows, unsigned int cols, unsigned long long ld, void* idx, void* val, void* st)
{
    return run(st, [=] {
        for (unsigned int r = 0; r < rows; r++)
        {
            const uint16_t* row = (const uint16_t*)x + r * ld;
            unsigned int best = 0;
            for (unsigned int v = 1; v < cols; v++) { best = wide(row[v]) > wide(row[best]) ? v : best; }
            ((int*)idx)[r] = (int)best;
            ((float*)val)[r] = wide(row[best]);
        }
    });
}

#include "decode_step.h"

#include "../../../include/cccc_b200_decoder.h"
#include "../../../include/cccc_cuda_b200.h"

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstring>

namespace cccc
{

namespace
{
bool fail(std::string* err, const std::string& what)
{
    if (err) { *err = what; }
    return false;
}

// the host bfloat16 constructor of the reference truncates (cccc/types.h:36-60)
uint16_t bf16Trunc(float f)
{
    uint32_t u;
    std::memcpy(&u, &f, 4);
    return (uint16_t)(u >> 16);
}

uint16_t bf16Round(float f)
{
    uint32_t u;
    std::memcpy(&u, &f, 4);
    if ((u & 0x7fffffffu) > 0x7f800000u) { return (uint16_t)((u >> 16) | 0x40); }
    u += 0x7fffu + ((u >> 16) & 1u);
    return (uint16_t)(u >> 16);
}

float halfToFloat(uint16_t h)
{
    const uint32_t sign = (uint32_t)(h & 0x8000u) << 16;
    uint32_t exp = (h >> 10) & 0x1fu, man = h & 0x3ffu, u;
    if (exp == 0)
    {
        if (man == 0) { u = sign; }
        else
        {
            int e = -1;
            do {
                man <<= 1;
                e++;
            } while (!(man & 0x400u));
            u = sign | ((uint32_t)(127 - 15 - e) << 23) | ((man & 0x3ffu) << 13);
        }
    }
    else if (exp == 31) { u = sign | 0x7f800000u | (man << 13); }
    else { u = sign | ((exp + 112) << 23) | (man << 13); }
    float f;
    std::memcpy(&f, &u, 4);
    return f;
}
}    // namespace

// ---- TensorParallel ----

TensorParallel::~TensorParallel()
{
    // The areas belong to this object, not to the ranks' GpuControl objects: those live on the ranks' threads and are
    // gone by the time the last owner of the TensorParallel lets go of it.
    for (int r = 0; r < world_; r++)
    {
        if (device_[r] < 0) { continue; }
        cudaSetDevice(device_[r]);
        if (recv_[r]) { cudaFree(recv_[r]); }
        if (flag_[r]) { cudaFree(flag_[r]); }
    }
}

void TensorParallel::barrier()
{
    std::unique_lock<std::mutex> lk(m_);
    const unsigned long long gen = generation_;
    if (++waiting_ == world_)
    {
        waiting_ = 0;
        generation_++;
        cv_.notify_all();
        return;
    }
    cv_.wait(lk, [&] { return generation_ != gen; });
}

bool TensorParallel::allOk(int rank, bool ok)
{
    {
        std::lock_guard<std::mutex> lk(m_);
        ok_[rank] = ok ? 1 : 0;
    }
    barrier();
    bool all = true;
    for (int r = 0; r < world_; r++) { all = all && ok_[r] != 0; }
    barrier();
    return all;
}

bool TensorParallel::join(int rank, GpuControl* gpu, unsigned int n_max, std::string* err)
{
    if (rank < 0 || rank >= world_ || !gpu) { return fail(err, "bad rank"); }
    gpu->setAsCurrent();
    n_max = (n_max + 3u) & ~3u;
    const size_t rb = cuda_b200_allreduce_recv_bytes(world_, n_max), fb = cuda_b200_fused_flag_bytes(world_);
    void *recv = nullptr, *flag = nullptr;
    bool ok = cudaMalloc(&recv, rb) == cudaSuccess && cudaMalloc(&flag, fb) == cudaSuccess;
    if (ok) { ok = cudaMemset(recv, 0, rb) == cudaSuccess && cudaMemset(flag, 0, fb) == cudaSuccess; }
    if (!ok) { cudaGetLastError(); }
    {
        std::lock_guard<std::mutex> lk(m_);
        device_[rank] = gpu->getDeviceID();
        recv_[rank] = recv;
        flag_[rank] = flag;
        n_max_ = n_max;
        if (!ok) { failed_ = true; }
    }
    barrier();    // every rank's areas exist
    // peer access to every other rank's device (the reference's multi-device mode uses cudaMemcpyPeer,
    // cccc/Matrix.cpp:498-517; the fused exchange stores straight into the peers' areas)
    for (int r = 0; r < world_ && !failed_; r++)
    {
        if (r == rank) { continue; }
        const int peer = device_[r];
        if (peer == gpu->getDeviceID()) { continue; }
        int can = 0;
        cudaDeviceCanAccessPeer(&can, gpu->getDeviceID(), peer);
        if (!can)
        {
            std::lock_guard<std::mutex> lk(m_);
            failed_ = true;
            break;
        }
        const cudaError_t e = cudaDeviceEnablePeerAccess(peer, 0);
        if (e == cudaErrorPeerAccessAlreadyEnabled) { cudaGetLastError(); }
        else if (e != cudaSuccess)
        {
            std::lock_guard<std::mutex> lk(m_);
            failed_ = true;
        }
    }
    cudaDeviceSynchronize();
    barrier();
    if (failed_) { return fail(err, "tensor parallel setup failed (allocation or peer access)"); }
    return true;
}

int TensorParallel::combineArgmax(int rank, int global_id, float value)
{
    {
        std::lock_guard<std::mutex> lk(m_);
        best_[rank] = value;
        id_[rank] = global_id;
    }
    barrier();
    int win = -1;
    float top = 0.f;
    for (int r = 0; r < world_; r++)
    {
        if (id_[r] < 0) { continue; }    // a shard of only NaN
        if (win < 0 || best_[r] > top)
        {
            win = id_[r];
            top = best_[r];
        }
    }
    last_best_[rank] = top;
    barrier();    // nobody overwrites the slots before all have read them
    return win;
}

float TensorParallel::combineAbsmax(int rank, float value)
{
    {
        std::lock_guard<std::mutex> lk(m_);
        absmax_[rank] = value;
    }
    barrier();
    float top = 0.f;
    for (int r = 0; r < world_; r++) { top = std::fmax(top, absmax_[r]); }
    barrier();
    return top;
}

void TensorParallel::gatherLogits(int rank, const uint16_t* shard, int n, float* full)
{
    {
        std::lock_guard<std::mutex> lk(m_);
        if (row_.size() != (size_t)world_ * n) { row_.assign((size_t)world_ * n, 0.f); }
    }
    barrier();    // the row has its size before anyone writes a slice
    for (int i = 0; i < n; i++)
    {
        const uint32_t u = (uint32_t)shard[i] << 16;
        std::memcpy(&row_[(size_t)rank * n + i], &u, 4);
    }
    barrier();
    std::memcpy(full, row_.data(), row_.size() * sizeof(float));
    barrier();
}

// ---- DecodeStep ----

DecodeStep::~DecodeStep()
{
    if (!gpu_) { return; }
    gpu_->setAsCurrent();
    gpu_->synchronize();
    if (program_) { cuda_decode_program_destroy(program_); }
    for (auto g : graphs_)
    {
        if (g) { cudaGraphExecDestroy(g); }
    }
    quantised_.clear();
    for (void* p : owned_) { gpu_->free(p); }
    if (h_ids_) { cudaFreeHost(h_ids_); }
    if (h_logits_) { cudaFreeHost(h_logits_); }
    if (h_meta_) { cudaFreeHost(h_meta_); }
}

void* DecodeStep::dmalloc(size_t bytes)
{
    void* p = gpu_->malloc(bytes);
    if (p) { owned_.push_back(p); }
    return p;
}

bool DecodeStep::loadLinear(const BinFile& f, const std::string& name, int N, int K, char kind, Linear* out, std::string* err)
{
    WeightShard sh;
    if (!loadWeightShard(f, name, N, K, kind, world_, rank_, &sh, err)) { return false; }
    out->n = sh.n;
    out->k = sh.k;
    if (Cublas::isQuantized(sh.dtype))
    {
        if (wt_ == CURRENT) { wt_ = sh.dtype; }
        if (sh.dtype != wt_) { return fail(err, "weight '" + name + "' has another quantised type than the first one"); }
        if (sh.dtype == FP4_E2M1 && sh.block_scales.empty()) { return fail(err, "weight '" + name + "' is FP4 without block scales"); }
        out->w = dmalloc(sh.weights.size());
        if (!out->w || cudaMemcpy(out->w, sh.weights.data(), sh.weights.size(), cudaMemcpyHostToDevice) != cudaSuccess)
        {
            return fail(err, "no device memory for '" + name + "'");
        }
        if (!sh.block_scales.empty())
        {
            out->s = dmalloc(sh.block_scales.size());
            if (!out->s || cudaMemcpy(out->s, sh.block_scales.data(), sh.block_scales.size(), cudaMemcpyHostToDevice) != cudaSuccess)
            {
                return fail(err, "no device memory for the block scales of '" + name + "'");
            }
        }
        out->inv = sh.quant_scale;
    }
    else
    {
        // BF16 / half / float tensor: quantise on the GPU while loading (cccc/Net.cpp:1142-1233 -> cccc/Matrix.cpp:301-355)
        if (!Cublas::isQuantized(cfg_.weight_data_type)) { return fail(err, "weight '" + name + "' is not quantised and no weight_data_type is set"); }
        if (wt_ == CURRENT) { wt_ = cfg_.weight_data_type; }
        if (wt_ != cfg_.weight_data_type) { return fail(err, "weight '" + name + "' would get another quantised type than the first one"); }
        const size_t n = (size_t)sh.n * sh.k;
        if (sh.dtype == HALF)
        {
            // the device converter takes float and BF16: widen half on the host
            std::vector<uint8_t> wide(n * 4);
            const uint16_t* src = (const uint16_t*)sh.weights.data();
            float* dst = (float*)wide.data();
            for (size_t i = 0; i < n; i++) { dst[i] = halfToFloat(src[i]); }
            sh.weights.swap(wide);
            sh.dtype = FLOAT;
        }
        Matrix m(sh.k, sh.n, 1, 1, sh.dtype, gpu_);
        if (!m.data() || cudaMemcpy(m.data(), sh.weights.data(), sh.weights.size(), cudaMemcpyHostToDevice) != cudaSuccess)
        {
            return fail(err, "no device memory for '" + name + "'");
        }
        if (tp_ && world_ > 1)
        {
            m.quantizeWeights(wt_, [&](float a) { return tp_->combineAbsmax(rank_, a); });
        }
        else { m.quantizeWeights(wt_); }
        if (m.getDataType() != wt_) { return fail(err, "quantising '" + name + "' failed"); }
        out->w = m.data();
        out->s = (void*)m.getBlockScaleData();
        out->inv = m.getQuantScale();
        if (keep_host_)
        {
            const size_t wb = wt_ == FP4_E2M1 ? n / 2 : n;
            sh.weights.resize(wb);
            cudaMemcpy(sh.weights.data(), out->w, wb, cudaMemcpyDeviceToHost);
            sh.block_scales.clear();
            if (out->s)
            {
                sh.block_scales.resize(n / 16);
                cudaMemcpy(sh.block_scales.data(), out->s, n / 16, cudaMemcpyDeviceToHost);
            }
            sh.dtype = wt_;
            sh.quant_scale = out->inv;
        }
        quantised_.push_back(std::move(m));
        quantised_on_load_++;
    }
    weight_bytes_ += (wt_ == FP4_E2M1 ? (size_t)sh.n * sh.k / 2 + (size_t)sh.n * sh.k / 16 : (size_t)sh.n * sh.k);
    if (keep_host_) { stored_.push_back(Stored{ name, std::move(sh) }); }
    return true;
}

bool DecodeStep::loadBf16(const BinFile& f, const std::string& name, size_t n, uint16_t** out, bool required, std::string* err)
{
    *out = nullptr;
    std::string key;
    DataType dt;
    if (!f.findTypedWeight(name, &key, &dt))
    {
        return required ? fail(err, "tensor '" + name + "' is missing") : true;
    }
    std::vector<uint16_t> host(n);
    if (dt == BFLOAT16)
    {
        if (f.entry(key).length != n * 2 || !f.read(key, 0, n * 2, host.data())) { return fail(err, "tensor '" + name + "' has the wrong size"); }
    }
    else if (dt == FLOAT)
    {
        // float checkpoints: to BF16 as the device conversion of the reference rounds (cccc/Net.cpp:1404-1440)
        std::vector<float> tmp(n);
        if (f.entry(key).length != n * 4 || !f.read(key, 0, n * 4, tmp.data())) { return fail(err, "tensor '" + name + "' has the wrong size"); }
        for (size_t i = 0; i < n; i++) { host[i] = bf16Round(tmp[i]); }
    }
    else if (dt == HALF)
    {
        if (f.entry(key).length != n * 2 || !f.read(key, 0, n * 2, host.data())) { return fail(err, "tensor '" + name + "' has the wrong size"); }
        for (size_t i = 0; i < n; i++) { host[i] = bf16Round(halfToFloat(host[i])); }
    }
    else { return fail(err, "tensor '" + name + "' must be BF16, half or float"); }
    *out = (uint16_t*)dmalloc(n * 2);
    if (!*out || cudaMemcpy(*out, host.data(), n * 2, cudaMemcpyHostToDevice) != cudaSuccess) { return fail(err, "no device memory for '" + name + "'"); }
    if (keep_host_) { plain_.emplace_back(name, std::move(host)); }
    return true;
}

bool DecodeStep::load(GpuControl* gpu, const BinFile& file, const ModelConfig& cfg, int max_batch, TensorParallel* tp, int rank, std::string* err)
{
    gpu_ = gpu;
    tp_ = tp;
    cfg_ = cfg;
    world_ = tp ? tp->world() : 1;
    rank_ = tp ? rank : 0;
    max_batch_ = max_batch;
    wt_ = CURRENT;
    gpu_->setAsCurrent();
    if (cfg.hidden <= 0 || cfg.layers <= 0 || cfg.head_dim <= 0 || cfg.max_context <= 0 || max_batch <= 0 || max_batch > 32)
    {
        return fail(err, "bad model configuration");
    }
    if (cfg.n_heads % world_ || cfg.n_kv_heads % world_ || cfg.ffn % world_ || cfg.vocab % world_)
    {
        return fail(err, "heads, ffn or vocabulary do not divide over the ranks");
    }
    H_ = cfg.n_heads / world_;
    Hkv_ = cfg.n_kv_heads / world_;
    q_loc_ = H_ * cfg.head_dim;
    kv_loc_ = Hkv_ * cfg.head_dim;
    ffn_loc_ = cfg.ffn / world_;
    vocab_loc_ = cfg.vocab / world_;
    qkv_ld_ = q_loc_ + 2 * kv_loc_;

    // With several ranks, the tensors are loaded first and the ranks agree that all of them succeeded before the
    // first step (whose exchange waits for every peer) is issued.
    bool ok = loadTensors(file, err);
    if (tp_ && world_ > 1 && !tp_->allOk(rank_, ok))
    {
        if (ok) { fail(err, "another rank failed to load"); }
        return false;
    }
    if (!ok) { return false; }
    // first use of the kernels allocates the library's per-device workspace: do it before any capture
    // (the step's stream does not wait for the default stream: its zeros are written on it)
    const bool cleared = cudaMemsetAsync(d_ids_, 0, (size_t)max_batch * 16, gpu_->stream()) == cudaSuccess;
    if (tp_) { tp_->barrier(); }
    const int rc = cleared ? issue(1, gpu_->stream(), false) : -1;
    gpu_->synchronize();
    const bool stepped = rc >= 0 && cuda_check_error("decode step warm-up") == 0;
    launches_per_step_ = rc;
    resetCache();
    if (tp_ && world_ > 1)
    {
        if (!tp_->allOk(rank_, stepped)) { return fail(err, "the first decode step failed"); }
    }
    else if (!stepped) { return fail(err, "the first decode step failed"); }
    return true;
}

bool DecodeStep::loadTensors(const BinFile& file, std::string* err)
{
    const ModelConfig& cfg = cfg_;
    const int max_batch = max_batch_;
    const int q_dim = cfg.n_heads * cfg.head_dim, kv_dim = cfg.n_kv_heads * cfg.head_dim;
    layers_.resize(cfg.layers);
    layers_loaded_ = 0;
    for (int i = 0; i < cfg.layers; i++)
    {
        Layer& L = layers_[i];
        const std::string s = "_" + std::to_string(i);
        if (!loadLinear(file, "W_q" + s, q_dim, cfg.hidden, 'c', &L.q, err) || !loadLinear(file, "W_k" + s, kv_dim, cfg.hidden, 'c', &L.k, err)
            || !loadLinear(file, "W_v" + s, kv_dim, cfg.hidden, 'c', &L.v, err) || !loadLinear(file, "W_o" + s, cfg.hidden, q_dim, 'r', &L.o, err)
            || !loadLinear(file, "W_gate" + s, cfg.ffn, cfg.hidden, 'c', &L.gate, err) || !loadLinear(file, "W_up" + s, cfg.ffn, cfg.hidden, 'c', &L.up, err)
            || !loadLinear(file, "W_down" + s, cfg.hidden, cfg.ffn, 'r', &L.down, err))
        {
            return false;
        }
        layers_loaded_++;
        if (!loadBf16(file, "W_rms_attn" + s, cfg.hidden, &L.attn_norm, true, err) || !loadBf16(file, "W_rms_ffn" + s, cfg.hidden, &L.ffn_norm, true, err)
            || !loadBf16(file, "W_qnorm" + s, cfg.head_dim, &L.q_norm, cfg.qk_norm, err) || !loadBf16(file, "W_knorm" + s, cfg.head_dim, &L.k_norm, cfg.qk_norm, err))
        {
            return false;
        }
        if (!cfg.qk_norm) { L.q_norm = L.k_norm = nullptr; }
    }
    if (!cache_.init(gpu_, std::vector<KvLayerShape>((size_t)cfg.layers, { Hkv_, cfg.head_dim, cfg.head_dim }), 2, max_batch, cfg.max_context, err)) { return false; }
    if (!loadLinear(file, "W_lm_head", cfg.vocab, cfg.hidden, 'c', &lm_head_, err)) { return false; }
    if (!loadBf16(file, "W_emb", (size_t)cfg.vocab * cfg.hidden, &emb_, true, err) || !loadBf16(file, "W_rms_final", cfg.hidden, &final_norm_, true, err))
    {
        return false;
    }

    // RoPE tables, computed on the host in float and stored through the truncating host constructor
    // (cccc/NetCifa.cpp:431-475)
    {
        const int half = cfg.head_dim / 2;
        std::vector<uint16_t> c((size_t)cfg.max_context * half), s((size_t)cfg.max_context * half);
        for (int t = 0; t < cfg.max_context; t++)
        {
            for (int d = 0; d < half; d++)
            {
                const float ang = (float)t * std::pow(cfg.rope_theta, -2.0f * (float)d / (float)cfg.head_dim);
                c[(size_t)t * half + d] = bf16Trunc(std::cos(ang));
                s[(size_t)t * half + d] = bf16Trunc(std::sin(ang));
            }
        }
        cos_ = (uint16_t*)dmalloc(c.size() * 2);
        sin_ = (uint16_t*)dmalloc(s.size() * 2);
        if (!cos_ || !sin_) { return fail(err, "no device memory for the RoPE tables"); }
        cudaMemcpy(cos_, c.data(), c.size() * 2, cudaMemcpyHostToDevice);
        cudaMemcpy(sin_, s.data(), s.size() * 2, cudaMemcpyHostToDevice);
    }

    const size_t B = (size_t)max_batch;
    x_ = (uint16_t*)dmalloc(B * cfg.hidden * 2);
    xn_ = (uint16_t*)dmalloc(B * cfg.hidden * 2);
    tmp_ = (uint16_t*)dmalloc(B * cfg.hidden * 2);
    qkv_ = (uint16_t*)dmalloc(B * qkv_ld_ * 2);
    att_ = (uint16_t*)dmalloc(B * q_loc_ * 2);
    gu_ = (uint16_t*)dmalloc(B * 2 * ffn_loc_ * 2);
    h_ = (uint16_t*)dmalloc(B * ffn_loc_ * 2);
    logits_ = (uint16_t*)dmalloc(B * vocab_loc_ * 2);
    d_ids_ = (int*)dmalloc(B * 16);    // one block, one copy each way: ids, positions, slots, best
    d_pos_ = d_ids_ + B;
    d_slot_ = d_pos_ + B;
    d_best_ = (float*)(d_slot_ + B);
    if (!x_ || !xn_ || !tmp_ || !qkv_ || !att_ || !gu_ || !h_ || !logits_ || !d_ids_) { return fail(err, "no device memory for the step's buffers"); }
    // one pinned block: ids, positions and slots in; the device's block out; the status word
    if (cudaMallocHost((void**)&h_ids_, B * 28 + 4) != cudaSuccess) { return fail(err, "no pinned memory"); }
    std::memset(h_ids_, 0, B * 28 + 4);
    h_pos_ = h_ids_ + B;
    h_slot_ = h_pos_ + B;
    h_out_ = h_slot_ + B;
    h_best_ = (float*)(h_out_ + 3 * B);
    h_status_ = (unsigned int*)(h_best_ + B);
    if (cudaMallocHost((void**)&h_logits_, B * vocab_loc_ * 2) != cudaSuccess) { return fail(err, "no pinned memory for the logits"); }
    if (world_ > 1)
    {
        const size_t cb = cuda_b200_fused_counter_bytes();
        seq_counters_ = dmalloc(cb);
        if (!seq_counters_) { return fail(err, "no device memory"); }
        cudaMemset(seq_counters_, 0, cb);
        if (tp_->nMax() < (unsigned int)(B * cfg.hidden)) { return fail(err, "the exchange areas are smaller than max_batch * hidden"); }
    }
    graphs_.assign(2 * (max_batch + 1), nullptr);
    // The default stream's copies and the zeros above end before anything runs on the step's own stream, which is not ordered behind it.
    if (cudaDeviceSynchronize() != cudaSuccess) { return fail(err, "a CUDA error while loading"); }
    return true;
}

void DecodeStep::resetCache() { cache_.clear(); }

// A linear of a group: features from `out` on, rows of `ld` elements.
static cuda_wq_linear member(const void* w, const void* s, float inv, int n, uint16_t* out, int k, int ld)
{
    cuda_wq_linear g = {};
    g.W = w;
    g.blk_scales = s;
    g.Y = out;
    g.inv_scale = inv;
    g.alpha = 1.0f;
    g.N_out = (unsigned int)n;
    g.ldw = (unsigned int)k;
    g.ldy_m = (unsigned int)ld;
    g.ldy_n = 1;
    return g;
}

void DecodeStep::groupQkv(const Layer& L, uint16_t* out, cuda_wq_linear* g) const
{
    const Linear* l[3] = { &L.q, &L.k, &L.v };
    for (int j = 0; j < 3; out += l[j]->n, j++) { g[j] = member(l[j]->w, l[j]->s, l[j]->inv, l[j]->n, out, cfg_.hidden, qkv_ld_); }
}

void DecodeStep::groupGateUp(const Layer& L, uint16_t* out, cuda_wq_linear* g) const
{
    g[0] = member(L.gate.w, L.gate.s, L.gate.inv, ffn_loc_, out, cfg_.hidden, 2 * ffn_loc_);
    g[1] = member(L.up.w, L.up.s, L.up.inv, ffn_loc_, out + ffn_loc_, cfg_.hidden, 2 * ffn_loc_);
}

int DecodeStep::issue(int M, cudaStream_t st, bool direct)
{
    const unsigned int PDL = 1u, RES = 8u;
    const int wt = (int)wt_;
    const bool tp = world_ > 1;
    const unsigned int hid = cfg_.hidden;
    int n = 0, bad = 0;
    auto ok = [&](int rc) {
        if (rc != 0) { bad++; }
        n++;
    };
    auto norm = [&](const uint16_t* scale, bool pending) {
        ok(cuda_rms_norm_bf16(x_, pending ? tmp_ : nullptr, pending ? x_ : nullptr, xn_, scale, M, hid, cfg_.eps, st, PDL));
    };
    auto row_linear = [&](const Linear& L, const uint16_t* src) {
        if (tp)
        {
            ok(cuda_gemm_wq_bf16_allreduce(wt, L.w, L.s, L.inv, src, tmp_, hid, M, L.k, L.k, L.k, hid, 1, 1.0f, tp_->recvPtrs(), tp_->flagPtrs(),
                seq_counters_, tp_->nMax(), rank_, world_, st, PDL));
        }
        else { ok(cuda_gemm_wq_bf16(wt, L.w, L.s, L.inv, src, x_, hid, M, L.k, L.k, L.k, hid, 1, 1.0f, 1.0f, st, PDL | RES)); }
    };
    ok(cuda_embed_bf16(d_ids_, emb_, x_, hid, M, cfg_.vocab, st, PDL));
    bool pending = false;
    for (size_t i = 0; i < layers_.size(); i++)
    {
        const Layer& L = layers_[i];
        norm(L.attn_norm, pending);
        cuda_wq_linear g[3];
        groupQkv(L, qkv_, g);
        ok(cuda_gemm_wq_bf16_group(wt, 3, g, xn_, M, hid, hid, st, PDL));
        cuda_attn_decode a = attnArgs(i, M);
        ok(cuda_attn_decode_bf16(&a, st, PDL));
        row_linear(L.o, att_);
        norm(L.ffn_norm, tp);
        cuda_wq_linear u[2];
        groupGateUp(L, gu_, u);
        ok(cuda_gemm_wq_bf16_group(wt, 2, u, xn_, M, hid, hid, st, PDL));
        ok(cuda_swiglu_bf16(gu_, gu_ + ffn_loc_, h_, M, ffn_loc_, 2 * ffn_loc_, 2 * ffn_loc_, ffn_loc_, st, PDL));
        row_linear(L.down, h_);
        pending = tp;
    }
    norm(final_norm_, pending);
    ok(cuda_gemm_wq_bf16(wt, lm_head_.w, lm_head_.s, lm_head_.inv, xn_, direct ? h_logits_ : logits_, vocab_loc_, M, hid, hid, hid, vocab_loc_, 1, 1.0f, 0.0f, st, PDL));
    if (!direct) { ok(cuda_argmax_bf16(logits_, M, vocab_loc_, vocab_loc_, d_ids_, d_best_, st)); }
    return bad ? -1 : n;
}

cuda_attn_decode DecodeStep::attnArgs(size_t layer, int M) const
{
    const Layer& L = layers_[layer];
    cuda_attn_decode a = {};
    a.q = qkv_;
    a.k = qkv_ + q_loc_;
    a.v = qkv_ + q_loc_ + kv_loc_;
    a.q_norm = L.q_norm;
    a.k_norm = L.k_norm;
    a.cos_tab = cos_;
    a.sin_tab = sin_;
    a.k_cache = cache_.k((int)layer);
    a.v_cache = cache_.v((int)layer);
    a.pos = d_pos_;
    a.slot = d_slot_;
    a.out = att_;
    a.ldq = a.ldk = a.ldv = qkv_ld_;
    a.ldo = q_loc_;
    a.B = M;
    a.H = H_;
    a.Hkv = Hkv_;
    a.head_dim = cfg_.head_dim;
    a.T_max = cfg_.max_context;
    a.epsilon = cfg_.eps;
    a.dk = 0.f;
    return a;
}

bool DecodeStep::reservePrompts(int tokens)
{
    prompt_cap_ = 0;
    if (world_ != 1 || tokens <= 0 || (cfg_.head_dim != 64 && cfg_.head_dim != 128)) { return false; }
    gpu_->setAsCurrent();
    const size_t T = (size_t)tokens, meta = (size_t)(4 * tokens + 4 * max_batch_) * 4, work = cuda_b200_attention_work_bytes((unsigned int)cfg_.head_dim);
    const size_t owned = owned_.size();
    px_ = (uint16_t*)dmalloc(T * cfg_.hidden * 2);
    pxn_ = (uint16_t*)dmalloc(T * cfg_.hidden * 2);
    pqkv_ = (uint16_t*)dmalloc(T * qkv_ld_ * 2);
    patt_ = (uint16_t*)dmalloc(T * q_loc_ * 2);
    pgu_ = (uint16_t*)dmalloc(T * 2 * ffn_loc_ * 2);
    ph_ = (uint16_t*)dmalloc(T * ffn_loc_ * 2);
    d_meta_ = (int*)dmalloc(meta);
    attn_work_ = dmalloc(work);
    const bool all = px_ && pxn_ && pqkv_ && patt_ && pgu_ && ph_ && d_meta_ && attn_work_;
    if (!all || (!h_meta_ && cudaMallocHost((void**)&h_meta_, meta) != cudaSuccess) || cudaMemset(attn_work_, 0, work) != cudaSuccess)
    {
        cudaGetLastError();    // no room: what was taken goes back, prompts go through the decode step
        while (owned_.size() > owned)
        {
            gpu_->free(owned_.back());
            owned_.pop_back();
        }
        return false;
    }
    cudaDeviceSynchronize();
    prompt_cap_ = tokens;
    return true;
}

int DecodeStep::prompt(const std::vector<PromptEntry>& entries, const std::vector<int>& want, int* next_ids, uint16_t* logits)
{
    const unsigned int PDL = 1u, RES = 8u;
    int tokens = 0, max_n = 0, max_len = 0;
    for (const auto& e : entries)
    {
        tokens += e.n;
        max_n = std::max(max_n, e.n);
        max_len = std::max(max_len, e.pos + e.n);
    }
    if (tokens == 0) { return 0; }
    if (tokens > prompt_cap_ || (int)entries.size() > max_batch_) { return -1; }
    for (int w : want)
    {
        if (w < 0 || w >= tokens) { return -1; }    // (a place may be wanted several times)
    }
    gpu_->setAsCurrent();
    cudaStream_t st = gpu_->stream();
    // per token: id, position, slot, entry; per entry: slot, position, first token, tokens
    const int C = prompt_cap_, B = max_batch_;
    int *ids = h_meta_, *pos = ids + C, *slot = pos + C, *owner = slot + C, *e_slot = owner + C, *e_pos = e_slot + B, *e_start = e_pos + B, *e_n = e_start + B;
    int at = 0;
    for (size_t e = 0; e < entries.size(); e++)
    {
        const PromptEntry& E = entries[e];
        e_slot[e] = E.slot;
        e_pos[e] = E.pos;
        e_start[e] = at;
        e_n[e] = E.n;
        for (int i = 0; i < E.n; i++, at++)
        {
            ids[at] = E.tokens[i];
            pos[at] = E.pos + i;
            slot[at] = E.slot;
            owner[at] = (int)e;
        }
    }
    if (cudaMemcpyAsync(d_meta_, h_meta_, (size_t)(4 * C + 4 * B) * 4, cudaMemcpyHostToDevice, st) != cudaSuccess) { return 1; }
    auto dev = [&](const int* host) { return d_meta_ + (host - h_meta_); };
    cuda_b200_batch batch = {};
    batch.slot = dev(e_slot);
    batch.pos = dev(e_pos);
    batch.start = dev(e_start);
    batch.n = dev(e_n);
    batch.token_entry = dev(owner);
    batch.entries = (unsigned int)entries.size();
    batch.tokens = (unsigned int)tokens;
    batch.max_n = (unsigned int)max_n;
    batch.max_len = (unsigned int)max_len;
    const int wt = (int)wt_;
    const unsigned int hid = (unsigned int)cfg_.hidden, M = (unsigned int)tokens;
    int n = 0, bad = 0;
    auto ok = [&](int rc) {
        if (rc != 0) { bad++; }
        n++;
    };
    auto row_linear = [&](const Linear& L, const uint16_t* src) {
        ok(cuda_gemm_wq_bf16(wt, L.w, L.s, L.inv, src, px_, hid, M, L.k, L.k, L.k, hid, 1, 1.0f, 1.0f, st, PDL | RES));
    };
    ok(cuda_embed_bf16(dev(ids), emb_, px_, hid, M, cfg_.vocab, st, 0));
    for (size_t i = 0; i < layers_.size(); i++)
    {
        const Layer& L = layers_[i];
        ok(cuda_rms_norm_bf16(px_, nullptr, nullptr, pxn_, L.attn_norm, M, hid, cfg_.eps, st, PDL));
        cuda_wq_linear g[3];
        groupQkv(L, pqkv_, g);
        ok(cuda_gemm_wq_bf16_group(wt, 3, g, pxn_, M, hid, hid, st, PDL));
        cuda_attn_decode a = attnArgs(i, tokens);
        a.q = pqkv_;
        a.k = pqkv_ + q_loc_;
        a.v = pqkv_ + q_loc_ + kv_loc_;
        a.out = pqkv_;
        a.ldo = (unsigned int)qkv_ld_;
        a.pos = dev(pos);
        a.slot = dev(slot);
        ok(cuda_attn_append_bf16(&a, st, PDL));
        cuda_b200_attention t = {};
        t.qkvg = pqkv_;
        t.out = patt_;
        t.k_cache = cache_.k((int)i);
        t.v_cache = cache_.v((int)i);
        t.work = attn_work_;
        t.ld = (unsigned int)qkv_ld_;
        t.ldo = (unsigned int)q_loc_;
        t.H = (unsigned int)H_;
        t.Hkv = (unsigned int)Hkv_;
        t.dim = t.vdim = (unsigned int)cfg_.head_dim;
        t.k_ld = (unsigned int)cache_.kLd((int)i);
        t.v_ld = (unsigned int)cache_.vLd((int)i);
        t.T_max = (unsigned int)cache_.rows();
        t.slots = (unsigned int)cache_.slots();
        t.no_append = 1;
        t.scale = 1.0f / std::sqrt((float)cfg_.head_dim);
        ok(cuda_b200_attention_rows((int)BFLOAT16, &t, &batch, st, PDL, 0));
        row_linear(L.o, patt_);
        ok(cuda_rms_norm_bf16(px_, nullptr, nullptr, pxn_, L.ffn_norm, M, hid, cfg_.eps, st, PDL));
        cuda_wq_linear u[2];
        groupGateUp(L, pgu_, u);
        ok(cuda_gemm_wq_bf16_group(wt, 2, u, pxn_, M, hid, hid, st, PDL));
        ok(cuda_swiglu_bf16(pgu_, pgu_ + ffn_loc_, ph_, M, ffn_loc_, 2 * ffn_loc_, 2 * ffn_loc_, ffn_loc_, st, PDL));
        row_linear(L.down, ph_);
    }
    // the wanted rows, a decode batch at a time: gathered, normalised, through the head
    for (size_t w0 = 0; w0 < want.size() && !bad; w0 += (size_t)max_batch_)
    {
        const int rows = (int)std::min((size_t)max_batch_, want.size() - w0);
        for (int i = 0; i < rows; i++) { h_ids_[i] = want[w0 + i]; }
        cudaMemcpyAsync(d_ids_, h_ids_, (size_t)rows * 4, cudaMemcpyHostToDevice, st);
        ok(cuda_embed_bf16(d_ids_, px_, x_, hid, rows, M, st, 0));
        ok(cuda_rms_norm_bf16(x_, nullptr, nullptr, xn_, final_norm_, rows, hid, cfg_.eps, st, PDL));
        ok(cuda_gemm_wq_bf16(wt, lm_head_.w, lm_head_.s, lm_head_.inv, xn_, logits_, vocab_loc_, rows, hid, hid, hid, vocab_loc_, 1, 1.0f, 0.0f, st, PDL));
        ok(cuda_argmax_bf16(logits_, rows, vocab_loc_, vocab_loc_, d_ids_, d_best_, st));
        cudaMemcpyAsync(h_out_, d_ids_, (size_t)rows * 4, cudaMemcpyDeviceToHost, st);
        if (logits) { cudaMemcpyAsync(h_logits_, logits_, (size_t)rows * vocab_loc_ * 2, cudaMemcpyDeviceToHost, st); }
        if (cudaStreamSynchronize(st) != cudaSuccess) { return 1; }
        if (logits) { std::memcpy(logits + w0 * vocab_loc_, h_logits_, (size_t)rows * vocab_loc_ * 2); }
        for (int i = 0; i < rows && next_ids; i++) { next_ids[w0 + i] = h_out_[i]; }
    }
    last_launches_ = n;
    if (cudaStreamSynchronize(st) != cudaSuccess) { return 1; }    // the pinned arrays are reused by the next pass
    if (cuda_check_error("prompt") != 0 || cuda_b200_decoder_check("prompt") != 0) { return 1; }
    return bad ? 1 : 0;
}

bool DecodeStep::buildProgram()
{
    if (program_) { return true; }
    if (world_ > 1) { return false; }
    const unsigned int RES = 8u, PAIRED = 16u;
    const unsigned int hid = cfg_.hidden;
    ::cuda_decode_program* p = nullptr;
    if (cuda_decode_program_create(&p, (int)wt_, 1) != 0) { return false; }
    bool good = true;
    auto lin = [](const Linear& L, void* Y, unsigned int ldw, unsigned int ldy, float beta) {
        cuda_wq_linear g = {};
        g.W = L.w;
        g.blk_scales = L.s;
        g.Y = Y;
        g.inv_scale = L.inv;
        g.alpha = 1.0f;
        g.beta = beta;
        g.N_out = L.n;
        g.ldw = ldw;
        g.ldy_m = ldy;
        g.ldy_n = 1;
        return g;
    };
    auto input = [&](int mode, const void* x, unsigned int ld, const void* w) {
        cuda_decode_input in = {};
        in.mode = mode;
        in.x = x;
        in.ldx = ld;
        in.norm_weight = w;
        in.epsilon = cfg_.eps;
        return in;
    };
    for (size_t i = 0; i < layers_.size() && good; i++)
    {
        const Layer& L = layers_[i];
        cuda_wq_linear g[3] = { lin(L.q, qkv_, hid, qkv_ld_, 0.f), lin(L.k, qkv_ + q_loc_, hid, qkv_ld_, 0.f), lin(L.v, qkv_ + q_loc_ + kv_loc_, hid, qkv_ld_, 0.f) };
        cuda_decode_input in = input(1, x_, hid, L.attn_norm);
        good = good && cuda_decode_program_add_linears(p, 3, g, &in, hid, 0) == 0;
        cuda_attn_decode a = attnArgs(i, 1);
        good = good && cuda_decode_program_add_attention(p, &a) == 0;
        cuda_wq_linear o = lin(L.o, x_, q_loc_, hid, 1.0f);
        in = input(0, att_, q_loc_, nullptr);
        good = good && cuda_decode_program_add_linears(p, 1, &o, &in, q_loc_, RES) == 0;
        cuda_wq_linear gu[2] = { lin(L.gate, h_, hid, ffn_loc_, 0.f), lin(L.up, h_, hid, ffn_loc_, 0.f) };
        in = input(1, x_, hid, L.ffn_norm);
        good = good && cuda_decode_program_add_linears(p, 2, gu, &in, hid, PAIRED) == 0;
        cuda_wq_linear d = lin(L.down, x_, ffn_loc_, hid, 1.0f);
        in = input(0, h_, ffn_loc_, nullptr);
        good = good && cuda_decode_program_add_linears(p, 1, &d, &in, ffn_loc_, RES) == 0;
    }
    if (good)
    {
        cuda_wq_linear h = lin(lm_head_, logits_, hid, vocab_loc_, 0.f);
        cuda_decode_input in = input(1, x_, hid, final_norm_);
        good = cuda_decode_program_add_linears(p, 1, &h, &in, hid, 0) == 0 && cuda_decode_program_finalize(p) == 0;
    }
    if (!good)
    {
        cuda_decode_program_destroy(p);
        return false;
    }
    program_ = p;
    return true;
}

bool DecodeStep::useProgram(bool on)
{
    if (!on)
    {
        use_program_ = false;
        return true;
    }
    gpu_->setAsCurrent();
    use_program_ = buildProgram();
    return use_program_;
}

int DecodeStep::step(const int* token_ids, const int* positions, int M, int* next_ids, float* best_logits, uint16_t* logits_host, const int* slots)
{
    int rc = launch(token_ids, positions, M, logits_host != nullptr, true, slots);
    if (rc == 0) { rc = finish(next_ids, best_logits); }
    if (rc == 0 && logits_host) { std::memcpy(logits_host, h_logits_, (size_t)M * vocab_loc_ * 2); }
    return rc;
}

int DecodeStep::launch(const int* token_ids, const int* positions, int M, bool logits, bool choice, const int* slots)
{
    if (M < 1 || M > max_batch_) { return -1; }
    gpu_->setAsCurrent();
    cudaStream_t st = gpu_->stream();
    for (int i = 0; i < M; i++)
    {
        h_ids_[i] = token_ids[i];
        h_pos_[i] = positions[i];
        h_slot_[i] = slots ? slots[i] : i;
    }
    // ids, positions and slots lie one behind the other, here and on the device
    auto upload = [&] { return cudaMemcpyAsync(d_ids_, h_ids_, (size_t)max_batch_ * 12, cudaMemcpyHostToDevice, st) == cudaSuccess; };
    // the chosen ids and, behind two other arrays, their logits; the status word
    auto download = [&](bool chosen) {
        if (chosen) { cudaMemcpyAsync(h_out_, d_ids_, (size_t)max_batch_ * 16, cudaMemcpyDeviceToHost, st); }
        return cuda_b200_status(h_status_, st);
    };
    int rc = 0;
    // Logits that the host wants without the greedy choice, which reads them again, are written into its memory by the head's linear:
    // they cross the bus while the weights are read.
    bool direct = false;
    if (use_program_ && M == 1 && program_)
    {
        rc = upload() ? 0 : 1;
        rc |= cuda_embed_bf16(d_ids_, emb_, x_, cfg_.hidden, 1, cfg_.vocab, st, 0);
        rc |= cuda_decode_program_launch(program_, st);
        rc |= cuda_argmax_bf16(logits_, 1, vocab_loc_, vocab_loc_, d_ids_, d_best_, st);
        rc |= download(true);
        last_launches_ = 3;
    }
    else
    {
        direct = logits && !choice && world_ == 1 && M <= kDirectRows;
        cudaGraphExec_t& step = graphs_[M + (direct ? max_batch_ + 1 : 0)];
        if (!step)
        {
            // the first step for this M records the launches, and the copies around them; later ones replay the graph
            cudaGraph_t graph = nullptr;
            if (cudaStreamBeginCapture(st, cudaStreamCaptureModeThreadLocal) != cudaSuccess) { return 1; }
            const bool sent = upload();
            const int n = issue(M, st, direct);
            const bool good = download(!direct) == 0 && sent;
            const cudaError_t e = cudaStreamEndCapture(st, &graph);
            if (n < 0 || !good || e != cudaSuccess || !graph)
            {
                if (graph) { cudaGraphDestroy(graph); }
                cudaGetLastError();
                return n < 0 ? -1 : 1;
            }
            cudaGraphExec_t exec = nullptr;
            const cudaError_t ei = cudaGraphInstantiate(&exec, graph, 0);
            cudaGraphDestroy(graph);
            if (ei != cudaSuccess) { return 1; }
            step = exec;
        }
        // every rank is about to launch: the exchange inside the row-parallel linears waits for the peers
        if (tp_ && world_ > 1) { tp_->barrier(); }
        rc = cudaGraphLaunch(step, st) == cudaSuccess ? 0 : 1;
        last_launches_ = launches_per_step_ - (direct ? 1 : 0);
    }
    if (logits && !direct) { cudaMemcpyAsync(h_logits_, logits_, (size_t)M * vocab_loc_ * 2, cudaMemcpyDeviceToHost, st); }
    running_ = M;
    if (rc != 0) { finish(h_out_, nullptr); }    // nothing stays under way
    return rc;
}

int DecodeStep::finish(int* next_ids, float* best_logits)
{
    int rc = 0;
    gpu_->setAsCurrent();
    if (cudaStreamSynchronize(gpu_->stream()) != cudaSuccess) { rc = 1; }
    if ((rc != 0 || *h_status_ != 0 || cudaPeekAtLastError() != cudaSuccess) && cuda_check_error("decode step") != 0) { rc = 1; }
    for (int i = 0; i < running_; i++)
    {
        int id = h_out_[i] < 0 ? -1 : h_out_[i] + rank_ * vocab_loc_;
        float best = h_best_[i];
        if (tp_ && world_ > 1)
        {
            id = tp_->combineArgmax(rank_, id, best);
            best = tp_->lastBest(rank_);
        }
        next_ids[i] = id;
        if (best_logits) { best_logits[i] = best; }
    }
    return rc;
}

bool DecodeStep::saveNamedWeights(const std::string& path, std::string* err) const
{
    if (world_ != 1) { return fail(err, "a cache file holds whole tensors: load on one rank to write it"); }
    if (stored_.empty()) { return fail(err, "keepHostCopies(true) before load() keeps what this writes"); }
    BinWriter w;
    for (const auto& s : stored_) { w.addQuantised(s.name, s.shard); }
    for (const auto& t : plain_) { w.add("weight_bf16_" + t.first, t.second.data(), t.second.size() * 2); }
    return w.save(path) ? true : fail(err, "cannot write '" + path + "'");
}

}    // namespace cccc

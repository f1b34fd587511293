// The quantised cccc LLM (DecodeStep) behind the LanguageModel interface, for the registry, the scheduler and the command
// line.  config.json: {"architecture": "cccc-llm", "hidden", "n_heads", "n_kv_heads", "head_dim", "ffn", "vocab", "layers",
// "rope_theta", "eps", "qk_norm", and optionally "weights" (container file, default model.bin) and "weight_data_type"
// ("fp8_e4m3", "fp8_e5m2", "fp4_e2m1": quantise while loading)}.  Prompts run in passes of many tokens (DecodeStep::prompt);
// sequences that decode together share a step.
#include "decode_step.h"
#include "language_model.h"

#include <algorithm>
#include <cstring>

namespace cccc
{

namespace
{
class QuantisedLlm : public LanguageModel
{
public:
    bool load(const ModelOptions& o, const Json& c, std::string* err)
    {
        if (o.dtype != BFLOAT16) { return fail(err, "this model runs in bfloat16 activations only"); }
        if (o.noise_weights) { return fail(err, "this model needs its weight file"); }
        ModelConfig m;
        m.hidden = (int)c["hidden"].number();
        m.n_heads = (int)c["n_heads"].number();
        m.n_kv_heads = (int)c["n_kv_heads"].number();
        m.head_dim = (int)c["head_dim"].number();
        m.ffn = (int)c["ffn"].number();
        m.vocab = (int)c["vocab"].number();
        m.layers = (int)c["layers"].number();
        m.rope_theta = (float)c["rope_theta"].number(10000.0);
        m.eps = (float)c["eps"].number(1e-6);
        m.qk_norm = c["qk_norm"].boolean();
        m.max_context = o.max_context;
        const std::string& t = c["weight_data_type"].string();
        if (t == "fp8_e4m3") { m.weight_data_type = FP8_E4M3; }
        else if (t == "fp8_e5m2") { m.weight_data_type = FP8_E5M2; }
        else if (t == "fp4_e2m1") { m.weight_data_type = FP4_E2M1; }
        else if (!t.empty()) { return fail(err, "no weight_data_type '" + t + "'"); }
        if (m.n_heads <= 0 || m.n_kv_heads <= 0 || m.ffn <= 0 || m.vocab <= 0) { return fail(err, "config.json lacks a size"); }
        const std::string path = o.dir + "/" + (c.has("weights") ? c["weights"].string() : "model.bin");
        BinFile f;
        if (gpu_.init(o.device) != 0) { return fail(err, "cannot open CUDA device " + std::to_string(o.device)); }
        if (!f.open(path)) { return fail(err, "cannot open '" + path + "'"); }
        vocab_ = m.vocab;
        batch_ = std::min(o.max_sequences, 32);
        if (!step_.load(&gpu_, f, m, batch_, nullptr, 0, err)) { return false; }
        // a step never has more tokens than the cache has rows
        const long long most = std::min<long long>({ o.max_step_tokens, kMostPromptTokens, (long long)o.max_context * batch_ });
        if (most > 1) { step_.reservePrompts((int)most); }
        return true;
    }
    int vocab() const override { return vocab_; }
    KvCache& cache() override { return step_.cache(); }
    int launchesLastStep() const override { return launches_; }
    size_t weightBytes() const override { return step_.weightBytes(); }

    int step(const std::vector<StepEntry>& entries, float* logits, int* choice) override
    {
        if (!valid(entries)) { return -1; }
        launches_ = 0;
        std::vector<size_t> first(entries.size());
        size_t wanted = 0, longest = 0, tokens = 0;
        for (size_t e = 0; e < entries.size(); e++)
        {
            first[e] = wanted;
            wanted += entries[e].want.size();
            longest = std::max(longest, entries[e].tokens.size());
            tokens += entries[e].tokens.size();
        }
        // Either way a pass reads the weights once, and a decode step is one graph: many tokens at once only where that takes fewer.
        // (Passes of one token never do, passes of two do not for two sequences.)
        const size_t cap = (size_t)step_.promptTokens();
        if (cap > 0 && (tokens + cap - 1) / cap < longest) { return prompts(entries, first, logits, choice); }
        // one token of all entries that have one after the other; the graph of a step takes them all
        for (size_t i = 0; i < longest; i++)
        {
            int rc = launch(entries, i, logits != nullptr, choice != nullptr);
            if (rc == 0) { rc = finish(entries, i, first, logits, choice); }
            if (rc != 0) { return 1; }
        }
        return 0;
    }

    int begin(std::vector<StepEntry> entries, bool logits, bool choice) override
    {
        const int rc = LanguageModel::begin(std::move(entries), logits, choice);
        started_ = rc == 0 && !held_.empty();
        for (const auto& e : held_) { started_ = started_ && e.tokens.size() == 1; }
        if (!started_) { return rc; }
        launches_ = 0;
        started_rc_ = launch(held_, 0, logits, choice);
        return 0;
    }
    int end(float* logits, int* choice) override
    {
        if (!started_) { return LanguageModel::end(logits, choice); }
        started_ = false;
        logits = held_logits_ ? logits : nullptr;
        choice = held_choice_ ? choice : nullptr;
        std::vector<size_t> first(held_.size());
        for (size_t e = 1; e < held_.size(); e++) { first[e] = first[e - 1] + held_[e - 1].want.size(); }
        return started_rc_ == 0 && finish(held_, 0, first, logits, choice) == 0 ? 0 : 1;
    }

private:
    static constexpr int kMostPromptTokens = 2048;    // of a pass: more bring the linears nothing, and cost memory

    // Passes of up to promptTokens() tokens; a long entry goes on in the next one.  first[e]: the place of entry e's results.
    int prompts(const std::vector<StepEntry>& entries, const std::vector<size_t>& first, float* logits, int* choice)
    {
        std::vector<size_t> done(entries.size(), 0);
        for (;;)
        {
            std::vector<DecodeStep::PromptEntry> pass;
            std::vector<size_t> count(entries.size(), 0);
            std::vector<int> want;
            std::vector<size_t> place;
            size_t at = 0;
            for (size_t e = 0; e < entries.size(); e++)
            {
                const StepEntry& E = entries[e];
                count[e] = std::min((size_t)step_.promptTokens() - at, E.tokens.size() - done[e]);
                if (count[e] == 0) { continue; }
                pass.push_back({ E.slot, cache().length(E.slot), (int)count[e], E.tokens.data() + done[e] });
                for (size_t w = 0; w < E.want.size(); w++)
                {
                    const size_t t = (size_t)E.want[w];
                    if (t < done[e] || t >= done[e] + count[e]) { continue; }
                    want.push_back((int)(at + t - done[e]));
                    place.push_back(first[e] + w);
                }
                at += count[e];
            }
            if (at == 0) { return 0; }
            std::vector<uint16_t> rows(logits ? want.size() * vocab_ : 0);
            std::vector<int> next(want.size());
            if (step_.prompt(pass, want, next.data(), logits ? rows.data() : nullptr) != 0) { return 1; }
            launches_ += step_.lastLaunches();
            for (size_t i = 0; i < want.size(); i++)
            {
                if (choice) { choice[place[i]] = next[i]; }
                if (logits) { widen(rows.data() + i * vocab_, logits + place[i] * vocab_); }
            }
            for (size_t e = 0; e < entries.size(); e++)
            {
                done[e] += count[e];
                if (count[e]) { cache().setLength(entries[e].slot, cache().length(entries[e].slot) + (int)count[e]); }
            }
        }
    }

    // The i-th tokens of the entries that have one, as one step.
    int launch(const std::vector<StepEntry>& entries, size_t i, bool logits, bool choice)
    {
        std::vector<int> ids, pos, slot;
        bool any = false;
        for (const auto& e : entries)
        {
            if (i >= e.tokens.size()) { continue; }
            ids.push_back(e.tokens[i]);
            slot.push_back(e.slot);
            pos.push_back(cache().length(e.slot));
            any = any || std::count(e.want.begin(), e.want.end(), (int)i);
        }
        return step_.launch(ids.data(), pos.data(), (int)ids.size(), logits && any, choice, slot.data());
    }
    int finish(const std::vector<StepEntry>& entries, size_t i, const std::vector<size_t>& first, float* logits, int* choice)
    {
        std::vector<int> next(entries.size());
        if (step_.finish(next.data(), nullptr) != 0) { return 1; }
        launches_ += step_.lastLaunches();
        size_t k = 0;
        for (size_t e = 0; e < entries.size(); e++)
        {
            const StepEntry& E = entries[e];
            if (i >= E.tokens.size()) { continue; }
            cache().setLength(E.slot, cache().length(E.slot) + 1);
            for (size_t w = 0; w < E.want.size(); w++)
            {
                if (E.want[w] != (int)i) { continue; }
                if (choice) { choice[first[e] + w] = next[k]; }
                if (logits) { widen(step_.hostLogits() + k * vocab_, logits + (first[e] + w) * vocab_); }
            }
            k++;
        }
        return 0;
    }

    // a BF16 number is the upper half of a float (vectorised: a row of logits is on the way of every step)
    __attribute__((optimize("O3"))) void widen(const uint16_t* __restrict row, float* __restrict out) const
    {
        uint32_t* __restrict bits = (uint32_t* __restrict)(void*)out;
        for (int v = 0; v < vocab_; v++) { bits[v] = (uint32_t)row[v] << 16; }
    }

    static bool fail(std::string* err, const std::string& what)
    {
        if (err) { *err = what; }
        return false;
    }
    GpuControl gpu_;
    DecodeStep step_;
    int vocab_ = 0, batch_ = 1, launches_ = 0;
    bool started_ = false;    // between begin() and end(): the step is under way (started_rc_ 0) or could not be started
    int started_rc_ = 0;
};

const bool g_registered = ModelRegistry::add("cccc-llm", [](const ModelOptions& o, const Json& config, std::string* err) {
    std::unique_ptr<QuantisedLlm> m(new QuantisedLlm());
    if (!m->load(o, config, err)) { m.reset(); }
    return std::unique_ptr<LanguageModel>(std::move(m));
});
}    // namespace

}    // namespace cccc

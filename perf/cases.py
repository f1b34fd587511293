"""What this library is measured on: the linears of a decoder layer with quantised weights at the token counts of decoding
and of prompts, the decode attention beside them, and whole requests - prompts, then tokens one by one - through the served
models of the three families.  Sizes are those of the benchmark (Qwen3-8B and Llama-3.1-8B layers) and, for the served models,
halves of them, so that a model folder stays under a gigabyte.

Kinds of cases:
  linear     one 4096 x 4096 linear on its own
  layer      the linears of one layer as a decoder calls them: q+k+v, o, gate+up, down (four calls)
  attention  the decode attention of one layer: norm, rotation, append and softmax over `context` cached rows
  request    `sequences` requests that arrive together: their prompts in one step, then `decode` steps of one token each,
             with the logits on the host after every step, where a sampler wants them
"""
import ctypes
import importlib.util
import json
import math
import os
import struct
import sys
import tempfile
import zlib

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _package():
    """The package directory carries a hyphen: imported by path."""
    name = "cccc_lite_b200"
    if name not in sys.modules:
        path = os.path.join(ROOT, "cccc-lite_b200")
        spec = importlib.util.spec_from_file_location(name, os.path.join(path, "__init__.py"), submodule_search_locations=[path])
        sys.modules[name] = importlib.util.module_from_spec(spec)
        spec.loader.exec_module(sys.modules[name])
    return sys.modules[name]


# ---- the cases -----------------------------------------------------------------------------------------------------
# hidden, q, kv and feed-forward sizes of a layer
LAYERS = {"qwen3-8b": (4096, 4096, 1024, 12288), "llama-3.1-8b": (4096, 4096, 1024, 14336)}
HEADS, KV_HEADS, HEAD_DIM, ROWS = 32, 8, 128, 4096


def listed():
    return [
        # the smallest call there is: one token through one linear, where latency counts
        dict(name="linear_fp8_1", kind="linear", weights="e5m2", scaled=False, tokens=1),
        # a layer of the benchmark's decode token, one user
        dict(name="layer_fp8_1", kind="layer", model="qwen3-8b", weights="e5m2", scaled=False, tokens=1),
        # the same with thirty-two users in a batch, weights with the scale that quantising on load gives them
        dict(name="layer_fp8_32", kind="layer", model="qwen3-8b", weights="e4m3", scaled=True, tokens=32),
        # four-bit weights, a small batch
        dict(name="layer_fp4_8", kind="layer", model="llama-3.1-8b", weights="fp4", scaled=True, tokens=8),
        # FP8 activations (dynamic scale), a large batch or a short prompt
        dict(name="layer_w8a8_64", kind="layer", model="qwen3-8b", weights="w8a8", scaled=True, tokens=64),
        # a ragged prompt of ordinary length
        dict(name="layer_fp4_301", kind="layer", model="llama-3.1-8b", weights="fp4", scaled=True, tokens=301),
        # the benchmark's prompt
        dict(name="layer_fp8_2048", kind="layer", model="qwen3-8b", weights="e5m2", scaled=False, tokens=2048),
        # long contexts: one user, thirty-two users
        dict(name="attention_1", kind="attention", sequences=1, context=4096),
        dict(name="attention_32", kind="attention", sequences=32, context=4096),
        # whole requests through the served models
        dict(name="request_quantised", kind="request", family="quantised", sequences=4, prompt=256, decode=24),
        dict(name="request_fakilorn", kind="request", family="fakilorn", sequences=8, prompt=192, decode=24),
        dict(name="request_tazunex", kind="request", family="tazunex", sequences=8, prompt=192, decode=24),
    ]


def _log_uniform(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["linear", "layer", "layer", "layer", "attention", "request", "request"])
    if kind in ("linear", "layer"):
        weights = rng.choice(["e5m2", "e4m3", "fp4", "w8a8"])
        case = dict(kind=kind, weights=weights, scaled=weights in ("fp4", "w8a8") or rng.random() < 0.5, tokens=_log_uniform(rng, 1, 2048))
        if kind == "layer":
            case["model"] = "qwen3-8b" if case["tokens"] > 1500 else rng.choice(sorted(LAYERS))
        return case
    if kind == "attention":
        return dict(kind=kind, sequences=_log_uniform(rng, 1, 32), context=_log_uniform(rng, 64, ROWS))
    sequences = _log_uniform(rng, 1, 8)
    return dict(kind=kind, family=rng.choice(["quantised", "fakilorn", "tazunex"]), sequences=sequences,
                prompt=_log_uniform(rng, 16, min(400, 1024 // sequences)), decode=_log_uniform(rng, 4, 24))


# ---- quantised weights ---------------------------------------------------------------------------------------------
FP4_TABLE = (0.0, 0.5, 1.0, 1.5, 2.0, 3.0, 4.0, 6.0)


def _generator(seed, salt=0):
    return torch.Generator(device="cuda").manual_seed((int(seed) * 1000003 + salt) % (1 << 62))


def _quantise(w, weights, scaled):
    """A float matrix as (bytes, block scales or None, multiplier), with the scales that quantising a checkpoint gives."""
    if weights == "fp4":
        blocks = w.reshape(-1, 16)
        top = blocks.abs().amax(1, keepdim=True).clamp_min(1e-10)
        edges = torch.tensor([0.25, 0.75, 1.25, 1.75, 2.5, 3.5, 5.0], device=w.device)
        code = torch.bucketize((blocks * (6.0 / top)).abs(), edges).to(torch.uint8) | ((blocks < 0).to(torch.uint8) << 3)
        code = code.reshape(-1, 2)
        return (code[:, 0] | (code[:, 1] << 4)).reshape(w.shape[0], -1).contiguous(), (top / 6.0).to(torch.float8_e4m3fn).view(torch.uint8).reshape(-1), 1.0
    most, kind = (57344.0, torch.float8_e5m2) if weights == "e5m2" else (448.0, torch.float8_e4m3fn)
    inv = float((w.abs().max() / most).float()) if scaled else 1.0
    return (w / inv).clamp(-most, most).to(kind).view(torch.uint8), None, inv


def _dequantise(q, weights):
    """The matrix the format defines - BF16 numbers - in 64 bits (W8A8: without the rounding, its scale applies to the sums)."""
    W, S, inv = q
    if weights == "fp4":
        table = torch.tensor(FP4_TABLE + tuple(-v for v in FP4_TABLE), device=W.device)
        v = torch.stack([table[(W & 15).int()], table[(W >> 4).int()]], -1).reshape(-1, 16)
        return (v * S.view(torch.float8_e4m3fn).float()[:, None]).to(torch.bfloat16).double().reshape(W.shape[0], -1)
    v = W.view(torch.float8_e5m2 if weights == "e5m2" else torch.float8_e4m3fn).float()
    return v.double() * inv if weights == "w8a8" else (v * inv).to(torch.bfloat16).double()


def _quantised_activations(x):
    """The dynamic activation quantiser of the W8A8 mode: one scale per tensor, magnitudes truncated to E4M3; in 64 bits."""
    top = x.float().abs().max()
    v = x.float() * torch.full_like(top, 448.0).div(top)
    step = torch.exp2(torch.floor(torch.log2(v.abs().clamp_min(2.0 ** -6))) - 3)
    return torch.trunc(v / step).mul(step).clamp(-448, 448).double() * top.div(448.0).double()


# ---- linear, layer -------------------------------------------------------------------------------------------------
def _calls(case):
    """(input width, output widths) of the calls of one pass."""
    if case["kind"] == "linear":
        return [(4096, [4096])]
    hidden, q, kv, ff = LAYERS[case["model"]]
    return [(hidden, [q, kv, kv]), (q, [hidden]), (hidden, [ff, ff]), (ff, [hidden])]


def _linear_inputs(case, seed):
    calls = []
    for i, (K, Ns) in enumerate(_calls(case)):
        g = _generator(seed, i)
        x = torch.randn(case["tokens"], K, device="cuda", generator=g).to(torch.bfloat16)
        calls.append((K, x, [_quantise(torch.randn(N, K, device="cuda", generator=g) * 0.02, case["weights"], case["scaled"]) for N in Ns]))
    return calls


def _prepare_linear(case, seed):
    capi = _package().capi
    calls = []
    for K, x, quantised in _linear_inputs(case, seed):
        y = [torch.zeros(case["tokens"], q[0].shape[0], dtype=torch.bfloat16, device="cuda") for q in quantised]
        group = capi.make_group([dict(W=W, S=S, inv=inv, Y=t, N=t.shape[1]) for (W, S, inv), t in zip(quantised, y)], K)
        calls.append((K, x, quantised, y, group))
    return dict(capi=capi, tokens=case["tokens"], weights=case["weights"], calls=calls,
                type={"e5m2": capi.FP8_E5M2, "e4m3": capi.FP8_E4M3, "fp4": capi.FP4_E2M1, "w8a8": capi.FP8_E4M3}[case["weights"]])


def _run_linear(s):
    capi, M, out = s["capi"], s["tokens"], []
    for K, x, quantised, y, group in s["calls"]:
        # flags 1: the calls of a chain may overlap their neighbours' ends, as in the decode step
        if len(y) > 1:
            rc = capi.gemm_w8a8_bf16_group(group, x, 0.0, M, K, flags=1) if s["weights"] == "w8a8" else capi.gemm_wq_bf16_group(s["type"], group, x, M, K, flags=1)
        else:
            W, S, inv = quantised[0]
            N = y[0].shape[1]
            rc = capi.gemm_w8a8_bf16(W, inv, x, 0.0, y[0], N, M, K, flags=1) if s["weights"] == "w8a8" else capi.gemm_wq_bf16(s["type"], W, S, inv, x, y[0], N, M, K, flags=1)
        if rc:
            raise RuntimeError("a linear failed: %d" % rc)
        out += y
    return out


def _exact_linear(case, seed):
    out = []
    for K, x, quantised in _linear_inputs(case, seed):
        v = _quantised_activations(x) if case["weights"] == "w8a8" else x.double()
        out += [v @ _dequantise(q, case["weights"]).T for q in quantised]
    return out


def _work_linear(case):
    M, each = case["tokens"], {"fp4": 0.5 + 1 / 16}.get(case["weights"], 1.0)
    return dict(bytes=sum(sum(N * K * each + 2 * M * N for N in Ns) + 2 * M * K for K, Ns in _calls(case)),
                flops=sum(2 * M * N * K for K, Ns in _calls(case) for N in Ns))


# ---- attention -----------------------------------------------------------------------------------------------------
def _rope_tables(rows, dim, theta):
    """cos and sin as the models keep them: truncated to BF16."""
    a = torch.arange(rows, dtype=torch.float64)[:, None] * theta ** (-2.0 * torch.arange(dim // 2, dtype=torch.float64) / dim)
    cut = lambda t: torch.from_numpy((t.float().numpy().view(np.uint32) >> 16).astype(np.uint16).view(np.int16)).view(torch.bfloat16).cuda()
    return cut(a.cos()), cut(a.sin())


def _attention_inputs(case, seed):
    B, g = case["sequences"], _generator(seed)
    r = lambda *shape, scale=1.0: (torch.randn(*shape, device="cuda", generator=g) * scale).to(torch.bfloat16)
    qkv = r(B, (HEADS + 2 * KV_HEADS) * HEAD_DIM)
    norms = [(1 + 0.2 * torch.randn(HEAD_DIM, device="cuda", generator=g)).to(torch.bfloat16) for _ in range(2)]
    return qkv, norms, r(B, KV_HEADS, case["context"], HEAD_DIM), r(B, KV_HEADS, case["context"], HEAD_DIM), _rope_tables(case["context"], HEAD_DIM, 1e6)


def _prepare_attention(case, seed):
    """Sequences of slightly different lengths, as in a batch of users; the longest has context - 1 cached rows."""
    capi, B = _package().capi, case["sequences"]
    qkv, norms, k, v, (cos, sin) = _attention_inputs(case, seed)
    pos = torch.tensor(_positions(case), dtype=torch.int32, device="cuda")
    out = torch.zeros(B, HEADS * HEAD_DIM, dtype=torch.bfloat16, device="cuda")
    at = [qkv.data_ptr() + 2 * HEAD_DIM * n for n in (0, HEADS, HEADS + KV_HEADS)]
    desc = capi.make_attn_decode(q=at[0], k=at[1], v=at[2], k_cache=k, v_cache=v, pos=pos, out=out, cos_tab=cos, sin_tab=sin, q_norm=norms[0], k_norm=norms[1],
                                 B=B, H=HEADS, Hkv=KV_HEADS, head_dim=HEAD_DIM, T_max=case["context"], ldq=qkv.shape[1], ldk=qkv.shape[1], ldv=qkv.shape[1])
    return dict(capi=capi, desc=desc, out=out, k=k, v=v, keep=(qkv, norms, cos, sin, pos))


def _positions(case):
    return [case["context"] - 1 - (i * case["context"] // 8) // max(1, case["sequences"]) for i in range(case["sequences"])]


def _run_attention(s):
    rc = s["capi"].attn_decode_bf16(s["desc"], flags=1)
    if rc:
        raise RuntimeError("the attention failed: %d" % rc)
    return [s["out"], s["k"], s["v"]]


def _norm_rotate(x, weight, cos, sin, eps):
    """RMS norm over the last axis, then the half-rotate form of rotary positions."""
    x = x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps) * weight if weight is not None else x
    a, b = x.chunk(2, -1)
    return torch.cat([a * cos - b * sin, b * cos + a * sin], -1)


def _exact_attention(case, seed):
    qkv, norms, k, v, (cos, sin) = _attention_inputs(case, seed)
    qn, kn, cos, sin, out = norms[0].double(), norms[1].double(), cos.double(), sin.double(), []
    k, v = k.double(), v.double()
    for b, p in enumerate(_positions(case)):
        q, kk, vv = qkv[b].double().reshape(-1, HEAD_DIM).split([HEADS, KV_HEADS, KV_HEADS])
        k[b, :, p] = _norm_rotate(kk, kn, cos[p], sin[p], 1e-6)
        v[b, :, p] = vv
        q = _norm_rotate(q, qn, cos[p], sin[p], 1e-6).reshape(KV_HEADS, -1, HEAD_DIM)
        out.append((torch.softmax(q @ k[b, :, :p + 1].transpose(1, 2) / math.sqrt(HEAD_DIM), -1) @ v[b, :, :p + 1]).reshape(-1))
    return [torch.stack(out), k, v]


def _work_attention(case):
    rows = sum(p + 1 for p in _positions(case))
    return dict(bytes=4 * rows * KV_HEADS * HEAD_DIM + case["sequences"] * 4 * (HEADS + KV_HEADS) * HEAD_DIM, flops=4 * rows * HEADS * HEAD_DIM)


# ---- requests through the served models ------------------------------------------------------------------------------
CONTEXT, SLOTS, WIDTH, VOCAB, FF = 1024, 8, 2048, 32768, 6144
SERVED_HEADS, SERVED_KV = 16, 4


def _config(family):
    if family == "quantised":
        return dict(architecture="cccc-llm", hidden=WIDTH, n_heads=SERVED_HEADS, n_kv_heads=SERVED_KV, head_dim=HEAD_DIM, ffn=FF, vocab=VOCAB, layers=4, rope_theta=1e6,
                    eps=1e-6, qk_norm=True)
    if family == "fakilorn":
        mixer = dict(heads=SERVED_HEADS, kv_heads=SERVED_KV, dim=HEAD_DIM, vdim=HEAD_DIM, scale=HEAD_DIM ** -0.5, v_mix=True)
        experts = dict(kind="moe", router=dict(experts=16, top=4), expert=dict(ff=768), shared=dict(ff=768))
        return dict(architecture="Fakilorn", width=WIDTH, vocab=VOCAB, embedding=dict(scale=8.0), logit_scale=1.0, norm=dict(eps=1e-5),
                    layers=[dict(type="attention", mixer=mixer, mlp=m) for m in (dict(kind="dense", ff=FF), dict(kind="dense", ff=FF), experts)])
    mask, rot = dict(size=CONTEXT), lambda dims: dict(base=1e6, dims=dims)
    mixers = [("mlstm", dict(heads=4, dim=256, vdim=512, gate_cap=15.0)),
              ("attention", dict(heads=SERVED_HEADS, kv_heads=SERVED_KV, dim=HEAD_DIM, vdim=HEAD_DIM, scale=HEAD_DIM ** -0.5, mask=mask, rot=rot(HEAD_DIM))),
              ("latent_attention", dict(heads=SERVED_HEADS, dim=128, rot_dim=64, vdim=128, q_rank=768, kv_rank=512, scale=192 ** -0.5, mask=mask, rot=rot(64)))]
    return dict(architecture="Tazunex", width=WIDTH, vocab=VOCAB, norm=dict(eps=1e-6), logit_softcap=30.0,
                layers=[dict(type=t, mixer=m, mlp=dict(kind="dense", ff=FF)) for t, m in mixers])


def _shapes(c):
    """name -> shape of the tensors of a model."""
    out, W = {}, WIDTH
    if c["architecture"] == "cccc-llm":
        q, kv = c["n_heads"] * c["head_dim"], c["n_kv_heads"] * c["head_dim"]
        for i in range(c["layers"]):
            out.update({"W_%s_%d" % (n, i): s for n, s in dict(q=(q, W), k=(kv, W), v=(kv, W), o=(W, q), gate=(FF, W), up=(FF, W), down=(W, FF)).items()})
            out.update({"W_rms_attn_%d" % i: (W,), "W_rms_ffn_%d" % i: (W,), "W_qnorm_%d" % i: (c["head_dim"],), "W_knorm_%d" % i: (c["head_dim"],)})
        out.update({"W_lm_head": (VOCAB, W), "W_emb": (VOCAB, W), "W_rms_final": (W,)})
        return out
    out["embed"] = (VOCAB, W)
    bias = c["architecture"] == "Fakilorn"
    norm = lambda n: out.update({n: (W,), n + ".b": (W,)} if bias else {n: (W,)})
    for i, L in enumerate(c["layers"]):
        m, f, p = L["mixer"], L["mlp"], "l%d." % i
        H, d, dv = m["heads"], m["dim"], m["vdim"]
        for n in ("norm1", "norm2") if bias else ("norm1", "norm2", "norm1b", "norm2b"):
            norm(p + n)
        if bias:
            t = dict(q=(H * d, W), k=(m["kv_heads"] * d, W), v=(m["kv_heads"] * dv, W), g=(H * dv, W), o=(W, H * dv), vmix=())
        elif L["type"] == "mlstm":
            t = {"q": (H * d, W), "k": (H * d, W), "v": (H * dv, W), "g": (H * dv, W), "o": (W, H * dv), "norm": (H * dv,), "i": (H, W), "i.b": (H,), "f": (H, W), "f.b": (H,)}
        elif L["type"] == "attention":
            t = {"q": (H * d, W), "k": (m["kv_heads"] * d, W), "q.norm": (H * d,), "k.norm": (m["kv_heads"] * d,), "sink": (H,), "o": (W, H * dv)}
        else:
            r, R, Q = m["rot_dim"], m["kv_rank"], m["q_rank"]
            t = {"dq": (Q, W), "dq.norm": (Q,), "uq": (H * (d + r), Q), "dkv": (R + r, W), "dkv.norm": (R,), "uk": (H * d, R), "uv": (H * dv, R), "g": (H, W), "o": (W, H * dv)}
        out.update({p + "mix." + n: s for n, s in t.items()})
        if f["kind"] == "moe":
            out[p + "mlp.router"], out[p + "mlp.shared.sg"] = (f["router"]["experts"], W), (1, W)
            for n, ff in [("e%d." % j, f["expert"]["ff"]) for j in range(f["router"]["experts"])] + [("shared.", f["shared"]["ff"])]:
                out.update({p + "mlp." + n + "gate": (ff, W), p + "mlp." + n + "up": (ff, W), p + "mlp." + n + "down": (W, ff)})
        else:
            out.update({p + "mlp." + n: s for n, s in (("gate", (FF, W)), ("up", (FF, W)), ("down", (W, FF))) if n != "gate" or not bias})
    norm("final.norm")
    return out


def _weights(family):
    """The model's tensors in BF16 on the GPU, the same in every process: linears N(0, 1 / inputs), norms near 1, small branches
    and forget gates that mostly keep (random recurrences with other weights are ill conditioned)."""
    out = {}
    for name, shape in _shapes(_config(family)).items():
        a = torch.randn(shape, device="cuda", generator=_generator(zlib.crc32(name.encode())))
        leaf = name.rsplit(".", 1)[-1]
        if name.endswith(".f.b"):
            a = 3 + 2 * a
        elif name.endswith("vmix"):
            a = 0.5 + 0.1 * a
        elif name.endswith(".b") and "norm" in name:
            a = 0.1 * a
        elif "norm" in leaf or "rms" in name or "qnorm" in name or "knorm" in name:
            a = (1 + 0.2 * a) * (0.035 if leaf in ("norm1b", "norm2b") else 1.0)
        elif name == "embed":
            a = a / math.sqrt(WIDTH) if family == "fakilorn" else 0.02 * (a + 0.4 * torch.randn(WIDTH, device="cuda", generator=_generator(7)))
        elif len(shape) == 2 and name != "W_emb":
            a = a / math.sqrt(shape[1]) * (3.0 if name.endswith((".mix.i", ".mix.f")) else 1.0)
        if name.endswith("l0.mix.k") and family == "tazunex":
            a = 0.9 * out["l0.mix.q"].float() + 0.44 * a
        out[name] = a.to(torch.bfloat16)
    return out


def _is_linear(name):
    return name.startswith("W_") and "norm" not in name and "rms" not in name and name != "W_emb"


def _bytes(t):
    return t.contiguous().reshape(-1).view(torch.uint8).cpu().numpy().tobytes()


def _folder(family):
    """The model's folder, written once: the weights are the same for every seed, the tokens are not."""
    top = os.path.join(tempfile.gettempdir(), "cccc_b200_models_%d" % os.getuid())
    path = os.path.join(top, "%s_%08x" % (family, zlib.crc32(json.dumps(_config(family), sort_keys=True).encode())))
    if os.path.isdir(path):
        return path
    os.makedirs(top, exist_ok=True)
    new = tempfile.mkdtemp(dir=top)
    with open(os.path.join(new, "config.json"), "w") as f:
        json.dump(_config(family), f)
    blobs = {}
    for name, t in _weights(family).items():
        if family == "quantised" and _is_linear(name):
            W, _, inv = _quantise(t.float(), "e4m3", True)
            blobs["weight_fp8_e4m3_" + name], blobs["scale_" + name] = (_bytes(W), None), (struct.pack("<f", inv), None)
        else:
            blobs[("weight_bf16_" if family == "quantised" else "") + name] = (_bytes(t), list(t.shape))
    at, index, head = 0, "", {}
    for name, (b, shape) in blobs.items():
        index += "%s = %d,%d\n" % (name, at, len(b))
        head[name] = dict(dtype="BF16", shape=shape, data_offsets=[at, at + len(b)])
        at += len(b)
    with open(os.path.join(new, "model.bin" if family == "quantised" else "model.safetensors"), "wb") as f:
        if family == "quantised":
            f.write(b"CFG_BIN INI" + bytes(21) + struct.pack("<Q", len(index)) + index.encode())
        else:
            h = json.dumps(head).encode()
            h += b" " * (-len(h) % 8)
            f.write(struct.pack("<Q", len(h)) + h)
        for b, _ in blobs.values():
            f.write(b)
    try:
        os.rename(new, path)
    except OSError:  # somebody else was first
        pass
    return path


def _lengths(case):
    """Prompts of unlike lengths around `prompt`."""
    S = case["sequences"]
    return [max(1, round(case["prompt"] * (0.5 + (i + 1) / (S + 1)))) for i in range(S)]


def _tokens(case, seed):
    r = np.random.default_rng(seed)
    return [[int(t) for t in r.integers(0, VOCAB, n + case["decode"])] for n in _lengths(case)]


def _prepare_request(case, seed):
    pkg = _package()
    lib = pkg.hostapi.lib()
    for name, (res, args) in pkg.serve.SYMBOLS.items():
        getattr(lib, name).restype, getattr(lib, name).argtypes = res, args

    class Served(pkg.serve.Model):
        """serve.Model over the built libraries as they are."""

        def __init__(self, folder):
            self.h, self.lib, err = None, lib, ctypes.create_string_buffer(1024)
            self.h = lib.cccc_model_open(os.fsencode(folder), 0, pkg.serve.BFLOAT16, CONTEXT, SLOTS, 2048, 0, err, 1024)
            if not self.h:
                raise RuntimeError(err.value.decode())
            self.vocab = self.info(0)

        def __del__(self):
            self.close()

    return dict(model=Served(_folder(case["family"])), tokens=_tokens(case, seed), decode=case["decode"])


def _run_request(s):
    m, out = s["model"], []
    D = s["decode"]
    slots = [m.open_slot() for _ in s["tokens"]]
    entries = [(slot, t[:-D], [len(t) - D - 1]) for slot, t in zip(slots, s["tokens"])]
    for i in range(D + 1):
        logits, _ = m.step(entries)
        out.append(np.frombuffer(logits, np.float32).reshape(len(slots), -1))
        entries = [(slot, [t[len(t) - D + i]], [0]) for slot, t in zip(slots, s["tokens"])] if i < D else []
    for slot in slots:
        m.close_slot(slot)
    return out


def _exact_request(case, seed):
    """The whole sequences at once, without a cache, padded to the longest (later tokens do not change earlier ones)."""
    tokens, D = _tokens(case, seed), case["decode"]
    T = max(len(t) for t in tokens)
    ids = torch.tensor([t + [0] * (T - len(t)) for t in tokens], device="cuda")
    family, c = case["family"], _config(case["family"])
    w = _weights(family)
    if family == "quantised":
        w = {n: _dequantise(_quantise(t.float(), "e4m3", True), "e4m3").to(torch.bfloat16) if _is_linear(n) else t for n, t in w.items()}
    x = {"quantised": _forward_quantised, "fakilorn": _forward_fakilorn, "tazunex": _forward_tazunex}[family](c, w, ids)
    rows = torch.stack([torch.stack([x[b, n - 1 + i] for b, n in enumerate(_lengths(case))]) for i in range(D + 1)])
    head = w["W_lm_head" if family == "quantised" else "embed"].double()
    z = rows @ head.T
    return list((c["logit_softcap"] * torch.tanh(z / c["logit_softcap"]) if family == "tazunex" else z).unbind(0))


def _softmax_attention(q, k, v, scale, sink=None):
    """q [T, H, d], k, v [T, G, .] of one sequence, causal; sink [H]: a score that takes part in the denominator only."""
    T, H = q.shape[:2]
    k, v = (a.repeat_interleave(H // a.shape[1], 1).transpose(0, 1) for a in (k, v))
    s = (q.transpose(0, 1) @ k.transpose(1, 2)) * scale
    s = s.masked_fill(torch.ones(T, T, dtype=torch.bool, device=s.device).triu(1), -math.inf)
    if sink is not None:
        s = torch.cat([s, sink[:, None, None].expand(H, T, 1)], -1)
    return (torch.softmax(s, -1)[..., :T] @ v).transpose(0, 1)


def _rms(x, weight, eps):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps) * weight


def _forward_quantised(c, w, ids):
    H, G, d, eps = c["n_heads"], c["n_kv_heads"], c["head_dim"], c["eps"]
    W = lambda n: w[n].double()
    cos, sin = (t.double()[:, None] for t in _rope_tables(ids.shape[1], d, c["rope_theta"]))
    x = W("W_emb")[ids]
    for i in range(c["layers"]):
        h = _rms(x, W("W_rms_attn_%d" % i), eps)
        q, k, v = ((h @ W("W_%s_%d" % (n, i)).T).unflatten(-1, (-1, d)) for n in "qkv")
        q, k = _norm_rotate(q, W("W_qnorm_%d" % i), cos, sin, eps), _norm_rotate(k, W("W_knorm_%d" % i), cos, sin, eps)
        x = x + torch.stack([_softmax_attention(*a, d ** -0.5) for a in zip(q, k, v)]).flatten(2) @ W("W_o_%d" % i).T
        h = _rms(x, W("W_rms_ffn_%d" % i), eps)
        x = x + (torch.nn.functional.silu(h @ W("W_gate_%d" % i).T) * (h @ W("W_up_%d" % i).T)) @ W("W_down_%d" % i).T
    return _rms(x, W("W_rms_final"), eps)


def _forward_fakilorn(c, w, ids):
    eps, W, first = c["norm"]["eps"], lambda n: w[n].double(), None
    norm = lambda x, n: torch.nn.functional.layer_norm(x, x.shape[-1:], W(n), W(n + ".b"), eps)
    gated = lambda h, p: (torch.nn.functional.silu(h @ W(p + "gate").T) * (h @ W(p + "up").T)) @ W(p + "down").T
    x = W("embed")[ids] * c["embedding"]["scale"]
    for i, L in enumerate(c["layers"]):
        p, m, f = "l%d." % i, L["mixer"], L["mlp"]
        h = norm(x, p + "norm1")
        q, k, v = ((h @ W(p + "mix." + n).T).unflatten(-1, (m["heads"] if n == "q" else m["kv_heads"], -1)) for n in "qkv")
        q, k = _rms(q, 1.0, eps), _rms(k, 1.0, eps)
        mix = float(w[p + "mix.vmix"])
        first, v = (v, v) if first is None else (first, (1 - mix) * v + mix * first)
        o = torch.stack([_softmax_attention(*a, m["scale"]) for a in zip(q, k, v)]).flatten(2)
        x = x + (o * torch.sigmoid(h @ W(p + "mix.g").T)) @ W(p + "mix.o").T
        h, p = norm(x, p + "norm2"), p + "mlp."
        if f["kind"] == "dense":
            x = x + torch.relu(h @ W(p + "up").T) ** 2 @ W(p + "down").T
            continue
        best = (h @ W(p + "router").T).topk(f["router"]["top"], -1)
        share = torch.zeros(*h.shape[:2], f["router"]["experts"], dtype=h.dtype, device=h.device).scatter(-1, best.indices, torch.softmax(best.values, -1))
        x = x + torch.sigmoid(h @ W(p + "shared.sg").T) * gated(h, p + "shared.") + sum(share[..., j:j + 1] * gated(h, p + "e%d." % j) for j in range(share.shape[-1]))
    return norm(x, "final.norm")


def _forward_tazunex(c, w, ids):
    eps, W, T = c["norm"]["eps"], lambda n: w[n].double(), ids.shape[1]
    gelu = lambda z: torch.nn.functional.gelu(z, approximate="tanh")

    def rotate(x, r, pairs):
        n, dims = torch.arange(T, dtype=torch.float64, device="cuda")[:, None, None], r["dims"]
        a = n * r["base"] ** (-2.0 * torch.arange(dims // 2, dtype=torch.float64, device="cuda") / dims)
        u, v = (x[..., :dims:2], x[..., 1:dims:2]) if pairs else x[..., :dims].chunk(2, -1)
        t = u * a.cos() - v * a.sin(), v * a.cos() + u * a.sin()
        return torch.cat([torch.stack(t, -1).flatten(-2) if pairs else torch.cat(t, -1), x[..., dims:]], -1)

    def attention(h, m, p):
        raw, q = h @ W(p + "k").T, _rms(h @ W(p + "q").T, W(p + "q.norm"), eps).unflatten(-1, (m["heads"], -1))
        k = _rms(raw, W(p + "k.norm"), eps).unflatten(-1, (m["kv_heads"], -1))
        q, k, v = rotate(q, m["rot"], False), rotate(k, m["rot"], False), raw.unflatten(-1, (m["kv_heads"], -1))
        return torch.stack([_softmax_attention(*a, m["scale"], W(p + "sink")) for a in zip(q, k, v)]).flatten(2) @ W(p + "o").T

    def latent(h, m, p):
        d, R, H = m["dim"], m["kv_rank"], m["heads"]
        q = (_rms(h @ W(p + "dq").T, W(p + "dq.norm"), eps) @ W(p + "uq").T).unflatten(-1, (H, -1))
        down = h @ W(p + "dkv").T
        latents, k_rot = _rms(down[..., :R], W(p + "dkv.norm"), eps), rotate(down[..., None, R:], m["rot"], True)
        k = torch.cat([(latents @ W(p + "uk").T).unflatten(-1, (H, -1)), k_rot.expand(-1, -1, H, -1)], -1)
        q = torch.cat([q[..., :d], rotate(q[..., d:], m["rot"], True)], -1)
        o = torch.stack([_softmax_attention(*a, m["scale"]) for a in zip(q, k, (latents @ W(p + "uv").T).unflatten(-1, (H, -1)))])
        return (o * torch.sigmoid(h @ W(p + "g").T)[..., None]).flatten(2) @ W(p + "o").T

    def mlstm(h, m, p):
        H, d, dv, cap = m["heads"], m["dim"], m["vdim"], m["gate_cap"]
        q, k, v = ((h @ W(p + n).T).unflatten(-1, (H, -1)) for n in "qkv")
        q = q * d ** -0.5
        gate = lambda n: cap * torch.tanh((h @ W(p + n).T + W(p + n + ".b")) / cap)
        log_i, log_f = gate("i"), torch.nn.functional.logsigmoid(gate("f"))
        zeros = lambda *s: torch.zeros(h.shape[0], H, *s, dtype=h.dtype, device=h.device)
        S, n, top, out = zeros(d, dv), zeros(d), zeros(), []
        for t in range(T):
            new = torch.maximum(log_f[:, t] + top, log_i[:, t])
            keep, add, top = torch.exp(log_f[:, t] + top - new), torch.exp(log_i[:, t] - new), new
            S = keep[..., None, None] * S + (add[..., None] * k[:, t])[..., None] * v[:, t, :, None]
            n = keep[..., None] * n + add[..., None] * k[:, t]
            z = torch.maximum((n * q[:, t]).sum(-1).abs(), torch.exp(-top)) + 1e-6
            out.append((q[:, t, :, None] @ S).squeeze(2) / z[..., None])
        o = _rms(torch.stack(out, 1), 1.0, eps).flatten(2) * W(p + "norm") * torch.sigmoid(h @ W(p + "g").T)
        return o @ W(p + "o").T

    x = W("embed")[ids]
    for i, L in enumerate(c["layers"]):
        p = "l%d." % i
        y = {"attention": attention, "latent_attention": latent, "mlstm": mlstm}[L["type"]](_rms(x, W(p + "norm1"), eps), L["mixer"], p + "mix.")
        x = x + _rms(y, W(p + "norm1b"), eps)
        h = _rms(x, W(p + "norm2"), eps)
        x = x + _rms((gelu(h @ W(p + "mlp.gate").T) * (h @ W(p + "mlp.up").T)) @ W(p + "mlp.down").T, W(p + "norm2b"), eps)
    return _rms(x, W("final.norm"), eps)


def _work_request(case):
    """Weights and caches once per step, the linears' and the attention's arithmetic once per token."""
    c, S, D = _config(case["family"]), case["sequences"], case["decode"]
    lengths, shapes = _lengths(case), _shapes(c)
    each = 1 if case["family"] == "quantised" else 2
    table = VOCAB * WIDTH
    linears = sum(s[0] * s[1] for n, s in shapes.items() if len(s) == 2 and n not in ("W_emb", "embed", "W_lm_head"))
    experts = sum(s[0] * s[1] for n, s in shapes.items() if ".mlp.e" in n)
    active, read = linears - experts * 3 // 4, linears - experts + experts * (1 - 0.75 ** S)    # four of sixteen experts for each token
    tokens = sum(lengths) + S * D
    pairs = sum((n + D) * (n + D + 1) / 2 for n in lengths)
    rows = sum(sum(n + i for i in range(D)) for n in lengths)
    if case["family"] == "tazunex":
        heads, cache, state = 2 * SERVED_HEADS * 256 + 2 * SERVED_HEADS * 320, 2 * (SERVED_KV * 256 + 576), 8 * 4 * 256 * 512
    else:
        layers = c["layers"] if case["family"] == "quantised" else len(c["layers"])
        heads, cache, state = 4 * layers * SERVED_HEADS * HEAD_DIM, 4 * layers * SERVED_KV * HEAD_DIM, 0
    return dict(bytes=each * (linears + table + D * (read + table)) + cache * (rows + tokens) + state * S * D + 4 * S * (D + 1) * VOCAB,
                flops=2 * active * tokens + 2 * table * S * (D + 1) + heads * pairs)


# ---- what is asked of a case ----------------------------------------------------------------------------------------
def prepare(case, seed):
    return dict({"linear": _prepare_linear, "layer": _prepare_linear, "attention": _prepare_attention, "request": _prepare_request}[case["kind"]](case, seed), kind=case["kind"])


def run(state):
    return {"linear": _run_linear, "layer": _run_linear, "attention": _run_attention, "request": _run_request}[state["kind"]](state)


def exact(case, seed):
    return {"linear": _exact_linear, "layer": _exact_linear, "attention": _exact_attention, "request": _exact_request}[case["kind"]](case, seed)


def work(case):
    return {"linear": _work_linear, "layer": _work_linear, "attention": _work_attention, "request": _work_request}[case["kind"]](case)


def tolerance(case):
    """Linears: one rounding to BF16.  Attention: scores and probabilities are BF16 tensors too.  Requests: BF16 activations
    through a few layers, and a router or a recurrence that may decide a close call the other way."""
    if case["kind"] in ("linear", "layer"):
        return dict(rel=6e-3, max=0.02)
    return dict(rel=0.02, max=0.1) if case["kind"] == "attention" else dict(rel=0.03, max=0.25)

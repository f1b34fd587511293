"""Prompts of the quantised model in passes of many tokens: the append kernel against the decode attention's own append bit for
bit, and the served model's logits against token-by-token decoding of the same sequences."""
import json

import numpy as np
import pytest

from __graft_entry__ import load_package
from oracle import oracle as O
from tests._util import capi, from_dev_u16, to_dev

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("hd,H,Hkv,tokens,norm", [(128, 4, 1, 1, True), (128, 16, 2, 37, True), (128, 3, 3, 5, False), (64, 8, 4, 130, True), (64, 1, 1, 3, False)])
def test_append_has_the_bits_of_the_decode_kernel(hd, H, Hkv, tokens, norm):
    import torch

    c, T, rng = capi(), 64, np.random.default_rng(hd + tokens)
    bf = lambda *s: to_dev(O.f32_to_bf16_bits(rng.standard_normal(s).astype(np.float32)))
    ld = (H + 2 * Hkv) * hd + 8
    x = bf(tokens, ld)
    # a query head that is a copy of a key head: both take the same norm and rotation
    x[:, :hd] = x[:, H * hd:(H + 1) * hd]
    w, cos, sin = bf(hd), bf(T, hd // 2), bf(T, hd // 2)
    pos = torch.from_numpy(rng.integers(0, T, tokens).astype(np.int32)).cuda()
    pos[0] = T - 1
    slot = torch.arange(tokens - 1, -1, -1, dtype=torch.int32, device="cuda")
    at = lambda n: x.data_ptr() + 2 * n * hd
    out = {}
    for name, B in (("append", tokens), ("decode", tokens)):
        k, v = torch.zeros(tokens, Hkv, T, hd, dtype=torch.int16, device="cuda"), torch.zeros(tokens, Hkv, T, hd, dtype=torch.int16, device="cuda")
        q = torch.zeros(tokens, H * hd, dtype=torch.int16, device="cuda")
        p = pos
        d = c.make_attn_decode(q=at(0), k=at(H), v=at(H + Hkv), k_cache=k, v_cache=v, pos=p, out=q, cos_tab=cos, sin_tab=sin, q_norm=w if norm else None,
                               k_norm=w if norm else None, B=B, H=H, Hkv=Hkv, head_dim=hd, T_max=T, ldq=ld, ldk=ld, ldv=ld, slot=slot)
        if H // Hkv not in (1, 2, 4, 8) and name == "decode":
            pytest.skip("the decode kernel takes other head counts")
        assert (c.attn_append_bf16 if name == "append" else c.attn_decode_bf16)(d) == 0 and c.check_error(name) == 0
        out[name] = (k, v, q, p)
    k, v, q, p = out["append"]
    assert torch.equal(k, out["decode"][0]) and torch.equal(v, out["decode"][1])
    rows = k[slot.long(), 0, p.long()]
    assert torch.equal(q[:, :hd], rows)
    # a position past the cache: the queries are still written, the cache is not
    before = k.clone()
    far = torch.full_like(p, T - 1)
    d = c.make_attn_decode(q=at(0), k=at(H), v=at(H + Hkv), k_cache=k, v_cache=v, pos=far, out=q, cos_tab=cos, sin_tab=sin, B=tokens, H=H, Hkv=Hkv, head_dim=hd,
                           T_max=T - 1, ldq=ld, ldk=ld, ldv=ld, slot=slot)
    assert c.attn_append_bf16(d) == 0 and c.check_error("append past the end") == 0 and torch.equal(k, before)


@pytest.fixture(scope="module")
def folder(tmp_path_factory):
    from tests.test_gpu_decode_model import make_model
    from tests.test_gpu_host_step import container_entries, small_cfg
    from tests.test_loader_cpu import write_container

    d, cfg = tmp_path_factory.mktemp("quantised"), small_cfg(True)
    write_container(str(d / "model.bin"), container_entries(O.FP8_E5M2, cfg, make_model(O.FP8_E5M2, cfg, seed=4)))
    (d / "config.json").write_text(json.dumps(dict(architecture="cccc-llm", hidden=cfg.hidden, n_heads=cfg.n_heads, n_kv_heads=cfg.n_kv_heads, head_dim=cfg.head_dim,
                                                   ffn=cfg.ffn, vocab=cfg.vocab, layers=cfg.layers, rope_theta=cfg.rope_theta, eps=cfg.eps, qk_norm=cfg.qk_norm)))
    return str(d), cfg


def error(got, want):
    return float(np.sqrt(((got - want) ** 2).mean(1)).max() / want.std())


# cap 400: passes of up to 400 tokens; 48: longer steps run in several, which cut entries anywhere
@pytest.mark.parametrize("cap", [400, 48])
def test_prompts_match_decoding_token_by_token(folder, cap):
    d, cfg = folder
    m = load_package().serve.Model(d, max_context=256, max_sequences=3, max_step_tokens=cap)
    rng = np.random.default_rng(cap)
    seqs = [[int(t) for t in rng.integers(0, cfg.vocab, n)] for n in (150, 33, 2)]
    want = []
    for s in seqs:
        slot = m.open_slot()
        want.append(np.concatenate([np.array(m.step([(slot, [t], [0])])[0]).reshape(1, -1) for t in s]))
        m.close_slot(slot)
    # BF16 activations through the same layers, the scores of a prompt in float: as far apart as two decode batches are
    bar = 0.03
    for cuts in ([1.0], [0.1, 0.5, 1.0], [0.5, 0.55, 0.6, 1.0]):
        slots, at = [m.open_slot() for _ in seqs], [0] * len(seqs)
        got = [[] for _ in seqs]
        for part in cuts:
            entries = []
            for i, s in enumerate(seqs):
                n = int(round(len(s) * part)) - at[i]
                if n > 0:
                    entries.append((slots[i], s[at[i]:at[i] + n], list(range(n - 1, -1, -1))))
            lg, ch = m.step(entries, choice=True)
            lg, at_row = np.array(lg).reshape(len(ch), -1), 0
            for slot, t, _ in entries:
                i = slots.index(slot)
                got[i].append(lg[at_row:at_row + len(t)][::-1])
                assert ch[at_row:at_row + len(t)] == [int(np.argmax(r)) for r in lg[at_row:at_row + len(t)]]
                at_row += len(t)
                at[i] += len(t)
                assert m.slot_length(slot) == at[i]
        for i, s in enumerate(seqs):
            assert error(np.concatenate(got[i]), want[i]) < bar, (cuts, i, error(np.concatenate(got[i]), want[i]))
            m.close_slot(slots[i])
    m.close()


@pytest.mark.parametrize("hd,H,Hkv", [(128, 4, 2), (64, 8, 1)])
def test_append_past_the_cache_writes_the_queries_alone(hd, H, Hkv):
    import torch

    c, T, tokens, rng = capi(), 32, 9, np.random.default_rng(hd)
    bf = lambda *s: to_dev(O.f32_to_bf16_bits(rng.standard_normal(s).astype(np.float32)))
    x, w, cos, sin = bf(tokens, (H + 2 * Hkv) * hd), bf(hd), bf(T, hd // 2), bf(T, hd // 2)
    pos = torch.full((tokens,), T - 1, dtype=torch.int32, device="cuda")
    pos[3] = T - 2    # the last row of the smaller cache
    out = {}
    for rows in (T, T - 1):
        k, v, q = torch.zeros(tokens, Hkv, rows, hd, dtype=torch.int16, device="cuda"), torch.zeros(tokens, Hkv, rows, hd, dtype=torch.int16, device="cuda"), torch.zeros(
            tokens, H * hd, dtype=torch.int16, device="cuda")
        at = lambda n: x.data_ptr() + 2 * n * hd
        d = c.make_attn_decode(q=at(0), k=at(H), v=at(H + Hkv), k_cache=k, v_cache=v, pos=pos, out=q, cos_tab=cos, sin_tab=sin, q_norm=w, k_norm=w, B=tokens, H=H, Hkv=Hkv,
                               head_dim=hd, T_max=rows, ldq=x.shape[1], ldk=x.shape[1], ldv=x.shape[1])
        assert c.attn_append_bf16(d) == 0 and c.check_error("append") == 0
        out[rows] = (k, v, q)
    (k, v, q), (k1, v1, q1) = out[T], out[T - 1]
    assert bool(q.any(1).all()) and torch.equal(q, q1)
    k[:, :, T - 1], v[:, :, T - 1] = 0, 0    # what the smaller cache has no row for
    assert bool(k[3].any()) and torch.equal(k[:, :, :T - 1], k1) and torch.equal(v[:, :, :T - 1], v1)

"""No GPU needed: the host side of the served quantised model - loading, steps, their halves, prompts in passes - over a stand-in
for the device (tests/fake_device.cpp), which runs the default stream's work as late as the runtime allows."""
import json
import os
import struct
import subprocess
import sys

import numpy as np
import pytest

from __graft_entry__ import ROOT, load_package
from tests.test_loader_cpu import write_container

HIDDEN, HEADS, KV, DIM, FF, VOCAB, LAYERS = 128, 2, 1, 64, 128, 256, 2

PRELUDE = """
import ctypes as C, json, os, sys
import numpy as np
sys.path.insert(0, %r)
from __graft_entry__ import load_package
serve = load_package().serve
fake = C.CDLL(os.environ["LD_PRELOAD"])
fake.fake_seen.restype = C.c_ulonglong
seen = lambda: dict(zip(("wild", "decode", "prompt", "bytes"), (fake.fake_seen(i) for i in range(4))))

def rows(logits):
    return np.array(logits, np.float32).reshape(-1, %d)

def bf16(x):
    u = np.float32(x).view(np.uint32)
    return ((u + 0x7FFF + ((u >> 16) & 1)) & 0xFFFF0000).astype(np.uint32).view(np.float32)

def expected(tokens):
    out = np.repeat(np.float32(tokens)[:, None], %d, 1)
    for r, t in zip(out, tokens):
        r[t] = bf16(t + 1000)
    return out

FOLDER = sys.argv[1]
""" % (ROOT, VOCAB, VOCAB)


@pytest.fixture(scope="module")
def run(tmp_path_factory):
    """Runs a program over the stand-in; what it prints last, as JSON."""
    top = tmp_path_factory.mktemp("served")
    shim = str(top / "fake_device.so")
    subprocess.check_call(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", "-I/usr/local/cuda/include", "-o", shim, os.path.join(ROOT, "tests", "fake_device.cpp")])
    load_package().serve.library("cccc-llm")    # built before anything is preloaded
    e = {}
    for i in range(LAYERS):
        for n, (N, K) in dict(q=(HEADS * DIM, HIDDEN), k=(KV * DIM, HIDDEN), v=(KV * DIM, HIDDEN), o=(HIDDEN, HEADS * DIM), gate=(FF, HIDDEN), up=(FF, HIDDEN),
                              down=(HIDDEN, FF)).items():
            e["weight_fp8_e4m3_W_%s_%d" % (n, i)], e["scale_W_%s_%d" % (n, i)] = bytes(N * K), struct.pack("<f", 1.0)
        e["weight_bf16_W_rms_attn_%d" % i] = e["weight_bf16_W_rms_ffn_%d" % i] = bytes(2 * HIDDEN)
    e["weight_fp8_e4m3_W_lm_head"], e["scale_W_lm_head"] = bytes(VOCAB * HIDDEN), struct.pack("<f", 1.0)
    e["weight_bf16_W_emb"] = np.repeat((np.arange(VOCAB, dtype=np.float32).view(np.uint32) >> 16).astype(np.uint16), HIDDEN).tobytes()
    e["weight_bf16_W_rms_final"] = bytes(2 * HIDDEN)
    write_container(str(top / "model.bin"), e)
    (top / "config.json").write_text(json.dumps(dict(architecture="cccc-llm", hidden=HIDDEN, n_heads=HEADS, n_kv_heads=KV, head_dim=DIM, ffn=FF, vocab=VOCAB,
                                                     layers=LAYERS, rope_theta=1e4, eps=1e-6, qk_norm=False)))

    def go(program):
        r = subprocess.run([sys.executable, "-c", PRELUDE + program, str(top)], env=dict(os.environ, LD_PRELOAD=shim), capture_output=True, text=True, timeout=300)
        assert r.returncode == 0, r.stderr[-2000:]
        return json.loads(r.stdout.strip().splitlines()[-1])

    return go


def test_the_first_step_finds_its_ids_positions_and_slots_cleared(run):
    assert run("""
m = serve.Model(FOLDER, max_context=16, max_sequences=3)
print(json.dumps(seen()))
""")["wild"] == 0


def test_steps_and_prompts_over_the_stand_in(run):
    s = run("""
m = serve.Model(FOLDER, max_context=32, max_sequences=3)
a, b = m.open_slot(), m.open_slot()
ok = True
lg, ch = m.step([(b, [7, 9, 11], [2, 0]), (a, [5], [0])], choice=True)
ok &= np.array_equal(rows(lg), expected([11, 7, 5])) and ch == [11, 7, 5]
lg, ch = m.step([(a, [200], [0]), (b, [3], [0])], choice=True)
ok &= np.array_equal(rows(lg), expected([200, 3])) and ch == [200, 3] and [m.slot_length(x) for x in (a, b)] == [2, 4]
print(json.dumps(dict(seen(), ok=bool(ok))))
""")
    assert s["ok"] and s["wild"] == 0 and s["prompt"] == LAYERS


def test_the_halves_of_a_step_give_what_begin_was_told_of(run):
    s = run("""
m = serve.Model(FOLDER, max_context=32, max_sequences=3)
a = m.open_slot()
ints = lambda *v: (C.c_int * max(1, len(v)))(*v)
def halves(tokens, want, logits, choice):
    lg, ch = np.full((len(want), m.vocab), -1, np.float32), ints(*[-1] * len(want))
    assert m.lib.cccc_model_step_begin(m.h, 1, ints(a), ints(len(tokens)), ints(*tokens), ints(len(want)), ints(*want), logits, choice) == 0
    assert m.lib.cccc_model_step_end(m.h, lg.ctypes.data_as(C.POINTER(C.c_float)), ch) == 0
    e = [tokens[w] for w in want]
    return bool(np.array_equal(lg, expected(e)) if logits else (lg == -1).all()), list(ch) == (e if choice else [-1] * len(want))
out = [halves(t, w, lg, ch) for t, w in (([9], [0]), ([4, 8], [1, 0])) for lg, ch in ((1, 1), (0, 1), (1, 0), (0, 0))]
print(json.dumps(out))
""")
    assert s == [[True, True]] * 8


def test_places_wanted_several_times_in_a_step_of_several_passes(run):
    s = run("""
m = serve.Model(FOLDER, max_context=64, max_sequences=2, max_step_tokens=8)
a, b = m.open_slot(), m.open_slot()
tokens, want = list(range(20, 30)), [9] * 7 + [0, 9, 3]       # the second pass has two tokens and eight wants
lg, ch = m.step([(b, [100], [0]), (a, tokens, want)], choice=True)
e = [100] + [tokens[w] for w in want]
print(json.dumps([bool(np.array_equal(rows(lg), expected(e))), ch == e, m.slot_length(a)]))
""")
    assert s == [True, True, 10]


@pytest.mark.parametrize("vocab", [1 << 46, 1 << 62])    # beyond the address space, beyond what a size can say
def test_a_step_without_memory_for_its_logits_has_not_run(vocab):
    class Lib:
        begun = 0

        def cccc_model_step_begin(self, *_):
            self.begun += 1
            return 0

        def cccc_model_step_end(self, *_):
            return 0

    serve = load_package().serve
    m = serve.Model.__new__(serve.Model)
    m.lib, m.h, m.vocab = Lib(), None, vocab
    with pytest.raises(MemoryError):
        m.step([(0, [1], [0])], choice=True)
    assert m.lib.begun == 0
    assert m.step([(0, [1], [0])], logits=False, choice=True) == (None, [0]) and m.lib.begun == 1


def test_prompts_hold_no_more_than_a_step_can_have(run):
    bytes_at = [run("""
m = serve.Model(FOLDER, max_context=16, max_sequences=3, max_step_tokens=%d)
a = m.open_slot()
assert np.array_equal(rows(m.step([(a, [1] * 16, [15])])[0]), expected([1]))
print(json.dumps(seen()))
""" % n)["bytes"] for n in (32, 48, 4096)]
    assert bytes_at[0] < bytes_at[1] == bytes_at[2]


# (tokens of the sequences, tokens of a pass) -> passes, or 0: decode steps, one for each place of the longest sequence
@pytest.mark.parametrize("lengths,cap,passes", [((10,), 1, 0), ((10,), 2, 5), ((10, 10), 2, 0), ((10, 9), 2, 0), ((10, 7), 2, 9), ((1, 2), 4096, 1), ((8, 8, 8), 3, 0)])
def test_prompts_run_in_passes_where_that_takes_fewer(run, lengths, cap, passes):
    s = run("""
lengths, cap = %r
m = serve.Model(FOLDER, max_context=16, max_sequences=3, max_step_tokens=cap)
before = seen()
e = [(m.open_slot(), [10 * i + j for j in range(n)], [0, n - 1]) if n > 1 else (m.open_slot(), [10 * i], [0]) for i, n in enumerate(lengths)]
lg, ch = m.step(e, choice=True)
want = [t[w] for _, t, ws in e for w in ws]
ok = ch == want and np.array_equal(rows(lg), expected(want)) and [m.slot_length(x) for x, _, _ in e] == list(lengths)
print(json.dumps(dict(ok=bool(ok), **{n: seen()[n] - before[n] for n in ("decode", "prompt", "wild")})))
""" % ((lengths, cap),))
    assert s == dict(ok=True, decode=0 if passes else LAYERS * max(lengths), prompt=LAYERS * passes, wild=0)

"""A step in two halves (cccc_model_step_begin / _end, what serve.Model.step calls) against the step in one, which it has the bits
of: decode steps that are started ahead, steps that are not (prompts, entries without wants), results that are not taken."""
import ctypes as C
import json

import numpy as np
import pytest

from __graft_entry__ import load_package
from oracle import fakilorn as F
from tests.test_gpu_fakilorn import CONFIGS, tokens_for
from tests.test_gpu_prompt import folder  # noqa: F401 (a fixture)

pytestmark = pytest.mark.gpu


def ints(values):
    values = list(values)
    return (C.c_int * max(1, len(values)))(*values)


def flat(entries):
    return (len(entries), ints(s for s, _, _ in entries), ints(len(t) for _, t, _ in entries), ints(x for _, t, _ in entries for x in t),
            ints(len(w) for _, _, w in entries), ints(x for _, _, w in entries for x in w))


# rows of the four pieces that go to the host one after the other: fewer, as many, uneven
@pytest.mark.parametrize("n", [1, 3, 4, 9])
def test_the_halves_give_the_bits_of_the_whole(tmp_path, n):
    c = CONFIGS["odd"]
    (tmp_path / "config.json").write_text(json.dumps(c))
    F.write_safetensors(str(tmp_path / "model.safetensors"), F.random_weights(c, seed=5))
    serve = load_package().serve
    a, b = (serve.Model(str(tmp_path), max_context=64, max_sequences=9) for _ in range(2))
    V, slots = a.vocab, [(a.open_slot(), b.open_slot()) for _ in range(n)]
    assert all(x == y for x, y in slots)
    slots = [x for x, _ in slots][::-1]    # entries in another order than their slots
    steps = [[(s, tokens_for(c, 3 + s, s), [2 + s, 0]) for s in slots]]
    steps += [[(s, tokens_for(c, 1, 100 * i + s), [0]) for s in slots] for i in range(4)]
    steps += [[(s, tokens_for(c, 1, s), [] if s % 2 else [0]) for s in slots], [(s, tokens_for(c, 1 + s % 2, s), [0]) for s in slots]]
    for i, e in enumerate(steps):
        wanted = sum(len(w) for _, _, w in e)
        want, ids = np.zeros((wanted, V), np.float32), ints([0] * wanted)
        assert a.lib.cccc_model_step(a.h, *flat(e), want.ctypes.data_as(C.POINTER(C.c_float)), ids) == 0
        got, chosen = b.step(e, logits=i != 3, choice=i != 4)
        assert (got is None) == (i == 3) and (got is None or np.array_equal(np.frombuffer(got, np.float32).reshape(wanted, V), want))
        assert chosen is None if i == 4 else chosen == list(ids[:wanted])
        assert [b.slot_length(s) for s in slots] == [a.slot_length(s) for s in slots]
    # begun, and its results not taken: the next step does not see any of it
    e = steps[1]
    assert b.lib.cccc_model_step_begin(b.h, *flat(e), 1, 0) == 0 and b.lib.cccc_model_step_end(b.h, None, None) == 0
    a.step(e)
    assert np.array_equal(np.array(a.step(steps[2])[0]), np.array(b.step(steps[2])[0]))
    # entries that cannot run: nothing to end
    assert b.lib.cccc_model_step_begin(b.h, *flat([(slots[0], [c["vocab"]], [0])]), 1, 0) == -1
    a.close(), b.close()


def test_the_halves_of_the_quantised_model(folder):  # noqa: F811
    serve = load_package().serve
    d, cfg = folder
    a, b = (serve.Model(d, max_context=64, max_sequences=3) for _ in range(2))
    rng = np.random.default_rng(3)
    slots = [(a.open_slot(), b.open_slot())[0] for _ in range(3)]
    token = lambda n=1: [int(t) for t in rng.integers(0, cfg.vocab, n)]
    steps = [[(s, token(5 + s), [0, 4]) for s in slots], [(s, token(), [0]) for s in slots], [(s, token(), [] if s else [0]) for s in slots], [(slots[1], token(2), [1, 0])],
             [(s, token(), [0]) for s in slots[::-1]], [(s, token(), [0]) for s in slots]]
    for i, e in enumerate(steps):
        wanted = sum(len(w) for _, _, w in e)
        want, got, ids = np.zeros((wanted, cfg.vocab), np.float32), np.full((wanted, cfg.vocab), -1, np.float32), [ints([-1] * wanted) for _ in range(2)]
        pointer = lambda x: x.ctypes.data_as(C.POINTER(C.c_float))
        assert a.lib.cccc_model_step(a.h, *flat(e), pointer(want), ids[0]) == 0
        assert b.lib.cccc_model_step_begin(b.h, *flat(e), i != 4, i != 3) == 0 and b.lib.cccc_model_step_end(b.h, pointer(got), ids[1]) == 0
        assert np.array_equal(got, want) if i != 4 else (got == -1).all()
        assert list(ids[1]) == (list(ids[0]) if i != 3 else [-1] * wanted)
        assert [b.slot_length(s) for s in slots] == [a.slot_length(s) for s in slots]
    a.close(), b.close()


@pytest.mark.parametrize("n", [1, 8, 16, 17])
def test_logits_alone_are_those_beside_the_choice(tmp_path, n):
    """Up to sixteen rows the head writes logits that nothing chooses from into the host's memory; steps of both kinds by turns."""
    c = CONFIGS["odd"]
    (tmp_path / "config.json").write_text(json.dumps(c))
    F.write_safetensors(str(tmp_path / "model.safetensors"), F.random_weights(c, seed=6))
    serve = load_package().serve
    a, b = (serve.Model(str(tmp_path), max_context=64, max_sequences=n) for _ in range(2))
    slots = [(a.open_slot(), b.open_slot())[0] for _ in range(n)]
    for i in range(8):
        e = [(s, tokens_for(c, 1, 7 * i + s), [0]) for s in slots]
        want, chosen = a.step(e, choice=True)
        got, none = b.step(e, choice=i in (3, 6))
        assert got == want and (none is None or none == chosen)
    a.close(), b.close()


@pytest.mark.parametrize("n", [1, 16, 17])
def test_logits_alone_of_the_quantised_model(folder, n):  # noqa: F811
    serve = load_package().serve
    d, cfg = folder
    a, b = (serve.Model(d, max_context=64, max_sequences=n) for _ in range(2))
    slots = [(a.open_slot(), b.open_slot())[0] for _ in range(n)]
    for i in range(6):
        e = [(s, [(31 * i + 7 * s) % cfg.vocab], [0]) for s in slots]
        want, chosen = a.step(e, choice=True)
        got, none = b.step(e, choice=i == 3)
        assert got == want and (none is None or none == chosen)
    a.close(), b.close()

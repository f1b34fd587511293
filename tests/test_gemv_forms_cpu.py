"""The forms of the decode kernel: the default call, the allocation-free one and the one with the exchange fused in give the same bits.  All
forms do where whole row blocks are dealt out; a split k range is cut between a form's stages, so there the three have to take one form."""
import ctypes
import os
import subprocess

import pytest

from __graft_entry__ import ROOT

LOW, LONG, TALL = range(3)
DEFAULT, STATIC = 64 << 20, 256 * 2 * 32 * 8 * 4    # bytes for partial tiles


@pytest.fixture(scope="module")
def forms(tmp_path_factory):
    top = tmp_path_factory.mktemp("forms")
    (top / "forms.cpp").write_text('''
#include "%s/cccc-lite_b200/csrc/gemv_form.cuh"
extern "C" int form(int fp4, unsigned M, unsigned K, unsigned long long low, unsigned long long tall, int sms, int world, size_t bytes)
{
    return (int)b200::gemv_form(fp4 != 0, M, K, low, tall, sms, world, bytes);
}
extern "C" int whole(unsigned rows, int fp4, unsigned long long blocks, unsigned K, int sms) { return b200::gemv_whole_blocks(rows, fp4 != 0, blocks, K, sms); }
''' % ROOT)
    so = str(top / "forms.so")
    subprocess.check_call(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", "-o", so, str(top / "forms.cpp")])
    L = ctypes.CDLL(so)
    L.form.argtypes = [ctypes.c_int, ctypes.c_uint, ctypes.c_uint, ctypes.c_ulonglong, ctypes.c_ulonglong, ctypes.c_int, ctypes.c_int, ctypes.c_size_t]
    L.whole.argtypes = [ctypes.c_uint, ctypes.c_int, ctypes.c_ulonglong, ctypes.c_uint, ctypes.c_int]
    return L


def cut(L, fp4, M, K, Ns, sms, world, nbytes):
    """What the sums of a launch depend on: nothing but whole blocks, or the rows and the stage that a split is made of."""
    low, tall = sum((N + 31) // 32 for N in Ns), sum((N + 63) // 64 for N in Ns)
    f = L.form(fp4, M, K, low, tall, sms, world, nbytes)
    assert not (fp4 and f != LOW)
    rows, blocks = (64, tall) if f == TALL else (32, low)
    if L.whole(rows, fp4, blocks, K, sms):
        return f, "whole"
    stage = {LOW: (2048 if M <= 2 else 1024) * (2 if fp4 else 1), LONG: 2048, TALL: 1024}[f]
    return f, (rows, stage)


@pytest.mark.parametrize("sms", [132, 148])
@pytest.mark.parametrize("fp4", [0, 1])
def test_the_cut_of_k_is_the_same_in_all_calls(forms, fp4, sms):
    seen = set()
    for M in (1, 2, 3, 8):
        for K in [256 * i for i in (1, 4, 8, 16, 24, 32, 40, 50, 54, 56, 64, 68, 96, 100, 112)]:
            for N in (8, 64, 1000, 1024, 2048, 4096, 4736, 5120, 6144, 8192, 9472, 9473, 24576, 28672, 151936):
                for Ns in ((N,), (N, 1024, 1024)):
                    form, want = cut(forms, fp4, M, K, Ns, sms, 0, DEFAULT)
                    seen.add((form, want))
                    assert cut(forms, fp4, M, K, Ns, sms, 0, STATIC)[1] == want, (M, K, Ns)
                    assert cut(forms, fp4, M, K, Ns, sms, 2, DEFAULT)[1] == want, (M, K, Ns)
    # the forms that there are, and a launch of each schedule
    assert {f for f, _ in seen} == ({LOW} if fp4 else {LOW, LONG, TALL}) and len({w for _, w in seen}) > 1


def test_calls_with_the_exchange_take_the_form_of_32_rows(forms):
    for M in range(1, 9):
        for N, K in ((4096, 4096), (6144, 4096), (24576, 4096), (4096, 12288), (5120, 12800)):
            assert forms.form(0, M, K, (N + 31) // 32, (N + 63) // 64, 148, 2, DEFAULT) == LOW

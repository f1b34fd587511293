"""Decode attention where its tiles, splits and clusters end: positions at the edges of 16-row tiles and of splits, one split up to
sixteen, splits without rows, a split in more rounds than the GPU has slots for, query heads per kv head 1 to 8, both head sizes;
against the oracle's composition of the reference's ops (tests/test_gpu_decode_ops.py)."""
import numpy as np
import pytest

from tests.test_gpu_decode_ops import attention_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("hd", [64, 128])
@pytest.mark.parametrize("G", [1, 2, 4, 8])
@pytest.mark.parametrize("T_max", [15, 64, 129, 1024])
def test_edges_of_tiles_and_splits(T_max, G, hd):
    pos = [p for p in (0, 1, 15, 16, 17, 31, 63, 64, 127, 128, 129, 255, 511, 1023) if p <= T_max]    # T_max itself: no row left for it
    attention_case(len(pos), 2 * G, 2, hd, T_max, pos, G != 2, T_max + G + hd, strided=G == 4)


# sixteen splits of one sequence: the last ones empty, the owner first or last
@pytest.mark.parametrize("pos", [0, 5, 240, 255, 256, 1000, 4000, 4095])
def test_a_cluster_of_sixteen(pos):
    attention_case(1, 8, 2, 128, 4096, [pos], True, pos, strided=True)


# Few scores where sequences are short: a score that lies within its sum's FP32 error of a BF16 rounding boundary goes either way
# (about one in 3000), which moves its head's outputs by up to 2^-6 p (1 - p) |v - out| for 2 <= |score| < 4 - with p near a half as
# much as 1.6 times the bar; among 4480 heads of about thirty rows one such is to be expected, among 280 not.
@pytest.mark.parametrize("B,Hkv,T_max", [(6, 8, 700), (64, 8, 300), (40, 4, 530), (3, 1, 2048), (70, 1, 64)])
def test_counts_of_sequences(B, Hkv, T_max):
    rng = np.random.default_rng(B)
    attention_case(B, 4 * Hkv, Hkv, 128, T_max, [int(p) for p in rng.integers(0, T_max, B)], False, B, strided=True)

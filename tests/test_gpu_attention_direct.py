"""attention_direct (kernel 4) where its splits and clusters end: one sequence over sixteen splits, the last ones empty and the new row in
the first or last of them, several tokens per entry (two row tiles), more clusters than the GPU has slots for; against the numpy
statement of tests/test_gpu_decoder_ops.py."""
import numpy as np
import pytest

from tests.test_gpu_decoder_ops import BF16, Attn, D, close  # noqa: F401 (D is a fixture)

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("pos", [0, 15, 16, 255, 256, 1000, 4080, 4095])
@pytest.mark.parametrize("n", [1, 3])
def test_a_cluster_of_sixteen(D, pos, n):  # noqa: F811
    pos = min(pos, 4096 - n)
    a = Attn(D, BF16, 8, 2, 128, 128, [(0, pos, n)], T_max=4096, slots=1, scale=0.1, seed=pos + n)
    close(a.run(4).reshape(n, -1), a.reference().reshape(n, -1), BF16, pos, 1.5)


@pytest.mark.parametrize("H,Hkv,dim,vdim,S", [(8, 8, 128, 128, 60), (20, 2, 64, 64, 3), (3, 1, 72, 136 - 8, 5), (64, 16, 32, 16, 24)])
def test_counts_of_units(D, H, Hkv, dim, vdim, S):  # noqa: F811
    rng = np.random.default_rng(H)
    a = Attn(D, BF16, H, Hkv, dim, vdim, [(s, int(p), 1) for s, p in enumerate(rng.integers(0, 500, S))], T_max=512, slots=S, scale=0.2, v_mix=2, seed=S)
    close(a.run(4).reshape(S, -1), a.reference().reshape(S, -1), BF16, (H, S), 1.5)

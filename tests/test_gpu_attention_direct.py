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


@pytest.mark.parametrize("pos", [5, 600])    # one split, several
@pytest.mark.parametrize("sink", [True, False])
def test_scores_of_minus_infinity(D, pos, sink):  # noqa: F811
    """Every key of the first sequence scores minus infinity: its weights are zero beside a sink and undefined without one; the second
    sequence is as ever."""
    import torch

    H, Hkv, d, T = 4, 2, 64, 640
    g = torch.Generator(device="cuda").manual_seed(pos)
    bf = lambda *s: torch.randn(*s, device="cuda", generator=g, dtype=torch.bfloat16)
    x, K, V, out = bf(2, H * d), bf(2, Hkv, T, d), bf(2, Hkv, T, d), torch.full((2, H * d), 7.0, device="cuda", dtype=torch.bfloat16)
    x[0], K[0] = 1.0, -float("inf")
    keep = [torch.tensor(m, dtype=torch.int32, device="cuda") for m in ([0, 1], [pos, pos], [0, 1], [1, 1], [0, 1])]
    s, work = torch.tensor([0.0, 1.0, -2.0, 3.0], device="cuda"), torch.zeros(D.attention_work_bytes(d), dtype=torch.uint8, device="cuda")
    a = D.fill(D.Attention, qkvg=x, out=out, k_cache=K, v_cache=V, work=work, sink=s if sink else None, ld=H * d, ldo=H * d, H=H, Hkv=Hkv, dim=d, vdim=d, k_ld=d, v_ld=d,
               T_max=T, slots=2, no_append=1, scale=0.125)
    b = D.fill(D.Batch, slot=keep[0], pos=keep[1], start=keep[2], n=keep[3], token_entry=keep[4], entries=2, tokens=2, max_n=1, max_len=pos + 1)
    assert D.attention(BF16, a, b, kernel=4) == 0 and D.check() == 0
    assert bool((out[0] == 0).all()) if sink else bool(out[0].isnan().all())
    for h in range(H):
        z = x[1].view(H, d)[h].double() @ K[1, h // 2, :pos + 1].double().T * 0.125
        w = torch.softmax(torch.cat([z, s[h:h + 1].double()]), 0)[:-1] if sink else torch.softmax(z, 0)
        want = w @ V[1, h // 2, :pos + 1].double()
        assert float((out[1].view(H, d)[h].double() - want).abs().max()) < 2.0 ** -7 * float(want.abs().max())


# units that clusters of more than eight have room for and that they have not; a last cluster beyond one round
@pytest.mark.parametrize("H,Hkv,d,S,n", [(16, 8, 128, 2, 1), (4, 4, 64, 5, 1), (4, 2, 128, 3, 4), (8, 8, 128, 4, 4), (16, 4, 64, 33, 4)])
def test_long_contexts(D, H, Hkv, d, S, n):  # noqa: F811
    T = 9000 if S < 10 else 1500
    rng = np.random.default_rng(S)
    a = Attn(D, BF16, H, Hkv, d, d, [(s, T - n if s == 0 else int(rng.integers(0, T - n)), n) for s in range(S)], T_max=T, slots=S, scale=0.1, seed=S)
    close(a.run(4).reshape(S * n, -1), a.reference().reshape(S * n, -1), BF16, (H, Hkv, S, n), 1.5)

"""Decode attention where its tiles, splits and clusters end: positions at the edges of 16-row tiles and of splits, one split up to
sixteen, splits without rows, a split in more rounds than the GPU has slots for, query heads per kv head 1 to 8, both head sizes;
against the oracle's composition of the reference's ops (tests/test_gpu_decode_ops.py)."""
import numpy as np
import pytest

from tests._util import assert_close_rows, capi
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


def long_case(B, Hkv, G, hd, T_max, pos, seed):
    """Caches made on the device, queries and keys as they are (no norm, a rotation by nothing); against the reference's roundings of
    scores and weights in float64."""
    import torch

    c, g = capi(), torch.Generator(device="cuda").manual_seed(seed)
    bf = lambda *s: torch.randn(*s, device="cuda", generator=g, dtype=torch.bfloat16)
    H = G * Hkv
    q, k, v, K, V = bf(B, H, hd), bf(B, Hkv, hd), bf(B, Hkv, hd), bf(B, Hkv, T_max, hd), bf(B, Hkv, T_max, hd)
    cos, sin = torch.ones(T_max, hd // 2, device="cuda", dtype=torch.bfloat16), torch.zeros(T_max, hd // 2, device="cuda", dtype=torch.bfloat16)
    out, p = torch.zeros(B, H * hd, device="cuda", dtype=torch.bfloat16), torch.tensor(pos, dtype=torch.int32, device="cuda")
    desc = c.make_attn_decode(q=q, k=k, v=v, k_cache=K, v_cache=V, pos=p, out=out, cos_tab=cos, sin_tab=sin, B=B, H=H, Hkv=Hkv, head_dim=hd, T_max=T_max)
    rc = c.attn_decode_bf16(desc)
    assert c.check_error("long") == 0
    if rc != 0:
        return rc
    want = torch.empty(B, H, hd, dtype=torch.float64, device="cuda")
    for b, at in enumerate(pos):
        assert torch.equal(K[b, :, at], k[b]) and torch.equal(V[b, :, at], v[b])
        for h in range(Hkv):
            s = ((q[b, h * G:(h + 1) * G].double() @ K[b, h, :at + 1].double().T).float() * (1.0 / np.float32(np.sqrt(np.float32(hd))))).to(torch.bfloat16)
            w = torch.softmax(s.double(), -1).to(torch.bfloat16)
            want[b, h * G:(h + 1) * G] = w.double() @ V[b, h, :at + 1].double()
    assert_close_rows(out.float().cpu().numpy().reshape(B * H, hd), want.cpu().numpy().reshape(B * H, hd), (B, Hkv, G, hd, T_max))
    return 0


# caches so long that the scores of a split take the shared memory of two or three CTAs
@pytest.mark.parametrize("B,Hkv,G,hd,T_max", [(16, 8, 8, 128, 32768), (9, 8, 8, 64, 40000), (16, 4, 4, 128, 65536), (1, 1, 8, 128, 65536), (1, 2, 1, 128, 32768)])
def test_long_caches(B, Hkv, G, hd, T_max):
    rng = np.random.default_rng(B)
    pos = [T_max - 1] + [int(x) for x in rng.integers(0, T_max, B - 1)]
    assert long_case(B, Hkv, G, hd, T_max, pos, G) == 0
    assert long_case(1, 1, G, hd, 256, [200], G) == 0    # a small cache after a large one


@pytest.mark.parametrize("hd", [64, 128])
@pytest.mark.parametrize("G", [1, 2, 4, 8])
def test_the_longest_cache_that_is_served(G, hd):
    import torch

    floats = torch.cuda.get_device_properties(0).shared_memory_per_block_optin // 4 - ((3 * G + 5) * hd + 260 * G + 256 + max(2048 * G, 8192))
    most = floats // G // 32 * 32 * 16
    assert long_case(1, 1, G, hd, most, [most - 1], G) == 0
    assert long_case(3, 2, G, hd, most, [most // 2, 0, most - 1], G) == 0
    assert long_case(1, 1, G, hd, most + 1, [0], G) == -1


def test_many_short_sequences():
    """4480 heads of about thirty rows.  A score within its sum's error of a BF16 rounding boundary may go either way; a head beyond the
    bar has to have such scores, and to be within it for one way of rounding them."""
    import itertools

    import torch

    c, g, B, Hkv, G, hd, T_max = capi(), torch.Generator(device="cuda").manual_seed(7), 70, 16, 4, 128, 64
    bf = lambda *s: torch.randn(*s, device="cuda", generator=g, dtype=torch.bfloat16)
    q, k, v, K, V = bf(B, Hkv, G, hd), bf(B, Hkv, hd), bf(B, Hkv, hd), bf(B, Hkv, T_max, hd), bf(B, Hkv, T_max, hd)
    cos, sin = torch.ones(T_max, hd // 2, device="cuda", dtype=torch.bfloat16), torch.zeros(T_max, hd // 2, device="cuda", dtype=torch.bfloat16)
    pos = torch.randint(0, T_max, (B,), device="cuda", generator=g, dtype=torch.int32)
    out = torch.zeros(B, Hkv, G, hd, device="cuda", dtype=torch.bfloat16)
    d = c.make_attn_decode(q=q, k=k, v=v, k_cache=K, v_cache=V, pos=pos, out=out, cos_tab=cos, sin_tab=sin, B=B, H=G * Hkv, Hkv=Hkv, head_dim=hd, T_max=T_max)
    assert c.attn_decode_bf16(d) == 0 and c.check_error("short") == 0
    q, K, V, out, pos, scale = q.cpu().double(), K.cpu().double(), V.cpu().double(), out.cpu().double(), pos.cpu().tolist(), float(np.float32(1 / np.sqrt(np.float32(hd))))
    to_bf = lambda x: x.float().to(torch.bfloat16).double()

    def error(scores, b, h, j, n):
        want = to_bf(torch.softmax(scores, -1)) @ V[b, h, :n]
        return float(((out[b, h, j] - want).abs() / want.abs().clamp_min(float(want.square().mean().sqrt()))).max())

    beyond = 0
    for b, h, j in itertools.product(range(B), range(Hkv), range(G)):
        n = pos[b] + 1
        s = K[b, h, :n] @ q[b, h, j] * scale
        if error(to_bf(s), b, h, j, n) <= 1e-2:
            continue
        # eight steps of sixteen products, each cut or rounded at 2^-23 of what has been added up, within a step as much again
        e = K[b, h, :n].abs() @ q[b, h, j].abs() * scale * 2.0 ** -19
        low, high = to_bf(s - e), to_bf(s + e)
        near = (low != high).nonzero().flatten().tolist()
        assert 1 <= len(near) <= 8, (b, h, j, near)
        ways = []
        for pick in itertools.product((0, 1), repeat=len(near)):
            z = to_bf(s).clone()
            for i, p in zip(near, pick):
                z[i] = high[i] if p else low[i]
            ways.append(error(z, b, h, j, n))
        assert min(ways) <= 1e-2, (b, h, j, min(ways))
        beyond += 1
    assert beyond <= 8    # about one is to be expected

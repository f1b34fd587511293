"""The wide streaming kernel (more than 128 tokens: CTA pairs, up to 384 tokens per tile, k slices as a cluster) against the CPU
oracle at the GEMM bar, and bit for bit on one-hot activations, where the output IS the dequantised weight.  Flags bits 8-10 = 7
take it wherever it accepts the shape; without them it is taken by its estimate."""
import numpy as np
import pytest

from oracle import oracle as O
from tests._util import assert_close, capi, from_dev_u16, to_dev
from tests.test_gpu_onehot import expected_bits, fp4_matrix, fp8_matrix, run_onehot

pytestmark = pytest.mark.gpu

WTS = [O.FP8_E5M2, O.FP8_E4M3, O.FP4_E2M1]
WIDE = 7 << 8


def run(wt, W, blk, inv, X, N, M, K, Y0=None, flags=WIDE, **kw):
    import torch

    c = capi()
    dW, dX, dB = to_dev(W), to_dev(X), to_dev(blk) if blk is not None else None
    size = (M - 1) * kw.get("ldy_m", N) + (N - 1) * kw.get("ldy_n", 1) + 1
    dY = to_dev(Y0) if Y0 is not None else torch.zeros(size, dtype=torch.float32 if flags & 4 else torch.int16, device="cuda")
    before = c.launch_count()
    assert c.gemm_wq_bf16(wt, dW, dB, inv, dX, dY, N, M, K, flags=flags, **kw) == 0
    assert c.check_error("wide") == 0 and c.launch_count() == before + 1
    return dY.cpu().numpy() if flags & 4 else from_dev_u16(dY)


# tokens at the edges of the tile widths (one UMMA up to 256, two up to 384, several tiles), a last tile of one token and one whose
# second UMMA is empty; features that end inside either CTA of a pair; one k slice of 256 up to slices of unequal length
@pytest.mark.parametrize("wt", WTS)
@pytest.mark.parametrize("N,K,M", [(128, 256, 129), (256, 512, 144), (300, 1280, 256), (129, 768, 257), (1000, 2304, 272), (384, 512, 383), (512, 4096, 384), (64, 256, 385),
                                   (200, 1024, 513), (257, 512, 769), (5, 256, 1153)])
def test_matches_the_oracle(wt, N, K, M):
    W, blk, inv, X = O.make_inputs(wt, N, K, M, seed=N + M, scaled=True)
    _, y32 = O.linear_wq_bf16(wt, W, blk, inv, X, N, M, K)
    for flags in (WIDE, WIDE | 1, 1):
        assert_close(O.bf16_bits_to_f32(run(wt, W, blk, inv, X, N, M, K, flags=flags)).reshape(M, N), y32, (wt, N, K, M, flags))


@pytest.mark.parametrize("wt", WTS)
def test_alpha_beta_strides_and_output_modes(wt):
    N, K, M = 203, 512, 150
    ldw, ldx = K + 256, K + 8
    rng = np.random.default_rng(3)
    Wd, blkd, inv, Xd = O.make_inputs(wt, N, ldw, M, seed=13, scaled=False)
    X = np.zeros((M, ldx), np.uint16)
    X[:, :K] = Xd.reshape(M, ldw)[:, :K]
    for ldy_m, ldy_n, size in ((1, M + 3, N * (M + 3)), (N + 1, 1, M * (N + 1))):
        Y0 = O.f32_to_bf16_bits(rng.standard_normal(size).astype(np.float32))
        kw = dict(ldw=ldw, ldx=ldx, alpha=0.25, beta=1.5, ldy_m=ldy_m, ldy_n=ldy_n)
        Yo, _ = O.linear_wq_bf16(wt, Wd, blkd, inv, X, N, M, K, Y=Y0, **kw)
        Y = run(wt, Wd, blkd, inv, X, N, M, K, Y0=Y0.copy(), **kw)
        assert_close(O.bf16_bits_to_f32(Y[:Yo.size]), O.bf16_bits_to_f32(Yo), (wt, ldy_m))
    # float32 output: the unrounded sums (K = 512 products of BF16 numbers, summed in float32 in another order)
    _, y32 = O.linear_wq_bf16(wt, Wd, blkd, inv, X, N, M, K, ldw=ldw, ldx=ldx)
    got = run(wt, Wd, blkd, inv, X, N, M, K, flags=WIDE | 4, ldw=ldw, ldx=ldx).reshape(M, N)
    assert np.abs(got - y32).max() <= 1e-5 * np.sqrt(np.mean(y32.astype(np.float64) ** 2)) * np.sqrt(K)


@pytest.mark.parametrize("wt", WTS)
@pytest.mark.parametrize("N,K,M", [(203, 512, 150), (4, 256, 129), (260, 4096, 385)])
@pytest.mark.parametrize("mode", [0, 8])
def test_rows_that_lie_on_8_bytes_have_the_same_bits(wt, N, K, M, mode):
    """Four elements of Y at once where its rows allow it, the added Y among them, else one by one: the same bits, and nothing beside the rows."""
    W, blk, inv, X = O.make_inputs(wt, N, K, M, seed=N, scaled=True)
    Y0 = O.f32_to_bf16_bits(np.random.default_rng(M).standard_normal((M, N)).astype(np.float32))
    got = []
    for ld in ((N + 3) // 4 * 4 + 4, (N + 3) // 4 * 4 + 5):
        Y = np.full((M, ld), 0x1234, np.uint16)
        Y[:, :N] = Y0
        got.append(run(wt, W, blk, inv, X, N, M, K, Y0=Y, flags=WIDE | mode, ldy_m=ld, alpha=0.75, beta=1.5).reshape(M, ld))
        assert (got[-1][:, N:] == 0x1234).all()
    assert np.array_equal(got[0][:, :N], got[1][:, :N]) and not np.array_equal(got[0][:, :N], Y0)


@pytest.mark.parametrize("wt", WTS)
@pytest.mark.parametrize("M", [130, 512])
def test_weights_are_dequantised_bit_exactly(wt, M):
    N, K = 508, 512
    W, S = fp4_matrix(N, K) if wt == O.FP4_E2M1 else (fp8_matrix(wt, N, K), None)
    for inv in ((1.0,) if wt == O.FP4_E2M1 else (1.0, 0.25, 0.37)):
        positions = [(np.arange(M) * 37 + 11 + s) % K for s in range(0, K, M)]
        run_onehot(wt, W, S, inv, expected_bits(wt, W, S, inv, N, K), N, K, M, positions, flags=WIDE)


@pytest.mark.parametrize("wt", WTS)
def test_a_group_is_one_launch(wt):
    import torch

    c, K, M = capi(), 1024, 200
    Ns = (300, 128, 64)
    items, want = [], []
    X = O.make_inputs(wt, 8, K, M, seed=1)[3]
    for i, N in enumerate(Ns):
        W, blk, inv, _ = O.make_inputs(wt, N, K, M, seed=20 + i, scaled=True)
        want.append(O.linear_wq_bf16(wt, W, blk, inv, X, N, M, K)[1])
        items.append(dict(W=to_dev(W), S=to_dev(blk) if blk is not None else None, inv=inv, N=N, Y=torch.zeros(M * N, dtype=torch.int16, device="cuda")))
    before = c.launch_count()
    assert c.gemm_wq_bf16_group(wt, c.make_group(items, K), to_dev(X), M, K, flags=1) == 0
    assert c.check_error("wide group") == 0 and c.launch_count() == before + 1
    for it, y, N in zip(items, want, Ns):
        assert_close(O.bf16_bits_to_f32(from_dev_u16(it["Y"])).reshape(M, N), y, (wt, N))

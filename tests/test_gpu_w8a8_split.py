"""W8A8 with k slices (24 to 64 tokens by default, more where k is long; flags bits 8-10 = 4 take it at any count) against the
CPU oracle, and the rule that the result does not depend on how many CTAs share the k range."""
import numpy as np
import pytest

from oracle import oracle as O
from tests._util import assert_close, capi, from_dev_u16, to_dev
from tests.test_gpu_w8a8 import run

pytestmark = pytest.mark.gpu

SPLIT = 4 << 8


# tokens at the edges of the 64- and 128-token tiles; features that end inside a tile; k of one block (three slices empty), of
# unequal slices, and long enough that every stage is used again
@pytest.mark.parametrize("flags", [SPLIT, SPLIT | 1])
@pytest.mark.parametrize("act_scale", [0.0, 0.0123])
@pytest.mark.parametrize("N,K,M", [(128, 128, 33), (5, 256, 48), (300, 640, 64), (129, 896, 65), (1000, 4096, 100), (256, 12288, 128), (2500, 1024, 129), (384, 256, 300),
                                   (6144, 2048, 64), (20000, 512, 40), (4096, 1152, 97)])
def test_matches_the_oracle(N, K, M, act_scale, flags):
    W, _, w_inv, X = O.make_inputs(O.FP8_E4M3, N, K, M, seed=N + M, scaled=True)
    y32, _, _ = O.linear_w8a8(W, w_inv, X, N, M, K, act_scale=act_scale)
    assert_close(O.bf16_bits_to_f32(run(W, w_inv, X, act_scale, N, M, K, flags=flags)).reshape(M, N), y32, (N, K, M, act_scale))


# the line at 24 tokens, and at 16384 activations (below, the quantiser finds the maximum itself and the streaming kernel runs)
@pytest.mark.parametrize("act_scale", [0.0, 0.0123])
@pytest.mark.parametrize("N,K,M", [(1000, 1024, 23), (1000, 1024, 24), (640, 4096, 31), (300, 640, 25), (300, 768, 25), (129, 512, 32), (129, 640, 32)])
def test_the_line_below_32_tokens(N, K, M, act_scale):
    W, _, w_inv, X = O.make_inputs(O.FP8_E4M3, N, K, M, seed=N + M, scaled=True)
    y32, _, _ = O.linear_w8a8(W, w_inv, X, N, M, K, act_scale=act_scale)
    assert_close(O.bf16_bits_to_f32(run(W, w_inv, X, act_scale, N, M, K)).reshape(M, N), y32, (N, K, M, act_scale))


@pytest.mark.parametrize("M", [34, 70])
def test_float32_strides_and_accumulate(M):
    """float32 output: sums of 1024 products in another order than float64's, 2^-24 per addition at most; transposed output with
    alpha and beta; rows of Y that are not 8-byte aligned."""
    N, K = 203, 1024
    W, _, w_inv, X = O.make_inputs(O.FP8_E4M3, N, K, M, seed=5, scaled=True)
    y32, _, _ = O.linear_w8a8(W, w_inv, X, N, M, K)
    Yf = run(W, w_inv, X, 0.0, N, M, K, flags=4 | SPLIT).reshape(M, N)
    rms = np.sqrt(np.mean(np.square(y32), axis=1, keepdims=True))
    assert np.max(np.abs(Yf - y32) / np.maximum(np.abs(y32), rms)) < 1e-5
    rng = np.random.default_rng(4)
    ya, _, _ = O.linear_w8a8(W, w_inv, X, N, M, K, alpha=0.25)
    Y0 = O.f32_to_bf16_bits(rng.standard_normal((N, M + 3)).astype(np.float32))
    got = O.bf16_bits_to_f32(run(W, w_inv, X, 0.0, N, M, K, Y0=Y0.copy(), alpha=0.25, beta=1.5, ldy_m=1, ldy_n=M + 3, flags=SPLIT)[:N * (M + 3)]).reshape(N, M + 3)
    assert_close(got[:, :M].T.copy(), (ya.T + 1.5 * O.bf16_bits_to_f32(Y0)[:, :M]).T.copy(), "alpha beta strides")
    assert np.array_equal(got[:, M:], O.bf16_bits_to_f32(Y0)[:, M:])
    for ldy in (N + 1, N + 2):
        assert_close(O.bf16_bits_to_f32(np.resize(run(W, w_inv, X, 0.0, N, M, K, ldy_m=ldy, flags=SPLIT), M * ldy)).reshape(M, ldy)[:, :N], y32, ldy)


@pytest.mark.parametrize("K,M", [(1024, 64), (8192, 100)])
def test_the_bits_do_not_depend_on_the_grid(K, M):
    """The same 128 features alone (four CTAs per tile), with others in a group, and as part of a matrix whose tiles fill the GPU
    without cutting k."""
    import torch

    c, most = capi(), 40960 if K < 4096 else 20480
    W, _, w_inv, X = O.make_inputs(O.FP8_E4M3, most, K, M, seed=1, scaled=True)
    W = W.reshape(most, K)
    dX = to_dev(X)

    def linear(n):
        y = torch.zeros(M, n, dtype=torch.int16, device="cuda")
        assert c.gemm_w8a8_bf16(to_dev(W[:n].copy()), w_inv, dX, 0.0, y, n, M, K, flags=1) == 0 and c.check_error("grid") == 0
        return y[:, :128]

    alone = linear(128)
    for n in (6144, most):
        assert torch.equal(linear(n), alone)
    items = [dict(W=to_dev(W[:n].copy()), S=None, inv=w_inv, N=n, Y=torch.zeros(M, n, dtype=torch.int16, device="cuda")) for n in (128, 9000, 4096)]
    assert c.gemm_w8a8_bf16_group(c.make_group(items, K), dX, 0.0, M, K) == 0 and c.check_error("group") == 0
    assert torch.equal(items[0]["Y"], alone)


# k slices: all matrices within the line (129 to 8448 features with K from 4096 on, up to 128 tokens); CTA pairs in all their forms where k is shorter, or the tokens are more
@pytest.mark.parametrize("M,K,features", [(65, 4096, (129, 1000, 4096, 6144, 8448)), (100, 4096, (256, 1024, 4096, 8448)), (128, 5120, (512, 5120, 8448)), (100, 2048, (128, 6144, 20480)),
                                          (129, 4096, (128, 4096, 24576))])
def test_the_bits_do_not_depend_on_the_matrix(M, K, features):
    import torch

    c = capi()
    (W,), X = on_device([max(features)], K, M, 3)
    first = min(features)

    def linear(n):
        y = torch.zeros(M, n, dtype=torch.float32, device="cuda")
        assert c.gemm_w8a8_bf16(W, 0.01, X, 0.0, y, n, M, K, flags=5) == 0 and c.check_error("matrix") == 0
        return y

    alone = linear(first)
    for n in features:
        assert torch.equal(linear(n)[:, :first], alone), n
    Ns = (features[-1], first, features[1])
    items = [dict(W=W[:n], S=None, inv=0.01, N=n, Y=torch.zeros(M, n, dtype=torch.float32, device="cuda")) for n in Ns]
    assert c.gemm_w8a8_bf16_group(c.make_group(items, K), X, 0.0, M, K, flags=5) == 0 and c.check_error("group") == 0
    for it in items:
        assert torch.equal(it["Y"][:, :first], alone)


# q, k and v of a model, or of a rank's share of one: one quantisation (two kernels with the scale found) and one linear
@pytest.mark.parametrize("Ns,K", [((4096, 1024, 1024), 4096), ((4096, 512, 512), 4096), ((2048, 256, 256), 4096), ((5120, 1024, 1024), 5120), ((8192, 256, 256), 5120)])
@pytest.mark.parametrize("M", [65, 128])
def test_q_k_and_v_are_one_launch(Ns, K, M):
    import torch

    c = capi()
    Ws, X = on_device(Ns, K, M, 4)
    items = [dict(W=W, S=None, inv=0.01, N=N, Y=torch.zeros(M, N, dtype=torch.bfloat16, device="cuda")) for W, N in zip(Ws, Ns)]
    before = c.launch_count()
    assert c.gemm_w8a8_bf16_group(c.make_group(items, K), X, 0.0, M, K) == 0 and c.check_error("group") == 0
    assert c.launch_count() - before == 3


@pytest.mark.parametrize("M", [20, 64])
def test_the_largest_magnitude_is_found_wherever_it_lies(M):
    """One scale for the tensor: every block of the search has to count."""
    N, K = 128, 4096
    W, _, w_inv, X0 = O.make_inputs(O.FP8_E4M3, N, K, M, seed=M, scaled=True)
    for at in (0, 5, M * K // 2 + 8191, M * K - 1):
        X = X0.reshape(-1).copy()
        X[at] = O.f32_to_bf16_bits(np.array([300.0], np.float32))[0]
        y32, _, _ = O.linear_w8a8(W, w_inv, X.reshape(X0.shape), N, M, K)
        assert_close(O.bf16_bits_to_f32(run(W, w_inv, X.reshape(X0.shape), 0.0, N, M, K)).reshape(M, N), y32, (M, at))


@pytest.mark.parametrize("y_type", [3, 4])
def test_e4m3_activations_where_they_lie(y_type):
    """cuda_gemm_fp8_fp8 at 70 tokens: no quantiser before the linear; BF16 and E4M3 output."""
    import torch

    c, N, K, M = capi(), 600, 1024, 70
    W, _, w_inv, _ = O.make_inputs(O.FP8_E4M3, N, K, M, seed=2, scaled=True)
    Xq = O.float_to_fp8(np.random.default_rng(0).standard_normal(M * K).astype(np.float32), O.FP8_E4M3, 32.0)
    y = ((O.fp8_to_float(Xq, O.FP8_E4M3, 1.0).reshape(M, K).astype(np.float64) @ O.fp8_to_float(W, O.FP8_E4M3, 1.0).reshape(N, K).astype(np.float64).T)
         * (float(np.float32(w_inv)) / 32.0)).astype(np.float32)
    out = torch.zeros(M * N, dtype=torch.int16 if y_type == 3 else torch.uint8, device="cuda")
    dW, dX = to_dev(W), to_dev(Xq)
    assert c.lib().cuda_gemm_fp8_fp8(dW.data_ptr(), w_inv, dX.data_ptr(), 1 / 32, out.data_ptr(), y_type, N, M, K, K, K, N, 1, 1.0, 0.0, None, SPLIT) == 0
    assert c.check_error("fp8 x fp8") == 0
    if y_type == 3:
        assert_close(O.bf16_bits_to_f32(from_dev_u16(out)).reshape(M, N), y, "bf16")
    else:    # a code is a 6-12 % step: sums that differ in their last bits may land on either side of one
        want = O.float_to_fp8(O.bf16_bits_to_f32(O.f32_to_bf16_bits(y)).reshape(-1), O.FP8_E4M3, 1.0)
        diff = np.abs(out.cpu().numpy().astype(np.int16) - want.astype(np.int16))
        assert diff.max() <= 1 and np.mean(diff != 0) < 2e-3


def on_device(Ns, K, M, seed=0):
    import torch

    g = torch.Generator(device="cuda").manual_seed(seed)
    Ws = [torch.randint(0, 256, (N, K), dtype=torch.uint8, device="cuda", generator=g) for N in Ns]
    for W in Ws:
        W[(W & 0x7F) == 0x7F] = 0    # not a number in E4M3
    return Ws, torch.randn(M, K, device="cuda", generator=g).to(torch.bfloat16)


# the lines between the k slices and the CTA pairs, in tiles of 128 features x 128 tokens: a wave and a quarter up to 128 tokens, two slices of
# every tile at once above; and where k is too short or the tokens too many
@pytest.mark.parametrize("M,K,beyond", [(65, 8192, 0), (128, 8192, 0), (128, 8192, 1), (129, 8192, 0), (129, 8192, 1), (256, 12288, 0), (256, 12288, 1), (257, 8192, 1), (65, 8064, 1)])
def test_the_line_above_64_tokens(M, K, beyond):
    """Sums of k slices and of the whole k range differ in their last bits: the float32 outputs say which kernel ran."""
    import torch

    c, sms = capi(), torch.cuda.get_device_properties(0).multi_processor_count
    tiles = 5 * sms // 4 if M <= 128 else 9 * sms // 20 // 2    # of features
    if M > 256 or K < 8192:
        tiles = 0
    N = 128 * tiles + (1 if beyond else 0)
    (W,), X = on_device([N], K, M)
    out = {}
    for form in (0, 1, 4):
        out[form] = torch.zeros(M, N, dtype=torch.float32, device="cuda")
        assert c.gemm_w8a8_bf16(W, 0.01, X, 0.0, out[form], N, M, K, flags=4 | form << 8) == 0 and c.check_error("line") == 0
    assert not torch.equal(out[1], out[4])
    assert torch.equal(out[0], out[1 if beyond else 4])


@pytest.mark.parametrize("M,K,tiles,slices", [(65, 4096, 2, True), (65, 4096, 1, False), (128, 8064, 66, True), (128, 4096, 67, False), (129, 4096, 32, False), (100, 3968, 32, False)])
def test_the_line_of_shorter_k(M, K, tiles, slices):
    """As above, for k below 8192: two tiles of features to nine twentieths of the SMs (66 of 148), up to 128 tokens."""
    import torch

    c, sms = capi(), torch.cuda.get_device_properties(0).multi_processor_count
    N = 128 * (tiles if tiles < 60 else 9 * sms // 20 + tiles - 66) - (5 if slices else 0)
    (W,), X = on_device([N], K, M, 2)
    out = {}
    for form in (0, 1, 4):
        out[form] = torch.zeros(M, N, dtype=torch.float32, device="cuda")
        assert c.gemm_w8a8_bf16(W, 0.01, X, 0.0, out[form], N, M, K, flags=5 | form << 8) == 0 and c.check_error("line") == 0
    assert not torch.equal(out[1], out[4])
    assert torch.equal(out[0], out[4 if slices else 1])


@pytest.mark.parametrize("order,launches", [((4352, 256, 384), 4), ((256, 4352, 384), 5), ((256, 384, 4096), 3), ((4352, 4480, 9000), 3)])
def test_members_of_a_group_take_the_kernels_they_would_take_alone(order, launches):
    import torch

    c, M, K = capi(), 129, 8192
    Ws, X = on_device(order, K, M, 1)
    items = [dict(W=W, S=None, inv=0.01 * (i + 1), N=N, Y=torch.zeros(M, N, dtype=torch.float32, device="cuda")) for i, (W, N) in enumerate(zip(Ws, order))]
    before = c.launch_count()
    assert c.gemm_w8a8_bf16_group(c.make_group(items, K), X, 0.0, M, K, flags=4) == 0 and c.check_error("group") == 0
    assert c.launch_count() - before == launches
    for it in items:
        y = torch.zeros_like(it["Y"])
        assert c.gemm_w8a8_bf16(it["W"], it["inv"], X, 0.0, y, it["N"], M, K, flags=4) == 0 and c.check_error("alone") == 0
        assert torch.equal(y, it["Y"])

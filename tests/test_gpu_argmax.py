"""cuda_argmax_bf16 where its rounds of 16 logits per thread end, with and without 16-byte rows: the first of equal largest values
wherever it lies, NaN ahead of it, rows that begin past the others' ends."""
import numpy as np
import pytest

from tests._util import capi

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cols", [1, 7, 16383, 16384, 16385, 32768, 40001])
@pytest.mark.parametrize("pad", [0, 8, 3])
def test_the_first_maximum(cols, pad):
    import torch

    c, rng = capi(), np.random.default_rng(cols)
    ld = (cols + 7) // 8 * 8 + pad
    spots = sorted({0, cols // 2, max(0, cols - 2), cols - 1, min(cols - 1, 8191), min(cols - 1, 8192), min(cols - 1, 16384)})
    x = torch.from_numpy(rng.standard_normal((len(spots), ld)).astype(np.float32)).to(torch.bfloat16)
    x[:, cols:] = 99.0
    for r, s in enumerate(spots):
        x[r, s], x[r, cols - 1] = 50.0, 50.0
        if s > 3:
            x[r, 1] = float("nan")
    idx, val = torch.zeros(len(spots), dtype=torch.int32, device="cuda"), torch.zeros(len(spots), device="cuda")
    assert c.argmax_bf16(x.cuda(), len(spots), cols, idx, val, ld=ld) == 0 and c.check_error("argmax") == 0
    assert idx.tolist() == spots and val.tolist() == [50.0] * len(spots)

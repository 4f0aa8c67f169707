"""Per-column fp8 layers (format 3): the weights that enter the products are those of the block-scaled format, for any number of tokens."""
import numpy as np
import pytest

from oracle import linear as OL
from oracle.numerics import BF16, F16, rn

from test_linear_gpu import DevLinear

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [F16, BF16])
@pytest.mark.parametrize("scale", [1e-6, 2e-3, 0.3])
def test_fp8_weights_are_those_of_the_block_format(lib, dtype, scale):
    """w = T(e4m3) *_T T(scale) below 25 tokens too, as for format 2 and for more tokens.  Two ones per row of x: whatever order they are summed
    in, the output is the sum of two weights rounded once.  Scales down to products below f16's normal range."""
    K, N = 384, 256
    rng = np.random.default_rng(8)
    w8 = rng.integers(0, 0x7F, (K, N)).astype(np.uint8) | (rng.integers(0, 2, (K, N)) << 7).astype(np.uint8)
    s = np.repeat((scale * (1 + rng.random((K // 128, N // 128)))).astype(np.float32), 128, 1)
    cols, blocks = DevLinear(lib, K, N, 3, dtype, w8, scales=s), DevLinear(lib, K, N, 2, dtype, w8, scales=s[:, ::128].copy())
    w = OL.dequant_fp8_cols(w8, s, 128, dtype)
    for m in (1, 8, 13, 24, 25):
        x, at = np.zeros((m, K), np.float32), np.stack([rng.choice(K, 2, replace=False) for _ in range(m)])
        np.put_along_axis(x, at, 1, 1)
        y = cols.forward(x)
        assert np.array_equal(y, rn(w[at[:, 0]] + w[at[:, 1]], dtype)) and np.array_equal(y, blocks.forward(x))

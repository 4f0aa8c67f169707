"""Linear layers of a few tokens (linear_thin_kernel): the edges of its 8-token tiles, its splits of features and K, and every weight
format against the numpy oracle; strided and packed neighbours of the kernel.

Tolerance: as test_linear_gpu / test_linear_fp8_gpu -- T's rounding of the output (f16 2^-11, bf16 2^-8 relative) and, for fp8, of the
oracle's weights."""
import ctypes as C

import numpy as np
import pytest

from oracle import linear as OL
from oracle.numerics import BF16, F16, rn

from harness import from_dev_T, to_dev_T
from test_linear_fp8_gpu import _fp8_cols
from test_linear_gpu import DevLinear, _assert_close, _mk_u4

pytestmark = pytest.mark.gpu


def _layer(lib, fmt, dtype, K, N, rng, bias=None):
    if fmt == "u4":
        q, s, z = _mk_u4(rng, K, N)
        s = rn(s, dtype)
        return DevLinear(lib, K, N, 1, dtype, q, s, z, bias=bias), OL.dequant_u4(q, s, z, dtype)
    if fmt == "fp8":
        w8, s = _fp8_cols(rng, K, N)
        return DevLinear(lib, K, N, 3, dtype, w8, scales=s, bias=bias), OL.dequant_fp8_cols(w8, s, 128, dtype)
    w = rn((rng.standard_normal((K, N)) * 0.1 / np.sqrt(K)).astype(np.float32), dtype)
    return DevLinear(lib, K, N, 0, dtype, w, bias=bias), w


def _close(got, ref, dtype):
    _assert_close(got, ref, atol=2e-4 if dtype == F16 else 2e-3, rtol=2e-3 if dtype == F16 else 1.6e-2)


# one k-group; nine (a remainder for every number of warps along K); N on both sides of 16 * 296 and 32 * 296 features, and one CTA
@pytest.mark.parametrize("K,N", [(128, 128), (1152, 384), (256, 4736), (256, 4864), (384, 9472), (384, 9600), (128, 19072)])
@pytest.mark.parametrize("fmt,dtype", [("u4", F16), ("u4", BF16), ("fp8", F16), ("fp8", BF16), ("dense", F16), ("dense", BF16)])
def test_thin_matches_oracle(lib, fmt, dtype, K, N):
    rng = np.random.default_rng(K + N)
    bias = rn((rng.standard_normal(N) * 0.05).astype(np.float32), dtype)
    lin, w = _layer(lib, fmt, dtype, K, N, rng, bias)
    x = rn(rng.standard_normal((25, K)).astype(np.float32), dtype)
    ref = OL.linear(x, w, dtype, bias=bias)
    for m in (1, 7, 8, 9, 16, 17, 24, 25):                 # 25: the tcgen05 kernel
        _close(lin.forward(x[:m]), ref[:m], dtype)


@pytest.mark.parametrize("fmt,dtype", [("u4", F16), ("fp8", BF16), ("dense", F16)])
@pytest.mark.parametrize("m", [3, 16])
def test_thin_gated_silu(lib, fmt, dtype, m):
    K, N = 640, 2048
    rng = np.random.default_rng(m)
    lin, w = _layer(lib, fmt, dtype, K, N, rng)
    x = rn(rng.standard_normal((m, K)).astype(np.float32), dtype)
    _close(lin.forward(x, epilogue=1), OL.linear_gated_silu(x, w, dtype), dtype)


def test_thin_strides_and_neighbours(lib):
    """Rows of x and y further apart than they are long: what lies between them is neither read as data nor written."""
    import torch
    K, N, m = 512, 384, 11
    rng = np.random.default_rng(5)
    lin, w = _layer(lib, "u4", F16, K, N, rng)
    x = rn(rng.standard_normal((m, K)).astype(np.float32), F16)
    wide = torch.full((m, K + 24), float("nan"), dtype=torch.float16, device="cuda")
    wide[:, :K] = to_dev_T(x, F16)
    y = torch.full((m + 1, N + 8), 7.0, dtype=torch.float16, device="cuda")
    lin.L.check(lib.b200_linear_forward(C.byref(lin.d), wide.data_ptr(), wide.stride(0), m, y.data_ptr(), y.stride(0), 0, lin.ws.data_ptr(), lin.ws.numel(),
                                        torch.cuda.current_stream().cuda_stream), "forward")
    torch.cuda.synchronize()
    _close(from_dev_T(y[:m, :N].contiguous(), F16), OL.linear(x, w, F16), F16)
    assert (y[:m, N:] == 7).all() and (y[m] == 7).all()


def test_outputs_over_the_inputs(lib):
    """y in x's own memory: every output depends on all of x's row, as if x had been read first."""
    import torch
    K, m = 512, 5
    rng = np.random.default_rng(6)
    lin, w = _layer(lib, "dense", F16, K, K, rng)
    x = rn(rng.standard_normal((m, K)).astype(np.float32), F16)
    buf = to_dev_T(x, F16)
    lin.L.check(lib.b200_linear_forward(C.byref(lin.d), buf.data_ptr(), K, m, buf.data_ptr(), K, 0, lin.ws.data_ptr(), lin.ws.numel(),
                                        torch.cuda.current_stream().cuda_stream), "forward")
    torch.cuda.synchronize()
    _close(from_dev_T(buf, F16), OL.linear(x, w, F16), F16)


def test_nan_and_infinity_stay_in_their_rows(lib):
    """A token with an infinity or a NaN does not change the other tokens of its tile; a NaN weight (e4m3 0x7f) is a NaN in its column only."""
    K, N, m = 256, 256, 6
    rng = np.random.default_rng(7)
    w8, s = _fp8_cols(rng, K, N)
    w8 = w8.copy()
    w8[17, 33] = 0x7F
    lin = DevLinear(lib, K, N, 3, BF16, w8, scales=s)
    x = rn(rng.standard_normal((m, K)).astype(np.float32), BF16)
    x[2, 100], x[4, 3] = np.inf, np.nan
    y = lin.forward(x)
    assert np.isnan(y[:, 33]).all() and np.isnan(y[4]).all() and not np.isfinite(y[2]).any()
    keep = np.delete(np.arange(N), 33)
    clean = OL.dequant_fp8_cols(np.where(w8 == 0x7F, 0, w8).astype(np.uint8), s, 128, BF16)
    for t in (0, 1, 3, 5):
        _close(y[t][keep], OL.linear(x[t:t + 1], clean, BF16)[0][keep], BF16)

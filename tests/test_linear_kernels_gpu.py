"""Each kernel of the linear layers in its steady state and at few tokens, whichever of them b200_linear_forward takes.

1. linear_thin_kernel over more k-groups than its rings hold, for every number of warps along K (8, 4, 2), both widths of a warp's tile and one to three token
   tiles: stages of X refilled, weights reloaded, an odd last group.  Weights are exact in T (scales are powers of two), so a float64 product is the
   reference and the bound is the output's rounding plus K / 16 + 16 float sums of terms up to |x| |w|.
2. The tcgen05 kernel below 25 tokens (through packed activations), with plain and subnormal u4 layouts, against the numpy oracle."""
import ctypes as C

import numpy as np
import pytest

from oracle import linear as OL
from oracle.numerics import BF16, F16, rn

from harness import from_dev_T, to_dev_T
from test_linear_fp8_gpu import _fp8_cols
from test_linear_gpu import DevLinear, _assert_close, _layout_flag, _mk_u4

pytestmark = pytest.mark.gpu

FEW = 1
STEADY = {
    "u4": [(8064, 2048, (1, 9, 16)), (4096, 2048, (17, 24)), (4224, 6144, (8, 9)), (4096, 6144, (24,)), (3328, 9600, (1, 16)), (2688, 9600, (24,)), (2176, 19072, (8,))],
    "fp8": [(8064, 2048, (1, 16)), (4224, 6144, (8, 9)), (6016, 5120, (17, 24)), (3328, 9600, (1, 16, 24)), (2176, 19072, (8,))],
    "dense": [(8064, 2048, (1, 8)), (4096, 2048, (9, 24)), (4096, 4608, (16,)), (4224, 6144, (8,)), (2944, 6144, (9,)), (3200, 5120, (24,)), (3328, 9600, (1,)), (1920, 9600, (16,)), (1664, 9600, (17,)),
              (2176, 19072, (8,))],
}


@pytest.mark.parametrize("fmt,dtype", [("u4", "f16"), ("u4", "bf16"), ("fp8", "f16"), ("fp8", "bf16"), ("dense", "f16"), ("dense", "bf16")])
def test_few_tokens_over_many_k_groups(lib, fmt, dtype):
    import torch
    from lmdeploy_b200 import _lib as L
    from lmdeploy_b200.turbomind.runtime import PreparedLinear
    lib.b200_linear_load_plans(None)
    T, eps = (torch.float16, 2.0 ** -11) if dtype == "f16" else (torch.bfloat16, 2.0 ** -8)
    st = torch.cuda.current_stream().cuda_stream
    for K, N, ms in STEADY[fmt]:
        g = torch.Generator(device="cuda").manual_seed(K + N)
        s = z = None
        scale = 2.0 ** torch.randint(-9, -5, (K // 128, N), generator=g, device="cuda").float()
        wide = scale.double().repeat_interleave(128, 0)
        if fmt == "u4":
            w = torch.randint(-2**31, 2**31 - 1, (K, N // 8), generator=g, device="cuda", dtype=torch.int32)
            s, z = scale.to(T), torch.full((K // 128, N), 8.0, device="cuda").to(T)
            ref_w = (torch.stack([(w >> (4 * i)) & 15 for i in range(8)], -1).view(K, N).double() - 8) * wide
        elif fmt == "fp8":
            w, s = torch.randn(K, N, generator=g, device="cuda").to(torch.float8_e4m3fn), scale
            ref_w = w.double() * wide
            w = w.view(torch.uint8)
        else:
            w = (torch.randn(K, N, generator=g, device="cuda") * 0.02).to(T)
            ref_w = w.double()
        pl = PreparedLinear(lib, K, N, {"u4": L.FMT_U4, "fp8": L.FMT_FP8_COL, "dense": L.FMT_DENSE}[fmt], dtype, "cuda")
        pl.prepare(lib, w, s, z)
        for m in ms:
            assert lib.b200_linear_kernel(C.byref(pl.desc), m, 0) == FEW, (K, N, m)
            x = torch.randn(m, K, generator=g, device="cuda").to(T)
            ws = torch.zeros(lib.b200_linear_workspace_bytes(C.byref(pl.desc), m), dtype=torch.uint8, device="cuda")
            y = torch.full((m + 1, N), 7.0, dtype=T, device="cuda")
            L.check(lib.b200_linear_forward(C.byref(pl.desc), x.data_ptr(), K, m, y.data_ptr(), N, 0, ws.data_ptr(), ws.numel(), st), "forward")
            ref, terms = x.double() @ ref_w, x.double().abs() @ ref_w.abs()
            assert ((y[:m].double() - ref).abs() <= eps * ref.abs() + (K / 16 + 16) * 2.0 ** -23 * terms).all(), (K, N, m)
            assert (y[m] == 7).all()


def _packed(lib, lin, x, dtype):
    import torch
    m, K, N, mt, st = x.shape[0], lin.K, lin.N, max(16, (x.shape[0] + 15) // 16 * 16), torch.cuda.current_stream().cuda_stream
    dx = to_dev_T(x, dtype)
    xp, y = torch.zeros(K // 8, mt, 8, dtype=dx.dtype, device="cuda"), torch.zeros(m, N, dtype=dx.dtype, device="cuda")
    lin.L.check(lib.b200_pack_activations(dx.data_ptr(), K, m, K, mt, 0 if dtype == F16 else 1, xp.data_ptr(), st), "pack")
    lin.L.check(lib.b200_linear_forward_packed(C.byref(lin.d), xp.data_ptr(), mt, m, y.data_ptr(), N, 0, 0, lin.ws.data_ptr(), lin.ws.numel(), st), "packed")
    torch.cuda.synchronize()
    return from_dev_T(y, dtype)


@pytest.mark.parametrize("shape", [(256, 128), (1024, 256), (4096, 6144), (14336, 4096)])
def test_u4_packed_at_few_tokens(lib, shape):
    K, N = shape
    rng = np.random.default_rng(K + N)
    q, s, z = _mk_u4(rng, K, N)
    lin = DevLinear(lib, K, N, 1, F16, q, s, z)
    x = rn(rng.standard_normal((24, K)).astype(np.float32), F16)
    ref = OL.linear(x, OL.dequant_u4(q, s, z, F16), F16)
    for m in (1, 3, 16, 24):
        _assert_close(_packed(lib, lin, x[:m], F16), ref[:m])


@pytest.mark.parametrize("dtype", [F16, BF16])
@pytest.mark.parametrize("shape", [(1024, 256), (512, 384), (4096, 4096)])
def test_fp8_packed_at_few_tokens(lib, shape, dtype):
    K, N = shape
    rng = np.random.default_rng(K + N)
    w8, scale = _fp8_cols(rng, K, N)
    lin = DevLinear(lib, K, N, 3, dtype, w8, scales=scale)
    x = rn(rng.standard_normal((17, K)).astype(np.float32), dtype)
    ref = OL.linear(x, OL.dequant_fp8_cols(w8, scale, 128, dtype), dtype)
    for m in (1, 17):
        _assert_close(_packed(lib, lin, x[:m], dtype), ref[:m], atol=2e-4 if dtype == F16 else 2e-3, rtol=2e-3 if dtype == F16 else 1.6e-2)


@pytest.mark.parametrize("m", [17, 33])
@pytest.mark.parametrize("packed", [False, True])
def test_u4_layouts_in_both_kernels(lib, m, packed):
    """The plain layout (a scale of 0.5 and more keeps a whole f16 tensor in it) and the subnormal one; 17 tokens row-major is the few-token kernel."""
    K, N = 1024, 256
    rng = np.random.default_rng(77)
    w = (rng.standard_normal((K, N)) * 0.1 / np.sqrt(K)).astype(np.float32)
    x = rn(rng.standard_normal((m, K)).astype(np.float32), F16)
    for plain in (False, True):
        if plain:
            w[:128, :64] *= 3000.0
        q, s, z = OL.quantize_groupwise_u4(w, 128)
        lin = DevLinear(lib, K, N, 1, F16, q, s, z)
        assert _layout_flag(lin) == (0 if plain else 1)
        y = _packed(lib, lin, x, F16) if packed else lin.forward(x)
        _assert_close(y, OL.linear(x, OL.dequant_u4(q, s, z, F16), F16), atol=2e-3 if plain else 2e-4, rtol=2e-3)

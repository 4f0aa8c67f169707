"""Weights written and used on one stream with nothing in between: a layer's calls see all of what b200_linear_prepare in front of them wrote
(they are launched before the kernel ahead has ended), and b200_linear_forward what any kernel in front of it wrote."""
import ctypes as C

import pytest

pytestmark = pytest.mark.gpu


def _weights(torch, fmt, T, K, N, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    if fmt == 1:
        q = torch.randint(-2**31, 2**31 - 1, (K, N // 8), generator=g, device="cuda", dtype=torch.int32)
        s = (torch.rand(K // 128, N, generator=g, device="cuda") * 0.01 + 0.001).to(T)
        if seed % 2:
            s[0, 0] = 0.75                                  # f16: the whole tensor keeps the plain layout, so the layout flag changes too
        return q, s, torch.full((K // 128, N), 8.0, device="cuda").to(T)
    if fmt == 0:
        return (torch.randn(K, N, generator=g, device="cuda") * 0.02).to(T), None, None
    w = torch.randn(K, N, generator=g, device="cuda").to(torch.float8_e4m3fn).view(torch.uint8)
    return w, torch.rand(K // 128, N // 128 if fmt == 2 else N, generator=g, device="cuda") * 0.02 + 0.001, None


class Layer:
    def __init__(self, lib, fmt, dtype, K, N, m):
        import torch
        from lmdeploy_b200 import _lib as L
        from lmdeploy_b200.turbomind.runtime import PreparedLinear
        self.lib, self.L, self.torch, self.K, self.N, self.m = lib, L, torch, K, N, m
        self.T = torch.float16 if dtype == "f16" else torch.bfloat16
        self.pl = PreparedLinear(lib, K, N, fmt, dtype, "cuda")
        self.sets = [_weights(torch, fmt, self.T, K, N, s) for s in (0, 1)]
        self.mt = max(16, (m + 15) // 16 * 16)
        self.ws = torch.zeros(lib.b200_linear_workspace_bytes(C.byref(self.pl.desc), m), dtype=torch.uint8, device="cuda")
        self.x = torch.randn(m, K, device="cuda", generator=torch.Generator(device="cuda").manual_seed(5)).to(self.T)
        self.xp = torch.zeros(K // 8, self.mt, 8, dtype=self.T, device="cuda")
        self.st = torch.cuda.current_stream().cuda_stream
        L.check(lib.b200_pack_activations(self.x.data_ptr(), K, m, K, self.mt, 0 if dtype == "f16" else 1, self.xp.data_ptr(), self.st), "pack")

    def prepare(self, i):
        self.pl.prepare(self.lib, *self.sets[i])

    def forward(self, y, packed):
        if packed:
            self.L.check(self.lib.b200_linear_forward_packed(C.byref(self.pl.desc), self.xp.data_ptr(), self.mt, self.m, y.data_ptr(), self.N, 0, 0, self.ws.data_ptr(),
                                                             self.ws.numel(), self.st), "packed")
        else:
            self.L.check(self.lib.b200_linear_forward(C.byref(self.pl.desc), self.x.data_ptr(), self.K, self.m, y.data_ptr(), self.N, 0, self.ws.data_ptr(), self.ws.numel(), self.st),
                         "forward")

    def expected(self, packed):
        out = []
        for i in (0, 1):
            self.prepare(i)
            self.torch.cuda.synchronize()
            out.append(self.torch.zeros(self.m, self.N, dtype=self.T, device="cuda"))
            self.torch.cuda.synchronize()
            self.forward(out[-1], packed)
            self.torch.cuda.synchronize()
        return out


# 2048 x 4096: 8 to 16 MB to write; 256 x 37888: the dense head's kernel at 128 tokens
@pytest.mark.parametrize("fmt,dtype,K,N", [(0, "f16", 2048, 4096), (0, "bf16", 256, 37888), (1, "f16", 2048, 4096), (1, "bf16", 2048, 4096), (2, "f16", 2048, 4096), (3, "bf16", 2048, 4096)])
@pytest.mark.parametrize("m", [1, 24, 64, 128])
@pytest.mark.parametrize("packed", [False, True])
def test_prepare_then_forward(lib, fmt, dtype, K, N, m, packed):
    import torch
    layer = Layer(lib, fmt, dtype, K, N, m)
    ref = layer.expected(packed)
    assert not (ref[0] == ref[1]).all()
    ys = [torch.zeros_like(ref[0]) for _ in range(16)]
    torch.cuda.synchronize()
    for i, y in enumerate(ys):
        layer.prepare(i % 2)
        layer.forward(y, packed)
    torch.cuda.synchronize()
    assert all((y == ref[i % 2]).all() for i, y in enumerate(ys))


@pytest.mark.parametrize("fmt,dtype", [(0, "f16"), (1, "f16"), (2, "bf16"), (3, "f16")])
@pytest.mark.parametrize("m", [1, 24, 64, 128])
def test_any_kernel_then_forward(lib, fmt, dtype, m):
    """Prepared weights exchanged by a kernel of the program's own."""
    import torch
    layer = Layer(lib, fmt, dtype, 2048, 4096, m)
    ref = layer.expected(False)
    blobs = []
    for i in (0, 1):
        layer.prepare(i)
        blobs.append(layer.pl.storage.clone())
    flip = blobs[0] ^ blobs[1]
    ys = [torch.zeros_like(ref[0]) for _ in range(16)]
    torch.cuda.synchronize()
    for i, y in enumerate(ys):                              # set 1 lies there: 0, 1, 0, ..
        torch.bitwise_xor(layer.pl.storage, flip, out=layer.pl.storage)
        layer.forward(y, False)
    torch.cuda.synchronize()
    assert all((y == ref[i % 2]).all() for i, y in enumerate(ys))

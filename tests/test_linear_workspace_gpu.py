"""Linear layers on packed activations whose K is split over CTAs: the partial sums lie in the caller's workspace, of which multiples of eight bytes are enough (the
activations, which need more, come from elsewhere).  Same sums, bit for bit."""
import ctypes as C

import pytest

from test_linear_order_gpu import Layer

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fmt,dtype", [(0, "bf16"), (1, "f16"), (3, "bf16")])
@pytest.mark.parametrize("K,N", [(2048, 512), (3584, 1280)])
@pytest.mark.parametrize("m", [33, 128])
@pytest.mark.parametrize("gated", [0, 1])
def test_workspace_at_multiples_of_eight_bytes(lib, fmt, dtype, K, N, m, gated):
    import torch
    layer, nout = Layer(lib, fmt, dtype, K, N, m), N // 2 if gated else N
    layer.prepare(0)
    room = torch.zeros(layer.ws.numel() + 16, dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    out = []
    for at in (0, 8):
        y = torch.full((m, nout), float("nan"), dtype=layer.T, device="cuda")
        layer.L.check(lib.b200_linear_forward_packed(C.byref(layer.pl.desc), layer.xp.data_ptr(), layer.mt, m, y.data_ptr(), nout, gated, 0, room.data_ptr() + at,
                                                     layer.ws.numel(), layer.st), "packed")
        torch.cuda.synchronize()
        room.zero_()                                        # arrival counters lie at the workspace's start
        out.append(y)
    assert torch.isfinite(out[0]).all() and torch.equal(out[0], out[1])

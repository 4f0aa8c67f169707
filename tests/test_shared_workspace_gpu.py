"""One workspace for prefill attention and for decode attention of every batch size, as a model's steps use it: the arrival counters of the decode
kernel's in-kernel fix-up stay zero whatever ran before, so that the one-launch form still merges the segments that CTAs share."""
import ctypes as C

import numpy as np
import pytest

from harness import PagedCase, from_dev_T

pytestmark = pytest.mark.gpu


def _decode(lib, case, ws, flags):
    import torch
    from lmdeploy_b200 import _lib as L
    p = case.params(lib, workspace=ws)
    plan = torch.zeros(case.B + 1, dtype=torch.int32, device="cuda")
    L.check(lib.b200_decode_attention_plan(plan.data_ptr(), p.cu_k_len, p.finished, case.B, p.stream), "plan")
    p.plan, p.debug_flags = plan.data_ptr(), flags
    case.d_out.zero_()                                  # a segment that nobody merges would keep what stands here
    L.check(lib.b200_decode_attention(C.byref(p)), "b200_decode_attention")
    torch.cuda.synchronize()
    return from_dev_T(case.d_out, case.dtype).view(np.uint16).copy()


@pytest.mark.parametrize("heads", [(8, 2), (32, 8)])
def test_prefill_and_decode_share_a_workspace(lib, heads):
    import torch
    from lmdeploy_b200 import _lib as L
    cases = [PagedCase(batch_hist=h, num_heads=heads[0], num_kv_heads=heads[1], kv_bits=8, seed=len(h)) for h in ([2047, 700, 4100], [63, 1500] * 8)]
    for c in cases:
        c.upload()
    nbytes = max(max(lib.b200_decode_attention_workspace_bytes(c.B, *heads), lib.b200_prefill_attention_workspace_bytes(c.B, heads[0])) for c in cases)
    own = [_decode(lib, c, None, 4) for c in cases]     # three kernels, no counters
    ws = torch.zeros(nbytes, dtype=torch.uint8, device="cuda")
    for first, then in [(0, 0), (0, 1), (1, 0), (1, 1)]:
        p = cases[first].params(lib, workspace=ws)
        L.check(lib.b200_prefill_attention(C.byref(p)), "b200_prefill_attention")
        assert np.array_equal(_decode(lib, cases[then], ws, 8), own[then]), (first, then)
        assert np.array_equal(_decode(lib, cases[1 - then], ws, 8), own[1 - then]), (first, then)

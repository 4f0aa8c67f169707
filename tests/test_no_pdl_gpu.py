"""B200_NO_PDL turns programmatic dependent launches off in the hybrid library too: the edges of a captured attention say which kind they are."""
import ctypes as C
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SCRIPT = """
import ctypes as C, sys
sys.path.insert(0, sys.argv[1])
import torch
from lmdeploy_b200 import _hybrid_lib as H
lib, n, heads, kv, d = H.load(), 256, 4, 2, 128
i32 = dict(dtype=torch.int32, device="cuda")
pool = torch.randn(4, 64 * 2 * kv * d, device="cuda").bfloat16()
ptrs = (pool.data_ptr() + torch.arange(4, device="cuda") * pool.shape[1] * 2).contiguous()
cu, seq, pos = torch.tensor([0, 4], **i32), torch.zeros(n, **i32), torch.arange(n, **i32)
qn, scores, ml = torch.randn(n, heads * d, device="cuda"), torch.zeros(n, heads, 256, device="cuda"), torch.zeros(n, heads, 1, 2, device="cuda")
part, y = torch.zeros(n, 1, heads * d, device="cuda"), torch.zeros(n, heads * d, dtype=torch.bfloat16, device="cuda")
a = H.WindowArgs(n=n, heads=heads, kv_heads=kv, dim=d, vdim=d, block_len=64, splits=1, scale=d ** -0.5, eps=1e-6, ld=1, maps=1, out_scale=1.0, ld_y=heads * d, score_ld=256, dtype=H.BF16,
                 sequences=1)
a.q = a.k = a.v = a.qn = qn.data_ptr()
a.tok_seq, a.tok_pos, a.block_ptrs, a.cu_blocks, a.v_off = seq.data_ptr(), pos.data_ptr(), ptrs.data_ptr(), cu.data_ptr(), 64 * kv * d * 2
a.scores, a.ml, a.o_part, a.y = scores.data_ptr(), ml.data_ptr(), part.data_ptr(), y.data_ptr()
g, s = torch.cuda.CUDAGraph(keep_graph=True), torch.cuda.Stream()
torch.cuda.synchronize()
with torch.cuda.graph(g, stream=s):
    a.stream = s.cuda_stream
    H.check(lib.b200h_window_attention(C.byref(a)), "window_attention")
drv, graph, count = C.CDLL("libcuda.so.1"), C.c_void_p(g.raw_cuda_graph()), C.c_size_t(0)
assert drv.cuGraphGetEdges_v2(graph, None, None, None, C.byref(count)) == 0
ends, data = (C.c_void_p * count.value)(), ((C.c_uint8 * 8) * count.value)()
assert drv.cuGraphGetEdges_v2(graph, ends, (C.c_void_p * count.value)(), data, C.byref(count)) == 0
print("edges", count.value, "programmatic", sum(e[2] == 1 for e in data))
"""


@pytest.mark.parametrize("off,programmatic", [(False, 1), (True, 0)])
def test_hybrid_attention_follows_the_switch(off, programmatic):
    env = {k: v for k, v in os.environ.items() if k != "B200_NO_PDL"}
    if off:
        env["B200_NO_PDL"] = "1"
    r = subprocess.run([sys.executable, "-c", SCRIPT, ROOT], env=env, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
    assert r.stdout.split()[-4:] == ["edges", "1", "programmatic", str(programmatic)]     # plan -> attention

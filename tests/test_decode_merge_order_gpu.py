"""Decode attention of a few long sequences: the pieces of a sequence are summed in ascending order whichever kernel merges them, so outputs do not depend
on how many sequences a step has beside it (and the steps of a model stay what they were, byte for byte).

Keys are zero, so every softmax weight is one and a piece is a sum of values: large ones, small ones, the large ones negated, small ones.  In order the
large sum swallows bits of the small values behind it; in any other order it does not.  Sums of a piece are exact in float, so a float32 loop is
the reference, bit for bit."""
import ctypes as C
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

D, PAGE = 128, 64


def _attend(lib, values, heads, flags):
    import torch
    from lmdeploy_b200 import _lib as L
    tiles = values.shape[0]
    pool = torch.zeros(tiles, 1, 2, PAGE, D, dtype=torch.float16, device="cuda")          # one kv head: keys, values
    pool[:, 0, 1] = torch.from_numpy(values).cuda()[:, None]
    i32 = dict(dtype=torch.int32, device="cuda")
    ptrs = pool.data_ptr() + torch.arange(tiles, device="cuda") * pool[0].numel() * 2
    qkv = torch.zeros(1, (heads + 2) * D, dtype=torch.float16, device="cuda")              # the new token's key and value are zero
    qkv[:, :heads * D] = torch.randn(heads * D, device="cuda").half()
    cu_q, cu_k, cu_b = torch.tensor([0, 1], **i32), torch.tensor([0, tiles * PAGE], **i32), torch.tensor([0, tiles], **i32)
    out, ws = torch.zeros(1, heads * D, dtype=torch.float16, device="cuda"), torch.zeros(lib.b200_decode_attention_workspace_bytes(1, heads, 1), dtype=torch.uint8, device="cuda")
    p = L.AttentionParams()
    p.out, p.q, p.stride = out.data_ptr(), qkv.data_ptr(), qkv.stride(0)
    p.k, p.v = p.q + 2 * heads * D, p.q + 2 * (heads + 1) * D
    p.cu_q_len, p.cu_k_len, p.block_ptrs, p.cu_block_nums = cu_q.data_ptr(), cu_k.data_ptr(), ptrs.data_ptr(), cu_b.data_ptr()
    p.block_len, p.token_num, p.batch_size, p.max_k_len = PAGE, 1, 1, tiles * PAGE
    p.num_heads, p.num_kv_heads, p.size_per_head, p.inv_sqrt_dh = heads, 1, D, math.log2(math.e) / math.sqrt(D)
    p.rope = L.RopeConfig(type=1, dim=D, base=1e4)
    p.workspace, p.workspace_bytes, p.stream, p.debug_flags = ws.data_ptr(), ws.numel(), torch.cuda.current_stream().cuda_stream, flags
    L.check(lib.b200_decode_attention(C.byref(p)), "decode_attention")
    torch.cuda.synchronize()
    return out.cpu().numpy().reshape(heads, D)


@pytest.mark.parametrize("heads", [1, 6, 8])
@pytest.mark.parametrize("flags", [0, 8])                # 8: merged inside the main kernel
@pytest.mark.parametrize("tiles", [40, 200, 900])        # a piece per tile: a third of and more than one pass over pieces; a few tiles per piece
def test_pieces_are_summed_in_order(lib, tiles, heads, flags):
    grid = lib.b200_decode_attention_grid(0, 0)
    t, d = np.arange(tiles)[:, None], np.arange(D)[None]
    small = (2 * ((7 * t + 3 * d) % 16) + 1.0) / (1 if tiles > grid else 64)
    quarter = 4 * t // tiles
    values = np.where(quarter == 0, 60000.0, np.where(quarter == 2, -60000.0, small)).astype(np.float16)
    sums = values.astype(np.float64) * np.where(t == tiles - 1, PAGE - 1, PAGE)
    cuts = [tiles * c // grid for c in range(grid + 1)] if tiles > grid else range(tiles + 1)
    acc, free = np.zeros(D, np.float32), sums.sum(0)
    for a, b in zip(cuts[:-1], cuts[1:]):
        piece = sums[a:b].sum(0)
        assert (piece == piece.astype(np.float32)).all()
        acc = (acc + piece.astype(np.float32)).astype(np.float32)
    ref = (acc / np.float32(tiles * PAGE)).astype(np.float16)
    assert tiles != 200 or ((ref != (free / (tiles * PAGE)).astype(np.float16)).mean() > 0.5)                 # the order is seen
    out = _attend(lib, values, heads, flags)
    assert (out == ref[None]).all()

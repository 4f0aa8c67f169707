"""Decode attention over int4 pages, whose consumer warps take two tiles of 64 keys at a time: runs of tiles that end on either side of two and of a sequence's
last tile, pages of one and of two tiles (copied in four and in six parts), values whose scales let codes through as they are in all, some or none of
the tiles, scores that grow from tile to tile.  Many sequences share one history, so that a CTA has dozens of tiles in a row; against 64 bits."""
import ctypes as C

import numpy as np
import pytest

from oracle import attention as OA
from oracle.numerics import BF16, F16, rn

from harness import PagedCase

pytestmark = pytest.mark.gpu

BATCH = 200
U = {F16: 2.0 ** -11, BF16: 2.0 ** -8}                                      # half a unit in the last place, relative


def _run(case, lib, qkv, G, plan=False):
    """BATCH sequences over the pages of `case` (one sequence), each with a last page of its own for its new token -> [BATCH, G, 128]."""
    import torch
    from lmdeploy_b200 import _lib as L
    from harness import from_dev_T, to_dev_T
    case.upload()
    hist = int(case.hist[0])
    own = case.d_pool[case.block_tables[0][-1]].repeat(BATCH, 1)            # a page that is not full holds cached tokens too
    ptrs = case.d_block_ptrs.repeat(BATCH, 1)
    ptrs[:, -1] = own.data_ptr() + torch.arange(BATCH, device="cuda") * case.cache.block_bytes
    cu = torch.arange(BATCH + 1, dtype=torch.int32, device="cuda")
    cu_k, cu_blocks = cu * (hist + 1), cu * ptrs.shape[1]
    d_qkv = to_dev_T(qkv, case.dtype)
    out = torch.zeros(BATCH, G * 128, dtype=d_qkv.dtype, device="cuda")
    ws = torch.zeros(lib.b200_decode_attention_workspace_bytes(BATCH, G, 1), dtype=torch.uint8, device="cuda")
    p = case.params(lib, workspace=ws)
    p.out, p.q, p.k, p.v = out.data_ptr(), d_qkv.data_ptr(), d_qkv.data_ptr() + G * 256, d_qkv.data_ptr() + (G + 1) * 256
    p.cu_q_len, p.cu_k_len, p.block_ptrs, p.cu_block_nums = cu.data_ptr(), cu_k.data_ptr(), ptrs.data_ptr(), cu_blocks.data_ptr()
    p.token_num = p.batch_size = BATCH
    if plan:                                                                # the caller's: keys are streamed, and segments looked up, beside the prologue
        tiles = torch.zeros(BATCH + 1, dtype=torch.int32, device="cuda")
        L.check(lib.b200_decode_attention_plan(tiles.data_ptr(), p.cu_k_len, p.finished, BATCH, p.stream), "plan")
        p.plan = tiles.data_ptr()
    L.check(lib.b200_decode_attention(C.byref(p)), "b200_decode_attention")
    torch.cuda.synchronize()
    return from_dev_T(out, case.dtype).reshape(BATCH, G, 128)


def pages(hist, block_len, G, dtype, odd):
    """(a sequence's pages, queries | keys | values of BATCH new tokens behind it)"""
    case = PagedCase(batch_hist=[hist], num_heads=G, num_kv_heads=1, kv_bits=4, block_len=block_len, dtype=dtype, seed=G, rope=OA.RopeParam(type=OA.ROPE_NULL))
    rng = np.random.default_rng(hist)
    tok = np.arange(hist)[:, None, None]
    # constant vectors (scale 0) do not go through as codes: one warp's keys (four groups of four, 16 apart) of every third tile; every third tile; all
    flat = {"none": tok < 0, "warps": (tok // 64 % 3 == 1) & (tok // 4 % 4 == 2), "tiles": tok // 64 % 3 == 1, "all": tok >= 0}[odd]
    k = rn(rng.standard_normal((hist, 1, 128)).astype(np.float32), dtype)
    v = rn(np.where(flat, 0.5 * (tok % 7) - 1.5, rng.standard_normal((hist, 1, 128))).astype(np.float32), dtype)
    OA.process_kv(case.cache, case.block_tables[0], case.layer, 0, k, v, case.rope, None, None)
    return case, rn(rng.standard_normal((BATCH, (G + 2) * 128)).astype(np.float32), dtype)


class Exact:
    """Outputs in 64 bits over the pages' keys and values and, for every output, how far a correct one may be off at worst and the square of how far it is
    off on average.

    A weight is rounded to T (u of its term), and so is the result.  bf16 kernels round keys and values to T as well, which the de-quantised pages have
    behind them; in f16 they are not rounded, but for values that do not go through as codes (constant vectors here, which are exact).  Scores are float sums
    (2^-16 of the products' magnitudes is ample), outputs float sums of terms up to twice the largest value; the mean leaves both out.  Roundings of different weights do not know of one
    another: uniform ones have a mean square of a third of u^2."""

    def __init__(self, case, qkv, G):
        hist = int(case.hist[0])
        self.dtype, self.G, self.qkv, self.u = case.dtype, G, qkv, U[case.dtype]
        new = OA.PagedKvCache(len(qkv), 1, case.layout, case.dtype)
        for b in range(len(qkv)):
            new.write_token(b, 0, 0, 0, qkv[b, G * 128:(G + 1) * 128], qkv[b, (G + 1) * 128:])
        stored, OA.kv_dequant = OA.kv_dequant, stored_or_64(OA.kv_dequant, case.dtype)
        try:
            cached = case.cache.read_tokens(case.block_tables[0], case.layer, 0, hist)
            self.kv = [[np.concatenate([c, n]).astype(np.float64) for c, n in zip(cached, new.read_tokens([b], 0, 0, 1))] for b in range(len(qkv))]
        finally:
            OA.kv_dequant = stored

    def weights(self, b):
        """(weights, sums of the magnitudes of each score's products) [G, keys]"""
        q = self.qkv[b, :self.G * 128].astype(np.float64).reshape(self.G, 128)
        s = q @ self.kv[b][0].T / np.sqrt(128.0)
        p = np.exp(s - s.max(-1, keepdims=True))
        return p / p.sum(-1, keepdims=True), np.abs(q) @ np.abs(self.kv[b][0]).T / np.sqrt(128.0)

    def __call__(self, b):
        p, mag = self.weights(b)
        V, u = self.kv[b][1], self.u
        ref, sums = p @ V, 2.0 ** -18 * np.abs(V).max() + 2.0 ** -24
        worst = (p * (2 * u + 2.0 ** -16 * mag)) @ np.abs(V) + u * np.abs(ref) + sums
        square = (u * u / 3) * (p ** 2 @ V ** 2 + ref ** 2)
        return ref, worst, square

    def check(self, got, every):
        """got(b) -> outputs [G, 128] of sequence b"""
        off, mean = [], []
        for b in range(0, len(self.qkv), every):
            ref, worst, square = self(b)
            err = np.abs(got(b) - ref)
            assert (err <= worst).all(), (b, float((err / worst).max()))
            off.append((err ** 2).mean()), mean.append(square.mean())
        # outputs show 0.6 to 0.8 of the expected mean, with a tile left out, taken twice or weighed with another's values 36 times it in bf16 and 290 times in f16
        assert np.mean(off) <= np.mean(mean), (np.mean(off) / np.mean(mean)) ** 0.5


def stored_or_64(stored, dtype):
    return stored if dtype == BF16 else lambda codes, scale, zero, _: codes * scale[:, None].astype(np.float64) + zero[:, None].astype(np.float64)


# 64 tiles or so for each of 200 sequences: 28 to 30 in a row per CTA of 444, cut anywhere
SHAPES = [(4031, 64, 4), (4032, 64, 4), (4095, 64, 8), (4096, 128, 4), (4160, 128, 1)]
ODD = ["none", "warps", "tiles", "all"]


@pytest.mark.parametrize("hist,block_len,G", SHAPES)
@pytest.mark.parametrize("dtype", [F16, BF16])
@pytest.mark.parametrize("odd", ODD)
def test_tiles_at_once(hist, block_len, G, dtype, odd, lib):
    case, qkv = pages(hist, block_len, G, dtype, odd)
    got = _run(case, lib, qkv, G)
    Exact(case, qkv, G).check(lambda b: got[b], 7)


@pytest.mark.parametrize("dtype", [F16, BF16])
def test_tiles_at_once_with_the_callers_plan(dtype, lib):
    case, qkv = pages(4095, 64, 4, dtype, "warps")
    got = _run(case, lib, qkv, 4, plan=True)
    Exact(case, qkv, 4).check(lambda b: got[b], 7)
    assert np.array_equal(got, _run(case, lib, qkv, 4))


@pytest.mark.parametrize("tile", [1, 2])
@pytest.mark.parametrize("at", [0, 3])
def test_a_tile_is_weighed_against_the_maxima_up_to_it(tile, at, lib):
    """Narrow values far from zero in the first tiles, zeros (in every other dimension) behind them, and in the first tile behind them a key of each warp whose
    score is 22 octaves above all others.  Weighed against the maximum of its own time a tile's weights are twice the least scale, rounded to 11 bits;
    against the loud keys', which come later, they would be subnormal numbers of 8.5 steps."""
    hist, G = 4095, 4
    case = PagedCase(batch_hist=[hist], num_heads=G, num_kv_heads=1, kv_bits=4, seed=1, rope=OA.RopeParam(type=OA.ROPE_NULL))
    k, v = np.zeros((hist, 1, 128), np.float32), np.zeros((hist, 1, 128), np.float32)
    v[:64 * tile] = 1.5
    v[:, :, ::2] += 2.0 ** -9                                               # scale 2^-9 / 15; from 2^-14 on codes go through as they are
    k[64 * tile + at + np.array([0, 20, 40, 60]), 0, 0] = 15.0
    OA.process_kv(case.cache, case.block_tables[0], case.layer, 0, k, v, case.rope, None, None)
    qkv = np.zeros((BATCH, (G + 2) * 128), np.float32)
    q = float(rn(np.float32(22 * np.log(2.0) * np.sqrt(128.0) / 15.0), F16))
    qkv[:, :G * 128:128] = q
    got, w = _run(case, lib, qkv, G)[:, :, 1::2], np.exp(-15.0 * q / np.sqrt(128.0))
    ref = 64 * tile * 1.5 * w / (4 + (hist + 1 - 4) * w)
    # the weights' rounding (2^-11), float sums in which parts some 20 times as large cancel, and the result's half step
    assert (np.abs(got - ref) <= 2.0 ** -10 * ref + 2.0 ** -25).all(), float(np.abs(got / ref - 1).max())

"""Decode attention over int8 / int4 pages in f16, whose codes enter the tensor cores unconverted: scales at and beyond the limits of that form (constant
vectors, tiny and huge ranges, both kinds side by side in one accumulator, narrow ranges far from zero, long tails of small weights), sequences around
64-token tiles, against 64-bit arithmetic on the de-quantised pages."""
import numpy as np
import pytest

from oracle import attention as OA
from oracle.numerics import F16, rn

from harness import PagedCase

pytestmark = pytest.mark.gpu

U = 2.0 ** -11                                                              # half a unit in the last place of f16, relative
LIMITS = {8: (2.0 ** -16, 0.5), 4: (2.0 ** -14, 2.0)}                       # scales between which codes enter as they are


def _rewrite(case, k, v):
    """k, v(b, tokens, first) -> values for cached tokens and the new one, in place of the case's own."""
    for b in range(case.B):
        h = int(case.hist[b])
        if h:
            OA.process_kv(case.cache, case.block_tables[b], case.layer, 0, k(b, h, 0), v(b, h, 0), case.rope, None, None)
        new = v(b, 1, h)
        case.qkv[b, (case.Hq + case.Hkv) * 128:] = new.reshape(-1)


def _dequant64(codes, scale, zero, dtype):
    return codes * scale[:, None].astype(np.float64) + zero[:, None].astype(np.float64)


def _exact(case, b, h, q):
    """(output of query q over the pages, how far a correct one may be off) in 64 bits; OA.kv_dequant is _dequant64."""
    K, V = case.cache.read_tokens(case.block_tables[b], case.layer, h, int(case.hist[b]) + 1)
    s = K @ q / np.sqrt(128.0)
    p = np.exp(s - s.max())
    p /= p.sum()
    o = p @ V
    # weights and, where a tile is de-quantised, values rounded to f16: U of each term; the result rounded to f16; float sums of terms up to twice the
    # largest value (code and zero parts cancel); steps of subnormal results
    return o, 2 * U * (p @ np.abs(V)) + U * np.abs(o) + 2.0 ** -18 * np.abs(V).max() + 2.0 ** -24


def _check(case, monkeypatch):
    q = OA.decode_prologue(case.qkv, None, None, None, case.hist, case.Hq, case.Hkv, 128, case.rope, F16)[0].astype(np.float64)
    out, pool = case.run_device()
    case.run_oracle()                                                       # appends the new tokens to the case's pages
    assert np.array_equal(pool, case.cache.pool)
    monkeypatch.setattr(OA, "kv_dequant", _dequant64)
    got, G = out.reshape(case.B, case.Hq, 128), case.Hq // case.Hkv
    for b in range(case.B):
        for h in range(case.Hkv):
            for g in range(G):
                ref, bar = _exact(case, b, h, q[b, h * G + g])
                err = np.abs(got[b, h * G + g] - ref)
                assert (err <= bar).all(), (b, h, g, float((err / bar).max()))


@pytest.mark.parametrize("kv_bits", [8, 4])
@pytest.mark.parametrize("scale", [1e-4, 2e-2, 1.0, 40.0, 3000.0, "mixed", "constant", 1e-3, 4.0, "min", "max", "offset"])
def test_scales_of_every_size(kv_bits, scale, monkeypatch):
    case = PagedCase(batch_hist=[0, 1, 63, 64, 65, 200, 700], num_heads=8, num_kv_heads=2, kv_bits=kv_bits, seed=5)
    rng = np.random.default_rng(7)

    def keys(b, n, first):
        return rn(rng.standard_normal((n, 2, 128)).astype(np.float32), F16)

    def values(b, n, first):
        tok, offset = first + np.arange(n)[:, None, None], 0.0
        x = rng.standard_normal((n, 2, 128))
        if scale == "mixed":
            f = 10.0 ** rng.integers(-4, 4, (n, 2, 1))
        elif scale == "constant":                                           # half of the vectors are one number throughout
            f, offset = rng.integers(0, 2, (n, 2, 1)), 0.25
        elif scale in ("min", "max"):
            # a warp's 16 keys are four groups of four consecutive tokens, 16 apart: two warps of each tile inside the limit, two outside (128 normal
            # values span about 5.4)
            inside = (tok // 4 % 4 + tok // 64) % 2 == 0
            wide = 1.7 if scale == "min" else 0.6
            f = LIMITS[kv_bits][scale == "max"] * (2 ** kv_bits - 1) / 5.4 * np.where(inside, wide, 1 / wide)
        elif scale == "offset":                                             # ranges of 64 f16 steps at most, far from zero
            f, offset = 2e-3, 0.75
        else:
            f = scale
        return rn((x * f + offset).astype(np.float32), F16)

    _rewrite(case, keys, values)
    _check(case, monkeypatch)


HIST, BATCH = 16384, 256


def _shared_pages(case, lib, qkv):
    """Decode attention of BATCH sequences over the pages of `case` (one sequence of HIST tokens, 4 / 1 heads), each with a last page of its own for its
    new token; qkv [BATCH, 6 * 128] -> outputs [BATCH, 4, 128].  So many tiles that a CTA has whole sequences."""
    import ctypes as C
    import torch
    from lmdeploy_b200 import _lib as L
    from harness import from_dev_T, to_dev_T
    case.upload()
    own = torch.zeros(BATCH, case.cache.block_bytes, dtype=torch.uint8, device="cuda")
    ptrs = case.d_block_ptrs.repeat(BATCH, 1)
    ptrs[:, -1] = own.data_ptr() + torch.arange(BATCH, device="cuda") * case.cache.block_bytes
    cu = torch.arange(BATCH + 1, dtype=torch.int32, device="cuda")
    cu_k, cu_blocks = cu * (HIST + 1), cu * ptrs.shape[1]
    d_qkv, out = to_dev_T(qkv, F16), torch.zeros(BATCH, 4 * 128, dtype=torch.float16, device="cuda")
    ws = torch.zeros(lib.b200_decode_attention_workspace_bytes(BATCH, 4, 1), dtype=torch.uint8, device="cuda")
    p = case.params(lib, workspace=ws)
    p.out, p.q, p.k, p.v = out.data_ptr(), d_qkv.data_ptr(), d_qkv.data_ptr() + 4 * 256, d_qkv.data_ptr() + 5 * 256
    p.cu_q_len, p.cu_k_len, p.block_ptrs, p.cu_block_nums = cu.data_ptr(), cu_k.data_ptr(), ptrs.data_ptr(), cu_blocks.data_ptr()
    p.token_num = p.batch_size = BATCH
    L.check(lib.b200_decode_attention(C.byref(p)), "b200_decode_attention")
    torch.cuda.synchronize()
    return from_dev_T(out, F16).reshape(BATCH, 4, 128)


@pytest.mark.parametrize("kv_bits,gap", [(8, 11.565), (8, 10.9), (4, 11.577), (4, 10.9)])
def test_long_tail_of_small_weights_over_narrow_values(kv_bits, gap, monkeypatch, lib):
    """One key holds most of the weight, 16 384 others exp(-gap) of it each, alike, over values whose scale lies just inside the lower limit: what
    rounding takes from one of them it takes from all."""
    case = PagedCase(batch_hist=[HIST], num_heads=4, num_kv_heads=1, kv_bits=kv_bits, seed=6, rope=OA.RopeParam(type=OA.ROPE_NULL))
    rng = np.random.default_rng(8)
    u = np.where(rng.integers(0, 2, 128) > 0, 1.0, -1.0)
    span = 5 if kv_bits == 8 else 1                                         # steps of 2^-10: scales of 1.9e-5 and 6.5e-5

    def keys(b, n, first):
        k = np.zeros((n, 1, 128), np.float32)
        k[n // 2, 0] = u * gap / np.sqrt(128.0)
        return rn(k, F16)

    def values(b, n, first):
        v = 1.0 + rng.integers(0, span + 1, (n, 1, 128)) * 2.0 ** -10
        if first == 0:
            v[n // 2] -= 2.0
        return rn(v.astype(np.float32), F16)

    _rewrite(case, keys, values)
    case.qkv[0, :4 * 128] = np.tile(u, 4)
    case.qkv[0, 4 * 128:5 * 128] = 0.0                                      # the new token's key: part of the tail
    got = _shared_pages(case, lib, np.repeat(case.qkv, BATCH, 0))
    case.run_oracle()
    monkeypatch.setattr(OA, "kv_dequant", _dequant64)
    ref, _ = _exact(case, 0, 0, u)
    tail = HIST * np.exp(-gap) * 1.01
    # the result rounded to f16; the tail's weights and values (the large weight is one, its scaled form a power of two times an f16 scale: exact); steps of
    # subnormal weights, of all keys that a warp has beside the large one (a CTA has at most 149 tiles, a warp 16 keys of each); values differ by two
    bar = U * np.abs(ref) + 2 * U * tail + 149 * 16 * 2.0 ** -25 * 2 + 2.0 ** -18
    err = np.abs(got - ref)
    assert (err <= bar).all(), float((err / bar).max())


@pytest.mark.parametrize("kv_bits", [8, 4])
def test_long_even_contexts_keep_their_bits(kv_bits, lib):
    """16 384 keys of like weight: the output is a hundredth of a value, so that sums which carried the values' offset would lose it."""
    import torch
    case = PagedCase(batch_hist=[HIST], num_heads=4, num_kv_heads=1, kv_bits=kv_bits, seed=9, rope=OA.RopeParam(type=OA.ROPE_NULL))
    rng = np.random.default_rng(10)
    qkv = rn(rng.standard_normal((BATCH, 6 * 128)).astype(np.float32), F16)
    got = torch.from_numpy(_shared_pages(case, lib, qkv).astype(np.float64))
    keep, OA.kv_dequant = OA.kv_dequant, _dequant64
    try:
        K, V = (torch.from_numpy(x) for x in case.cache.read_tokens(case.block_tables[0], case.layer, 0, HIST))
        new = [OA.PagedKvCache(BATCH, 1, case.layout, F16) for _ in range(1)][0]
        for b in range(BATCH):
            new.write_token(b, 0, 0, 0, qkv[b, 512:640], qkv[b, 640:])
        nk, nv = (torch.from_numpy(np.stack(x)) for x in zip(*[[y[0] for y in new.read_tokens([b], 0, 0, 1)] for b in range(BATCH)]))
    finally:
        OA.kv_dequant = keep
    q = torch.from_numpy(qkv[:, :512].astype(np.float64)).view(BATCH, 4, 128)
    s = torch.cat([q @ K.T, (q * nk[:, None]).sum(-1, keepdim=True)], -1) / np.sqrt(128.0)
    p = s.softmax(-1)
    ref = p[..., :HIST] @ V + p[..., HIST:] * nv[:, None]
    # at most four independent roundings to f16 -- keys (as an error of the weights of up to one score's size), weights, values, result -- each up to U,
    # evenly spread: U / sqrt(3) of the 2-norm
    assert float((got - ref).norm() / ref.norm()) <= U * (4 / 3) ** 0.5

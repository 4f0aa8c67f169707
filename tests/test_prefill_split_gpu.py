"""Prefill attention where its work list is cut: key tiles of 128 at their edges, a few tokens over a long history (many CTAs per piece), empty
tiles, GQA groups that leave rows unused, and the form for callers whose workspace holds the rotated queries alone."""
import numpy as np
import pytest

from oracle.numerics import BF16, F16

from test_prefill_attention_gpu import _prefill_case

pytestmark = pytest.mark.gpu


class _Call:
    """The library with another workspace (`more` bytes beyond the rotated queries, the least that the operator takes; None: all it asks for) and another
    word about the longest context."""

    def __init__(self, lib, more, keys):
        self.lib, self.more, self.keys = lib, more, keys

    def __getattr__(self, name):
        return getattr(self.lib, name)

    def b200_prefill_attention_workspace_bytes(self, tokens, heads):
        return self.lib.b200_prefill_attention_workspace_bytes(tokens, heads) if self.more is None else tokens * heads * 256 + self.more

    def b200_prefill_attention(self, ref):
        ref._obj.max_k_len = self.keys
        return self.lib.b200_prefill_attention(ref)


# shared keys; whole pieces for want of room; whole pieces and the short form for what the caller says of the contexts (not true here: any form is right)
@pytest.mark.parametrize("more,keys", [(None, 0), (0, 0), (20000, 0), (None, 200), (None, 128)])
@pytest.mark.parametrize("kv_bits,dtype,heads,q_lens,hists", [
    (8, F16, (8, 2), [127, 128, 129, 64, 65, 1], [0, 0, 0, 64, 63, 127]),
    (16, F16, (4, 1), [3, 40], [1500, 700]),
    (4, F16, (8, 1), [33, 17, 2], [129, 128, 1000]),
    (16, BF16, (7, 1), [19, 37, 300], [0, 128, 127]),
    (8, BF16, (2, 2), [257, 1], [255, 900]),
])
def test_cut_work_matches_oracle(lib, kv_bits, dtype, heads, q_lens, hists, more, keys):
    got, ref, pool, ref_pool = _prefill_case(_Call(lib, more, keys), q_lens=q_lens, hists=hists, Hq=heads[0], Hkv=heads[1], kv_bits=kv_bits,
                                             dtype=dtype, seed=sum(q_lens))
    assert np.array_equal(pool, ref_pool)
    # P is rounded to T before P.V and the output is rounded to T (half an ulp each, 2^-12 / 2^-9 relative to values up to 4): as for the whole prompts
    bar = 2e-3 if dtype == F16 else 2e-2
    assert np.isfinite(got).all() and np.abs(got - ref).max() <= bar


@pytest.mark.parametrize("dtype", [F16, BF16])
def test_largest_weight_of_a_row_is_exact(lib, dtype):
    """A row's largest score stands in its second key tile, 4.5 to 5.4 above the largest of the first: the weight it gets is one, whatever the tile before
    it had for a maximum, so that the output (that key's value, one, times a normalised weight) is off by its own rounding and little more."""
    import ctypes as C
    import torch
    from lmdeploy_b200 import _lib as L
    from harness import PagedCase, from_dev_T
    from oracle import attention as OA
    from oracle.numerics import rn
    hist, top = 140, 135
    case = PagedCase(batch_hist=[hist] * 64, num_heads=4, num_kv_heads=1, kv_bits=16, dtype=dtype, rope=OA.RopeParam(type=OA.ROPE_NULL))
    u = np.where(np.random.default_rng(1).integers(0, 2, 128) > 0, 1.0, -1.0).astype(np.float32)
    k, v = np.tile(-4.0 * u, (hist, 1, 1)), np.zeros((hist, 1, 128), np.float32)
    k[0], k[top], v[top] = 0.0, 0.5 * u, 1.0
    for table in case.block_tables:
        OA.process_kv(case.cache, table, case.layer, 0, k, v, case.rope, None, None)
    gaps = np.linspace(4.5, 5.4, 256)                                       # score of `top`: u.u * 0.5 * size / sqrt(128)
    size = rn((gaps / (64 / np.sqrt(128.0))).astype(np.float32), dtype)
    case.qkv[:, :512] = (size[:, None] * u).reshape(64, 512)
    case.qkv[:, 512:640], case.qkv[:, 640:] = -4.0 * u, 0.0
    case.upload()
    ws = torch.zeros(64 * 4 * 256, dtype=torch.uint8, device="cuda")        # no partials: one CTA has both tiles
    p = case.params(lib, workspace=ws)
    L.check(lib.b200_prefill_attention(C.byref(p)), "b200_prefill_attention")
    torch.cuda.synchronize()
    got = from_dev_T(case.d_out, dtype).reshape(256, 128).astype(np.float64)
    w = np.exp(-size.astype(np.float64) * 64 / np.sqrt(128.0))              # of key 0; the others' are e^-40
    half = 2.0 ** -12 if dtype == F16 else 2.0 ** -9                        # half a step between 0.5 and 1
    assert (np.abs(got - (1 / (1 + w))[:, None]) <= 1.02 * half + 4 * half * w[:, None]).all()

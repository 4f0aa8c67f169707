"""Prefill attention where its work list is cut: key tiles of 128 at their edges, a few tokens over a long history (many CTAs per piece), empty
tiles, GQA groups that leave rows unused, and the form for callers whose workspace holds the rotated queries alone."""
import numpy as np
import pytest

from oracle.numerics import BF16, F16

from test_prefill_attention_gpu import _prefill_case

pytestmark = pytest.mark.gpu


class _Workspace:
    """The library with a smaller workspace: `more` bytes beyond the rotated queries, the least that the operator takes."""

    def __init__(self, lib, more):
        self.lib, self.more = lib, more

    def __getattr__(self, name):
        return getattr(self.lib, name)

    def b200_prefill_attention_workspace_bytes(self, tokens, heads):
        return tokens * heads * 256 + self.more


@pytest.mark.parametrize("more", [None, 0, 20000])
@pytest.mark.parametrize("kv_bits,dtype,heads,q_lens,hists", [
    (8, F16, (8, 2), [127, 128, 129, 64, 65, 1], [0, 0, 0, 64, 63, 127]),
    (16, F16, (4, 1), [3, 40], [1500, 700]),
    (4, F16, (8, 1), [33, 17, 2], [129, 128, 1000]),
    (16, BF16, (7, 1), [19, 37, 300], [0, 128, 127]),
    (8, BF16, (2, 2), [257, 1], [255, 900]),
])
def test_cut_work_matches_oracle(lib, kv_bits, dtype, heads, q_lens, hists, more):
    got, ref, pool, ref_pool = _prefill_case(lib if more is None else _Workspace(lib, more), q_lens=q_lens, hists=hists, Hq=heads[0], Hkv=heads[1], kv_bits=kv_bits,
                                             dtype=dtype, seed=sum(q_lens))
    assert np.array_equal(pool, ref_pool)
    # P is rounded to T before P.V and the output is rounded to T (half an ulp each, 2^-12 / 2^-9 relative to values up to 4): as for the whole prompts
    bar = 2e-3 if dtype == F16 else 2e-2
    assert np.isfinite(got).all() and np.abs(got - ref).max() <= bar

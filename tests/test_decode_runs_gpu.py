"""Decode attention of a few sequences, whose pieces a CTA per query head merges (decode_reduce_heads_kernel): one piece, a few, sequences without
keys beside long ones; against the numpy oracle."""
import numpy as np
import pytest

from harness import PagedCase

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("heads,kv_heads,kv_bits", [(8, 1, 8), (4, 2, 4), (6, 1, 16)])
@pytest.mark.parametrize("hist", [[0], [63], [64], [127, 0], [200], [64 * 5 + 1], [64 * 18], [64 * 33 + 7, 3, 130]])
def test_few_sequences_match_the_oracle(hist, heads, kv_heads, kv_bits):
    case = PagedCase(batch_hist=hist, num_heads=heads, num_kv_heads=kv_heads, kv_bits=kv_bits, seed=len(hist) + sum(hist))
    out, pool = case.run_device()
    ref = case.run_oracle()
    assert (pool == case.cache.pool).all()
    # probabilities rounded to f16 (2^-11 each) and the output's own rounding, on values up to about one
    assert float(np.abs(out - ref).max()) <= 2e-3

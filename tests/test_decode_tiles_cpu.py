"""What the bars of the tests of decode attention over tiles can see: outputs made on the CPU in the kernel's arithmetic (weights and results rounded to T) stay below
them, and the same with a fault of a tile in them does not, for every dtype and pattern of values."""
import numpy as np
import pytest

from oracle.numerics import BF16, F16, rn

from test_decode_tiles_gpu import ODD, Exact, pages


def _tile(i):
    return slice(64 * i, 64 * i + 64)


def _out(exact, b, fault):
    p, _ = exact.weights(b)
    P, V = p / p.max(-1, keepdims=True), exact.kv[b][1].copy()
    taken = np.ones(len(V))
    if fault == "a tile left out":
        taken[_tile(20)] = 0
    elif fault == "a tile taken twice":
        taken[_tile(20)] = 2
    elif fault == "fifteen tiles not rescaled":
        taken[64 * 5:64 * 20] = 2
    elif fault == "another tile's values":
        V[_tile(20)], V[_tile(21)] = V[_tile(21)].copy(), V[_tile(20)].copy()
    # in f16 a weight is rounded with its value's scale, which is no power of two: as far off as T's rounding of the weight itself
    return rn(((rn(P.astype(np.float32), exact.dtype) * taken) @ V / (P * taken).sum(-1, keepdims=True)).astype(np.float32), exact.dtype)


@pytest.mark.parametrize("dtype", [F16, BF16])
@pytest.mark.parametrize("odd", ODD)
def test_faults_of_a_tile_exceed_the_bars(dtype, odd):
    case, qkv = pages(4031, 64, 4, dtype, odd)
    exact = Exact(case, qkv[::20], 4)
    exact.check(lambda b: _out(exact, b, None), 1)
    for fault in ("a tile left out", "a tile taken twice", "fifteen tiles not rescaled", "another tile's values"):
        with pytest.raises(AssertionError):
            exact.check(lambda b: _out(exact, b, fault), 1)

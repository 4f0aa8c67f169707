"""Which kernel a linear layer's call runs (host logic, no GPU)."""
import ctypes as C

import pytest

from lmdeploy_b200 import _lib as L

TILES, FEW, HEAD = range(3)


def kernel(lib, K, N, fmt, m, packed=0, dtype=0, prepared=None):
    return lib.b200_linear_kernel(C.byref(L.LinearDesc(K, N, fmt, dtype, 128, prepared, None)), m, packed)


@pytest.fixture
def plans(lib, tmp_path):
    """load(lines) -> replaces the plan table; the table is empty before and after."""
    lib.b200_linear_load_plans(None)

    def load(*lines):
        f = tmp_path / "plans.txt"
        f.write_text("\n".join(lines) + "\n")
        assert lib.b200_linear_load_plans(str(f).encode()) == len(lines)

    yield load
    lib.b200_linear_load_plans(None)


@pytest.mark.parametrize("packed", [0, 1])
@pytest.mark.parametrize("m,mt", [(65, 80), (128, 128)])
def test_a_plan_selects_the_kernel_it_was_measured_on_for_heads(lib, plans, m, mt, packed):
    K, N = 4096, 92544
    assert kernel(lib, K, N, L.FMT_DENSE, m, packed) == HEAD
    plans(f"PLAN 0 {mt} {N} {K} 1 1 0 0")
    assert kernel(lib, K, N, L.FMT_DENSE, m, packed) == TILES
    assert kernel(lib, K + 128, N, L.FMT_DENSE, m, packed) == HEAD           # another shape


def test_a_plan_selects_the_kernel_it_was_measured_on_for_few_tokens(lib, plans):
    assert kernel(lib, 4096, 6144, L.FMT_U4, 16) == FEW
    plans("PLAN 1 16 6144 4096 1 2 0 0")
    assert kernel(lib, 4096, 6144, L.FMT_U4, 16) == kernel(lib, 4096, 6144, L.FMT_U4, 1) == TILES
    assert kernel(lib, 4096, 6144, L.FMT_U4, 17) == FEW                       # 32 padded tokens: no plan


def test_who_reads_packed_activations_or_unaligned_weights(lib, plans):
    assert kernel(lib, 4096, 6144, L.FMT_U4, 1, packed=1) == TILES
    assert kernel(lib, 4096, 6144, L.FMT_FP8, 1) == TILES
    assert kernel(lib, 4096, 6144, L.FMT_U4, 1, prepared=1 << 20) == FEW
    assert kernel(lib, 4096, 6144, L.FMT_U4, 1, prepared=(1 << 20) + 16) == TILES
    assert kernel(lib, 4096, 6144, L.FMT_U4, 25) == TILES
    assert kernel(lib, 4096, 6144, 7, 1) == L.ERR_UNSUPPORTED and kernel(lib, 4096, 6144, L.FMT_U4, 129) == L.ERR_INVALID_ARG


# both sides of the lines between the kernels: (format, dtype, m, K, N, who was faster there)
@pytest.mark.parametrize("fmt,dtype,m,K,N,want", [
    (1, 0, 1, 4096, 6144, FEW), (1, 0, 8, 14336, 1024, FEW), (1, 0, 8, 4096, 22016, TILES), (1, 0, 9, 8192, 4096, FEW), (1, 0, 16, 14336, 1024, TILES),
    (1, 0, 16, 1024, 32768, TILES), (1, 0, 24, 4096, 6144, FEW), (1, 0, 24, 6144, 4096, TILES), (1, 1, 24, 8192, 1024, TILES),
    (3, 0, 8, 4096, 32000, FEW), (3, 1, 8, 4096, 22016, TILES), (3, 1, 8, 8192, 10240, FEW), (3, 1, 16, 4096, 14336, FEW), (3, 1, 16, 1024, 32768, TILES),
    (3, 0, 24, 4096, 8192, FEW), (3, 1, 24, 8192, 1024, TILES),
    (0, 0, 1, 4096, 32000, FEW), (0, 0, 8, 4096, 46336, TILES), (0, 0, 8, 14336, 1024, TILES), (0, 0, 8, 14336, 4096, FEW), (0, 0, 16, 4096, 4096, FEW), (0, 0, 16, 5120, 5120, TILES),
    (0, 1, 16, 8192, 1024, TILES), (0, 0, 24, 4096, 4096, FEW), (0, 0, 24, 4096, 1024, TILES), (0, 1, 24, 8192, 2048, TILES)])
def test_calls_go_to_the_faster_kernel(lib, plans, fmt, dtype, m, K, N, want):
    assert kernel(lib, K, N, fmt, m, dtype=dtype) == want

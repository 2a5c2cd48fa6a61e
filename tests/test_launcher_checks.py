"""Arguments that a kernel could not handle are refused by the launchers before anything is launched, so these calls need no GPU."""
import ctypes

import pytest

from dlslime_b200 import _lib

A, B, OUT, OFFS = 1 << 20, 2 << 20, 3 << 20, 4 << 20  # addresses that nothing dereferences
M, N, K = 300, 2048, 512

PLAIN = ["slime_gemm_bf16", "slime_gemm_bf16_pair", "slime_gemm_bf16_wide"]
GROUPED = ["slime_grouped_gemm_bf16", "slime_grouped_gemm_bf16_pair", "slime_grouped_gemm_bf16_wide", "slime_grouped_gemm_bf16_swapped"]


def _refused(name, *args):
    if not _lib.available():
        pytest.skip("kernel library not built")
    with pytest.raises(_lib.SlimeCudaError, match="aligned"):
        _lib.call(name, *args)


@pytest.mark.parametrize("shift", [2, 4])
@pytest.mark.parametrize("name", PLAIN)
def test_plain_products_refuse_an_output_between_two_vectors(name, shift):
    _refused(name, A, B, OUT + shift, M, N, K, K, K, N, None, None)


@pytest.mark.parametrize("shift", [2, 4])
def test_fp8_product_refuses_an_output_between_two_vectors(shift):
    import dlslime_b200.ops.gemm  # noqa: F401 (declares the launcher)

    _refused("slime_gemm_fp8_blockscaled", A, A, B, B, OUT + shift, M, N, K, K, K, N, None, None)


@pytest.mark.parametrize("ldc,shift", [(N, 4), (N + 1, 0), (N, 2)])
@pytest.mark.parametrize("name", GROUPED)
@pytest.mark.parametrize("epilogue", [0, 1])
def test_grouped_products_refuse_rows_between_two_vectors(name, epilogue, ldc, shift):
    bases = (ctypes.c_ulonglong * 8)()
    _refused(name, A, B, OUT + shift, OFFS, 4, M, N, K, K, K, ldc, epilogue, None, bases, 0, 0, None, None, None)

"""How the few-token tensor-core product is cut (host code, no device needed)."""
import ctypes

import pytest


@pytest.mark.parametrize("mode", [0, 2])
@pytest.mark.parametrize("sms", [16, 132, 148, 1000])
def test_a_partial_tile_fits_where_the_stages_lay(mode, sms):
    """With K split a block's 32-bit partial tile lies over its stages; behind them are the barriers and the rows' scales."""
    from torchless_rs_b200.csrc import build, gemm_bf16  # noqa: F401  (registers the library)
    lib = build.load_library("gemm_tc")
    split = set()
    for M in (1, 16, 17, 32, 33, 64, 65, 128, 129, 200, 256, 257, 600):
        for N in (8, 128, 200, 1024, 4096, 6144, 14336):
            for K in (64, 512, 1024, 4096, 14336):
                bn, splits, partial, room = (ctypes.c_int() for _ in range(4))
                lib.tl_gemm_tc_plan(M, N, K, mode, sms, *(ctypes.byref(x) for x in (bn, splits, partial, room)))
                assert bn.value in (16, 32, 64, 128, 256) and splits.value >= 1
                assert partial.value == (splits.value > 1) * (2 if mode == 2 else 1) * bn.value * 128 * 4
                assert partial.value <= room.value, (M, N, K, splits.value)
                split |= {bn.value} if splits.value > 1 else set()
    if sms >= 132:      # the sweep reaches splits of every tile that has room for them
        assert split == {16, 32, 64, 128} | ({256} if mode == 0 else set())


def test_32_bit_products_on_tensor_cores_go_by_rows_and_sizes_in_order():
    """More rows, columns or longer sums never send a 32-bit product back to the CUDA cores, and both sides of the line at K = 3072."""
    from torchless_rs_b200.csrc.gemm_f32 import GemmF32
    takes, sizes = GemmF32.takes, (64, 255, 341, 342, 512, 1024, 2048, 3071, 3072, 4095, 4096, 4736, 6144, 14336)
    for M in (1, 3, 4, 5, 8, 9, 100):
        for N in sizes:
            for K in sizes:
                if takes(M, N, K):
                    assert takes(M + 1, N, K) and takes(M, N + 1, K) and takes(M, N, K + 1), (M, N, K)
    for M in (4, 5, 8):
        assert takes(M, 1024, 4096) and takes(M, 512, 3072) and takes(M, 4096, 4032) and takes(M, 342, 3072)
        assert not takes(M, 341, 3072) and not takes(M, 1024, 3071) and not takes(M, 255, 4096)
    assert not takes(4, 4736, 2560) and takes(5, 4736, 2560) and not takes(3, 4096, 4096)

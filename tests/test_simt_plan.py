"""How the float32 product lays out its tiles (csrc/gemm_simt.cu; no GPU needed)."""
import ctypes

import pytest

from coheryn_ai_studio_b200 import ops


def plan(M, N, K):
    out = [ctypes.c_int() for _ in range(3)]
    ops.core().coheryn_gemm_simt_plan(ctypes.c_int(M), ctypes.c_int(N), ctypes.c_int(K), *[ctypes.byref(o) for o in out])
    return tuple(o.value for o in out)


# us measured on a B200 with tiles of 64 x 128 and of 16 x 64
@pytest.mark.parametrize("M,N,K,large,small", [
    (64, 16, 16, 7.6, 4.1), (2048, 64, 64, 10.7, 4.4), (64, 256, 128, 15.5, 5.9), (17, 3584, 512, 38.0, 16.7), (400, 512, 512, 41.3, 23.7),
    (33, 1536, 1536, 40.2, 25.7), (130, 1536, 1536, 42.4, 62.7), (700, 1000, 256, 24.7, 39.6), (200, 8960, 1536, 187, 399), (1300, 1536, 8960, 808, 2223)])
def test_the_faster_tile_is_taken(M, N, K, large, small):
    rows, columns, apart = plan(M, N, K)
    assert (rows, columns) == ((64, 128) if large < small else (16, 64))
    tiles = -(-M // rows) * -(-N // columns)
    assert apart == 1 or (apart > 1 and tiles < 296)


@pytest.mark.parametrize("M,N,K", [(640, 3584, 18944), (300, 3584, 18944), (1100, 1536, 8960), (200, 4095, 30000), (16, 3584, 18944), (1, 100, 1000000)])
def test_the_workspace_is_bounded(M, N, K):
    """64 MB, or the sums of one row tile: an eighth of a float32 weight's bytes (the last stretch may be short)."""
    lib = ops.core()
    floats = int(lib.coheryn_gemm_simt_workspace_floats(ctypes.c_int(M), ctypes.c_int(N), ctypes.c_int(K)))
    assert plan(M, N, K)[2] > 1 and 0 < floats <= max(1 << 24, N * (K + 512) // 8)

"""What the float32 product on the tensor cores asks for (csrc/gemm_f32_tc.cu; no GPU needed)."""
import pytest

from coheryn_ai_studio_b200 import ops


@pytest.mark.parametrize("M,N,K,act", [(2048, 17920, 1536, 0), (2048, 17920, 1536, 16), (2048, 1536, 8960, 0), (700, 1536, 8960, 16), (5000, 256, 4096, 0),
                                       (1, 151936, 1536, 0), (3000, 151936, 1536, 0), (3000, 151936, 1536, 16), (1500, 3584, 18944, 0), (640, 128, 100000, 0)])
def test_the_workspace_is_bounded(M, N, K, act):
    """128 MB, or what one tile of 160 rows needs (its terms; its results, where they wait for the activation or for other slices of k)."""
    floats = ops._f32_tc_workspace_floats(M, N, K, act)
    slices = max(1, round(148 / -(-N // 128)))
    assert 0 < floats <= max(1 << 25, 160 * (2 * K + slices * N)) + 64


# us measured on a B200 by this kernel and by the FMA kernel, the worst of 1 to 1,500 rows
@pytest.mark.parametrize("N,K,tc,fma", [(128, 256, 13.6, 9.1), (1024, 256, 11.9, 9.1), (256, 448, 18.2, 14.2), (512, 384, 14.7, 12.5), (4096, 256, 8.4, 8.7),
                                        (20000, 256, 15.0, 16.8), (256, 512, 15.5, 16.0), (128, 768, 15.8, 17.4), (1536, 1536, 17, 30), (17920, 1536, 38, 84)])
def test_the_faster_product_is_taken(N, K, tc, fma):
    from ctypes import c_int
    assert bool(ops.core().coheryn_gemm_f32_tc_pays(c_int(N), c_int(K))) == (tc < fma)

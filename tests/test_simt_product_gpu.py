"""The float32 product on the CUDA cores (csrc/gemm_simt.cu) at the edges of its tiles, of its stretches of k and of aligned
loads, against float64; and rows that do not depend on the other rows, bit for bit."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def product(x, w, bias, out_dtype, act=0):
    from coheryn_ai_studio_b200 import ops
    out = torch.full((x.shape[0], w.shape[0] + 3), float("nan"), dtype=out_dtype, device=DEV)[:, :w.shape[0]]
    ops.gemm_simt(x, w, bias, out, act)
    return out


@pytest.mark.parametrize("M,N,K,pad", [(1, 1, 1, 0), (16, 128, 512, 0), (17, 127, 513, 0), (64, 130, 511, 3), (65, 300, 1100, 0), (3, 257, 1540, 4),
                                       (200, 129, 36, 1), (130, 3000, 1025, 0), (70, 4100, 2052, 0)])
@pytest.mark.parametrize("kinds", ["fff", "fbf", "bbf", "bbb"])
def test_product_at_the_edges(M, N, K, pad, kinds):
    kind = {"f": torch.float32, "b": torch.bfloat16}
    g = torch.Generator(device=DEV).manual_seed(M + N + K)
    x = torch.randn((M, K + pad), device=DEV, generator=g).to(kind[kinds[0]])[:, pad:]
    w = torch.randn((N, K), device=DEV, generator=g).to(kind[kinds[1]])
    bias = torch.randn((N,), device=DEV, generator=g)
    got = product(x, w, bias, kind[kinds[2]]).double()
    want, size = x.double() @ w.double().T + bias.double(), x.double().abs() @ w.double().abs().T + bias.double().abs()
    # every term, every sum and the bias are rounded once: (K + 2) 2^-24 of the terms' size at most; a bfloat16 result is
    # rounded once more
    bound = size * (K + 2) * 2.0 ** -24 + (want.abs() * 2.0 ** -8 if kinds[2] == "b" else 0.0)
    assert bool(((got - want).abs() <= bound).all())


@pytest.mark.parametrize("N,K", [(200, 1600), (5000, 700), (4100, 2100)])
def test_a_row_does_not_depend_on_the_other_rows(N, K):
    g = torch.Generator(device=DEV).manual_seed(N)
    x, w = torch.randn((700, K), device=DEV, generator=g), torch.randn((N, K), device=DEV, generator=g)
    whole = product(x, w, None, torch.float32)
    for at, n in ((0, 1), (5, 16), (100, 17), (300, 400)):
        assert torch.equal(product(x[at:at + n], w, None, torch.float32), whole[at:at + n]), (at, n)


@pytest.mark.parametrize("M,rows,cols,N,K", [(5, 130, 24, 300, 48), (70, 256, 64, 512, 128), (65, 1, 3, 400, 10), (33, 128, 100, 200, 700)])
def test_block_diagonal_weight(M, rows, cols, N, K):
    """Leaving the zero blocks out changes no bit."""
    from coheryn_ai_studio_b200 import ops
    g = torch.Generator(device=DEV).manual_seed(N)
    x, w = torch.randn((M, K), device=DEV, generator=g), torch.randn((N, K), device=DEV, generator=g)
    w[:rows, cols:] = 0.0
    w[rows:, :cols] = 0.0
    out = torch.empty((M, N), device=DEV)
    ops.gemm_simt(x, w, None, out, blocks=(rows, cols))
    assert torch.equal(out, product(x, w, None, torch.float32))


# Small products in tiles of 16 x 64 (one and many of them across and down, a rest in each direction), sums of at most 32 values.
@pytest.mark.parametrize("M,N,K,pad", [(33, 65, 64, 0), (100, 64, 33, 2), (129, 300, 100, 0), (300, 200, 130, 0), (17, 130, 1030, 1), (500, 63, 32, 0),
                                       (40, 100, 30, 0), (1, 20, 5, 3)])
@pytest.mark.parametrize("kinds", ["fff", "fbf", "bbf", "bbb"])
def test_small_products(M, N, K, pad, kinds):
    test_product_at_the_edges(M, N, K, pad, kinds)


def test_rows_in_several_blocks_of_the_workspace():
    """330 rows whose 37 stretches' sums take the workspace in blocks of 64 and of 192 rows: the bits of the same rows by themselves."""
    g = torch.Generator(device=DEV).manual_seed(1)
    for N, K, kinds in ((3584, 18944, torch.bfloat16), (1800, 18900, torch.float32)):
        x, w = torch.randn((330, K), device=DEV, generator=g), (torch.randn((N, K), device=DEV, generator=g) * 0.1).to(kinds)
        whole = product(x, w, None, torch.float32)
        for at, n in ((0, 64), (60, 10), (127, 1), (200, 130)):
            assert torch.equal(product(x[at:at + n], w, None, torch.float32), whole[at:at + n]), (N, at, n)
        want = x[300:].double() @ w.double().T
        assert float((whole[300:].double() - want).norm() / want.norm()) <= 2e-6      # float32 sums of this length are near 1e-7


# One CTA over several stretches of k (a wide weight): both tiles, with aligned and with unaligned rows.
@pytest.mark.parametrize("M,N,K,pad", [(600, 4100, 2052, 0), (600, 4100, 2051, 1), (16, 19000, 2052, 4), (5, 18945, 4101, 0)])
@pytest.mark.parametrize("kinds", ["fff", "fbf", "bbf", "bbb"])
def test_several_stretches_per_cta(M, N, K, pad, kinds):
    from coheryn_ai_studio_b200 import ops
    assert ops._simt_workspace_floats(M, N, K) == 0
    test_product_at_the_edges(M, N, K, pad, kinds)

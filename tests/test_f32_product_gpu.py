"""The float32 product on the tensor cores (csrc/gemm_f32_tc.cu) at the edges of its tiles of features and tokens, of its stages and slices of
k, against float64 and the FMA product; rows that do not depend on the other rows; values that are not finite; and which weights it takes."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def product(x, w, bias=None, act=0):
    from coheryn_ai_studio_b200 import ops
    out = torch.full((x.shape[0], w.shape[0] + 3), float("nan"), device=DEV)[:, :w.shape[0]]
    assert ops._f32_tc_workspace_floats(x.shape[0], w.shape[0], w.shape[1], act) > 0
    ops.gemm_f32_tc(x, w, bias, out, act)
    return out


def operands(M, N, K, pad=0):
    g = torch.Generator(device=DEV).manual_seed(M + N + K)
    x = torch.randn((M, K + pad), device=DEV, generator=g)[:, pad:]
    return x, torch.randn((N, K), device=DEV, generator=g), torch.randn((N,), device=DEV, generator=g)


@pytest.mark.parametrize("M,N,K,pad", [(1, 128, 256, 0), (16, 129, 260, 1), (17, 200, 316, 0), (33, 255, 320, 3), (65, 1000, 324, 0), (96, 130, 1540, 4),
                                       (128, 257, 576, 0), (161, 3000, 1028, 0), (320, 128, 4096, 0), (150, 12928, 256, 0), (700, 1536, 4100, 0)])
@pytest.mark.parametrize("act", [0, 16])
def test_product_at_the_edges(M, N, K, pad, act):
    x, w, bias = operands(M, N, K, pad)
    got = product(x, w, bias, act).double()
    want, size = x.double() @ w.double().T + bias.double(), x.double().abs() @ w.double().abs().T + bias.double().abs()
    # The terms left out are below 2^-24 of a product; 64 products are added to four large sums and about twenty small ones, cut at 24 bits;
    # the sums of K / 64 stages, of the slices and the bias are rounded once each: well inside (K + 2) 2^-24 of the terms' size, K >= 256
    bound = size * (K + 2) * 2.0 ** -24
    if act:      # GELU's slope stays below 1.13; its own error functions are good to a few units in the last place
        want = torch.nn.functional.gelu(want)
        bound = 1.13 * bound + (size + 1.0) * 2.0 ** -20
    assert bool(((got - want).abs() <= bound).all())


def test_closer_to_float64_than_the_fma_product():
    from coheryn_ai_studio_b200 import ops
    for M, N, K in ((96, 1536, 8960), (40, 17920, 1536), (64, 256, 256)):
        x, w, _ = operands(M, N, K)
        want, fma = x.double() @ w.double().T, torch.empty((M, N), device=DEV)
        ops.gemm_simt(x, w, None, fma)
        assert float((product(x, w).double() - want).norm()) <= float((fma.double() - want).norm())


@pytest.mark.parametrize("N,K", [(200, 1600), (13000, 700), (4100, 2100)])
def test_a_row_does_not_depend_on_the_other_rows(N, K):
    x, w, _ = operands(700, N, K)
    whole = product(x, w)
    for at, n in ((0, 1), (5, 16), (100, 17), (50, 64), (50, 90), (50, 128), (300, 150), (300, 400)):
        assert torch.equal(product(x[at:at + n], w), whole[at:at + n]), (at, n)


def test_rows_in_several_blocks_of_the_workspace():
    x, w, _ = operands(1500, 3584, 18944)
    whole = product(x, w)
    for at, n in ((0, 160), (600, 200), (1340, 160)):
        assert torch.equal(product(x[at:at + n], w), whole[at:at + n]), at


@pytest.mark.parametrize("M", [20, 170])
@pytest.mark.parametrize("N", [300, 12900])
def test_values_that_are_not_finite(M, N):
    """Infinities, NaN and numbers whose nearest bfloat16 is infinite give what the FMA product gives."""
    from coheryn_ai_studio_b200 import ops
    x, w, bias = operands(M, N, 772)
    x[3, 7], x[5, 9], x[6, 1], x[7, 0], x[9, 771] = float("inf"), float("nan"), 3.4e38, -float("inf"), -3.4e38
    w[10, 3], w[11, 7], w[131] = -float("inf"), 0.0, 0.0
    got, want = product(x, w, bias), torch.empty((M, N), device=DEV)
    ops.gemm_simt(x, w, bias, want)
    assert torch.equal(got.isnan(), want.isnan())
    assert bool(((got == want) | want.isnan() | ((got - want).abs() <= 1e-4 * (1.0 + want.abs()))).all())


@pytest.mark.parametrize("M,N,K", [(24, 256, 512), (90, 300, 324), (170, 13000, 260), (20, 1536, 2304)])
@pytest.mark.parametrize("ex,ew", [(-100, 0), (-108, 20), (-114, 100), (0, -118), (-124, 120), (118, -135), (-140, 100), (-70, -60)])
def test_operands_under_the_terms_range(M, N, K, ex, ew):
    """Bits that lie under the terms' smallest number count where the other operand is large: the error is the FMA product's at most, and
    a few units of float32's own smallest number where the results come down to it."""
    from coheryn_ai_studio_b200 import ops
    x, w, bias = operands(M, N, K)
    x, w = (x.double() * 2.0 ** ex).float(), (w.double() * 2.0 ** ew).float()
    want, fma, got = x.double() @ w.double().T, torch.empty((M, N), device=DEV), product(x, w)
    ops.gemm_simt(x, w, None, fma)
    error, room = float((got.double() - want).norm()), K * 2.0 ** -149 * (M * N) ** 0.5      # one unit for every value of k
    assert error <= max(float((fma.double() - want).norm()), room)
    # the same beside operands of ordinary size: in some rows, in some features, at some k
    small, x, w = (x, w), torch.randn(M, K, device=DEV), torch.randn(N, K, device=DEV)
    x[::3], w[::5], x[:, ::7], w[:, 1::7] = small[0][::3], small[1][::5], small[0][:, ::7], small[1][:, 1::7]
    want, got = x.double() @ w.double().T, product(x, w, bias).double() - bias.double()
    size = x.double().abs() @ w.double().abs().T + bias.double().abs()
    assert bool(((got - want).abs() <= (K + 2) * 2.0 ** -24 * size + K * 2.0 ** -149).all())


def test_a_weight_that_the_kernel_before_writes():
    """The weight is fetched ahead, but not ahead of the kernel in front that is still writing it (and lets its successors start early)."""
    from coheryn_ai_studio_b200 import ops
    N, K = 12928, 1536
    x, gate_up, _ = operands(24, N, 2 * K)
    x, w, want = x[:, :K].contiguous(), torch.empty((N, K), device=DEV), torch.empty((N, K), device=DEV)
    code = ops.gated_epilogue_word("silu", None)
    ops.silu_mul(gate_up, want, code, 0.0)
    torch.cuda.synchronize()
    want = product(x, want)
    torch.cuda.synchronize()
    for _ in range(10):
        w.zero_()
        ops.silu_mul(gate_up, w, code, 0.0)
        assert torch.equal(product(x, w), want)


def test_which_products_it_takes():
    from coheryn_ai_studio_b200 import ops
    for M, N, K, taken in ((1, 128, 256, True), (5, 127, 256, False), (5, 128, 255, False), (5, 128, 252, False), (2000, 4000, 258, False)):
        assert (ops._f32_tc_workspace_floats(M, N, K, 0) > 0) == taken
    # an unaligned weight and mixed types go to the FMA product
    x, w, _ = operands(9, 300, 512)
    odd = torch.empty((300 * 512 + 1,), device=DEV)[1:].view(300, 512).copy_(w)
    out, want = torch.empty((9, 300), device=DEV), torch.empty((9, 300), device=DEV)
    ops.gemm_f32(x, odd, None, out)
    ops.gemm_simt(x, w, None, want)
    assert torch.equal(out, want)
    ops.gemm_f32(x, w.bfloat16(), None, out)
    ops.gemm_simt(x, w.bfloat16(), None, want)
    assert torch.equal(out, want)

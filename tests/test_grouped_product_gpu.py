"""The routed products by pairs of CTAs (csrc/gemm_tc.cu, gemm_tc_grouped_kernel) for groups of no, one and many rows, at the edges
of its row tiles and feature tiles, against float64."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("counts", [[0, 1, 31, 32, 33, 0], [255, 256, 257], [270, 0, 513, 600, 3], [2400], [64] * 40, [0, 0, 700]])
@pytest.mark.parametrize("N,K,gated,out_dtype", [(512, 256, True, torch.bfloat16), (256, 72, False, torch.float32), (300, 64, False, torch.bfloat16),
                                                 (130, 520, True, torch.float32), (40, 8, False, torch.float32), (2048, 1024, True, torch.bfloat16)])
def test_rows_of_groups(counts, N, K, gated, out_dtype):
    from coheryn_ai_studio_b200 import ops
    E = len(counts)
    g = torch.Generator(device=DEV).manual_seed(N + K + E)
    ids = torch.cat([torch.full((c,), e) for e, c in enumerate(counts)] + [torch.full((5,), E)])      # and some of no group
    ids = ids[torch.randperm(len(ids), generator=torch.Generator().manual_seed(1))].to(torch.int32).to(DEV)[:, None].contiguous()
    rows = ops.route_sort(ids, E, wide_tiles=True)
    x = torch.randn((len(ids), K), device=DEV, generator=g).to(torch.bfloat16)
    w = (torch.randn((E, N, K), device=DEV, generator=g) * K ** -0.5).to(torch.bfloat16)
    out = torch.full((len(ids), N // 2 if gated else N), 7.0, dtype=out_dtype, device=DEV)
    ops.gemm_bf16_tc_grouped(x, w, out, rows, ops.gated_epilogue_word("silu", None) if gated else 0)
    ops.check_tc_status(x.device)
    at = 0
    for e, c in enumerate(counts):
        y = x[at:at + c].double() @ w[e].double().T
        if gated:
            y = y[:, 0::2] * torch.sigmoid(y[:, 0::2]) * y[:, 1::2]
        # float32 sums of K products (2^-24 each, generously 1e-5 of unit-sized results), the gate's exponential, one rounding
        bound = 1e-4 + y.abs() * (2.0 ** -8 if out_dtype == torch.bfloat16 else 1e-5)
        assert bool(((out[at:at + c].double() - y).abs() <= bound).all()), e
        at += c
    assert bool((out[at:] == 7.0).all())

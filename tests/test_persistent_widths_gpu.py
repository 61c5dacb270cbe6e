"""The many-rows product's persistent kernel at each width of its tiles (csrc/gemm_tc.cu, persistent_width), with a rest in rows, columns
and k, plain and gated, against float64."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("M,N,width", [(1100, 4864, 160), (1090, 4730, 160), (1873, 3584, 192), (2048, 4740, 192), (1560, 4620, 224), (1537, 4490, 224),
                                       (1280, 7400, 256), (130, 37700, 256)])
@pytest.mark.parametrize("gated", [False, True])
def test_every_width(M, N, width, gated):
    from coheryn_ai_studio_b200 import ops
    assert int(ops.core().coheryn_gemm_tc_persistent_width(ctypes.c_int(M), ctypes.c_int(N))) == width
    K = 200
    g = torch.Generator(device=DEV).manual_seed(M + N)
    x = torch.randn((M, K), device=DEV, generator=g).to(torch.bfloat16)
    w = (torch.randn((N, K), device=DEV, generator=g) * K ** -0.5).to(torch.bfloat16)
    b = torch.randn((N,), device=DEV, generator=g)
    y = x.double() @ w.double().T
    if gated:
        y = y[:, 0::2] * torch.sigmoid(y[:, 0::2]) * y[:, 1::2]
    else:
        y = y + b.double()
    for dtype in (torch.bfloat16, torch.float32):
        out = torch.full((M + 1, y.shape[1]), 7.0, dtype=dtype, device=DEV)
        ops.set_gemm_pairs(False)
        try:
            ops.gemm_bf16_tc(x, w, None if gated else b, out[:M], gated=gated)
        finally:
            ops.set_gemm_pairs(True)
        ops.check_tc_status(x.device)
        # float32 sums of K products of unit-sized results, the gate's exponential, one rounding
        bound = 1e-4 + y.abs() * (2.0 ** -8 if dtype == torch.bfloat16 else 1e-5)
        assert bool(((out[:M].double() - y).abs() <= bound).all())
        assert bool((out[M:] == 7.0).all())

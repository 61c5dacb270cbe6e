"""The any-shape attention (csrc/attention_simple.cu) with the heads of a group in one block: every number of heads per block, both
register widths, shapes that go key by key, windows, slopes; and rows that do not depend on how many rows a call has, bit for bit."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def problem(T, before, nh, nkv, hd, hdv, dtype, page, shift=0):
    g = torch.Generator(device=DEV).manual_seed(T + nh + hd)
    pages = -(-(T + before) // page)
    order = torch.randperm(pages, generator=g, device=DEV).int()

    def pool(d):      # `shift` elements off an aligned address
        return torch.randn((pages * nkv * page * d + shift,), device=DEV, generator=g).to(dtype)[shift:].view(pages, nkv, page, d)
    k, v = pool(hd), pool(hdv)
    return torch.randn((T, nh * hd), device=DEV, generator=g).to(dtype), k, v, order[None].contiguous(), torch.arange(before, before + T, dtype=torch.int32, device=DEV)


def attend(q, k, v, table, pos, nh, nkv, hd, hdv, page, window, slopes):
    from coheryn_ai_studio_b200 import ops
    out = torch.full((q.shape[0], nh * hdv), float("nan"), dtype=q.dtype, device=DEV)
    ops.attention_simple(q, out, k, v, table, torch.zeros(q.shape[0], dtype=torch.int32, device=DEV), pos, nh, nkv, hd, page, window, hd ** -0.5,
                         v_head_dim=hdv, slopes=slopes, out_scale=1.25)
    return out


def exact(q, k, v, table, pos, nh, nkv, hd, hdv, window, slopes):
    K, V = (t[table[0].long()].transpose(1, 2).reshape(-1, nkv, t.shape[3]).double() for t in (k, v))
    s = torch.einsum("tghd,sgd->ghts", q.double().view(-1, nkv, nh // nkv, hd), K) * hd ** -0.5
    far = (pos[:, None] - torch.arange(K.shape[0], device=DEV)[None]).double()
    if slopes is not None:
        s = s - slopes.double().view(nkv, nh // nkv, 1, 1) * far
    seen = (far >= 0) & (far < (window or 1 << 30))
    return 1.25 * torch.einsum("ghts,sgd->tghd", torch.softmax(s.masked_fill(~seen, -1e300), -1), V).reshape(q.shape[0], -1)


@pytest.mark.parametrize("nh,nkv,hd,hdv", [(4, 4, 128, 128), (6, 3, 64, 32), (6, 2, 128, 128), (8, 2, 100, 60), (10, 2, 80, 80), (12, 2, 128, 128), (7, 1, 128, 64),
                                           (16, 2, 128, 128), (22, 2, 16, 16), (8, 2, 256, 256), (6, 2, 132, 128), (4, 2, 200, 256), (9, 3, 30, 30)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("T,before,window,shift", [(1, 0, None, 0), (3, 33, 20, 0), (160, 0, None, 0), (600, 0, 37, 0), (90, 300, None, 1)])
def test_against_float64(nh, nkv, hd, hdv, dtype, T, before, window, shift):
    q, k, v, table, pos = problem(T, before, nh, nkv, hd, hdv, dtype, 16, shift)
    slopes = torch.linspace(0.0, 0.3, nh, device=DEV) if window is None and T > 1 else None
    args = (q, k, v, table, pos, nh, nkv, hd, hdv)
    got, want = attend(*args, 16, window, slopes).double(), exact(*args, window, slopes)
    # sums of at most 700 float32 terms; bfloat16 results are rounded once
    assert float((got - want).norm() / want.norm()) <= (2e-6 if dtype == torch.float32 else 3e-3)


@pytest.mark.parametrize("nh,nkv,hd", [(12, 2, 128), (28, 4, 128), (8, 1, 64), (8, 2, 192)])
def test_a_row_does_not_depend_on_the_other_rows(nh, nkv, hd):
    q, k, v, table, pos = problem(500, 0, nh, nkv, hd, hd, torch.float32, 16)
    whole = attend(q, k, v, table, pos, nh, nkv, hd, hd, 16, None, None)
    for at, n in ((0, 1), (499, 1), (70, 20), (100, 80), (200, 300)):
        assert torch.equal(attend(q[at:at + n].contiguous(), k, v, table, pos[at:at + n].contiguous(), nh, nkv, hd, hd, 16, None, None), whole[at:at + n]), (at, n)

"""Attention of steps that mix portions of prompts with many one-token requests: the prompt kernel's grid holds the portions only,
which each CTA finds among the requests (csrc/attention_tc.cu).  Against the float32-arithmetic kernel."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


# a portion first, last, behind more than 32 one-token requests; portions of no more than 16 rows per kv head stay with the
# decode kernel; none, one and all requests long
@pytest.mark.parametrize("lens", [[150] + [1] * 40, [1] * 40 + [150], [1] * 33 + [60] + [1] * 31 + [129, 2, 1, 300] + [1] * 7, [5, 1, 3, 2], [40, 129, 260]])
@pytest.mark.parametrize("nh,nkv,hd", [(12, 2, 128), (7, 1, 64), (4, 4, 128), (20, 1, 64)])
@pytest.mark.parametrize("two_tiles,cluster", [(None, 0), (True, 0), (False, 2)])
def test_portions_among_one_token_requests(lens, nh, nkv, hd, two_tiles, cluster):
    from coheryn_ai_studio_b200 import ops
    page, rng = 16, np.random.default_rng(len(lens) + hd)
    before = [int(rng.integers(0, 200)) for _ in lens]
    total = [n + b for n, b in zip(lens, before)]
    need = [-(-n // page) for n in total]
    order = rng.permutation(sum(need) + 1)
    tables = np.full((len(lens), max(need)), -1, np.int32)
    for i, n in enumerate(need):
        tables[i, :n] = order[sum(need[:i]):sum(need[:i + 1])]
    t32 = lambda a: torch.as_tensor(np.asarray(a, np.int32)).to(DEV)
    g = torch.Generator(device=DEV).manual_seed(3)
    b16 = lambda *s: torch.randn(s, device=DEV, generator=g).to(torch.bfloat16)
    kc, vc = b16(sum(need) + 1, nkv, page, hd), b16(sum(need) + 1, nkv, page, hd)
    T = sum(lens)
    q = b16(T, nh * hd)
    req = np.repeat(np.arange(len(lens)), lens)
    pos = np.concatenate([np.arange(b, b + n) for n, b in zip(lens, before)])
    got, want = torch.zeros_like(q), torch.zeros_like(q)
    args = (t32(tables), t32(req), t32(pos), nh, nkv, hd, page, None, hd ** -0.5)
    hints = dict(cu_q=t32(np.concatenate([[0], np.cumsum(lens)])), kv_lens=t32(total), q_lens=lens, max_kv_len=max(total))
    ops.set_attention_tc_two_tiles(hd, two_tiles)
    ops.set_attention_tc_cluster(hd, cluster)
    try:
        ops.attention_rows(q, got, kc, vc, *args, **hints)
    finally:
        ops.set_attention_tc_two_tiles(hd, None)
        ops.set_attention_tc_cluster(hd, 0)
    ops.attention_rows(q, want, kc, vc, *args, force_simple=True)
    ops.check_tc_status(q.device)
    # probabilities rounded to bfloat16 before the values (2^-8 for values of unit spread) and two rounded outputs
    bound = 2.0 ** -8 + 1.5 * 2.0 ** -8 * want.float().abs()
    assert bool(((got.float() - want.float()).abs() <= bound).all())

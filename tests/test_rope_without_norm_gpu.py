"""Rotation and cache writes of units without a norm against float64: rotated widths with and without channels that stay, one
and two maps, more items than one round of threads takes, mixed values, rows without a slot, and a row stride that sends the
same values through the kernel for unaligned rows."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("q_units,k_units,G,dk,rot,dv,mix,dtype", [
    (24, 4, 2, 64, 64, 128, 0.0, torch.bfloat16),
    (3, 2, 1, 24, 8, 20, 0.25, torch.float32),
    (40, 8, 8, 128, 96, 128, 0.5, torch.float32),
    (2, 1, 1, 4, 0, 4, 0.0, torch.float32),
    (5, 3, 3, 256, 256, 68, 0.0, torch.bfloat16),
])
@pytest.mark.parametrize("shift", [0, 1])
def test_units_rotated_without_a_norm(q_units, k_units, G, dk, rot, dv, mix, dtype, shift):
    from coheryn_ai_studio_b200 import ops
    gen = torch.Generator().manual_seed(q_units * dk + rot)
    T, page_size, pages = 37, 16, 4
    nq, nk, nv = q_units * dk, k_units * dk, G * dv
    rows = torch.randn(T, nq + nk + nv + shift, generator=gen)
    positions = torch.randint(0, 4096, (T,), generator=gen, dtype=torch.int32)
    slots = torch.randperm(pages * page_size, generator=gen)[:T].to(torch.int32)
    slots[3] = -1
    exact = 1.0 / 10000.0 ** (torch.arange(rot // 2, dtype=torch.float64) * 2 / max(rot, 1))
    high = exact.float()
    freq = torch.stack([high, (exact - high.double()).float()], 1).contiguous()
    first = torch.randn(T, nv, generator=gen) if mix else None
    M = k_units // G

    def turned(x, units):
        x = x.double().view(T, units, dk).clone()
        angle = positions.double()[:, None] * exact[None]
        c, s = angle.cos()[:, None] * 1.5, angle.sin()[:, None] * 1.5
        a, b = x[..., :rot // 2].clone(), x[..., rot // 2:rot].clone()
        x[..., :rot // 2], x[..., rot // 2:rot] = a * c - b * s, b * c + a * s
        return x

    want_q, want_k = turned(rows[:, :nq], q_units), turned(rows[:, nq:nq + nk], k_units)
    want_v = rows[:, nq + nk:nq + nk + nv].double()
    if mix:
        want_v = (1 - mix) * want_v + mix * first.double()
    dev = rows.cuda()
    k_cache = torch.full((pages, G, page_size, M * dk), 7.0, dtype=dtype, device="cuda")
    v_cache = torch.full((pages, G, page_size, dv), 7.0, dtype=dtype, device="cuda")
    q = ops.unit_norm_rope_kv_write(dev[:, :nq], dev[:, nq:nq + nk], dev[:, nq + nk:nq + nk + nv], None, None, 1e-6, positions.cuda(),
                                    freq.cuda() if rot else None, rot, 1.5, slots.cuda(), k_cache, v_cache, q_units, k_units, G, dk,
                                    dv, page_size, dtype, v_first=first.cuda() if mix else None, mix=mix)
    # an angle is a sum of two parts with a relative error of 2^-47 in all; sines, cosines and their combination are within a
    # few units in the last place of 1.5, and two products are added; bfloat16 results (8 significant bits) round once more by 2^-8
    rel = 2.0 ** -8 if dtype == torch.bfloat16 else 0.0
    scale = 1.5 * rows.abs().max().item()

    def same(got, want):
        error = (got.double().cpu() - want).abs()
        assert bool((error <= rel * want.abs() * 1.01 + 16 * 2.0 ** -23 * scale).all()), error.max()

    same(q.view(T, q_units, dk), want_q)
    written = torch.zeros(pages, page_size, dtype=torch.bool)
    for t in range(T):
        if slots[t] < 0:
            continue
        p, o = divmod(int(slots[t]), page_size)
        written[p, o] = True
        same(k_cache[p, :, o].reshape(k_units, dk), want_k[t])
        same(v_cache[p, :, o].reshape(-1), want_v[t])
    assert bool((k_cache.cpu().permute(0, 2, 1, 3)[~written] == 7.0).all()) and bool((v_cache.cpu().permute(0, 2, 1, 3)[~written] == 7.0).all())

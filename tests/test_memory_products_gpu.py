"""The two products of the chunked matrix memory (csrc/memory_chunks_tc.cu) at the edges of their tiles: 64 key channels, 128 and 256
value channels, chunks of 64 tokens, rows that allow no 16-byte loads."""
import numpy as np
import pytest
import torch

import plain_kapudra as plain
from test_chunked_scans_gpu import DEV, dev, step_of

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dk,dv,lens,dtype", [
    (1, 1, [48, 63], torch.float32), (63, 127, [64], torch.float32), (65, 129, [128, 65], torch.bfloat16), (64, 128, [192], torch.bfloat16),
    (129, 5, [127], torch.float32), (256, 256, [64, 129], torch.float32), (255, 253, [96], torch.bfloat16)])
@pytest.mark.parametrize("scale", [1.0, 3e4])
def test_products_at_the_edges_of_their_tiles(dk, dv, lens, dtype, scale):
    from coheryn_ai_studio_b200 import ops
    heads, cap, n, lib = 2, 10.0, sum(lens), ops.recurrent()
    rng = np.random.default_rng(dk + dv)
    f = lambda *s: rng.normal(size=s)
    q, k, v, gate = f(n, heads * dk), f(n, heads * dk), f(n, heads * dv) * scale, f(n, heads * dv) * 40      # gates shut to 1e-38 and open
    gi, gf, bi, bf, weight = f(n, heads), f(n, heads) + 3.0, f(heads), f(heads), f(heads * dv)
    first = f(len(lens), heads * (dk * dv + dk + 1))
    first[:, :heads * dk * dv] *= scale
    state, step = dev(first), step_of(lens, list(range(len(lens))), True)
    qkv, out = dev(np.concatenate([q, k, v], axis=1)), torch.empty((n, heads * dv), dtype=dtype, device=DEV)
    assert lib.coheryn_memory_chunk_floats(n // 48 + len(lens), heads, dk, dv) > 0
    pays = lib.coheryn_memory_chunks_pay
    try:
        lib.coheryn_memory_chunks_pay = lambda *a: 1      # the chunks whatever the scan would cost
        ops.matrix_memory_scan(qkv[:, :heads * dk], qkv[:, heads * dk:2 * heads * dk], qkv[:, 2 * heads * dk:], dev(gi), dev(gf), dev(bi),
                               dev(bf), cap, state, step, heads, dk, dv, out, dev(weight), dev(gate), 1e-5)
    finally:
        lib.coheryn_memory_chunks_pay = pays
    i, g = cap * np.tanh((gi + bi) / cap), plain.log_sigmoid(cap * np.tanh((gf + bf) / cap))
    o, room, at = np.zeros((n, heads, dv)), np.zeros((n, heads)), 0
    for r, length in enumerate(lens):
        for h in range(heads):
            S = first[r][:heads * dk * dv].reshape(heads, dk, dv)[h].copy()
            nn = first[r][heads * dk * dv:heads * dk * (dv + 1)].reshape(heads, dk)[h].copy()
            m = first[r][heads * dk * (dv + 1) + h]
            size, nsize = np.abs(S), np.abs(nn)
            for t in range(at, at + length):
                qt, kt, vt = q[t].reshape(heads, dk)[h] * dk ** -0.5, k[t].reshape(heads, dk)[h], v[t].reshape(heads, dv)[h]
                m_new = max(g[t, h] + m, i[t, h])
                a, b, m = np.exp(g[t, h] + m - m_new), np.exp(i[t, h] - m_new), m_new
                S, nn = a * S + b * np.outer(kt, vt), a * nn + b * kt
                size, nsize = a * size + b * np.outer(np.abs(kt), np.abs(vt)), a * nsize + b * np.abs(kt)
                den = max(abs(nn @ qt), np.exp(-m)) + 1e-6
                o[t, h] = (S.T @ qt) / den
                # sums of magnitudes over the result's: what the rounding of a float32 recurrence is multiplied by
                room[t, h] = (size.T @ np.abs(qt)).max() / den / max(np.sqrt((o[t, h] ** 2).mean()), 1e-300) + nsize @ np.abs(qt) / den
            got = state[r].cpu().numpy()[:heads * dk * dv].reshape(heads, dk, dv)[h]
            assert np.abs(got - S).max() <= 4 * (length + 8) * 2.0 ** -24 * size.max()
        at += length
    want = plain.rms(o, 1e-5).reshape(n, heads, dv) * weight.reshape(heads, dv) * plain.sigmoid(gate).reshape(n, heads, dv)
    # One rounding per term of a sum, 2^-24 of the sum of magnitudes each; dk + dv + 64 terms and the handful of factors around them.
    bound = (dk + 64 + 32) * 2.0 ** -24 * room[..., None] * np.abs(weight).max() * np.maximum(1.0, np.abs(plain.rms(o, 1e-5)).max(-1, keepdims=True))
    bound = bound + (2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -21) * np.abs(want) + 1e-37
    got = out.double().cpu().numpy().reshape(n, heads, dv)
    assert (np.abs(got - want) <= bound).all(), (np.abs(got - want) / bound).max()


@pytest.mark.parametrize("dk,dv", [(64, 128), (128, 256), (200, 72), (256, 128)])
def test_error_no_larger_than_that_of_multiply_adds(dk, dv):
    """A chunk's outputs against float64: no further off than the same products by the FMA kernel, whatever the number of key channels."""
    from coheryn_ai_studio_b200 import ops
    H, T, lib = 4, 64, ops.recurrent()
    g = torch.Generator(device=DEV).manual_seed(dk)
    f = lambda *s: torch.randn(s, device=DEV, generator=g)
    q, k, v, gates, state = f(T, H * dk), f(T, H * dk), f(T, H * dv), f(T, 2 * H), f(1, H * (dk * dv + dk + 1))
    gates[:, :H] -= 2.0
    gates[:, H:] += 4.5
    state[:, -H:] = 0.0
    first, qkv, out, zero = state[0].clone(), torch.cat([q, k, v], dim=1), torch.empty((T, H * dv), device=DEV), torch.zeros(H, device=DEV)
    pays = lib.coheryn_memory_chunks_pay
    try:
        lib.coheryn_memory_chunks_pay = lambda *a: 1
        ops.matrix_memory_scan(qkv[:, :H * dk], qkv[:, H * dk:2 * H * dk], qkv[:, 2 * H * dk:], gates[:, :H], gates[:, H:], zero, zero, 15.0, state,
                               step_of([T], [0], True), H, dk, dv, out, torch.ones(H * dv, device=DEV), torch.full((T, H * dv), 40.0, device=DEV), 1e-6)
    finally:
        lib.coheryn_memory_chunks_pay = pays
    cap = lambda z: 15.0 * torch.tanh(z.double() / 15.0)
    i, F = cap(gates[:, :H]), torch.nn.functional.logsigmoid(cap(gates[:, H:])).cumsum(0)
    errors = [0.0, 0.0, 0.0]
    for h in range(H):
        rows = lambda x, d: x[:, h * d:(h + 1) * d].contiguous()
        qh, kh, vh = rows(q, dk), rows(k, dk), rows(v, dv)
        S, n = first[h * dk * dv:(h + 1) * dk * dv].view(dk, dv), first[H * dk * dv + h * dk:H * dk * dv + (h + 1) * dk]
        each = F[:, h, None] - F[None, :, h] + i[None, :, h]
        each.masked_fill_(torch.ones(T, T, device=DEV).triu(1).bool(), -float("inf"))
        m = torch.maximum(each.max(1).values, F[:, h])
        w, a = (each - m[:, None]).exp(), (F[:, h] - m).exp()

        def outputs(product, dtype):
            s = product((qh.to(dtype) * dk ** -0.5), kh.to(dtype)) * w.to(dtype)
            den = torch.maximum((a.to(dtype) * (qh.to(dtype) * dk ** -0.5 * n.to(dtype)).sum(1) + s.sum(1)).abs(), (-m).exp().to(dtype)) + 1e-6
            o = (a[:, None].to(dtype) * product(qh.to(dtype) * dk ** -0.5, S.T.contiguous().to(dtype)) + product(s, vh.T.contiguous().to(dtype))) / den[:, None]
            return (o.double() / (o.double().square().mean(1, keepdim=True) + 1e-6).sqrt())

        def fma(x, y):
            got = torch.empty((x.shape[0], y.shape[0]), device=DEV)
            ops.gemm_simt(x.contiguous(), y, None, got)
            return got

        want = outputs(lambda x, y: x @ y.T, torch.float64)
        for e, got in enumerate((rows(out, dv).double(), outputs(fma, torch.float32))):
            errors[e] += float((got - want).square().sum())
        errors[2] += float(want.square().sum())
    assert errors[0] <= errors[1], [(e / errors[2]) ** 0.5 for e in errors[:2]]


@pytest.mark.parametrize("dk,dv", [(64, 128), (96, 200)])
@pytest.mark.parametrize("where,value", [("v", float("nan")), ("k", float("inf")), ("q", float("nan")), ("state", float("-inf")), ("v", 3.4e38)])
def test_values_that_are_not_finite_stay_in_their_chunks(dk, dv, where, value):
    """A bad value reaches its head's chunk and, through the state, the later ones; other heads, requests and earlier chunks keep their bits."""
    from coheryn_ai_studio_b200 import ops
    H, lens, lib = 3, [150, 70], ops.recurrent()
    T = sum(lens)
    g = torch.Generator(device=DEV).manual_seed(dk)
    f = lambda *s: torch.randn(s, device=DEV, generator=g)
    clean, gates, gate, first, zero = f(T, H * (2 * dk + dv)), f(T, 2 * H), f(T, H * dv), f(2, H * (dk * dv + dk + 1)), torch.zeros(H, device=DEV)
    first[:, -H:] = 0.0
    pays, got = lib.coheryn_memory_chunks_pay, []
    try:
        lib.coheryn_memory_chunks_pay = lambda *a: 1
        for bad in (False, True):
            qkv, state, out = clean.clone(), first.clone(), torch.empty((T, H * dv), device=DEV)
            if bad:      # head 1 of the first request; token 70 is the second chunk's
                at = {"q": dk + 5, "k": H * dk + dk + 5, "v": 2 * H * dk + dv + 7}
                if where == "state":
                    state[0, dk * dv + 3 * dv + 7] = value
                else:
                    qkv[70, at[where]] = value
            ops.matrix_memory_scan(qkv[:, :H * dk], qkv[:, H * dk:2 * H * dk], qkv[:, 2 * H * dk:], gates[:, :H], gates[:, H:], zero, zero, 15.0, state,
                                   step_of(lens, [0, 1], True), H, dk, dv, out, torch.ones(H * dv, device=DEV), gate, 1e-5)
            got.append((out.view(T, H, dv), state))
    finally:
        lib.coheryn_memory_chunks_pay = pays
    ops.check_tc_status(DEV)
    (want, want_state), (out, state) = got
    assert torch.isfinite(want).all() and torch.isfinite(want_state).all()
    assert torch.equal(out[:, 0], want[:, 0]) and torch.equal(out[:, 2], want[:, 2]) and torch.equal(out[150:], want[150:])
    assert torch.equal(state[1], want_state[1])
    start = 0 if where == "state" else 64
    assert torch.equal(out[:start, 1], want[:start, 1])
    assert not torch.isfinite(out[70, 1]).all()
    if where != "q":      # the norm over the value channels takes it to all of them, the state to the chunks behind
        assert not torch.isfinite(out[130:150, 1]).any() and not torch.isfinite(state[0]).all()
    else:
        assert torch.isfinite(out[128:150, 1]).all() and torch.equal(state[0], want_state[0])


@pytest.mark.parametrize("what", ["v", "state", "k"])
def test_operands_under_the_terms_range(what):
    """Operands under 2^-110: a result is off by 2^-133 of each at most, times the other operand."""
    from coheryn_ai_studio_b200 import ops
    H, T, dk, dv, lib = 2, 64, 64, 128, ops.recurrent()
    g = torch.Generator(device=DEV).manual_seed(5)
    f = lambda *s: torch.randn(s, device=DEV, generator=g)
    q, k, v, state = f(T, H * dk), f(T, H * dk), f(T, H * dv), f(1, H * (dk * dv + dk + 1))
    state[:, H * dk * dv:] = 0.0
    for name, t in (("v", v), ("k", k), ("state", state)):
        if name == what or (name == "state" and what != "state") or (name == "v" and what == "state"):
            t.mul_(2.0 ** -124 if name == what else 0.0)
    first, qkv, zero, out = state.clone(), torch.cat([q, k, v], dim=1), torch.zeros(H, device=DEV), torch.empty((T, H * dv), device=DEV)
    pays = lib.coheryn_memory_chunks_pay
    try:
        lib.coheryn_memory_chunks_pay = lambda *a: 1      # the gates are open: log f = 0 to 1e-6, log i = 0
        ops.matrix_memory_scan(qkv[:, :H * dk], qkv[:, H * dk:2 * H * dk], qkv[:, 2 * H * dk:], torch.zeros(T, H, device=DEV),
                               torch.full((T, H), 1e4, device=DEV), zero, zero, 15.0, state, step_of([T], [0], True), H, dk, dv, out,
                               torch.ones(H * dv, device=DEV), torch.full((T, H * dv), 40.0, device=DEV), 1e-6)
    finally:
        lib.coheryn_memory_chunks_pay = pays
    for h in range(H):
        S, kh, vh = first[0, h * dk * dv:(h + 1) * dk * dv].view(dk, dv).double(), k[:, h * dk:(h + 1) * dk].double(), v[:, h * dv:(h + 1) * dv].double()
        want, got = S + kh.T @ vh, state[0, h * dk * dv:(h + 1) * dk * dv].view(dk, dv).double()
        # the gates and float32's sums as everywhere; what the split cuts off
        bound = (T + 32) * 2.0 ** -23 * (S.abs() + kh.abs().T @ vh.abs()) + 2.0 ** -133 * (kh.abs().sum(0)[:, None] + vh.abs().sum(0)[None, :])
        assert bool(((got - want).abs() <= bound).all())
    assert bool(torch.isfinite(out).all()) and float(out.abs().max()) < 1e-25      # (the norm's eps is larger than any of these)

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

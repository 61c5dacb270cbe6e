"""The gated delta rule and the matrix memory in chunks of 64 tokens (csrc/delta_chunks.cu, csrc/memory_chunks.cu) against the recurrences written token by token in float64,
at the edges of the runs it takes, of its chunks, blocks and tiles, and beside runs that stay with the scan."""
import types

import numpy as np
import pytest
import torch

import plain_kapudra as plain

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def dev(a, dtype=torch.float32):
    return torch.as_tensor(np.asarray(a)).to(DEV, dtype)


def step_of(lengths, slots, host=True):
    cu = np.concatenate([[0], np.cumsum(lengths)])
    st = types.SimpleNamespace(num_requests=len(lengths), num_tokens=int(cu[-1]), cu_q=dev(cu, torch.int32),
                               token_req=dev(np.repeat(np.arange(len(lengths)), lengths), torch.int32), state_slots=dev(slots, torch.int32))
    if host:
        st.q_lens = list(lengths)
    return st


def delta_inputs(rng, n, heads, groups, dk, dv, channel):
    f = lambda *s: rng.normal(size=s)
    return dict(q=f(n, groups * dk), k=f(n, groups * dk), v=f(n, heads * dv), beta=f(n, heads), step=f(n, heads * (dk if channel else 1)),
                gate=f(n, heads * dv))


def run_delta(parts, state, slots, bias, rate_log, weight, heads, groups, dk, dv, channel, act, host):
    from coheryn_ai_studio_b200 import ops
    cat = lambda key: dev(np.concatenate([d[key] for d in parts]))
    step = step_of([len(d["q"]) for d in parts], slots, host)
    qkv, G = torch.cat([cat("q"), cat("k"), cat("v")], dim=1), groups * dk
    out = torch.empty((step.num_tokens, heads * dv), device=DEV)
    ops.gated_delta_scan(qkv[:, :G], qkv[:, G:2 * G], qkv[:, 2 * G:], cat("beta"), cat("step"), dev(bias), dev(rate_log), state, step, heads,
                         groups, dk, dv, out, dev(weight), cat("gate"), 1e-5, decay_per_channel=channel, gate_activation=act)
    return out.cpu().numpy()


# The bounds are those of the token-by-token kernel's own test (2e-4 of the largest value): the chunks add the same float32
# products in another order.
@pytest.mark.parametrize("lens", [[47, 48], [64, 2, 65], [130, 1, 63], [257]])
@pytest.mark.parametrize("heads,groups,dk,dv,channel,act,host", [
    (4, 2, 20, 30, True, "sigmoid", True), (2, 1, 64, 64, False, "silu", True), (2, 2, 65, 72, True, "silu", False),
    (2, 1, 128, 128, True, "sigmoid", True), (1, 1, 128, 256, False, "sigmoid", False), (3, 1, 96, 144, True, "sigmoid", True)])
def test_gated_delta_rule_in_chunks(lens, heads, groups, dk, dv, channel, act, host):
    rng = np.random.default_rng(dk + dv + lens[0])
    parts = [delta_inputs(rng, n, heads, groups, dk, dv, channel) for n in lens]
    dc = dk if channel else 1
    # decays from nearly one to nothing: a chunk's product leaves float32's range in some channels and not in others
    bias, rate_log, weight = rng.uniform(-7, 3, size=heads * dc), rng.normal(size=heads), rng.normal(size=dv)
    slots = list(rng.permutation(len(lens) + 1)[:len(lens)])
    first = rng.normal(size=(len(lens) + 1, heads * dk * dv)) * 0.1
    state = dev(first)
    got = run_delta(parts, state, slots, bias, rate_log, weight, heads, groups, dk, dv, channel, act, host)
    after, at = state.cpu().numpy(), 0
    for d, slot in zip(parts, slots):
        n = len(d["q"])
        q = d["q"].reshape(n, groups, dk); k = d["k"].reshape(n, groups, dk)
        q = q / np.sqrt((q * q).sum(-1, keepdims=True) + 1e-6) * dk ** -0.5
        k = k / np.sqrt((k * k).sum(-1, keepdims=True) + 1e-6)
        decay = np.exp(-np.exp(rate_log)[None, :, None] * plain.softplus(d["step"] + bias).reshape(n, heads, dc))
        o = np.zeros((n, heads, dv))
        for h in range(heads):
            S, g = first[slot].reshape(heads, dk, dv)[h].copy(), h // (heads // groups)
            for t in range(n):
                S = decay[t, h][:, None] * S
                u = plain.sigmoid(d["beta"][t, h]) * (d["v"].reshape(n, heads, dv)[t, h] - S.T @ k[t, g])
                S = S + np.outer(k[t, g], u)
                o[t, h] = S.T @ q[t, g]
            end = after[slot].reshape(heads, dk, dv)[h]
            assert np.abs(end - S).max() <= 2e-4 * max(1.0, np.abs(S).max()), (slot, h)
        z = d["gate"].reshape(n, heads, dv)
        want = (plain.rms(o, 1e-5) * weight * plain.sigmoid(z) * (z if act == "silu" else 1.0)).reshape(n, heads * dv)
        assert np.abs(got[at:at + n] - want).max() <= 2e-4 * max(1.0, np.abs(want).max()), slot
        at += n
    untouched = [s for s in range(len(lens) + 1) if s not in slots]
    assert np.array_equal(after[untouched], dev(first[untouched]).cpu().numpy())


def test_a_runs_rows_do_not_depend_on_the_other_runs():
    """Bit for bit: alone, beside a run that goes chunk by chunk and beside one that goes token by token (at sizes where each run's
    own step and the common one take the same form, see test_chunk_choice.py)."""
    rng = np.random.default_rng(5)
    heads, groups, dk, dv = 2, 1, 64, 48
    parts = [delta_inputs(rng, n, heads, groups, dk, dv, True) for n in (100, 9, 47, 64)]
    bias, rate_log, weight = rng.normal(size=heads * dk), rng.normal(size=heads), rng.normal(size=dv)
    args = (bias, rate_log, weight, heads, groups, dk, dv, True, "sigmoid", True)
    state = torch.zeros((4, heads * dk * dv), device=DEV)
    both, at = run_delta(parts, state, [2, 0, 3, 1], *args), 0
    for d in parts:
        n = len(d["q"])
        alone = run_delta([d], torch.zeros((1, heads * dk * dv), device=DEV), [0], *args)
        assert np.array_equal(alone, both[at:at + n]), n
        at += n


@pytest.mark.parametrize("taps,channels,offset", [(2, 40, 0), (3, 36, 3), (4, 1028, 4), (4, 130, 1), (5, 24, 0)])
def test_short_convolution_by_runs_of_tokens(taps, channels, offset):
    """Runs shorter and longer than the taps and than a thread's tokens, aligned and unaligned columns, states of strided rows."""
    from coheryn_ai_studio_b200 import ops
    rng = np.random.default_rng(taps + channels)
    lens = [1, 2, 40, 3, 17]
    n = sum(lens)
    wide = dev(rng.normal(size=(n, channels + 12)))
    x = wide[:, offset:offset + channels]
    w = dev(rng.normal(size=(channels, taps)))
    keep = taps - 1
    state = dev(rng.normal(size=(6, 8 + keep * channels)))[:, 8:]
    slots = [4, 0, 5, 2, 1]
    before = state.double().cpu().numpy().reshape(6, keep, channels)
    y = ops.short_conv_silu(x, w, state, step_of(lens, slots)).double().cpu().numpy()
    xs, ws, at = x.double().cpu().numpy(), w.double().cpu().numpy(), 0
    after = state.cpu().numpy().reshape(6, keep, channels)
    for m, slot in zip(lens, slots):
        rows = np.concatenate([before[slot], xs[at:at + m]])
        want = plain.silu(sum(rows[j:j + m] * ws[:, j] for j in range(taps)))
        # a sum of `taps` products and the activation in float32
        assert np.abs(y[at:at + m] - want).max() <= 1e-5 * max(1.0, np.abs(want).max())
        assert np.array_equal(after[slot], rows[-keep:].astype(np.float32))
        at += m


# The bound is that of the token-by-token kernel's own test: a float32 recurrence is itself up to 5e-4 from float64 where a row's
# output nearly cancels before its norm.
@pytest.mark.parametrize("lens", [[47, 48], [64, 2, 65], [130, 1, 63], [257]])
@pytest.mark.parametrize("heads,dk,dv,cap,open_gate,host", [
    (3, 20, 30, 9.0, False, True), (2, 64, 128, 15.0, True, True), (2, 72, 130, 8.0, False, False), (1, 128, 256, 15.0, True, False),
    (1, 256, 144, 12.0, False, True)])
def test_matrix_memory_in_chunks(lens, heads, dk, dv, cap, open_gate, host):
    from coheryn_ai_studio_b200 import ops
    rng = np.random.default_rng(dk + dv + lens[0])
    f = lambda *s: rng.normal(size=s)
    parts = [dict(q=f(n, heads * dk), k=f(n, heads * dk), v=f(n, heads * dv), gi=f(n, heads) * 3, gf=f(n, heads) * 3 + (6.0 if open_gate else -6.0),
                  gate=f(n, heads * dv)) for n in lens]       # forget gates held open, or shut: exponents from 0 to hundreds in a chunk
    bi, bf, weight = f(heads), f(heads), f(heads * dv)
    size = heads * (dk * dv + dk + 1)
    slots = list(rng.permutation(len(lens) + 1)[:len(lens)])
    first = f(len(lens) + 1, size) * 0.3
    state, step = dev(first), step_of(lens, slots, host)
    cat = lambda key: dev(np.concatenate([d[key] for d in parts]))
    qkv, gates = torch.cat([cat("q"), cat("k"), cat("v")], dim=1), torch.cat([cat("gi"), cat("gf")], dim=1)
    out = torch.empty((step.num_tokens, heads * dv), device=DEV)
    ops.matrix_memory_scan(qkv[:, :heads * dk], qkv[:, heads * dk:2 * heads * dk], qkv[:, 2 * heads * dk:], gates[:, :heads], gates[:, heads:],
                           dev(bi), dev(bf), cap, state, step, heads, dk, dv, out, dev(weight), cat("gate"), 1e-5)
    got, after, at = out.cpu().numpy(), state.cpu().numpy(), 0
    for d, slot in zip(parts, slots):
        n = len(d["q"])
        li = cap * np.tanh((d["gi"] + bi) / cap)
        lf = plain.log_sigmoid(cap * np.tanh((d["gf"] + bf) / cap))
        o = np.zeros((n, heads, dv))
        for h in range(heads):
            S = first[slot][:heads * dk * dv].reshape(heads, dk, dv)[h].copy()
            nn = first[slot][heads * dk * dv:heads * dk * (dv + 1)].reshape(heads, dk)[h].copy()
            m = first[slot][heads * dk * (dv + 1) + h]
            q, k, v = d["q"].reshape(n, heads, dk)[:, h] * dk ** -0.5, d["k"].reshape(n, heads, dk)[:, h], d["v"].reshape(n, heads, dv)[:, h]
            for t in range(n):
                m_new = max(lf[t, h] + m, li[t, h])
                a, b, m = np.exp(lf[t, h] + m - m_new), np.exp(li[t, h] - m_new), m_new
                S, nn = a * S + b * np.outer(k[t], v[t]), a * nn + b * k[t]
                o[t, h] = (S.T @ q[t]) / (max(abs(nn @ q[t]), np.exp(-m)) + 1e-6)
            assert np.abs(after[slot][:heads * dk * dv].reshape(heads, dk, dv)[h] - S).max() <= 2e-4 * max(1.0, np.abs(S).max())
            assert np.abs(after[slot][heads * dk * dv:heads * dk * (dv + 1)].reshape(heads, dk)[h] - nn).max() <= 2e-4 * max(1.0, np.abs(nn).max())
            assert abs(after[slot][heads * dk * (dv + 1) + h] - m) <= 2e-5 * max(1.0, abs(m))
        want = plain.rms(o, 1e-5).reshape(n, heads * dv) * weight * plain.sigmoid(d["gate"])
        assert np.abs(got[at:at + n] - want).max() <= 1e-3 * max(1.0, np.abs(want).max()), slot
        at += n


@pytest.mark.parametrize("kind,dk,dv", [("gated_delta_rule", 64, 128), ("gated_delta_rule", 24, 40), ("matrix_memory", 64, 64), ("matrix_memory", 128, 48)])
def test_float32_mixers_keep_their_bits_however_a_sequence_is_cut(kind, dk, dv):
    """A float32 mixer over 200 tokens in one step, in four portions (two of them long enough for chunks), and beside another
    request: the same outputs and the same state, bit for bit."""
    from coheryn_ai_studio_b200.config.spec import PartSpec
    from coheryn_ai_studio_b200.parts.base import MIXERS, LayerCache, Runtime, build_part
    g = torch.Generator(DEV).manual_seed(dk + dv)
    params = dict(hidden_size=96, num_heads=2, head_dim=dk, v_head_dim=dv, eps=1e-6)
    params.update(dict(num_kv_heads=1, conv_taps=4, decay_rank=16, gate_rank=16) if kind == "gated_delta_rule" else dict(gate_cap=15.0))
    part = build_part(MIXERS, "mixer", PartSpec(kind, params), Runtime(torch.float32, torch.device(DEV)))
    ranks = {"a1": (16, 96), "a2": (part.decay_size, 16), "g1": (16, 96), "g2": (2 * dv, 16)} if kind == "gated_delta_rule" else {}
    part.bind({n: torch.randn(ranks.get(n, s.shape), generator=g, device=DEV) * (ranks.get(n, s.shape)[-1] ** -0.5 if len(s.shape) > 1 else 1.0)
               for n, s in part.tensor_specs().items()})
    x, other = torch.randn((200, 96), generator=g, device=DEV), torch.randn((120, 96), generator=g, device=DEV)
    size = part.cache_requirement().shape

    def run(cuts, beside=0):
        state, outs, at = torch.zeros((2,) + tuple(size), device=DEV), [], 0
        for n in cuts:
            rows, lens, slots = x[at:at + n], [n], [1]
            if beside:
                rows, lens, slots = torch.cat([other[:beside], rows]), [beside, n], [0, 1]
            y = part.forward(rows.contiguous(), step_of(lens, slots), LayerCache("state", state=state))
            outs.append(y[sum(lens) - n:])
            at += n
        return torch.cat(outs), state[1]

    want, end = run([200])
    assert want.shape[0] == 200 and bool(want.isfinite().all()) and float(want.abs().max()) > 0
    for got, state in (run([64, 1, 70, 65]), run([1, 199]), run([130, 70], beside=120)):
        assert torch.equal(got, want) and torch.equal(state, end)


@pytest.mark.parametrize("heads,dk,dv", [(2, 24, 200), (1, 128, 256), (3, 64, 72), (1, 192, 80), (2, 256, 130)])
def test_long_portions_token_by_token(heads, dk, dv):
    """The scans of long portions, whose heads' columns go to several CTAs (norm and gate in a kernel of their own), and of the
    short ones between them, continuing each other's state: sizes that chunks take too, and more key channels than they take.  The
    bounds are those of the scans' own tests."""
    from coheryn_ai_studio_b200 import ops
    rng = np.random.default_rng(dv + dk)
    cuts, eps, cap = [130, 1, 70, 2, 64, 33], 1e-6, 9.0
    n = sum(cuts)
    f = lambda *s: rng.normal(size=s)
    d = dict(delta_inputs(rng, n, heads, 1, dk, dv, True), mq=f(n, heads * dk), mk=f(n, heads * dk), gi=f(n, heads) * 2, gf=f(n, heads) * 2 + 3.0)
    bias, rate_log, weight, bi, bf, wm = f(heads * dk), f(heads) * 0.5, f(dv), f(heads), f(heads), f(heads * dv)
    unit = lambda a: a / np.sqrt((a * a).sum(-1, keepdims=True) + 1e-6)
    decay = np.exp(-np.exp(rate_log)[None, :, None] * plain.softplus(d["step"] + bias).reshape(n, heads, dk))
    v, per = d["v"].reshape(n, heads, dv), lambda a: a.reshape(n, heads, dk)
    o = np.stack([plain.gated_delta_rule(unit(d["q"]) * dk ** -0.5, unit(d["k"]), v[:, h], plain.sigmoid(d["beta"][:, h]), decay[:, h])
                  for h in range(heads)], axis=1)
    want_d = (plain.rms(o, eps) * weight).reshape(n, heads * dv) * plain.sigmoid(d["gate"])
    li = cap * np.tanh((d["gi"] + bi) / cap); lf = plain.log_sigmoid(cap * np.tanh((d["gf"] + bf) / cap))
    o = np.stack([plain.matrix_memory(per(d["mq"])[:, h] * dk ** -0.5, per(d["mk"])[:, h], v[:, h], li[:, h], lf[:, h]) for h in range(heads)], axis=1)
    want_m = plain.rms(o, eps).reshape(n, heads * dv) * wm * plain.sigmoid(d["gate"])
    state_d, state_m = torch.zeros((2, heads * dk * dv), device=DEV), torch.zeros((2, heads * (dk * dv + dk + 1)), device=DEV)
    at = 0
    for m in cuts:
        step, cat = step_of([m], [1]), lambda *keys: dev(np.concatenate([d[k][at:at + m] for k in keys], axis=1))
        out = torch.empty((m, heads * dv), device=DEV)
        qkv = cat("q", "k", "v")
        ops.gated_delta_scan(qkv[:, :dk], qkv[:, dk:2 * dk], qkv[:, 2 * dk:], cat("beta"), cat("step"), dev(bias), dev(rate_log), state_d, step,
                             heads, 1, dk, dv, out, dev(weight), cat("gate"), eps, in_chunks=False)
        ref = want_d[at:at + m]
        assert np.abs(out.cpu().numpy() - ref).max() <= 3e-4 * max(1.0, np.abs(ref).max()), ("delta", at, m)
        qkv, gates, c = cat("mq", "mk", "v"), cat("gi", "gf"), heads * dk
        ops.matrix_memory_scan(qkv[:, :c], qkv[:, c:2 * c], qkv[:, 2 * c:], gates[:, :heads], gates[:, heads:], dev(bi), dev(bf), cap, state_m, step,
                               heads, dk, dv, out, dev(wm), cat("gate"), eps, in_chunks=False)
        ref = want_m[at:at + m]
        assert np.abs(out.cpu().numpy() - ref).max() <= 1e-3 * max(1.0, np.abs(ref).max()), ("memory", at, m)
        at += m


@pytest.mark.parametrize("taps,channels,offset", [(2, 256, 0), (3, 260, 4), (2, 65, 0), (3, 129, 1), (4, 24, 0)])
def test_short_convolution_wide_and_narrow(taps, channels, offset):
    """Rows by four channels and by one per thread, and too few channels for a CTA."""
    test_short_convolution_by_runs_of_tokens(taps, channels, offset)


def test_short_convolution_of_a_million_tokens():
    """One run of 2^20 + 50 tokens: more sixteens of tokens than a grid's second dimension holds."""
    from coheryn_ai_studio_b200 import ops
    n, channels, taps = (1 << 20) + 50, 65, 3
    g = torch.Generator(DEV).manual_seed(2)
    x, w, state = (torch.randn(s, generator=g, device=DEV) for s in ((n, channels), (channels, taps), (1, (taps - 1) * channels)))
    rows = torch.cat([state.reshape(taps - 1, channels), x])
    step = types.SimpleNamespace(num_requests=1, num_tokens=n, cu_q=dev([0, n], torch.int32), token_req=torch.zeros(n, dtype=torch.int32, device=DEV),
                                 state_slots=dev([0], torch.int32), q_lens=[n])
    y = ops.short_conv_silu(x, w, state, step)
    for at in (0, 524288, n - 100):
        s = sum(rows[at + j:at + j + 100].double() * w[:, j].double() for j in range(taps))
        want = s * torch.sigmoid(s)
        assert float((y[at:at + 100].double() - want).abs().max()) <= 1e-5 * max(1.0, float(want.abs().max()))
    assert torch.equal(state.reshape(taps - 1, channels), x[n - taps + 1:])


@pytest.mark.parametrize("kind,heads,dk,dv,lens", [("delta", 16, 128, 128, [4000, 70, 3000]), ("memory", 8, 128, 256, [9000, 70, 9000])])
def test_more_chunks_than_the_scratch_holds(kind, heads, dk, dv, lens):
    """A step whose chunks' scratch would pass its bound goes in several groups of chunks, the last run's state from one to the next:
    the same bits as each long run alone, which fits at once."""
    from coheryn_ai_studio_b200 import ops
    g, n = torch.Generator(DEV).manual_seed(3), sum(lens)
    f = lambda *s: torch.randn(s, generator=g, device=DEV)
    size = heads * (dk * dv + (dk + 1 if kind == "memory" else 0))
    qkv, step_pre, pair, gate, weight = f(n, heads * (2 * dk + dv)), f(n, heads * dk), f(n, 2 * heads), f(n, heads * dv), f(heads * dv)
    bias, small, c = f(heads * dk), f(2 * heads), heads * dk

    def run(a, b, lens):
        rows, out = slice(a, b), torch.empty((b - a, heads * dv), device=DEV)
        state, step = torch.zeros((len(lens), size), device=DEV), step_of(lens, list(range(len(lens))))
        q, k, v = qkv[rows, :c], qkv[rows, c:2 * c], qkv[rows, 2 * c:]
        if kind == "delta":
            ops.gated_delta_scan(q, k, v, pair[rows, :heads], step_pre[rows], bias, small[:heads].contiguous(), state, step, heads, heads, dk, dv, out,
                                 weight[:dv].contiguous(), gate[rows], 1e-5)
        else:
            ops.matrix_memory_scan(q, k, v, pair[rows, :heads], pair[rows, heads:], small[:heads].contiguous(), small[heads:].contiguous(), 15.0, state,
                                   step, heads, dk, dv, out, weight, gate[rows], 1e-5)
        return out, state

    both, state = run(0, n, lens)
    for i in (0, 2):
        a = sum(lens[:i])
        alone, end = run(a, a + lens[i], [lens[i]])
        assert torch.equal(alone, both[a:a + lens[i]]) and torch.equal(end[0], state[i]) and bool(alone.isfinite().all())

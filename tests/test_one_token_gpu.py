"""Steps of one token per request (csrc/recurrent_one.cu): the bits of the token-by-token scans, which an unaligned state still takes, for every
size of key channels that the scans are built for, both widths of values, runs of no token beside one of two, decays per head and channel."""
import types

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def step_of(lens):
    cu = torch.tensor([sum(lens[:i]) for i in range(len(lens) + 1)], dtype=torch.int32, device=DEV)
    return types.SimpleNamespace(num_requests=len(lens), cu_q=cu, state_slots=torch.arange(len(lens), dtype=torch.int32, device=DEV).flip(0).contiguous(),
                                 q_lens=list(lens))


def state_of(values, shift):
    """The same values, `shift` elements off a 16-byte boundary."""
    rows, n = values.shape
    pitch = -(-n // 4) * 4
    view = torch.zeros((rows * pitch + 4,), device=DEV)[shift:shift + rows * pitch].view(rows, pitch)[:, :n]
    return view.copy_(values)


LENS = [[1], [1, 1, 1, 1, 1], [0, 2, 1]]


@pytest.mark.parametrize("lens", LENS)
@pytest.mark.parametrize("heads,groups,dk,dv", [(2, 1, 16, 4), (3, 3, 30, 60), (2, 2, 48, 128), (4, 2, 64, 132), (2, 1, 96, 256), (12, 4, 128, 128),
                                                (2, 2, 100, 200), (1, 1, 192, 128), (2, 1, 256, 100), (1, 1, 200, 200)])
@pytest.mark.parametrize("channel,act", [(True, "sigmoid"), (False, "silu")])
def test_delta_rule(lens, heads, groups, dk, dv, channel, act):
    from coheryn_ai_studio_b200 import ops
    g = torch.Generator(device=DEV).manual_seed(dk + dv)
    f = lambda *s: torch.randn(s, device=DEV, generator=g)
    T, B, dc = sum(lens), len(lens), dk if channel else 1
    qkv, beta, pre, gate = f(T, 2 * groups * dk + heads * dv), f(T, heads), f(T, heads * dc), f(T, heads * dv)
    bias, rate, weight, first = f(heads * dc), f(heads), f(dv), f(B, heads * dk * dv)
    got = []
    for shift in (0, 1):
        state, out = state_of(first, shift), torch.empty((T, heads * dv), device=DEV)
        ops.gated_delta_scan(qkv[:, :groups * dk], qkv[:, groups * dk:2 * groups * dk], qkv[:, 2 * groups * dk:], beta, pre, bias, rate, state,
                             step_of(lens), heads, groups, dk, dv, out, weight, gate, 1e-5, decay_per_channel=channel, gate_activation=act)
        got.append((out, state.clone()))
    assert torch.isfinite(got[0][0]).all() and torch.equal(got[0][0], got[1][0]) and torch.equal(got[0][1], got[1][1])
    assert not torch.equal(got[0][1][B - lens.index(1) - 1], first[B - lens.index(1) - 1])


@pytest.mark.parametrize("lens", LENS)
@pytest.mark.parametrize("heads,dk,dv", [(2, 16, 4), (3, 30, 60), (2, 48, 128), (4, 64, 132), (8, 128, 256), (2, 100, 200), (1, 192, 128), (2, 256, 100), (1, 200, 200)])
def test_matrix_memory(lens, heads, dk, dv):
    from coheryn_ai_studio_b200 import ops
    g = torch.Generator(device=DEV).manual_seed(dk + dv)
    f = lambda *s: torch.randn(s, device=DEV, generator=g)
    T, B = sum(lens), len(lens)
    qkv, gates, gate = f(T, heads * (2 * dk + dv)), 3 * f(T, 2 * heads), f(T, heads * dv)
    bi, bf, weight, first = f(heads), f(heads), f(heads * dv), f(B, heads * (dk * dv + dk + 1))
    got = []
    for shift in (0, 1):
        state, out = state_of(first, shift), torch.empty((T, heads * dv), device=DEV)
        ops.matrix_memory_scan(qkv[:, :heads * dk], qkv[:, heads * dk:2 * heads * dk], qkv[:, 2 * heads * dk:], gates[:, :heads], gates[:, heads:], bi, bf,
                               15.0, state, step_of(lens), heads, dk, dv, out, weight, gate, 1e-5)
        got.append((out, state.clone()))
    assert torch.isfinite(got[0][0]).all() and torch.equal(got[0][0], got[1][0]) and torch.equal(got[0][1], got[1][1])

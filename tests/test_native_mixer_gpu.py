"""A recurrent mixer enqueued by one call into the library (csrc/mixer_runner.cu) gives the bits of its operations run one by one: decode steps,
prompts that go in chunks, mixed and empty runs, widths on both sides of the products' row thresholds, a row stride, the open form."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def weights(specs, seed):
    g = torch.Generator(device=DEV).manual_seed(seed)
    return {n: torch.randn([32 if d < 0 else d for d in s.shape], device=DEV, generator=g).mul_(0.05).to(torch.bfloat16) for n, s in specs.items()}


def step_of(lens):
    from coheryn_ai_studio_b200.parts.base import StepContext
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)
    T = sum(lens)
    cu = [sum(lens[:i]) for i in range(len(lens) + 1)]
    return StepContext(num_tokens=T, num_requests=len(lens), token_ids=i32([0] * T), positions=i32([0] * T),
                       token_req=i32([r for r, n in enumerate(lens) for _ in range(n)]), cu_q=i32(cu), kv_lens=i32(lens), block_tables=[], slots=[],
                       state_slots=i32(list(range(len(lens)))[::-1]), q_lens=list(lens), kv_lens_host=list(lens), max_q_len=max(lens), max_kv_len=max(lens))


DELTA = dict(hidden_size=256, num_heads=4, num_kv_heads=2, head_dim=64, v_head_dim=72, conv_taps=4, eps=1e-6)
CASES = [("gated_delta_rule", dict(DELTA, decay_rank=32, gate_rank=32)), ("gated_delta_rule", dict(DELTA, decay="head", low_rank=False, gate_activation="silu")),
         ("matrix_memory", dict(hidden_size=256, num_heads=4, head_dim=64, v_head_dim=128, gate_cap=15.0, eps=1e-6, out_scale=0.5))]


@pytest.mark.parametrize("kind,params", CASES)
@pytest.mark.parametrize("lens", [[1], [1] * 20, [1] * 40, [7, 0, 3], [130, 1, 64], [700], [300, 2, 900]])
def test_one_call_equals_the_operations(kind, params, lens):
    from coheryn_ai_studio_b200 import ops
    from coheryn_ai_studio_b200.config.spec import PartSpec
    from coheryn_ai_studio_b200.parts import model, native_mixer  # noqa: F401  (registers the parts)
    from coheryn_ai_studio_b200.parts.base import MIXERS, LayerCache, Runtime, build_part
    part = build_part(MIXERS, "mixer", PartSpec(kind, params), Runtime(torch.bfloat16, torch.device(DEV)))
    part.bind(weights(part.tensor_specs(), 3))
    step, width = step_of(lens), params["num_heads"] * params["v_head_dim"]
    g = torch.Generator(device=DEV).manual_seed(len(lens))
    x = torch.randn((step.num_tokens, 256 + 8), device=DEV, generator=g).to(torch.bfloat16)[:, :256]
    first = torch.randn((len(lens),) + tuple(part.cache_requirement().shape), device=DEV, generator=g) * 0.1
    got = []
    for native in (False, True):
        ops.set_native_block(native)
        try:
            before = native_mixer.runs
            a, b = (LayerCache("state", state=first.clone()) for _ in range(2))
            y = part.forward(x, step, a)
            opened = torch.zeros((step.num_tokens, width + 16), dtype=torch.bfloat16, device=DEV)
            part.forward_open(x, step, b, [opened[:, 8:8 + width]])
            got.append((y, a.state, opened, b.state))
            assert native_mixer.runs - before == (2 if native else 0)
        finally:
            ops.set_native_block(True)
    for one, other in zip(*got):
        assert torch.isfinite(one).all() and torch.equal(one, other)


def test_what_it_leaves_to_the_operations():
    """Other types and steps without tokens."""
    from coheryn_ai_studio_b200.config.spec import PartSpec
    from coheryn_ai_studio_b200.parts import model, native_mixer  # noqa: F401
    from coheryn_ai_studio_b200.parts.base import MIXERS, LayerCache, Runtime, build_part
    kind, params = CASES[0]
    part = build_part(MIXERS, "mixer", PartSpec(kind, params), Runtime(torch.float32, torch.device(DEV)))
    part.bind({n: t.float() for n, t in weights(part.tensor_specs(), 3).items()})
    assert part.native is None
    part = build_part(MIXERS, "mixer", PartSpec(kind, params), Runtime(torch.bfloat16, torch.device(DEV)))
    part.bind(weights(part.tensor_specs(), 3))
    before, state = native_mixer.runs, torch.zeros((1,) + tuple(part.cache_requirement().shape), device=DEV)
    step = step_of([1])
    out = torch.empty((1, 0, 256), device=DEV)
    step.num_tokens = 0
    assert not part.native.run(torch.empty((0, 256), dtype=torch.bfloat16, device=DEV), step, state, None, out[0]) and native_mixer.runs == before
    assert not part.native.run(torch.zeros((1, 256), device=DEV), step, state, None, torch.empty((1, 256), device=DEV))

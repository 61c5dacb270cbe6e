"""A recurrent mixer enqueued by one call into the library (csrc/mixer_runner.cu) gives the bits of its operations run one by one: decode steps,
prompts that go in chunks, mixed and empty runs, widths on both sides of the products' row thresholds, a row stride, the open form, the layer sizes of
the models.  What does not fit the part's sizes never reaches the library."""
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


def broken(kind, params, name):
    """The part's weights with one of them of another size."""
    from coheryn_ai_studio_b200.config.spec import PartSpec
    from coheryn_ai_studio_b200.parts import model, native_mixer  # noqa: F401
    from coheryn_ai_studio_b200.parts.base import MIXERS, Runtime, build_part
    part = build_part(MIXERS, "mixer", PartSpec(kind, params), Runtime(torch.bfloat16, torch.device(DEV)))
    w = weights(part.tensor_specs(), 3)
    if name is not None:
        w[name] = w[name][:-1].contiguous() if name != "o" else w[name][:, :-8].contiguous()
    part.bind(w)
    return part


@pytest.mark.parametrize("kind,params,name", [(k, p, n) for k, p in CASES for n in
                                              (("norm", "i.b", "f.b", "o", "q", "g") if k == "matrix_memory" else ("norm", "A_log", "dt_bias", "v.conv", "o", "v", "b"))])
def test_weights_of_another_size_are_refused(kind, params, name):
    """... by the operations' own checks, and the library's sequence is not run."""
    from coheryn_ai_studio_b200 import ops
    from coheryn_ai_studio_b200.parts import native_mixer
    from coheryn_ai_studio_b200.parts.base import LayerCache
    part, step, before = broken(kind, params, name), step_of([1, 1]), native_mixer.runs
    assert part.native is None
    state = torch.zeros((2,) + tuple(part.cache_requirement().shape), device=DEV)
    with pytest.raises((AssertionError, ops.KernelError)):
        part.forward(torch.zeros((2, 256), dtype=torch.bfloat16, device=DEV), step, LayerCache("state", state=state))
    assert native_mixer.runs == before


@pytest.mark.parametrize("kind,params", CASES)
def test_states_and_steps_that_do_not_fit_are_refused(kind, params):
    from coheryn_ai_studio_b200 import ops
    from coheryn_ai_studio_b200.parts import native_mixer
    from coheryn_ai_studio_b200.parts.base import LayerCache
    part, before = broken(kind, params, None), native_mixer.runs
    assert part.native is not None
    width = part.cache_requirement().shape[0]
    x = torch.zeros((2, 256), dtype=torch.bfloat16, device=DEV)
    good = torch.zeros((2, width), device=DEV)
    for state in (good[:, :-1], good[:, :width - 4], torch.zeros((2, width + 4), device=DEV), torch.zeros((2, width)), good.bfloat16(), good[:, :part.dk]):
        with pytest.raises((AssertionError, ops.KernelError)):
            part.forward(x, step_of([1, 1]), LayerCache("state", state=state))
    for spoil in ("cu_q", "state_slots", "token_req"):
        if spoil == "token_req" and kind == "matrix_memory":
            continue      # (its operations do not read them)
        step = step_of([1, 1])
        setattr(step, spoil, getattr(step, spoil)[:-1])
        with pytest.raises((AssertionError, ops.KernelError)):
            part.forward(x, step, LayerCache("state", state=good))
    # where the results go: another place, or a host tensor
    for out in (torch.empty((2, 256)), torch.empty((3, 256), device=DEV), torch.empty((2, 256), dtype=torch.bfloat16, device=DEV)):
        assert not part.native.run(x, step_of([1, 1]), good, None, out)
    for opened in (torch.empty((2, params["num_heads"] * params["v_head_dim"]), dtype=torch.bfloat16), torch.empty((2, 8), dtype=torch.bfloat16, device=DEV)):
        assert not part.native.run(x, step_of([1, 1]), good, opened, None)
    assert native_mixer.runs == before
    part.forward(x, step_of([1, 1]), LayerCache("state", state=good))
    assert native_mixer.runs == before + 1


SIZES = [("gated_delta_rule", dict(hidden_size=1536, num_heads=12, num_kv_heads=12, head_dim=128, v_head_dim=128, conv_taps=4, eps=1e-6, decay_rank=64, gate_rank=64)),
         ("gated_delta_rule", dict(hidden_size=2048, num_heads=16, num_kv_heads=16, head_dim=64, v_head_dim=64, conv_taps=4, eps=1e-6, decay="head", low_rank=False,
                                   gate_activation="silu")),
         ("matrix_memory", dict(hidden_size=1536, num_heads=8, head_dim=128, v_head_dim=256, gate_cap=15.0, eps=1e-6))]


@pytest.mark.parametrize("kind,params", SIZES)
@pytest.mark.parametrize("lens", [[1], [1] * 32, [61, 1, 200], [513]])
def test_one_call_equals_the_operations_at_the_models_sizes(kind, params, lens):
    from coheryn_ai_studio_b200 import ops
    from coheryn_ai_studio_b200.parts import native_mixer
    from coheryn_ai_studio_b200.parts.base import LayerCache
    part, step = broken(kind, params, None), step_of(lens)
    g = torch.Generator(device=DEV).manual_seed(len(lens))
    x = torch.randn((step.num_tokens, params["hidden_size"]), device=DEV, generator=g).to(torch.bfloat16)
    first = torch.randn((len(lens),) + tuple(part.cache_requirement().shape), device=DEV, generator=g) * 0.1
    got = []
    for native in (False, True):
        ops.set_native_block(native)
        try:
            before, cache = native_mixer.runs, LayerCache("state", state=first.clone())
            got.append((part.forward(x, step, cache), cache.state))
            assert native_mixer.runs - before == (1 if native else 0)
        finally:
            ops.set_native_block(True)
    for one, other in zip(*got):
        assert torch.isfinite(one).all() and torch.equal(one, other)

"""Which tensors a recurrent mixer may hand to the library's one call (parts/native_mixer.py; no GPU needed): those of the shapes that the part
names, and no others."""
import pytest
import torch

from coheryn_ai_studio_b200.config.spec import PartSpec
from coheryn_ai_studio_b200.parts import model  # noqa: F401  (registers the parts)
from coheryn_ai_studio_b200.parts.base import MIXERS, Runtime, build_part
from coheryn_ai_studio_b200.parts.native_mixer import NativeMixer, shapes_fit

DELTA = dict(hidden_size=64, num_heads=4, num_kv_heads=2, head_dim=8, v_head_dim=16, conv_taps=4, eps=1e-6)


@pytest.mark.parametrize("kind,params", [
    ("gated_delta_rule", DELTA), ("gated_delta_rule", dict(DELTA, decay="head", low_rank=False)),
    ("matrix_memory", dict(hidden_size=64, num_heads=4, head_dim=8, v_head_dim=16, gate_cap=15.0, eps=1e-6))])
def test_shapes(kind, params):
    part = build_part(MIXERS, "mixer", PartSpec(kind, params), Runtime(torch.bfloat16, torch.device("cpu")))
    specs = part.tensor_specs()
    good = {n: torch.zeros([5 if d < 0 else d for d in s.shape], dtype=torch.bfloat16) for n, s in specs.items()}
    assert shapes_fit(specs, good)
    for n, t in good.items():
        for axis in range(t.dim()):
            if specs[n].shape[axis] > 0:
                assert not shapes_fit(specs, dict(good, **{n: t.narrow(axis, 0, t.shape[axis] - 1)})), (n, axis)
        assert not shapes_fit(specs, dict(good, **{n: t.reshape(-1, 1, 1)}))


def test_tensors_on_the_host_are_left_to_the_operations():
    t = torch.zeros((4, 4), dtype=torch.bfloat16)
    assert NativeMixer.build({}, dict(w_in=t, w_o=t, bias_a=t[0], bias_b=t[0], norm_w=t[0]), True, 4) is None

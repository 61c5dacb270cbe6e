"""Whether a step's long runs go in chunks or token by token (csrc/recurrent.cu, coheryn_*_chunks_pay; no GPU needed): at sizes where
both forms were measured (B200), most of them a third apart or more, the choice is the faster one."""
import types

import pytest

from coheryn_ai_studio_b200 import ops


def choice(kind, heads, dk, dv, lens, host=True):
    lib = ops.recurrent()
    step = types.SimpleNamespace(num_requests=len(lens), num_tokens=sum(lens))
    if host:
        step.q_lens = lens
    return ops._chunked_runs(lib, getattr(lib, f"coheryn_{kind}_chunks_pay"), step, sum(lens), heads, dk, dv)


# us by the scan and in chunks
@pytest.mark.parametrize("kind,heads,dk,dv,lens,scan,chunks", [
    ("delta", 12, 128, 128, [48], 72, 97), ("delta", 12, 128, 128, [64], 67, 106), ("delta", 12, 128, 128, [48] * 8, 76, 131),
    ("delta", 12, 128, 128, [64] * 16, 180, 194), ("delta", 12, 128, 128, [512], 312, 130), ("delta", 12, 64, 128, [48] * 32, 145, 196),
    ("delta", 16, 64, 64, [96] * 32, 182, 290), ("delta", 16, 64, 64, [192], 268, 73), ("delta", 4, 32, 64, [48] * 128, 74, 178),
    ("delta", 4, 32, 64, [192] * 4, 217, 71), ("delta", 2, 64, 64, [1] * 64 + [200], 272, 82), ("delta", 12, 128, 128, [1] * 64 + [50] * 3, 145, 180),
    ("memory", 8, 128, 256, [256] * 32, 1344, 455), ("memory", 8, 128, 256, [192], 155, 65), ("memory", 4, 64, 64, [96], 164, 55),
    ("memory", 2, 32, 128, [320], 169, 62), ("memory", 8, 128, 256, [64] * 16, 184, 85), ("memory", 8, 64, 128, [1] * 64 + [400], 631, 88),
    ("memory", 8, 128, 256, [48], 139, 63),
])
def test_the_faster_form_is_taken(kind, heads, dk, dv, lens, scan, chunks):
    got = choice(kind, heads, dk, dv, lens)[0]
    assert (got > 0) == (chunks < scan), (got, scan, chunks)


def test_what_is_cut_into_chunks():
    for lens, cut in (([100, 9, 47, 64], 2), ([100], 1), ([64], 1), ([47], 0)):
        assert choice("delta", 2, 64, 48, lens)[1] == cut
    assert choice("delta", 12, 128, 128, [1021, 407, 130, 2]) == (16 + 7 + 3, 3, True)
    assert choice("delta", 12, 128, 128, [1021, 407]) == (16 + 7, 2, False)
    assert choice("memory", 8, 128, 256, [2048, 47, 48]) == (32 + 1, 2, True)
    chunks, runs, rest = choice("delta", 12, 128, 128, [1021, 407, 130, 2], host=False)       # the lengths are the device's alone
    assert chunks >= 26 and runs >= 3 and rest
    assert choice("delta", 12, 192, 128, [2048]) == (0, 0, True)                              # more key channels than the chunks take
    assert choice("memory", 8, 128, 256, [1] * 64) == (0, 0, True) and choice("delta", 2, 16, 16, []) == (0, 0, True)


def test_the_chunks_scratch_is_bounded():
    """256 MB whatever the step, and what the chunks need below that."""
    import ctypes
    lib = ops.recurrent()
    for f, heads, dk, dv in ((lib.coheryn_delta_chunk_floats, 16, 128, 128), (lib.coheryn_delta_chunk_floats, 2, 20, 30),
                             (lib.coheryn_memory_chunk_floats, 8, 128, 256), (lib.coheryn_memory_chunk_floats, 64, 256, 256)):
        floats = [int(f(*(ctypes.c_int(x) for x in (chunks, heads, dk, dv)))) for chunks in (1, 2, 10000)]
        assert floats[1] == 2 * floats[0] or floats[1] == floats[0] > 1 << 25
        assert floats[2] <= 1 << 26 and floats[2] >= (1 << 26) - floats[0] or floats[2] == 10000 * floats[0]

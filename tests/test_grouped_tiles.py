"""How the routed products cut the groups' rows into tiles (csrc/gemm_tc.cu, GroupCursor; no GPU needed)."""
import ctypes

import pytest

from coheryn_ai_studio_b200 import ops


@pytest.mark.parametrize("counts", [[0, 1, 31, 32, 33, 0], [255, 256, 257, 513], [2048, 2049, 0, 2305, 5000], [0], [64] * 40, list(range(0, 4000, 97))])
def test_groups_are_cut_into_equal_tiles(counts):
    offsets = [sum(counts[:g]) for g in range(len(counts) + 1)]
    room = sum(counts) // 256 + len(counts)
    out = (ctypes.c_int * (4 * room + 4))()
    n = ops.core().coheryn_gemm_tc_grouped_tiles((ctypes.c_int * len(offsets))(*offsets), ctypes.c_int(len(counts)), out, ctypes.c_int(room))
    assert n == sum(-(-c // 256) for c in counts) <= room          # the fewest, and the launch counts on no more
    tiles = [tuple(out[4 * i:4 * i + 4]) for i in range(n)]
    for g, c in enumerate(counts):
        mine = [t for t in tiles if t[0] == g]
        at = offsets[g]
        for _, row0, rows, cols in mine:
            assert row0 == at and 0 < rows <= cols <= 256 and cols % 32 == 0 and cols - rows < 32
            at += rows
        assert at == offsets[g + 1]
        assert len({t[3] for t in mine[:-1]}) <= 1 and all(t[2] == t[3] for t in mine[:-1])      # equal but for the last
    assert [t[0] for t in tiles] == sorted(t[0] for t in tiles)

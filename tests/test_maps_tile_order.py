"""The order in which the row tiles of the attention with score maps start (csrc/attention_maps_tc.cu): every tile once, those that
see the most keys first, whether the prompt fills its chunks, ends inside one or is shorter than one."""
import ctypes

import pytest

from coheryn_ai_studio_b200 import ops

ROWS = 64       # rows of a tile


@pytest.mark.parametrize("chunk", [0, 48, 64, 128, 1024, 1600])
@pytest.mark.parametrize("tiles", [1, 2, 7, 16, 17, 24, 32, 45])
def test_row_tiles_with_the_most_keys_start_first(tiles, chunk):
    lib = ops.maps_attention_lib(64, 128, 2)
    order = (ctypes.c_int * tiles)()
    lib.coheryn_maps_tile_order(ctypes.c_int(tiles), ctypes.c_int(chunk), order)
    order = list(order)
    assert sorted(order) == list(range(tiles))
    # the keys that a tile's last row sees; chunks of less than a row tile hide less than a tile's worth of each other
    keys = [(t + 1) * ROWS if chunk < ROWS else ((t + 1) * ROWS - 1) % chunk + 1 for t in order]
    assert all(a >= b for a, b in zip(keys, keys[1:])), (order, keys)

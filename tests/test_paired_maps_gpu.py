"""Prompt portions of the attention with two maps, where two warps share a row tile's rows: one to many key tiles (the ring of
three), portions that begin inside a row tile, chunks that hold none, one or two row tiles and a remainder, pages of 12
positions, requests of unequal length, heads normalised or not."""
import math

import numpy as np
import pytest
import torch

from test_tutunex_gpu import Paged, bf, plain_maps, write_and_attend

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dk,dv,chunk,page,head_norm", [
    (64, 128, None, 16, True), (64, 128, 130, 12, False), (64, 96, 64, 12, True), (16, 32, 70, 8, True), (48, 64, 40, 16, False),
])
def test_two_maps_in_long_portions(dk, dv, chunk, page, head_norm):
    from coheryn_ai_studio_b200 import ops
    rng = np.random.default_rng(dk + dv)
    heads, G, lam, scale, eps = 4, 2, 0.55, 1.0 / math.sqrt(dk), 1e-5
    lengths = [405, 33, 131]
    seqs = []
    for n in lengths:
        q, k, v = (bf(rng.normal(size=(n, heads * 2 * dk)) * 1.5), bf(rng.normal(size=(n, G * 2 * dk)) * 1.5), bf(rng.normal(size=(n, G * dv))))
        seqs.append((q, k, v, plain_maps(q, k, v, heads, G, dk, dv, 2, scale, lam, chunk, False, head_norm, eps, 0.7)))
    cache = Paged(lengths, G, 2 * dk, dv, page, torch.bfloat16, seed=dk)
    for portion in ([(0, 0, 300), (1, 0, 32), (2, 0, 2)], [(0, 300, 105), (2, 2, 129)]):
        step = cache.step(portion)
        rows = lambda i: np.concatenate([seqs[r][i][a:a + n] for r, a, n in portion])
        got = write_and_attend(cache, step, rows(0), rows(1), rows(2), heads, dk, 2, ops, chunk=chunk, sink=False, scale=scale, lam=lam,
                               head_norm=head_norm, out_scale=0.7, eps=eps)
        # results are rounded to bfloat16 (8 significant bits: 2^-8); the weights are held to 2^-16 and sums to float32, which
        # a norm of the heads enlarges by the reciprocal of their root mean square (not above 30 here)
        assert (np.abs(got - rows(3)) <= 2.0 ** -8 * np.abs(rows(3)) + 30 * 2.0 ** -15).all(), np.abs(got - rows(3)).max()


def test_normalised_heads_of_short_row_tiles_repeat_to_the_bit():
    """Row tiles whose first warps are the last to work: 2 to 47 rows behind 0 to 96 earlier positions, so that some pairs of warps
    have no row (or no key of the last key tile) and exchange their sums of squares while another pair still exchanges the last
    tile's weights.  Forty launches give the same bits, and those of the plain attention within its bound."""
    from coheryn_ai_studio_b200 import ops
    rng = np.random.default_rng(11)
    dk, dv, heads, G, lam, eps, page = 64, 128, 12, 2, 0.55, 1e-5, 16
    scale = 1.0 / math.sqrt(dk)
    runs = [(0, 2), (32, 16), (64, 17), (96, 5), (32, 32), (0, 33), (64, 47), (96, 24)]
    lengths = [first + n for first, n in runs]
    seqs = []
    for n in lengths:
        q, k, v = (bf(rng.normal(size=(n, heads * 2 * dk)) * 1.5), bf(rng.normal(size=(n, G * 2 * dk)) * 1.5), bf(rng.normal(size=(n, G * dv))))
        seqs.append((q, k, v, plain_maps(q, k, v, heads, G, dk, dv, 2, scale, lam, None, False, True, eps, 0.7)))
    cache = Paged(lengths, G, 2 * dk, dv, page, torch.bfloat16, seed=3)
    for portion in ([(r, 0, first) for r, (first, _) in enumerate(runs) if first], [(r, first, n) for r, (first, n) in enumerate(runs)]):
        rows = lambda i: np.concatenate([seqs[r][i][a:a + n] for r, a, n in portion])
        step, want = cache.step(portion), None
        for _ in range(40):
            got = write_and_attend(cache, step, rows(0), rows(1), rows(2), heads, dk, 2, ops, sink=False, scale=scale, lam=lam,
                                   head_norm=True, out_scale=0.7, eps=eps)
            want = got if want is None else want
            assert np.array_equal(got, want)
        # (the bound of the test above)
        assert (np.abs(got - rows(3)) <= 2.0 ** -8 * np.abs(rows(3)) + 30 * 2.0 ** -15).all(), np.abs(got - rows(3)).max()

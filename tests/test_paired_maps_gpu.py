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

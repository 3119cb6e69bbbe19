"""Segment adjacency at the edges of its per-tile pair sets: whole and ragged
tiles, sets that fill up (every pixel its own segment), and labels at the ends
of the int range; equal to the oracle."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape,low,high", [
    ((32, 64), 0, 3), ((33, 65), 0, 40), ((31, 63), -5, 5),
    ((64, 128), 0, 1 << 20),                 # more pairs than a tile's set holds
    ((96, 200), -(1 << 31), (1 << 31) - 1),
    ((1, 300), 0, 2), ((300, 1), 0, 2), ((2, 2), 0, 1), ((1, 1), 7, 7),
    ((40, 70), 9, 9)])                       # one segment: no pair
def test_pairs_of_tiles(cuda, shape, low, high):
    import torch
    from split_gb300 import ccl
    h, w = shape
    lab = np.random.default_rng(h * 1000 + w).integers(low, high, size=shape, endpoint=True)
    lab = lab.astype(np.int32)
    keys = torch.full((8 * h * w,), -77, dtype=torch.int32, device=cuda)
    adj = torch.full((8 * h * w,), -77, dtype=torch.int32, device=cuda)
    n = ccl.segment_adjacency(torch.from_numpy(lab).to(cuda), keys, adj)
    rk, ra = oracle.segment_adjacency(lab)
    assert n == len(rk)
    assert np.array_equal(keys.cpu().numpy()[:n], rk)
    assert np.array_equal(adj.cpu().numpy()[:n], ra)
    assert (keys.cpu().numpy()[n:] == -77).all()   # nothing past the pairs

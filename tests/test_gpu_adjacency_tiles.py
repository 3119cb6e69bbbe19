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


@pytest.mark.parametrize("shape,cell", [
    ((12, 12), 1), ((12, 13), 1),            # 1012 and 1102 keys: one sorted tile, two
    ((200, 300), 60),                        # few pairs, each from several tiles
    ((300, 500), 3),                         # 16700 segments, pairs that tiles share
    ((128, 129), 1), ((129, 129), 1)])       # 130558 keys are ranked, 131584 sorted by digits
def test_ranked_and_sorted_keys(cuda, shape, cell):
    import torch
    from split_gb300 import ccl
    h, w = shape
    y, x = np.mgrid[0:h, 0:w]
    ids = np.random.default_rng(cell).permutation(h * w).astype(np.int32) - 500
    lab = ids[y // cell * w + x // cell]
    keys = torch.full((8 * h * w,), -77, dtype=torch.int32, device=cuda)
    adj = torch.full((8 * h * w,), -77, dtype=torch.int32, device=cuda)
    ws = None
    for _ in range(2):
        ws = ccl.Workspace(ccl.segment_adjacency_workspace(w, h), cuda) if ws is None else ws
        n = ccl.segment_adjacency(torch.from_numpy(lab).to(cuda), keys, adj, ws)
        rk, ra = oracle.segment_adjacency(lab)
        assert n == len(rk)
        assert np.array_equal(keys.cpu().numpy()[:n], rk)
        assert np.array_equal(adj.cpu().numpy()[:n], ra)
    assert (keys.cpu().numpy()[n:] == -77).all()

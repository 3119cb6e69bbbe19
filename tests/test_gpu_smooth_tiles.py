"""Smooth-boundary merge at the edges of its tiles and of their pair tables:
whole and ragged tiles, labels addressed at odd bytes of a line, more pairs
than a tile's table holds, one segment; equal to the oracle, twice through one
workspace."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape,block,salt,offset", [
    ((32, 64), 16, 0.0, 0), ((33, 65), 12, 0.0, 1), ((31, 63), 9, 0.0, 3),
    ((70, 130), 33, 0.0, 2), ((96, 200), 7, 0.0, 0),
    ((64, 128), 32, 0.2, 0), ((65, 131), 40, 0.3, 2),   # single pixels: 1000 pairs a tile
    ((1, 300), 40, 0.0, 0), ((300, 1), 40, 0.0, 1), ((1, 1), 1, 0.0, 0), ((40, 70), 99, 0.0, 0)])
def test_merge_over_tiles(cuda, shape, block, salt, offset):
    import torch
    from split_gb300 import ccl
    h, w = shape
    rng = np.random.default_rng(100 * h + w)
    y, x = np.mgrid[0:h, 0:w]
    seg = (y // block * block * w + x // block * block).astype(np.int32)
    base = seg
    seg = np.where(rng.random((h, w)) < salt, y * w + x, seg).astype(np.int32)
    # classes whose mutual boundaries are smooth, other boundaries sharp
    pts = (rng.integers(0, 3, size=h * w)[base.ravel()] * 0.4
           + rng.random((3, h * w)) * 0.02).astype(np.float32)
    buf = torch.empty(h * w + 4, dtype=torch.int32, device=cuda)
    got = buf[offset:offset + h * w].view(h, w)
    got.copy_(torch.from_numpy(seg))
    dev = torch.from_numpy(pts).to(cuda)
    ws, ref = None, seg
    for threshold in (0.05, 2.0):
        ref = oracle.merge_smooth(ref, pts, threshold)
        ws = ccl.merge_smooth_boundaries(dev, 0, got, ws, threshold)
        ws.check("merge_smooth")
        assert np.array_equal(got.cpu().numpy(), ref)


def test_workspace_across_sizes(cuda):
    """One workspace for images of different sizes, back and forth."""
    import torch
    from split_gb300 import ccl
    ws = ccl.Workspace(ccl.merge_smooth_boundaries_workspace(300, 200), cuda)
    for w, h in ((300, 200), (70, 50), (290, 190), (300, 200), (128, 64), (300, 200)):
        rng = np.random.default_rng(w)
        y, x = np.mgrid[0:h, 0:w]
        seg = (y // 9 * 9 * w + x // 9 * 9).astype(np.int32)
        pts = (rng.integers(0, 3, size=h * w)[seg.ravel()] * 0.4
               + rng.random((3, h * w)) * 0.02).astype(np.float32)
        got = torch.from_numpy(seg).to(cuda)
        ccl.merge_smooth_boundaries(torch.from_numpy(pts).to(cuda), 0, got, ws, 0.05)
        ws.check("merge_smooth")
        assert np.array_equal(got.cpu().numpy(), oracle.merge_smooth(seg, pts, 0.05)), (w, h)


@pytest.mark.parametrize("shape,block", [((20, 20), 1), ((48, 64), 3), ((33, 130), 2)])
def test_more_pairs_than_a_tile_holds(cuda, shape, block):
    """Tiles that fill their table several times over."""
    import torch
    from split_gb300 import ccl
    h, w = shape
    rng = np.random.default_rng(h + w)
    y, x = np.mgrid[0:h, 0:w]
    seg = (y // block * block * w + x // block * block).astype(np.int32)
    seg[:, : w // 4] = 0     # and one large segment with many neighbours
    pts = rng.random((3, h * w)).astype(np.float32)
    got = torch.from_numpy(seg).to(cuda)
    ws = ccl.merge_smooth_boundaries(torch.from_numpy(pts).to(cuda), 0, got, None, 2.0)
    ws.check("merge_smooth")
    assert np.array_equal(got.cpu().numpy(), oracle.merge_smooth(seg, pts, 2.0))


def test_after_a_refused_call(cuda):
    """More pairs than the global table holds is an error; the workspace is then as
    good as new."""
    import torch
    from split_gb300 import ccl
    from split_gb300._native import SplitError
    h, w = 48, 64
    pts = torch.rand((3, h * w), device=cuda)
    seg = torch.arange(h * w, dtype=torch.int32, device=cuda).view(h, w)
    ws = ccl.merge_smooth_boundaries(pts, 0, seg.clone(), None, 0.5)
    with pytest.raises(SplitError):
        ws.check("merge_smooth")
    y, x = np.mgrid[0:h, 0:w]
    lab = (y // 8 * 8 * w + x // 8 * 8).astype(np.int32)
    got = torch.from_numpy(lab).to(cuda)
    ccl.merge_smooth_boundaries(pts, 0, got, ws, 2.0)
    ws.check("merge_smooth")
    assert np.array_equal(got.cpu().numpy(), oracle.merge_smooth(lab, pts.cpu().numpy(), 2.0))

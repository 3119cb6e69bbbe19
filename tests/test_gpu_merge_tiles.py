"""Small-segment merge at the edges of its per-tile tables: segments inside a
tile (decided there), across tiles (global table), more segments or pairs than
a tile's tables hold, and workspaces used twice; bit-exact against the
oracle."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("policy", [0, 1])
@pytest.mark.parametrize("shape,block,values,P", [
    ((32, 64), 1, 3, 50),       # one tile of speckle
    ((32, 64), 1, 1000, 2),     # more single-pixel segments than the tile's table holds
    ((33, 65), 2, 40, 6),       # the last tiles are one pixel wide or high
    ((64, 128), 2, 1000, 6),    # more pairs than the decision launch's tables hold
    ((200, 330), 3, 5, 30),     # mixed sizes, many inside their tiles
    ((200, 330), 1, 60, 9),     # pair tables nearly full
    ((256, 320), 40, 9, 2000),  # every segment crosses tiles
    ((1, 500), 1, 4, 3), ((500, 1), 1, 4, 3)])
def test_merge_tile_tables(cuda, policy, shape, block, values, P):
    import torch
    from split_gb300 import ccl
    h, w = shape
    rng = np.random.default_rng(h * 7 + w + block)
    ws = None
    for k in range(2):   # the second call finds the workspace as the first left it
        lab = rng.integers(0, values, size=(h // block + 1, w // block + 1))
        lab = np.ascontiguousarray(lab.repeat(block, 0).repeat(block, 1)[:h, :w]).astype(np.int32)
        lab[:, : w // 3] = 0 if k else lab[:, : w // 3]   # a large segment beside the speckle
        seg = oracle.ccl(lab, 8 if k else 4, k)
        chroma = (rng.integers(0, 256, size=(2, h * w)) / 256.0).astype(np.float32)
        want = oracle.merge_small(seg, P, policy, chroma)
        g = torch.from_numpy(seg).to(cuda)
        ws = ccl.merge_small_segments(torch.from_numpy(chroma).to(cuda), g, ws, P, policy=policy)
        torch.cuda.synchronize()
        ws.check("merge")
        assert np.array_equal(g.cpu().numpy(), want), k


@pytest.mark.parametrize("policy", [0, 1])
def test_merge_overflow_from_dense_tiles(cuda, policy):
    """The pair pass leaves every tile to the decision launch, whose sixteen
    blocks then overflow the global table: all of them have to go on to the
    class-by-class decision together."""
    import torch
    from split_gb300 import ccl
    h, w, block, P = 256, 512, 2, 6
    rng = np.random.default_rng(11 + policy)
    lab = rng.integers(0, 1000, size=(h // block, w // block))
    seg = oracle.ccl(np.ascontiguousarray(lab.repeat(block, 0).repeat(block, 1)).astype(np.int32),
                     8, 0)
    chroma = (rng.integers(0, 256, size=(2, h * w)) / 256.0).astype(np.float32)
    want = oracle.merge_small(seg, P, policy, chroma)
    ws = None
    for k in range(3):
        g = torch.from_numpy(seg).to(cuda)
        ws = ccl.merge_small_segments(torch.from_numpy(chroma).to(cuda), g, ws, P, policy=policy)
        torch.cuda.synchronize()
        ws.check("merge")
        assert np.array_equal(g.cpu().numpy(), want), k


@pytest.mark.parametrize("policy", [0, 1])
@pytest.mark.parametrize("step,P", [(2, 1 << 20), (3, 1 << 20), (2, 2)])
def test_merge_many_neighbours(cuda, policy, step, P):
    """Backgrounds that are themselves below P and border tens of thousands of
    single pixels: thousands of pairs of one segment in the global table."""
    import torch
    from split_gb300 import ccl
    h, w = 900, 777
    y, x = np.mgrid[0:h, 0:w]
    base = np.where(x < w // 2, 0, w // 2)   # two backgrounds side by side
    lab = np.where((y % step == 1) & (x % step == 1), y * w + x, base).astype(np.int32)
    rng = np.random.default_rng(step)
    chroma = (rng.integers(0, 256, size=(2, h * w)) / 256.0).astype(np.float32)
    want = oracle.merge_small(lab, P, policy, chroma)
    g = torch.from_numpy(lab).to(cuda)
    ws = ccl.merge_small_segments(torch.from_numpy(chroma).to(cuda), g, None, P, policy=policy)
    torch.cuda.synchronize()
    ws.check("merge")
    assert np.array_equal(g.cpu().numpy(), want)


@pytest.mark.parametrize("policy", [0, 1])
def test_merge_after_refused_call(cuda, policy):
    """A call that gives up leaves nothing behind for the next one."""
    import torch
    from split_gb300 import ccl
    from split_gb300._native import SplitError
    h, w = 64, 128
    y, x = np.mgrid[0:h, 0:w]
    rng = np.random.default_rng(5)
    chroma = (rng.integers(0, 256, size=(2, h * w)) / 256.0).astype(np.float32)
    ch = torch.from_numpy(chroma).to(cuda)
    # one segment on half of the pixels, every other pixel its own: more pairs of
    # one segment than half the table
    many = np.where((x + y) % 2 == 1, y * w + x, 0).astype(np.int32)
    g = torch.from_numpy(many).to(cuda)
    ws = ccl.merge_small_segments(ch, g, None, h * w + 1, policy=policy)
    with pytest.raises(SplitError):
        ws.check("merge")
    seg = oracle.ccl(rng.integers(0, 3, size=(h, w)).astype(np.int32), 4, 0)
    want = oracle.merge_small(seg, 9, policy, chroma)
    g = torch.from_numpy(seg).to(cuda)
    ccl.merge_small_segments(ch, g, ws, 9, policy=policy)
    ws.check("merge")
    assert np.array_equal(g.cpu().numpy(), want)

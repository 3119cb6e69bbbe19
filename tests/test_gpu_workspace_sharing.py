"""One workspace used by different calls in turn: the two merges, which keep
state between calls, find it again or clear what another call has left."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu

W, H = 160, 96
OTHERS = ["adjacency", "edges", "compress", "label", "cluster", "cluster_wide", "assign", "update",
          "update_wide", "shading", "lab_beta", "pipeline", "smooth", "small", "smooth_size", "small_size"]


class Shared:
    def __init__(self, cuda):
        import torch
        from split_gb300 import ccl, kmeans, pipeline
        self.cuda, n = cuda, W * H
        self.rng = np.random.default_rng(3)
        self.rgb = torch.from_numpy(self.rng.integers(0, 256, (H, W, 3)).astype(np.uint8)).to(cuda)
        self.pipe = pipeline.Pipeline(W, H, pipeline.Params(nclusters=8, kmeans_iters=2,
                                                            merge_P=20), cuda)
        need = max(ccl.segment_adjacency_workspace(W, H), self.pipe.ws.nbytes,
                   kmeans.calculate_centroids_workspace(n, n, 3),
                   kmeans.cluster_workspace_2d(n, W, 100, 5),
                   ccl.merge_smooth_boundaries_workspace(W, H),
                   ccl.merge_small_segments_workspace(W, H))
        self.ws = ccl.Workspace(need, cuda)

    def smooth(self, w=W, h=H):
        import torch
        from split_gb300 import ccl
        y, x = np.mgrid[0:h, 0:w]
        seg = (y // 9 * 9 * w + x // 9 * 9).astype(np.int32)
        pts = (self.rng.integers(0, 3, size=h * w)[seg.ravel()] * 0.4
               + self.rng.random((3, h * w)) * 0.02).astype(np.float32)
        got = torch.from_numpy(seg).to(self.cuda)
        ccl.merge_smooth_boundaries(torch.from_numpy(pts).to(self.cuda), 0, got, self.ws, 0.05)
        self.ws.check("merge_smooth")
        assert np.array_equal(got.cpu().numpy(), oracle.merge_smooth(seg, pts, 0.05))

    def small(self, w=W, h=H):
        import torch
        from split_gb300 import ccl
        lab = self.rng.integers(0, 3, size=(h, w)).astype(np.int32)
        lab[h // 2:] //= 2
        seg = oracle.ccl(lab, 4, 0)
        got = torch.from_numpy(seg).to(self.cuda)
        ccl.merge_small_segments(None, got, self.ws, 12, policy=ccl.MOST_BOUNDARY)
        self.ws.check("merge_small")
        assert np.array_equal(got.cpu().numpy(), oracle.merge_small(seg, 12, 0))

    def call(self, name):
        """One call of another entry point through the workspace."""
        import torch
        from split_gb300 import ccl, color, kmeans, sfs
        n, d, ws = W * H, self.cuda, self.ws
        many = torch.arange(n, dtype=torch.int32, device=d).view(H, W)
        ints = lambda m: torch.empty(m * n, dtype=torch.int32, device=d)
        how = dict(layout=kmeans.RGB8, dim=5, width=W)
        if name == "adjacency":
            ccl.segment_adjacency(many, ints(8), ints(8), ws)
        elif name == "edges":
            ccl.segment_adjacency_edges(many, ints(16), ws)
        elif name == "compress":
            ccl.compress_labels(many.clone(), ws)
        elif name == "label":
            ccl.connected_components(many, ws, torch.empty_like(many), connectivity=8)
        elif name in ("cluster", "cluster_wide", "assign"):
            c = torch.rand((5, 100 if name == "cluster_wide" else 8), device=d)
            lab = torch.empty(n, dtype=torch.int32, device=d)
            if name == "assign":
                kmeans.label_points(c, self.rgb, lab, ws, **how)
            else:
                kmeans.cluster(self.rgb, c, lab, ws, 3, -1.0, **how)
        elif name in ("update", "update_wide"):
            k = 8 if name == "update" else n
            kmeans.calculate_centroids(many.view(-1) % k, torch.rand((3, n), device=d),
                                       torch.zeros((3, k), device=d), ws, dim=3, width=W)
        elif name == "shading":
            sfs.estimate_normals(torch.rand((H, W), device=d), (0.3, 0.2, 1.0),
                                 torch.empty((3, n), device=d), 1.0, max_iter=3, temp=ws)
        elif name == "lab_beta":
            color.pack_lab_beta(self.rgb, torch.empty((3, n), device=d), temp=ws)
        elif name == "pipeline":
            self.pipe.ws = ws
            self.pipe.run(self.rgb, torch.rand((5, 8), device=d))
        elif name.startswith("smooth"):
            self.smooth(*((70, 50) if name.endswith("size") else (W, H)))
        elif name.startswith("small"):
            self.small(*((70, 50) if name.endswith("size") else (W, H)))
        torch.cuda.synchronize()


@pytest.mark.parametrize("other", OTHERS)
def test_merges_after_other_calls(cuda, other):
    s = Shared(cuda)
    for merge in (s.smooth, s.small, s.smooth, s.smooth, s.small, s.small):
        merge()
        s.call(other)
        merge()


def test_smooth_call_numbers_run_out(cuda):
    """The number that marks a call's results starts again after 2^32 calls."""
    import torch
    s = Shared(cuda)
    s.smooth()
    # the header: status, barrier (2), counter (2), result, stamp (2), call number
    s.ws.view[:256].view(torch.int32)[8] = -3
    for _ in range(4):
        s.smooth()


def test_batches_in_turn_in_one_arena(cuda):
    """Two layouts, one of them twice in a row, and another call in between, in one
    arena: every batch's segments are those of fresh buffers."""
    import torch
    from split_gb300 import batch, ccl, pipeline
    params = pipeline.Params(merge_P=40, xy_scale=0.01)
    shapes = [[(200, 150, 8, 3), (90, 70, 4, 2)], [(120, 110, 8, 3)]]
    rng = np.random.default_rng(9)
    imgs = [[rng.integers(0, 256, (h, w, 3)).astype(np.uint8) for w, h, _, _ in s] for s in shapes]
    cents = [[rng.random((5, k)).astype(np.float32) for _, _, k, _ in s] for s in shapes]

    def run(i, arena):
        b = batch.Batch(shapes[i], params, cuda, arena=arena)
        b.load(imgs[i], cents[i])
        b.run()
        torch.cuda.synchronize()
        b.ws.check("batch")
        return [b.segment_labels_of(k).clone() for k in range(len(shapes[i]))]

    want = [run(i, None) for i in range(2)]
    arena = batch.Arena(cuda)
    run(0, arena)
    lab = torch.arange(60 * 60, dtype=torch.int32, device=cuda).view(60, 60)
    out = [torch.empty(8 * 3600, dtype=torch.int32, device=cuda) for _ in range(2)]
    for i in (0, 1, 0, 0, -1, 0, 1, -1, 1, 1, 0):
        if i < 0:
            need = ccl.segment_adjacency_workspace(60, 60)
            ccl.segment_adjacency(lab, *out, ccl.Workspace.over(arena.ws_buf, need))
            continue
        for got, ref in zip(run(i, arena), want[i]):
            assert torch.equal(got, ref)

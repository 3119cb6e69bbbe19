"""Performance cases of the segmentation framework.

Each case is one piece of work that a program does through the public entry
points: whole frames through the pipeline (single, captured, batched, served),
and the single stages a program calls by themselves (clustering of planar
features, large palettes, stress labellings, segment rendering, region graphs,
shape from shading).  Sizes come from the framework's own configurations,
tests and benchmark.  `listed()` names them, `draw()` gives more of the same
ranges, `prepare()` makes what a program holds before the call, `run()` is one
pass, `work()` the bytes and operations that pass cannot do without and
`exact()` the floating outputs in 64 bits.
"""
from __future__ import annotations

import math
import random

import torch

from split_gb300 import batch, ccl, kmeans, pipeline, serve, sfs, synth
from split_gb300._util import Workspace

XY = 0.1   # xy_scale of the 5-D features everywhere
LAB_BETA = 3   # pipeline features: the sample's (beta, a*, b*)


# ------------------------------------------------------------------ the cases
def listed():
    return [
        # One photograph-sized frame, the benchmark's configuration: 16
        # clusters over colour and position, 8-connected, merge below 256 px,
        # 3x3 erosion, normals.  What a single-image user runs.
        dict(name="frame_4k", kind="frame", width=3840, height=2160, cells=256, palette=16,
             k=16, dim=5, iters=20, conn=8, max_index=False, merge_p=256, chroma=False,
             erode=1, normals=True, features=1, captured=False),
        # A thumbnail replayed from its captured graph (previews, video at low
        # resolution): the smallest frame, where launches and latency are all.
        dict(name="frame_thumb", kind="frame", width=160, height=128, cells=12, palette=0,
             k=4, dim=5, iters=10, conn=8, max_index=False, merge_p=64, chroma=False,
             erode=1, normals=True, features=1, captured=True),
        # The plain 512x512 configuration: 8 clusters over colour alone, 10
        # iterations, 4-connected, merge below 64 px, labels only.
        dict(name="frame_512", kind="frame", width=512, height=512, cells=32, palette=0,
             k=8, dim=3, iters=10, conn=4, max_index=False, merge_p=64, chroma=False,
             erode=0, normals=False, features=1, captured=False),
        # The reference sample's own settings on an odd-sized image: Lab + beta
        # features, maximum-index 4-connected labels, nearest-chroma merge,
        # erosion by 10.
        dict(name="frame_sample", kind="frame", width=1283, height=957, cells=96, palette=0,
             k=10, dim=3, iters=15, conn=4, max_index=True, merge_p=100, chroma=True,
             erode=10, normals=True, features=LAB_BETA, captured=False),
        # An offline job over a folder of uneven images: sides 128 to 2048,
        # K from {4, 8, 16, 32}, 10 to 20 iterations, one launch sequence.
        dict(name="batch_48", kind="batch", images=48, mix=48, side_min=128, side_max=2048),
        # A burst of requests at the continuous-batching server, host memory
        # to host memory: sides log-uniform in [256, 2048].
        dict(name="serve_burst", kind="serve", images=12, mix=12, side_min=256, side_max=2048),
        # The labelling and merge stress: a maze with one serpentine component
        # and about 10^5 blobs, labels given.  The largest call.
        dict(name="maze_8k", kind="maze", width=8192, height=8192, conn=8, merge_p=64),
        # A drop-in caller of the reference's kmeans::cluster: planar float
        # colour features, an odd-sized 720p frame.
        dict(name="cluster_planar", kind="planar", width=1279, height=719, cells=64, k=24,
             iters=15),
        # A large palette (256 clusters) learned on one 1440p frame and applied
        # to the next one (label_points).
        dict(name="palette_256", kind="palette", width=2560, height=1440, cells=256, k=256,
             dim=5, iters=10),
        # The sample's render step on a fragmented 1080p segmentation:
        # compress the segment labels, take each segment's mean colour, paint.
        dict(name="render_1080p", kind="render", width=1920, height=1080, cells=3000,
             speckle=0.01),
        # Region graph of a 1080p labelling: merge across smooth boundaries,
        # then the sorted adjacency of the segments that are left.
        dict(name="regions_1080p", kind="regions", width=1920, height=1080, cells=400,
             speckle=0.002, threshold=0.05),
        # Shape from shading of a VGA image to the reference's tolerance and
        # sweep limit: the iterative solver, one long latency-bound call.
        dict(name="shading_vga", kind="shading", width=640, height=480, smoothness=1.0,
             max_iter=1500),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["frame", "frame", "frame", "sample", "batch", "serve", "maze", "planar",
                       "palette", "render", "regions", "shading"])
    if kind == "frame":
        w, h = _log(rng, 128, 3840), _log(rng, 128, 2160)
        px = w * h
        full = rng.random() < 0.7
        return dict(kind="frame", width=w, height=h, cells=max(8, min(256, px // 8000)),
                    palette=rng.choice([0, 16]), k=rng.choice([4, 8, 16, 32]),
                    dim=rng.choice([3, 5, 5]), iters=rng.randint(10, 20),
                    conn=rng.choice([4, 8]), max_index=False,
                    merge_p=rng.choice([64, 256]), chroma=False, erode=1 if full else 0,
                    normals=full, features=rng.choice([1, 1, 2]),
                    captured=rng.random() < 0.5)
    if kind == "sample":
        w, h = _log(rng, 200, 2200), _log(rng, 200, 1600)
        return dict(kind="frame", width=w, height=h, cells=rng.randint(24, 160), palette=0,
                    k=rng.randint(6, 16), dim=3, iters=rng.randint(8, 20), conn=4,
                    max_index=True, merge_p=100, chroma=True, erode=rng.randint(2, 12),
                    normals=True, features=LAB_BETA, captured=False)
    if kind == "batch":
        return dict(kind="batch", images=_log(rng, 3, 48), mix=rng.randrange(1 << 20),
                    side_min=128, side_max=rng.choice([512, 1024, 2048]))
    if kind == "serve":
        return dict(kind="serve", images=_log(rng, 1, 12), mix=rng.randrange(1 << 20),
                    side_min=256, side_max=2048)
    if kind == "maze":
        return dict(kind="maze", width=_log(rng, 500, 8192), height=_log(rng, 500, 8192),
                    conn=rng.choice([4, 8]), merge_p=rng.choice([16, 64, 256]))
    if kind == "planar":
        return dict(kind="planar", width=_log(rng, 100, 2560), height=_log(rng, 100, 1440),
                    cells=rng.randint(16, 128), k=rng.randint(3, 64), iters=rng.randint(5, 20))
    if kind == "palette":
        return dict(kind="palette", width=_log(rng, 256, 2560), height=_log(rng, 256, 1440),
                    cells=256, k=rng.randint(65, 512), dim=rng.choice([3, 5]),
                    iters=rng.randint(3, 10))
    if kind == "render":
        return dict(kind="render", width=_log(rng, 200, 3840), height=_log(rng, 200, 2160),
                    cells=rng.randint(20, 3000), speckle=rng.choice([0.0, 0.002, 0.02]))
    if kind == "regions":
        return dict(kind="regions", width=_log(rng, 200, 1920), height=_log(rng, 200, 1080),
                    cells=rng.randint(20, 600), speckle=rng.choice([0.0, 0.002, 0.01]),
                    threshold=0.05)
    return dict(kind="shading", width=_log(rng, 64, 1280), height=_log(rng, 64, 720),
                smoothness=rng.choice([0.3, 1.0, 3.0]), max_iter=rng.choice([200, 400]))


# ------------------------------------------------------------------ inputs
def _dev():
    return torch.device("cuda", torch.cuda.current_device())


def _gen(seed):
    g = torch.Generator(device=_dev())
    g.manual_seed(int(seed))
    return g


def _cells(g, w, h, cells):
    """Voronoi partition: (H, W) index of the nearest of `cells` random sites."""
    d = _dev()
    cx = torch.rand(cells, generator=g, device=d) * w
    cy = torch.rand(cells, generator=g, device=d) * h
    dx = (torch.arange(w, device=d, dtype=torch.float32)[:, None] - cx[None]).square()
    dy = (torch.arange(h, device=d, dtype=torch.float32)[:, None] - cy[None]).square()
    out = torch.empty((h, w), dtype=torch.int64, device=d)
    step = max(1, (1 << 27) // max(1, w * cells))
    for r in range(0, h, step):
        out[r:r + step] = (dy[r:r + step, None, :] + dx[None]).argmin(-1)
    return out


def _image(g, w, h, cells, palette=0, gradient=False, sigma=4.0):
    """RGB8 photograph stand-in: flat-coloured cells, optional palette and
    illumination gradient, Gaussian sensor noise."""
    d = _dev()
    idx = _cells(g, w, h, cells)
    if palette:
        colours = torch.rand((palette, 3), generator=g, device=d) * 255.0
        colour = colours[torch.randint(palette, (cells,), generator=g, device=d)]
    else:
        colour = torch.rand((cells, 3), generator=g, device=d) * 255.0
    img = colour[idx]
    if gradient:
        img = img * torch.linspace(0.6, 1.0, w, device=d)[None, :, None]
    img = img + torch.randn(img.shape, generator=g, device=d) * sigma
    return img.round().clamp(0, 255).to(torch.uint8).contiguous()


def _picks(g, rgb, k, dim):
    """Initial centroids: the features of k random pixels, planar (dim, k)."""
    h, w = rgb.shape[:2]
    at = torch.randint(h * w, (k,), generator=g, device=rgb.device)
    c = [rgb.reshape(-1, 3)[at, j].float() / 255.0 for j in range(3)]
    if dim == 5:
        c += [XY * (at % w).float(), XY * (at // w).float()]
    return torch.stack(c).contiguous()


def _lab64(rgb):
    """(L*, a*, b*) of (H, W, 3) bytes clamped to >= 1/255, in 64 bits."""
    v = (rgb.double() / 255.0).clamp_min(1.0 / 255.0)
    lin = torch.where(v > 0.04045, ((v + 0.055) / 1.055) ** 2.4, v / 12.92) * 100.0
    m = torch.tensor([[0.4124564, 0.3575761, 0.1804375], [0.2126729, 0.7151522, 0.0721750],
                      [0.0193339, 0.1191920, 0.9503041]], dtype=torch.float64, device=rgb.device)
    white = torch.tensor([95.047, 100.0, 108.883], dtype=torch.float64, device=rgb.device)
    t = lin @ m.T / white
    f = torch.where(t > 0.008856, t.clamp_min(1e-30) ** (1.0 / 3.0), 7.787 * t + 16.0 / 116.0)
    return 116.0 * f[..., 1] - 16.0, 500.0 * (f[..., 0] - f[..., 1]), 200.0 * (f[..., 1] - f[..., 2])


def _segments(g, w, h, cells, speckle):
    """A fragmented labelling as connected_components gives it: every segment
    named by its smallest pixel index, `speckle` of the pixels their own."""
    d = _dev()
    n = w * h
    idx = _cells(g, w, h, cells).view(-1)
    pix = torch.arange(n, device=d)
    single = torch.rand(n, generator=g, device=d) < speckle
    idx = torch.where(single, cells + pix, idx)
    first = torch.full((cells + n,), n, dtype=torch.int64, device=d)
    first.scatter_reduce_(0, idx, pix, "amin")
    return first[idx].to(torch.int32)


def _shapes(case):
    """(width, height, K, iterations) of a mix of images: part of the case."""
    rng = random.Random(case["mix"])
    lo, hi = case["side_min"], case["side_max"]
    if case["kind"] == "batch":
        return [(rng.randint(lo, hi), rng.randint(lo, hi), rng.choice([4, 8, 16, 32]),
                 rng.randint(10, 20)) for _ in range(case["images"])]
    return [(_log(rng, lo, hi), _log(rng, lo, hi), rng.choice([8, 16, 32]), 20)
            for _ in range(case["images"])]


def _params(case):
    return pipeline.Params(
        nclusters=case["k"], dim=case["dim"], xy_scale=XY, kmeans_iters=case["iters"],
        features=case["features"], connectivity=case["conn"],
        convention=ccl.MAX_INDEX if case["max_index"] else ccl.MIN_INDEX,
        merge_P=case["merge_p"], merge_policy=ccl.REF_CHROMA if case["chroma"] else
        ccl.MOST_BOUNDARY, erode_radius=case["erode"], compute_normals=case["normals"])


def prepare(case, seed):
    g = _gen(seed)
    d = _dev()
    kind = case["kind"]
    s = {"case": case, "kind": kind}
    if kind in ("batch", "serve"):
        shapes = _shapes(case)
        imgs = [_image(g, w, h, 32) for w, h, _, _ in shapes]
        cents = [_picks(g, im, k, 5) for im, (_, _, k, _) in zip(imgs, shapes)]
        s["images"], s["centroids0"], s["shapes"] = imgs, cents, shapes
        if kind == "batch":
            b = batch.Batch(shapes, pipeline.Params(), d)
            for i, (im, c) in enumerate(zip(imgs, cents)):
                b.rgb_of(i).copy_(im)
                b.centroids_of(i).copy_(c)
            s["batch"], s["c0"] = b, b.centroids.clone()
        else:
            px = sum((w * h + 63) // 64 * 64 for w, h, _, _ in shapes)
            s["server"] = serve.Server(pipeline.Params(compute_normals=False), device=d,
                                       reserve_pixels=px)
            s["host"] = [(im.cpu().pin_memory(), c.cpu().pin_memory())
                         for im, c in zip(imgs, cents)]
        return s
    w, h = case["width"], case["height"]
    n = w * h
    if kind == "frame":
        rgb = _image(g, w, h, case["cells"], case["palette"], bool(case["palette"]),
                     3.0 if case["palette"] else 4.0)
        if case["features"] == LAB_BETA:
            at = torch.randint(n, (case["k"],), generator=g, device=d)
            _, a, b = _lab64(rgb.view(-1, 3)[at])
            c0 = torch.stack([torch.zeros_like(a), a, b]).float()
        else:
            c0 = _picks(g, rgb, case["k"], case["dim"])
        s.update(rgb=rgb, c0=c0.contiguous(), pipe=pipeline.Pipeline(w, h, _params(case), d))
        if case["captured"]:
            s["pipe"].centroids.copy_(s["c0"])
            s["pipe"].capture(rgb)
    elif kind == "maze":
        s["labels"] = torch.from_numpy(synth.maze_labels(int(seed), w, h)).to(d)
        s["out"] = torch.empty((h, w), dtype=torch.int32, device=d)
        s["sizes"] = torch.empty(n, dtype=torch.int32, device=d)
        s["ccl_ws"] = Workspace(ccl.connected_components_workspace(w, h), d)
        s["merge_ws"] = Workspace(ccl.merge_small_segments_workspace(w, h), d)
    elif kind == "planar":
        rgb = _image(g, w, h, case["cells"])
        s["points"] = (rgb.view(n, 3).float() / 255.0).T.contiguous()
        s["c0"] = _picks(g, rgb, case["k"], 3)
        s["centroids"] = torch.empty_like(s["c0"])
        s["labels"] = torch.empty(n, dtype=torch.int32, device=d)
        s["ws"] = Workspace(kmeans.cluster_workspace_2d(n, w, case["k"], 3), d)
    elif kind == "palette":
        s["rgb"] = _image(g, w, h, case["cells"], sigma=8.0)
        s["next"] = _image(g, w, h, case["cells"], sigma=8.0)
        s["c0"] = _picks(g, s["rgb"], case["k"], case["dim"])
        s["centroids"] = torch.empty_like(s["c0"])
        s["labels"] = torch.empty(n, dtype=torch.int32, device=d)
        s["next_labels"] = torch.empty(n, dtype=torch.int32, device=d)
        s["ws"] = Workspace(kmeans.cluster_workspace_2d(n, w, case["k"], case["dim"]), d)
    elif kind in ("render", "regions"):
        s["segments"] = _segments(g, w, h, case["cells"], case["speckle"])
        s["labels"] = torch.empty((h, w), dtype=torch.int32, device=d)
        rgb = _image(g, w, h, case["cells"])
        s["points"] = (rgb.view(n, 3).float() / 255.0).T.contiguous()
        if kind == "render":
            s["painted"] = torch.empty((3, n), dtype=torch.float32, device=d)
            s["compress_ws"] = Workspace(ccl.compress_labels_workspace(n), d)
        else:
            s["smooth_ws"] = Workspace(ccl.merge_smooth_boundaries_workspace(w, h), d)
            s["adjacency_ws"] = Workspace(ccl.segment_adjacency_workspace(w, h), d)
            s["keys"] = torch.zeros(8 * n, dtype=torch.int32, device=d)
            s["adjacency"] = torch.zeros(8 * n, dtype=torch.int32, device=d)
    else:
        lum = _lab64(_image(g, w, h, 40, sigma=2.0))[0] / 100.0
        yy = torch.linspace(-1, 1, h, device=d, dtype=torch.float64)[:, None]
        xx = torch.linspace(-1, 1, w, device=d, dtype=torch.float64)[None]
        dome = (1.0 - 0.4 * (xx * xx + yy * yy)).clamp_min(0.05)
        s["shading"] = (0.3 * lum + 0.7 * dome).float().contiguous()
        s["normals"] = torch.empty((3, n), dtype=torch.float32, device=d)
        s["iterations"] = torch.zeros(1, dtype=torch.int32, device=d)
        s["ws"] = sfs.estimate_normals(s["shading"], LIGHT, s["normals"], 1.0, max_iter=0)
    return s


LIGHT = (0.3, -0.2, 1.0)


# ------------------------------------------------------------------ one pass
def run(s):
    kind, case = s["kind"], s["case"]
    if kind == "frame":
        p = s["pipe"]
        if case["captured"]:
            p.centroids.copy_(s["c0"], non_blocking=True)
            p.replay()
        else:
            p.run(s["rgb"], s["c0"])
        return {"clusters": p.cluster_labels, "segments": p.segment_labels,
                "normals": p.normals, "centroids": p.centroids}
    if kind == "batch":
        b = s["batch"]
        b.centroids.copy_(s["c0"], non_blocking=True)
        b.run()
        return {"clusters": b.cluster_labels, "segments": b.segment_labels,
                "normals": b.normals, "centroids": b.centroids}
    if kind == "serve":
        reqs = [serve.Request(i, rgb, k, it, c) for i, ((rgb, c), (_, _, k, it)) in
                enumerate(zip(s["host"], s["shapes"]))]
        s["server"].serve(reqs, realtime=False)
        return {"segments": [r.segment_labels for r in reqs],
                "centroids": [r.centroids_out for r in reqs]}
    if kind == "maze":
        ccl.connected_components(s["labels"], s["ccl_ws"], s["out"], connectivity=case["conn"],
                                 convention=ccl.MIN_INDEX, sizes=s["sizes"])
        ccl.merge_small_segments(None, s["out"], s["merge_ws"], case["merge_p"],
                                 policy=ccl.MOST_BOUNDARY, sizes=s["sizes"])
        return s["out"]
    if kind == "planar":
        s["centroids"].copy_(s["c0"], non_blocking=True)
        kmeans.cluster(s["points"], s["centroids"], s["labels"], s["ws"], case["iters"], -1.0,
                       width=case["width"])
        return {"labels": s["labels"], "centroids": s["centroids"]}
    if kind == "palette":
        s["centroids"].copy_(s["c0"], non_blocking=True)
        how = dict(layout=kmeans.RGB8, dim=case["dim"], width=case["width"], xy_scale=XY)
        kmeans.cluster(s["rgb"], s["centroids"], s["labels"], s["ws"], case["iters"], -1.0, **how)
        kmeans.label_points(s["centroids"], s["next"], s["next_labels"], s["ws"], **how)
        return {"labels": s["labels"], "next": s["next_labels"], "centroids": s["centroids"]}
    if kind == "render":
        labels = s["labels"].view(-1)
        labels.copy_(s["segments"])
        count = ccl.compress_labels(labels, s["compress_ws"])
        means = torch.zeros((3, count), dtype=torch.float32, device=labels.device)
        s["means_ws"] = kmeans.calculate_centroids(labels, s["points"], means, s.get("means_ws"),
                                                   width=case["width"])
        kmeans.propagate_centroids(labels, means, s["painted"])
        return {"labels": labels, "painted": s["painted"]}
    if kind == "regions":
        s["labels"].view(-1).copy_(s["segments"])
        ccl.merge_smooth_boundaries(s["points"], 0, s["labels"], s["smooth_ws"],
                                    case["threshold"])
        count = ccl.segment_adjacency(s["labels"], s["keys"], s["adjacency"], s["adjacency_ws"])
        return {"labels": s["labels"], "keys": s["keys"], "adjacency": s["adjacency"],
                "count": count}
    sfs.estimate_normals(s["shading"], LIGHT, s["normals"], case["smoothness"],
                         max_iter=case["max_iter"], temp=s["ws"],
                         iterations_out=s["iterations"])
    return {"normals": s["normals"], "sweeps": s["iterations"]}


# ------------------------------------------------------------------ floors
def work(case):
    """Inputs read once, outputs written once; operations: one distance per
    pixel and iteration for a clustering (bounds decide the rest), one block
    solve per pixel and sweep for the relaxation."""
    kind = case["kind"]
    if kind in ("batch", "serve"):
        shapes = _shapes(case)
        px = sum(w * h for w, h, _, _ in shapes)
        it = sum(w * h * i for w, h, _, i in shapes)
        return {"bytes": px * (3 + 4 + 4 + 12 if kind == "batch" else 3 + 4), "flops": it * 15}
    n = case["width"] * case["height"]
    if kind == "frame":
        return {"bytes": n * (3 + 4 + 4 + (12 if case["normals"] else 0)),
                "flops": n * case["iters"] * 3 * case["dim"]}
    if kind == "maze":
        return {"bytes": 8 * n, "flops": 0}
    if kind == "planar":
        return {"bytes": 16 * n, "flops": n * case["iters"] * 9}
    if kind == "palette":
        return {"bytes": 14 * n, "flops": n * (case["iters"] + 1) * 3 * case["dim"]}
    if kind == "render":
        return {"bytes": n * (4 + 4 + 12 + 12), "flops": 3 * n}
    if kind == "regions":
        return {"bytes": n * (4 + 4 + 12), "flops": 0}
    # intensity in, normals out; per pixel and sweep 3 x 4 neighbour adds, the
    # 3 x 3 block solve and the residual; the tolerance is met after about 45
    # sweeps per unit of smoothness
    sweeps = min(case["max_iter"], 45 * case["smoothness"])
    return {"bytes": 16 * n, "flops": 60 * n * sweeps}


# ------------------------------------------------------------------ 64 bits
def _features64(rgb, dim):
    h, w = rgb.shape[:2]
    f = [rgb[..., j].reshape(-1).double() / 255.0 for j in range(3)]
    if dim == 5:
        i = torch.arange(h * w, device=rgb.device)
        f += [XY * (i % w).double(), XY * (i // w).double()]
    return torch.stack(f)


def _nearest64(p, c):
    lab = torch.empty(p.shape[1], dtype=torch.int64, device=p.device)
    step = max(1, (1 << 28) // c.shape[1])
    for a in range(0, p.shape[1], step):
        q = p[:, a:a + step]
        d2 = torch.zeros((q.shape[1], c.shape[1]), dtype=torch.float64, device=p.device)
        for x, m in zip(q, c):
            d2 += (x[:, None] - m[None]).square_()
        lab[a:a + step] = d2.argmin(1)
    return lab


def _means64(p, lab, k, old):
    n = torch.bincount(lab, minlength=k).double()
    new = torch.stack([torch.bincount(lab, weights=x, minlength=k) for x in p])
    return torch.where(n > 0, new / n.clamp_min(1.0), old)


def _lloyd64(p, c0, iters):
    c = c0.double()
    for _ in range(iters):
        c = _means64(p, _nearest64(p, c), c.shape[1], c)
    return c


def _normals64(height, depth=1.0):
    """Sobel normals of an (H, W) height map: zero beyond the rows' ends,
    differences between clamped neighbours, unit length."""
    def smooth(a, dim):
        b = 2.0 * a
        n = a.shape[dim]
        b.narrow(dim, 1, n - 1).add_(a.narrow(dim, 0, n - 1))
        b.narrow(dim, 0, n - 1).add_(a.narrow(dim, 1, n - 1))
        return b

    def step(a, dim):
        n = a.shape[dim]
        i = torch.arange(n, device=a.device)
        return a.index_select(dim, (i + 1).clamp_max(n - 1)) - \
            a.index_select(dim, (i - 1).clamp_min(0))
    gx, gy = step(smooth(height, 0), 1), step(smooth(height, 1), 0)
    v = torch.stack([gx, gy, torch.full_like(gx, 1.0 / max(0.001, depth))])
    return (v / v.square().sum(0).sqrt()).reshape(3, -1)


def _frame_normals64(rgb):
    return _normals64(_lab64(rgb)[0] / 100.0)


def _relax64(shading, smoothness, max_iter, tol=1e-5):
    s = shading.double()
    h, w = s.shape
    light = torch.tensor(LIGHT, dtype=torch.float64, device=s.device)
    light = (light / light.square().sum().sqrt())[:, None, None]
    lam2 = 2.0 * smoothness
    r = torch.arange(h, device=s.device)[:, None]
    c = torch.arange(w, device=s.device)[None]
    val = 4.0 - ((r == 0) | (r == h - 1)).double() - ((c == 0) | (c == w - 1)).double()
    colour = (r + c) % 2
    x = torch.zeros((3, h, w), dtype=torch.float64, device=s.device)
    x[2] = 1.0

    def around(x):
        t = torch.zeros_like(x)
        t[:, 1:] += x[:, :-1]
        t[:, :-1] += x[:, 1:]
        t[:, :, 1:] += x[:, :, :-1]
        t[:, :, :-1] += x[:, :, 1:]
        return t
    b = light * s
    limit = (tol * tol) * b.square().sum()
    sweeps = 0
    while True:
        res = b - light * (light * x).sum(0) - lam2 * (val * x - around(x))
        if sweeps >= max_iter or bool(res.square().sum() <= limit):
            break
        for k in (0, 1):
            rhs = b + lam2 * around(x)
            q = (light * rhs).sum(0) / (lam2 * val + 1.0)
            x = torch.where(colour == k, (rhs - light * q) / (lam2 * val), x)
        sweeps += 1
    x[2].abs_()
    return (x / x.square().sum(0).sqrt()).reshape(3, -1)


def exact(case, seed):
    kind = case["kind"]
    if kind in ("maze", "regions"):
        return None   # whole numbers only
    s = prepare(case, seed)
    if kind == "frame":
        lab = case["features"] == LAB_BETA   # beta jumps between -mu, 0 and mu at thresholds
        return {"clusters": None, "segments": None,
                "normals": _frame_normals64(s["rgb"]) if case["normals"] else None,
                "centroids": None if lab else
                _lloyd64(_features64(s["rgb"], case["dim"]), s["c0"], case["iters"])}
    if kind in ("batch", "serve"):
        cents = [_lloyd64(_features64(im, 5), c, it) for im, c, (_, _, _, it) in
                 zip(s["images"], s["centroids0"], s["shapes"])]
        if kind == "serve":
            return {"segments": None, "centroids": cents}
        b = s["batch"]
        c64, n64 = s["c0"].double(), torch.zeros_like(b.normals, dtype=torch.float64)
        for i, (im, c) in enumerate(zip(s["images"], cents)):
            c64[b.coffsets[i]:b.coffsets[i] + c.numel()] = c.reshape(-1)
            v = _frame_normals64(im).reshape(-1)
            n64[3 * b.offsets[i]:3 * b.offsets[i] + v.numel()] = v
        return {"clusters": None, "segments": None, "normals": n64, "centroids": c64}
    if kind == "planar":
        return {"labels": None, "centroids": _lloyd64(s["points"].double(), s["c0"],
                                                      case["iters"])}
    if kind == "palette":
        return {"labels": None, "next": None, "centroids": _lloyd64(
            _features64(s["rgb"], case["dim"]), s["c0"], case["iters"])}
    if kind == "render":
        _, lab = torch.unique(s["segments"], return_inverse=True)
        k = int(lab.max()) + 1
        p = s["points"].double()
        zero = torch.zeros((3, k), dtype=torch.float64, device=p.device)
        return {"labels": None, "painted": _means64(p, lab, k, zero)[:, lab]}
    return {"normals": _relax64(s["shading"], case["smoothness"], case["max_iter"]),
            "sweeps": None}

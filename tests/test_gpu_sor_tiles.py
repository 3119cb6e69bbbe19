"""Shape-from-shading normals at the edges of the solver's pixel split: odd
and even widths, rows longer than a block, a last block that is nearly empty,
several pixels per thread, and intensities far from 1 (the residual is summed
scaled)."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape,scale,sweeps,tol", [
    ((32, 64), 1.0, 9, 0.0),        # one block exactly full
    ((33, 65), 1.0, 9, 0.0),        # one pixel row past it, odd width
    ((2, 2), 1.0, 40, 1e-5),
    ((3, 4099), 1.0, 7, 0.0),       # rows longer than a block's threads
    ((4099, 3), 1.0, 7, 0.0),
    ((701, 499), 1.0, 5, 0.0),      # every SM, two pixels of a colour per thread
    ((40, 50), 1e20, 200, 1e-4),    # squares beyond FP32 without the scaling
    ((40, 50), 1e-15, 12, 1e-5)])
def test_sor_pixel_split(cuda, shape, scale, sweeps, tol):
    import torch
    from split_gb300 import sfs
    rng = np.random.default_rng(shape[0] * 131 + shape[1])
    s = (rng.random(shape) * scale).astype(np.float32)
    light = (0.3, -0.2, 1.0)
    ref, ref_it = oracle.estimate_normals_rb(s, light, 1.0, sweeps, tol)
    out = torch.empty((3, s.size), dtype=torch.float32, device=cuda)
    its = torch.zeros(1, dtype=torch.int32, device=cuda)
    ws = sfs.estimate_normals(torch.from_numpy(s).to(cuda), light, out, 1.0, max_iter=sweeps,
                              tol=tol, iterations_out=its)
    torch.cuda.synchronize()
    ws.check("estimate_normals")
    assert abs(int(its.item()) - ref_it) <= (1 if tol > 0 else 0)
    got = out.cpu().numpy().astype(np.float64)
    ang = np.arctan2(np.linalg.norm(np.cross(got.T, ref.T), axis=1), (got * ref).sum(0))
    assert ang.max() <= 1e-4   # FP32 rounding of some tens of operations per sweep


def _relax_f32(s, light, lam, sweeps):
    """|b|^2 and the squared residual before each sweep of the FP32 relaxation,
    both summed exactly; the light's components are used as given."""
    import math
    f = np.float32
    h, w = s.shape
    L = [f(v) for v in light]
    LL = f(f(L[0] * L[0] + L[1] * L[1]) + L[2] * L[2])
    lam2 = f(2) * f(lam)
    r, c = np.mgrid[0:h, 0:w]
    v = (4 - ((r == 0) | (r == h - 1)).astype(int) - ((c == 0) | (c == w - 1)).astype(int)).astype(f)
    x = np.zeros((3, h, w), f)
    x[2] = 1

    def nsum(x):
        S = np.zeros_like(x)
        S[:, 1:] += x[:, :-1]
        S[:, :, 1:] += x[:, :, :-1]
        S[:, :, :-1] += x[:, :, 1:]
        S[:, :-1] += x[:, 1:]
        return S

    out = []
    for k in range(sweeps):
        S = nsum(x)
        lx = (L[0] * x[0] + L[1] * x[1]) + L[2] * x[2]
        e = np.stack([s * L[d] - (L[d] * lx + lam2 * (v * x[d] - S[d])) for d in range(3)])
        assert e.dtype == f
        out.append(math.fsum((e.astype(np.float64) ** 2).ravel()))
        for colour in range(2):
            S = nsum(x)
            rv = [s * L[d] + lam2 * S[d] for d in range(3)]
            cc = lam2 * v
            q = ((L[0] * rv[0] + L[1] * rv[1]) + L[2] * rv[2]) / (cc + LL)
            new = np.stack([(rv[d] - L[d] * q) / cc for d in range(3)])
            x = np.where((r + c) % 2 == colour, new, x)
    b2 = math.fsum((s.astype(np.float64) ** 2).ravel()) * float(LL)
    return b2, out


def _sweeps(cuda, s, light, max_iter, tol):
    import torch
    from split_gb300 import sfs
    out = torch.empty((3, s.size), dtype=torch.float32, device=cuda)
    its = torch.full((1,), -1, dtype=torch.int32, device=cuda)
    ws = sfs.estimate_normals(torch.from_numpy(s).to(cuda), light, out, 1.0, max_iter=max_iter,
                              tol=float(tol), iterations_out=its)
    ws.check("estimate_normals")
    return int(its.item()), out.cpu().numpy()


@pytest.mark.parametrize("shape,scale", [((40, 50), 1.0), ((33, 65), 1e-12), ((301, 200), 1e12)])
def test_stop_is_that_of_fp64_sums(cuda, shape, scale):
    """Tolerances whose limit is the next one above and below the residual of a
    sweep: the sweep count follows the exact sums."""
    rng = np.random.default_rng(shape[0])
    s = (rng.random(shape) * scale).astype(np.float32)
    # (0, 3, 4) / 5 in the library's float steps, whether or not they are fused
    L = (0.0, np.float32(3) * np.float32(0.2), np.float32(4) * np.float32(0.2))
    b2, r2 = _relax_f32(s, L, 1.0, 12)
    for k in (0, 3, 10):
        assert all(v > r2[k] * 1.001 for v in r2[:k])
        tol = np.float32(np.sqrt(r2[k] / b2))
        while float(tol) ** 2 * b2 < r2[k] * (1 + 1e-12):
            tol = np.nextafter(tol, np.float32(np.inf))
        below = tol
        while float(below) ** 2 * b2 > r2[k] * (1 - 1e-12):
            below = np.nextafter(below, np.float32(0))
        assert _sweeps(cuda, s, (0.0, 3.0, 4.0), 100, tol)[0] == k
        want = next(i for i in range(12) if r2[i] <= float(below) ** 2 * b2)
        assert want > k and _sweeps(cuda, s, (0.0, 3.0, 4.0), 100, below)[0] == want


def test_intensities_that_are_not_finite(cuda):
    """An infinite |b| meets every residual at once; NaN meets none."""
    s = np.random.default_rng(1).random((40, 50)).astype(np.float32)
    s[7, 9] = np.inf
    its, out = _sweeps(cuda, s, (1.0, 2.0, 2.0), 9, 1e-5)
    assert its == 0 and (out[2] == 1).all() and (out[:2] == 0).all()
    s[7, 9] = np.nan
    assert _sweeps(cuda, s, (1.0, 2.0, 2.0), 9, 1e-5)[0] == 9


@pytest.mark.parametrize("shape", [(1, 1), (1, 700), (40, 50), (33, 65), (480, 640)])
def test_workspace_without_the_unknowns(cuda, shape):
    """A workspace of one size for every image: the same normals and sweeps, bit
    for bit; a smaller one is refused."""
    import torch
    from split_gb300 import _native as N
    from split_gb300._util import Workspace, ptr, stream_handle
    s = np.random.default_rng(sum(shape)).random(shape).astype(np.float32)
    dev, its = torch.from_numpy(s).to(cuda), torch.zeros(2, dtype=torch.int32, device=cuda)
    out = torch.zeros((2, 3, s.size), dtype=torch.float32, device=cuda)
    lib = N.load()
    sizes = (lib.split_estimate_normals_workspace_size(shape[1], shape[0]), 65792)
    for tol in (0.0, 1e-2):
        for k, nbytes in enumerate(sizes):
            ws = Workspace(nbytes, cuda)
            N.check(lib.split_estimate_normals(
                ptr(dev), shape[1], shape[0], 0.3, -0.2, 1.0, 1.0, 40, tol, ptr(out[k]),
                ptr(its[k:]), ws.ptr, nbytes, stream_handle()), "estimate_normals")
            ws.check("estimate_normals")
        assert torch.equal(its[0], its[1]) and torch.equal(out[0], out[1])
    assert lib.split_estimate_normals(
        ptr(dev), shape[1], shape[0], 0.3, -0.2, 1.0, 1.0, 40, 0.0, ptr(out[0]), ptr(its), ws.ptr,
        65792 - 256, stream_handle()) != N.OK

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

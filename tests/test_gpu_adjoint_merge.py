"""The exact adjoint with rows merged, at the sizes from which residuals that may be
zero for the most part take two and four rays a thread, against the CPU
restatement of the march.

Tolerance: as for the other merged scatters the terms are the march's own and only
the order of the FP32 additions differs: 1e-5 relative L2 for some hundred terms a
voxel, which a residual live on a few rows of every view keeps."""
import numpy as np
import pytest

import oracle_bind as ob

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("det,ds,views", [((403, 389), 0.25, 4), ((403, 389), 0.25, 20), ((409, 397), 0.40, 7)])
def test_the_adjoint_matches_the_march(cuda, det, ds, views):
    import torch

    import spacetimetomography_b200 as stt

    dims, off = (40, 36, 44), (0.5, -0.7, 0.3)
    angles = np.linspace(0.0, 5.9, views)
    scan = ob.Scan(dims, det, ds=ds, off=off)
    W, H = det
    ctx = stt.Context(0)
    ctx.set_geometry(dims, scan.sp, det, ds, scan.sid, scan.sdd, angles, off)
    rng = np.random.default_rng(views)
    y = np.zeros((views, H, W), np.float32)
    for v in range(views):  # runs of rows that start inside a thread's group, and single rays
        for j in rng.integers(0, H - 6, max(1, 40 // views)):
            y[v, j:j + rng.integers(1, 6)] = rng.uniform(-1, 1, W)
        y[v, rng.integers(0, H, 30), rng.integers(0, W, 30)] = 1.0
    want = np.zeros(dims[::-1])
    for v, a in enumerate(angles):
        want += ob.fp_adjoint32(scan, ob.view_angle(a), y[v]).astype(np.float64)
    bar = torch.ones(dims[::-1], device=cuda)
    ctx.fp_vjp(torch.from_numpy(y).to(cuda), bar)
    assert ob.rel_l2(bar.cpu().numpy() - 1.0, want) < 1e-5
    ctx.close()

"""The voxel backprojection's columns at the edges of their tiles, against the
FP64 oracle: extents around the 32 x 4 blocks and the 8 to 20 voxel columns,
magnifications on both sides of what the row table holds (below one row per
voxel, and past it, where the kernel walks the column), a detector smaller than
the volume's shadow, and both storages.  Every variant gives the same bits, and a
BF16-stored volume the FP32 result of the same values, rounded.

Tolerance: the suite's 1e-4 relative L2 of the update (the FP32 coordinates put
a tap's position off by a few 1e-5 pixel).  The reference's cutoff at 2 pixels
from the border is a jump, so voxels that project within 1e-3 pixel of it are
left out of the comparison (they may take either side in FP32)."""
import numpy as np
import pytest

import oracle_bind as ob

pytestmark = pytest.mark.gpu

CASES = [  # dims, detector, ds, sid, sdd, offset
    ((31, 16, 5), (64, 40), 1.0, 600.0, 1000.0, (0.0, 0.0, 0.0)),
    ((33, 17, 4), (70, 44), 1.0, 600.0, 1000.0, (0.6, -0.4, 0.3)),
    ((65, 41, 9), (60, 31), 1.0, 300.0, 500.0, (0.0, 0.0, 0.0)),      # shadow larger than the detector
    ((40, 20, 40), (33, 29), 3.0, 600.0, 1000.0, (0.0, 0.0, 0.0)),    # under one row per voxel
    ((24, 60, 24), (90, 150), 0.7, 200.0, 340.0, (0.0, 0.0, 0.0)),    # about 2.4 rows: shorter columns
    ((20, 33, 21), (160, 240), 0.3, 150.0, 300.0, (0.0, 0.0, 0.0)),   # about 7 rows: the walk
    ((2, 2, 2), (9, 8), 1.0, 600.0, 1000.0, (0.0, 0.0, 0.0)),
]
ANGLES = np.deg2rad([0.0, 40.0, 90.0, 201.0, 313.0])


def _far_from_the_cutoff(scan, angle):
    nx, ny, nz = scan.dims
    z, y, x = np.meshgrid(*(np.arange(n, dtype=np.float64) for n in (nz, ny, nx)), indexing="ij")
    c, s = np.cos(angle), np.sin(angle)
    p = [(q - (n - 1) * 0.5) for q, n in zip((x, y, z), (nx, ny, nz))]
    ox, oy, oz = scan.off
    cam = [c * p[0] + s * p[2] - ox, p[1] - oz, -s * p[0] + c * p[2] - scan.sid + oy]
    W, H = scan.det
    ok = np.ones(x.shape, bool)
    for a, n in ((0, W), (1, H)):
        u = (n - 1) * 0.5 + cam[a] / -cam[2] * scan.sdd / scan.ds
        ok &= (np.abs(u - 2) > 1e-3) & (np.abs(u - (n - 2)) > 1e-3)
    return ok


@pytest.mark.parametrize("case", range(len(CASES)))
def test_columns_match_the_oracle(cuda, case):
    import torch

    import spacetimetomography_b200 as stt

    dims, det, ds, sid, sdd, off = CASES[case]
    scan = ob.Scan(dims, det, ds=ds, sid=sid, sdd=sdd, off=off)
    nx, ny, nz = dims
    W, H = det
    ctx = stt.Context(0)
    ctx.set_geometry(dims, scan.sp, det, ds, sid, sdd, ANGLES, off)
    rng = np.random.default_rng(case)
    corr = rng.normal(size=(H, W)).astype(np.float32)
    start = torch.from_numpy(rng.uniform(0.5, 2.0, (nz, ny, nx)).astype(np.float32)).to(cuda)
    start16 = start.to(torch.bfloat16)
    c = torch.from_numpy(corr).to(cuda)
    moved = 0
    for v, a in enumerate(ANGLES):
        outs = []
        for bv in range(5):
            ctx.set_tuning(0, 0, bv)
            vol = start.clone()
            ctx.bp_voxel(c, vol, 0.3, 2.5, v)
            outs.append(vol.cpu().numpy())
            narrow, wide = start16.clone(), start16.float()
            ctx.bp_voxel(c, narrow, 0.3, 2.5, v)
            ctx.bp_voxel(c, wide, 0.3, 2.5, v)
            assert torch.equal(narrow, wide.to(torch.bfloat16)), f"BF16 storage, variant {bv}, view {v}"
        for bv in range(1, 5):
            np.testing.assert_array_equal(outs[0], outs[bv], err_msg=f"variant {bv}, view {v}")
        first = start.cpu().numpy()
        ref = ob.bp_voxel64(scan, ob.view_angle(a), corr, 0.3, 2.5, first)
        ok = _far_from_the_cutoff(scan, a)
        scale = np.linalg.norm((ref - first)[ok])
        moved += scale > 0
        err = np.linalg.norm((outs[0] - ref)[ok])
        assert err <= 1e-4 * scale, f"view {v}: {err / scale}"
    assert moved == len(ANGLES) or min(dims) == 2
    ctx.close()

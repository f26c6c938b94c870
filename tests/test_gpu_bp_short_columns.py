"""The voxel backprojection at magnifications that take columns of four voxels: against
the FP64 oracle and, bit for bit, the other column lengths, both storages.

Tolerance and the voxels left out near the reference's cutoff: as for the longer
columns (1e-4 relative L2 of the update; 1e-3 pixel)."""
import ctypes as C

import numpy as np
import pytest

import oracle_bind as ob
from test_gpu_bp_columns import _far_from_the_cutoff


@pytest.mark.parametrize("rows,n,want", [(1.6, 256, 16), (2.4, 128, 12), (5.0, 96, 8), (6.0, 96, 4), (11.6, 64, 4),
                                         (11.8, 64, 8), (6.0, 256, 8)])
def test_column_lengths(rows, n, want):
    from spacetimetomography_b200 import build

    build.build_libstt()
    from spacetimetomography_b200._lib import lib

    f = lib.stt_internal_bp_len
    f.argtypes, f.restype = [C.c_double, C.c_longlong], C.c_int
    assert f(rows, n**3) == want


CASES = [  # dims, detector, ds, sid, sdd: 5.6 to 11 rows a voxel where the volume is nearest
    ((33, 21, 20), (200, 190), 0.3, 160.0, 270.0),
    ((31, 18, 33), (300, 280), 0.25, 150.0, 300.0),
    ((40, 13, 35), (150, 60), 0.3, 130.0, 300.0),
    ((5, 3, 6), (64, 48), 0.2, 100.0, 200.0),
]


@pytest.mark.gpu
@pytest.mark.parametrize("case", range(len(CASES)))
def test_short_columns_match_the_oracle(cuda, case):
    import torch

    import spacetimetomography_b200 as stt

    dims, det, ds, sid, sdd = CASES[case]
    scan = ob.Scan(dims, det, ds=ds, sid=sid, sdd=sdd)
    nx, ny, nz = dims
    W, H = det
    angles = np.deg2rad([0.0, 33.0, 90.0, 251.0])
    ctx = stt.Context(0)
    ctx.set_geometry(dims, scan.sp, det, ds, sid, sdd, angles)
    rng = np.random.default_rng(case)
    corr = rng.normal(size=(H, W)).astype(np.float32)
    start = torch.from_numpy(rng.uniform(0.5, 2.0, (nz, ny, nx)).astype(np.float32)).to(cuda)
    c = torch.from_numpy(corr).to(cuda)
    for v, a in enumerate(angles):
        outs = []
        for bv in range(5):
            ctx.set_tuning(0, 0, bv)
            vol = start.clone()
            ctx.bp_voxel(c, vol, 0.3, 2.5, v)
            outs.append(vol)
            narrow, wide = start.to(torch.bfloat16), start.to(torch.bfloat16).float()
            ctx.bp_voxel(c, narrow, 0.3, 2.5, v)
            ctx.bp_voxel(c, wide, 0.3, 2.5, v)
            assert torch.equal(narrow, wide.to(torch.bfloat16))
        for bv in range(1, 5):
            assert torch.equal(outs[0], outs[bv]), f"variant {bv}, view {v}"
        first = start.cpu().numpy()
        ref = ob.bp_voxel64(scan, ob.view_angle(a), corr, 0.3, 2.5, first)
        ok = _far_from_the_cutoff(scan, a)
        scale = np.linalg.norm((ref - first)[ok])
        assert scale > 0 and np.linalg.norm((outs[0].cpu().numpy() - ref)[ok]) <= 1e-4 * scale
    ctx.close()

"""The scatters with neighbouring detector rows merged (two or four rays a
thread) against the CPU restatement of the same FP32 march: the ray-driven
backprojection's contributions and weights and the exact adjoint, on detectors
whose rows and columns end inside a block, off-centre and anisotropic volumes,
rays that miss, and the march's restart before the entry.

Tolerance: the terms are the march's own (products rounded once more); only the
order of the float additions differs, over some hundred terms a voxel: 1e-5
relative L2, the suite's bound for a reordered scatter. A volume of eight voxels gets half a
million terms in each, and an FP32 sum of that many rounds by more than that in
any order: there the corrections are compared a patch of 4 x 8 rays at a time (the
rest of the correction zero, which adds nothing), some hundred terms a voxel again."""
import numpy as np
import pytest

import oracle_bind as ob

pytestmark = pytest.mark.gpu

CASES = [  # dims, detector, pixel, spacing, offset: rows per voxel and rays choose how many merge; in patches
    ((40, 36, 44), (403, 389), 0.25, 1.0, (0.0, 0.0, 0.0), False),   # two rays a thread, the adjoint four
    ((24, 50, 17), (391, 401), 0.33, 1.3, (1.5, -2.0, 0.7), False),  # the same, a ragged last column of rows
    ((33, 20, 31), (253, 241), 1.5, 1.0, (0.3, 0.1, -0.4), False),   # one, the adjoint two; most rays miss
    ((2, 2, 2), (390, 386), 0.02, 1.0, (0.0, 0.0, 0.0), True),   # every cell on a face
    ((40, 36, 44), (431, 421), 0.23, 1.0, (0.2, 0.0, -0.3), False),  # four
]
ANGLES = np.array([0.0, 0.6, np.pi / 2, 3.9])


@pytest.mark.parametrize("case", range(len(CASES)))
def test_merged_scatters_match_the_march(cuda, case):
    import torch

    import spacetimetomography_b200 as stt

    dims, det, ds, sp, off, patches = CASES[case]
    scan = ob.Scan(dims, det, ds=ds, spacing=sp, off=off)
    nx, ny, nz = dims
    W, H = det
    ctx = stt.Context(0)
    ctx.set_geometry(dims, scan.sp, det, ds, scan.sid, scan.sdd, ANGLES, off)
    rng = np.random.default_rng(case)
    corr = rng.uniform(0.1, 1.0, (len(ANGLES), H, W)).astype(np.float32)
    corr[:, ::7, ::5] = 0  # the adjoint skips a zero, the backprojection adds its weights

    def parts(image):
        if not patches:
            return [image]
        out = []
        for j in (0, H // 8 * 4, (H - 1) // 4 * 4):  # (the last one of H % 4 rows)
            for i in (0, W // 2 - 4, W - 8):
                out.append(np.zeros_like(image))
                out[-1][..., j:j + 4, i:i + 8] = image[..., j:j + 4, i:i + 8]
        return out

    for v, a in enumerate(ANGLES):
        for image in (corr[v], np.ones((H, W), np.float32)):  # (the weights are the contributions of ones)
            for q, part in enumerate(parts(image)):
                c, w = torch.zeros((nz, ny, nx), device=cuda), torch.zeros((nz, ny, nx), device=cuda)
                ctx.bp_ray_scatter(torch.from_numpy(part).to(cuda), c, w, v)
                # (gmode 1: the kernels' FP64 ray set-up)
                c_ref, w_ref = ob.bp_ray_scatter32(scan, ob.view_angle(a), part, gmode=1)
                assert ob.rel_l2(c.cpu().numpy(), c_ref) < 1e-5, f"contributions, view {v}, part {q}"
                assert patches or ob.rel_l2(w.cpu().numpy(), w_ref) < 1e-5, f"weights, view {v}"
                assert np.array_equal(w.cpu().numpy() > 0, w_ref > 0), f"touched voxels, view {v}"
    for q, part in enumerate(parts(corr)):
        adj_ref = np.zeros((nz, ny, nx))
        for v, a in enumerate(ANGLES):
            adj_ref += ob.fp_adjoint32(scan, ob.view_angle(a), part[v]).astype(np.float64)
        vol_bar = torch.ones((nz, ny, nx), device=cuda)
        ctx.fp_vjp(torch.from_numpy(part).to(cuda), vol_bar)
        assert ob.rel_l2(vol_bar.cpu().numpy() - 1.0, adj_ref) < 1e-5, f"adjoint, part {q}"
    ctx.close()

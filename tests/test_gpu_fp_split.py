"""The texture forms of the forward projector against the load forms, bit for
bit: views of few rays (each ray shared between the warps of a block), the
boundary between the two texture forms, ragged detectors, rays that miss, the
march's restart before the entry (a non-zero boundary, an off-centre volume),
both storages, volumes projected from a mirror (their slices are not aligned) and
volumes no texture takes.  A context's default choice,
each tuned variant and the slab-staged kernel with textures beside it agree."""
import numpy as np
import pytest

import oracle_bind as ob

pytestmark = pytest.mark.gpu

CASES = [  # dims, detector, spacing, offset
    ((32, 24, 40), (8, 5), 1.0, (0.0, 0.0, 0.0)),         # one block
    ((64, 64, 64), (61, 45), 1.3, (1.5, -2.0, 0.7)),
    ((16, 8, 12), (90, 71), 1.0, (0.0, 0.0, 0.0)),        # most rays miss
    ((48, 40, 44), (192, 128), 1.0, (0.5, -0.3, 0.2)),    # 24576 rays: the last shared view
    ((48, 40, 44), (193, 128), 1.0, (0.5, -0.3, 0.2)),    # the first that is not
    ((33, 17, 21), (40, 37), 1.0, (0.0, 0.0, 0.0)),       # unaligned slices: through a mirror
    ((2, 2, 2), (40, 37), 1.0, (0.0, 0.0, 0.0)),
    ((30, 31, 29), (200, 160), 1.0, (0.3, 0.0, 0.0)),     # a mirror, and rays past the shared views
    ((1024, 130, 6), (64, 40), 1.0, (0.0, 0.0, 0.0)),     # slices past the texture width: loads
]
ANGLES = np.array([0.0, 0.05, 0.5, 0.785, 1.3, np.pi / 2, 2.36, 3.3, 4.4, 5.5])


@pytest.mark.parametrize("case", range(len(CASES)))
@pytest.mark.parametrize("storage", ["f32", "bf16"])
def test_texture_forms_equal_loads(cuda, case, storage):
    import torch

    import spacetimetomography_b200 as stt

    dims, det, sp, off = CASES[case]
    scan = ob.Scan(dims, det, spacing=sp, off=off)
    nx, ny, nz = dims
    W, H = det
    ctx = stt.Context(0)
    ctx.set_geometry(dims, scan.sp, det, scan.ds, scan.sid, scan.sdd, ANGLES, off)
    g = torch.Generator(device=cuda)
    g.manual_seed(case)
    vol = torch.rand((nz, ny, nx), device=cuda, generator=g) + 0.25  # a boundary that is not empty
    b = torch.rand((len(ANGLES), H, W), device=cuda, generator=g) * 30
    if storage == "bf16":
        vol, b = vol.to(torch.bfloat16), b.to(torch.bfloat16)
    wide, bw = vol.float(), b.float()
    # the load form of the projection: the correction of a load variant, per view
    load = stt.Context(0)
    load.set_geometry(dims, scan.sp, det, scan.ds, scan.sid, scan.sdd, ANGLES, off)
    load.set_tuning(0, 0, 0, staged_bins=0)
    state, corr = torch.zeros((H, W), device=cuda), torch.zeros((H, W), device=cuda)
    proj, rl, count = (torch.zeros((len(ANGLES), H, W), device=cuda) for _ in range(3))
    ctx.fp_typed(vol, proj, raylen=rl, weight=count)
    one = [torch.zeros((1, H, W), device=cuda) for _ in range(3)]
    other = torch.zeros((H, W), device=cuda)
    for v in range(len(ANGLES)):
        load.fp_correction(wide, bw[v], state, corr, v)
        hit = count[v] > 0
        # c = (b - Ax) / (L + 1) from the texture form's projection and lengths
        L = torch.where(hit, rl[v], state)
        assert torch.equal((bw[v] - proj[v]) / (L + 1.0), corr), f"projection, view {v}"
        assert torch.equal(state[hit], rl[v][hit])
        ctx.fp_typed(vol, one[0], view0=v, nviews=1, raylen=one[1], weight=one[2])  # one view: fewer rays
        assert torch.equal(one[0][0], proj[v]) and torch.equal(one[2][0], count[v]), f"view {v} on its own"
        if storage == "f32":
            for tuned in (None, 10, 11):
                if tuned is not None:
                    ctx.set_tuning(tuned, 0, 0, staged_bins=0x1F0 if nx % 4 == 0 and nz % 4 == 0 else 0)
                st = torch.where(hit, torch.zeros_like(state), state)
                ctx.fp_correction(vol, b[v], st, other, v)
                assert torch.equal(other, corr), f"correction, variant {tuned}, view {v}"
                assert torch.equal(st[hit], rl[v][hit])
    ctx.poll_status()
    # one sweep, default choice against loads: the projections, copies and backprojections in order
    perm = np.random.default_rng(case).permutation(len(ANGLES)).astype(np.int32)
    outs = []
    for tuned in (False, True):
        c = stt.Context(0)
        c.set_geometry(dims, scan.sp, det, scan.ds, scan.sid, scan.sdd, ANGLES, off)
        if tuned:
            c.set_tuning(0, 0, 0, staged_bins=0, fp_variant_bf16=0)
        x, st = vol.clone(), torch.zeros((H, W), device=cuda)
        c.sart_sweep(x, b, perm, 0.3, 5.0, 0, st)
        outs.append((x, st))
        c.close()
    assert torch.equal(outs[0][0], outs[1][0]) and torch.equal(outs[0][1], outs[1][1])
    ctx.close()
    load.close()


@pytest.mark.parametrize("storage", ["f32", "bf16"])
@pytest.mark.parametrize("bp_mode", [0, 1])
def test_solver_frames_through_mirrors(cuda, storage, bp_mode):
    """Two frames of unaligned slices: the projector's default form (each frame's
    mirror kept current by the backprojection) against loads.  Voxel
    backprojection bit for bit; ray backprojection within the reordering of its
    float atomics."""
    import torch

    import spacetimetomography_b200 as stt

    F, V, dims, det = 2, 7, (29, 27, 31), (44, 40)
    nx, ny, nz = dims
    W, H = det
    g = torch.Generator(device=cuda)
    g.manual_seed(3)
    rand = lambda *s: torch.rand(s, device=cuda, generator=g)  # noqa: E731
    vol, proj = rand(F + 1, nz, ny, nx), rand(F, V, H, W) * 20
    flow = (rand(F, 3, nz, ny, nx) - 0.5) * 2
    cut = (3, 3, 3, 5, 3, 3, 6, 5)
    outs = []
    for tuned in (False, True):
        ctx = stt.Context(0)
        ctx.set_geometry(dims, (1.0, 1.0, 1.0), det, 1.0, 600.0, 1000.0, np.arange(F * V) * 0.7, (0.0, 0.0, 0.0))
        if tuned:
            ctx.set_tuning(0, 0, 0, staged_bins=0, fp_variant_bf16=0)
        z = lambda *s: torch.zeros(s, device=cuda)  # noqa: E731
        st = dict(vol=vol.clone(), xbar=vol.clone(), xprev=z(F, nz, ny, nx), ytv=z(F, 3, nz, ny, nx),
                  ytp=z(F, nz, ny, nx), ybc=z(F, nz, ny, nx), flow=flow, proj=proj)
        if storage == "bf16":
            for k in ("vol", "xbar", "xprev", "proj"):
                st[k] = st[k].to(torch.bfloat16)
        s = stt.Solver(ctx, st, F, V, stt.PdParams(gmax=5.0, cut=cut), bp_mode=bp_mode, roi_cut=cut, seed=5,
                       storage=storage)
        s.iterate(2)
        torch.cuda.synchronize()
        s.poll_status()
        outs.append({k: st[k].float().cpu().numpy() for k in ("vol", "xbar", "xprev", "ytv", "ytp", "ybc")})
        s.close()
        ctx.close()
    for k in outs[0]:
        if bp_mode == 0:
            np.testing.assert_array_equal(outs[0][k], outs[1][k], err_msg=k)
        else:
            scale = np.linalg.norm(outs[1][k])
            assert np.linalg.norm(outs[0][k] - outs[1][k]) <= (1e-2 if storage == "bf16" else 1e-4) * scale, k

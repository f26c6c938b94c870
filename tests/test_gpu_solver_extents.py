"""The solver's warps on volumes that take 64-bit offsets: extents of two voxels, whose
samples must not leave the volume, and more than 2^30 voxels, whose flow's third plane
lies past 2^31."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

NAMES = dict(vol=1, xbar=1, xprev=0, ytv=0, ytp=0, ybc=0, flow=0)  # (vol and xbar hold one frame more)


def _solve(stt, torch, cuda, dims, state, mode, storage, frames):
    ctx = stt.Context(0)
    ctx.set_geometry(dims, (1.0, 1.0, 1.0), (24, 20), 2.0, 300.0, 500.0, np.linspace(0.2, 5.0, 2 * frames))
    pd = stt.PdParams(tv_w=0.02, tp_w=0.1, bc_w=0.5, huber_factor=0.9, gmax=3.0, cut=(0,) * 8)
    s = stt.Solver(ctx, state, frames, 2, pd, seed=3, mode=mode, storage=storage)
    s.iterate(2)
    torch.cuda.synchronize()
    s.poll_status()
    s.close()
    ctx.close()


@pytest.mark.parametrize("dims", [(2, 9, 7), (8, 2, 7), (12, 6, 2), (2, 2, 2), (33, 17, 2)])
@pytest.mark.parametrize("storage", ["f32", "bf16"])
@pytest.mark.parametrize("frames", [1, 2])
def test_an_extent_of_two(cuda, dims, storage, frames):
    import torch

    import spacetimetomography_b200 as stt

    nx, ny, nz = dims
    dt = torch.bfloat16 if storage == "bf16" else torch.float32
    outs = []
    for mode in (stt.SOLVE_PLAIN, stt.SOLVE_STREAMS, stt.SOLVE_GRAPH, stt.SOLVE_PERSISTENT):
        for around in (0.0, float("nan"), 1e30):  # what lies before and behind every array
            g = torch.Generator(device=cuda)
            g.manual_seed(5)
            state = {}
            for name, more in NAMES.items():
                shape = (frames + more,) + ((3,) if name in ("ytv", "flow") else ()) + (nz, ny, nx)
                kind = dt if name in ("vol", "xbar", "xprev") else torch.float32
                n, pad = int(np.prod(shape)), 8 * nx * ny
                room = torch.full((n + 2 * pad,), around, device=cuda, dtype=kind)
                state[name] = room[pad:pad + n].view(shape)
                state[name].copy_(torch.rand(shape, device=cuda, generator=g) * (1.0 if name != "flow" else 0.9))
            state["proj"] = (torch.rand((frames, 2, 20, 24), device=cuda, generator=g) * 10).to(dt)
            _solve(stt, torch, cuda, dims, state, mode, storage, frames)
            outs.append({k: state[k].float().clone() for k in NAMES})
    for o in outs[1:]:
        for k in NAMES:
            assert torch.isfinite(o[k]).all() and torch.equal(o[k], outs[0][k]), k


def test_past_2_30_voxels(cuda):
    import torch

    import spacetimetomography_b200 as stt

    nz, ny, nx, short, edge = 1040, 1024, 1024, 16, 4
    assert 2 * nz * ny * nx > 2**31
    g = torch.Generator(device=cuda)
    g.manual_seed(5)
    ends = torch.rand((short, ny, nx), device=cuda, generator=g)
    step = (0.25, -0.5, 0.75)  # (coordinates exact in FP32 at either depth)
    results = []
    for depth in (short, nz):
        shape = (depth, ny, nx)
        z = lambda *s: torch.zeros(s + shape, device=cuda)  # noqa: E731
        state = dict(vol=z(2), xbar=z(2), xprev=z(1), ytv=z(1, 3), ytp=z(1), ybc=z(1), flow=z(1, 3),
                     proj=torch.zeros((1, 1, 5, 5), device=cuda))
        state["xbar"][1, -short:] = ends
        for a in range(3):
            state["flow"][0, a] = step[a]
        ctx = stt.Context(0)
        ctx.set_geometry((nx, ny, depth), (1.0, 1.0, 1.0), (5, 5), 1.0, 2000.0, 3000.0, [0.0])
        pd = stt.PdParams(tv_w=0.02, tp_w=0.1, bc_w=0.5, huber_factor=0.9, gmax=3.0, cut=(0,) * 8)
        s = stt.Solver(ctx, state, 1, 1, pd, seed=3, mode=stt.SOLVE_STREAMS)
        s.iterate(1)
        torch.cuda.synchronize()
        s.poll_status()
        results.append(state["ybc"][0, -short + edge:-1].clone())
        s.close()
        ctx.close()
        del state, s, ctx
        torch.cuda.empty_cache()
    assert torch.equal(*results) and float(results[0].abs().max()) > 0.05

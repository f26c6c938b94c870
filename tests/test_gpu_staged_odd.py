"""Volumes of extents that the slab-staged projector does not take: the tuner stages
no view of them, and a solver whose choice stages some runs the launches of one
that stages none (no z-fastest copies that nothing would read)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

DET, VIEWS = (72, 64), 10


def _context(stt, dims):
    ctx = stt.Context(0)
    ctx.set_geometry(dims, (1.0, 1.0, 1.0), DET, 1.2, 600.0, 1000.0, np.linspace(0.1, 6.0, VIEWS))
    return ctx


def _launches(stt, torch, cuda, ctx, dims, storage):
    nx, ny, nz = dims
    dt = torch.bfloat16 if storage == "bf16" else torch.float32
    z = lambda *s: torch.zeros(s, device=cuda, dtype=dt)  # noqa: E731
    f = lambda *s: torch.zeros(s, device=cuda)  # noqa: E731
    state = dict(vol=z(2, nz, ny, nx), xbar=z(2, nz, ny, nx), xprev=z(1, nz, ny, nx), ytv=f(1, 3, nz, ny, nx),
                 ytp=f(1, nz, ny, nx), ybc=f(1, nz, ny, nx), flow=f(1, 3, nz, ny, nx),
                 proj=torch.rand((1, VIEWS, DET[1], DET[0]), device=cuda).to(dt))
    pd = stt.PdParams(tv_w=0.02, tp_w=0.0, bc_w=0.0, huber_factor=0.9, gmax=5.0)
    s = stt.Solver(ctx, state, 1, VIEWS, pd, seed=1, storage=storage)
    s.iterate(1)
    torch.cuda.synchronize()
    n = s.stats()[0]
    s.close()
    return n


@pytest.mark.parametrize("storage", ["f32", "bf16"])
@pytest.mark.parametrize("dims", [(41, 36, 40), (40, 36, 41), (43, 41, 45)])
def test_nothing_is_copied_for_views_that_cannot_be_staged(cuda, dims, storage):
    import torch

    import spacetimetomography_b200 as stt

    ctx = _context(stt, dims)
    counts = []
    for staged in (0, 0x1FF):
        ctx.set_tuning(10, 0, 0, staged_bins=staged, fp_variant_bf16=1)
        counts.append(_launches(stt, torch, cuda, ctx, dims, storage))
    assert counts[0] == counts[1]
    ctx.close()


@pytest.mark.parametrize("dims,none16", [((43, 41, 45), True), ((44, 40, 52), True), ((48, 40, 56), False)])
def test_the_tuner_stages_nothing_without_boxes(cuda, dims, none16):
    import spacetimetomography_b200 as stt

    ctx = _context(stt, dims)
    t = ctx.autotune()
    if dims[0] % 4:
        assert t["staged_bins"] == 0
    if none16:  # BF16 boxes take multiples of 8
        assert t["staged_bins_bf16"] == 0
    ctx.close()

"""stt_get_tuning reports what a context runs, and setting back what was read
changes nothing: an untuned context stays untuned, with the same launches, for
volumes whose texture binds, whose mirror does, and that no texture admits."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

DET, VIEWS = (72, 64), 10


def _context(stt, dims):
    ctx = stt.Context(0)
    ctx.set_geometry(dims, (1.0, 1.0, 1.0), DET, 2.0, 1200.0, 2000.0, np.linspace(0.1, 6.0, VIEWS))
    return ctx


def _round_trip(ctx, **changed):
    """The C struct read, some fields changed, and set."""
    from spacetimetomography_b200._lib import Tuning, lib

    t = Tuning()
    assert lib.stt_get_tuning(ctx._h, C.byref(t)) == 0
    for k, v in changed.items():
        setattr(t, k, v)
    assert lib.stt_set_tuning(ctx._h, C.byref(t)) == 0


def _solver_launches(stt, torch, cuda, ctx, dims, storage):
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


# 372 x 364 texels a slice are past the texture width (131072)
@pytest.mark.parametrize("dims,admits", [((48, 40, 56), True), ((41, 37, 43), True), ((372, 364, 8), False)])
@pytest.mark.parametrize("storage", ["f32", "bf16"])
def test_setting_what_was_read_changes_nothing(cuda, dims, admits, storage):
    import torch

    import spacetimetomography_b200 as stt

    fresh, trip = _context(stt, dims), _context(stt, dims)
    before = trip.get_tuning()
    assert not before["tuned"]
    assert (before["fp_variant"], before["staged_bins"]) == ((10, 0) if admits else (5, 0x1E0))
    assert (before["fp_variant_bf16"], before["staged_bins_bf16"]) == ((1, 0) if admits else (0, 0x1E0))
    _round_trip(trip)
    assert trip.get_tuning() == before
    want = _solver_launches(stt, torch, cuda, fresh, dims, storage)
    assert _solver_launches(stt, torch, cuda, trip, dims, storage) == want
    _round_trip(trip, bp_variant=1)  # one field of another kernel: the projector keeps its form
    assert _solver_launches(stt, torch, cuda, trip, dims, storage) == want
    after = trip.get_tuning()
    assert after["tuned"] and after["bp_variant"] == 1
    assert all(after[k] == before[k] for k in ("fp_variant", "staged_bins", "fp_variant_bf16", "staged_bins_bf16"))
    for c in (fresh, trip):
        c.close()


def test_choices_that_are_set_are_kept(cuda):
    import spacetimetomography_b200 as stt

    ctx = _context(stt, (48, 40, 56))
    for fp, bins, fp16, bins16 in ((0, 0x1E0, 0, 0x1E0), (10, 0x100, 1, 0x80), (11, 0, 0, 0), (5, 0x1E0, 1, 0)):
        ctx.set_tuning(fp, 3, 2, staged_bins=bins, fp_variant_bf16=fp16, staged_bins_bf16=bins16, ray_variant=1)
        _round_trip(ctx)
        t = ctx.get_tuning()
        assert (t["fp_variant"], t["staged_bins"], t["fp_variant_bf16"], t["staged_bins_bf16"]) == (fp, bins, fp16, bins16)
        assert (t["slab_variant"], t["bp_variant"], t["ray_variant"], t["tuned"]) == (3, 2, 1, True)
    ctx.close()


def test_a_tuned_context_is_tuned_whatever_it_chose(cuda):
    import spacetimetomography_b200 as stt

    ctx = _context(stt, (40, 40, 48))
    before = ctx.get_tuning()
    assert ctx.autotune()["tuned"] and ctx.get_tuning()["tuned"]
    ctx.set_tuning(before["fp_variant"], 0, 0, staged_bins=before["staged_bins"])
    assert ctx.get_tuning()["tuned"]
    again = _context(stt, (40, 40, 48))
    assert again.autotune()["from_cache"] and again.get_tuning()["tuned"]
    for c in (ctx, again):
        c.close()

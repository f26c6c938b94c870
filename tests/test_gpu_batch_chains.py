"""A batch whose instances ask for tuning makes its solvers several times; the
last ones still count every instance of the batch, on which the projector's form
depends."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _chains(batch, count):
    from spacetimetomography_b200._lib import lib

    f = lib.stt_internal_batch_chains
    f.argtypes, f.restype = [C.c_void_p, C.c_int], C.c_int
    return [f(batch._h, i) for i in range(count)]


@pytest.mark.parametrize("tuned", [(False, False, False), (True, True, True), (False, True, False)])
@pytest.mark.parametrize("dims", [(40, 36, 44), (41, 37, 43)])
def test_solvers_count_every_instance(cuda, dims, tuned):
    import torch

    import spacetimetomography_b200 as stt

    items = []
    for k, tune in enumerate(tuned):
        ctx = stt.Context(0)
        ctx.set_geometry(dims, (1.0, 1.0, 1.0), (64, 56), 1.2, 600.0, 1000.0, np.linspace(0.1, 5.0, 6))
        pd = stt.PdParams(tv_w=0.02, tp_w=0.0, bc_w=0.0, huber_factor=0.9, gmax=5.0)
        if any(tuned):  # views staged, so that the batch times both ways
            ctx.set_tuning(0, 0, 0, staged_bins=0x1FF)
        items.append(dict(ctx=ctx, vol=torch.zeros(dims[::-1], device=cuda),
                          proj=torch.rand((6, 56, 64), device=cuda), pd=pd, seed=k, autotune=tune))
    batch = stt.Batch(items, mode=stt.SOLVE_GRAPH)
    assert _chains(batch, len(items)) == [len(items)] * len(items)
    batch.close()
    for i in items:
        i["ctx"].close()


@pytest.mark.parametrize("asked", [True, False])
def test_slow_choices_give_way_to_the_untuned_ones(cuda, asked):
    """Instances that ask for tuning and whose contexts hold a far slower projector
    (loads, every view staged) end with the untuned choices; those that do not ask
    keep theirs."""
    import torch

    import spacetimetomography_b200 as stt

    dims, det = (128, 128, 128), (128, 128)
    items = []
    for k in range(3):
        ctx = stt.Context(0)
        ctx.set_geometry(dims, (1.0, 1.0, 1.0), det, 2.0, 600.0, 1000.0, np.linspace(0.1, 6.0, 24))
        default = ctx.get_tuning()
        ctx.set_tuning(3, 0, 0, staged_bins=0x1FF)
        pd = stt.PdParams(tv_w=0.02, tp_w=0.0, bc_w=0.0, huber_factor=0.9, gmax=5.0)
        items.append(dict(ctx=ctx, vol=torch.zeros(dims[::-1], device=cuda), proj=torch.rand((24,) + det, device=cuda),
                          pd=pd, seed=k, autotune=asked))
    batch = stt.Batch(items, mode=stt.SOLVE_GRAPH)
    for i in items:
        assert i["ctx"].get_tuning()["fp_variant"] == (default["fp_variant"] if asked else 3)
    batch.close()
    for i in items:
        i["ctx"].close()

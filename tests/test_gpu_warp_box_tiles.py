"""The boxed warp at the edges of its 32 x 8 blocks against the CPU restatement,
bit for bit: extents of one tile and one past it, the smallest volume, a
velocity that lands on nodes (fractions of zero on every axis, or on one), steps
that leave the volume, and a box that is not the grid's."""
import numpy as np
import pytest

import oracle_bind as ob

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(3, 3, 3), (4, 8, 32), (5, 9, 33), (3, 7, 31), (9, 17, 65)])
@pytest.mark.parametrize("kind", ["zero", "nodes", "one axis", "rough", "far"])
@pytest.mark.parametrize("scale", [1.0, 1.37])
def test_warp_box_tiles(cuda, shape, kind, scale):
    import torch

    import spacetimetomography_b200 as stt

    rng = np.random.default_rng(sum(shape))
    vel = rng.normal(size=(3,) + shape).astype(np.float32)
    if kind == "zero":
        vel[:] = 0
    elif kind == "nodes":
        vel = np.round(vel).astype(np.float32)
    elif kind == "one axis":
        vel[0] = vel[2] = 0
    elif kind == "far":
        vel *= 50
    src = rng.normal(size=(2,) + shape).astype(np.float32)
    box = tuple(scale * n for n in shape[::-1])
    out = stt.warp_box(torch.from_numpy(vel).to(cuda), torch.from_numpy(src).to(cuda), -1.0, box)
    np.testing.assert_array_equal(out.cpu().numpy(), ob.warp_box32(vel, src, -1.0, box))

"""The flow's fused iterations (a dual step and the next primal step in one
kernel) at the edges of their tiles and of their place between residual checks,
against the CPU restatement of the reference's level: bit for bit.

Extents on both sides of the 31 x 4 column tiles and of the runs along z,
ROIs that touch the faces, iteration counts on both sides of a check, a second
warp, and the norm without the Huber factor."""
import numpy as np
import pytest

import oracle_bind as ob

pytestmark = pytest.mark.gpu


def _run(shape, roi, max_iter, n_warps, norm=4, tol=0.0, seed=0):
    import torch

    import spacetimetomography_b200 as stt

    rng = np.random.default_rng(seed)
    i1 = ob.blur32(rng.uniform(0, 1, shape).astype(np.float32), 1.0)
    i2 = ob.blur32(rng.uniform(0, 1, shape).astype(np.float32), 1.0)
    v0 = rng.normal(scale=0.2, size=(3,) + shape).astype(np.float32)
    y0 = rng.normal(scale=0.1, size=(10,) + shape).astype(np.float32)
    f = stt.Flow(shape, stt.FlowParams(tol=tol, max_iter=max_iter, n_warps=n_warps, norm=norm, scales=1))
    d = lambda a: torch.from_numpy(a.copy()).cuda()  # noqa: E731
    V, Y = d(v0), d(y0)
    f.level(d(i1), d(i2), V, Y, roi)
    torch.cuda.synchronize()
    its, _ = f.stats()
    f.close()
    v, y, ref_its = ob.flow_level32(i1, i2, v0, y0, roi, tol=tol, max_iter=max_iter, n_warps=n_warps, norm=norm)[:3]
    np.testing.assert_array_equal(V.cpu().numpy(), v)
    np.testing.assert_array_equal(Y.cpu().numpy(), y)
    return its


@pytest.mark.parametrize("shape", [(3, 3, 3), (5, 4, 31), (6, 5, 32), (4, 8, 62), (7, 9, 63), (33, 3, 30), (40, 13, 5)])
@pytest.mark.parametrize("roi", [(0, 0, 0, 0, 0, 0), (1, 0, 0, 1, 1, 0)])
def test_tile_edges(cuda, shape, roi):
    _run(shape, roi, max_iter=11, n_warps=2, seed=sum(shape))


@pytest.mark.parametrize("last", [1, 2, 3, 48, 49, 50, 51, 52, 53, 99, 100, 101, 150])
def test_iteration_counts_around_the_checks(cuda, last):
    _run((6, 7, 33), (1, 1, 0, 1, 1, 1), max_iter=last - 1, n_warps=2, norm=4 if last % 2 else 2, seed=last)


def test_a_warp_that_stops_on_its_residual(cuda):
    its = _run((12, 10, 40), (0, 0, 0, 0, 0, 0), max_iter=400, n_warps=3, tol=0.9, seed=5)
    assert all(k % 50 == 0 and k < 401 for k in its), its


@pytest.mark.parametrize("shape", [(85, 88, 99), (90, 90, 90), (106, 104, 105), (109, 110, 111)])
def test_volumes_around_the_l2(cuda, shape):
    """Both sides of the sizes whose dual and primal steps run as two kernels."""
    _run(shape, (2, 1, 3, 1, 2, 4), max_iter=6, n_warps=1, seed=shape[0])

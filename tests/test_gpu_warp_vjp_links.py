"""The warp's vector-Jacobian product, whose rows of atomics are merged between
neighbouring lanes, on rows that end inside a warp and flows that link all of its
lanes, some or none: steps within a cell, stretched and squeezed along x (several
lanes in one cell), sheared, and far out of the volume.

The images are linear, so no sample reaches its clamp's corners and the oracle
in FP64 takes the same branches.  Tolerance: a traced coordinate below 128 is rounded
some four times by up to 3.8e-6, so fractions are 4e-6 off and the weights, whose
slopes are about one per axis, 1e-5 relative: 2e-5; the velocity's gradient goes
through a second sample: 4e-5.  The gradient's oracle is the kernel itself with no
two lanes linked (a fifth of the output's columns at a time: the product is linear
in them): the reference's slope jumps where a coordinate meets a node, which the
stretched and squeezed rows of odd length do, and FP32 and FP64 round to different
sides of it."""
import numpy as np
import pytest

import oracle_bind as ob

pytestmark = pytest.mark.gpu

FLOWS = {  # v = v0 + G (x, y, z)
    "step": ((0.37, -0.23, 0.41), np.diag([0.011, 0.007, 0.013])),
    "stretch": ((0.2, 0.3, -0.4), np.diag([0.6, 0.01, 0.01])),
    "squeeze": ((0.2, 0.3, -0.4), np.diag([-0.7, 0.01, 0.01])),
    "shear": ((0.1, 0.2, 0.3), np.array([[0.02, 0.3, 0.1], [0.25, 0.01, 0.2], [0.15, -0.2, 0.01]])),
    "far": ((40.0, -30.0, 25.0), np.diag([0.011, 0.007, 0.013])),
}


def _grid(shape):
    z, y, x = np.mgrid[0:shape[0], 0:shape[1], 0:shape[2]].astype(np.float64)
    return np.stack([x, y, z])


@pytest.mark.parametrize("shape", [(4, 4, 4), (5, 6, 31), (6, 9, 32), (5, 7, 33), (4, 5, 65)])
@pytest.mark.parametrize("flow", sorted(FLOWS))
def test_linked_rows(cuda, shape, flow):
    import torch

    import spacetimetomography_b200 as stt

    rng = np.random.default_rng(sum(shape))
    v0, g = FLOWS[flow]
    xyz = _grid(shape)
    c = np.array([(n - 1) * 0.5 for n in shape[::-1]])
    vel = (np.array(v0)[:, None, None, None] + np.tensordot(g, xyz - c[:, None, None, None], 1)).astype(np.float32)
    src = np.stack([np.tensordot(w, xyz, 1) for w in ((0.5, 0.3, 0.7), (-0.2, 0.9, 0.4))]).astype(np.float32)
    bar = rng.normal(size=src.shape).astype(np.float32)
    d = lambda a: torch.from_numpy(a).to(cuda)  # noqa: E731
    sb, vb = torch.zeros(src.shape, device=cuda), torch.zeros(vel.shape, device=cuda)
    stt.warp_vjp(d(vel), d(src), 1.0, d(bar), sb, vb)
    rs, rv = ob.warp_vjp64(vel.astype(np.float64), src.astype(np.float64), 1.0, bar.astype(np.float64))
    assert ob.rel_l2(sb.cpu().numpy(), rs) < 2e-5
    apart = np.zeros(vel.shape)
    for k in range(5):
        some = np.zeros_like(bar)
        some[..., k::5] = bar[..., k::5]
        part = torch.zeros(vel.shape, device=cuda)
        stt.warp_vjp(d(vel), d(src), 1.0, d(some), None, part)
        apart += part.cpu().numpy()
    assert ob.rel_l2(vb.cpu().numpy(), apart) < 4e-5
    if flow in ("step", "shear", "far"):
        assert ob.rel_l2(vb.cpu().numpy(), rv) < 4e-5


def test_rough_fields_conserve(cuda):
    """Random images and flows (clamped samples between linked ones): a sample's
    weights sum to one on either branch, so the totals are kept per channel."""
    import torch

    import spacetimetomography_b200 as stt

    rng = np.random.default_rng(4)
    shape = (12, 18, 70)
    vel, src = rng.normal(size=(3,) + shape) * 0.6, rng.normal(size=(2,) + shape)
    bar = rng.uniform(0.5, 1.5, size=src.shape)
    bar[:, ::2, ::3, ::7] = 0
    d = lambda a: torch.from_numpy(a.astype(np.float32)).to(cuda)  # noqa: E731
    sb = torch.zeros(src.shape, device=cuda)
    stt.warp_vjp(d(vel), d(src), 1.0, d(bar), sb, None)
    np.testing.assert_allclose(sb.double().sum((1, 2, 3)).cpu().numpy(), bar.sum((1, 2, 3)), rtol=1e-5)

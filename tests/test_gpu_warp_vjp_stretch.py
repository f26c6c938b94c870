"""The warp's velocity gradient where neighbouring lanes share cells (stretched and
squeezed rows), against the FP64 oracle: outputs whose traced coordinates come within
2e-3 of a node on any axis, where the reference's slope jumps, carry no gradient; the
images are linear, so no sample reaches its clamp's corners.

Tolerance: that of the flows without such rows, 4e-5 (fractions 4e-6 off, through two
samples)."""
import numpy as np
import pytest

import oracle_bind as ob

pytestmark = pytest.mark.gpu

FLOWS = {  # v = v0 + G (x, y, z)
    "stretch": ((0.213, 0.307, -0.411), np.diag([0.6, 0.013, 0.017])),
    "squeeze": ((0.213, 0.307, -0.411), np.diag([-0.7, 0.013, 0.017])),
    "both": ((0.113, -0.207, 0.311), np.array([[0.5, 0.1, 0.0], [0.05, -0.6, 0.1], [0.0, 0.1, 0.4]])),
}


@pytest.mark.parametrize("shape", [(6, 8, 12), (5, 6, 31), (6, 9, 32), (5, 7, 33), (7, 9, 66)])
@pytest.mark.parametrize("flow", sorted(FLOWS))
def test_shared_cells(cuda, shape, flow):
    import torch

    import spacetimetomography_b200 as stt

    rng = np.random.default_rng(sum(shape))
    v0, g = FLOWS[flow]
    z, y, x = np.mgrid[0:shape[0], 0:shape[1], 0:shape[2]].astype(np.float64)
    xyz = np.stack([x, y, z])
    dims = np.array(shape[::-1], np.float64)[:, None, None, None]
    c = (dims - 1) * 0.5
    v0 = np.array(v0)[:, None, None, None]
    field = lambda p: v0 + np.tensordot(g, np.clip(p, 1, dims - 2) - c, 1)  # noqa: E731
    vel = (v0 + np.tensordot(g, xyz - c, 1)).astype(np.float32)
    src = np.stack([np.tensordot(w, xyz, 1) for w in ((0.5, 0.3, 0.7), (-0.2, 0.9, 0.4))]).astype(np.float32)
    # the trace in grid coordinates: dt = 1 steps back along the flow
    first = xyz - field(xyz)
    last = 0.5 * (xyz + first) - 0.5 * field(first)
    near = np.zeros(shape, bool)
    for p in (first, last):
        inside = (p > 1 - 2e-3) & (p < dims - 2 + 2e-3)  # (past these the coordinate is held, on a node, without a slope)
        near |= (inside & (np.abs(p - np.round(p)) < 2e-3)).any(axis=0)
    bar = rng.normal(size=src.shape).astype(np.float32)
    bar[:, near] = 0
    assert near.mean() < 0.3
    d = lambda a: torch.from_numpy(a).to(cuda)  # noqa: E731
    sb, vb = torch.zeros(src.shape, device=cuda), torch.zeros(vel.shape, device=cuda)
    stt.warp_vjp(d(vel), d(src), 1.0, d(bar), sb, vb)
    rs, rv = ob.warp_vjp64(vel.astype(np.float64), src.astype(np.float64), 1.0, bar.astype(np.float64))
    assert ob.rel_l2(sb.cpu().numpy(), rs) < 2e-5
    assert ob.rel_l2(vb.cpu().numpy(), rv) < 4e-5

"""The voxel backprojection from a detector of more than 2^32 pixels: the rows past
that offset are read where they lie.  The correction depends on the row alone, so
a narrow detector of the same rows gives the same update but for the rounding of
the x weights.

Tolerance: a Catmull-Rom row sums four products whose weights add up to 1 and to
at most 1.25 in absolute value; weights, products and sums each round by 2^-24,
some 12 roundings on either side of the comparison, and the y weights multiply
that by at most 1.25: 2 x 12 x 1.25^2 x 2^-24 < 2.3e-6 of the largest row value."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_rows_past_2_32_pixels(cuda):
    import torch

    import spacetimetomography_b200 as stt

    dims, H = (8, 600, 8), 1024
    rows = torch.from_numpy(np.random.default_rng(2).normal(size=H).astype(np.float32)).to(cuda)
    out = []
    for W in (64, 4_500_000):
        ctx = stt.Context(0)
        ctx.set_geometry(dims, (1.0, 1.0, 1.0), (W, H), 1.0, 600.0, 1000.0, [0.0])
        corr = rows[:, None].expand(H, W).contiguous()
        vol = torch.full(dims[::-1], 10.0, device=cuda)
        ctx.bp_voxel(corr, vol, 1.0, 100.0, 0)
        out.append(vol.cpu().numpy().astype(np.float64) - 10.0)
        ctx.close()
    # the last rows that voxels reach lie past 2^32 pixels of the wide detector
    last = (H - 1) / 2 + (dims[1] - 1) / 2 * 1000.0 / (600.0 + (dims[2] - 1) / 2)
    assert (last - 2) * 4_500_000 > 2**32
    bound = 2.3e-6 * float(rows.abs().max()) + 2 * 14.0 * 2.0**-24  # (the volume's own rounding, at 14 at most)
    assert np.abs(out[1] - out[0]).max() <= bound
    assert (np.abs(out[0][:, -8:]) > 1e-3).mean() > 0.5

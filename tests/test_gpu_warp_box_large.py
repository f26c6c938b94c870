"""The boxed warp of a grid of more than 2^31 voxels: its first and last planes
are, bit for bit, those of a short grid with the same values (a uniform flow of
quarter voxels, whose coordinates are exact in FP32 on either grid)."""
import pytest

pytestmark = pytest.mark.gpu


def test_warp_box_past_2_31_voxels(cuda):
    import torch

    import spacetimetomography_b200 as stt

    nz, ny, nx, short, edge = 2056, 1024, 1024, 16, 3
    assert nz * ny * nx > 2**31
    g = torch.Generator(device=cuda)
    g.manual_seed(5)
    step = (0.25, -0.5, 0.75)
    ends = [torch.randn((short, ny, nx), device=cuda, generator=g) for _ in range(2)]
    want = []
    for src in ends:
        vel = torch.stack([torch.full_like(src, s) for s in step])
        want.append(stt.warp_box(vel, src, -1.0, (nx, ny, short)))
    src = torch.zeros((nz, ny, nx), device=cuda)
    src[:short], src[-short:] = ends
    vel = torch.empty((3, nz, ny, nx), device=cuda)
    for a in range(3):
        vel[a] = step[a]
    out = stt.warp_box(vel, src, -1.0, (nx, ny, nz))
    assert torch.equal(out[: short - edge], want[0][: short - edge])
    assert torch.equal(out[edge - short :], want[1][edge:])
    assert float(out[-1].abs().max()) > 0.5

"""A call's projections are the same bits whichever form its size and views lead to:
all views in one call, one by one, and from a copy of the volume at another
alignment.  A call that no copy of the volume pays for makes none."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

FORMS = [  # dims, detector, degrees: along z, along x, both, with and without slices that a texture steps over
    ((128, 96, 112), (160, 150), [0, 4, 9, 178, 357]),
    ((127, 95, 111), (160, 150), [0, 4, 9, 178, 357]),
    ((127, 95, 111), (160, 150), [12, 20, 24, 160, 337]),
    ((96, 96, 88), (420, 410), [88, 90, 93, 268, 271]),
    ((95, 97, 88), (420, 410), [88, 90, 93, 268, 271]),
    ((95, 97, 88), (96, 80), [0, 30, 60, 90, 135]),
]


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("case", range(len(FORMS)))
def test_every_form_gives_the_same_bits(cuda, case, dtype):
    import torch

    import spacetimetomography_b200 as stt

    dims, det, degrees = FORMS[case]
    ctx = stt.Context(0)
    ctx.set_geometry(dims, (1.0, 1.0, 1.0), det, 2.0 * max(dims) / det[0], 600.0, 1000.0, np.deg2rad(degrees))
    g = torch.Generator(device=cuda)
    g.manual_seed(case)
    vol = torch.rand(dims[::-1], device=cuda, generator=g).to(getattr(torch, dtype))
    shape = (len(degrees), det[1], det[0])
    together = ctx.fp_typed(vol, torch.zeros(shape, device=cuda))
    for v in range(len(degrees)):
        one = ctx.fp_typed(vol, torch.zeros((1,) + shape[1:], device=cuda), view0=v, nviews=1)
        assert torch.equal(one[0], together[v]), f"view {v}"
    room = torch.zeros(vol.numel() + 1, device=cuda, dtype=vol.dtype)  # a base one element off: no texture binds
    room[1:] = vol.reshape(-1)
    off = room[1:].reshape(vol.shape)
    assert torch.equal(ctx.fp_typed(off, torch.zeros(shape, device=cuda)), together)
    if dtype == "float32":
        b = torch.rand(shape, device=cuda, generator=g)
        for v in range(len(degrees)):
            out = []
            for x in (vol, off):
                rl, corr = torch.zeros(shape[1:], device=cuda), torch.zeros(shape[1:], device=cuda)
                out.append(ctx.fp_correction(x, b[v], rl, corr, v).clone())
            want = (b[v] - together[v]) / (rl + 1.0)
            assert torch.equal(out[0], want) and torch.equal(out[1], want), f"correction of view {v}"
    ctx.close()


def test_no_copy_where_none_pays(cuda):
    import torch

    import spacetimetomography_b200 as stt

    n = 255
    ctx = stt.Context(0)
    ctx.set_geometry((n, n, n), (1.0, 1.0, 1.0), (512, 512), 1.0, 600.0, 1000.0, np.deg2rad([0.0, 40.0]))
    vol = torch.rand((n, n, n), device=cuda)
    proj = torch.zeros((1, 512, 512), device=cuda)
    rl, corr = torch.zeros((512, 512), device=cuda), torch.zeros((512, 512), device=cuda)
    bytes_of = 4 * n**3

    def taken(call):
        torch.cuda.synchronize()
        free = torch.cuda.mem_get_info()[0]
        call()
        torch.cuda.synchronize()
        return free - torch.cuda.mem_get_info()[0]

    first = stt.Context(0)  # (the kernels are loaded)
    first.set_geometry((64, 64, 64), (1.0, 1.0, 1.0), (512, 512), 1.0, 600.0, 1000.0, np.deg2rad([0.0, 40.0]))
    first.fp(vol, torch.zeros((2, 512, 512), device=cuda))
    first.fp_correction(vol, proj[0], rl, corr, 0)
    first.close()
    assert taken(lambda: ctx.fp(vol, proj, view0=0, nviews=1)) < bytes_of // 2
    assert taken(lambda: ctx.fp_correction(vol, proj[0], rl, corr, 0)) < bytes_of // 2
    assert taken(lambda: ctx.fp(vol, proj, view0=1, nviews=1)) >= bytes_of  # an oblique view: the copy pays
    ctx.close()

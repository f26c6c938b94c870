"""A batch whose views are too many to be shared between warps when its instances
run side by side, and an instance of it alone, whose views are: the same bits."""
import numpy as np
import pytest

import oracle_bind as ob

pytestmark = pytest.mark.gpu


def _instances(stt, cuda, count, bf16):
    import torch

    dims, det, angles = (40, 36, 32), (96, 90), np.linspace(0.1, 5.9, 5)  # 8640 rays: shared by up to 7 chains
    scan = ob.Scan(dims, det)
    out = []
    for k in range(count):
        ctx = stt.Context(0)
        ctx.set_geometry(dims, scan.sp, det, scan.ds, scan.sid, scan.sdd, angles, (0.3, 0.0, 0.0))
        g = torch.Generator(device=cuda)
        g.manual_seed(k)
        vol = torch.rand(dims[::-1], device=cuda, generator=g)
        proj = torch.rand((len(angles), det[1], det[0]), device=cuda, generator=g) * 30
        if bf16:
            vol, proj = vol.to(torch.bfloat16), proj.to(torch.bfloat16)
        sigma = 0.9 / 8.0
        pd = stt.PdParams(sigma=sigma, tau=1.0, tv_w=0.01, tp_w=0.0, bc_w=0.0, huber_factor=1.0 / (1.0 + sigma),
                          gmax=10.0, cut=(1, 1, 1, 1, 1, 1, 2, 2))
        out.append(dict(ctx=ctx, vol=vol, proj=proj, bp_mode=0, alpha=0.3, pd=pd, seed=k + 3,
                        roi_cut=(1, 1, 1, 1, 1, 1, 2, 2), storage="bf16" if bf16 else "f32"))
    return out


@pytest.mark.parametrize("bf16", [False, True])
@pytest.mark.parametrize("count", [7, 8])
def test_shared_views_of_a_batch(cuda, count, bf16):
    import torch

    import spacetimetomography_b200 as stt

    many, one = _instances(stt, cuda, count, bf16), _instances(stt, cuda, count, bf16)[-1:]
    for inst in (many, one):
        batch = stt.Batch(inst, mode=stt.SOLVE_GRAPH)
        batch.iterate(2)
        torch.cuda.synchronize()
        batch.close()
    assert torch.equal(many[-1]["vol"], one[0]["vol"])

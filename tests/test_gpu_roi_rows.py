"""The region-of-interest mask at the end of a SART call, on volumes whose rows
end inside a thread's eight: vol * mask of the oracle, bit for bit (so a masked
voxel keeps its sign and a NaN, a kept one everything)."""
import numpy as np
import pytest

import oracle_bind as ob

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ny", [2, 7, 8, 9, 23, 64])
@pytest.mark.parametrize("cut", [(1, 1, 1, 1, 1, 1, 3, 2), (0, 0, 0, 0, 0, 0, 0, 0), (40, 0, 0, 0, 0, 0, 0, 0)])
@pytest.mark.parametrize("bf16", [False, True])
def test_mask_rows(cuda, ny, cut, bf16):
    import torch

    import spacetimetomography_b200 as stt

    dims = (33, ny, 18)
    scan = ob.Scan(dims, (8, 8), ds=8.0)
    ctx = stt.Context(0)
    ctx.set_geometry(dims, scan.sp, (8, 8), 8.0, scan.sid, scan.sdd, np.zeros(1), (0, 0, 0))
    v = np.random.default_rng(ny).normal(size=(18, ny, 33)).astype(np.float32)
    v[::3, :, ::5] = np.nan
    v[1::3, :, 1::5] = np.inf
    vol = torch.from_numpy(v).to(cuda)
    mask = torch.from_numpy(ob.roi_mask(dims, cut).reshape(18, ny, 33).astype(np.float32)).to(cuda)
    if bf16:
        vol = vol.to(torch.bfloat16)
    want = (vol.float() * mask).to(vol.dtype)
    proj = torch.zeros((1, 8, 8), device=cuda, dtype=vol.dtype)
    ctx.sart_sweep(vol, proj, np.zeros(0, np.int32), 0.3, 1.0, 0, torch.zeros((8, 8), device=cuda), roi_cut=cut)
    nan = torch.isnan(want)
    assert torch.equal(torch.isnan(vol), nan)
    assert torch.equal(vol[~nan], want[~nan])
    assert torch.equal(torch.signbit(vol[~nan]), torch.signbit(want[~nan]))
    ctx.close()

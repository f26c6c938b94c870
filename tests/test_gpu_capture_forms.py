"""A context that has projected one view may be captured projecting others: whatever
copies and textures they would use outside a capture, those that are not there yet
are done without, and the replay gives the same bits."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ANGLES = np.deg2rad([0.0, 91.0, 268.0, 40.0, 180.0])


@pytest.mark.parametrize("dims,det", [((48, 40, 44), (96, 80)), ((47, 41, 45), (96, 80)), ((47, 41, 45), (420, 400)),
                                      ((48, 40, 44), (420, 400)), ((372, 364, 8), (60, 50))])
@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
def test_other_views_than_the_first_call_s(cuda, dims, det, dtype):
    import torch

    import spacetimetomography_b200 as stt

    def context():
        ctx = stt.Context(0)
        ctx.set_geometry(dims, (1.0, 1.0, 1.0), det, 2.0 * max(dims) / det[0], 1200.0, 2000.0, ANGLES)
        return ctx

    vol = torch.rand(dims[::-1], device=cuda).to(getattr(torch, dtype))
    n, shape = len(ANGLES), (len(ANGLES), det[1], det[0])
    plain, ctx = context(), context()
    want = plain.fp_typed(vol, torch.zeros(shape, device=cuda))
    b = torch.rand(shape, device=cuda)
    corr_want = []
    if dtype == "float32":
        for v in range(n):
            corr = torch.zeros(shape[1:], device=cuda)
            plain.fp_correction(vol, b[v], torch.zeros(shape[1:], device=cuda), corr, v)
            corr_want.append(corr)
    out, corr = torch.zeros(shape, device=cuda), torch.zeros(shape, device=cuda)
    lens = torch.zeros(shape, device=cuda)
    ctx.fp_typed(vol, out, view0=0, nviews=1)
    torch.cuda.synchronize()
    s, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=s):
        ctx.fp_typed(vol, out, stream=s)
        ctx.fp_typed(vol, out[1:3], view0=1, nviews=2, stream=s)
        if dtype == "float32":
            for v in range(n):
                ctx.fp_correction(vol, b[v], lens[v], corr[v], v, stream=s)
    out.zero_()
    torch.cuda.synchronize()
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(out, want)
    for v, w in enumerate(corr_want):
        assert torch.equal(corr[v], w), v
    del graph
    for c in (plain, ctx):
        c.close()

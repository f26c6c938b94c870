"""Calls of one context that overlap on several streams, on volumes whose slices
no texture binds (the projections gather from a mirror that the context keeps):
each gets its own volume's projections, bit for bit those of the call alone,
also when one of them is the replay of a captured graph, and when the context had
another geometry between the capture and the replay."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

DIMS, DET = (151, 149, 150), (200, 180)
ANGLES = np.deg2rad([33.0, 127.0, 40.0, 215.0, 310.0, 50.0])


def _context(stt, dims=DIMS):
    ctx = stt.Context(0)
    ctx.set_geometry(dims, (1.0, 1.0, 1.0), DET, 1.5, 600.0, 1000.0, ANGLES)
    return ctx


def _volumes(torch, cuda, dtype, count):
    g = torch.Generator(device=cuda)
    g.manual_seed(3)
    return [torch.rand(DIMS[::-1], device=cuda, generator=g).to(dtype) for _ in range(count)]


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
def test_two_streams(cuda, dtype):
    import torch

    import spacetimetomography_b200 as stt

    vols = _volumes(torch, cuda, getattr(torch, dtype), 4)
    ctx = _context(stt)
    want = []
    for v in vols:
        want.append(ctx.fp_typed(v, torch.zeros((len(ANGLES), DET[1], DET[0]), device=cuda)))
    streams = [torch.cuda.Stream() for _ in vols]
    out = [torch.zeros_like(w) for w in want]
    torch.cuda.synchronize()
    for _ in range(10):
        for o in out:
            o.zero_()
        torch.cuda.synchronize()
        for v, o, s in zip(vols, out, streams):
            ctx.fp_typed(v, o, stream=s)
        torch.cuda.synchronize()
        for w, o in zip(want, out):
            assert torch.equal(w, o)
    ctx.close()


def test_a_replay_beside_calls(cuda):
    import torch

    import spacetimetomography_b200 as stt

    a, b = _volumes(torch, cuda, torch.float32, 2)
    ctx = _context(stt)
    shape = (len(ANGLES), DET[1], DET[0])
    want = [ctx.fp(v, torch.zeros(shape, device=cuda)) for v in (a, b)]
    torch.cuda.synchronize()
    graph, oa, ob = torch.cuda.CUDAGraph(), torch.zeros(shape, device=cuda), torch.zeros(shape, device=cuda)
    s = torch.cuda.Stream()
    with torch.cuda.graph(graph, stream=s):
        for _ in range(3):
            ctx.fp(a, oa, stream=s)
    other = torch.cuda.Stream()
    for k in range(10):
        oa.zero_()
        ob.zero_()
        torch.cuda.synchronize()
        if k % 2:
            ctx.fp(b, ob, stream=other)
        with torch.cuda.stream(s):
            graph.replay()
        ctx.fp(b, ob, stream=other)
        torch.cuda.synchronize()
        assert torch.equal(oa, want[0]) and torch.equal(ob, want[1])
    # another geometry for a while, then the first one again: the graph still replays
    small = tuple(n - 10 for n in DIMS)
    ctx.set_geometry(small, (1.0, 1.0, 1.0), DET, 1.5, 600.0, 1000.0, ANGLES)
    c = torch.rand(small[::-1], device=cuda)
    oc = ctx.fp(c, torch.zeros(shape, device=cuda))
    fresh = _context(stt, small)
    assert torch.equal(oc, fresh.fp(c, torch.zeros(shape, device=cuda)))
    ctx.set_geometry(DIMS, (1.0, 1.0, 1.0), DET, 1.5, 600.0, 1000.0, ANGLES)
    oa.zero_()
    torch.cuda.synchronize()
    with torch.cuda.stream(s):
        graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(oa, want[0])
    fresh.close()
    del graph
    ctx.close()

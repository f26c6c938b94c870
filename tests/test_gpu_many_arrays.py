"""A context that is given one array after another: each is projected from its own
texture, however many came before (no copy of a volume that binds itself), and a
captured projection stays valid while others come and go."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ANGLES = np.deg2rad([33.0, 127.0, 250.0])


def _context(stt, n, det):
    ctx = stt.Context(0)
    ctx.set_geometry((n, n, n), (1.0, 1.0, 1.0), (det, det), 2.0 * n / det, 600.0, 1000.0, ANGLES)
    return ctx


def test_no_volume_is_copied_for_want_of_a_texture(cuda):
    import torch

    import spacetimetomography_b200 as stt

    n, det = 128, 96
    ctx = _context(stt, n, det)
    room = torch.rand((44, n, n, n), device=cuda)  # 8 MiB each
    proj = torch.zeros((len(ANGLES), det, det), device=cuda)
    free = []
    for vol in room:
        ctx.fp(vol, proj)
        torch.cuda.synchronize()
        free.append(torch.cuda.mem_get_info()[0])
    assert free[0] - free[-1] < 4 * n**3 // 2
    ctx.close()


def test_hundreds_of_arrays_and_a_capture(cuda):
    import torch

    import spacetimetomography_b200 as stt

    n, det, count = 16, 40, 700
    ctx = _context(stt, n, det)
    room = torch.rand((count, n, n, n), device=cuda)
    shape = (len(ANGLES), det, det)
    kept = torch.zeros(shape, device=cuda)
    ctx.fp(room[0], kept)
    want = kept.clone()
    s, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=s):
        ctx.fp(room[0], kept, stream=s)
    out = torch.zeros((count,) + shape, device=cuda)
    for vol, o in zip(room, out):
        ctx.fp(vol, o)
    torch.cuda.synchronize()
    for k in range(0, count, 90):
        fresh = _context(stt, n, det)
        assert torch.equal(out[k], fresh.fp(room[k], torch.zeros(shape, device=cuda))), k
        fresh.close()
    assert torch.equal(out[0], want)
    kept.zero_()
    torch.cuda.synchronize()
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(kept, want)
    del graph
    ctx.close()

"""Enhancement of frames that are rewritten right before each call, with nothing waited for in
between: in the stream, and in a caller's captured graph whose frame comes from a side stream."""
import pytest

import piv_b200 as P

pytestmark = pytest.mark.gpu


def test_rewritten_frames(cuda):
    import torch

    Nx, Ny = 1000, 700
    base = torch.randint(0, 256, (Ny, Nx), device="cuda", generator=torch.Generator("cuda").manual_seed(3), dtype=torch.int32)
    frames = [(base * (k + 1) % 251).to(torch.uint8) for k in range(3)]
    m = P.mhe_gpu()
    assert m.init(Nx, Ny, 40, 0.91)
    want = []
    for f in frames:
        torch.cuda.synchronize()
        assert m.processsing(f)
        torch.cuda.synchronize()
        want.append(m.d_enhanced.clone())
    src, got = frames[0].clone(), []
    for k in range(60):
        src.copy_(frames[k % 3])
        assert m.processsing(src)
        got.append(m.d_enhanced.clone())
    torch.cuda.synchronize()
    assert all(torch.equal(g, want[k % 3]) for k, g in enumerate(got))

    factor, res = torch.ones(1, dtype=torch.int32, device="cuda"), torch.empty_like(src)
    side, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        cur = torch.cuda.current_stream()
        side.wait_stream(cur)
        with torch.cuda.stream(side):
            x = (base * factor % 251).to(torch.uint8)
        cur.wait_stream(side)
        src.copy_(x)
        assert m.processsing(src)
        res.copy_(m.d_enhanced)
    for k in (2, 0, 1, 1):
        factor.fill_(k + 1)
        graph.replay()
        assert torch.equal(res, want[k]), k
    torch.cuda.synchronize()
    m.freemem()

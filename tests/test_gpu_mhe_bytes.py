"""Histogram equalisation of tiles whose rows start off a word: tiles narrower and wider than the
warp that walks them, in the pair's launch and on its own, against the oracle."""
import numpy as np
import pytest

import piv_b200 as P
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ws,thresh", [(1, 0.3), (2, 0.3), (5, 0.91), (7, 0.91), (31, 0.91), (32, 0.91), (33, 0.91), (40, 0.91),
                                       (64, 0.91), (65, 0.5), (97, 0.91), (150, 0.91)])
def test_unaligned_tiles_exact(cuda, ws, thresh):
    import torch

    Nx, Ny = 2 * max(ws, 40) + 1 + 2 * (ws % 2), max(150, 2 * ws + 3)
    assert Nx % 4  # rows off the word
    rng = np.random.default_rng(ws)
    f1 = rng.integers(0, 256, (Ny, Nx), dtype=np.uint8)
    f2 = (rng.gamma(2.0, 20.0, (Ny, Nx)).clip(0, 255)).astype(np.uint8)
    want = O.mhe(f1, ws, thresh), O.mhe(f2, ws, thresh)
    p = P.default_params(Nx=Nx, Ny=Ny, if_mhe=1, mhe_ws=ws, mhe_thresh=thresh, ws_x1=16, ws_y1=16, spacing_x1=8,
                         spacing_y1=8, Npass1=1, Npass2=0)
    with P.Engine(p) as e:
        e.set_images(f1, f2)
        e.prep()
        got = e.frames()
    assert np.array_equal(got[0], want[0]) and np.array_equal(got[1], want[1])
    m = P.mhe_gpu()
    assert m.init(Nx, Ny, ws, thresh)
    assert m.processsing(torch.from_numpy(f1).cuda())
    assert np.array_equal(m.d_enhanced.cpu().numpy().reshape(Ny, Nx), want[0])
    m.freemem()

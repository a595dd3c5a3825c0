"""Histogram equalisation of both frames in one launch: odd widths (unaligned rows), widths that
end inside a vector load, and tiles that do not divide the frame, each frame against the oracle."""
import numpy as np
import pytest

import piv_b200 as P
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("Nx,Ny,ws", [(97, 81, 40), (256, 128, 40), (161, 120, 16), (200, 99, 25), (640, 403, 136)])
def test_both_frames_exact(cuda, Nx, Ny, ws):
    rng = np.random.default_rng(Nx)
    f1 = rng.integers(0, 256, (Ny, Nx), dtype=np.uint8)
    f2 = (rng.gamma(2.0, 20.0, (Ny, Nx)).clip(0, 255)).astype(np.uint8)
    p = P.default_params(Nx=Nx, Ny=Ny, if_mhe=1, mhe_ws=ws, mhe_thresh=0.91, ws_x1=16, ws_y1=16, spacing_x1=8, spacing_y1=8,
                         Npass1=1, Npass2=0)
    with P.Engine(p) as e:
        for a, b in ((f1, f2), (f2, f1)):  # the levels of the pair before are cleared
            e.set_images(a, b)
            e.prep()
            g = e.frames()
            assert np.array_equal(g[0], O.mhe(a, ws, 0.91)) and np.array_equal(g[1], O.mhe(b, ws, 0.91))

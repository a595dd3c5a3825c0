"""Deformation by a caller-set predictor that holds NaN or infinities: exactly the pixels of the cells
with such a corner are NaN, all others are the bits of a run with numbers there.  Spacings of both
kernels, at the frame's border and inside."""
import numpy as np
import pytest

import piv_b200 as P

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sp", [(8, 8), (16, 16), (12, 12), (5, 7), (8, 6)], ids=lambda s: f"{s[0]}x{s[1]}")
@pytest.mark.parametrize("value", [np.nan, np.inf, -np.inf])
def test_cells_with_a_bad_corner(cuda, sp, value):
    Nx, Ny, ws = 301, 207, 16
    p = P.default_params(Nx=Nx, Ny=Ny, ws_x1=ws, ws_y1=ws, spacing_x1=sp[0], spacing_y1=sp[1], Npass1=2, Npass2=0)
    f1, f2 = P.synth_pair(P.synth_params(Nx, Ny, seed=4))
    rng = np.random.default_rng(sp[0])
    with P.Engine(p) as e:
        e.set_images(f1, f2)
        e.prep()
        nx, ny, nt = e.geom["Nx_vec"][0], e.geom["Ny_vec"][0], e.geom["Nt_vec"][0]
        d = rng.normal(0, 2, (2, nt)).astype(np.float32)
        bad = rng.random((2, nt)) < 0.03
        bad[0, 0] = bad[1, -1] = True
        out = []
        for v in (np.float32(0), np.float32(value)):
            q = np.where(bad, v, d)
            e.set_field(0, q[0], q[1], np.ones(nt, np.uint8))
            e.pass_grid1(1)
            out.append(e.deformed(0).copy())
    cells = []
    for n, N, s in ((nx, out[0].shape[1], sp[0]), (ny, out[0].shape[0], sp[1])):
        c = (np.arange(N) - (ws // 2 - 3 * s)) // s  # the cell's first corner in the extended field
        cells.append((np.clip(c - 3, 0, n - 1), np.clip(c - 2, 0, n - 1)))
    any_bad = bad.any(0).reshape(ny, nx)
    want = np.zeros(out[0].shape, bool)
    for y in cells[1]:
        for x in cells[0]:
            want |= any_bad[y[:, None], x[None, :]]
    assert want.any() and not want.all()
    assert np.array_equal(np.isnan(out[1]), want)
    assert np.array_equal(out[1][~want].view(np.uint32), out[0][~want].view(np.uint32))

"""The deformation kernels' runs: spacings that take the 8-pixel runs (powers of two or not) and the
column walk (cells of many rows, of a few, of one), odd extents, displacements that reach over every
border or far outside, against 64-bit NumPy on the zero-extended frame; and a NaN vector, whose runs fall back pixel by pixel:
the pixels beside it keep their bits."""
import numpy as np
import pytest

import piv_b200 as P
from oracle import oracle as O

pytestmark = pytest.mark.gpu

CASES = [(16, 16, 211, 83), (32, 8, 150, 129), (48, 24, 301, 150), (24, 12, 277, 111), (16, 5, 133, 97),
         (16, 4, 140, 90), (16, 1, 47, 35), (40, 20, 190, 301)]


def _deform(img, g, sp, ws, fx, fy):
    """Bilinear displacement, then bilinear interpolation of the zero-extended frame, in 64 bits."""
    nx, ny, w, h = g.Nx_vec[0], g.Ny_vec[0], g.Nx_aug[0], g.Ny_aug[0]

    def cells(n, count):
        t = (np.arange(n) - (ws // 2 - 3 * sp)) / sp
        i = np.floor(t).astype(int)
        return np.clip(i - 3, 0, count - 1), np.clip(i - 2, 0, count - 1), t - i

    (x0, x1, ax), (y0, y1, ay) = cells(w, nx), cells(h, ny)
    ay = ay[:, None]

    def sample(f):
        f = f.reshape(ny, nx).astype(np.float64)
        top = f[y0][:, x0] * (1 - ax) + f[y0][:, x1] * ax
        return top * (1 - ay) + (f[y1][:, x0] * (1 - ax) + f[y1][:, x1] * ax) * ay

    px = np.arange(w) + sample(fx) - g.Nx_left[0]
    py = np.arange(h)[:, None] + sample(fy) - g.Ny_left[0]
    i, j = np.floor(px).astype(int), np.floor(py).astype(int)
    a, b = px - i, py - j

    def tap(r, c):
        ok = (r >= 0) & (r < img.shape[0]) & (c >= 0) & (c < img.shape[1])
        return np.where(ok, img[np.clip(r, 0, img.shape[0] - 1), np.clip(c, 0, img.shape[1] - 1)], 0.0)

    return ((1 - a) * (1 - b) * tap(j, i) + a * (1 - b) * tap(j, i + 1) + (1 - a) * b * tap(j + 1, i) +
            a * b * tap(j + 1, i + 1))


@pytest.mark.parametrize("ws,sp,Nx,Ny", CASES, ids=lambda v: str(v))
def test_deformation_runs(cuda, ws, sp, Nx, Ny):
    f1, f2 = P.synth_pair(P.synth_params(Nx, Ny, ppp=0.05, seed=17))
    p = P.default_params(Nx=Nx, Ny=Ny, if_mhe=0, ws_x1=ws, ws_y1=ws, spacing_x1=sp, spacing_y1=sp, Npass1=2, Npass2=0)
    op = O.params_from(p)
    _, g = O.geometry(op)
    nx, ny = g.Nx_vec[0], g.Ny_vec[0]
    yy, xx = np.mgrid[0:ny, 0:nx].astype(np.float32)
    with P.Engine(p) as e:
        e.set_images(f1, f2)
        e.prep()

        def run(fx, fy):
            e.set_field(0, fx, fy, np.ones(nx * ny, np.uint8))
            e.pass_grid1(1)
            return e.deformed(0)

        for ax, ay in ((1.7, -2.2), (45.0, -38.0), (-3e3, 9e3)):
            fx = (ax * (1 + 0.3 * np.sin(xx / 2))).astype(np.float32).ravel()
            fy = (ay * (1 + 0.2 * np.cos(yy / 3))).astype(np.float32).ravel()
            got = run(fx, fy)
            want = _deform(f2, g, sp, ws, fx, fy)
            # positions below 512 px, rounded four times in FP32: 2 ulp = 6.1e-5 px per axis, times
            # at most 255 grey levels / px each; weights and sums of them: 8 roundings of 255
            assert np.abs(got - want).max() <= 2 * 255 * 6.1e-5 + 8 * 255 * 6e-8, (ax, ay)
            fx[(ny // 2) * nx + nx // 2] = np.nan
            bad = run(fx, fy)
            hit = np.isnan(bad)
            assert hit.any() and hit.sum() <= (2 * sp) ** 2 + 4 * sp * max(Nx, Ny) * (nx < 3 or ny < 3)
            assert np.array_equal(bad[~hit], got[~hit])

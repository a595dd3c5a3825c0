"""The fused correlation kernels' staged pixel rows and packed transforms: every shape at
spacings that take each form of the row copies (16-, 8- and 4-byte), odd window counts that leave
a last window without a partner, and all-zero windows, on the undeformed and the deformed pass.
The oracle is NumPy's 64-bit FFT of the engine's own frames."""
import numpy as np
import pytest

import piv_b200 as P

pytestmark = pytest.mark.gpu

SHAPES = [(8, 8), (12, 12), (16, 16), (24, 24), (32, 32), (48, 48), (64, 64), (48, 24), (24, 48), (32, 16), (16, 32),
          (64, 32), (32, 64)]


def _planes(f1, f2, g, sp, ws):
    """|IFFT(conj(F1) F2)|, fftshifted, of every window; f1, f2 padded to the grid's extent."""
    nx, ny = g["Nx_vec"][0], g["Ny_vec"][0]
    out = np.empty((nx * ny, ws[1], ws[0]))
    for w in range(nx * ny):
        y, x = (w // nx) * sp, (w % nx) * sp
        a, b = f1[y:y + ws[1], x:x + ws[0]], f2[y:y + ws[1], x:x + ws[0]]
        c = np.fft.ifft2(np.conj(np.fft.fft2(a)) * np.fft.fft2(b)) if a.any() and b.any() else np.zeros(a.shape)
        out[w] = np.fft.fftshift(np.abs(c))
    return out


@pytest.mark.parametrize("shape", SHAPES, ids=[f"{x}x{y}" for x, y in SHAPES])
@pytest.mark.parametrize("sp", [5, 6, 8])
def test_planes_match_numpy(cuda, monkeypatch, shape, sp):
    ws = shape
    Nx, Ny = 5 * sp + 2 * ws[0] + 1, 3 * sp + ws[1] + 2  # a few windows; odd counts among the spacings
    f1, f2 = P.synth_pair(P.synth_params(Nx, Ny, ppp=0.05, field=P.PIV_FIELD_UNIFORM, a=0.7, b=-0.4, seed=31 + sp))
    f1[: ws[1] // 2 + sp, : ws[0] // 2 + sp] = 0  # the first window has no frame 1
    p = P.default_params(Nx=Nx, Ny=Ny, ws_x1=ws[0], ws_y1=ws[1], spacing_x1=sp, spacing_y1=sp, Npass1=2, Npass2=0,
                         insert_threshold_p1=2.0)
    for variant in range(8):
        monkeypatch.setenv("PIV_XCORR_VARIANT", f"{variant},0")
        try:
            e = P.Engine(p)
        except P.PivError:
            assert variant > 1
            break
        with e:
            e.set_images(f1, f2)
            g = e.geom
            ext = np.zeros((2, g["Ny_aug"][0], g["Nx_aug"][0]))
            top, left = g["Ny_left"][0], g["Nx_left"][0]
            ext[0, top:top + Ny, left:left + Nx], ext[1, top:top + Ny, left:left + Nx] = f1, f2
            nt = g["Nt_vec"][0]
            e.prep()
            for j in range(2):
                e.pass_grid1(j)
                second = ext[1] if j == 0 else e.deformed(0).astype(np.float64)
                want = _planes(ext[0], second, g, sp, ws)
                got = e.cc_planes(0, 0, nt)
                peak = want.max((1, 2), keepdims=True)
                # FP32 transforms of at most 64x64 points: 2e-6 of the window's peak, as the other
                # plane tests; exactly zero where a frame's window is
                assert (np.abs(got - want) <= 2e-6 * peak).all(), (variant, j)
                e.validate_grid1()

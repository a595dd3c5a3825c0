"""The general-size correlation kernel's radix stages (2, 3, 4, 5, 7, 11, 13 and a larger prime in
both dimensions) against NumPy's 64-bit FFT, planes in shared memory and in the workspace, and its
two peak searches (a top-list per thread up to 8 saved peaks, rounds of an arg-max above) against
each other."""
import numpy as np
import pytest

import piv_b200 as P

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ws", [(20, 28), (52, 44), (60, 36), (76, 4), (4, 100), (96, 52), (256, 84)],
                         ids=lambda w: f"{w[0]}x{w[1]}")
def test_stages_and_peak_lists(cuda, ws):
    sp = 12
    Nx, Ny = ws[0] + 4 * sp + 3, ws[1] + 3 * sp + 1
    f1, f2 = P.synth_pair(P.synth_params(Nx, Ny, ppp=0.05, field=P.PIV_FIELD_UNIFORM, a=1.3, b=0.6, seed=ws[0]))
    lists = []
    for nps in (3, 8, 12):
        p = P.default_params(Nx=Nx, Ny=Ny, ws_x1=ws[0], ws_y1=ws[1], spacing_x1=sp, spacing_y1=sp, Npass1=1, Npass2=0,
                             Npeak_save=nps)
        with P.Engine(p) as e:
            e.set_images(f1, f2)
            e.prep()
            e.pass_grid1(0)
            g, nt = e.geom, e.geom["Nt_vec"][0]
            lists.append([v for v in e.peaks(0)] + list(e.field(0)[2:]))
            if nps == 3:
                ext = np.zeros((2, g["Ny_aug"][0], g["Nx_aug"][0]))
                top, left = g["Ny_left"][0], g["Nx_left"][0]
                ext[:, top:top + Ny, left:left + Nx] = f1, f2
                got = e.cc_planes(0, 0, nt)
                for w in range(nt):
                    y, x = (w // g["Nx_vec"][0]) * sp, (w % g["Nx_vec"][0]) * sp
                    a, b = ext[:, y:y + ws[1], x:x + ws[0]]
                    c = np.abs(np.fft.fftshift(np.fft.ifft2(np.conj(np.fft.fft2(a)) * np.fft.fft2(b))))
                    assert (np.abs(got[w] - c) <= 2e-6 * c.max()).all(), w
    # the lists agree on the peaks that they share, to the bit
    assert np.array_equal(lists[0][0], lists[1][0]) and np.array_equal(lists[1][0], lists[2][0])
    for k in range(1, 6):
        assert np.array_equal(lists[0][k], lists[1][k][:, :3]) and np.array_equal(lists[1][k], lists[2][k][:, :8])

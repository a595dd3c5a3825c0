"""An all-zero frame-1 window whose deformed frame-2 window holds NaN pixels (a caller-set
predictor that is no number).  Its correlation is zero, so the window that shares its inverse
transform keeps its own candidates: they are those of the same run with a number in that place,
for every fused shape and variant and the general-size kernel."""
import numpy as np
import pytest

import piv_b200 as P

pytestmark = pytest.mark.gpu

SHAPES = [(8, 8), (12, 12), (16, 16), (24, 24), (32, 32), (48, 48), (64, 64), (48, 24), (24, 48), (32, 16), (16, 32),
          (64, 32), (32, 64), (40, 40)]


@pytest.mark.parametrize("first", [True, False], ids=["first_of_pair", "second_of_pair"])
@pytest.mark.parametrize("ws", SHAPES, ids=[f"{x}x{y}" for x, y in SHAPES])
def test_partner_of_a_zero_window_keeps_its_candidates(cuda, monkeypatch, ws, first):
    sp = (ws[0] // 2, ws[1] // 2)
    Nx, Ny = 8 * sp[0] + ws[0], 4 * sp[1] + ws[1]
    f1, f2 = P.synth_pair(P.synth_params(Nx, Ny, ppp=0.08, field=P.PIV_FIELD_UNIFORM, a=0.4, b=-0.3, seed=17))
    p = P.default_params(Nx=Nx, Ny=Ny, ws_x1=ws[0], ws_y1=ws[1], spacing_x1=sp[0], spacing_y1=sp[1], Npass1=2, Npass2=0)
    g = P.geometry(p)
    nx = g["Nx_vec"][0]
    wy = 2
    wx = next(x for x in range(2, nx - 2) if ((wy * nx + x) % 2 == 0) == first)
    zero, side = wy * nx + wx, -1 if first else 1  # the NaN vector lies on the side away from the partner
    partner = zero - side
    f1 = f1.copy()
    y0, x0 = wy * sp[1] - g["Ny_left"][0], wx * sp[0] - g["Nx_left"][0]
    f1[y0:y0 + ws[1], x0:x0 + ws[0]] = 0
    tried = 0
    for variant in range(8):
        monkeypatch.setenv("PIV_XCORR_VARIANT", f"{variant},0")
        try:
            e = P.Engine(p)
        except P.PivError as err:
            assert err.status == P.PIV_ERR_ARG and tried >= 3, err  # past the shape's last variant
            break
        with e:
            e.set_images(f1, f2)
            e.prep()
            nt = e.geom["Nt_vec"][0]
            got = []
            for value in (0.0, np.nan):
                d = np.zeros(nt, np.float32)
                d[zero + side] = value
                e.set_field(0, d, d, np.ones(nt, np.uint8))
                e.pass_grid1(1)
                cut = e.deformed(0)[:, (wx - side) * sp[0]:][wy * sp[1]:wy * sp[1] + ws[1], :ws[0]]
                assert not np.isnan(cut).any()  # the partner sees none of it
                cnt, idx, val = e.peaks(0)
                _, _, dx, dy, ok = e.field(0)
                assert cnt[zero] == 0 and not ok[zero].any()
                got.append((cnt[partner], idx[partner], val[partner], dx[partner], dy[partner], ok[partner]))
            assert got[0][0] > 0
            for a, b in zip(*got):
                assert np.array_equal(a, b), variant
            tried += 1

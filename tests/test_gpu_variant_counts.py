"""The tile variants of every fused window shape: how many there are, which one each index names,
and that an index past the last is refused by name.  Every other failure to create an engine is one."""
import pytest

import piv_b200 as P

pytestmark = pytest.mark.gpu

# (windows per CTA, threads per CTA) by index
VARIANTS = {(8, 8): [(32, 128), (16, 128), (32, 256)], (12, 12): [(16, 96), (8, 96), (16, 192)],
            (16, 16): [(16, 128), (8, 128), (16, 256), (4, 64)], (24, 24): [(8, 96), (4, 96), (8, 192), (2, 64)],
            (32, 32): [(8, 128), (4, 128), (2, 64), (8, 256), (4, 64), (4, 128)],
            (48, 48): [(4, 96), (2, 96), (2, 64), (4, 192)], (64, 64): [(2, 128), (4, 128), (2, 64), (4, 256)],
            (48, 24): [(4, 96), (2, 64), (2, 96), (8, 192)], (24, 48): [(4, 96), (2, 64), (4, 128), (8, 192)],
            (32, 16): [(8, 128), (4, 64), (8, 256)], (16, 32): [(8, 128), (4, 64), (8, 256)],
            (64, 32): [(4, 128), (2, 64), (2, 128)], (32, 64): [(4, 128), (2, 64), (2, 128)]}


@pytest.mark.parametrize("shape", VARIANTS, ids=lambda s: f"{s[0]}x{s[1]}")
@pytest.mark.parametrize("nps", [4, 8])
def test_every_index(cuda, monkeypatch, capfd, shape, nps):
    wx, wy = shape
    f1, f2 = P.synth_pair(P.synth_params(3 * wx + 5, 3 * wy + 2, seed=wx))
    p = P.default_params(Nx=3 * wx + 5, Ny=3 * wy + 2, ws_x1=wx, ws_y1=wy, spacing_x1=wx // 2, spacing_y1=wy // 2, Npass1=2,
                         Npass2=0, Npeak_save=nps)
    fields = []
    for index, cta in enumerate(VARIANTS[shape]):
        monkeypatch.setenv("PIV_XCORR_VARIANT", f"{index},0")
        with P.Engine(p) as e:
            assert tuple(e.xcorr_config(0)[:2]) == cta
            e.set_images(f1, f2)
            e.run_pair()
            fields.append([a.tobytes() for a in e.field(0)])
    assert all(f == fields[0] for f in fields)
    capfd.readouterr()
    monkeypatch.setenv("PIV_XCORR_VARIANT", f"{len(VARIANTS[shape])},0")
    with pytest.raises(P.PivError) as err:
        P.Engine(p)
    assert err.value.status == P.PIV_ERR_ARG
    assert f"grid 1 has {len(VARIANTS[shape])} variants" in str(err.value) + capfd.readouterr().err

"""Synchronous readback through the pinned halves: components of several parts and a ragged last
one, left-out arrays, pinned destinations, and the raw selection, against the queued readback."""
import ctypes as C

import numpy as np
import pytest

import piv_b200 as P

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("Nx,Ny,sp", [(90, 70, 16), (1100, 701, 3)], ids=["one_part", "many_parts"])
def test_field_in_parts(cuda, Nx, Ny, sp):
    import torch

    f1, f2 = P.synth_pair(P.synth_params(Nx, Ny, ppp=0.04, field=P.PIV_FIELD_UNIFORM, a=1.3, b=-0.6, seed=3))
    p = P.default_params(Nx=Nx, Ny=Ny, if_mhe=0, ws_x1=16, ws_y1=16, spacing_x1=sp, spacing_y1=sp, Npass1=1, Npass2=0)
    with P.Engine(p) as e:
        e.set_images(f1, f2)
        e.run_pair()
        nt = e.geom["Nt_vec"][0]
        for sel in (0, 1):
            n = nt * (p.Npeak_save if sel == 0 else 1)
            want = e.field_wait(e.field_async(sel))
            got = e.field(sel)
            for a, b in zip(got, want):
                assert np.array_equal(np.ravel(a), np.ravel(b))
            # pinned destinations take the copies directly; a left-out array changes nothing else
            pin = torch.full((n,), -7.0, pin_memory=True)
            valid = np.full(n + 1, 9, np.uint8)
            rc = P.lib().piv_get_field(e.h, sel, None, None, None, C.cast(pin.data_ptr(), C.POINTER(C.c_float)),
                                       valid.ctypes.data_as(C.POINTER(C.c_uint8)))
            assert rc == 0
            assert np.array_equal(pin.numpy(), np.ravel(want[3]))
            assert np.array_equal(valid[:n], np.ravel(want[4])) and valid[n] == 9
            assert P.lib().piv_get_field(e.h, sel, None, None, None, None, None) == 0

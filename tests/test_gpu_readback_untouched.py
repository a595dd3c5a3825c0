"""What a readback does to the caller's arrays: when it reports a device error it leaves the results'
arrays alone, and pinned coordinates too (a copy of them may be in flight); fresh arrays cost one
page fault a page (not a read fault and a write fault)."""
import ctypes as C
import mmap
import resource

import numpy as np
import pytest

import piv_b200 as P

pytestmark = pytest.mark.gpu


def _fp(a):
    return a.ctypes.data_as(C.POINTER(C.c_float))


def _u8(a):
    return a.ctypes.data_as(C.POINTER(C.c_uint8))


def _wait(e, sel, *arrays):
    t = e.field_async(sel)[0]
    return lambda: P.lib().piv_field_wait(e.h, t, *arrays)


def _get(e, sel, *arrays):
    return lambda: P.lib().piv_get_field(e.h, sel, *arrays)


@pytest.mark.parametrize("read", [_get, _wait], ids=["get", "wait"])
@pytest.mark.parametrize("pinned", [False, True], ids=["pageable", "pinned"])
def test_an_error_leaves_the_results_alone(cuda, monkeypatch, read, pinned):
    import torch

    monkeypatch.setenv("PIV_TEST_FILL_CAP", "1")
    p = P.default_params(Nx=400, Ny=300, ws_x1=32, ws_y1=32, spacing_x1=16, spacing_y1=16, Npass1=1, Npass2=0)
    with P.Engine(p) as e:
        nx, ny, nt = e.geom["Nx_vec"][0], e.geom["Ny_vec"][0], e.geom["Nt_vec"][0]
        valid = np.ones((ny, nx, p.Npeak_save), np.uint8)
        valid[3:13, 4:14] = 0  # a hole that one iteration does not fill
        z = np.zeros((nt, p.Npeak_save), np.float32)
        e.set_candidates(0, z, z, valid.reshape(nt, -1))
        e.validate_grid1(2, 5, 2.0, 2.0, 0)
        keep = [torch.full((nt,), 7.0, pin_memory=pinned) for _ in range(4)]
        a = [t.numpy() for t in keep]
        ok = np.full(nt, 9, np.uint8)
        assert read(e, 1, *map(_fp, a), _u8(ok))() == P.PIV_ERR_DEVICE
        assert all((v == 7.0).all() for v in a[2:]) and (ok == 9).all()
        xs = 8 + 16 * np.arange(nx)
        assert (a[0] == 7.0).all() if pinned else np.array_equal(a[0].reshape(ny, nx)[0], xs)
        e.set_candidates(0, z, z, np.ones((nt, p.Npeak_save), np.uint8))
        e.validate_grid1(2, 5, 2.0, 2.0, 0)
        assert read(e, 1, *map(_fp, a), _u8(ok))() == 0
        assert np.array_equal(a[0].reshape(ny, nx)[0], xs) and (a[2] == 0).all() and (ok == 1).all()


@pytest.mark.parametrize("read", [_get, _wait], ids=["get", "wait"])
def test_fresh_pages_fault_once(cuda, read):
    p = P.default_params(Nx=1400, Ny=1100, ws_x1=16, ws_y1=16, spacing_x1=4, spacing_y1=4, Npass1=1, Npass2=0)
    with P.Engine(p) as e:
        nt = e.geom["Nt_vec"][0]
        n = nt * p.Npeak_save
        e.set_images(*P.synth_pair(P.synth_params(1400, 1100, seed=2)))
        e.run_pair()
        e.synchronize()
        faults = []
        for _ in range(3):
            maps = [mmap.mmap(-1, 4 * n, flags=mmap.MAP_PRIVATE | mmap.MAP_ANONYMOUS) for _ in range(3)]
            for m in maps:
                m.madvise(mmap.MADV_NOHUGEPAGE)
            a = [np.frombuffer(m, np.float32, n) for m in maps[:2]]
            ok = np.frombuffer(maps[2], np.uint8, n)
            call = read(e, 0, None, None, _fp(a[0]), _fp(a[1]), _u8(ok))
            before = resource.getrusage(resource.RUSAGE_SELF).ru_minflt
            assert call() == 0
            faults.append(resource.getrusage(resource.RUSAGE_SELF).ru_minflt - before)
        pages = 9 * n / mmap.PAGESIZE
        assert min(faults) <= 1.2 * pages, (faults, pages)

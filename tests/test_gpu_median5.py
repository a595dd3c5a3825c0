"""The 5x5 median kernel: grids smaller than the stencil, borders, holes (the sort of partial
neighbourhoods), counts that end inside a CTA, one to three passes with and without the hole
fill, against the C oracle; and neighbourhoods with infinities and NaN (candidates set by the
caller), against the compare-exchange network that the other stencils use, in NumPy."""
import numpy as np
import pytest

import piv_b200 as P
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _engine(nx, ny, nps):
    p = P.default_params(Nx=8 * nx + 8, Ny=8 * ny + 8, if_mhe=0, ws_x1=16, ws_y1=16, spacing_x1=8, spacing_y1=8, Npass1=1,
                         ws_x2=8, ws_y2=8, spacing_x2=8, spacing_y2=8, Npass2=1, Npeak_save=nps)
    e = P.Engine(p)
    f = np.full((p.Ny, p.Nx), 7, np.uint8)
    e.set_images(f, f)
    e.prep()
    return e, e.geom["Nx_vec"][1], e.geom["Ny_vec"][1]


def _candidates(rng, n, nps, holes):
    dx, dy = (np.round(rng.normal(0, 1, (n, nps)) * 64).astype(np.float32) / 64 for _ in range(2))  # ties too
    return dx, dy, (rng.random((n, nps)) >= holes).astype(np.uint8)


@pytest.mark.parametrize("grid", [(1, 1), (3, 2), (9, 4), (13, 11)], ids=lambda g: f"{g[0]}x{g[1]}")
@pytest.mark.parametrize("holes", [0.0, 0.3, 0.85])
def test_matches_oracle(cuda, grid, holes):
    rng = np.random.default_rng(7 * grid[0] + int(10 * holes))
    for nps in (1, 4):
        e, nx, ny = _engine(*grid, nps)
        with e:
            dx, dy, v = _candidates(rng, nx * ny, nps, holes)
            for npm, fill, minn in ((1, 0, 5), (1, 1, 1), (2, 1, 5), (3, 0, 3), (3, 1, 24)):
                e.set_candidates(1, dx, dy, v)
                e.validate_grid2(npm, minn, 2.0, 2.0, 0, fill)
                _, _, gx, gy, gv = e.field(3)
                wx, wy, wv, _ = O.validate(dx.ravel(), dy.ravel(), v.ravel(), nx, ny, nps, 5, 5, 3, 3, npm, minn, 2.0,
                                           0, fill)
                # the chosen candidates themselves, so exact; filled holes: FP32 means of at most
                # 8 values of at most 6, in another order
                assert np.array_equal(gv, wv), (nps, npm, fill, minn)
                tol = 1e-5 if fill else 0
                assert np.abs(gx - wx).max() <= tol and np.abs(gy - wy).max() <= tol, (nps, npm, fill, minn)


def _network(w, k0):
    """The bitonic merges of sizes k0..32 over 32 slots, fminf and fmaxf dropping NaN."""
    w = w.copy()
    k = k0
    while k <= 32:
        j = k // 2
        while j:
            for i in range(32):
                if i ^ j > i:
                    lo, hi = np.fmin(w[i], w[i ^ j]), np.fmax(w[i], w[i ^ j])
                    w[i], w[i ^ j] = (hi, lo) if i & k else (lo, hi)
            j //= 2
        k *= 2
    return w


def _median(w, n):
    return w[n // 2] if n % 2 else (w[n // 2] + w[n // 2 - 1]) / np.float32(2)


@pytest.mark.parametrize("holes", [0.0, 0.3])
def test_nonfinite_neighbours(cuda, holes):
    rng = np.random.default_rng(5)
    e, nx, ny = _engine(12, 9, 1)
    with e:
        dx, dy, v = _candidates(rng, nx * ny, 1, holes)
        bad = rng.permutation(nx * ny)[:9]
        dx[bad[:6], 0] = np.float32([np.nan, np.inf, -np.inf, np.nan, np.inf, np.nan])
        dy[bad[6:], 0] = np.float32([np.inf, np.nan, -np.inf])
        e.set_candidates(1, dx, dy, v)
        e.validate_grid2(1, 5, 2.0, 2.0, 0, 0)
        _, _, gx, gy, gv = e.field(3)
    with np.errstate(all="ignore"):
        for q in range(nx * ny):
            ok = v[q, 0] != 0
            for c in (dx[:, 0], dy[:, 0]):
                w = np.full(32, np.inf, np.float32)
                n = 0
                for t in range(25):
                    x, y = q % nx + t % 5 - 2, q // nx + t // 5 - 2
                    if t != 12 and 0 <= x < nx and 0 <= y < ny and v[y * nx + x, 0]:
                        w[t] = c[y * nx + x]
                        n += 1
                if n < 5:
                    ok = False
                    break
                w = _network(w, 2)
                med = _median(w, n)
                mad = _median(_network(np.where(np.arange(32) < n, np.abs(w - med), np.inf).astype(np.float32), 32), n)
                ok = ok and bool(np.abs(c[q] - med) / (mad + np.float32(0.1)) < 2)
            assert bool(gv[q]) == ok, q
            if ok:
                assert gx[q] == dx[q, 0] and gy[q] == dy[q, 0]

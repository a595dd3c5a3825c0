"""The 5x5 median kernel where most neighbourhoods hold infinities or NaN (candidates set by the
caller): medians that are no number, warps whose every lane needs the exchange network, and a
neighbour count that no vector reaches, against the network in NumPy."""
import numpy as np
import pytest

from test_gpu_median5 import _candidates, _engine, _median, _network

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("minn", [1, 24])
@pytest.mark.parametrize("values,share", [((np.inf,), 0.05), ((np.inf, -np.inf), 0.4), ((np.inf,), 0.8), ((np.nan,), 0.02),
                                          ((np.nan,), 0.5), ((np.nan, np.inf, -np.inf, 3e38), 0.6)],
                         ids=["inf5", "both40", "inf80", "nan2", "nan50", "mixed60"])
def test_dense_nonfinite(cuda, values, share, minn):
    rng = np.random.default_rng(int(100 * share) + len(values) + minn)
    e, nx, ny = _engine(13, 10, 2)
    n = nx * ny
    with e:
        d = _candidates(rng, n, 2, 0.05)
        v = d[2]
        for c in d[:2]:
            bad = rng.random((n, 2)) < share
            c[bad] = rng.choice(np.float32(values), int(bad.sum()))
        e.set_candidates(1, *d)
        e.validate_grid2(1, minn, 2.0, 2.0, 0, 0)
        _, _, gx, gy, gv = e.field(3)
    with np.errstate(all="ignore"):
        for q in range(n):
            ok = v[q] != 0
            for c in d[:2]:
                w = np.full(32, np.inf, np.float32)
                k = 0
                for t in range(25):
                    x, y = q % nx + t % 5 - 2, q // nx + t // 5 - 2
                    if t != 12 and 0 <= x < nx and 0 <= y < ny and v[y * nx + x, 0]:
                        w[t] = c[y * nx + x, 0]
                        k += 1
                if k < minn:
                    ok = np.zeros(2, bool)
                    break
                w = _network(w, 2)
                med = _median(w, k)
                mad = _median(_network(np.where(np.arange(32) < k, np.abs(w - med), np.inf).astype(np.float32), 32), k)
                ok = ok & (np.abs(c[q] - med) / (mad + np.float32(0.1)) < 2)
            assert bool(gv[q]) == bool(ok.any()), q
            if ok.any():
                i = int(ok.argmax())
                assert gx[q] == d[0][q, i] and gy[q] == d[1][q, i]

"""The predictor's gradients where the tiled kernels' ranges end: rows longer than a segment of 32
pixels (split across segments) and than a run of 8, single rows, columns and vectors, several rows
per segment, and batches that leave a last CTA and a last split partly empty.  The oracle is the
float64 restatement of the network; the SIMT forward keeps the pre-activations' signs its own."""
import numpy as np
import pytest

import piv_b200 as P
from oracle import learned as L

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(1, 1, 1), (2, 1, 41), (1, 37, 3), (5, 4, 33), (3, 17, 16), (9, 8, 8)],
                         ids=lambda s: "x".join(map(str, s)))
def test_gradients_match_oracle(cuda, monkeypatch, shape):
    import torch

    monkeypatch.setenv("PIV_NET_TC", "0")
    N, H, W = shape
    rng = np.random.default_rng(100 + W)
    x = rng.normal(0, 0.5, (N, 81, H, W)).astype(np.float32)
    label = rng.normal(0, 1, (N, 2, H, W)).astype(np.float32)
    mask = (rng.random((N, H, W)) > 0.15).astype(np.float32)
    mask.flat[0] = 1
    with P.PredictorNet(seed=5) as net:
        params = net.params()
        for (_, b_off, cout, _) in L.layout()[0]:
            params[b_off:b_off + cout] = rng.normal(0, 0.05, cout)
        net.set_params(params)
        d = [torch.from_numpy(v).cuda() for v in (x, label, mask)]
        got = []
        for _ in range(2):  # a second call finds the workspaces of the first
            loss = net.loss_grad(*d, N, H, W)
            got.append(net.grads())
    want_loss, want, _ = L.loss_and_grad(params.astype(np.float64), x.astype(np.float64), label.astype(np.float64),
                                         mask.astype(np.float64))
    assert np.array_equal(got[0], got[1])
    assert abs(loss - want_loss) <= 1e-5 * (1 + abs(want_loss))
    # FP32 sums over at most N*H*W*9 products: the bar of the other gradient tests
    for i, (w_off, b_off, cout, _) in enumerate(L.layout()[0]):
        for lo, hi in ((w_off, b_off), (b_off, b_off + cout)):
            err = np.linalg.norm(got[0][lo:hi] - want[lo:hi]) / max(np.linalg.norm(want[lo:hi]), 1e-12)
            assert err < 2e-4, (i, lo == b_off, err)

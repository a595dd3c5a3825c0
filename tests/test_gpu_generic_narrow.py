"""The general-size kernel's windows narrower than a warp, whose rows share its lanes: row counts
that the lanes divide and that they do not, against NumPy and between the peak searches."""
import pytest

from test_gpu_generic_stages import test_stages_and_peak_lists as _planes_and_peaks

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ws", [(4, 36), (8, 36), (12, 44), (20, 20), (24, 40), (28, 60), (12, 512), (4, 1024)],
                         ids=lambda w: f"{w[0]}x{w[1]}")
def test_narrow(cuda, ws):
    _planes_and_peaks(cuda, ws)

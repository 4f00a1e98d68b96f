"""Edge weights where their rows start to be staged (24 samples), up to the most
samples, and on the last, partly filled warp: equal to the restated graph."""
import pytest

from test_gpu_parity import _graph_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("S", [23, 24, 25, 32, 33, 44, 45, 63, 64])
def test_staged_rows(gpu_ctx, orc, S):
    g = _graph_case(gpu_ctx, orc, 6, 401, S, seed=300 + S)
    assert len(g["src"]) > 0

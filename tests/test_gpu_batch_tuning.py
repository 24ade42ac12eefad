"""cfd_batch_autotune also times the tiling it starts from. One long, narrow
grid has too few lines for the chip along x, so that a sweep's time falls with
the segments a line is cut into; a batch that starts with many must not be left
with fewer, which would be times as slow."""
import numpy as np
import pytest

from cfd_inwsl_b200 import zone
from tests.util import make_info, quadrant_state

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("segments", [None, 16, 48])
def test_autotune_keeps_many_segments(segments):
    from tests.conftest import gpu_available
    if not gpu_available():
        pytest.skip("no CUDA device")
    n = (16384, 8)
    b = zone.BlockBatch([make_info(2, list(n), [0, 1, 0, 1, 0, 0])])
    b.set_cons(0, quadrant_state(n, np.random.default_rng(1)))
    if segments:
        b.set_tiling(1, 1, segments)
    choice = b.autotune()
    assert choice[0]["segments_per_line"] >= (segments or 16)
    b.close()

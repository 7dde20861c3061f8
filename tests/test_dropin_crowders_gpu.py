"""The repulsive crowder form in the energy kernel's two- and four-block CTA shapes, and its
non-crowder sum beside it, against the FP64 oracle (bounds: test_dropin_blocks_gpu.py)."""
import numpy as np
import pytest

from test_dropin_blocks_gpu import check, cut
from test_dropin_gpu import L, synthetic_packed  # noqa: F401  (L: fixture)

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [33 * 128 + 1, 39 * 128 + 5])  # 34 and 40 tiles
def test_repulsive_crowders(L, refdata, n):  # noqa: F811
    rng = np.random.default_rng(n)
    pos, meta = cut(*synthetic_packed(rng, 24, [60, 150, 97], 260.0, 0.1, crowders=40), n)
    assert (meta[:, 3] == -1.0).sum() > 1000
    check(L, refdata, pos, meta, 260.0, rc=True)

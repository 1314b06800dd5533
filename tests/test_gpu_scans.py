"""The operand scans of the modular scheme at the edges of their chunks.

Grids and results against the exact-integer model (bit for bit) where K does
not fill a scan's batch (8 or 16 values), slice (32 rows), chunk (256 rows) or
the chunks merged inside the column split (K <= 1024), on rows and columns
whose exponents rise or fall all along, are zero, or lie around the exponent
below which the scan goes element by element (2^-862).
"""
import numpy as np
import pytest

import ozaki2_model
from test_gpu_ozaki2 import check_grid, run_dev_grid

pytestmark = pytest.mark.gpu


def _vectors(rng, count, k):
    """count vectors of length k: the special ones first, then wide exponents."""
    x = rng.uniform(1, 2, (count, k)) * rng.choice([-1.0, 1.0], (count, k))
    x *= np.exp2(rng.integers(-20, 21, (count, k)))
    steps = np.minimum(np.arange(k), 900)
    x[0] = 0.0
    x[1] = np.ldexp(1.5, -400 + steps)             # every element raises the exponent
    x[2] = np.ldexp(-1.25, 300 - steps)            # none after the first does
    x[3] = np.ldexp(x[3], -860)                    # around the element-by-element limit
    x[4] = np.ldexp(x[4], -1040)                   # subnormal values among them
    x[5, : k // 2] = 0.0                           # a zero half, then values
    return x


@pytest.mark.parametrize("k", [1, 7, 31, 33, 255, 257, 1024, 1025, 2304])
def test_grids_at_scan_edges(phpc, torch_cuda, k):
    rng = np.random.default_rng(k)
    a = _vectors(rng, 9, k)
    b = np.ascontiguousarray(_vectors(rng, 33, k).T)
    got, grid = run_dev_grid(phpc, torch_cuda, a, b, np.zeros((9, 33)), 13)
    check_grid(a, b, grid, 13)
    want = ozaki2_model.gemm(a, b, None, 13, grid)
    normal = (np.abs(want) >= np.finfo(float).tiny) | (want == 0)  # subnormal results round twice
    np.testing.assert_array_equal(got[normal], want[normal])

"""calcNCCAlt and calcSQDAlt through tap quads and pairs (scan_sum_kernel), against the oracle.

Rows of fewer samples than a warp, of one more than one or two warps' worth, moving images larger and
smaller than the fixed one, one and three channels; and an image so wide that a row's lambda has more
runs than the kernel keeps (lanes step explicitly).  Tolerance as in test_gpu_parity.py.
"""
import numpy as np
import pytest

import oracle as O
from conftest import close_costs
from cugridsearch_b200 import synthetic as S

pytestmark = pytest.mark.gpu


def _run(cuda, cost, moving, fixed, lo, hi, cnt):
    import torch
    import cugridsearch_b200 as cgs
    grid = cgs.CudaGrid.from_ranges(lo, hi, cnt)
    costs = torch.full((grid.numElements(),), 7.0e30, dtype=torch.float32, device=cuda)
    to = lambda a: cgs.CudaImage(torch.from_numpy(np.ascontiguousarray(a)).to(cuda))
    cgs.search(cost, to(moving), to(fixed), grid, costs=costs)
    torch.cuda.synchronize()
    c = costs.cpu().numpy()
    c32, c64 = O.search(cost, O.make_grid(lo, hi, cnt), O.Image(moving), O.Image(fixed))
    bad = close_costs(c, c32, c64, cost)
    assert not bad.any(), (int(bad.sum()), c[bad][:4], c64[bad][:4])
    return c


@pytest.mark.parametrize("cost", ["NCC_ALT", "SQD_ALT"])
@pytest.mark.parametrize("size,msize,channels", [(5, 5, 1), (20, 33, 3), (33, 31, 1), (65, 64, 3), (97, 130, 3)])
def test_ragged_rows(cuda, lib, cost, size, msize, channels):
    pair = S.small_pair(700 + size, size=size, count=3, cost=cost, msize=msize, channels=channels)
    _run(cuda, cost, pair.moving, pair.fixed, *pair.grid_args())


@pytest.mark.parametrize("cost", ["NCC_ALT", "SQD_ALT"])
def test_wide_rows_step_explicitly(cuda, lib, cost):
    rng = np.random.default_rng(7)
    w = 70000  # lambda 0.25 .. 70000 passes 19 binades
    fixed = rng.uniform(0, 255, (2, w)).astype(np.float32)
    moving = np.roll(fixed, 3, axis=1)
    lo, hi = [0, 1, 1, 0, -0.25, 0, 0, 0], [0, 1, 1, 0, 0.25, 0, 0, 0]
    c = _run(cuda, cost, moving, fixed, lo, hi, [1, 1, 1, 1, 3, 1, 1, 1])
    assert (c != 123123.0).any()


@pytest.mark.parametrize("channels", [1, 3])
@pytest.mark.parametrize("cost", ["NCC_ALT", "SQD_ALT"])
def test_no_data_pixels(cuda, lib, cost, channels):
    """A block of the type's lowest value in the fixed image: finite samples, whose squares overflow as the
    reference's do (calcNCCAlt 0, not NaN)."""
    pair = S.small_pair(41, size=33, count=3, cost=cost, channels=channels)
    pair.fixed = pair.fixed.copy()
    pair.fixed[5:9, 10:20] = np.finfo(np.float32).min
    with np.errstate(all="ignore"):
        c = _run(cuda, cost, pair.moving, pair.fixed, *pair.grid_args())
    assert np.isnan(c).any() == (cost == "SQD_ALT")

"""Fixed pixels that are not finite, or so large that they swamp their row's sums in FP64, must not reach
the cost of a grid point whose overlap misses them; a row of zeros beside other pixels sums to exactly 0.

Nor may they, in either image, move the shift of the zero-mean sums away from the pixels.  The fixed
rows' sums over an overlap come from prefix sums (span kernels), which such pixels poison for
the rest of their row.  Checked against the oracle, one and three channels, single and batch, whole and
split tasks; tolerances as in conftest.close_costs.
"""
import numpy as np
import pytest

import oracle as O
from conftest import close_costs
from cugridsearch_b200 import synthetic as S
from test_span_gpu import _env, _run

pytestmark = pytest.mark.gpu
COSTS = ["SQD_REF", "NCC_REF"]
LOWEST = float(np.finfo(np.float32).min)


def _pair(cost, h, w, channels, seed=31):
    """A grid whose overlaps lie at the right, the left or across a fixed image."""
    p = S.small_pair(seed, size=max(h, w), count=3, cost=cost, channels=channels)
    p.fixed = np.ascontiguousarray(p.fixed[:h, :w])
    p.moving = np.ascontiguousarray(p.moving[:h, :w])
    p.lo[4], p.hi[4] = -0.45 * w, 0.45 * w
    p.lo[5], p.hi[5] = -0.1 * h, 0.1 * h
    return p


def _outliers(p, value):
    """`value` at the left of the fixed image in every third row, and at one pixel a quarter across."""
    f = p.fixed.copy()
    h, w = f.shape[:2]
    f[2:h:3, :2] = value
    f[h // 2, w // 4] = value
    return f


def _oracle(p, cost, fixed):
    return O.search(cost, O.make_grid(*p.grid_args()), O.Image(p.moving), O.Image(fixed))


def _runs(cuda, p, cost):
    """A search, one on the span kernel whatever the width (self-checking), and a batch."""
    out = [_run(cuda, p, cost)[1]]
    if p.fixed.shape[2] == 1:
        with _env(CGS_SPAN_CHECK=1):
            out.append(_run(cuda, p, cost)[1])
        out.append(_batch(cuda, p, cost))
    return out


def _batch(cuda, p, cost):
    import torch
    import cugridsearch_b200 as cgs
    mov, fix = (cgs.CudaImage(torch.from_numpy(x).to(cuda)) for x in (p.moving, p.fixed))
    grid = cgs.CudaGrid.from_ranges(*p.grid_args())
    costs, out = torch.empty(grid.numElements(), device=cuda), cgs.result_buffer(cuda)
    with cgs.Batch([cgs.BatchPair(cost, mov, fix, grid, out, costs)]) as b:
        b.launch()
        torch.cuda.synchronize()
    return costs.cpu().numpy()


def _clear(p, fixed, moving):
    """The points whose overlap misses the NaN pixels of the images (calcNCC and zero-mean NCC have the
    same map; the oracle's zero-mean NCC takes whole images' means, so NaN spreads to all its points)."""
    q = S.Pair(fixed, moving, p.gt, p.lo, p.hi, p.count)
    clear = np.isfinite(_oracle(q, "NCC_REF", np.ascontiguousarray(fixed))[1])
    assert 0.2 < clear.mean() < 0.8
    return clear


def _check(cuda, cost, h, w, channels, value):
    p = _pair(cost, h, w, channels)
    clear = _clear(p, _outliers(p, np.float32("nan")), p.moving)
    c32, c64 = _oracle(p, cost, p.fixed)  # at clear points the outliers' values are not read
    p.fixed = np.ascontiguousarray(_outliers(p, value))
    for c in _runs(cuda, p, cost):
        bad = close_costs(c, c32, c64, cost) & clear
        assert not bad.any(), (int(bad.sum()), c[bad][:4], c64[bad][:4])
        if not np.isfinite(value):
            assert not np.isfinite(c[~clear]).any()


@pytest.mark.parametrize("value", [float("nan"), float("inf"), float("-inf"), 1e10, LOWEST])
@pytest.mark.parametrize("h,w,channels", [(30, 41, 1), (20, 300, 1), (30, 70, 3)])
@pytest.mark.parametrize("cost", COSTS + ["ZNCC"])
def test_outliers_outside_the_overlap(cuda, lib, cost, h, w, channels, value):
    _check(cuda, cost, h, w, channels, value)


@pytest.mark.parametrize("channels", [1, 3])
@pytest.mark.parametrize("cost", COSTS)
def test_overlap_of_zeros(cuda, lib, cost, channels):
    """Overlaps of zeros that begin in the 32 columns of other pixels: SQD +inf and NCC NaN there, as the
    oracle's."""
    p = _pair(cost, 40, 41, channels)
    p.fixed = np.ascontiguousarray(p.fixed + np.float32(0.1))
    p.fixed[:, 12:] = 0.0
    c32, c64 = _oracle(p, cost, p.fixed)
    assert 0.2 < (~np.isfinite(c64)).mean() < 0.8
    for c in _runs(cuda, p, cost):
        bad = close_costs(c, c32, c64, cost)
        assert not bad.any(), (int(bad.sum()), c[bad][:4], c32[bad][:4], c64[bad][:4])


@pytest.mark.parametrize("value", [float("nan"), 1e10, LOWEST])
@pytest.mark.parametrize("channels", [1, 3])
def test_moving_outliers_outside_the_overlap(cuda, lib, channels, value):
    """Moving pixels that no sample of a point reads: its zero-mean cost is the oracle's."""
    p = _pair("ZNCC", 30, 41, channels)
    moving = p.moving.copy()
    moving[::3, 30:32] = np.nan
    clear = _clear(p, p.fixed, np.ascontiguousarray(moving))
    c32, c64 = _oracle(p, "ZNCC", p.fixed)
    moving[::3, 30:32] = value
    p.moving = np.ascontiguousarray(moving)
    c = _run(cuda, p, "ZNCC")[1]
    bad = close_costs(c, c32, c64, "ZNCC") & clear
    assert not bad.any(), (int(bad.sum()), c[bad][:4], c64[bad][:4])


@pytest.mark.parametrize("channels", [1, 3])
def test_sad_beyond_fp32(cuda, lib, channels):
    """No-data pixels of the type's lowest value inside the overlap: the reference's FP32 sum overflows, and the
    cost is +inf on every kernel."""
    p = S.small_pair(47, size=70, count=2, cost="SAD_AVG", channels=channels)
    p.fixed = p.fixed.copy()
    p.fixed[12, 30] = p.fixed[50, 40] = LOWEST  # a band each: its FP32 sums hold it
    c32, c64 = _oracle(p, "SAD_AVG", np.ascontiguousarray(p.fixed))
    assert np.isinf(c32).any()
    for c in _runs(cuda, p, "SAD_AVG") + [_run(cuda, p, "SAD_AVG", per_sample_decisions=True)[1]]:
        bad = close_costs(c, c32, c64, "SAD_AVG")
        assert not bad.any(), (int(bad.sum()), c[bad][:4], c32[bad][:4], c64[bad][:4])

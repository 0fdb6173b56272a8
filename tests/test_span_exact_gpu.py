"""The span kernel of the exact-sampling costs (cgs_span_exact.cuh: SAD_AVG, SQD_REF and NCC_REF with
one or three channels) at the edges of its tiles, blocks and bands, against the FP64 oracle:

* fixed images one pixel around a 32-column block, a 256-column (three channels: 64-column) tile and a
  16-row band, moving images of another size;
* the self-checking build (CGS_SPAN_CHECK=1, one channel) finds every sample's quad in its window, and
  windows that do not fit the stage (CGS_SPAN_CAP) give the same bits from global memory;
* grids whose perspective lets w change sign (points without spans);
* a 1 x 1 fixed image, whose SAD is one sample: bit for bit the oracle's, so that coordinates, quotients
  and interpolation round as the reference's.
"""
import numpy as np
import pytest

import oracle as O
from conftest import close_costs
from cugridsearch_b200 import synthetic as S
from test_span_gpu import _env, _run

pytestmark = pytest.mark.gpu
COSTS = ["SAD_AVG", "SQD_REF", "NCC_REF"]


def _pair(seed, cost, h, w, mh, mw, channels, count=2, u8=False):
    size = max(h, w, mh, mw, 16)
    p = S.small_pair(seed, size=size, count=count, cost=cost, channels=channels, u8=u8)
    p.fixed = np.ascontiguousarray(p.fixed[:h, :w])
    p.moving = np.ascontiguousarray(p.moving[:mh, :mw])
    span = 0.1 * min(h, w, mh, mw)
    p.lo[4:6], p.hi[4:6] = -span, span
    return p


def _oracle_agrees(pair, cost, c):
    g = O.make_grid(*pair.grid_args())
    c32, c64 = O.search(cost, g, O.Image(pair.moving), O.Image(pair.fixed))
    bad = close_costs(c, c32, c64, cost)
    assert not bad.any(), (int(bad.sum()), c[bad][:4], c32[bad][:4], c64[bad][:4])


@pytest.mark.parametrize("cost", COSTS)
@pytest.mark.parametrize("h,w,mh,mw,channels", [(15, 31, 20, 33, 1), (16, 32, 16, 32, 1), (17, 33, 14, 40, 1),
                                                (33, 257, 37, 250, 1), (1, 256, 3, 256, 1), (48, 5, 48, 5, 1),
                                                (17, 65, 19, 61, 3), (16, 64, 16, 64, 3), (31, 129, 33, 140, 3)])
def test_edges_match_oracle(cuda, lib, cost, h, w, mh, mw, channels):
    pair = _pair(500 + h + w, cost, h, w, mh, mw, channels, u8=channels == 3)
    with _env(**({"CGS_SPAN_CHECK": 1} if channels == 1 else {})):
        _, c = _run(cuda, pair, cost)
    _oracle_agrees(pair, cost, c)


@pytest.mark.parametrize("cost", COSTS)
def test_plain_checked_and_global_taps_agree(cuda, lib, cost):
    pair = _pair(7, cost, 70, 130, 75, 120, 1, count=3)
    _, c0 = _run(cuda, pair, cost)
    with _env(CGS_SPAN_CHECK=1):
        _, c1 = _run(cuda, pair, cost)
    with _env(CGS_SPAN_CAP=1024):
        _, c2 = _run(cuda, pair, cost)
    np.testing.assert_array_equal(c1.view(np.uint32), c0.view(np.uint32))
    np.testing.assert_array_equal(c2.view(np.uint32), c0.view(np.uint32))
    pair.fixed, pair.moving = np.repeat(pair.fixed, 3, 2), np.repeat(pair.moving, 3, 2)
    _, c3 = _run(cuda, pair, cost)
    with _env(CGS_SPAN_CAP=1024):
        _, c4 = _run(cuda, pair, cost)
    np.testing.assert_array_equal(c4.view(np.uint32), c3.view(np.uint32))
    _oracle_agrees(pair, cost, c3)


@pytest.mark.parametrize("channels", [1, 3])
@pytest.mark.parametrize("cost", COSTS)
def test_points_without_spans(cuda, lib, cost, channels):
    pair = _pair(11, cost, 24, 40, 24, 40, channels, count=3)
    pair.lo[6:8], pair.hi[6:8] = -0.06, 0.06  # w changes sign inside the image at the outer values
    _, c = _run(cuda, pair, cost)
    _oracle_agrees(pair, cost, c)


def test_one_sample_is_the_references_bit_for_bit(cuda, lib):
    pair = _pair(13, "SAD_AVG", 1, 1, 64, 64, 1, count=4)
    pair.fixed[:] = 0.0
    pair.lo[4:6], pair.hi[4:6] = -60.3, 3.7
    pair.moving = np.random.default_rng(3).uniform(0, 255, pair.moving.shape).astype(np.float32)
    _, c = _run(cuda, pair, "SAD_AVG")
    g = O.make_grid(*pair.grid_args())
    c32, _ = O.search("SAD_AVG", g, O.Image(pair.moving), O.Image(pair.fixed))
    assert np.isfinite(c32).sum() > 1000
    np.testing.assert_array_equal(c[np.isfinite(c32)].view(np.uint32), c32[np.isfinite(c32)].view(np.uint32))
    np.testing.assert_array_equal(np.isfinite(c), np.isfinite(c32))


@pytest.mark.parametrize("h,w,mh,mw", [(17, 65, 19, 61), (16, 64, 16, 64), (31, 129, 33, 140)])
@pytest.mark.parametrize("bins", [8, 32])
def test_three_channel_mi_is_the_per_sample_kernels(cuda, lib, h, w, mh, mw, bins):
    """Equal counts and the same cost function: the same bits, at the edges of blocks and bands."""
    pair = _pair(700 + w, "MI", h, w, mh, mw, 3, u8=True)
    _, c = _run(cuda, pair, "MI", mi_bins=bins)
    _, c0 = _run(cuda, pair, "MI", mi_bins=bins, per_sample_decisions=True)
    np.testing.assert_array_equal(c.view(np.uint32), c0.view(np.uint32))


@pytest.mark.parametrize("h,w", [(15, 31), (17, 33), (33, 257), (2, 64)])
def test_one_channel_mi_is_the_per_sample_kernels(cuda, lib, h, w):
    """The guarded fast samples at the same edges, with values beyond both ends of the bins."""
    pair = _pair(800 + w, "MI", h, w, h + 3, w - 2, 1)
    pair.moving = pair.moving * 1.5 - 40.0
    with _env(CGS_SPAN_CHECK=1):
        _, c = _run(cuda, pair, "MI")
    _, c0 = _run(cuda, pair, "MI", per_sample_decisions=True)
    np.testing.assert_array_equal(c.view(np.uint32), c0.view(np.uint32))


@pytest.mark.parametrize("cost", COSTS + ["ZNCC"])
def test_split_tasks_equal_whole_ones(cuda, lib, cost):
    """256 points of a 200 x 180 image are four tasks, split over their 13 bands in a single search and
    whole in a batch: the same bits."""
    import torch
    import cugridsearch_b200 as cgs
    pair = _pair(21, cost, 200, 180, 190, 200, 1)
    res, c = _run(cuda, pair, cost)
    mov, fix = (cgs.CudaImage(torch.from_numpy(x).to(cuda)) for x in (pair.moving, pair.fixed))
    grid = cgs.CudaGrid.from_ranges(*pair.grid_args())
    costs, out = torch.empty(grid.numElements(), device=cuda), cgs.result_buffer(cuda)
    with cgs.Batch([cgs.BatchPair(cost, mov, fix, grid, out, costs)]) as b:
        b.launch()
        torch.cuda.synchronize()
    np.testing.assert_array_equal(costs.cpu().numpy().view(np.uint32), c.view(np.uint32))
    assert cgs.read_result(out).index == res.index
    _oracle_agrees(pair, cost, c)


@pytest.mark.parametrize("cost,channels,tuning", [("SAD_AVG", 1, {"warps_per_block": 5}),
                                                  ("SQD_REF", 3, {"warps_per_block": 32}),
                                                  ("NCC_REF", 1, {"warps_per_block": 1}),
                                                  ("MI", 3, {"points_per_warp": 4})])  # 278 KB of histograms
def test_tunings_of_no_per_sample_kernel_are_refused(cuda, lib, cost, channels, tuning):
    """As on the per-sample kernel, although the span kernel has its own plan."""
    import cugridsearch_b200 as cgs
    pair = _pair(3, cost, 20, 20, 20, 20, channels)
    for per_sample in (False, True):
        with pytest.raises(cgs.CgsError):
            _run(cuda, pair, cost, per_sample_decisions=per_sample, **tuning)
    for tuning in ({"warps_per_block": 8}, {"points_per_warp": 1}):
        _run(cuda, pair, cost, **tuning)


@pytest.mark.parametrize("channels", [1, 3])
@pytest.mark.parametrize("cost", COSTS + ["MI"])
@pytest.mark.parametrize("h,w", [(1, 300), (9, 70), (70, 9), (33, 33)])
def test_rows_along_the_moving_images_edges(cuda, lib, cost, channels, h, w):
    """No rotation, unit scale and whole pixels: the edge rows are band pixels from end to end (1 to 300,
    around the 8 that a lane takes by itself and the 32 of a warp), with and without a slight tilt."""
    pair = _pair(900 + w, cost, h, w, h + 2, w + 1, channels, u8=channels == 3)
    pair.lo[:] = [0, 1, 1, 0, -8, -2, 0, -2e-6]
    pair.hi[:] = [2e-6, 1, 1, 0, 8, 2, 0, 0]
    pair.count[:] = [2, 1, 1, 1, 5, 5, 1, 2]
    with _env(**({"CGS_SPAN_CHECK": 1} if channels == 1 and cost != "MI" else {})):  # narrow ones too
        _, c = _run(cuda, pair, cost)
    if cost == "MI":
        _, c0 = _run(cuda, pair, cost, per_sample_decisions=True)
        np.testing.assert_array_equal(c.view(np.uint32), c0.view(np.uint32))
    _oracle_agrees(pair, cost, c)


@pytest.mark.parametrize("channels", [1, 3])
@pytest.mark.parametrize("cost", COSTS + ["MI"])
@pytest.mark.parametrize("h,w", [(40, 8), (20, 16), (20, 24), (20, 28), (20, 33), (20, 44), (20, 48), (1, 300)])
def test_narrow_images(cuda, lib, cost, channels, h, w):
    """Widths around the lines of span_pays, which run on the per-sample kernel or the span kernel."""
    pair = _pair(950 + w, cost, h, w, h, w, channels, u8=channels == 3)
    _, c = _run(cuda, pair, cost)
    _oracle_agrees(pair, cost, c)
    if channels == 1 and cost != "MI":
        with _env(CGS_SPAN_CHECK=1):  # the span kernel
            _, c1 = _run(cuda, pair, cost)
        _oracle_agrees(pair, cost, c1)
        _, c2 = _run(cuda, pair, cost, per_sample_decisions=True)
        if w < 28 or 33 <= w < 44:
            np.testing.assert_array_equal(c.view(np.uint32), c2.view(np.uint32))
        elif w in (28, 48):
            np.testing.assert_array_equal(c.view(np.uint32), c1.view(np.uint32))


@pytest.mark.parametrize("cost", COSTS + ["MI"])
@pytest.mark.parametrize("h,w,mh,mw", [(17, 65, 19, 61), (16, 64, 16, 64), (31, 129, 33, 140), (20, 24, 24, 20)])
def test_three_channel_windows_are_in_bounds(cuda, lib, cost, h, w, mh, mw):
    """The self-checking build finds every sample of three planes in its block's window, with the plain
    build's bits, from windows and (a small stage) from global memory."""
    pair = _pair(640 + w, cost, h, w, mh, mw, 3, u8=True)
    with _env(CGS_SPAN_CHECK=1):
        _, c = _run(cuda, pair, cost)
        with _env(CGS_SPAN_CAP=1024):
            _, c1 = _run(cuda, pair, cost)
    np.testing.assert_array_equal(c1.view(np.uint32), c.view(np.uint32))
    _oracle_agrees(pair, cost, c)
    if w > 32:  # wide enough for the span kernel
        _, c0 = _run(cuda, pair, cost)
        np.testing.assert_array_equal(c0.view(np.uint32), c.view(np.uint32))


@pytest.mark.parametrize("cost", COSTS)
def test_three_channel_split_tasks(cuda, lib, cost):
    """64 points of a tall image, one task split over its bands, and the same points among 148 tasks, which
    fill the GPU whole: the same bits per point."""
    pair = _pair(23, cost, 104, 66, 100, 68, 3)
    pair.count[:] = [2, 1, 1, 1, 4, 4, 2, 1]
    _, few = _run(cuda, pair, cost)
    n = [2, 37, 2, 2, 4, 4, 2, 2]
    pair.count[:] = n
    for a, step in ((1, 0.001), (2, 0.01), (3, 0.01), (7, 1e-6)):  # the few's value is the first of the many's
        pair.hi[a] = pair.lo[a] + step * (n[a] - 1)
    _, many = _run(cuda, pair, cost)
    pick = many.reshape(n[::-1])[0, :, :, :, 0, 0, 0, :].reshape(-1)
    np.testing.assert_array_equal(pick.view(np.uint32), few.view(np.uint32))
    _oracle_agrees(pair, cost, many)


@pytest.mark.parametrize("channels", [1, 3])
@pytest.mark.parametrize("cost", ["SAD_AVG", "NCC_REF", "MI"])
def test_one_wide_row(cuda, lib, cost, channels):
    """A row too wide for the per-sample kernel's shared memory, which one row of few points otherwise takes."""
    rng = np.random.default_rng(9)
    pair = _pair(3, cost, 1, 16, 3, 16, channels)
    pair.fixed = rng.uniform(0, 255, (1, 30000, channels)).astype(np.float32)
    pair.moving = np.ascontiguousarray(np.repeat(np.roll(pair.fixed, 2, axis=1), 3, axis=0))
    pair.lo[:] = [0, 1, 1, 0, -3, -0.25, 0, 0]
    pair.hi[:] = [0, 1, 1, 0, 3, 1.25, 0, 0]
    pair.count[:] = [1, 1, 1, 1, 4, 3, 1, 1]
    _, c = _run(cuda, pair, cost)
    _oracle_agrees(pair, cost, c)

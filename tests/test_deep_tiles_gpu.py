"""Small maps on the deep tiles (8 coarse cells of the innermost axis) that large series
run on, against the FP64 oracle: whole and ragged innermost ends, either axis innermost,
odd axis counts, central differences and unequal gradient ranges. Launches of few (tile,
volume) items get shallow tiles, so these have volumes enough;
tests/test_tile_depth_cpu.py checks that they do."""
import numpy as np
import pytest

from tests.parity import assert_parity, tol_for

pytestmark = pytest.mark.gpu

SMOOTH = dict(gradient_smooth=1, main_range=1, x_range=1, y_range=1, z_range=1)
RANGES = dict(gradient_smooth=1, main_range=2, x_range=2, y_range=1, z_range=0)
CENTRAL = dict(gradient_smooth=0)

CASES = [
    # (mag x, y, z), (T, D, H, W), axes, method, gradient
    ((2, 2, 2), (160, 8, 8, 8), 6, 1, SMOOTH),    # y innermost, one whole tile of 16
    ((2, 2, 2), (80, 7, 7, 17), 6, 3, SMOOTH),    # 14 of 16 subvoxels
    ((2, 2, 2), (80, 7, 7, 17), 6, 1, RANGES),
    ((4, 4, 2), (80, 7, 8, 8), 6, 3, SMOOTH),     # y innermost, 32 deep
    ((4, 4, 2), (60, 9, 15, 5), 6, 1, CENTRAL),   # 60 in two tiles
    ((2, 2, 4), (80, 8, 7, 9), 6, 1, SMOOTH),     # z innermost
    ((2, 2, 4), (60, 15, 6, 9), 6, 1, RANGES),
    ((1, 2, 5), (80, 7, 8, 19), 6, 1, SMOOTH),    # 21 cells of x per tile, 35 of 40 subvoxels
    ((3, 3, 3), (100, 7, 7, 6), 5, 1, SMOOTH),    # odd axis count: nothing at a quarter turn
    ((1, 1, 1), (100, 15, 15, 17), 6, 1, SMOOTH),
    ((2, 2, 1), (100, 9, 8, 9), 4, 1, CENTRAL),
    ((5, 5, 5), (60, 8, 8, 6), 3, 1, SMOOTH),     # the deepest magnification
]


@pytest.mark.parametrize("mag,shape,axes,method,grad", CASES)
@pytest.mark.parametrize("dtype", [np.uint16, np.float32])
def test_deep_tiles_match_oracle(ctx, oracle_mod, mag, shape, axes, method, grad, dtype):
    from rfba_gb300 import synth
    from rfba_gb300.srrf import Config
    kw = dict(mag=mag, method=method, axes_in_ring=axes, itc=0, **grad)
    T, D, H, W = shape
    x = synth.render(synth.make_scene(60 + axes, T, (W, H, D), 8), (W, H, D), 60 + axes, dtype)
    got = ctx.forward(Config.make(**kw), np.ascontiguousarray(x))
    ref = oracle_mod.srrf_region(x.astype(np.float32), oracle_mod.make_conf(**kw))
    assert_parity(got, ref, tol_for(method), f"{mag} {shape} axes {axes}")

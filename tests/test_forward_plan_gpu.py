"""The forward kernel's plan choices against the FP64 oracle: both tile axis orders,
both tile depths with exact and ragged ends along every axis, rings without a
sample on the tile's innermost axis (odd axis counts), and rings whose tables do
not fit the kernel parameters."""
import numpy as np
import pytest

from tests.parity import assert_parity, tol_for

pytestmark = pytest.mark.gpu

SMOOTH = dict(gradient_smooth=1, x_range=1, y_range=1, z_range=1)
CASES = [
    # (mag x, y, z), (T, D, H, W), axes, method
    ((2, 2, 2), (3, 8, 8, 8), 6, 1),      # whole tiles: 16 x 8 x 16 subvoxels
    ((2, 2, 2), (2, 7, 9, 17), 6, 1),     # one subvoxel row or more past a tile on every axis
    ((4, 4, 2), (3, 6, 8, 8), 6, 3),      # y innermost, 32 deep
    ((4, 4, 2), (2, 5, 9, 5), 6, 1),
    ((2, 2, 4), (3, 8, 6, 9), 6, 1),      # z innermost
    ((3, 5, 1), (2, 9, 7, 6), 6, 1),
    ((1, 2, 5), (2, 9, 8, 19), 6, 1),     # 21 cells of x per tile
    ((3, 3, 3), (3, 7, 5, 6), 5, 1),      # odd axis count: nothing at a quarter turn
    ((2, 3, 2), (3, 7, 6, 8), 3, 3),
    ((2, 2, 2), (2, 7, 7, 7), 12, 1),     # tables in global memory
    ((2, 4, 2), (2, 6, 6, 7), 32, 1),     # the largest ring
]


@pytest.mark.parametrize("mag,shape,axes,method", CASES)
def test_plan_choice_matches_oracle(ctx, oracle_mod, mag, shape, axes, method):
    from rfba_gb300 import synth
    from rfba_gb300.srrf import Config
    kw = dict(mag=mag, method=method, axes_in_ring=axes, itc=0, **SMOOTH)
    T, D, H, W = shape
    scene = synth.make_scene(40 + axes, T, (W, H, D), 8)
    for dtype in (np.uint16, np.float32):
        x = synth.render(scene, (W, H, D), 40 + axes, dtype)
        got = ctx.forward(Config.make(**kw), np.ascontiguousarray(x))
        ref = oracle_mod.srrf_region(x.astype(np.float32), oracle_mod.make_conf(**kw))
        assert_parity(got, ref, tol_for(method), f"{mag} {shape} axes {axes} {np.dtype(dtype).name}")

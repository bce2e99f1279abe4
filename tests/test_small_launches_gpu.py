"""The tiles that launches of few (tile, volume) items get: two coarse cells deep at
innermost magnifications of 5 and more, and the adjoint's at half their depth, beside
their full depth; against the FP64 oracle and the FP64 adjoint with the other
configurations' tolerances. tests/test_tile_depth_cpu.py checks the depths."""
import numpy as np
import pytest

from tests.parity import assert_parity, rel_linf, tol_for
from tests.test_adjoint_gpu import _case, _gmap, _gpu

pytestmark = pytest.mark.gpu

SMOOTH = dict(gradient_smooth=1, main_range=1, x_range=1, y_range=1, z_range=1)

# (mag, axes, (T, D, H, W)) with two-cell tiles
FLAT = [((5, 5, 5), 6, (2, 6, 6, 7)), ((6, 6, 6), 5, (2, 6, 5, 7)), ((7, 7, 7), 4, (2, 5, 6, 6)),
        ((8, 8, 8), 6, (1, 6, 5, 6)), ((2, 3, 8), 6, (2, 7, 8, 9)), ((1, 6, 2), 13, (2, 8, 7, 19)),
        ((3, 1, 7), 14, (2, 6, 9, 8))]
GRADIENTS = [SMOOTH, dict(gradient_smooth=0), dict(gradient_smooth=1, main_range=2, x_range=1, y_range=3, z_range=0)]


@pytest.mark.parametrize("mag,axes,shape", FLAT)
@pytest.mark.parametrize("grad", range(3))
def test_two_cell_tiles_match_oracle(ctx, oracle_mod, mag, axes, shape, grad):
    from rfba_gb300 import synth
    from rfba_gb300.srrf import Config
    kw = dict(mag=mag, method=1, axes_in_ring=axes, **GRADIENTS[grad])
    T, D, H, W = shape
    for dtype in (np.uint16, np.float32):
        x = synth.render(synth.make_scene(axes, T, (W, H, D), 8), (W, H, D), axes, dtype)
        got = ctx.forward(Config.make(**kw), np.ascontiguousarray(x))
        ref = oracle_mod.srrf_region(x.astype(np.float32), oracle_mod.make_conf(**kw))
        assert_parity(got, ref, tol_for(1), f"{mag} axes {axes} {np.dtype(dtype).name}")


# (mag, axes, (T, D, H, W), the adjoint's depth)
ADJOINT = [((2, 2, 2), 6, (5, 9, 8, 9), 4), ((2, 2, 2), 6, (80, 7, 7, 9), 8), ((4, 4, 2), 6, (5, 7, 8, 8), 4),
           ((4, 4, 2), 5, (80, 7, 8, 8), 8), ((3, 3, 3), 6, (5, 7, 7, 7), 4), ((3, 3, 3), 6, (60, 7, 7, 7), 8),
           ((1, 1, 1), 6, (8, 15, 15, 17), 4), ((1, 1, 1), 6, (160, 8, 8, 17), 8), ((5, 5, 5), 4, (5, 6, 6, 6), 2),
           ((2, 3, 8), 4, (5, 7, 8, 7), 2), ((2, 3, 8), 4, (60, 7, 8, 7), 4),
           ((8, 8, 6), 3, (5, 6, 5, 5), 2), ((2, 2, 2), 14, (5, 8, 8, 8), 8)]


@pytest.mark.parametrize("mag,axes,shape,depth", ADJOINT)
def test_adjoint_depths_match_fp64_adjoint(ctx, oracle_mod, mag, axes, shape, depth):
    from rfba_gb300 import srrf
    O = oracle_mod
    kw = dict(mag=mag, method=3, itc=0, trac_order=2, axes_in_ring=axes, **SMOOTH)
    x, sh = _case(90 + axes, *shape, drift=0.25)
    m, din, dsh = _gpu(ctx, srrf.Config.make(**kw), x, sh)
    mo = O.forward_shifted(x, O.make_conf(**kw), sh)
    assert_parity(m, mo, 1e-4, f"{mag} axes {axes} forward")
    _, din_o, dsh_o = O.adjoint(x, O.make_conf(**kw), _gmap(mo), sh)
    assert rel_linf(din, din_o) < 2e-4 and rel_linf(dsh, dsh_o) < 2e-4


# (mag, volume (D, H, W), volumes): the whole series has full tiles, an eighth of it half tiles
SERIES = [((1, 1, 1), (8, 8, 17), 160), ((2, 2, 2), (7, 7, 9), 80), ((3, 3, 3), (7, 7, 7), 64), ((4, 4, 2), (7, 8, 8), 80),
          ((4, 4, 4), (7, 6, 7), 32), ((5, 5, 5), (7, 6, 7), 24), ((6, 6, 6), (6, 6, 7), 16), ((7, 7, 7), (6, 5, 6), 16),
          ((8, 8, 8), (5, 6, 6), 16)]


@pytest.mark.parametrize("mag,volume,n", SERIES)
def test_adjoint_depths_agree(ctx, mag, volume, n):
    """With the temporal mean and intensity weighting off a volume's dL/dI does not
    depend on the others, so a series in eighths gives the same in half tiles as whole in
    full ones: the same terms, summed in shares of up to 32 tiles instead of 8. 32
    roundings of 2^-24 on sums up to 4 times the largest value are 8e-6 of it; 2e-5 is
    allowed."""
    import torch
    from rfba_gb300 import srrf
    cfg = srrf.Config.make(mag=mag, method=1, intensity_w=0, axes_in_ring=5, **SMOOTH)
    x, _ = _case(sum(mag), n, *volume)
    xd = torch.from_numpy(x).cuda()
    g = torch.from_numpy(np.random.default_rng(7).standard_normal([m * v for m, v in zip(mag[::-1], volume)]).astype(np.float32)).cuda()
    whole, _ = ctx.backward(cfg, xd, None, g)
    parts = [ctx.backward(cfg, c.contiguous(), None, g / 8)[0] for c in xd.split(n // 8)]
    torch.cuda.synchronize()
    scale = whole.abs().max().item()
    assert scale > 0 and (whole - torch.cat(parts)).abs().max().item() < 2e-5 * scale

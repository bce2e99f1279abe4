"""Rings at the size where their tables move from the kernel parameters to global
memory, which the forward and the adjoint do at different sizes: maps at both tile
depths against the FP64 oracle, dL/dI against the FP64 adjoint. Tolerances as for the
other configurations."""
import numpy as np
import pytest

from tests.parity import assert_parity, rel_linf, tol_for
from tests.test_adjoint_gpu import _case, _gmap, _gpu

pytestmark = pytest.mark.gpu

SMOOTH = dict(gradient_smooth=1, main_range=1, x_range=1, y_range=1, z_range=1)

# (mag, axes, (T, D, H, W) that gets deep tiles)
RINGS = [((2, 2, 2), 9, (80, 7, 7, 9)), ((2, 2, 2), 12, (80, 7, 7, 9)), ((2, 2, 2), 13, (80, 7, 7, 9)),
         ((2, 2, 2), 14, (80, 7, 7, 9)), ((3, 2, 1), 14, (40, 9, 15, 12)), ((1, 5, 2), 13, (100, 7, 7, 20))]


@pytest.mark.parametrize("mag,axes,shape", RINGS)
@pytest.mark.parametrize("deep", [False, True])
def test_map_matches_oracle(ctx, oracle_mod, mag, axes, shape, deep):
    from rfba_gb300 import synth
    from rfba_gb300.srrf import Config
    kw = dict(mag=mag, method=1, axes_in_ring=axes, **SMOOTH)
    T, D, H, W = shape if deep else (2,) + shape[1:]
    x = synth.render(synth.make_scene(axes, T, (W, H, D), 8), (W, H, D), axes, np.uint16)
    got = ctx.forward(Config.make(**kw), np.ascontiguousarray(x))
    ref = oracle_mod.srrf_region(x.astype(np.float32), oracle_mod.make_conf(**kw))
    assert_parity(got, ref, tol_for(1), f"{mag} axes {axes}")


@pytest.mark.parametrize("mag,axes", [((2, 2, 2), 12), ((2, 2, 2), 13), ((2, 2, 2), 14), ((3, 2, 1), 14), ((1, 4, 2), 9)])
def test_adjoint_matches_fp64_adjoint(ctx, oracle_mod, mag, axes):
    from rfba_gb300 import srrf
    O = oracle_mod
    kw = dict(mag=mag, method=3, itc=0, trac_order=2, axes_in_ring=axes, **SMOOTH)
    x, sh = _case(70 + axes, 5, 8, 8, 8, drift=0.25)
    m, din, dsh = _gpu(ctx, srrf.Config.make(**kw), x, sh)
    mo = O.forward_shifted(x, O.make_conf(**kw), sh)
    assert_parity(m, mo, 1e-4, f"{mag} axes {axes} forward")
    _, din_o, dsh_o = O.adjoint(x, O.make_conf(**kw), _gmap(mo), sh)
    assert rel_linf(din, din_o) < 2e-4 and rel_linf(dsh, dsh_o) < 2e-4

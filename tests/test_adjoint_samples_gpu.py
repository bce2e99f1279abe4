"""Ill-conditioned ring samples in the radiality adjoint.

A sample whose gradient nearly follows the ring direction, or nearly vanishes, has a
derivative that amplifies the rounding of the interpolated gradient. The adjoint forms
it in one fixed order of operations, whatever the plan's axis order, the launch and
however many such samples there are. With the temporal mean and intensity weighting
off, identical volumes have identical dL/dI, so every volume is compared with the
first: their sums differ only in the order in which tiles add to a voxel.

Tolerance: a voxel of dL/dI is a sum of at most 8 tiles' shares (16 x 8 x 16 or more
subvoxels at magnification 2, halo 3), each at most a few times the largest dL/dI and
the same in every volume. The order in which they add is not: 8 roundings of 2^-24 on
sums up to 4 times the largest value are 2e-6 of it, and ten times that is allowed.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SAME_VOLUME_TOL = 2e-5


def _cfg(**kw):
    from rfba_gb300 import srrf
    base = dict(mag=2, method=1, intensity_w=0, gradient_smooth=1, main_range=1, x_range=1, y_range=1, z_range=1)
    base.update(kw)
    return srrf.Config.make(**base)


def _ramp(rng, shape, direction, noise):
    """A ramp of slope 1 along direction (x, y, z) with noise relative to its slope."""
    d, h, w = shape
    z, y, x = np.meshgrid(np.arange(d), np.arange(h), np.arange(w), indexing="ij")
    v = direction[0] * x + direction[1] * y + direction[2] * z
    return (v + noise * rng.standard_normal(shape)).astype(np.float32)


def _backward(ctx, cfg, x):
    import torch
    xd = torch.from_numpy(x).cuda()
    m = ctx.forward_shifted(cfg, xd, None)
    g = torch.from_numpy(np.random.default_rng(1).standard_normal(tuple(m.shape)).astype(np.float32)).cuda()
    g = torch.where(torch.isfinite(m), g, torch.zeros_like(g))
    din, _ = ctx.backward(cfg, xd, None, g)
    torch.cuda.synchronize()
    return din.cpu().numpy(), g.cpu().numpy()


def _worst(din):
    scale = np.abs(din[0]).max()
    assert np.isfinite(din).all() and scale > 0
    return np.abs(din - din[:1]).max() / scale


@pytest.mark.parametrize("mag", [(2, 2, 2), (2, 4, 2)])
def test_tiny_gradients_have_one_derivative(ctx, mag):
    """Gradients so small that every sample is under the guard of 1 / sqrt(c2 g2): more
    than 4 million samples a volume."""
    rng = np.random.default_rng(3)
    vol = np.ldexp(rng.uniform(100, 600, (32, 32, 32)), -50).astype(np.float32)
    din, _ = _backward(ctx, _cfg(mag=mag), np.repeat(vol[None], 8, 0))
    e = _worst(din)
    assert e < SAME_VOLUME_TOL, e


@pytest.mark.parametrize("mag,direction", [((2, 2, 2), (1, 0, 0)), ((2, 2, 2), (0, 0, 1)), ((2, 4, 2), (0, 1, 0)),
                                           ((4, 2, 4), (0.5, 0.75 ** 0.5, 0))])
def test_any_number_of_samples_is_corrected(ctx, mag, direction):
    """Gradients within 1e-4 or so of a ring direction at every voxel: two of each
    subvoxel's samples, 0.5 million or more a volume."""
    rng = np.random.default_rng(4)
    vol = _ramp(rng, (32, 32, 32), direction, 3e-5)
    din, _ = _backward(ctx, _cfg(mag=mag), np.repeat(vol[None], 4, 0))
    e = _worst(din)
    assert e < SAME_VOLUME_TOL, e


def test_corrections_beyond_two_billion_subvoxels(ctx):
    """The same samples in the last planes of a map of 2.26e9 subvoxels against the
    region that holds only those planes."""
    import torch
    if torch.cuda.mem_get_info()[0] < 160 << 30:
        pytest.skip("needs 160 GB of device memory")
    n, planes = 164, 64
    rng = np.random.default_rng(5)
    x = torch.from_numpy(_ramp(rng, (n, n, n), (1, 0, 0), 3e-5)[None]).cuda()
    cfg = _cfg(mag=8, axes_in_ring=2)
    N = 8 * n
    g = torch.zeros((N, N, N), device="cuda")
    gen = torch.Generator(device="cuda").manual_seed(2)
    g[N - planes:].normal_(generator=gen)
    c = srrf_context()
    try:
        din, _ = c.backward(cfg, x, None, g)
        reg, _ = c.backward_region(cfg, x, None, (0, 0, N - planes), (N, N, N), g[N - planes:].contiguous())
        torch.cuda.synchronize()
        scale = reg.abs().max().item()
        e = (din - reg).abs().max().item() / scale
    finally:
        c.close()
        del g, x
        torch.cuda.empty_cache()
    assert scale > 0 and e < SAME_VOLUME_TOL, e


def srrf_context():
    from rfba_gb300 import srrf
    return srrf.Context(0)

"""Tomography calls at the edges of what the device holds: FP64 gradients that run short
of scratch, and quadratures of more nodes than a block has room for."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _paths(dp, ctx, nodes, n_rays, seed=3):
    import torch
    phys = dp.create_physics(ctx=ctx)
    grid = dp.VoxelGrid(48, 44, 24, (-240.0, -220.0, 0.0), 10.0)
    rng = np.random.default_rng(seed)
    rho = rng.uniform(1500.0, 3000.0, grid.ncell)
    o = np.column_stack([rng.uniform(-200, 200, n_rays), rng.uniform(-180, 180, n_rays), np.zeros(n_rays)])
    rays = dp.make_rays(o, rng.uniform(0.0, 80.0, n_rays), rng.uniform(0.0, 360.0, n_rays))
    paths = dp.TomoPaths(phys, grid, rays, nodes, side_density=2500.0)
    cuda = lambda x: torch.tensor(x, dtype=torch.float64, device=paths.dev)  # noqa: E731
    return paths, cuda(rho), cuda(rng.uniform(0.5, 1.5, n_rays))


def test_fp64_gradient_short_of_scratch():
    """With room for a few CTAs' terms only, the gradient is the same, bit for bit; with
    room for none the call says so and the next one runs."""
    import dpgpu as dp
    ctx = dp.Context(0)
    limit = lambda n: dp.check(dp.load().dp_set_debug_scratch(ctx.h, n), ctx.h)  # noqa: E731
    E = np.geomspace(1.0, 1e5, 40)
    paths, rho, cot = _paths(dp, ctx, (E, np.ones(40), 0.1 * E), 3000)
    per_cta = 4 * 512 * paths.max_segments
    limit(8 * paths.nnz + 20 * per_cta)
    few = [x.cpu().numpy() for x in paths.eval(rho, cot, precision="fp64")[:2]]
    limit(-1)
    full = [x.cpu().numpy() for x in paths.eval(rho, cot, precision="fp64")[:2]]
    assert dp.load().dp_scratch_bytes(ctx.h) > 8 * paths.nnz + 100 * per_cta
    for a, b in zip(few, full):
        np.testing.assert_array_equal(a, b)
    other = dp.Context(0)
    paths, rho, cot = _paths(dp, other, (E, np.ones(40), 0.1 * E), 3000)
    dp.check(dp.load().dp_set_debug_scratch(other.h, 4096), other.h)
    with pytest.raises(dp.DpError, match="allocation"):
        paths.eval(rho, cot, precision="fp64")
    dp.check(dp.load().dp_set_debug_scratch(other.h, -1), other.h)
    for a, b in zip(paths.eval(rho, cot, precision="fp64")[:2], full):
        np.testing.assert_array_equal(a.cpu().numpy(), b)


def test_mixed_with_thousands_of_nodes():
    """90 copies of 100 nodes have the 100 nodes' mean.  A node's coefficient 2 w / N is
    rounded to FP32 on either side (2^-23 together, 2^-22 allowed), and a segment's
    entry is summed in FP32 over 282 groups of nodes of one sign (282 2^-24)."""
    import dpgpu as dp
    E, q = np.geomspace(1.0, 1e5, 100), np.where(np.arange(100) % 2, 1.0, -1.0)
    out = []
    for k in (1, 90):
        paths, rho, cot = _paths(dp, dp.default_context(), [np.tile(x, k) for x in (E, q, 0.1 * E)], 60)
        f, g, _ = paths.eval(rho, cot, precision="mixed")
        np.testing.assert_array_equal(paths.eval(rho, precision="mixed")[0].cpu().numpy(), f.cpu().numpy())
        out.append((f.cpu().numpy(), g.cpu().numpy()))
    (f0, g0), (f1, g1) = out
    assert (f0 > 0).all()
    np.testing.assert_allclose(f1, f0, rtol=2.0 ** -22, atol=0)
    np.testing.assert_allclose(g1, g0, rtol=0, atol=282 * 2.0 ** -24 * np.abs(g0).max())

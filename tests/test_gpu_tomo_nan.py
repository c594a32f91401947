"""Invalid values in the FP64 tomography: a NaN density ends every node of the rays
that cross its cell, whichever its sign (0/0 on an x86 host has it set), and a NaN node
energy ends its node.  Their flux is 0 and they add nothing to the gradient; the other
rays and nodes keep every bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

NAN = {"plus": np.nan, "minus": -np.float64(np.nan)}


@pytest.fixture(scope="module")
def scene():
    import dpgpu as dp
    phys = dp.create_physics()
    grid = dp.VoxelGrid(12, 10, 8, (-60.0, -50.0, 0.0), 10.0)
    rng = np.random.default_rng(8)
    rho = rng.uniform(1500.0, 3000.0, grid.ncell)
    o = np.column_stack([rng.uniform(-50, 50, 60), rng.uniform(-40, 40, 60), np.zeros(60)])
    rays = dp.make_rays(o, rng.uniform(0.0, 70.0, 60), rng.uniform(0.0, 360.0, 60))
    return dp, phys, grid, rho, rays, rng.uniform(0.5, 1.5, 60)


@pytest.mark.parametrize("sign", list(NAN))
def test_nan_density(scene, sign):
    dp, phys, grid, rho, rays, cot = scene
    E = np.geomspace(0.5, 1e5, 40)
    model = dp.TomoModel(phys, grid, (E, np.ones(40), 0.1 * E), side_density=2500.0, precision="fp64")
    flux, grad = model.vjp(rho, rays, cot)
    cell = int(np.argmax(np.abs(grad)))
    heavy, bad = rho.copy(), rho.copy()
    heavy[cell] *= 1.5
    bad[cell] = NAN[sign]
    assert np.signbit(bad[cell]) == (sign == "minus")
    crosses = model.forward(heavy, rays) != flux
    assert 0 < crosses.sum() < len(rays)
    f, g = model.vjp(bad, rays, cot)
    np.testing.assert_array_equal(f, np.where(crosses, 0.0, flux))
    np.testing.assert_array_equal(model.forward(bad, rays), f)
    np.testing.assert_array_equal(g, model.vjp(rho, rays, np.where(crosses, 0.0, cot))[1])


@pytest.mark.parametrize("sign", list(NAN))
def test_nan_node(scene, sign):
    dp, phys, grid, rho, rays, cot = scene
    E = np.geomspace(0.5, 1e5, 40)
    q, w = np.ones(40), 0.1 * E
    bad, w0 = E.copy(), w.copy()
    bad[7], w0[7] = NAN[sign], 0.0
    a = dp.TomoModel(phys, grid, (bad, q, w), side_density=2500.0, precision="fp64").vjp(rho, rays, cot)
    b = dp.TomoModel(phys, grid, (E, q, w0), side_density=2500.0, precision="fp64").vjp(rho, rays, cot)
    for x, y in zip(a, b):
        np.testing.assert_array_equal(x, y)


@pytest.mark.parametrize("e", [1e300, 1e160, 1e140, np.inf, -np.inf, -1.0, -0.1, -0.05, 0.0, 1e-300])
def test_node_far_off_the_grid(oracle, e):
    """Squares of such energies overflow or are negative; the reference's operations give
    a finite flux.  Against the oracle, whose derivative at an infinite energy is NaN
    (the node is clamped there and has none)."""
    import dpgpu as dp
    orc = oracle.default_physics((oracle.STANDARD_ROCK, oracle.AIR))
    phys = dp.upload_physics([orc.table(0), orc.table(1)], ["StandardRock", "Air"])
    grid = dp.VoxelGrid(6, 6, 4, (-30.0, -30.0, 0.0), 10.0)
    rho = np.random.default_rng(1).uniform(1500.0, 3000.0, grid.ncell)
    rays = dp.make_rays([[0.0, 0.0, 0.0]] * 5 + [[900.0, 0.0, 0.0]], [0.0, 20.0, 40.0, 60.0, 80.0, 10.0], np.arange(6) * 50.0)
    nodes = (np.array([0.5, e, 100.0]), np.array([1.0, 0.0, 1.0]), np.array([1.0, 2.0, 3.0]))
    model = dp.TomoModel(phys, grid, nodes, side_density=2500.0, precision="fp64")
    flux, grad = model.vjp(rho, rays, np.ones(6))
    of, og = oracle.tomo_vjp(orc, 0, 1, np.array([6, 6, 4], np.int32), np.array([-30.0, -30.0, 0.0, 10.0, 10.0, 10.0]), rho,
                             2500.0, rays, nodes, np.ones(6))
    np.testing.assert_allclose(flux, of, rtol=1e-9, atol=0)
    if np.isinf(e):
        assert np.isfinite(grad).all() and (grad != 0).any()
    else:
        np.testing.assert_allclose(grad, og, rtol=1e-7, atol=1e-10 * np.abs(og).max())


@pytest.mark.parametrize("sign", list(NAN))
def test_nan_node_mixed(scene, sign):
    dp, phys, grid, rho, rays, cot = scene
    E = np.geomspace(0.5, 1e5, 40)
    q, w = np.ones(40), 0.1 * E
    bad, w0 = E.copy(), w.copy()
    bad[7], w0[7] = NAN[sign], 0.0
    a = dp.TomoModel(phys, grid, (bad, q, w), side_density=2500.0, precision="mixed").vjp(rho, rays, cot)
    b = dp.TomoModel(phys, grid, (E, q, w0), side_density=2500.0, precision="mixed").vjp(rho, rays, cot)
    for x, y in zip(a, b):
        np.testing.assert_array_equal(x, y)

"""The FP64 tomography kernel at its edges against the oracle's reverse sweep:
one node, a full warp of nodes and more than one; nodes below the energy grid,
at its top and carried past it by the rock; rays that miss the grid, of one
segment and of more than two 32-segment tiles.

Both sides are FP64 and differ by the rounding of up to 10^2 segments
(~1e-13); the tolerances are those of the other FP64 comparisons of this model
(1e-9 on the flux, 1e-7 and 1e-10 of the largest entry on the gradient)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def scene(oracle):
    import dpgpu as dp
    orc = oracle.default_physics((oracle.STANDARD_ROCK, oracle.AIR))
    phys = dp.upload_physics([orc.table(0), orc.table(1)], ["StandardRock", "Air"])
    grid = dp.VoxelGrid(40, 36, 20, (-200.0, -180.0, 0.0), 10.0)
    rng = np.random.default_rng(4)
    rho = rng.uniform(800.0, 3200.0, grid.ncell)
    zen = np.concatenate([rng.uniform(0.0, 85.0, 40), [0.0, 89.5]])
    o = np.column_stack([rng.uniform(-190, 190, 42), rng.uniform(-170, 170, 42), np.zeros(42)])
    o[0], o[1], o[2] = (900.0, 0.0, 0.0), (0.0, 0.0, 250.0), (0.5, 0.5, 199.0)
    rays = dp.make_rays(o, zen, rng.uniform(0.0, 360.0, 42))
    return dp, orc, phys, grid, rho, rays


NODES = {"one": [3.0], "warp": np.geomspace(1.0, 1e6, 32), "more": np.geomspace(2e-3, 1e6, 33),
         "ends": np.concatenate([[2e-4, 1e-3, 9e8, 9.9e8, 1e9, 2e9], np.geomspace(1e-2, 1e8, 40)])}


@pytest.mark.parametrize("which", list(NODES))
def test_flux_and_gradient_match_oracle(scene, oracle, which):
    dp, orc, phys, grid, rho, rays = scene
    E = np.asarray(NODES[which], float)
    nodes = (E, np.where(np.arange(len(E)) % 3, 0.0, 1.0), 0.1 * E)
    cot = np.random.default_rng(1).uniform(0.5, 1.5, len(rays))
    model = dp.TomoModel(phys, grid, nodes, side_density=2500.0, precision="fp64")
    flux, grad = model.vjp(rho, rays, cot)
    dims = np.array([grid.nx, grid.ny, grid.nz], np.int32)
    geom = np.array([*grid.origin, *grid.pitch])
    of, og = oracle.tomo_vjp(orc, 0, 1, dims, geom, rho, 2500.0, rays, nodes, cot)
    np.testing.assert_allclose(flux, of, rtol=1e-9, atol=0)
    np.testing.assert_array_equal(model.forward(rho, rays), flux)
    np.testing.assert_allclose(grad, og, rtol=1e-7, atol=1e-10 * np.abs(og).max())

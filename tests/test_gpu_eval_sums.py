"""The mixed tomography kernel's sums over nodes, taken four segments at a time:
rays of 1 to 9 segments, node counts around a warp's lanes, against the sum of
one-node evaluations of the same rays.

A node's term does not depend on its lane; the two differ by the roundings of the
term's weight and of a tree of at most 7 additions: 16 2^-24 of the sum of
magnitudes."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_nodes", [1, 2, 31, 32, 33, 70])
def test_jacobian_is_the_sum_of_its_nodes(n_nodes):
    import dpgpu as dp
    import torch
    phys = dp.create_physics()
    rng = np.random.default_rng(n_nodes)
    E = np.geomspace(2e-3, 1e6, n_nodes) if n_nodes > 1 else np.array([3.0])
    q, w = np.where(np.arange(n_nodes) % 2, -1.0, 1.0), 0.1 * E
    for nz in range(1, 10):
        grid = dp.VoxelGrid(4, 4, nz, (-20.0, -20.0, 0.0), 10.0)
        o = np.column_stack([rng.uniform(-19, 19, 6), rng.uniform(-19, 19, 6), np.zeros(6)])
        rays = dp.make_rays(o, np.array([0.0, 0.0, 0.0, 20.0, 45.0, 70.0]), rng.uniform(0, 360, 6))
        rho = rng.uniform(1500.0, 2900.0, grid.ncell)

        def jac(sl):
            paths = dp.TomoPaths(phys, grid, rays, (E[sl], q[sl], w[sl]), side_density=2500.0)
            out = torch.empty(paths.nnz, dtype=torch.float64, device=paths.dev)
            paths.eval(torch.tensor(rho, device=paths.dev), torch.ones(6, dtype=torch.float64, device=paths.dev),
                       precision="mixed", jac=out)
            return out.cpu().numpy()

        one = np.array([jac(slice(k, k + 1)) for k in range(n_nodes)]) / n_nodes
        assert np.all(np.abs(jac(slice(None)) - one.sum(0)) <= 16 * 2.0 ** -24 * np.abs(one).sum(0))

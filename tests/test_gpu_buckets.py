"""J^T r, J v and the column sums over a grid's buckets at the edges of how their
entries are dealt, against numpy on the product's own Jacobian: grids of less than
32 cells and of no multiple of 128, empty cells, rays off the grid, buckets around
32 entries (a lane's share), some 500 to 1000 entries in 32 cells (what a warp
stages), and a bucket past 2048 (a warp's share), its rays in runs.

The Jacobian is the same on both sides; a sum of n <= 4000 terms differs by
n 2^-53 of the sum of their magnitudes, 5e-13.  The iterates are within 1e-10."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# grid, rays, detectors (0: one per ray), side cell
SCENES = {"one": ((3, 3, 3), 1, 1, -1), "few": ((5, 5, 5), 12, 0, 3), "lane": ((9, 7, 6), 500, 0, -1),
          "stage": ((13, 11, 9), 1800, 0, -1), "hot": ((10, 9, 7), 4000, 1, 77),
          "sparse": ((30, 29, 11), 40, 2, -1)}


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("which", list(SCENES))
def test_bucket_sums_match_numpy(which, precision):
    import dpgpu as dp
    import torch
    (nx, ny, nz), n, n_det, side = SCENES[which]
    rng = np.random.default_rng(7)
    grid = dp.VoxelGrid(nx, ny, nz, (-5.0 * nx, -5.0 * ny, 0.0), 10.0)
    o = np.column_stack([rng.uniform(-4.9, 4.9, n) * nx, rng.uniform(-4.9, 4.9, n) * ny, np.zeros(n)])
    if n_det:
        o = o[np.arange(n) % n_det]
    if n > 20:
        o[-3:] = (5000.0, 0.0, 0.0)  # off the grid
    rays = dp.make_rays(o, rng.uniform(0.0, 80.0, n), rng.uniform(0.0, 360.0, n))
    paths = dp.TomoPaths(dp.create_physics(), grid, rays, dp.csda_energy_quadrature(16, 1.0, 1e6),
                         side_cell=side, side_density=2500.0)
    T = lambda a: torch.tensor(np.ascontiguousarray(a, np.float64), device=paths.dev)
    rho0 = rng.uniform(1500.0, 2900.0, grid.ncell)
    flux = lambda x: paths.eval(T(x), precision=precision)[0].cpu().numpy()
    obs = flux(rho0 * rng.uniform(0.97, 1.03, grid.ncell))

    jac = torch.empty(paths.nnz, dtype=torch.float64, device=paths.dev)
    cot = rng.normal(size=n)
    f0, grad, _ = paths.eval(T(rho0), T(cot), precision=precision, jac=jac)
    f0 = f0.cpu().numpy()
    rp, col, _ = paths.csr()
    row, val = np.repeat(np.arange(n), np.diff(rp)), jac.cpu().numpy()
    J = np.zeros((n, grid.ncell))
    np.add.at(J, (row[col >= 0], col[col >= 0]), val[col >= 0])
    mag = np.abs(J).T @ np.abs(cot)
    assert np.all(np.abs(grad.cpu().numpy() - J.T @ cot) <= 1e-12 * mag)

    box, r = (500.0, 3500.0), f0 - obs
    one = lambda s: np.where(s == 0, 1.0, s)
    x, hist = paths.solve(T(obs), T(rho0), method="sart", n_iter=1, box=box, precision=precision)
    ref = np.clip(rho0 - 0.2 * (J.T @ (r / one(np.abs(J).sum(1)))) / one(np.abs(J).sum(0)), *box)
    np.testing.assert_allclose(x.cpu().numpy(), ref, rtol=1e-10)
    assert hist[0] == pytest.approx(np.linalg.norm(r), rel=1e-10)

    W, mu = 1.0 / obs ** 2, 10.0
    x, _ = paths.solve(T(obs), T(rho0), method="gn", n_iter=1, weight=T(W), cg_iter=1, lm_damping=mu, box=box,
                       precision=precision)
    g, D = J.T @ (W * r), (W[:, None] * J * J).sum(0)
    D = np.maximum(D, 1e-12 * D.max())
    p = -g / ((1 + mu) * D)
    step = p * (-g @ p) / (p @ (J.T @ (W * (J @ p)) + mu * D * p))
    cost = lambda f: 0.5 * np.sum(W * (f - obs) ** 2)
    for k in range(10):  # the line search
        ref = np.clip(rho0 + 0.5 ** k * step, *box)
        if cost(flux(ref)) < cost(f0):
            break
    np.testing.assert_allclose(x.cpu().numpy(), ref, rtol=1e-10)

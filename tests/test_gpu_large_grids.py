"""Energy grids of many nodes, up to the largest that the tables of each kernel leave
room for, against the oracle.  The tolerances are those of each model's other
comparisons: a finer grid adds no operation to a step."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _physics(oracle, n):
    import dpgpu as dp
    orc = oracle.default_physics((oracle.STANDARD_ROCK, oracle.AIR, oracle.WATER), n=n)
    return dp, orc, dp.upload_physics([orc.table(i) for i in range(3)], ["StandardRock", "Air", "Water"])


@pytest.mark.parametrize("n", [720, 721, 764])
def test_mixed_csda(oracle, n):
    dp, orc, phys = _physics(oracle, n)
    t, rho, el = 100.0, 2650.0, 45.0
    E, q, w = dp.mc_samples(phys, energy_min=1.0, energy_max=100.0, n_samples=4096, seed=11)
    c, d = dp.csda_flux_samples(phys, E, q, w, precision="mixed", rock_thickness=t, rock_density=rho, elevation=el)
    oc, od = oracle.backward_mc_csda(orc, 0, 1, t, rho, el, E, q, w)
    assert (oc > 0).sum() > 100
    for x, ox, atol in ((c, oc, 1e-12 * oc.max()), (d, od, 1e-6 * np.abs(od).max())):
        assert (np.abs(x - ox) > 2e-6 * np.abs(ox) + atol).mean() <= 2e-3
        np.testing.assert_allclose(x, ox, rtol=1e-3, atol=atol)
        assert x.sum() == pytest.approx(ox.sum(), rel=1e-6)


@pytest.mark.parametrize("n", [1709, 2420])
def test_fp64_water_fraction(oracle, n):
    """The columns that the corrections read stay out of shared memory from 1709 nodes on."""
    import test_gpu_wtomo as T
    dp, orc, phys = _physics(oracle, n)
    rng = np.random.default_rng(2)
    wf = rng.uniform(0.0, 0.5, 12)
    seg = lambda k: [dp.CellSegment(int(c), float(rng.uniform(2.0, 40.0))) for c in rng.integers(1, 13, k)]  # noqa: E731
    paths = [dp.DirectionalPath(z, 0.0, seg(k), 0.0, 0.0, 5.0 * k, 60.0, True) for k, z in enumerate((0.0, 20.0, 45.0, 65.0))]
    c = T.CORR["correction"]
    corr = [1, c["kappa_strag"], c["kappa_hard"], c["resid_a"], c["resid_b"], c["resid_c"], c["resid_d"], 0, 0.0, 0.0]
    cfg, site = dp.MaterialConfig(1, 3, 2, 1, 2650.0, 1000.0, 1800.0, 20.0), dp.SiteConfig(963.0, 3e4)
    shallow, samples = np.arange(12) % 2 == 0, T._samples(dp, 33, 4)
    try:
        dp.set_csda_correction(**c)
        f, seg_ptr, cells, jac = dp.csda_flux_batch(phys, shallow, cfg, site, paths, wf, samples)
    finally:
        dp.set_csda_correction(enabled=False)
    of, og = T._oracle(oracle, orc, wf, paths, samples, corr, shallow.astype(np.uint8), [0, 2, 1, 0],
                       (2650.0, 1000.0, 1800.0, 20.0))
    assert (of > 0).all()
    np.testing.assert_allclose(f, of, rtol=1e-10, atol=0)
    np.testing.assert_allclose(T._per_cell_first(seg_ptr, cells, jac), og, rtol=1e-8, atol=1e-12 * np.abs(og).max())


@pytest.mark.parametrize("n", [3400, 5000])
def test_fp64_tomography(oracle, n):
    """The columns that a ray reads at its ends stay out of shared memory (3400 nodes:
    with the gradient only), and two warps find room where four do otherwise (5000)."""
    import dpgpu as dp
    orc = oracle.default_physics((oracle.STANDARD_ROCK, oracle.AIR), n=n)
    phys = dp.upload_physics([orc.table(0), orc.table(1)], ["StandardRock", "Air"])
    grid = dp.VoxelGrid(40, 36, 20, (-200.0, -180.0, 0.0), 10.0)
    rng = np.random.default_rng(4)
    rho = rng.uniform(800.0, 3200.0, grid.ncell)
    o = np.column_stack([rng.uniform(-190, 190, 12), rng.uniform(-170, 170, 12), np.zeros(12)])
    rays = dp.make_rays(o, rng.uniform(0.0, 85.0, 12), rng.uniform(0.0, 360.0, 12))
    E = np.concatenate([[2e-4, 1e-3, 9e8, 2e9], np.geomspace(1e-2, 1e8, 37)])
    nodes = (E, np.where(np.arange(len(E)) % 3, 0.0, 1.0), 0.1 * E)
    cot = rng.uniform(0.5, 1.5, len(rays))
    model = dp.TomoModel(phys, grid, nodes, side_density=2500.0, precision="fp64")
    flux, grad = model.vjp(rho, rays, cot)
    dims, geom = np.array([grid.nx, grid.ny, grid.nz], np.int32), np.array([*grid.origin, *grid.pitch])
    of, og = oracle.tomo_vjp(orc, 0, 1, dims, geom, rho, 2500.0, rays, nodes, cot)
    np.testing.assert_allclose(flux, of, rtol=1e-9, atol=0)
    np.testing.assert_array_equal(model.forward(rho, rays), flux)
    np.testing.assert_allclose(grad, og, rtol=1e-7, atol=1e-10 * np.abs(og).max())

"""Histories and samples that start exactly on nodes of the energy grid (the ordinary
input of a scan over tabulated energies), on grids where the device's logarithm of
such an energy and the table's differ by a last place, against the oracle.

A node has the same energy in both its intervals, so nothing is gained or lost there: the
tolerances are those of the other FP64 comparisons of each model."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# grids with such a node near 1 GeV (0.9659 and 0.9771 GeV), and a coarser one
GRIDS = [(200, 1e-3, 1e8), (200, 1e-3, 1e4), (80, 1e-3, 1e6)]


@pytest.fixture(scope="module", params=GRIDS, ids=["1e8", "1e4", "80"])
def setting(request, oracle):
    import dpgpu as dp
    n, lo, hi = request.param
    orc = oracle.default_physics((oracle.STANDARD_ROCK, oracle.AIR, oracle.WATER), n=n, Kmin=lo, Kmax=hi, coulomb=True)
    phys = dp.upload_physics([orc.table(i) for i in range(3)], ["StandardRock", "Air", "Water"],
                             materials=(dp.STANDARD_ROCK, dp.AIR, dp.WATER))
    E = np.asarray(orc.column(0, "E"), float)
    return dp, orc, phys, E[(E > 0.05) & (E < 100.0)]


def test_histories(setting, oracle):
    """As the other histories: 1e-9, and rounding flips a decision in under 1 %."""
    dp, orc, phys, nodes = setting
    E = np.tile(nodes, 1 + 1000 // len(nodes))
    n = len(E)
    rng = np.random.default_rng(1)
    q, w = np.where(rng.random(n) > 0.5, 1.0, -1.0), 2.0 * E
    rock, air = dp.MaterialMixture(phys, 1), dp.MaterialMixture(phys, 2)
    geo = dict(thickness=rng.uniform(1.0, 30.0, n), density=rng.uniform(2000.0, 2800.0, n),
               elevation=rng.uniform(30.0, 90.0, n), primary_altitude=np.full(n, 1300.0))
    c, st, steps, Ef = dp.mc_histories(phys, rock, air, E, q, w, seed=5, precision="fp64", **geo)
    oc, ost, osteps, oE = oracle.mc_histories(orc, [0], 1, geo["thickness"], geo["density"], geo["elevation"],
                                              geo["primary_altitude"], E, q, w, seed=5)
    assert (st == 0).all() and (ost == 0).all()
    near = lambda a, b: np.abs(a - b) <= 1e-9 * np.maximum(np.abs(a), np.abs(b)) + 1e-300  # noqa: E731
    same = near(c, oc) & (steps == osteps) & near(Ef[:, 0], oE)
    assert (~same).sum() <= 0.01 * n, (~same).sum()


def test_water_fraction_samples(setting, oracle):
    """As the other FP64 walks: 1e-10 on the flux, 1e-8 on the Jacobian.  The first
    sample of every path starts on its node with no step before it."""
    from test_gpu_wtomo import _oracle, _per_cell_first
    dp, orc, phys, nodes = setting
    rng = np.random.default_rng(3)
    wf = rng.uniform(0.0, 0.9, 9)
    seg = lambda *c: [dp.CellSegment(int(k), float(rng.uniform(1e-3, 60.0))) for k in c]  # noqa: E731
    P = dp.DirectionalPath
    paths = [P(0.0, 0.0, [], 0.0, 0.0, 0.0, 0.0, True), P(10.0, 0.0, [], 0.0, 0.0, 120.0, 50.0, True),
             P(60.0, 0.0, seg(*range(1, 10)), 0.0, 0.0, 5.0, 500.0, True)]
    cfg, site = dp.MaterialConfig(1, 3, 2, -1, 2650.0, 1000.0, 0.0, 0.0), dp.SiteConfig(963.0, 3e4)
    E = nodes[:256]
    samples = [dp.EnergySample(float(e), 1.0 if k % 2 else -1.0, 0.1 * float(e)) for k, e in enumerate(E)]
    f, seg_ptr, cells, jac = dp.csda_flux_batch(phys, np.zeros(9, bool), cfg, site, paths, wf, samples)
    of, og = _oracle(oracle, orc, wf, paths, samples, [0] * 10)
    np.testing.assert_allclose(f, of, rtol=1e-10, atol=0)
    np.testing.assert_allclose(_per_cell_first(seg_ptr, cells, jac), og, rtol=1e-8, atol=1e-12 * np.abs(og).max())

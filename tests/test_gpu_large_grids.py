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

"""CSDA histories whose source altitude lies inside the rock, at its top or less than a
step of air above it (a survey under a mountain higher than the given altitude): they
end there, in both forms of the FP64 program and in mixed precision.  Against the oracle
with the tolerances of the models' other comparisons."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# thickness, density, elevation, altitude, histories: the first four by warp (few, or
# thick rock), then by thread (many behind thin rock)
GEO = [(100.0, 2650.0, 45.0, 50.0, 200), (100.0, 2650.0, 45.0, 100.0, 200), (100.0, 2650.0, 45.0, 100.5, 200),
       (2000.0, 2650.0, 90.0, 1500.0, 6000), (5.0, 2650.0, 70.0, 3.0, 6000), (5.0, 2650.0, 70.0, 5.0, 6000)]


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("geo", GEO, ids=[f"{g[3]:g} of {g[0]:g} m" for g in GEO])
def test_histories_end_at_the_altitude(oracle, geo, precision):
    import dpgpu as dp
    orc = oracle.default_physics((oracle.STANDARD_ROCK, oracle.AIR))
    phys = dp.upload_physics([orc.table(0), orc.table(1)], ["StandardRock", "Air"])
    t, rho, el, H, n = geo
    rng = np.random.default_rng(int(H))
    E = np.tile(np.exp(rng.uniform(np.log(0.01), np.log(1e6), 200)), n // 200)
    q = np.where(np.arange(n) % 2, 1.0, -1.0)
    c, d = dp.csda_flux_samples(phys, E, q, np.ones(n), rock_thickness=t, rock_density=rho, elevation=el,
                                primary_altitude=H, precision=precision)
    oc, od = oracle.backward_mc_csda(orc, 0, 1, t, rho, el, E, q, np.ones(n), primary_altitude=H)
    assert (oc > 0).sum() > n // 2
    if precision == "fp64":
        np.testing.assert_allclose(c, oc, rtol=1e-9, atol=0)
        np.testing.assert_allclose(d, od, rtol=1e-8, atol=1e-12 * np.abs(od).max())
    else:
        assert (np.abs(c - oc) > 2e-6 * np.abs(oc) + 1e-12 * oc.max()).mean() <= 2e-3
        np.testing.assert_allclose(c, oc, rtol=1e-3, atol=1e-12 * oc.max())

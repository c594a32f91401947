"""The two forms of the FP64 CSDA histories (one per warp in batches of up to 32
steps, one per thread): counts around a group and a warp, and geometries that
leave the batches at every point: no rock, less than one step of it, rock thick
and thin enough for every air step rule, level and downward lines, energies at
the ends of the table and a low source ceiling.

Against the oracle both are FP64 programs of up to 10^3 steps (rounding ~1e-12;
1e-9 and, for the derivative with its cancellations, 1e-8 as in the other FP64
comparisons).  The forms differ from one another by the rounding of the batches'
closed forms only: 1e-11, and the same number of steps."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

GEO = {"thick": (100.0, 2650.0, 45.0, (1.0, 100.0)), "thin": (5.0, 2650.0, 70.0, (0.5, 20.0)),
       "no rock": (0.0, 2650.0, 80.0, (0.2, 1e3)), "sliver": (1e-6, 1800.0, 30.0, (1e-3, 10.0)),
       "flat": (20.0, 2000.0, 3.0, (1.0, 1e4)), "level": (20.0, 2650.0, 0.0, (1.0, 100.0)),
       "down": (20.0, 2650.0, -30.0, (1.0, 100.0)), "ends": (50.0, 2650.0, 60.0, (1e-3, 9e8))}


@pytest.fixture(scope="module")
def setup(oracle):
    import dpgpu as dp
    orc = oracle.default_physics((oracle.STANDARD_ROCK, oracle.AIR))
    return dp, orc, dp.upload_physics([orc.table(0), orc.table(1)], ["StandardRock", "Air"])


def _samples(n, erange):
    rng = np.random.default_rng(n)
    E = np.exp(rng.uniform(*np.log(erange), n))
    return E, np.where(rng.random(n) > 0.5, 1.0, -1.0), rng.uniform(0.5, 2.0, n)


@pytest.mark.parametrize("n", [1, 33, 1217, 6001])
@pytest.mark.parametrize("which", list(GEO))
def test_histories_match_oracle(setup, oracle, which, n):
    dp, orc, phys = setup
    t, rho, el, erange = GEO[which]
    E, q, w = _samples(n, erange)
    if which == "ends":
        E[0] = 1e-3
    c, d = dp.csda_flux_samples(phys, E, q, w, rock_thickness=t, rock_density=rho, elevation=el)
    oc, od = oracle.backward_mc_csda(orc, 0, 1, t, rho, el, E, q, w)
    np.testing.assert_allclose(c, oc, rtol=1e-9, atol=0)
    np.testing.assert_allclose(d, od, rtol=1e-8, atol=1e-12 * np.abs(od).max())


@pytest.mark.parametrize("which", list(GEO))
@pytest.mark.parametrize("ceiling", [None, 30.0])
def test_forms_agree(setup, which, ceiling):
    """The same histories alone (by warp) and among 40000 (by thread where the
    rock is thin)."""
    dp, _, phys = setup
    t, rho, el, erange = GEO[which]
    E, q, w = _samples(200, erange)
    kw = dict(rock_thickness=t, rock_density=rho, elevation=el, source_energy_max=ceiling, steps=True)
    a = dp.csda_flux_samples(phys, E, q, w, **kw)
    b = dp.csda_flux_samples(phys, *(np.tile(x, 200) for x in (E, q, w)), **kw)
    np.testing.assert_array_equal(a[2], b[2][:200])
    for x, y in zip(a[:2], b[:2]):
        np.testing.assert_array_equal(y[:200], y[-200:])
        np.testing.assert_allclose(x, y[:200], rtol=1e-11, atol=1e-13 * np.abs(x).max())

"""How the stochastic kernels deal histories to their lanes: counts around one per
multiprocessor, one per warp, two per warp and all lanes, both precisions, longest
first and in index order.  A history draws from its own stream and its sums do not
depend on the histories beside it, so a run's histories are bitwise the first ones
of a longer run, and the order changes nothing."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def setting():
    import dpgpu as dp
    phys = dp.create_physics(materials=(dp.STANDARD_ROCK, dp.AIR, dp.WATER))
    return dp, phys


def _edges(precision, full):
    warps = 152 * (32 if precision == "mixed" else 8)
    n = [1, 31, 151, 152, 153, warps - 1, warps, warps + 1, 2 * warps + 1]
    return n + [32 * warps - 7, 32 * warps + 33] if full else n


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_histories_do_not_depend_on_their_number(setting, precision):
    dp, phys = setting
    rock, air = dp.MaterialMixture(phys, 1), dp.MaterialMixture(phys, 2)
    counts = _edges(precision, precision == "mixed")
    rng = np.random.default_rng(2)
    m = max(counts)
    E, q = np.exp(rng.uniform(0.0, np.log(1e3), m)), np.where(rng.random(m) > 0.5, 1.0, -1.0)
    geo = dict(thickness=rng.uniform(1.0, 8.0, m), density=rng.uniform(2000.0, 2800.0, m),
               elevation=rng.uniform(30.0, 90.0, m), primary_altitude=500.0)
    run = lambda n: dp.mc_histories(phys, rock, air, E[:n], q[:n], 2.0 * E[:n], seed=3, precision=precision,  # noqa: E731
                                    **{k: v[:n] if np.ndim(v) else v for k, v in geo.items()})
    ref = run(m)
    assert (ref[1] == 0).all() and (ref[2] > 0).all()
    for n in counts:
        for a, b in zip(run(n), ref):
            np.testing.assert_array_equal(a, b[:n])


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("n", [1, 153, 700, 6000])
def test_directions_do_not_depend_on_the_order(setting, precision, n):
    dp, phys = setting
    wf = np.linspace(0.0, 0.5, 9)
    cfg, site = dp.MaterialConfig(1, 3, 2, -1, 2650.0, 1000.0, 0.0, 0.0), dp.SiteConfig(963.0, 2000.0)
    seg = lambda *c: [dp.CellSegment(k, 1.5 * k) for k in c]  # noqa: E731
    P = dp.DirectionalPath
    paths = [P(0.0, 0.0, [], 0.0, 0.0, 0.0, 0.0, True), P(10.0, 0.0, seg(1, 2), 0.0, 0.0, 6.0, 50.0, True),
             P(30.0, 0.0, seg(2, 3), 0.0, 0.0, 1.0, 30.0, False), P(60.0, 0.0, seg(*range(1, 10)), 0.0, 0.0, 0.0, 90.0, True)]
    mats, dens = dp.build_cell_properties_for_mc(phys, np.zeros(9, bool), wf, cfg)
    batch = dp.DirBatch(phys, cfg, site, paths, mats, dens, None, n_samples=n, energy_min=0.1, energy_max=1e4)
    out, before = [], dp.get_mc_shape(phys.ctx, "dir", precision)
    try:
        for order in (0, 1):
            dp.set_mc_shape(phys.ctx, "dir", precision, order=order)
            out.append(batch.run(5, precision=precision, return_histories=True))
    finally:
        dp.set_mc_shape(phys.ctx, "dir", precision, order=before["order"])
    for k in out[0]:
        np.testing.assert_array_equal(out[0][k], out[1][k])

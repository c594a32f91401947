"""The FP64 water-fraction walk at the edges of its warps and of its air steps:
one sample, a full warp of samples and one more, paths of no cells and no rock
(energies from the foot of the grid enter the air, where the energy gain limits
the first steps), and steep and flat directions, against the oracle.

Both sides walk in FP64: 1e-10 on the flux and 1e-8 on the Jacobian, the
tolerances of the other FP64 comparisons of this model."""
import numpy as np
import pytest
from test_gpu_wtomo import _oracle, _per_cell_first, _samples, dp, orc_phys, phys  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_e", [1, 32, 33])
@pytest.mark.parametrize("corrected", [False, True])
def test_edges_match_oracle(dp, phys, oracle, orc_phys, n_e, corrected):  # noqa: F811
    rng = np.random.default_rng(n_e)
    wf = rng.uniform(0.0, 0.9, 9)
    seg = lambda *c: [dp.CellSegment(int(k), float(rng.uniform(1e-3, 60.0))) for k in c]  # noqa: E731
    P = dp.DirectionalPath
    paths = [P(0.0, 0.0, [], 0.0, 0.0, 0.0, 0.0, True), P(88.0, 0.0, [], 0.0, 0.0, 0.0, 2e4, True),
             P(10.0, 0.0, [], 0.0, 0.0, 120.0, 50.0, True), P(45.0, 0.0, seg(1), 0.0, 0.0, 0.0, 9.0, True),
             P(60.0, 0.0, seg(*range(1, 10), 4, 4), 0.0, 0.0, 5.0, 29999.9995, True),
             P(30.0, 0.0, seg(2, 3), 0.0, 0.0, 1.0, 30.0, False)]
    cfg, site = dp.MaterialConfig(1, 3, 2, -1, 2650.0, 1000.0, 0.0, 0.0), dp.SiteConfig(963.0, 3e4)
    samples = _samples(dp, n_e, 5)
    corr = [0] * 10
    try:
        if corrected:
            dp.set_csda_correction(enabled=True, kappa_strag=1.0, kappa_hard=7.0)
            corr = [1, 1.0, 7.0, 0.0, 0.0, 0.0, 0.0, 0, 0.0, 0.0]
        f, seg_ptr, cells, jac = dp.csda_flux_batch(phys, np.zeros(9, bool), cfg, site, paths, wf, samples)
    finally:
        dp.set_csda_correction(enabled=False)
    of, og = _oracle(oracle, orc_phys, wf, paths, samples, corr)
    assert np.isnan(f[-1]) and np.isfinite(f[:-1]).all()
    np.testing.assert_allclose(f[:-1], of[:-1], rtol=1e-10, atol=0)
    g = _per_cell_first(seg_ptr, cells, jac)
    np.testing.assert_allclose(g, og, rtol=1e-8, atol=1e-12 * np.abs(og).max())

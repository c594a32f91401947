"""The mixed-precision water-fraction walk, whose lanes step together: a batch of
samples against its samples one by one, over counts around a warp, samples that
leave the valid range in the rock or in the air beside ones that do not, segments of
no length and paths of no cells.

A sample's walk does not depend on its neighbours, so the two differ only by the
order of an FP64 sum: 2^-53 times 64 terms, 1e-14 of the sum of magnitudes."""
import numpy as np
import pytest
from test_gpu_wtomo import dp, orc_phys, phys  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_e", [2, 31, 33, 64])
def test_batch_is_its_samples(dp, phys, n_e):  # noqa: F811
    rng = np.random.default_rng(n_e)
    wf = rng.uniform(0.0, 0.9, 9)
    seg = lambda *c: [dp.CellSegment(int(k), float(rng.uniform(1e-3, 60.0))) for k in c]  # noqa: E731
    P = dp.DirectionalPath
    paths = [P(0.0, 0.0, [], 0.0, 0.0, 0.0, 0.0, True), P(88.0, 0.0, [], 0.0, 0.0, 0.0, 2e4, True),
             P(10.0, 0.0, seg(1) + [dp.CellSegment(2, 0.0)] + seg(3), 0.0, 0.0, 1200.0, 50.0, True),
             P(60.0, 0.0, seg(*range(1, 10), 4, 4), 0.0, 0.0, 5.0, 29999.9995, True)]
    cfg, site = dp.MaterialConfig(1, 3, 2, -1, 2650.0, 1000.0, 0.0, 0.0), dp.SiteConfig(963.0, 3e4)
    E = np.exp(rng.uniform(np.log(1e-3), np.log(1e6), n_e))
    E[::5] = 9.9e11
    E[1::7] = 1e-3
    E[4::5] = 9.99999e11  # some 10^6 GeV more end the walk: in the rock
    samples = [dp.EnergySample(e, (-1.0) ** k, 1.0) for k, e in enumerate(E)]
    run = lambda k: dp.csda_flux_batch(phys, np.zeros(9, bool), cfg, site, paths, wf,  # noqa: E731
                                       samples[k], precision="mixed")
    f, _, _, jac = run(slice(None))
    one = [run(slice(k, k + 1)) for k in range(n_e)]
    f1, j1 = np.array([o[0] for o in one]), np.array([o[3] for o in one])
    assert np.isfinite(f).all() and (f > 0.0).all() and (n_e == 2 or (f1 == 0.0).any())
    for a, b in ((f, f1), (jac, j1)):  # (the Jacobian from 1 MeV up is out of FP32's range in places)
        mean = b.sum(0) / n_e
        with np.errstate(invalid="ignore"):
            assert np.all((a == mean) | (np.abs(a - mean) <= 1e-13 * np.abs(b).sum(0) / n_e))

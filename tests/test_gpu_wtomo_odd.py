"""Odd input of the FP64 water-fraction walk: segments too short for a step (up to 1e-8 m,
or a NaN length on resident arrays) leave the flux alone whatever their cell holds."""
import numpy as np
import pytest
from test_gpu_wtomo import _samples, dp, orc_phys, phys  # noqa: F401

pytestmark = pytest.mark.gpu


def _batch(dp, phys, samples, lengths):  # noqa: F811
    segs = [[dp.CellSegment(1, 30.0), dp.CellSegment(2, 45.0)]]
    segs += [[segs[0][0], dp.CellSegment(5, x), segs[0][1]] for x in lengths]
    paths = [dp.DirectionalPath(30.0, 0.0, s, 0.0, 0.0, 4.0, 60.0, True) for s in segs]
    cfg, site = dp.MaterialConfig(1, 3, 2, -1, 2650.0, 1000.0, 0.0, 0.0), dp.SiteConfig(963.0, 3e4)
    return dp.CsdaBatch(phys, np.zeros(5, bool), cfg, site, paths, samples)


@pytest.mark.parametrize("w", [0.3, np.nan])
@pytest.mark.parametrize("resident", [False, True])
def test_segments_without_a_step(dp, phys, w, resident):  # noqa: F811
    b = _batch(dp, phys, _samples(dp, 40, 2), [0.0, 1e-8, 1e-300] + ([np.nan, -np.float64(np.nan)] if resident else []))
    if resident:
        b.to_device()
    flux, _ = b.run(np.array([0.1, 0.2, 0.0, 0.0, w]))
    assert flux[0] > 0
    np.testing.assert_array_equal(flux, np.full(len(flux), flux[0]))

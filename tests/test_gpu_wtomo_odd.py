"""Odd input of the FP64 water-fraction walk: segments too short for a step (up to 1e-8 m,
or a NaN length on resident arrays) leave the flux alone whatever their cell holds, and
an energy sample of zero walks from below the grid, where no derivative uses it."""
import numpy as np
import pytest
from test_gpu_wtomo import _oracle, _per_cell_first, _samples, dp, orc_phys, phys  # noqa: F401

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


def test_sample_of_zero_energy(dp, phys, oracle, orc_phys):  # noqa: F811
    """1e-10 on the flux, 1e-8 on the Jacobian, as the other FP64 walks."""
    samples = [dp.EnergySample(0.0, 1.0, 1.0), dp.EnergySample(3.0, -1.0, 1.0)]
    b = _batch(dp, phys, samples, [12.0])
    wf = np.array([0.1, 0.2, 0.0, 0.0, 0.6])
    segs = b.arrays["seg_ptr"]
    flux, jac = b.run(wf)
    paths = [dp.DirectionalPath(30.0, 0.0, [dp.CellSegment(int(b.arrays["seg_cell"][k]) + 1, float(b.arrays["seg_length"][k]))
                                            for k in range(segs[i], segs[i + 1])], 0.0, 0.0, 4.0, 60.0, True) for i in range(2)]
    of, og = _oracle(oracle, orc_phys, wf, paths, samples, [0] * 10)
    assert np.isfinite(og).all() and (of > 0).all()
    np.testing.assert_allclose(flux, of, rtol=1e-10, atol=0)
    g = _per_cell_first(segs, b.arrays["seg_cell"], jac)
    np.testing.assert_allclose(g, og, rtol=1e-8, atol=1e-12 * np.abs(og).max())


@pytest.mark.parametrize("e", [5e-324, 1e-310, 2.2250738585072014e-308, -5e-324, -1.0])
def test_sample_of_hardly_any_energy(dp, phys, e):  # noqa: F811
    """Subnormal and negative energies walk as zero does, from below the grid."""
    out = []
    for x in (e, 0.0 if e > -1.0 else -1.0 + 2.0 ** -52):
        b = _batch(dp, phys, [dp.EnergySample(x, 1.0, 1.0), dp.EnergySample(3.0, -1.0, 1.0)], [12.0])
        out.append(b.run(np.array([0.1, 0.2, 0.0, 0.0, 0.6])))
    assert np.isfinite(out[0][1]).all() and (out[0][0] > 0).all()
    for x, y in zip(*out):
        np.testing.assert_allclose(x, y, rtol=1e-12, atol=0)


def test_a_nan_length_spoils_the_jacobian(dp, phys):  # noqa: F811
    """On resident arrays, where no length is checked: no step, so the path's flux stands,
    but its whole Jacobian is NaN; the other paths keep theirs."""
    wf = np.array([0.1, 0.2, 0.0, 0.0, 0.3])
    good = _batch(dp, phys, _samples(dp, 40, 2), [5.0, 7.0]).to_device().run(wf)
    b = _batch(dp, phys, _samples(dp, 40, 2), [5.0, np.nan]).to_device()
    flux, jac = b.run(wf)
    p = b.arrays["seg_ptr"]
    np.testing.assert_array_equal(flux, [good[0][0], good[0][1], good[0][0]])
    np.testing.assert_array_equal(jac[:p[2]], good[1][:p[2]])
    assert np.isnan(jac[p[2]:p[3]]).all()

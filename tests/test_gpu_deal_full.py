"""The FP64 hand-out with full warps and past them, where lanes refill from the counter: a
run's histories are bitwise the first ones of a longer run, in both kernels and orders."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _lanes():
    import torch
    return 256 * torch.cuda.get_device_properties(0).multi_processor_count


@pytest.mark.parametrize("order", [0, 1])
def test_histories(order):
    import dpgpu as dp
    phys = dp.create_physics(materials=(dp.STANDARD_ROCK, dp.AIR, dp.WATER))
    rock, air = dp.MaterialMixture(phys, 1), dp.MaterialMixture(phys, 2)
    lanes, rng = _lanes(), np.random.default_rng(2)
    m = 2 * lanes + 33
    E, q = np.exp(rng.uniform(0.0, np.log(1e3), m)), np.where(rng.random(m) > 0.5, 1.0, -1.0)
    t = rng.uniform(0.5, 3.0, m)
    before = dp.get_mc_shape(phys.ctx, "mc", "fp64")
    try:
        dp.set_mc_shape(phys.ctx, "mc", "fp64", order=order)
        run = lambda n: dp.mc_histories(phys, rock, air, E[:n], q[:n], 2.0 * E[:n], seed=3, precision="fp64",  # noqa: E731
                                        thickness=t[:n], density=2650.0, elevation=70.0, primary_altitude=200.0)
        ref = run(m)
        assert (ref[1] == 0).all() and (ref[2] > 0).all()
        for n in (lanes - 7, lanes, lanes + 33):
            for a, b in zip(run(n), ref):
                np.testing.assert_array_equal(a, b[:n])
    finally:
        dp.set_mc_shape(phys.ctx, "mc", "fp64", order=before["order"])


def test_directions():
    """One direction of more samples than lanes: its first samples are those of a shorter run."""
    import dpgpu as dp
    phys = dp.create_physics(materials=(dp.STANDARD_ROCK, dp.AIR, dp.WATER))
    cfg, site = dp.MaterialConfig(1, 3, 2, -1, 2650.0, 1000.0, 0.0, 0.0), dp.SiteConfig(963.0, 1200.0)
    mats, dens = dp.build_cell_properties_for_mc(phys, np.zeros(2, bool), np.array([0.1, 0.3]), cfg)
    path = dp.DirectionalPath(20.0, 0.0, [dp.CellSegment(1, 1.5), dp.CellSegment(2, 1.0)], 0.0, 0.0, 2.0, 50.0, True)
    batch = lambda n: dp.DirBatch(phys, cfg, site, [path], mats, dens, None, n_samples=n, energy_min=0.5, energy_max=1e4)  # noqa: E731
    lanes = _lanes()
    run = lambda n: batch(n).run(5, precision="fp64", return_histories=True)  # noqa: E731
    ref = run(2 * lanes + 33)
    assert (ref["status"] == 0).all()
    for n in (lanes - 7, lanes + 33):
        out = run(n)
        for k in ("contrib", "status", "final"):
            np.testing.assert_array_equal(out[k], ref[k][:n])


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_few_histories_are_not_ordered(precision):
    """As many histories as multiprocessors or fewer: the launches of index order."""
    import dpgpu as dp
    import torch
    phys = dp.create_physics(materials=(dp.STANDARD_ROCK, dp.AIR, dp.WATER))
    cfg, site = dp.MaterialConfig(1, 3, 2, -1, 2650.0, 1000.0, 0.0, 0.0), dp.SiteConfig(963.0, 1200.0)
    mats, dens = dp.build_cell_properties_for_mc(phys, np.zeros(2, bool), np.array([0.1, 0.3]), cfg)
    path = dp.DirectionalPath(20.0, 0.0, [dp.CellSegment(1, 1.5), dp.CellSegment(2, 1.0)], 0.0, 0.0, 2.0, 50.0, True)
    sms, lib, before = torch.cuda.get_device_properties(0).multi_processor_count, dp.load(), dp.get_mc_shape(phys.ctx, "dir", precision)
    try:
        for n, more in ((1, False), (sms, False), (sms + 1, True)):
            batch = dp.DirBatch(phys, cfg, site, [path], mats, dens, None, n_samples=n, energy_min=0.5, energy_max=1e4)
            launches = []
            for order in (0, 1):
                dp.set_mc_shape(phys.ctx, "dir", precision, order=order)
                k = lib.dp_launch_count(phys.ctx.h)
                batch.run(5, precision=precision)
                launches.append(lib.dp_launch_count(phys.ctx.h) - k)
            assert (launches[0] > launches[1]) == more, (n, launches)
    finally:
        dp.set_mc_shape(phys.ctx, "dir", precision, order=before["order"])

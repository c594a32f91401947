"""Contexts in threads of their own, calling at once with launches of different shared
memory (ray lengths, grids, media): the results are those of the same calls alone, bit for
bit, and no launch fails."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _work(k, reps, out):
    import dpgpu as dp
    ctx = dp.Context(0)
    phys = dp.create_physics(materials=(dp.STANDARD_ROCK, dp.AIR, dp.WATER), n_energies=(200, 150, 600)[k], ctx=ctx)
    rng = np.random.default_rng(k)
    nx = (30, 12, 60)[k]
    grid = dp.VoxelGrid(nx, nx, 8, (-5.0 * nx, -5.0 * nx, 0.0), 10.0)
    rho = rng.uniform(1500.0, 3000.0, grid.ncell)
    rays = dp.make_rays(np.zeros((64, 3)), rng.uniform(0.0, 85.0, 64), rng.uniform(0.0, 360.0, 64))
    E = np.geomspace(1.0, 1e5, 20)
    rock = dp.MaterialMixture(phys, 1) if k else dp.MaterialMixture(phys, [1, 3, 2], [0.7, 0.25, 0.05])
    air = dp.MaterialMixture(phys, 2)
    for _ in range(reps):
        r = []
        for precision in ("fp64", "mixed"):
            r += dp.TomoModel(phys, grid, (E, np.ones(20), E), side_density=2500.0, precision=precision).vjp(rho, rays, np.ones(64))
            r += dp.mc_histories(phys, rock, air, E, np.ones(20), E, seed=2, precision=precision, thickness=5.0,
                                 density=2650.0, elevation=60.0, primary_altitude=200.0)
            r += dp.csda_flux_samples(phys, E, np.ones(20), E, rock_thickness=5.0, rock_density=2650.0, elevation=60.0,
                                      precision=precision)
        out.append([np.array(x) for x in r])


def test_threads_share_no_launch_settings():
    alone = [[] for _ in range(3)]
    for k in range(3):
        _work(k, 1, alone[k])
    got = [[] for _ in range(9)]
    threads = [threading.Thread(target=_work, args=(i % 3, 25, got[i])) for i in range(9)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for i, g in enumerate(got):
        assert len(g) == 25, i  # (a thread whose call failed has fewer)
        for r in g:
            for a, b in zip(r, alone[i % 3][0]):
                np.testing.assert_array_equal(a, b)

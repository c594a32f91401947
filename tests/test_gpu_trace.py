"""The ray march of the voxel tomography, three lanes per ray, against a
restatement of the reference's loop (examples/diff_flux_cube.jl:132-366): the same
cells and bitwise the same lengths, for odd origins and pitches, rays along axes,
from corners and faces, off the grid, downwards, of no length and with infinite
components, ray counts around a warp's ten, and scales that take the general march.
(No tolerance: every operation is a rounded FP64 one.)"""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def march(lo, pitch, n, o, u):
    hi = [lo[a] + n[a] * pitch[a] for a in range(3)]
    x, cells, lens, z_exit = list(o), [], [], o[2]
    for _ in range(1000):
        if any(x[a] < lo[a] or x[a] > hi[a] for a in range(3)):
            break
        i = [min(max(math.floor((x[a] - lo[a]) / pitch[a]) + 1, 1), n[a]) for a in range(3)]
        best, leaves = math.inf, True
        for a in range(3):
            if abs(u[a]) > 1e-10:
                up = u[a] > 0
                t = (lo[a] + (i[a] if up else i[a] - 1) * pitch[a] - x[a]) / u[a]
                if t > 1e-10 and t < best:
                    best, leaves = t, i[a] + 1 > n[a] if up else i[a] - 1 < 1
        if math.isinf(best):
            x = [x[a] + u[a] * 0.01 for a in range(3)]
            continue
        cells.append(i[0] - 1 + n[0] * (i[1] - 1 + n[1] * (i[2] - 1)))
        lens.append(best)
        x = [x[a] + u[a] * best for a in range(3)]
        z_exit = x[2]
        if leaves:
            break
    return cells, lens, z_exit < hi[2] - 2.220446049250313e-16


GRIDS = {"cube": ((-80.0, -80.0, 0.0), (10.0, 10.0, 10.0), (16, 16, 8)),
         "odd": ((-3.7, 12.3, -1.1), (0.1, 0.37, 1 / 3), (50, 21, 33)),
         "cell": ((0.0, 0.0, 0.0), (1.0, 2.0, 3.0), (1, 1, 1)),
         "large": ((-8e31, -8e31, 0.0), (1e31, 1e31, 1e31), (16, 16, 8))}


@pytest.mark.parametrize("count", [1, 10, 11, 29, 200])
@pytest.mark.parametrize("which", list(GRIDS))
def test_march_is_the_reference_march(which, count):
    import dpgpu as dp
    lo, pitch, n = GRIDS[which]
    rng = np.random.default_rng(count)
    size = np.array(n) * pitch
    rays = np.zeros((count, 7))
    rays[:, :3] = lo + rng.uniform(-0.02, 1.02, (count, 3)) * size
    face = rng.random((count, 3)) < 0.3  # on cell faces and corners
    on = lo + rng.integers(0, np.array(n) + 1, (count, 3)) * pitch
    rays[:, :3] = np.where(face, on, rays[:, :3])
    v = rng.normal(size=(count, 3))
    v[rng.random((count, 3)) < 0.15] = 0.0
    v /= np.maximum(np.linalg.norm(v, axis=1), 1e-300)[:, None]
    v[rng.random((count, 3)) < 0.02] = 1e-11
    if count > 20:
        v[3], v[7], v[11], v[12] = (0.0, 0.0, 0.0), (0.0, 0.0, 1.0), (0.3, 0.0, 4e30), (math.inf, 0.0, 0.1)
        v[13], v[14] = (1.0, 0.0, 0.0), (0.0, -1.0, 0.0)
        rays[13:15, :3] = np.array(lo) + 0.5 * np.array(pitch)
    rays[:, 3:6] = v
    rays[:, 6] = np.clip(np.abs(v[:, 2]), 0.0, 1.0)
    paths = dp.TomoPaths(dp.create_physics(), dp.VoxelGrid(*n, lo, pitch), rays, ([10.0], [0.0], [1.0]))
    rp, col, length = paths.csr()
    for r in range(count):
        cells, lens, side = march(lo, pitch, n, *rays[r, :6].reshape(2, 3).tolist())
        assert rp[r + 1] - rp[r] == len(cells) + side, r
        assert col[rp[r]:rp[r] + len(cells)].tolist() == cells, r
        assert length[rp[r]:rp[r] + len(cells)].tolist() == lens, r

"""The fused translation at pencil lengths around its batch (a pencil that ends
inside a batch, one that fills it, one cell more), with blocks that some cells
of a pencil lack and planes without a positive value (the remap is left out
there), against the oracle's trans_map_1d_amr.

Tolerance: face, reconstruction and integral differ from the exact mode's by a
few tens of single-precision roundings of at most the peak: below 1e-5 of it.
Block lists do not change."""
import numpy as np
import pytest

from vlasiator_b200.projects import maxwellian_cell

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim", [0, 1, 2])
@pytest.mark.parametrize("n", [1, 2, 3, 4, 5, 7, 8, 9, 11, 12, 13, 17])
def test_pencil_lengths(mesh, orc_sp, dim, n):
    from vlasiator_b200 import vlgpu
    grid = [2, 2, 2]
    grid[dim] = n
    k = int(np.prod(grid))
    rng = np.random.default_rng(10 * n + dim)
    gids, data = [], []
    for c in range(k):
        m = maxwellian_cell(mesh, 10 ** rng.uniform(5.5, 6.5), 2e5, rng.uniform(-2e5, 2e5, 3))
        keep = rng.uniform(size=m.n_blocks) > 0.2  # the others are missing
        d = m.data[keep].copy()
        d[rng.uniform(size=len(d)) < 0.1] = 0.0    # blocks of zeros
        d[rng.uniform(size=len(d)) < 0.05] *= -1e-6
        gids.append(m.gids[keep])
        data.append(d)
    dt = 0.7 * 3e5 / 1.2e6
    with vlgpu.Batch(mesh, k, 4 * sum(map(len, gids)) + 4096) as b:
        b.upload(gids, data)
        b.set_grid(grid, 3e5)
        b.translate(dim, dt)
        got = b.cells()
        b.sync()
    offs = np.concatenate([[0], np.cumsum([len(g) for g in gids])])
    want = orc_sp.translate(mesh, grid, offs, np.concatenate(gids), np.concatenate(data), dim, dt, 3e5)
    peak = max(float(d.max()) for d in data)
    for c in range(k):
        np.testing.assert_array_equal(got[c][0], gids[c])
        assert np.abs(got[c][1] - want[offs[c]:offs[c + 1]]).max() <= 1e-5 * peak


@pytest.mark.parametrize("dim", [0, 1, 2])
def test_planes_of_nan(mesh, dim):
    """A plane of NaN has no positive value, so the remap is left out there, also where every other value is positive;
    as the exact mode does it."""
    from vlasiator_b200 import vlgpu
    grid = [1, 1, 1]
    grid[dim] = n = 9
    gids = maxwellian_cell(mesh, 1e6, 2e5, (1e5, -2e5, 5e4)).gids
    rng = np.random.default_rng(dim)
    data = (1e-13 * rng.uniform(0.5, 1.0, (n, len(gids), 4, 4, 4))).astype(np.float32)  # [z][y][x]
    plane = [slice(None)] * 3
    plane[2 - dim] = 2
    data[(slice(None), slice(3, None, 5), *plane)] = np.nan
    data = data.reshape(n, len(gids), 64)
    got = {}
    for exact in (False, True):
        with vlgpu.Batch(mesh, n, 4 * n * len(gids) + 4096, exact=exact) as b:
            b.upload([gids] * n, list(data))
            b.set_grid(grid, 3e5)
            b.translate(dim, 0.7 * 3e5 / 1.2e6)
            got[exact] = np.stack([d for _, d in b.cells()])
            b.sync()
    assert np.isfinite(got[True]).all()
    assert np.abs(got[False] - got[True]).max() <= 1e-5 * 1e-13

"""A batch whose adjusted lists outgrow its capacity: the shortage is reported,
what follows stays inside the pools (in particular off the row of zeros behind
them, which stands for every block without data), and the batch is as good as
new after the next upload."""
import numpy as np
import pytest

from vlasiator_b200.projects import maxwellian_cell

pytestmark = pytest.mark.gpu

ENOMEM, CELL_NOMEM = 2, 4
CAPACITY = 1400


def _overflow(vl, mesh, b):
    """Blocks three apart, which fit; the adjustment wants the 27 blocks around each of them."""
    axis = np.arange(4, 60, 4)
    gids = np.sort(mesh.gid(*[q.ravel() for q in np.meshgrid(axis, axis, axis[:2])])).astype(np.uint32)
    n = len(gids)
    assert 3 * n <= CAPACITY < 3 * 27 * n
    b.upload([gids] * 3, [np.full((n, 64), 1e-13, np.float32)] * 3)
    b.adjust()
    with pytest.raises(vl.VlgpuError) as e:
        b.sync()
    assert e.value.code == ENOMEM and (b.status() & CELL_NOMEM).any()
    out_g, out_d = np.zeros(CAPACITY, np.uint32), np.zeros((CAPACITY, 64), np.float32)
    b.download_begin()  # makes the list that overflowed direct
    b.download_end(out_g, out_d)
    # the list asked for more than there is: no room for any block more
    with pytest.raises(vl.VlgpuError) as e:
        b.unpack_cells([1], [0], 0, 0)
    assert e.value.code == ENOMEM


def _advance(vl, mesh, before):
    """`before(batch)`, then every second block of a Maxwellian: the adjustment adds blocks without data, the sweeps
    read them."""
    cell = maxwellian_cell(mesh, 1e6, 4e5, (1e5, -2e5, 5e4))
    g, d = np.asarray(cell.gids)[::2], np.asarray(cell.data)[::2]
    with vl.Batch(mesh, 3, CAPACITY) as b:
        before(b)
        b.upload([g[:40], g[:0], g[40:90]], [d[:40], d[:0], d[40:90]])
        b.adjust()
        assert b.block_counts()[0] > 40 and b.block_counts()[2] > 50
        dv = float(mesh.dv[0])
        for dim in range(3):
            isect = np.zeros(4)
            isect[0], isect[1 + dim] = mesh.vmin[dim] + 0.3 * dv, dv
            b.map_1d(np.tile(isect, (3, 1)), dim)
        b.sync()
        assert not b.status().any()
        return b.cells()


def test_pools_after_an_overflowing_adjustment(mesh):
    from vlasiator_b200 import vlgpu
    clean = _advance(vlgpu, mesh, lambda b: None)
    for (g1, d1), (g2, d2) in zip(clean, _advance(vlgpu, mesh, lambda b: _overflow(vlgpu, mesh, b))):
        np.testing.assert_array_equal(g1, g2)
        assert np.array_equal(d1, d2)

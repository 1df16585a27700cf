"""Sweeps and adjustments use two blocks of counters in turn, each operation
leaving the other block zero.  A captured graph starts with the block it was
captured with; here it is replayed when the batch's turn is at the other one,
which a translation (it takes no turn) between sweeps brings about."""
import numpy as np
import pytest

from vlasiator_b200.mesh import CHARGE, MASS_PROTON
from vlasiator_b200.projects import sinewave_grid

pytestmark = pytest.mark.gpu

DIMS = (3, 2, 2)


def _run(mesh, graph):
    from vlasiator_b200 import vlgpu
    cells = sinewave_grid(DIMS, mesh)
    B = np.stack([c.B for c in cells])
    dt = 0.01 * 2 * np.pi * MASS_PROTON / (CHARGE * 5e-9)
    identity = np.tile([mesh.vmin[2], 0.0, 0.0, mesh.dv[2]], (len(cells), 1))
    with vlgpu.Batch(mesh, len(cells), 8 * sum(c.n_blocks for c in cells) + 65536) as b:
        b.upload([c.gids for c in cells], [c.data for c in cells])
        b.set_grid(DIMS, 3e5)
        b.accelerate(B, dt, 0)
        if graph:
            b.capture(0, "accel", [1, 2])
        # pools and lists are back where they were, the counters are not
        b.translate(0, 0.01)
        b.map_1d(identity, 2)
        b.adjust()
        b.adjust()
        b.accelerate_device(0)
        b.accelerate_device(0)
        if graph:
            for _ in range(2):
                b.replay(0)
        else:
            for _ in range(2):
                b.accelerate_device(1)
                b.accelerate_device(2)
        b.sync()
        assert not b.status().any()
        return b.cells()


def test_replay_at_the_other_turn(mesh):
    for (g1, d1), (g2, d2) in zip(_run(mesh, False), _run(mesh, True)):
        np.testing.assert_array_equal(g1, g2)
        assert np.array_equal(d1, d2)


def _vlasov(mesh, graph, odd):
    """Two Vlasov steps, captured or not; with `odd` after an odd number of translations since the capture."""
    from vlasiator_b200 import vlgpu
    cells = sinewave_grid(DIMS, mesh)
    B = np.stack([c.B for c in cells])
    identity = np.tile([mesh.vmin[2], 0.0, 0.0, mesh.dv[2]], (len(cells), 1))
    with vlgpu.Batch(mesh, len(cells), 8 * sum(c.n_blocks for c in cells) + 65536) as b:
        b.upload([c.gids for c in cells], [c.data for c in cells])
        b.set_grid(DIMS, 3e5)
        b.vlasov_step(B, 0.01, 0)
        if graph:
            b.capture(0, "vlasov", [1, 2], 0.01)
        if odd:
            b.translate(0, 0.01)
            b.map_1d(identity, 2)
            b.adjust()
            b.adjust()
        for _ in range(2):
            if graph:
                b.replay(0)
            else:
                b.vlasov_step_device(0.01, 1)
                b.vlasov_step_device(0.01, 2)
        b.sync()
        assert not b.status().any()
        return b.cells()


@pytest.mark.parametrize("odd", [False, True])
def test_vlasov_graph_at_either_turn(mesh, odd):
    for (g1, d1), (g2, d2) in zip(_vlasov(mesh, False, odd), _vlasov(mesh, True, odd)):
        np.testing.assert_array_equal(g1, g2)
        assert np.array_equal(d1, d2)


def test_replay_keeps_a_translations_report(mesh):
    """A translation that ran out of room is reported by the next sync, also past the replay of a graph that does not
    translate."""
    from vlasiator_b200 import vlgpu
    n = 16
    axis = np.arange(4, 60, 4)
    apart = np.sort(mesh.gid(*[q.ravel() for q in np.meshgrid(axis, axis, axis)])).astype(np.uint32)
    same = [apart[:4]] * n
    own = [apart[80 * c:80 * c + 80] for c in range(n)]  # every cell its own blocks: a pencil's union has all of them
    values = lambda lists: [np.full((len(g), 64), 1e-13, np.float32) for g in lists]  # noqa: E731
    B = np.tile([0.0, 0.0, 5e-9], (n, 1))
    dt = 0.001 * 2 * np.pi * MASS_PROTON / (CHARGE * 5e-9)
    capacity = 4096
    assert 80 * n * n > 4 * capacity  # the rows of the pencil's table
    with vlgpu.Batch(mesh, n, capacity) as b:
        b.set_grid((n, 1, 1), 3e5)
        b.upload(same, values(same))
        b.accelerate(B, dt, 0)
        b.sync()
        b.capture(0, "accel", [1, 2])
        b.upload(own, values(own))
        b.translate(0, 0.01)
        b.upload(same, values(same))
        b.adjust()
        b.accelerate_device(0)
        b.replay(0)
        with pytest.raises(vlgpu.VlgpuError) as e:
            b.sync()
        assert e.value.code == 2

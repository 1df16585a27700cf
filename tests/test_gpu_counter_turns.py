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

"""The kernels that take a cell per CTA (columnize, the adjustment's lists)
run with larger CTAs where the cells are few, and the adjustment's values are
summed in parts of 64 blocks (cells of up to 1024 blocks) or 128.  A cell's step must not depend on any of
that: the same cells alone, beside a few and beside many others come out
bit-identical, and equal to the oracle's adjustment and moments.

Sizes: no block, one block, the edges of a part of 64 (63 to 65, 127 to 129,
255 to 257 blocks), of the change to parts of 128 (1023 to 1025) and of a part
after it (1151 to 1153), more blocks than 64 parts of 128, and a cell whose
transverse plane exceeds the capped columnize launch (1024 entries)."""
import numpy as np
import pytest

from vlasiator_b200.mesh import CHARGE, MASS_PROTON
from vlasiator_b200.projects import maxwellian_cell

pytestmark = pytest.mark.gpu

COUNTS = (0, 1, 2, 63, 64, 65, 127, 128, 129, 255, 256, 257, 1023, 1024, 1025, 1151, 1152, 1153)


def _cells(mesh):
    base, more = (maxwellian_cell(mesh, 1e6, T, (1e5, -2e5, 5e4)) for T in (8e5, 2e6))
    assert len(more.gids) >= max(COUNTS)
    cells = [((base if n < 512 else more).gids[:n], (base if n < 512 else more).data[:n]) for n in COUNTS]
    hot = maxwellian_cell(mesh, 3e6, 1.2e7, (0.0, 3e5, 0.0))
    assert len(hot.gids) > 64 * 128
    cells.append((hot.gids, hot.data))
    # content at both ends of a long diagonal: a transverse box of 41 x 41 blocks
    far = np.sort(np.concatenate([mesh.gid(12 + 40 * k, 12 + 40 * k, 20 + np.arange(3)) for k in (0, 1)]))
    cells.append((far.astype(np.uint32), np.full((len(far), 64), 3e-14, np.float32)))
    return cells


def _run(vl, mesh, cells, copies):
    n = len(cells) * copies
    total = sum(len(g) for g, _ in cells) * copies
    with vl.Batch(mesh, n, 4 * total + 65536) as b:
        b.upload([cells[c % len(cells)][0] for c in range(n)], [cells[c % len(cells)][1] for c in range(n)])
        b.adjust()
        first = (b.cells()[-len(cells):], b.rho_loss()[-len(cells):].copy(), b.moments(second=True)[-len(cells):])
        b.upload([cells[c % len(cells)][0] for c in range(n)], [cells[c % len(cells)][1] for c in range(n)])
        B = np.tile([2e-9, -3e-9, 8e-9], (n, 1))
        dt = 0.01 * 2 * np.pi * MASS_PROTON / (CHARGE * np.linalg.norm(B[0]))
        for order in range(3):
            b.accelerate(B, dt, order)
        got = (b.cells()[-len(cells):], b.rho_loss()[-len(cells):].copy(), None)
        assert not (b.status() & ~np.uint32(1)).any()
        b.sync()
    return first, got


@pytest.fixture(scope="module")
def alone(mesh):
    from vlasiator_b200 import vlgpu
    return _run(vlgpu, mesh, _cells(mesh), 1)


def test_adjustment_against_oracle(alone, mesh, orc_sp):
    (got, loss, mom), _ = alone
    for c, (g, d) in enumerate(_cells(mesh)):
        if len(g) == 0:
            assert len(got[c][0]) == 0 and loss[c] == 0 and not mom[c].any()
            continue
        g2, d2, l2 = orc_sp.adjust(mesh, g, d, 1e-15)
        np.testing.assert_array_equal(got[c][0], g2)
        np.testing.assert_array_equal(got[c][1], d2)
        assert loss[c] == pytest.approx(l2, rel=1e-12, abs=1e-300)
        m = orc_sp.moments(mesh, g2, d2, MASS_PROTON, CHARGE)
        np.testing.assert_allclose(mom[c][:4], m[:4], rtol=1e-12, atol=1e-12 * np.abs(m[:4]).max())
        np.testing.assert_allclose(mom[c][9:15], m[9:15], rtol=0, atol=1e-9 * np.abs(m[9:15]).max())


@pytest.mark.parametrize("copies", [3, 20, 60])  # 60, 400 and 1200 cells: each CTA size
def test_same_in_every_batch_size(alone, mesh, copies):
    from vlasiator_b200 import vlgpu
    many = _run(vlgpu, mesh, _cells(mesh), copies)
    for a, b in zip(alone, many):
        for (g1, d1), (g2, d2) in zip(a[0], b[0]):
            np.testing.assert_array_equal(g1, g2)
            assert np.array_equal(d1, d2)
        np.testing.assert_array_equal(a[1], b[1])
        if a[2] is not None:
            np.testing.assert_array_equal(a[2], b[2])

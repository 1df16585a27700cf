"""The fused remap with two columns per lane (remap_pair_kernel) where its walk
branches: sets of one block, sets that do not fill a warp's four, columns with
gaps (also gaps of one block, and targets that two columns share), Lagrangian
cells wider and narrower than the mesh's (no edge, or several, in a source
cell), every sweep dimension.  Against the oracle's map_1d.

Tolerance: the edges are rounded as the reference rounds them, so the
difference is that of the reconstruction and of the running sums, a few tens
of single-precision roundings (6e-8) of at most the cell's peak: below 1e-5 of
the peak.  Block sets are equal."""
import numpy as np
import pytest

from vlasiator_b200.mesh import VelocityMesh

pytestmark = pytest.mark.gpu

MESH = VelocityMesh(vmin=(-2.4e6,) * 3, vmax=(2.4e6,) * 3, length=(40, 40, 40))


def _cell(rng, n_blocks, spread):
    """Blocks at random places of a box (so that columns have gaps), smooth times noisy values."""
    box = np.arange(spread ** 3)
    at = np.sort(rng.choice(box, size=min(n_blocks, len(box)), replace=False))
    x, y, z = at % spread, (at // spread) % spread, at // spread ** 2
    gids = np.sort(MESH.gid(x + 20 - spread // 2, y + 20 - spread // 2, z + 20 - spread // 2)).astype(np.uint32)
    data = (1e-13 * rng.uniform(0.0, 1.0, (len(gids), 64))).astype(np.float32)
    data[rng.uniform(size=data.shape) < 0.1] = 0.0
    return gids, data


@pytest.mark.parametrize("stretch", [0.45, 0.97, 1.0, 1.04, 2.3, 4.5])
@pytest.mark.parametrize("dim", [0, 1, 2])
def test_against_oracle(orc_sp, dim, stretch):
    from vlasiator_b200 import vlgpu
    rng = np.random.default_rng(100 * dim + int(10 * stretch))
    cells = [_cell(rng, n, s) for n, s in ((1, 1), (2, 3), (3, 2), (27, 3), (40, 6), (200, 8), (150, 10))]
    dv = float(MESH.dv[dim])
    isect = np.zeros((len(cells), 4))
    for c in range(len(cells)):
        shear = rng.uniform(-0.08, 0.08, 3) * dv
        shear[dim] = stretch * dv
        # the Lagrangian grid meets the mesh in the middle of both, so that
        # every target lies well inside the mesh
        isect[c, 0] = -80 * stretch * dv - 80 * (shear.sum() - shear[dim]) + rng.uniform(-2, 2) * dv
        isect[c, 1:] = shear
    with vlgpu.Batch(MESH, len(cells), 65536) as b:
        b.upload([g for g, _ in cells], [d for _, d in cells])
        b.map_1d(isect, dim)
        got, status = b.cells(), b.status()
    for c, (g, d) in enumerate(cells):
        assert status[c] == 0, f"cell {c}: status {status[c]}"
        g2, d2, _ = orc_sp.map_1d(MESH, g, d, isect[c], dim, 1e-15)
        o = np.argsort(g2)
        np.testing.assert_array_equal(got[c][0], g2[o])
        assert np.abs(got[c][1] - d2[o]).max() <= 1e-5 * max(d.max(), d2.max())


def test_more_sets_than_workers(orc_sp):
    """Sets beyond the warps' first ones come from the work counter: a batch with several times as many."""
    from vlasiator_b200 import vlgpu
    rng = np.random.default_rng(7)
    distinct = [_cell(rng, n, 8) for n in (5, 60, 180)]
    n = 700
    dv = float(MESH.dv[2])
    isect = np.tile([-80.3 * 1.01 * dv, 0.01 * dv, -0.01 * dv, 1.01 * dv], (n, 1))
    with vlgpu.Batch(MESH, n, 400000) as b:
        b.upload([distinct[c % 3][0] for c in range(n)], [distinct[c % 3][1] for c in range(n)])
        b.map_1d(isect, 2)
        got = b.cells()
        assert not b.status().any()
    for k, (g, d) in enumerate(distinct):
        g2, d2, _ = orc_sp.map_1d(MESH, g, d, isect[k], 2, 1e-15)
        o = np.argsort(g2)
        for c in range(k, n, 3):
            np.testing.assert_array_equal(got[c][0], g2[o])
            assert np.abs(got[c][1] - d2[o]).max() <= 1e-5 * d.max()


@pytest.mark.parametrize("recon", ["plm", "ppm"])
@pytest.mark.parametrize("bad", [np.nan, np.inf])
@pytest.mark.parametrize("dim", [0, 1, 2])
def test_what_is_not_finite_stays_where_it_is(orc_sp, dim, bad, recon):
    """Single values that are not finite reach the target cells that they overlap, and no others: their neighbours'
    reconstructions do without the faces they spoil.  Which cells those are the oracle says: a one among zeros is flat
    in its cell."""
    from vlasiator_b200 import vlgpu
    rng = np.random.default_rng(300 + dim)
    dv = float(MESH.dv[dim])
    cells, ones = [], []
    for n, spread in ((27, 3), (60, 6), (150, 10)):
        g, d = _cell(rng, n, spread)
        at = np.zeros(d.shape, bool)
        at[::3, rng.integers(0, 64)] = True  # in every third block: not two neighbours in a column
        ones.append(at.astype(np.float32))
        cells.append((g, np.where(at, np.float32(bad), d)))
    shear = np.array([0.03, -0.05, 0.02]) * dv
    shear[dim] = 1.02 * dv
    isect = np.array([-80 * 1.02 * dv - 80 * (shear.sum() - shear[dim]) + 0.4 * dv, *shear])
    with vlgpu.Batch(MESH, len(cells), 65536, recon=recon) as b:
        b.upload([g for g, _ in cells], [d for _, d in cells])
        b.map_1d(np.tile(isect, (len(cells), 1)), dim)
        got = b.cells()
        assert not b.status().any()
    for (g, _), at, (g2, d2) in zip(cells, ones, got):
        go, reached, _ = orc_sp.map_1d(MESH, g, at, isect, dim, 1e-15)
        o = np.argsort(go)
        np.testing.assert_array_equal(g2, go[o])
        assert np.isfinite(d2[reached[o] == 0.0]).all()
        assert not np.isfinite(d2[reached[o] > 1e-3]).any()

"""vlgpu_batch_pack_cells / _unpack_cells at the edges of their chunks and in
the states they meet: packing an adjusted (indirect) list without making it
direct, with blocks that have no data; replacing every cell, which leaves the
current state untouched until the block IDs are known to be good; replacing
some."""
import numpy as np
import pytest
import torch

from vlasiator_b200.projects import maxwellian_cell

pytestmark = pytest.mark.gpu

COUNTS = (0, 1, 63, 64, 65, 255, 256, 257, 600)


def _cells(mesh):
    c = maxwellian_cell(mesh, 1e6, 1e6, (1e5, -2e5, 5e4))
    assert len(c.gids) >= max(COUNTS)
    return [(c.gids[:n], c.data[:n]) for n in COUNTS]


def _packed(b, cells, capacity=20000):
    ids = torch.full((capacity,), -1, dtype=torch.int32, device="cuda")
    vals = torch.full((capacity, 64), -1.0, device="cuda")
    torch.cuda.synchronize()
    counts, used = b.pack_cells(np.asarray(cells, np.uint32), ids.data_ptr(), vals.data_ptr(), capacity)
    ids, vals = ids.cpu().numpy(), vals.cpu().numpy()
    assert (ids[used:] == -1).all() and (vals[used:] == -1).all()
    offs = np.concatenate([[0], np.cumsum(counts)]).astype(np.int64)
    return [(ids[offs[i]:offs[i + 1]].view(np.uint32), vals[offs[i]:offs[i + 1]]) for i in range(len(cells))]


def _same(a, b):
    for (g1, d1), (g2, d2) in zip(a, b):
        o1, o2 = np.argsort(g1), np.argsort(g2)
        np.testing.assert_array_equal(g1[o1], g2[o2])
        assert np.array_equal(d1[o1], d2[o2])


@pytest.fixture()
def batch(mesh):
    from vlasiator_b200 import vlgpu
    cells = _cells(mesh)
    with vlgpu.Batch(mesh, len(cells), 16384) as b:
        b.upload([g for g, _ in cells], [d for _, d in cells])
        yield b, cells


@pytest.mark.parametrize("adjusted", [False, True])
def test_pack(batch, adjusted):
    b, cells = batch
    if adjusted:
        b.adjust()
    every = list(range(len(cells)))
    got, again = _packed(b, every), _packed(b, every)
    _same(got, again)
    few = [7, 2, 2, 5]
    part = _packed(b, few)
    want = b.cells()  # (makes an adjusted state direct)
    _same(got, want)
    _same(part, [want[c] for c in few])
    if not adjusted:
        _same(got, cells)


@pytest.mark.parametrize("adjusted", [False, True])
def test_replace_all_and_some(batch, adjusted):
    from vlasiator_b200 import vlgpu
    b, cells = batch
    if adjusted:
        b.adjust()
    before = _packed(b, range(len(cells)))
    new = [(g[::-1].copy(), (2.0 * d[::-1]).copy()) for g, d in cells[::-1]]
    counts = [len(g) for g, _ in new]
    ids = torch.as_tensor(np.concatenate([g for g, _ in new]).view(np.int32).copy(), device="cuda")
    vals = torch.as_tensor(np.concatenate([d for _, d in new]), device="cuda")
    every = np.arange(len(cells), dtype=np.uint32)
    # a block ID outside the mesh: refused, nothing changed
    bad = ids.clone()
    bad[17] = 67 ** 3
    torch.cuda.synchronize()
    with pytest.raises(vlgpu.VlgpuError) as e:
        b.unpack_cells(every, counts, bad.data_ptr(), vals.data_ptr())
    assert e.value.code == 1
    _same(_packed(b, range(len(cells))), before)
    b.unpack_cells(every, counts, ids.data_ptr(), vals.data_ptr())
    _same(_packed(b, range(len(cells))), new)
    assert np.array_equal(b.block_counts(), counts)
    # some cells of what is there now
    b.unpack_cells([4, 1], [counts[0], counts[1]], ids.data_ptr(), vals.data_ptr())
    want = list(new)
    want[4], want[1] = new[0], new[1]
    _same(_packed(b, range(len(cells))), want)
    b.adjust()
    _same(b.cells(), _packed(b, range(len(cells))))


def test_no_room(mesh):
    """Replacing cells asks for room behind the rows in use, as it does when not every cell is replaced."""
    from vlasiator_b200 import vlgpu
    cells = _cells(mesh)
    total = sum(COUNTS)
    ids = torch.as_tensor(np.concatenate([g for g, _ in cells]).view(np.int32).copy(), device="cuda")
    vals = torch.as_tensor(np.concatenate([d for _, d in cells]), device="cuda")
    torch.cuda.synchronize()
    for room, fits in ((2 * total, True), (2 * total - 1, False)):
        with vlgpu.Batch(mesh, len(cells), room) as b:
            b.upload([g for g, _ in cells], [d for _, d in cells])
            every = np.arange(len(cells), dtype=np.uint32)
            if fits:
                b.unpack_cells(every, COUNTS, ids.data_ptr(), vals.data_ptr())
            else:
                with pytest.raises(vlgpu.VlgpuError) as e:
                    b.unpack_cells(every, COUNTS, ids.data_ptr(), vals.data_ptr())
                assert e.value.code == 2
            _same(b.cells(), cells)

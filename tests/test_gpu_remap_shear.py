"""The fused remap where the columns of one block face start many target cells
apart, up to and beyond what the ring of eight target blocks per set holds:
sweeps whose Lagrangian lines lean by several cells per transverse cell, as
a caller's own intersections or a rotation of 80 degrees and more in one step
give them.  A cell comes out right or reported by its status word.

PPM against the oracle's map_1d, PLM against the restatement below; block sets
from the oracle.  Tolerance as in test_gpu_remap_pair.py: the edges are rounded
as the reference rounds them, so the difference is that of the reconstruction
and of the running sums, a few tens of single-precision roundings (6e-8) of at
most the cell's peak: below 1e-5 of the peak."""
import os

import numpy as np
import pytest

from vlasiator_b200.mesh import VelocityMesh

MESH = VelocityMesh(vmin=(-5.76e6,) * 3, vmax=(5.76e6,) * 3, length=(96, 96, 96))
N_CELLS = 240
F = np.float32


def _cell(rng, dim, mild):
    """A few sets with columns of one to eight blocks, some with gaps, and a leaning sweep about the mesh's middle."""
    sizes = [int(rng.integers(1, 4)) for _ in range(3)]
    sizes[dim] = int(rng.integers(1, 9))
    xyz = np.stack([q.ravel() for q in np.meshgrid(*[np.arange(n) for n in sizes])], axis=1)
    xyz = xyz[rng.uniform(size=len(xyz)) < rng.choice([0.7, 1.0])]
    if len(xyz) == 0:
        xyz = np.zeros((1, 3), int)
    gids = np.sort(MESH.gid(*(xyz + 47).T)).astype(np.uint32)
    data = (1e-13 * rng.uniform(0.0, 1.0, (len(gids), 64))).astype(F)
    dv = float(MESH.dv[dim])
    stretch = rng.uniform(0.5, 3.0)
    # the sum of the transverse slopes, in target cells: the ring's limit lies between 8 and 10
    lean = rng.uniform(0.0, 2.0) if mild else rng.uniform(7.0, 10.0)
    part = rng.uniform(0.2, 0.8)
    shear = np.full(3, lean * part)
    shear[(dim + 1) % 3] = lean - lean * part
    shear = shear * rng.choice([-1, 1], 3) * stretch * dv
    shear[dim] = stretch * dv
    first = -192 * shear.sum() + rng.uniform(-2, 2) * dv
    return gids, data, np.array([first, *shear])


def _transverse(dim):
    """Strides in a block of the transverse cells i, j and of the sweep, and the mesh axes of the same."""
    return {0: ((16, 4, 1), (2, 1, 0)), 1: ((1, 16, 4), (0, 2, 1)), 2: ((1, 4, 16), (0, 1, 2))}[dim]


def plm_map_1d(mesh, gids, data, isect, dim):
    """One sweep with the linear reconstruction (superbee slopes): the target edges and the columns' target limits in
    the single precision of the reference (cpu_acc_map.cpp:307-338, 493-496), the values in 64 bits.  A dict of the
    blocks that receive something, by global ID."""
    (si, sj, sk), (ai, aj, ak) = _transverse(dim)
    dv, vmin = F(mesh.dv[dim]), F(mesh.vmin[dim])
    I0 = F(isect[0])
    di, dj, dk = F(isect[1 + ai]), F(isect[1 + aj]), F(isect[1 + ak])
    ijk = np.stack(mesh.indices(gids), axis=1)
    out = {}
    at = {tuple(q): n for n, q in enumerate(ijk)}
    lane = np.arange(16)
    off = (lane & 3) * si + (lane >> 2) * sj
    for a, b in sorted({(q[ai], q[aj]) for q in ijk}):
        ks = sorted(q[ak] for q in ijk if (q[ai], q[aj]) == (a, b))
        A, B = F(4 * a) + (lane & 3).astype(F), F(4 * b) + (lane >> 2).astype(F)
        im = F(I0 + A * di) + B * dj
        mx, mn = im.max(), im.min()
        for k0 in [k for k in ks if k - 1 not in ks]:
            k1 = k0
            while k1 + 1 in ks:
                k1 += 1
            lo = min(max(int((F(4 * k0) * dv + vmin - mx) / dk) // 4, 0), mesh.length[dim] - 1) * 4
            hi = min(max(int((F(4 * (k1 + 1)) * dv + vmin - mn) / dk) // 4, 0), mesh.length[dim] - 1) * 4 + 3
            col = []
            for k in range(k0, k1 + 1):
                q = [0, 0, 0]
                q[ai], q[aj], q[ak] = a, b, k
                col += [data[at[tuple(q)]][off + c * sk].astype(float) for c in range(4)]
            zero = np.zeros(16)
            col = np.stack([zero, *col, zero])
            right, left = col[2:] - col[1:-1], col[1:-1] - col[:-2]
            p, m = np.abs(right), np.abs(left)
            slope = np.where(right * left > 0, np.sign(right) * np.maximum(np.minimum(p, 2 * m), np.minimum(2 * p, m)), 0.0)
            v_l = F(F(4 * k0) * dv) + vmin
            for c in range(4 * (k1 + 1 - k0)):
                v0, d = col[c + 1], slope[c]
                g = np.floor((np.float64(v_l) - im) / dk).astype(int) - 1
                done = np.zeros(16)
                last = zero
                while (done < 1.0).any():
                    e = (g + 1).astype(F) * dk + im
                    u = np.clip((e - v_l).astype(F).astype(float) / float(dv), done, 1.0)
                    full = u * (v0 - 0.5 * d + 0.5 * u * d)
                    for l in np.flatnonzero(u > done):
                        t = min(max(int(g[l]), lo), hi)
                        q = [0, 0, 0]
                        q[ai], q[aj], q[ak] = a, b, t // 4
                        blk = out.setdefault(int(mesh.gid(*q)), np.zeros(64))
                        blk[off[l] + (t & 3) * sk] += full[l] - last[l]
                    done, last, g = u, full, g + 1
                v_l = F(v_l + dv)
    return out


def test_restatement_against_reference(mesh):
    """The PLM restatement of this file gives the fixtures of the reference's own PLM build."""
    z = np.load(os.path.join(os.path.dirname(__file__), "golden", "map1d_sp_plm.npz"))
    name = min((k.split("/")[0] for k in z.files), key=lambda n: len(z[f"{n}/gids_in"]))
    dim = [[0, 1, 2], [1, 2, 0], [2, 0, 1]][int(z[f"{name}/map_order"])][0]
    got = plm_map_1d(mesh, z[f"{name}/gids_in"], z[f"{name}/data_in"], z[f"{name}/isect"][4 * dim:4 * dim + 4], dim)
    rg, rd = z[f"{name}/sweep0_gids"], z[f"{name}/sweep0_data"]
    assert set(got) <= set(rg.tolist())
    dense = np.stack([got.get(int(g), np.zeros(64)) for g in rg])
    assert np.abs(dense - rd).max() <= 1e-5 * rd.max()


@pytest.mark.gpu
@pytest.mark.parametrize("recon", ["ppm", "plm"])
@pytest.mark.parametrize("dim", [0, 1, 2])
def test_right_or_reported(orc_sp, dim, recon):
    from vlasiator_b200 import vlgpu
    rng = np.random.default_rng(10 * dim + len(recon) + (recon == "plm"))
    cells = [_cell(rng, dim, mild=c % 8 == 0) for c in range(N_CELLS)]
    with vlgpu.Batch(MESH, len(cells), 400000, recon=recon) as b:
        b.upload([c[0] for c in cells], [c[1] for c in cells])
        b.map_1d(np.array([c[2] for c in cells]), dim)
        got, status = b.cells(), b.status()
        b.sync()
    clear, leaning = 0, 0
    for c, (g, d, isect) in enumerate(cells):
        if status[c]:
            assert not c % 8 == 0, f"cell {c} leans little and is reported: {status[c]}"
            continue
        clear += 1
        leaning += np.abs(np.delete(isect[1:], dim)).sum() > 8.4 * isect[1 + dim]
        g2, d2, _ = orc_sp.map_1d(MESH, g, d, isect, dim, 1e-15)
        o = np.argsort(g2)
        np.testing.assert_array_equal(got[c][0], g2[o])
        ref = d2[o]
        if recon == "plm":
            blocks = plm_map_1d(MESH, g, d, isect, dim)
            assert set(blocks) <= set(g2.tolist())
            ref = np.stack([blocks.get(int(q), np.zeros(64)) for q in g2[o]])
        err = np.abs(got[c][1] - ref).max() / max(d.max(), ref.max())
        assert err <= 1e-5, f"cell {c}: {err:.2e} of the peak, {isect[1:] / isect[1 + dim]}"
    # the test reaches both sides of the ring's limit
    assert clear >= len(cells) // 3 and leaning >= len(cells) // 20 and clear < len(cells)


@pytest.mark.gpu
@pytest.mark.parametrize("recon", ["ppm", "plm"])
@pytest.mark.parametrize("cells_off", [1000, 2 ** 20, 2 ** 21 + 190, 2 ** 22 + 190, 3e9])
def test_targets_far_above_are_reported(cells_off, recon):
    """A column that starts many target cells above the mesh is reported, also where the number of cells times the
    ring's slot size exceeds 32 bits and where the number itself does."""
    from vlasiator_b200 import vlgpu
    dv = float(MESH.dv[2])
    gids = np.sort(MESH.gid(47, 47, np.arange(46, 49))).astype(np.uint32)
    data = np.full((3, 64), 1e-13, F)
    # the first source cell lies cells_off target cells above the one with index zero
    isect = np.array([[MESH.vmin[2] + 4 * 46 * dv - cells_off * dv, 0.0, 0.0, dv]])
    with vlgpu.Batch(MESH, 1, 4096, recon=recon) as b:
        b.upload([gids], [data])
        b.map_1d(isect, 2)
        assert b.status()[0] == 3  # at the wall, and out of the ring's range
        b.sync()

"""The work that programs have this library do, as cases to be timed and compared.

Every case goes through the public entry points: ``vlgpu.Batch``, the C
function ``vlgpu_map_1d_noalloc`` and ``serve.Server``.  The velocity
distributions are those of the benchmark workloads (drifting Maxwellians with
n and T log-uniform, bi-Maxwellians of a given block count, the periodic
sine-wave grid), made on the GPU from the seed.

A batch's VDF lives on the device, so a pass puts the inputs into the batch
with ``unpack_cells`` (as a rank does with the cells it receives), advances
them, and takes the result out with ``pack_cells``; the timed work starts from
the same VDF each time.  (A translation keeps its block sets, so that case
goes on from where the last pass ended, as a program's time loop does.)
Results whose block sets depend on the values (a block is kept if some value
reaches the sparsity threshold, so a change of rounding can move a block at
the threshold) come as one dense velocity box per cell where there are many
cells; the others come as the packed block lists, zeros behind the last.  The
densities and temperatures belong to the case, so that its size is the same
for every seed; drifts, fields, axes and phases come from the seed.

``exact`` restates the same mathematics densely in 64 bits with torch.
"""
from __future__ import annotations

import ctypes
import math

import numpy as np
import torch

from vlasiator_b200 import serve, vlgpu
from vlasiator_b200.mesh import VelocityMesh

K_B, CHARGE, MASS = 1.3806503e-23, 1.60217653e-19, 1.67262158e-27
BLOCK = 1.2e5     # velocity block size, m/s: 4 cells of 30 km/s
MIN_VALUE = 1e-15
ROTATION = 0.01   # gyroperiods a step advances
DX = 3.0e5        # spatial cell size, m
DEV = "cuda"
STEPS = 6         # acceleration steps of a "step" pass: each dimension order twice
VLASOV_STEPS = 4  # whole Vlasov steps of a "vlasov" pass


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------
def listed():
    return [
        # one spatial cell per call from a host code's own device buffers, the
        # three dimensions in turn: the latency of the per-cell drop-in
        {"name": "call_small_cell", "kind": "call", "dist": "one", "cells": 1, "blocks": 0, "mesh_len": 67},
        # the same for a hot cell (the upper sizes of the serving stream)
        {"name": "call_large_cell", "kind": "call", "dist": "bimax", "cells": 1, "blocks": 15000, "mesh_len": 67},
        # the three sweeps of cpu_accelerate_cell with the reference
        # Makefile's default reconstruction
        {"name": "sweeps_pqm", "kind": "sweeps", "dist": "drift", "cells": 256, "blocks": 0, "mesh_len": 67,
         "recon": "pqm", "exact": False, "order": 0},
        # the bit-exact mode, as verification runs use it
        {"name": "sweeps_exact", "kind": "sweeps", "dist": "drift", "cells": 200, "blocks": 0, "mesh_len": 67,
         "recon": "ppm", "exact": True, "order": 1},
        # the single-cell gyration test: full acceleration steps of one cell
        {"name": "step_one_cell", "kind": "step", "dist": "one", "cells": 1, "blocks": 0, "mesh_len": 67},
        # a few large bi-Maxwellian cells in flight, as in the serving engine's batch
        {"name": "step_large_cells", "kind": "step", "dist": "bimax", "cells": 13, "blocks": 12000, "mesh_len": 67},
        # the batched-acceleration workload of the benchmark
        {"name": "step_batch", "kind": "step", "dist": "drift", "cells": 4096, "blocks": 0, "mesh_len": 67},
        # block adjustment and the moments with the pressure, as at start-up,
        # restart and output
        {"name": "adjust_moments", "kind": "adjust", "dist": "drift", "cells": 1024, "blocks": 0, "mesh_len": 67},
        # spatial translation along z, x, y of an uneven grid
        {"name": "translate_grid", "kind": "translate", "dist": "grid", "nx": 21, "ny": 9, "nz": 7, "mesh_len": 67,
         "exact": False},
        # whole Vlasov steps of a small grid: one rank's share of a coarse run
        {"name": "vlasov_small", "kind": "vlasov", "dist": "grid", "nx": 6, "ny": 5, "nz": 4, "mesh_len": 67},
        # whole Vlasov steps of the benchmark's sine-wave grid, halved along each axis
        {"name": "vlasov_grid", "kind": "vlasov", "dist": "grid", "nx": 32, "ny": 32, "nz": 8, "mesh_len": 67},
        # requests from host memory through the serving engine and back
        {"name": "serve_requests", "kind": "serve", "dist": "bimax", "cells": 12, "blocks": 3000, "mesh_len": 67},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["call", "sweeps", "sweeps", "step", "step", "step", "adjust", "translate", "vlasov", "vlasov",
                       "serve"])
    c = {"kind": kind}
    if kind == "call":
        c.update(dist="bimax", cells=1, blocks=_log(rng, 300, 15000), mesh_len=rng.randint(62, 96))
    elif kind == "sweeps":
        c.update(dist="drift", cells=_log(rng, 3, 512), blocks=0, mesh_len=rng.randint(62, 96),
                 recon=rng.choice(["plm", "ppm", "ppm", "pqm"]), exact=False, order=rng.randint(0, 2))
        c["exact"] = c["recon"] == "ppm" and rng.random() < 0.5
    elif kind == "step":
        if rng.random() < 0.4:
            c.update(dist="bimax", cells=_log(rng, 1, 40), blocks=_log(rng, 500, 12000), mesh_len=rng.randint(64, 80))
        else:
            c.update(dist="drift", cells=_log(rng, 2, 3000), blocks=0, mesh_len=rng.randint(62, 96))
    elif kind == "adjust":
        c.update(dist="drift", cells=_log(rng, 2, 2500), blocks=0, mesh_len=rng.randint(62, 96))
    elif kind in ("translate", "vlasov"):
        big = 40 if kind == "translate" else 24
        c.update(dist="grid", nx=_log(rng, 4, big), ny=_log(rng, 3, 16), nz=_log(rng, 3, 9),
                 mesh_len=rng.randint(62, 73))
        if kind == "translate":
            c["exact"] = rng.random() < 0.25
    else:
        c.update(dist="bimax", cells=_log(rng, 2, 16), blocks=_log(rng, 500, 4000), mesh_len=rng.randint(64, 80))
    return c


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _mesh(case):
    h = 0.5 * BLOCK * case["mesh_len"]
    return VelocityMesh(vmin=(-h,) * 3, vmax=(h,) * 3, length=(case["mesh_len"],) * 3)


def _directions(rng, n):
    d = rng.normal(size=(n, 3))
    return d / np.linalg.norm(d, axis=1, keepdims=True)


def _n_cells(case):
    return case["nx"] * case["ny"] * case["nz"] if case["dist"] == "grid" else case["cells"]


def _sizes(case):
    """Density and temperatures of every cell (of the grid: their means)."""
    k = _n_cells(case)
    rng = np.random.default_rng([k, case["mesh_len"], case.get("blocks", 0)])
    if case["dist"] == "drift":
        return 10.0 ** rng.uniform(5.0, 7.0, k), np.repeat((10.0 ** rng.uniform(5.0, 7.0, k))[:, None], 3, axis=1)
    if case["dist"] == "bimax":
        ratio = rng.uniform(0.5, 2.0, k)
        want = np.clip(case["blocks"] * np.exp(0.5 * rng.normal(size=k)), 200.0, 1.3 * case["blocks"])
        Tp = np.array([_temperature(w, r) for w, r in zip(want, ratio)])
        return np.full(k, 1e6), np.stack([Tp, Tp, ratio * Tp], axis=1)
    return np.full(k, 1e6), np.full((k, 3), 5e5 if case["dist"] == "one" else 1e6)


def _rows(case, wider):
    """Blocks that hold every cell's distribution `wider` blocks wider on each side."""
    n, T = _sizes(case)
    if case["dist"] == "grid":
        n, T = 1.1 * n, 1.05 * T
    return int(_estimate(n, T, 1.85 + wider).sum()) + 1024


def _plasma(case, seed):
    """Per cell: density, temperatures along three axes and those axes, bulk velocity, magnetic field."""
    rng = np.random.default_rng([seed, 77])
    k = _n_cells(case)
    dist = case["dist"]
    n, T = _sizes(case)
    R = np.broadcast_to(np.eye(3), (k, 3, 3)).copy()
    B = _directions(rng, k) * rng.uniform(5e-9, 50e-9, (k, 1))
    if dist == "drift":
        V = _directions(rng, k) * rng.uniform(0.0, 8.0e5, (k, 1))
    elif dist == "one":  # the gyrating Maxwellian of the single-cell test, at a seeded drift
        V = _directions(rng, k) * 1e5
        B = np.broadcast_to(np.array([0.0, 0.0, 1e-8]), (k, 3)).copy()
    elif dist == "bimax":
        V = _directions(rng, k) * rng.uniform(0.0, 6.0e5, (k, 1))
        b = B / np.linalg.norm(B, axis=1, keepdims=True)
        e1 = np.cross(b, np.where(np.abs(b[:, :1]) < 0.9, [[1.0, 0.0, 0.0]], [[0.0, 1.0, 0.0]]))
        e1 /= np.linalg.norm(e1, axis=1, keepdims=True)
        R = np.stack([e1, np.cross(b, e1), b], axis=1)
    else:  # a smooth wave through a periodic grid, cells x fastest
        nx, ny, nz = case["nx"], case["ny"], case["nz"]
        c = np.arange(k)
        ph = 2.0 * np.pi * (np.stack([(c % nx) / nx, (c // nx) % ny / ny, c // (nx * ny) / nz], axis=1)
                            + rng.uniform(size=3))
        n = n * (1.0 + 0.5 * np.sin(ph[:, 0])) * (1.0 + 0.1 * np.sin(ph[:, 1]))
        T = T * (1.0 + 0.1 * np.sin(ph[:, 2]))[:, None]
        V = np.array([4e5, 0.0, 0.0]) + 3e4 * np.sin(ph)
        B = np.broadcast_to(np.array([0.0, 0.0, 5e-9]), (k, 3)) + 1e-9 * np.sin(ph)
    return n, T, R, V, B


def _radius(n, T):
    """Largest speed (m/s), from the bulk, at which the density reaches the threshold."""
    peak = n * (MASS / (2.0 * np.pi * K_B)) ** 1.5 / np.sqrt(np.prod(T, axis=-1))
    return np.sqrt(2.0 * K_B * np.max(T, axis=-1) / MASS * np.log(np.maximum(peak / MIN_VALUE, 1.0)))


def _estimate(n, T, halo=1.85):
    """Blocks of the pruned Maxwellian: the ellipsoid above the threshold and its halo."""
    peak = n * (MASS / (2.0 * np.pi * K_B)) ** 1.5 / np.sqrt(np.prod(T, axis=-1))
    lg = np.log(np.maximum(peak / MIN_VALUE, 1.0))[..., None]
    return 4.0 / 3.0 * np.pi * np.prod(np.sqrt(2.0 * K_B * T / MASS * lg) / BLOCK + halo, axis=-1)


def _temperature(blocks, ratio):
    """Perpendicular temperature of the bi-Maxwellian with about `blocks` blocks."""
    lo, hi = 1e3, 1e8
    for _ in range(60):
        mid = math.sqrt(lo * hi)
        if _estimate(1e6, np.array([mid, mid, ratio * mid])) < blocks:
            lo = mid
        else:
            hi = mid
    return math.sqrt(lo * hi)


def _vdf(case, plasma):
    """(counts, IDs, values) of every cell's distribution sampled at the cell
    centres and pruned as the first block adjustment prunes it: the blocks
    with a value at the threshold and their neighbours, ascending ID."""
    n, T, R, V, _ = plasma
    L = case["mesh_len"]
    half = 0.5 * BLOCK * L
    k = len(n)
    rad = _radius(n, T)[:, None]
    lo = np.clip(np.floor((V - rad + half) / BLOCK).astype(int) - 1, 0, L - 1)
    hi = np.clip(np.floor((V + rad + half) / BLOCK).astype(int) + 1, 0, L - 1)
    size = (hi - lo + 1).max(axis=1)
    M = np.einsum("cai,ca,caj->cij", R, 1.0 / T, R) * (MASS / (2.0 * K_B))
    amp = n * (MASS / (2.0 * np.pi * K_B)) ** 1.5 / np.sqrt(np.prod(T, axis=1))
    by_size = np.argsort(size, kind="stable")
    cells, ids, vals = [], [], []
    a = 0
    while a < k:
        b = a + 1
        while b < k and (b + 1 - a) * int(size[by_size[b]]) ** 3 * 64 <= 1 << 24:
            b += 1
        sel = by_size[a:b]
        s = int(size[sel].max())
        t = lambda x: torch.as_tensor(np.ascontiguousarray(x), dtype=torch.float64, device=DEV)  # noqa: E731
        tl, th = torch.as_tensor(lo[sel], device=DEV), torch.as_tensor(hi[sel], device=DEV)
        ar = torch.arange(s, device=DEV)
        blk = tl[:, :, None] + ar                                    # cells, axis, block
        ok = blk <= th[:, :, None]
        ctr = -half + blk[..., None] * BLOCK + (torch.arange(4, device=DEV, dtype=torch.float64) + 0.5) * (BLOCK / 4)
        u = ctr - t(V[sel])[:, :, None, None]                        # cells, axis, block, cell of block
        C = len(sel)
        ux = u[:, 0].reshape(C, 1, 1, s, 1, 1, 4)
        uy = u[:, 1].reshape(C, 1, s, 1, 1, 4, 1)
        uz = u[:, 2].reshape(C, s, 1, 1, 4, 1, 1)
        m = t(M[sel]).reshape(C, 3, 3, 1, 1, 1, 1, 1, 1)
        q = ux * (m[:, 0, 0] * ux + 2.0 * (m[:, 0, 1] * uy + m[:, 0, 2] * uz)) \
            + (uy * (m[:, 1, 1] * uy + 2.0 * m[:, 1, 2] * uz) + m[:, 2, 2] * uz * uz)
        f = (t(amp[sel]).reshape(C, 1, 1, 1, 1, 1, 1) * torch.exp(-q)).to(torch.float32).reshape(C, s, s, s, 64)
        inside = ok[:, 2, :, None, None] & ok[:, 1, None, :, None] & ok[:, 0, None, None, :]
        content = (f >= MIN_VALUE).any(dim=-1) & inside
        keep = torch.nn.functional.max_pool3d(content.to(torch.float32)[:, None], 3, 1, 1)[:, 0].bool() & inside
        at = keep.nonzero()
        c = at[:, 0]
        gid = (tl[c, 0] + at[:, 3]) + L * ((tl[c, 1] + at[:, 2]) + L * (tl[c, 2] + at[:, 1]))
        cells.append(torch.as_tensor(sel, device=DEV)[c])
        ids.append(gid.to(torch.int32))
        vals.append(f[keep])
        a = b
    cell = torch.cat(cells)
    order = torch.argsort(cell, stable=True)
    counts = torch.bincount(cell, minlength=k).cpu().numpy().astype(np.uint32)
    ids = torch.cat(ids)[order]
    vals = torch.cat(vals)
    return counts, ids, vals[order].contiguous()


def _step_dt(B):
    return ROTATION * 2.0 * np.pi * MASS / (CHARGE * np.linalg.norm(B, axis=1))


def _rotation(B, dt):
    """The gyration over dt about B: rotation matrices."""
    b = np.linalg.norm(B, axis=1)
    u = B / b[:, None]
    ang = -dt * CHARGE * b / MASS
    s, c = np.sin(ang)[:, None, None], np.cos(ang)[:, None, None]
    K = np.zeros((len(B), 3, 3))
    K[:, 0, 1], K[:, 0, 2], K[:, 1, 2] = -u[:, 2], u[:, 1], -u[:, 0]
    K -= K.transpose(0, 2, 1)
    return c * np.eye(3) + s * K + (1.0 - c) * u[:, :, None] * u[:, None, :]


def _intersections(case, B, V, dt, order):
    """Per cell 12 numbers (x, y, z; intersection, di, dj, dk): where the lines
    of each of the three sweeps meet the planes of the grid that the gyration
    about V carries onto the mesh."""
    half, dv = 0.5 * BLOCK * case["mesh_len"], BLOCK / 4
    L = _rotation(B, dt).transpose(0, 2, 1)       # the way back
    t = V - np.einsum("cij,cj->ci", L, V)
    back = lambda p: np.einsum("cij,cj->ci", L, np.broadcast_to(p, V.shape)) + t  # noqa: E731
    e = np.eye(3)
    mid = np.full(3, -half + 0.5 * dv)
    meet = lambda p, d, q, nrm: p + (np.einsum("ci,ci->c", nrm, q - p)  # noqa: E731
                                     / np.einsum("ci,ci->c", nrm, d))[:, None] * d
    full = lambda v: np.broadcast_to(v, V.shape)  # noqa: E731
    out = np.zeros((len(V), 3, 4))
    for which in range(3):
        d = (order + which) % 3
        n = (d + 1) % 3
        base = np.where(np.arange(3) == d, -half, mid)
        pts = []
        for s in [np.zeros(3)] + [dv * e[a] for a in range(3)]:
            along = s[d] * e[d]
            if which == 0:    # mesh lines along d, planes carried back
                pts.append(meet(full(np.where(np.arange(3) == d, 0.0, mid) + s - along), full(e[d]),
                                back(-half * e[d] + along), L[:, :, d]))
            elif which == 1:  # lines along n carried back, mesh planes normal to n
                pts.append(meet(back(base + s - s[n] * e[n]), L[:, :, n], full((mid[n] + s[n]) * e[n]), full(e[n])))
            else:             # points carried back
                pts.append(back(base + s))
        p = np.stack([q[:, d] for q in pts], axis=1)
        out[:, d, 0] = p[:, 0]
        out[:, d, 1:] = p[:, 1:] - p[:, :1]
    return out.reshape(len(V), 12)


def _boxes(case, V):
    """Per cell, the first block and the size (x, y, z) of a box around its distribution; the size does not
    depend on the seed, and a box may reach beyond the mesh."""
    n, T = _sizes(case)
    if case["dist"] == "grid":
        n, T = 1.65 * n, 1.1 * T
    r = np.ceil(_radius(n, T) / BLOCK).astype(int)
    lo = np.floor((V + 0.5 * BLOCK * case["mesh_len"]) / BLOCK).astype(int) - r[:, None] - 2
    return lo, np.repeat(2 * r[:, None] + 5, 3, axis=1)


class _State:
    pass


DENSE_FROM = 8  # cells from which results that depend on the threshold come in dense boxes


def prepare(case, seed):
    s = _State()
    s.case = case
    kind = case["kind"]
    plasma = _plasma(case, seed)
    s.V, s.B = plasma[3], plasma[4]
    s.dt = _step_dt(s.B)
    s.counts, s.ids, s.vals = _vdf(case, plasma)
    s.mesh = _mesh(case)
    total, k = int(s.counts.sum()), len(s.counts)
    if kind == "call":
        s.isect = _intersections(case, s.B, s.V, s.dt, 0).reshape(k, 3, 4)
        room = min(65536, _rows(case, 2.5))
        s.out = [[torch.zeros(room, dtype=torch.int32, device=DEV), torch.zeros(room, 64, device=DEV), 0]
                 for _ in range(3)]
        s.lib = vlgpu.load()
        s.cmesh = vlgpu.CMeshT()
        for d in range(3):
            s.cmesh.vmin[d], s.cmesh.vmax[d], s.cmesh.len[d] = s.mesh.vmin[d], s.mesh.vmax[d], s.mesh.length[d]
        s.params = vlgpu.make_params(min_value=MIN_VALUE)
        s.offsets = np.concatenate([[0], np.cumsum(s.counts)]).astype(np.uint64)
        return s
    offsets = np.concatenate([[0], np.cumsum(s.counts)]).astype(np.int64)
    if kind == "serve":
        ids, vals = s.ids.cpu().numpy().view(np.uint32), s.vals.cpu().numpy()
        s.requests = [(ids[offsets[c]:offsets[c + 1]].copy(), vals[offsets[c]:offsets[c + 1]].copy(), s.B[c],
                       float(s.dt[c]), 1 + (5 * c + 2) % 6) for c in range(k)]
        rows = _rows(case, 1.0)
        s.host = [np.zeros(rows, np.int32), np.zeros((rows, 64), np.float32)]
        s.server = serve.Server(s.mesh, k, 585 * (8 * total + 65536))
        return s
    room = 4 * total + 65536
    s.batch = vlgpu.Batch(s.mesh, k, room, exact=False)
    if kind == "sweeps":
        s.batch.set_reconstruction(case["recon"])
        s.batch.set_exact(case["exact"])
        s.isect = _intersections(case, s.B, s.V, s.dt, case["order"])
    if kind in ("translate", "vlasov"):
        s.batch.set_grid((case["nx"], case["ny"], case["nz"]), DX)
        s.step = _grid_dt(case)
        if kind == "translate":
            s.batch.set_exact(case["exact"])
    s.batch.upload_packed(offsets, s.ids.cpu().numpy().view(np.uint32), s.vals.cpu().numpy())
    s.cells = np.arange(k, dtype=np.uint32)
    rows = _rows(case, 2.5 if kind == "sweeps" else 1.0)
    s.out = [torch.zeros(rows, dtype=torch.int32, device=DEV), torch.zeros(rows, 64, device=DEV), 0]
    s.dense = None
    if kind in ("step", "vlasov") and k >= DENSE_FROM:
        lo, size = _boxes(case, s.V)
        s.lo, s.size = torch.as_tensor(lo, device=DEV), torch.as_tensor(size, device=DEV)
        s.first = torch.cumsum(s.size.prod(dim=1), 0) - s.size.prod(dim=1)
        s.rows = int(s.size.prod(dim=1).sum())
        s.dense = torch.zeros(s.rows + 1, 64, device=DEV)
        s.filled = None
    torch.cuda.synchronize()
    return s


def _grid_dt(case):
    """0.8 of the time in which the fastest blocks cross a cell."""
    return 0.8 * DX / (4.0e5 + 9.0e5)


def _record(m):
    """The moment record by quantity."""
    return {"n": m[:, 0], "nV": m[:, 1:4], "rhom": m[:, 4], "V": m[:, 5:8], "rhoq": m[:, 8], "P": m[:, 9:15],
            "sum": m[:, 15]}


def _filled(out, used):
    """The buffers of block IDs and values, `used` rows of them written; out[2] remembers the rows of the last pass."""
    if out[2] > used:
        out[0][used:out[2]].zero_()
        out[1][used:out[2]].zero_()
    out[2] = used
    return {"ids": out[0], "vdf": out[1]}


def _take_out(s):
    """The batch's VDF: packed lists, or dense boxes."""
    if s.dense is not None:
        torch.cuda.current_stream().synchronize()  # the batch's stream does not wait for the last scatter
    ids, vals, _ = s.out
    counts, used = s.batch.pack_cells(s.cells, ids.data_ptr(), vals.data_ptr(), ids.shape[0])
    if s.dense is None:
        return {"counts": counts.astype(np.int64), **_filled(s.out, used)}
    if s.filled is not None:
        s.dense.index_fill_(0, s.filled, 0.0)
    c = torch.repeat_interleave(torch.as_tensor(counts.astype(np.int64)).to(DEV), output_size=used)
    g = ids[:used].to(torch.int64)
    L = s.case["mesh_len"]
    at = torch.stack([g % L, (g // L) % L, g // (L * L)], dim=1) - s.lo[c]
    size = s.size[c]
    inside = ((at >= 0) & (at < size)).all(dim=1)
    s.filled = torch.where(inside, s.first[c] + at[:, 0] + size[:, 0] * (at[:, 1] + size[:, 1] * at[:, 2]), s.rows)
    s.dense.index_copy_(0, s.filled, vals[:used])
    return {"vdf": s.dense[:s.rows]}


def run(s):
    kind = s.case["kind"]
    if kind == "call":
        k = len(s.counts)
        off, cnt, st = (np.zeros(k, np.uint32) for _ in range(3))
        p = lambda a, t: a.ctypes.data_as(ctypes.POINTER(t))  # noqa: E731
        res = {}
        for d in range(3):
            isect = np.ascontiguousarray(s.isect[:, d])
            ids, vals, _ = s.out[d]
            rc = s.lib.vlgpu_map_1d_noalloc(
                ctypes.byref(s.cmesh), ctypes.byref(s.params), k, p(s.offsets, ctypes.c_uint64), s.ids.data_ptr(),
                s.vals.data_ptr(), p(isect, ctypes.c_double), d, ids.data_ptr(), vals.data_ptr(), ids.shape[0],
                p(off, ctypes.c_uint32), p(cnt, ctypes.c_uint32), p(st, ctypes.c_uint32), None)
            if rc != 0:
                raise RuntimeError("vlgpu_map_1d_noalloc: %d" % rc)
            res["xyz"[d]] = _filled(s.out[d], int(cnt[0]))  # one cell: its blocks come first
        return res
    if kind == "serve":
        tickets = [s.server.submit(g, d, B, dt, steps) for g, d, B, dt, steps in s.requests]
        done = 0
        while done < len(tickets):
            done += s.server.tick()[2]
        got = [s.server.result(t) for t in tickets]
        a = 0
        for g in got:
            s.host[0][a:a + len(g[0])] = g[0].view(np.int32)
            s.host[1][a:a + len(g[0])] = g[1]
            a += len(g[0])
        s.host[0][a:] = 0
        s.host[1][a:] = 0.0
        return {"counts": np.array([len(g[0]) for g in got]), "ids": s.host[0], "vdf": s.host[1],
                "loss": np.array([g[3] for g in got])}
    b = s.batch
    if kind == "translate":
        for d in (2, 0, 1):
            b.translate(d, s.step)
        return _take_out(s)
    b.unpack_cells(s.cells, s.counts, s.ids.data_ptr(), s.vals.data_ptr())
    if kind == "sweeps":
        b.accelerate_with_intersections(s.isect, s.case["order"])
        return _take_out(s)
    if kind == "step":
        for q in range(STEPS):
            b.accelerate(s.B, s.dt, q % 3)
        return _take_out(s)
    if kind == "adjust":
        b.adjust()
        return {"moments": _record(b.moments(second=True)), **_take_out(s)}
    for q in range(VLASOV_STEPS):  # kind == "vlasov"
        b.vlasov_step(s.B, s.step, q % 3)
        r, mean = b.moments_r(), b.interpolated_moments()
    return {"r": _record(r), "mean": _record(mean), **_take_out(s)}


# ---------------------------------------------------------------------------
# what a pass cannot do without, and how close two correct results are
# ---------------------------------------------------------------------------
def work(case):
    blocks = float(_estimate(*_sizes(case)).sum())
    io = 260.0 * blocks                      # a block's ID and 64 values, once
    sweep, trans = 60.0 * 64 * blocks, 45.0 * 64 * blocks
    kind = case["kind"]
    if kind == "call":
        return {"bytes": 3 * 2 * io, "flops": 3 * sweep}
    if kind == "sweeps":
        return {"bytes": 2 * io, "flops": 3 * sweep}
    if kind == "step":
        return {"bytes": 2 * io, "flops": STEPS * (3 * sweep + 20.0 * 64 * blocks)}
    if kind == "adjust":
        return {"bytes": 2 * io, "flops": 20.0 * 64 * blocks}
    if kind == "translate":
        return {"bytes": 2 * io, "flops": 3 * trans}
    if kind == "vlasov":
        return {"bytes": 2 * io, "flops": VLASOV_STEPS * (3 * trans + 3 * sweep + 40.0 * 64 * blocks)}
    return {"bytes": 2 * io, "flops": 3.5 * (3 * sweep + 20.0 * 64 * blocks)}


def tolerance(case):
    """About four times what was measured between the single-precision results and the 64-bit ones.  A sweep
    places its edges in single precision, to 1e-5 of a cell: 3e-6 to 9e-6 after one to three sweeps, 1.4e-5 to
    2.9e-5 after six steps (and 2e-3 of the root mean square in a single value); a translation has no such
    edges (1e-7)."""
    kind = case["kind"]
    if kind == "adjust":
        # 64-bit sums in another order; the values are moved, not computed
        return {"rel": 1e-10, "max": 1e-9, "differ": 0.0}
    if kind == "translate":
        return {"rel": 5e-7, "max": 1e-4, "differ": 0.0}
    if kind in ("step", "serve", "vlasov"):
        return {"rel": 8e-5, "max": 1e-2, "differ": 1e-3}
    return {"rel": 3e-5, "max": 8e-3, "differ": 0.0}


# ---------------------------------------------------------------------------
# the same in 64 bits
# ---------------------------------------------------------------------------
def _shift(v, s):
    """Values s places further along the last axis, zeros beyond the ends."""
    if s == 0:
        return v
    o = torch.zeros_like(v)
    if s > 0:
        o[..., :-s] = v[..., s:]
    else:
        o[..., -s:] = v[..., :s]
    return o


def _superbee(a, b):
    """Limited slope from the right and left differences."""
    m = torch.maximum(torch.minimum(a.abs(), 2.0 * b.abs()), torch.minimum(2.0 * a.abs(), b.abs()))
    return torch.where(a * b > 0.0, torch.sign(a) * m, torch.zeros_like(a))


def _ppm64(vm1, v, vp1, fl, fr):
    s = _superbee(vp1 - v, v - vm1)
    fl, fr = torch.where(s == 0.0, v, fl), torch.where(s == 0.0, v, fr)
    fl = torch.where((vm1 - fl) * (fl - v) < 0.0, v - 0.5 * s, fl)
    fr = torch.where((vp1 - fr) * (fr - v) < 0.0, v + 0.5 * s, fr)
    d, e = fr - fl, v - 0.5 * (fl + fr)
    fl = torch.where(d * e > d * d / 6.0, 3.0 * v - 2.0 * fr, fl)
    d, e = fr - fl, v - 0.5 * (fl + fr)
    fr = torch.where(-d * d / 6.0 > d * e, 3.0 * v - 2.0 * fl, fr)
    return [fl, 3.0 * v - 2.0 * fl - fr, fl + fr - 2.0 * v]


def _coefficients(v, recon):
    vm1, vp1 = _shift(v, -1), _shift(v, 1)
    if recon == "plm":
        s = _superbee(vp1 - v, v - vm1)
        return [v - 0.5 * s, 0.5 * s]
    if recon == "ppm":
        fl = (-_shift(v, -2) + 7.0 * vm1 + 7.0 * v - vp1) / 12.0
        fr = (-vm1 + 7.0 * v + 7.0 * vp1 - _shift(v, 2)) / 12.0
        return _ppm64(vm1, v, vp1, fl, fr)

    def faces(o):
        w = [_shift(v, q + o) for q in range(-4, 4)]
        f = (533.0 * (w[3] + w[4]) - 139.0 * (w[2] + w[5]) + 29.0 * (w[1] + w[6]) - 3.0 * (w[0] + w[7])) / 840.0
        g = (7175.0 * (w[4] - w[3]) - 889.0 * (w[5] - w[2]) + 119.0 * (w[6] - w[1]) - 9.0 * (w[7] - w[0])) / 5040.0
        return f, g

    (fl, dl), (fr, dr) = faces(0), faces(1)
    z = torch.zeros_like(v)
    s = _superbee(vp1 - v, v - vm1)
    sg = torch.where(s > 0.0, 1.0, -1.0).to(v)
    flat = s == 0.0
    fl, fr = torch.where(flat, v, fl), torch.where(flat, v, fr)
    dl, dr = torch.where(flat, z, dl), torch.where(flat, z, dr)
    bad = ((vm1 - fl) * (fl - v) < 0.0) | (sg * dl < 0.0)
    fl, dl = torch.where(bad, v - 0.5 * s, fl), torch.where(bad, s, dl)
    bad = ((vp1 - fr) * (fr - v) < 0.0) | (sg * dr < 0.0)
    fr, dr = torch.where(bad, v + 0.5 * s, fr), torch.where(bad, s, dr)
    b0 = 60.0 * v - 24.0 * fr - 36.0 * fl + 3.0 * (dr - 3.0 * dl)
    b1 = -360.0 * v + 36.0 * dl - 24.0 * dr + 168.0 * fr + 192.0 * fl
    b2 = 360.0 * v + 30.0 * (dr - dl) - 180.0 * (fl + fr)
    disc = b1 * b1 - 4.0 * b0 * b2
    sq = torch.where(disc < 0.0, b1 + 200.0 * b2, torch.sqrt(disc.clamp(min=0.0)))
    pl, pr = 2.0 * (v - vm1), 2.0 * (vp1 - v)
    way = pl + pr
    wrong = torch.zeros_like(flat)
    for root in ((-b1 + sq) / (2.0 * b2), (-b1 - sq) / (2.0 * b2)):
        sl = dl + root * (b0 + root * (0.5 * b1 + root * b2 / 3.0))
        wrong |= (root >= 0.0) & (root <= 1.0) & (sl * way < 0.0)
    left = pl.abs() <= pr.abs()
    # the slopes collapsed to one edge, and to a monotone parabola where they still oppose the cell
    cl = torch.where(left, (10.0 * v - 2.0 * fr - 8.0 * fl) / 3.0, 10.0 * v - 6.0 * fl - 4.0 * fr)
    cr = torch.where(left, -10.0 * v + 6.0 * fr + 4.0 * fl, (-10.0 * v + 2.0 * fl + 8.0 * fr) / 3.0)
    ol = way * cl < 0.0
    orr = ~ol & (way * cr < 0.0)
    nfr = torch.where(ol, torch.where(left, 5.0 * v - 4.0 * fl, 0.5 * (5.0 * v - 3.0 * fl)), fr)
    ndr = torch.where(ol, torch.where(left, 20.0 * (v - fl), 10.0 / 3.0 * (v - fl)), torch.where(orr, z, cr))
    nfl = torch.where(orr, torch.where(left, 0.5 * (5.0 * v - 3.0 * fr), 5.0 * v - 4.0 * fr), fl)
    ndl = torch.where(orr, torch.where(left, 10.0 / 3.0 * (fr - v), 20.0 * (fr - v)), torch.where(ol, z, cl))
    fl, fr = torch.where(wrong, nfl, fl), torch.where(wrong, nfr, fr)
    dl, dr = torch.where(wrong, ndl, dl), torch.where(wrong, ndr, dr)
    return [fl, 0.5 * dl, 10.0 * v - 4.0 * fr - 6.0 * fl + 0.5 * (dr - 3.0 * dl),
            -15.0 * v + 1.5 * dl - dr + 7.0 * fr + 8.0 * fl, 6.0 * v + 0.5 * (dr - dl) - 3.0 * (fl + fr)]


# transverse axes (first, second) of a sweep along x, y, z, as array axes of (z, y, x)
_ACROSS = {0: (2, 1), 1: (0, 2), 2: (0, 1)}


def _targets(case, occ, lo, I, dim):
    """The target blocks of a sweep: every run of blocks along dim reaches
    from the lowest to the highest block that the corners of its cells meet,
    in single precision.  occ: blocks (z, y, x); lo: first block (x, y, z)."""
    f = np.float32
    L = case["mesh_len"]
    ax, bx = _ACROSS[dim]
    o = np.ascontiguousarray(np.transpose(occ, (2 - ax, 2 - bx, 2 - dim)))
    pad = np.pad(o.astype(np.int8), ((0, 0), (0, 0), (1, 1)))
    step = np.diff(pad, axis=2)
    a, b, first = np.nonzero(step == 1)
    _, _, last = np.nonzero(step == -1)
    last = last - 1
    i0, di, dj, dk = f(I[0]), f(I[1 + ax]), f(I[1 + bx]), f(I[1 + dim])
    A, B = [(4 * (a + lo[ax]) + q).astype(f) for q in (0, 3)], [(4 * (b + lo[bx]) + q).astype(f) for q in (0, 3)]
    corner = [(i0 + p * di) + q * dj for p in A for q in B]
    mx, mn = np.maximum.reduce(corner), np.minimum.reduce(corner)
    dv, vmin = f(BLOCK / 4), f(-0.5 * BLOCK * L)
    left, right = (4 * (first + lo[dim])).astype(f) * dv + vmin, (4 * (last + lo[dim] + 1)).astype(f) * dv + vmin
    fb = np.clip(np.trunc((left - mx) / dk).astype(int) // 4, 0, L - 1) - lo[dim]
    lb = np.clip(np.trunc((right - mn) / dk).astype(int) // 4, 0, L - 1) - lo[dim]
    mark = np.zeros((*o.shape[:2], o.shape[2] + 1), int)
    np.add.at(mark, (a, b, fb), 1)
    np.add.at(mark, (a, b, lb + 1), -1)
    t = np.cumsum(mark, axis=2)[..., :-1] > 0
    out = np.empty_like(occ)
    np.transpose(out, (2 - ax, 2 - bx, 2 - dim))[...] = t
    return out


def _sweep64(case, f, occ, lo, I, dim, recon):
    """One sweep of a dense cell f (z, y, x) whose first block is lo."""
    I = I.astype(np.float32).astype(np.float64)  # the sweeps take them in single precision
    ax, bx = _ACROSS[dim]
    new = _targets(case, occ, lo, I, dim)
    v = f.permute(2 - ax, 2 - bx, 2 - dim).contiguous()
    n = v.shape
    ar = lambda q, d: torch.arange(n[q], device=DEV, dtype=torch.float64) + 4.0 * lo[d]  # noqa: E731
    im = I[0] + ar(0, ax)[:, None] * I[1 + ax] + ar(1, bx)[None, :] * I[1 + bx]
    k = torch.arange(n[2] + 1, device=DEV, dtype=torch.float64)
    edge = (k + 4.0 * lo[dim]) * I[1 + dim] + im[..., None]
    pos = (edge + 0.5 * BLOCK * case["mesh_len"]) / (BLOCK / 4) - 4.0 * lo[dim]
    at = pos.floor().clamp(0, n[2] - 1)
    u = (pos - at).clamp(0.0, 1.0)
    at = at.to(torch.int64)
    total = torch.cumsum(v, dim=2) - v
    c = 0.0
    for a in reversed(_coefficients(v, recon)):
        c = (c + torch.gather(a, 2, at)) * u
    c = c + torch.gather(total, 2, at)
    out = torch.empty_like(f)
    out.permute(2 - ax, 2 - bx, 2 - dim).copy_(c[..., 1:] - c[..., :-1])
    keep = torch.as_tensor(new, device=DEV).repeat_interleave(4, 0).repeat_interleave(4, 1).repeat_interleave(4, 2)
    return out * keep, new


def _dilated(occ):
    """The +-1 neighbourhood of blocks (z, y, x)."""
    o = torch.as_tensor(occ, device=DEV).to(torch.float32)[None, None]
    return torch.nn.functional.max_pool3d(o, 3, 1, 1)[0, 0].bool().cpu().numpy()


def _by_block(f):
    """Dense (4nz, 4ny, 4nx) -> (nz, ny, nx, 64)."""
    z, y, x = (q // 4 for q in f.shape)
    return f.reshape(z, 4, y, 4, x, 4).permute(0, 2, 4, 1, 3, 5).reshape(z, y, x, 64)


def _adjusted(f, occ, more=None):
    """Block adjustment of a dense cell; more: further blocks to keep."""
    content = ((_by_block(f) >= MIN_VALUE).any(dim=-1).cpu().numpy()) & occ
    keep = _dilated(content)
    if more is not None:
        keep |= more
    t = torch.as_tensor(keep & occ, device=DEV).repeat_interleave(4, 0).repeat_interleave(4, 1).repeat_interleave(4, 2)
    return f * t, keep, content


def _moments64(case, f, lo):
    dv = BLOCK / 4
    ax = [-0.5 * BLOCK * case["mesh_len"] + (torch.arange(f.shape[2 - d], device=DEV, dtype=torch.float64)
                                             + 4.0 * lo[d] + 0.5) * dv for d in range(3)]
    vx, vy, vz = ax[0][None, None, :], ax[1][None, :, None], ax[2][:, None, None]
    s0 = f.sum()
    nV = torch.stack([(f * q).sum() for q in (vx, vy, vz)])
    V = nV / s0 if float(s0) else nV * 0.0
    u = [vx - V[0], vy - V[1], vz - V[2]]
    P = torch.stack([(f * u[a] * u[b]).sum() for a, b in ((0, 0), (1, 1), (2, 2), (1, 2), (0, 2), (0, 1))])
    d3 = dv ** 3
    n = s0 * d3
    rec = torch.cat([n[None], nV * d3, (n * MASS)[None], V, (n * CHARGE)[None], MASS * d3 * P, s0[None]])
    return rec.cpu().numpy()


def _dense_cells(case, counts, ids, vals, margin, common=False):
    """Per cell (f, occ, lo): the dense box around its blocks in 64 bits."""
    L = case["mesh_len"]
    off = np.concatenate([[0], np.cumsum(counts)]).astype(int)
    g = ids.cpu().numpy().astype(np.int64)
    at = np.stack([g % L, (g // L) % L, g // (L * L)], axis=1)
    lo = np.stack([at[off[c]:off[c + 1]].min(axis=0) for c in range(len(counts))])
    hi = np.stack([at[off[c]:off[c + 1]].max(axis=0) for c in range(len(counts))])
    if common:
        lo[:], hi[:] = lo.min(axis=0), hi.max(axis=0)
    lo, hi = np.maximum(lo - margin, 0), np.minimum(hi + margin, L - 1)
    out = []
    for c in range(len(counts)):
        sx, sy, sz = (int(q) for q in hi[c] - lo[c] + 1)
        p = at[off[c]:off[c + 1]] - lo[c]
        row = torch.as_tensor(p[:, 0] + sx * (p[:, 1] + sy * p[:, 2]), device=DEV)
        d = torch.zeros(sx * sy * sz, 64, device=DEV, dtype=torch.float64)
        d[row] = vals[off[c]:off[c + 1]].to(torch.float64)
        occ = torch.zeros(sx * sy * sz, dtype=torch.bool, device=DEV)
        occ[row] = True
        f = d.reshape(sz, sy, sx, 4, 4, 4).permute(0, 3, 1, 4, 2, 5).reshape(4 * sz, 4 * sy, 4 * sx)
        out.append([f.contiguous(), occ.reshape(sz, sy, sx).cpu().numpy(), lo[c].copy()])
    return out


def _lists(got, rows):
    """The lists of all cells one after another, zeros behind them."""
    ids, vdf = torch.cat([g for g, _ in got]), torch.cat([v for _, v in got])
    more = rows - len(ids)
    return {"ids": torch.nn.functional.pad(ids, (0, more)), "vdf": torch.nn.functional.pad(vdf, (0, 0, 0, more))}


def _listed_blocks(case, f, occ, lo, dim=0):
    """(IDs, values) in the order a sweep along dim leaves (dim 0: ascending ID)."""
    L = case["mesh_len"]
    ax, bx = _ACROSS[dim]
    q = np.stack(np.nonzero(np.transpose(occ, (2 - ax, 2 - bx, 2 - dim))))
    at = np.empty((3, q.shape[1]), int)
    at[ax], at[bx], at[dim] = q
    gid = (at[0] + lo[0]) + L * ((at[1] + lo[1]) + L * (at[2] + lo[2]))
    t = torch.as_tensor(at, device=DEV)
    return torch.as_tensor(gid.astype(np.int32), device=DEV), _by_block(f)[t[2], t[1], t[0]]


def _in_box(case, f, lo, box_lo, box_size):
    """The dense cell cut to or filled up to another box, as rows of blocks."""
    b = _by_block(f)
    out = torch.zeros(int(box_size[2]), int(box_size[1]), int(box_size[0]), 64, device=DEV, dtype=torch.float64)
    src, dst = [], []
    for d in (2, 1, 0):
        a = max(lo[d], box_lo[d])
        e = max(a, min(lo[d] + b.shape[2 - d], box_lo[d] + box_size[d]))
        src.append(slice(a - lo[d], e - lo[d]))
        dst.append(slice(a - box_lo[d], e - box_lo[d]))
    out[tuple(dst)] = b[tuple(src)]
    return out.reshape(-1, 64)


def _accelerated(case, f, occ, lo, B, dt, order):
    """One acceleration step of a dense cell, without its adjustment."""
    V = _moments64(case, f, lo)[5:8]
    I = _intersections(case, B[None], V[None], np.array([dt]), order).reshape(3, 4)
    for q in range(3):
        d = (order + q) % 3
        f, occ = _sweep64(case, f, occ, lo, I[d], d, "ppm")
    return f, occ


def _translated(case, cells, dim, dt):
    """One translation sweep of the whole grid, in place; every cell in the same box."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    N = (nx, ny, nz)[dim]
    lo = cells[0][2]
    half, dv = 0.5 * BLOCK * case["mesh_len"], BLOCK / 4
    shape = cells[0][0].shape
    v = -half + (torch.arange(shape[2 - dim], device=DEV, dtype=torch.float64) + 4.0 * lo[dim] + 0.5) * dv
    zt = (v * dt / DX).reshape([-1 if a == 2 - dim else 1 for a in range(3)])
    up = zt > 0.0
    z1, z2 = torch.where(up, 1.0 - zt, torch.zeros_like(zt)), torch.where(up, torch.ones_like(zt), -zt)
    grid = np.arange(nx * ny * nz).reshape(nz, ny, nx)
    for pencil in np.moveaxis(grid, 2 - dim, 2).reshape(-1, N):
        w = torch.stack([cells[c][0] for c in pencil])
        at = lambda s: torch.roll(w, -s, 0)  # noqa: E731
        fl = (-at(-2) + 7.0 * at(-1) + 7.0 * w - at(1)) / 12.0
        a = _ppm64(at(-1), w, at(1), fl, torch.roll(fl, -1, 0))
        gone = z2 * (a[0] + z2 * (a[1] + z2 * a[2])) - z1 * (a[0] + z1 * (a[1] + z1 * a[2]))
        out = w - gone + torch.where(up, torch.roll(gone, 1, 0), torch.roll(gone, -1, 0))
        for q, c in enumerate(pencil):
            keep = torch.as_tensor(cells[c][1], device=DEV)
            for r in range(3):
                keep = keep.repeat_interleave(4, r)
            cells[c][0] = out[q] * keep


def exact(case, seed):
    kind = case["kind"]
    plasma = _plasma(case, seed)
    V, B = plasma[3], plasma[4]
    dt = _step_dt(B)
    blocks = _estimate(plasma[0], plasma[1]).sum()
    most = {"call": 1e9, "sweeps": 5e5, "step": 2e5, "serve": 2e5, "adjust": 2e6, "translate": 1.5e6, "vlasov": 1.2e5}
    if blocks > most[kind] or len(dt) > 1500:
        return None
    counts, ids, vals = _vdf(case, plasma)
    if kind == "call":
        I = _intersections(case, B, V, dt, 0).reshape(-1, 3, 4)
        (f, occ, lo), = _dense_cells(case, counts, ids, vals, 3)
        res = {}
        for d in range(3):
            g = _listed_blocks(case, *_sweep64(case, f, occ, lo, I[0, d], d, "ppm"), lo, d)
            res["xyz"[d]] = _lists([g], min(65536, _rows(case, 2.5)))
        return res
    if kind == "sweeps":
        order = case["order"]
        I = _intersections(case, B, V, dt, order).reshape(-1, 3, 4)
        got = []
        for c, (f, occ, lo) in enumerate(_dense_cells(case, counts, ids, vals, 5)):
            for q in range(3):
                d = (order + q) % 3
                f, occ = _sweep64(case, f, occ, lo, I[c, d], d, case["recon"])
            got.append(_listed_blocks(case, f, occ, lo, (order + 2) % 3))
        return {"counts": np.array([len(g) for g, _ in got]), **_lists(got, _rows(case, 2.5))}
    if kind == "adjust":
        recs, got = [], []
        for f, occ, lo in _dense_cells(case, counts, ids, vals, 1):
            f, occ, _ = _adjusted(f, occ)
            recs.append(_moments64(case, f, lo))
            got.append(_listed_blocks(case, f, occ, lo))
        return {"moments": _record(np.stack(recs)), "counts": np.array([len(g) for g, _ in got]),
                **_lists(got, _rows(case, 1.0))}
    if kind == "translate":
        cells = _dense_cells(case, counts, ids, vals, 0, common=True)
        for d in (2, 0, 1):
            _translated(case, cells, d, _grid_dt(case))
        got = [_listed_blocks(case, f, occ, lo) for f, occ, lo in cells]
        return {"counts": counts.astype(np.int64), **_lists(got, _rows(case, 1.0))}
    if kind in ("step", "serve"):
        box_lo, box_size = _boxes(case, V)
        got = []
        for c, (f, occ, lo) in enumerate(_dense_cells(case, counts, ids, vals, 5)):
            for q in range(STEPS if kind == "step" else 1 + (5 * c + 2) % 6):
                f, occ = _accelerated(case, f, occ, lo, B[c], dt[c], q % 3)
                f, occ, _ = _adjusted(f, occ)
            got.append((f, occ, lo))
        if kind == "step" and len(got) >= DENSE_FROM:
            return {"vdf": torch.cat([_in_box(case, f, lo, box_lo[c], box_size[c])
                                      for c, (f, _, lo) in enumerate(got)])}
        got = [_listed_blocks(case, f, occ, lo) for f, occ, lo in got]
        res = {"counts": np.array([len(g) for g, _ in got]), **_lists(got, _rows(case, 1.0))}
        if kind == "serve":
            res["loss"] = None  # a sum of what lies below the threshold
        return res
    box_lo, box_size = _boxes(case, V)
    cells = _dense_cells(case, counts, ids, vals, 5, common=True)
    step = _grid_dt(case)
    shape = (case["nz"], case["ny"], case["nx"])
    for q in range(VLASOV_STEPS):
        for d in (2, 0, 1):
            _translated(case, cells, d, step)
        r = np.stack([_moments64(case, f, lo) for f, _, lo in cells])
        for c in range(len(cells)):
            f, occ, lo = cells[c]
            cells[c][0], cells[c][1] = _accelerated(case, f, occ, lo, B[c], step, q % 3)
        content = np.stack([(_by_block(f) >= MIN_VALUE).any(dim=-1).cpu().numpy() & occ for f, occ, _ in cells])
        near = content.reshape(*shape, *content.shape[1:])
        near = sum(np.roll(near, (a, b, c), (0, 1, 2)).astype(np.int8) for a in (-1, 0, 1) for b in (-1, 0, 1)
                   for c in (-1, 0, 1)).reshape(content.shape) > 0
        for c in range(len(cells)):
            cells[c][0], cells[c][1], _ = _adjusted(cells[c][0], cells[c][1], near[c])
        v = np.stack([_moments64(case, f, lo) for f, _, lo in cells])
    return {"r": _record(r), "mean": _record(0.5 * (r + v)),
            "vdf": torch.cat([_in_box(case, f, lo, box_lo[c], box_size[c]) for c, (f, _, lo) in enumerate(cells)])}

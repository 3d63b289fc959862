"""The screen of the D3Q27 cut-link kernel along the lattice's axes (csrc/d3q27_solids.cu, cut_cell),
restated in binary32 numpy and checked against the exact ray test on the CPU.

A candidate triangle's vertices are taken to the lattice's axes with the cell as origin, by the inverse
of the map that takes link directions to the body frame; a direction is dropped where, along some axis,
the triangle's interval misses its link (from 0 to -c) widened by 1e-3 and by 4e-6 of the farthest
coordinate. No (direction, triangle) pair that the exact test reports hit may be dropped: random
rotations, transforms that are not unit quaternions, mesh scales, small, large and sliver triangles.
"""
import numpy as np
import pytest

from test_cut_link_screens import DIRS, _mt_hits, _qrot, _quat

F = np.float32


@pytest.mark.parametrize("seed", [0, 1, 2, 3, 4, 5])
def test_axes_screen_keeps_every_hit(seed):
    rng = np.random.default_rng(100 + seed)
    hits_seen = 0
    for solid in range(40):
        q = _quat(rng)
        if solid % 4 == 3:
            q = (q * F(rng.uniform(0.7, 1.4))).astype(np.float32)  # no rotation any more
        scale = np.ones(3, np.float32) if solid % 3 else rng.uniform(0.5, 2.0, 3).astype(np.float32)
        inv_q = np.array([-q[0], -q[1], -q[2], q[3]], np.float32)
        centres = rng.uniform(-4, 4, (400, 1, 3))
        spread = rng.normal(0, 0.35, (400, 3, 3))
        spread[:60] *= 40.0  # large faces
        spread[60:160, 2] = spread[60:160, 0] * 0.5 + spread[60:160, 1] * 0.5 + rng.normal(0, 1e-4, (100, 3))  # slivers
        tris = (centres + spread).astype(np.float32)
        lds_all = (_qrot(inv_q, -DIRS) / scale).astype(np.float32)
        axis = {tuple(d): -l for d, l in zip(DIRS.astype(int), lds_all)}
        a = [axis[(1, 0, 0)], axis[(0, 1, 0)], axis[(0, 0, 1)]]
        rows = [np.cross(a[1], a[2]), np.cross(a[2], a[0]), np.cross(a[0], a[1])]
        det = F(np.dot(a[0], rows[0]))
        assert abs(det) > 1e-30
        w = np.array([(r * (F(1) / det)).astype(np.float32) for r in rows], np.float32)
        for _ in range(40):
            los = rng.uniform(-5, 5, 3).astype(np.float32)
            rel = (tris - los).astype(np.float32)
            lat = (rel[..., 0, None] * w[:, 0] + rel[..., 1, None] * w[:, 1] + rel[..., 2, None] * w[:, 2]).astype(np.float32)
            lo, hi = lat.min(axis=1), lat.max(axis=1)
            e = (F(4e-6) * np.maximum(-lo, hi).max(axis=1) + F(1e-3)).astype(np.float32)[:, None]
            for di in range(len(DIRS)):
                c = DIRS[di]
                if not c.any():
                    assert not _mt_hits(tris, los, lds_all[di]).any()  # the rest direction hits nothing
                    continue
                hit = _mt_hits(tris, los, lds_all[di])
                if not hit.any():
                    continue
                hits_seen += int(hit.sum())
                keep = ~np.any((lo > np.maximum(-c, 0) + e) | (hi < np.minimum(-c, 0) - e), axis=1)
                assert np.all(keep[hit]), (seed, solid, di)
    assert hits_seen > 200

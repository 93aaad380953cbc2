"""Mesh and heightmap pairs of a step run on a warp each, their triangle
loops split over the lanes: the contacts of a step equal rbps_batch_collide's
(one thread a pair) on the same poses, bit for bit, at face counts around the
32 lanes and cell counts below and above them."""
import numpy as np
import pytest

from rbps_b200 import abi, scenes

pytestmark = pytest.mark.gpu


def _drop(spec, seed):
    """The bodies moved into the ground's surface, so that many touch."""
    rng = np.random.default_rng(seed)
    spec.bodies["position"][1:, 1] = rng.uniform(-0.4, 0.6, len(spec.bodies) - 1)
    return spec


def _mesh(faces, second=False):
    spec = _drop(scenes.mesh_world(seed=faces, n=60, rows=17, cols=17), faces)
    verts, tris = spec.meshes[0]
    order = np.random.default_rng(faces).permutation(len(tris))[:faces]
    spec.meshes = [(verts, tris[order])]
    if second:  # a small mesh body over the ground mesh, and a plane under both
        small = verts[:40] * 0.1, tris[:20] % 40
        spec.meshes.append(small)
        spec.colliders["shape"][-1] = abi.SHAPE_MESH
        spec.colliders["hull"][-1] = 1
        plane = spec.colliders[:1].copy()
        plane["shape"], plane["hull"], plane["params"] = abi.SHAPE_PLANE, 0, (0.0, 1.0, 0.0, -0.2)
        spec.colliders = np.concatenate([spec.colliders, plane])
    return spec


def _terrain(rows, cell, scale=1.0):
    spec = _drop(scenes.terrain_world(seed=rows, n=60, rows=rows, cols=rows, cell=cell), rows)
    spec.colliders["params"][1:, :3] *= scale
    return spec


CASES = {
    "mesh_1": lambda: _mesh(1), "mesh_31": lambda: _mesh(31), "mesh_32": lambda: _mesh(32), "mesh_33": lambda: _mesh(33),
    "mesh_512": lambda: _mesh(512), "mesh_mesh_plane": lambda: _mesh(200, second=True),
    "cells_1": lambda: _terrain(2, 9.0), "cells_few": lambda: _terrain(33, 0.5),
    "cells_many": lambda: _terrain(65, 0.1, scale=2.0),  # tens to hundreds of cells under a shape
}


@pytest.mark.parametrize("name", sorted(CASES))
def test_step_contacts_equal_collide(rbps, name):
    spec = CASES[name]()
    b = rbps.Batch.from_scene(scenes.Scene(name, 1.0 / 60.0, 1, 1, [spec]), abi.PRECISION_FP64, abi.SOLVE_COLORED,
                              max_pairs_per_world=1 << 14)
    b.set_dump(True)
    b.step(1)
    got = b.contacts(0)
    tri = np.isin(spec.colliders["shape"], (abi.SHAPE_MESH, abi.SHAPE_HEIGHTMAP))
    a, c = np.meshgrid(np.nonzero(tri)[0], np.arange(len(tri)), indexing="ij")
    keep = (a != c) & (spec.colliders["body_id"][a] != spec.colliders["body_id"][c])
    a, c = a[keep], c[keep]
    pose = np.concatenate([spec.bodies["position"], spec.bodies["orientation"]], axis=1)
    hit = {}
    for x, y in ((a, c), (c, a)):
        m = b.collide(spec.colliders[x], pose[spec.colliders["body_id"][x]], spec.colliders[y],
                      pose[spec.colliders["body_id"][y]])
        hit.update({(int(i), int(j)): r for i, j, r in zip(x, y, m) if r["status"] == abi.COLLIDE_HIT})
    rows = {(int(r["collider_a"]), int(r["collider_b"])): r for r in got
            if tri[r["collider_a"]] or tri[r["collider_b"]]}
    assert {frozenset(k) for k in rows} == {frozenset(k) for k in hit}
    assert rows or name in ("mesh_1", "cells_1")  # one face or cell may meet nothing
    for k, r in rows.items():
        assert r["penetration_depth"] == hit[k]["depth"][0]
        np.testing.assert_array_equal(r["normal"], hit[k]["normal"])

"""The transport's shortcuts against the general path they stand in for: the
octree walk's plane rejection against the C restatement of octree::propagate,
which tests every listed triangle."""
import ctypes as C

import numpy as np
import pytest

from nebula_b200 import formats


def library_geometry(oracle, tris):
    """The restatement's geometry on the library's own octree (and what keeps
    its arrays alive)."""
    import nebula_b200 as nb
    o = nb.HostOctree(nb.triangles_from_tri_array(tris))
    t = o.triangles
    verts = np.ascontiguousarray(np.concatenate([t["r0"], t["e1"], t["e2"]], 1), np.float32)
    mats = np.ascontiguousarray(np.stack([t["mat_in"], t["mat_out"]], 1), np.int32)
    extent = 2 * np.sqrt(np.float32((o.halfsize.astype(np.float32) ** 2).sum()))
    g = oracle.Geometry(o.octree_data.ctypes.data, verts.ctypes.data, mats.ctypes.data, (C.c_float * 3)(*o.center),
                        (C.c_float * 3)(*o.halfsize), float(extent))
    return o, g, (verts, mats)


def sliver_soup(seed=11, n=400):
    """Random triangles of every shape: equilateral to needles of 1:5000,
    some of zero area, some sharing planes and edges."""
    rng = np.random.default_rng(seed)
    out = np.zeros(n, formats.TRI_DTYPE)
    a = rng.uniform(-60, 60, (n, 3))
    e = rng.normal(size=(n, 3)) * 10.0 ** rng.uniform(-1, 1.7, (n, 1))
    f = rng.normal(size=(n, 3)) * 10.0 ** rng.uniform(-2.5, 1.3, (n, 1))
    out["v"] = np.stack([a, a + e, a + f + e * rng.choice([0.0, 1.0], (n, 1))], 1).astype(np.float32)
    out["v"][:8, 2] = out["v"][:8, 1]                      # zero area
    out["v"][8:40, :, 2] = 5.0                             # one shared plane
    out["mat_in"] = rng.integers(0, 3, n)
    out["mat_out"] = formats.VACUUM
    return out


@pytest.mark.gpu
@pytest.mark.parametrize("name", ["cube", "grating", "rough", "holes", "slivers"])
def test_rays_match_the_walk_that_tests_every_triangle(name, inputs, ray_sampler):
    import nebula_b200 as nb
    import oracle
    tris = sliver_soup() if name == "slivers" else inputs[name]
    o, g, keep = library_geometry(oracle, tris)
    ctx = nb.setup(tris, [inputs["si"]], device=0)
    n = 60000
    pos, d, dist = ray_sampler(o.center - o.halfsize, o.center + o.halfsize, n, seed=17, z_focus=o.center[2])
    # rays that start on a triangle and graze its plane, and very short ones
    t = o.triangles
    k = n // 4
    pick = np.random.default_rng(5).integers(0, len(t), k)
    u = np.random.default_rng(6).random((k, 2)).astype(np.float32)
    pos[-k:] = t["r0"][pick] + u[:, :1] * t["e1"][pick] + u[:, 1:] * (1 - u[:, :1]) * t["e2"][pick]
    graze = t["e1"][pick] * u[:, 1:] - t["e2"][pick] * u[:, :1] + 1e-4 * d[-k:]
    length = np.linalg.norm(graze, axis=1, keepdims=True)
    ok = length[:, 0] > 1e-6
    d[-k:][ok] = (graze / np.maximum(length, 1e-6))[ok]
    dist[-k // 2:] *= np.float32(0.01)
    rng = np.random.default_rng(3)
    ign = np.where(rng.random(n) < 0.3, rng.integers(0, len(t), n), -1).astype(np.int32)
    imat = rng.choice([-123, 0, 1], n).astype(np.int32)
    gd, gt = ctx.ray_query(pos, d, dist, ign, imat)
    od, ot = np.zeros(n, np.float32), np.zeros(n, np.int32)
    oracle.port().nbo_propagate_batch(C.byref(g), pos, d, dist, ign, imat, n, od, ot)
    ctx.close()
    assert (ot >= 0).sum() > n // 100
    assert np.array_equal(gt, ot)
    assert np.array_equal(gd.view(np.uint32), od.view(np.uint32))

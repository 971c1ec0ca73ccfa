"""The transport's shortcuts against the general path they stand in for: the
octree walk's plane rejection against the C restatement of octree::propagate,
which tests every listed triangle; and whole runs, whose steps skip the walk
where the clearance map allows it and share a warp's electrons among its
lanes, against the same cascades taken one nbx_step_query at a time, which
walk every step."""
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


def cascades_step_by_step(ctx, prim, uid_base=0):
    """Per-primary SE and BSE counts and the event totals (steps, inelastic,
    elastic, boundary) of whole cascades, every electron advanced by single
    general steps."""
    import nebula_b200 as nb
    n = len(prim)
    e = np.zeros(n, nb.ELECTRON_DTYPE)
    e["pos"], e["dir"], e["E"] = prim[:, 0:3], prim[:, 3:6], prim[:, 6]
    e["mat"], e["last_tri"] = formats.VACUUM, -1
    e["tag"], e["uid"] = np.arange(n), uid_base + np.arange(n)
    se, bse, events = np.zeros(n, np.uint32), np.zeros(n, np.uint32), np.zeros(4, np.int64)
    while len(e):
        e, st, ev, new, has = ctx.step_query(e)
        events += [len(e)] + [(ev == k).sum() for k in (1, 2, 3)]
        hit = e[st == 2]
        np.add.at(se, hit["tag"][hit["E"] < 50], 1)
        np.add.at(bse, hit["tag"][hit["E"] >= 50], 1)
        e = np.concatenate([e[st == 0], new[has == 1]])
    return se, bse, events


def soup_in_a_block(seed=4):
    """A block of material 0 with the sliver soup just below its top face:
    arbitrary material changes, edges and needles in every cell."""
    from nebula_b200 import generators as g
    t = sliver_soup(seed, 600)
    t["v"] *= np.float32(0.4)
    t["v"][:, :, 2] -= np.float32(30.0)
    t["mat_out"] = np.random.default_rng(seed).integers(0, 3, len(t))
    return np.concatenate([g.cube_geometry(size=(300.0, 300.0, 200.0)), t])


@pytest.mark.gpu
@pytest.mark.parametrize("model", ["kieft", "penn"])
@pytest.mark.parametrize("name", ["cube", "grating_small", "rough", "holes", "soup", "vast"])
def test_run_equals_single_steps(name, model, inputs):
    import nebula_b200 as nb
    from nebula_b200 import generators as g
    # "vast": a domain whose clearance map needs cells above the usual size
    tris = (soup_in_a_block() if name == "soup" else
            g.cube_geometry(size=(60000.0, 60000.0, 30000.0)) if name == "vast" else inputs[name])
    top = {"cube": 1.0, "grating_small": 75.0, "rough": 20.0, "holes": 10.0, "soup": 1.0, "vast": 1.0}[name]
    recs = g.scan_beam(9, 9, 12, 500.0, spacing=8.0, origin=(-36.0, -36.0), z_start=top, seed=23,
                       energies=[120.0, 500.0, 2000.0])
    prim = np.concatenate([recs["pos"], recs["dir"], recs["E"][:, None]], 1).astype(np.float32)
    ctx = nb.setup(tris, [inputs["si"], inputs["sio2"], inputs["w"]], device=0, seed=77, inelastic=model)
    ctx.push(prim, np.arange(len(prim), dtype=np.uint32))
    ctx.run()
    s = ctx.stats()
    got = ctx.tag_counts(0, len(prim))
    se, bse, events = cascades_step_by_step(ctx, prim)
    ctx.close()
    assert events[1:].sum() > 20 * len(prim)
    assert np.array_equal(got[0], se) and np.array_equal(got[1], bse)
    assert [s[k] for k in ("steps", "events_inelastic", "events_elastic", "events_boundary")] == events.tolist()


def strip_sheets(length, width, span=70.0, n_sheets=12, gap=2.0, seed=5):
    """Parallel sheets in a general direction, cut into strips of two
    triangles, materials 0 and 1 in turn: where a rounded edge is extruded
    along a line, the exact test's rounding grows with the strips' length
    over their width and with their length."""
    q = np.linalg.qr(np.random.default_rng(seed).normal(size=(3, 3)))[0]
    shift = np.random.default_rng(seed).uniform(0, width, n_sheets)
    k, half = int(span / width), 0.5 * length * q[:, 0]
    v = []
    for s in range(n_sheets):
        o = np.array([0.0, 0.0, -12.0]) + q[:, 2] * gap * (s - n_sheets / 2) + q[:, 1] * shift[s]
        for j in range(k):
            a, b = o + q[:, 1] * (j - k / 2) * width, o + q[:, 1] * (j + 1 - k / 2) * width
            v += [(a - half, a + half, b + half), (a - half, b + half, b - half)]
    t = np.zeros(len(v), formats.TRI_DTYPE)
    t["v"] = np.array(v)
    t["mat_in"], t["mat_out"] = np.repeat(np.arange(n_sheets) % 2, 2 * k), np.repeat((np.arange(n_sheets) + 1) % 2, 2 * k)
    return t


def points_and_needles(n=4000, seed=1):
    """Triangles without an area, edges from 1 pm to 4 nm, on the block's top
    face and below it."""
    rng = np.random.default_rng(seed)
    p = rng.uniform([-40, -40, -20], [40, 40, 0], (n, 3))
    p[: n // 2, 2] = 0.0
    e = rng.normal(size=(n, 3)) * 10.0 ** rng.uniform(-3, 0.6, (n, 1))
    e[: n // 2, 2] = 0.0
    t = np.zeros(n, formats.TRI_DTYPE)
    t["v"] = np.stack([p, p + e, p + e * rng.choice([0.0, 0.5, 1.0, 2.0], (n, 1))], 1)
    t["mat_in"], t["mat_out"] = rng.integers(0, 2, n), rng.integers(0, 2, n)
    return t


@pytest.mark.gpu
@pytest.mark.parametrize("length,width", [(1000.0, 0.3), (3000.0, 1.0), (8000.0, 1.0), (4000.0, 4.0), (0.0, 0.0)])
def test_run_equals_single_steps_near_strips(length, width, inputs):
    import nebula_b200 as nb
    from nebula_b200 import generators as g
    extra = strip_sheets(length, width) if length else points_and_needles()
    tris = np.concatenate([g.cube_geometry(size=(300.0, 300.0, 200.0)), extra])
    recs = g.scan_beam(9, 9, 12, 500.0, spacing=4.0, origin=(-18.0, -18.0), z_start=1.0, seed=23,
                       energies=[120.0, 500.0, 2000.0])
    prim = np.concatenate([recs["pos"], recs["dir"], recs["E"][:, None]], 1).astype(np.float32)
    ctx = nb.setup(tris, [inputs["si"], inputs["sio2"]], device=0, seed=77)
    ctx.push(prim, np.arange(len(prim), dtype=np.uint32))
    ctx.run()
    s = ctx.stats()
    got = ctx.tag_counts(0, len(prim))
    se, bse, events = cascades_step_by_step(ctx, prim)
    ctx.close()
    assert events[3] > (20000 if length else 5000)   # most of them in the strips
    assert np.array_equal(got[0], se) and np.array_equal(got[1], bse)
    assert [s[k] for k in ("steps", "events_inelastic", "events_elastic", "events_boundary")] == events.tolist()


@pytest.mark.gpu
def test_fine_mesh_in_a_vast_domain():
    """A whole mesh in one cell of the map: setting the geometry takes
    milliseconds (370 ms when a thread went over all triangles)."""
    import time
    import nebula_b200 as nb
    from nebula_b200 import generators as g
    tris = np.concatenate([g.cube_geometry(size=(1e6, 1e6, 1e6)), g.rough_geometry(n=256, size=200.0)])
    o = nb.HostOctree(nb.triangles_from_tri_array(tris))
    ctx = nb.Context(device=0)
    took = []
    for _ in range(5):
        t = time.perf_counter()
        ctx.set_geometry(o)
        took.append(time.perf_counter() - t)
    ctx.close()
    assert min(took) < 0.1, took


@pytest.mark.gpu
def test_refused_geometry_changes_nothing(inputs):
    """A geometry that nbx_set_geometry refuses leaves the one before it whole;
    one that fails for want of memory leaves none."""
    import nebula_b200 as nb
    import torch
    from nebula_b200 import generators as g
    ctx = nb.setup(inputs["cube"], [inputs["si"]], device=0, seed=3)
    recs = g.scan_beam(8, 8, 8, 500.0, z_start=1.0, seed=2)
    ctx.set_tag_range(len(recs))
    other = nb.HostOctree(nb.triangles_from_tri_array(inputs["rough"]))
    other._p.contents.triangles[5].mat_in = 40000
    got = []
    for again in (False, True):
        if again:
            with pytest.raises(nb.NbxError) as e:
                ctx.set_geometry(other)
            assert e.value.code == -1
        ctx.reset_tallies()
        ctx.set_uid_base(0)
        ctx.push_records(recs)
        ctx.run()
        got.append(np.stack(ctx.tag_counts(0, len(recs))))
    assert np.array_equal(*got) and got[0].sum() > 0
    other._p.contents.triangles[5].mat_in = 0
    big = nb.HostOctree(nb.triangles_from_tri_array(g.rough_geometry(n=256, size=500.0)))
    hold = [torch.empty(torch.cuda.mem_get_info()[0] - (4 << 20), dtype=torch.uint8, device="cuda")]
    with pytest.raises(nb.NbxError) as e:
        ctx.set_geometry(big)
    assert e.value.code == -2
    hold.clear()
    torch.cuda.empty_cache()
    with pytest.raises(nb.NbxError) as e:
        ctx.run()
    assert e.value.code == -6
    ctx.set_geometry(big)
    ctx.push_records(recs)
    ctx.run()
    ctx.close()


@pytest.mark.gpu
@pytest.mark.parametrize("spare", [1500, 400])
def test_map_when_memory_is_short(spare, inputs):
    """With little device memory left the map takes an eighth of it at most,
    its coarse grid included (here 200 MB at the usual cell), and larger cells
    before it is given up; runs are the same."""
    import nebula_b200 as nb
    import torch
    from nebula_b200 import generators as g
    far = np.zeros(1, formats.TRI_DTYPE)   # one small triangle that makes the domain 6 um wide
    far["v"] = np.array([5700.0, 5700.0, -5700.0]) + np.array([[0, 0, 0], [5, 0, 0], [0, 5, 0]])
    far["mat_in"] = far["mat_out"] = formats.VACUUM
    tris = np.concatenate([g.cube_geometry(size=(300.0, 300.0, 300.0)), far])
    recs = g.scan_beam(8, 8, 8, 500.0, z_start=1.0, seed=2)
    o = nb.HostOctree(nb.triangles_from_tri_array(tris))
    got = []
    for short in (True, False):
        ctx = nb.Context(device=0, seed=3)
        ctx.add_material(nb.HostMaterial(inputs["si"]))
        hold = None
        if short:
            torch.cuda.init()
            hold = torch.empty(torch.cuda.mem_get_info()[0] - (spare << 20), dtype=torch.uint8, device="cuda")
        free = torch.cuda.mem_get_info()[0]
        ctx.set_geometry(o)
        took = free - torch.cuda.mem_get_info()[0]
        if short:
            assert took < free // 8 + (16 << 20), (took, free)   # (and a few MB of triangles, in 2 MB pages)
        m = ctx.clearance()
        assert 0 < m["bytes"] <= took
        assert m["cell"] > 4 if short else m["cell"] == 4
        ctx.set_tag_range(len(recs))
        ctx.push_records(recs)
        ctx.run()
        got.append(np.stack(ctx.tag_counts(0, len(recs))))
        ctx.close()
        del hold
        torch.cuda.empty_cache()
    assert np.array_equal(*got) and got[0].sum() > 0


@pytest.mark.gpu
def test_table_indices_at_the_edges(inputs):
    """Table lookups whose index is clamped: below and above the axes, on
    every grid point and its neighbours, huge, infinite and NaN coordinates
    (the restatement's floor-to-int turns the last three into index 0)."""
    import ctypes as C
    import nebula_b200 as nb
    import oracle
    m = nb.HostMaterial(inputs["si"])
    ctx = nb.Context(device=0)
    ctx.add_material(m)
    P = oracle.port()
    for name in ("el_imfp", "in_imfp", "el_icdf", "in_icdf", "ion"):
        a, (x0, xs, y0, ys) = m.tables[name]
        a = np.ascontiguousarray(a, np.float32)
        grid = np.float32(x0) + np.arange(a.shape[0], dtype=np.float32) / np.float32(xs)
        x = np.concatenate([grid, np.nextafter(grid, np.float32(-np.inf)), np.nextafter(grid, np.float32(np.inf)),
                            np.array([-1e30, -5, 5e9, 1e30, np.inf, -np.inf, np.nan], np.float32)]).astype(np.float32)
        y = np.resize(np.array([0.0, 1e-7, 0.5, 0.9999999, 1.0, -0.25, 1.75, 1e12], np.float32), len(x))
        got = ctx.table_query(0, name, x, y)
        if name.endswith("imfp"):
            t = oracle.Table1D(len(a), x0, xs, a.ctypes.data)
            want = [P.nbo_table1d_get(C.byref(t), float(v)) for v in x]
        else:
            t = oracle.Table2D(a.shape[0], a.shape[1], x0, xs, y0, ys, a.ctypes.data)
            f = P.nbo_table2d_get_rounddown if name == "ion" else P.nbo_table2d_get
            want = [f(C.byref(t), float(v), float(w)) for v, w in zip(x, y)]
        assert np.array_equal(got, np.array(want, np.float32), equal_nan=True), name
    ctx.close()


@pytest.mark.gpu
@pytest.mark.parametrize("mode", ["plain", "weighted", "network"])
def test_launch_shapes_and_shallow_stacks_change_nothing(mode, inputs):
    """The same per-primary tallies whatever the launch shape and the stacks'
    depth, and with queues that fill whole ranges, one primary and none."""
    import nebula_b200 as nb
    from nebula_b200 import generators as g
    recs = g.scan_beam(16, 12, 11, 2000.0, spacing=4.0, origin=(-32.0, -24.0), seed=9)
    want = None
    for variant, block, depth in ((3, 256, 16), (3, 256, 1), (2, 32, 1), (4, 128, 2), (7, 128, 1), (4, 256, 64)):
        ctx = nb.setup(inputs["grating_small"], [inputs["si"]], device=0, seed=5)
        ctx.set_tag_range(len(recs))
        if mode != "plain":
            ctx.build_surface_map([-150, -150, -60], [150, 150, 60], 2.0, 20.0)
            ctx.mlp_set_params(nb.mlp_init_params(3))
            ctx.set_mode("learned", rr_threshold=0.6, split_threshold=0.65, max_roulette_exp=3)
            if mode == "weighted":
                ctx.set_importance_table(16, 16, 8)
        ctx.set_tuning(variant, block, depth, 2)
        got = []
        for n in (len(recs), 1, 0, 149):
            ctx.reset_tallies()
            ctx.set_uid_base(0)
            ctx.push_records(recs[:n])
            ctx.run()
            s = ctx.stats()
            got += [ctx.tag_counts(0, len(recs)), ctx.tag_weights(0, len(recs)),
                    [s[k] for k in ("steps", "events_elastic", "events_inelastic", "events_boundary", "secondaries",
                                    "terminated", "detected", "primaries_done", "queue_overflow")]]
        ctx.close()
        want = want or got
        for a, b in zip(got, want):
            assert all(np.array_equal(x, y) for x, y in zip(a, b)), (variant, block, depth)
    assert want[0][0].sum() > 100 and want[2][-1] == 0


@pytest.mark.gpu
@pytest.mark.parametrize("mode", ["plain", "weighted", "network"])
def test_secondaries_through_the_queue(mode, inputs):
    """Stacks of one electron per thread and enough primaries for a warp to
    fill its 32: secondaries then go through the next generations' queues (in
    learned mode with their weights), and every tally is that of a run that needs
    no queue."""
    import nebula_b200 as nb
    from nebula_b200 import generators as g
    recs = g.scan_beam(40, 40, 25, 5000.0, spacing=2.0, origin=(-40.0, -40.0), seed=9)
    got = []
    for shape in ((3, 256, 64), (2, 32, 1)):
        ctx = nb.setup(inputs["grating_small"], [inputs["si"]], device=0, seed=5, capacity=1 << 24)
        ctx.set_tag_range(len(recs))
        if mode != "plain":
            ctx.build_surface_map([-150, -150, -60], [150, 150, 60], 2.0, 20.0)
            ctx.mlp_set_params(nb.mlp_init_params(3))
            ctx.set_mode("learned", rr_threshold=0.3, split_threshold=0.3, max_roulette_exp=3)
            if mode == "weighted":
                ctx.set_importance_table(16, 16, 8)
        ctx.set_tuning(*shape, 2)
        ctx.push_records(recs)
        ctx.run()
        s = ctx.stats()
        assert (s["generations"] > 1) == (shape[2] == 1), s["generations"]
        got.append(list(ctx.tag_counts(0, len(recs))) + list(ctx.tag_weights(0, len(recs))) +
                   [s[k] for k in ("steps", "events_elastic", "events_inelastic", "events_boundary", "secondaries",
                                   "splits", "roulette_killed", "terminated", "detected", "primaries_done")])
        assert s["queue_overflow"] == 0 and s["primaries_done"] == len(recs)
        if mode != "plain":
            assert got[-1][2].sum() < 0.75 * got[-1][0].sum()   # most secondaries carry a weight of one half
        ctx.close()
    assert all(np.array_equal(a, b) for a, b in zip(*got))


@pytest.mark.gpu
def test_deposits_do_not_depend_on_the_launch(inputs):
    """The same set of energy-deposit records whatever the launch shape."""
    import nebula_b200 as nb
    from nebula_b200 import generators as g
    recs = g.scan_beam(12, 12, 8, 500.0, spacing=4.0, origin=(-24.0, -24.0), seed=9)
    want = None
    for shape in ((3, 256, 16), (2, 32, 1), (7, 128, 2), (4, 256, 64)):
        ctx = nb.setup(inputs["grating_small"], [inputs["si"]], device=0, seed=5, record_deposits=True,
                       deposit_capacity=1 << 23)
        ctx.set_tuning(*shape, 2)
        ctx.push_records(recs)
        ctx.run()
        s = ctx.stats()
        d = ctx.flush_deposits()
        ctx.close()
        assert s["deposits_dropped"] == 0 and len(d) == s["deposits"] > 100000
        x = d.view(np.uint32).reshape(len(d), -1)
        x = x[np.lexsort(x.T)]
        want = x if want is None else want
        assert np.array_equal(x, want), shape


@pytest.mark.gpu
def test_sample_mode_covers_the_queue(inputs):
    """Sample mode takes every primary once, whatever its launch shape and the
    ranges the queue is cut into (one, several an SM, fewer primaries than
    ranges, one shared cursor): the event totals of a plain run, and the same
    set of samples each time."""
    import nebula_b200 as nb
    from nebula_b200 import generators as g
    recs = g.scan_beam(60, 40, 16, 500.0, spacing=2.0, origin=(-60.0, -40.0), seed=9)   # 38,400: two ranges an SM
    keys = ("primaries_done", "steps", "events_elastic", "events_inelastic", "events_boundary", "secondaries",
            "terminated", "detected_se", "detected_bse")
    want = None
    for mode, shape, shared in (("plain", (3, 256), 0), ("sample", (3, 256), 0), ("sample", (2, 32), 0),
                                ("sample", (7, 128), 0), ("sample", (4, 256), 1)):
        ctx = nb.setup(inputs["grating_small"], [inputs["si"]], device=0, seed=5, shared_pop=shared)
        ctx.set_tag_range(len(recs))
        ctx.build_surface_map([-150, -150, -60], [150, 150, 60], 2.0, 20.0)
        ctx.set_tuning(*shape, 64, 2)
        if mode == "sample":
            ctx.set_sample_capacity(1 << 21)
            ctx.set_mode("sample")
        got = []
        for n in (len(recs), 149, 1):
            ctx.reset_tallies()
            ctx.set_uid_base(0)
            ctx.push_records(recs[:n])
            ctx.run()
            s = ctx.stats()
            got.append([s[k] for k in keys])
            assert s["primaries_done"] == n
            if mode == "sample":
                x = np.column_stack(ctx.get_samples(1 << 21, with_cost=True))
                got.append(x[np.lexsort(x.T)])
        ctx.close()
        if mode == "plain":
            totals = got
            continue
        assert got[0::2] == totals, (shape, shared)
        want = want or got[1::2]
        assert all(np.array_equal(a, b) for a, b in zip(got[1::2], want)), (shape, shared)
    assert len(want[0]) > 1000

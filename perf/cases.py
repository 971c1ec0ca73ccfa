"""Performance cases: the simulations a user of nebula_b200 runs.

Every simulation case is one frame of a scan through the library's public
calls: the tallies are reset, the primaries go in from page-locked host
buffers (or stay in device buffers for the allocation-free call), the
transport runs every cascade to its end and the frame's results come back.
Geometries, materials, beams and modes are those of the repository's
benchmark scans and tests; the sizes run from a 1,024-primary preview tile,
where latency counts, to half of the benchmark's grating frame.
"""
import functools
import math
import os
import tempfile

import numpy as np
import torch

import nebula_b200 as nb
from nebula_b200 import generators as g

MATERIALS = {"cube": ("si",), "grating": ("si",), "rough": ("si",), "holes": ("sio2", "w", "si")}
# Events (elastic + inelastic + boundary) per primary of each scan at 1 keV,
# by inelastic model; they grow about in proportion to the energy.
EVENTS_PER_KEV = {"cube": (560, 200), "grating": (650, 300), "rough": (545, 160), "holes": (424, 311)}
# Floating-point operations an event cannot do without: two free paths, one
# table interpolation, the rotation of a direction, the step to the new
# position and one ray-triangle test.
FLOPS_PER_EVENT = 150
MIXED = (300.0, 1000.0, 3000.0, 5000.0)
Z_START = {"cube": 1.0, "grating": 75.0, "rough": 25.0, "holes": 10.0}
# Surface map of the learned mode: box height, cell and largest distance (nm).
MAP_Z = {"grating": (-60.0, 60.0, 2.0, 20.0), "rough": (-40.0, 30.0, 2.0, 10.0), "holes": (-170.0, 15.0, 4.0, 10.0)}


def scan(name, workload, nx, ny, per_pixel, energy, spacing, model="kieft", mode="plain", size=0):
    """A frame of nx x ny pixels; `energy` 0 is the mixed beam, `size` the
    geometry's extent (samples a side of the rough slab, holes a side)."""
    return {"name": name, "workload": workload, "nx": nx, "ny": ny, "per_pixel": per_pixel, "energy": energy,
            "spacing": spacing, "model": model, "mode": mode, "size": size}


def listed():
    return [
        # preview of one tile while the operator focuses: 1,024 primaries
        scan("tile", "grating", 8, 8, 16, 500.0, 1.0),
        # half of the benchmark's grating frame: 3.28 M primaries
        scan("grating_frame", "grating", 256, 128, 100, 500.0, 1.0),
        # the yield of a flat sample at one point, with detected records
        scan("cube_records", "cube", 1, 1, 10000, 1000.0, 1.0, mode="records"),
        # mixed beam energies on a rough slab (voltage series of one field)
        scan("rough_mixed", "rough", 101, 99, 20, 0.0, 4.0, size=256),
        # contact holes, three materials, a patch of 4 x 4 holes in the array
        scan("holes", "holes", 128, 128, 20, 1000.0, 2.5, size=16),
        # the reference's stock inelastic model on each of the three scans
        scan("grating_penn", "grating", 256, 63, 25, 500.0, 1.0, model="penn"),
        scan("rough_penn", "rough", 127, 61, 15, 1000.0, 3.0, model="penn", size=128),
        scan("holes_penn", "holes", 97, 85, 12, 1000.0, 2.5, model="penn", size=8),
        # a host application that owns the device memory: device buffers,
        # allocation-free call
        scan("device_buffers", "grating", 53, 29, 13, 500.0, 4.0, mode="noalloc"),
        # learned roulette, decisions from the importance table, cost-aware
        scan("learned_table", "rough", 128, 128, 10, 0.0, 3.0, mode="table", size=256),
        # learned roulette, network evaluated for every newborn, weight window
        scan("learned_network", "grating", 128, 64, 20, 500.0, 2.0, mode="network"),
        # fitting the escape-probability network to recorded newborns and
        # scoring them with the result
        {"name": "fit_network", "mode": "train", "records": 200003, "epochs": 2, "batch": 8192},
    ]


def draw(rng):
    """One more case: any of the listed kinds, 1,000 primaries upwards."""
    kind = rng.choice(["plain", "plain", "plain", "plain", "records", "noalloc", "table", "network", "train"])
    if kind == "train":
        return {"mode": "train", "records": int(round(math.exp(rng.uniform(math.log(9e3), math.log(5e5))))),
                "epochs": rng.randint(1, 3), "batch": rng.choice([1024, 4096, 8192, 16384])}
    workload = rng.choice(["grating", "rough", "holes"] if kind in ("plain", "table", "network")
                          else ["cube", "grating", "rough", "holes"])
    model = rng.choice(["kieft", "kieft", "penn"])
    # the allocation-free call's fixed scratch is for beams up to about 1 keV
    energy = rng.choice([300.0, 500.0, 1000.0] if kind == "noalloc" else [300.0, 500.0, 1000.0, 2000.0, 5000.0, 0.0])
    size = {"rough": rng.choice([64, 100, 128, 256]), "holes": rng.choice([3, 4, 8, 16])}.get(workload, 0)
    top = 65000 if kind == "noalloc" else 100000 if kind == "records" else 1000000
    top = min(top, 0.5 * 3.2768e6 * 325 / events_per_primary(workload, model, energy))
    n = math.exp(rng.uniform(math.log(1000), math.log(top)))
    per_pixel = rng.choice([1, 7, 16, 20, 33, 100])
    nx = max(1, min(256, int(math.sqrt(n / per_pixel) * rng.uniform(0.6, 1.6))))
    ny = max(1, int(n / per_pixel / nx))
    if kind == "noalloc":
        ny = max(1, min(ny, 65536 // (nx * per_pixel)))
    # the scanned field stays on the sample
    field = {"cube": 400.0, "grating": 400.0, "rough": 1.5 * size, "holes": 70.0 * size}[workload]
    spacing = min(rng.choice([0.5, 1.0, 2.5]), field / max(nx, ny))
    c = scan("", workload, nx, ny, per_pixel, energy, spacing, model=model, mode=kind, size=size)
    del c["name"]
    return c


def events_per_primary(workload, model, energy):
    kev = (energy or sum(MIXED) / len(MIXED)) / 1000.0
    return EVENTS_PER_KEV[workload][model == "penn"] * kev


def primaries(case):
    return case["nx"] * case["ny"] * case["per_pixel"]


@functools.lru_cache(maxsize=None)
def material(kind):
    """Path of a synthetic material file, written once per process."""
    return g.make_material(os.path.join(tempfile.mkdtemp(prefix="nbx_cases_"), kind + ".mat"), kind)


def geometry(case):
    w, size = case["workload"], case["size"]
    if w == "cube":
        return g.cube_geometry()
    if w == "grating":
        return g.grating_geometry()
    if w == "rough":
        return g.rough_geometry(n=size, size=size * 1000.0 / 512)   # the benchmark's sampling of the height field
    return g.contact_hole_geometry(n_holes=size)


def network(seed):
    """Parameters like a trained escape-probability network's: seeded hidden
    layers, the output layer fitted to a logit that falls with the distance
    to the surface and rises with energy and with flight toward it."""
    p = nb.mlp_init_params(seed).astype(np.float64)
    x = np.zeros((4096, 16))
    rng = np.random.default_rng(seed)
    x[:, 0:2] = rng.random((4096, 2))
    x[:, 2] = rng.uniform(-1, 1, 4096)
    x[np.arange(4096), 3 + rng.integers(0, 3, 4096)] = 1.0
    silu = lambda v: v / (1.0 + np.exp(-v))
    h = silu(x @ p[:1024].reshape(64, 16).T + p[1024:1088])
    h = silu(h @ p[1088:5184].reshape(64, 64).T + p[5184:5248])
    logit = -2.0 - 7.0 * x[:, 1] + 1.5 * x[:, 2] + 3.0 * x[:, 0]
    w = np.linalg.lstsq(np.concatenate([h, np.ones((4096, 1))], 1), logit, rcond=None)[0]
    p[5248:5312] = w[:64]
    p[5760] = w[64]
    return p.astype(np.float32)


def training_records(case, seed):
    """Newborn electrons' features and escape labels."""
    rng = np.random.default_rng(seed)
    n = case["records"]
    f = np.zeros((n, 6), np.float32)
    f[:, 0] = rng.random(n) ** 2
    f[:, 1] = rng.random(n)
    f[:, 2] = rng.uniform(-1, 1, n)
    f[:, 3] = 1.0
    p = 1.0 / (1.0 + np.exp(2.0 + 7.0 * f[:, 1] - 1.5 * f[:, 2] - 3.0 * f[:, 0]))
    return f, (rng.random(n) < p).astype(np.float32)


def prepare(case, seed):
    if case["mode"] == "train":
        # the network lives in a context; its geometry plays no part
        ctx = nb.setup(g.cube_geometry(), [material("si")])
        f, y = training_records(case, seed)
        return {"case": case, "ctx": ctx, "features": f, "labels": y, "params": nb.mlp_init_params(seed % 1000)}
    w, mode = case["workload"], case["mode"]
    nx, ny, n = case["nx"], case["ny"], primaries(case)
    ctx = nb.setup(geometry(case), [material(k) for k in MATERIALS[w]], seed=0x78C7E39B ^ (seed & 0xFFFF),
                   inelastic=case["model"], record_detected=mode == "records", record_capacity=1 << 20)
    recs = g.scan_beam(nx, ny, case["per_pixel"], case["energy"], spacing=case["spacing"],
                       origin=(-0.5 * nx * case["spacing"], -0.5 * ny * case["spacing"]), z_start=Z_START[w],
                       seed=seed, energies=None if case["energy"] else MIXED)
    prim = nb.host_empty((n, 7), np.float32)
    prim[:, 0:3] = recs["pos"]
    prim[:, 3:6] = recs["dir"]
    prim[:, 6] = recs["E"]
    tags = nb.host_empty(n, np.uint32)
    tags[:] = np.arange(n, dtype=np.uint32)
    state = {"case": case, "ctx": ctx, "prim": prim, "tags": tags, "n": n, "pixels": nx * ny}
    if mode == "noalloc":
        state["d_prim"] = torch.from_numpy(prim).cuda()
        state["d_tags"] = torch.from_numpy(tags.view(np.int32)).cuda()
        state["d_se"] = torch.zeros(n, dtype=torch.int32, device="cuda")
        state["d_bse"] = torch.zeros(n, dtype=torch.int32, device="cuda")
        return state
    ctx.set_tag_range(n)
    ctx.set_pixel_map(recs["py"].astype(np.uint32) * nx + recs["px"].astype(np.uint32))
    if mode in ("table", "network"):
        z0, z1, cell, d_max = MAP_Z[w]
        rx, ry = 0.5 * nx * case["spacing"] + 20.0, 0.5 * ny * case["spacing"] + 20.0
        ctx.build_surface_map([-rx, -ry, z0], [rx, ry, z1], cell, d_max)
        ctx.mlp_set_params(network(7))
        if mode == "table":
            # cost-aware survival without splitting: sub-cascade cost (steps)
            # growing with the newborn's energy
            ctx.set_mode("learned", rr_threshold=0.05, split_threshold=2.0, max_roulette_exp=4)
            cost = np.tile(np.exp(np.linspace(0.0, 6.0, 32)), (len(MATERIALS[w]), 1))
            ctx.set_learned_cost(cost, 2.5, 9.0, 400.0)
            ctx.set_importance_table(48, 32, 16)
        else:
            ctx.set_mode("learned", rr_threshold=0.05, split_threshold=0.5, max_roulette_exp=3)
    return state


def run(state):
    ctx, mode = state["ctx"], state["case"]["mode"]
    if mode == "train":
        case = state["case"]
        ctx.mlp_set_params(state["params"])
        losses = ctx.mlp_train(state["features"], state["labels"], epochs=case["epochs"], batch=case["batch"],
                               lr=1e-3, seed=1)
        return {"losses": losses, "params": ctx.mlp_get_params(), "escape": ctx.mlp_predict(state["features"])}
    n = state["n"]
    if mode == "noalloc":
        state["d_se"].zero_()
        state["d_bse"].zero_()
        torch.cuda.current_stream().synchronize()   # the call reads its buffers on the context's own stream
        counts = nb.run_noalloc(ctx, state["d_prim"].data_ptr(), state["d_tags"].data_ptr(), n, 0,
                                state["d_se"].data_ptr(), state["d_bse"].data_ptr(), n)
        return {"se": state["d_se"], "bse": state["d_bse"], "events": np.array(list(counts.values()), np.int64)}
    ctx.reset_tallies()
    ctx.set_uid_base(0)
    ctx.push(state["prim"], state["tags"])
    ctx.run()
    out = {"yields": ctx.pixel_yields(None, state["pixels"]), "spectrum": ctx.spectrum()[0].astype(np.int64)}
    if mode == "records":
        # the device appends records in arrival order: put them in scan order,
        # in an image of fixed size (three records a primary, zeros after the last)
        rec = ctx.flush_detected()
        rec = rec[np.lexsort((rec["E"], rec["tag"]))][:3 * n]
        out["records"] = np.zeros((3 * n, 7), np.float32)
        out["record_tags"] = np.zeros(3 * n, np.int64)
        for k, name in ((slice(0, 3), "pos"), (slice(3, 6), "dir"), (6, "E")):
            out["records"][:len(rec), k] = rec[name]
        out["record_tags"][:len(rec)] = rec["tag"]
    elif mode == "plain":
        se, bse = ctx.tag_counts(0, n)
        out.update(se=se.view(np.int32), bse=bse.view(np.int32))
    else:
        out["se_weight"], out["bse_weight"] = ctx.tag_weights(0, n)
    return out


def work(case):
    if case["mode"] == "train":
        rows = case["records"] * case["epochs"]
        # forward, and twice that backward, of the 6 -> 64 -> 64 -> 1 network
        return {"bytes": case["records"] * 32 + 2 * 4 * 5768,
                "flops": (6 * rows + 2 * case["records"]) * (6 * 64 + 64 * 64 + 64)}
    n = primaries(case)
    return {"bytes": n * (28 + 4) + n * 8 + case["nx"] * case["ny"] * 40,
            "flops": int(n * events_per_primary(case["workload"], case["model"], case["energy"]) * FLOPS_PER_EVENT)}


def exact(case, seed):
    """The transport's outputs are whole numbers and random trajectories, and
    the fit follows the library's own shuffle: none has a value apart from
    the library's random streams."""
    return None

"""Shared fixtures.  Tests marked ``gpu`` need a CUDA device (B200); the
rest run on CPU.  Inputs are generated by the seeded synthetic generators."""
import os
import sys

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
if ROOT not in sys.path:
    sys.path.insert(0, ROOT)


def pytest_configure(config):
    config.addinivalue_line("markers", "gpu: needs a CUDA device")


def _skip_without_reference():
    """Tests against the reference's own build are skipped where it is missing
    (it needs the reference's source tree)."""
    import oracle
    try:
        return (yield)
    except oracle.ReferenceMissing as e:
        pytest.skip(str(e))


@pytest.hookimpl(wrapper=True)
def pytest_runtest_setup(item):
    return (yield from _skip_without_reference())


@pytest.hookimpl(wrapper=True)
def pytest_runtest_call(item):
    return (yield from _skip_without_reference())


@pytest.fixture(scope="session")
def oracle_built():
    import oracle
    oracle.build()
    return oracle


@pytest.fixture(scope="session")
def inputs(tmp_path_factory):
    """Synthetic materials and geometries shared by the tests."""
    from nebula_b200 import formats, generators as g
    d = tmp_path_factory.mktemp("inputs")
    out = {"dir": str(d)}
    out["si"] = g.make_material(str(d / "si.mat"), "si")
    out["sio2"] = g.make_material(str(d / "sio2.mat"), "sio2")
    out["w"] = g.make_material(str(d / "w.mat"), "w")
    out["cube"] = g.cube_geometry()
    out["grating"] = g.grating_geometry()
    out["grating_small"] = g.grating_geometry(n_lines=7, length=400.0)
    out["rough"] = g.rough_geometry(n=64, size=200.0, seed=5)
    # 3 x 3 contact holes (22,052 triangles): SiO2-like film, W-like plugs,
    # Si-like substrate
    out["holes"] = g.contact_hole_geometry(n_holes=3, seed=2)
    for name in ("cube", "grating", "rough", "holes"):
        p = str(d / (name + ".tri"))
        formats.write_tri(p, out[name])
        out[name + "_tri"] = p
    return out


def random_rays(geom_lo, geom_hi, n, seed, z_focus=0.0, z_sigma=40.0):
    rng = np.random.default_rng(seed)
    lo = np.asarray(geom_lo, np.float32)
    hi = np.asarray(geom_hi, np.float32)
    pos = (lo + (hi - lo) * rng.random((n, 3))).astype(np.float32)
    half = n // 2
    pos[:half, 2] = rng.normal(z_focus, z_sigma, half).astype(np.float32)
    d = rng.normal(size=(n, 3)).astype(np.float32)
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    # a few exactly axis-aligned directions (division by zero paths)
    k = n // 16
    d[:k] = 0
    d[np.arange(k), rng.integers(0, 3, k)] = rng.choice([-1.0, 1.0], k)
    dist = rng.exponential(50.0, n).astype(np.float32)
    dist[: n // 32] = np.float32(1e9)
    return pos, d.astype(np.float32), dist


@pytest.fixture(scope="session")
def ray_sampler():
    return random_rays

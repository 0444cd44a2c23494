"""The four-wide tree's walks against the oracle's binary walk: hit ids,
distances, barycentrics and occlusion bit for bit on the trees and rays where
its conservative boxes, its octant order or its way back to the binary walk
could go wrong."""
import numpy as np
import pytest

import pathtracingtutorial_b200 as pt
from oracle.pyoracle import Oracle
from pathtracingtutorial_b200 import scenes

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def oracle():
    return Oracle()


def _soup(pos):
    """Triangles given as (n, 3, 3) positions."""
    n = len(pos)
    v = np.zeros(3 * n, pt.VERTEX_DTYPE)
    v["position"] = pos.reshape(-1, 3)
    v["normal"] = (0, 1, 0)
    f = np.zeros(n, pt.FACE_DTYPE)
    f["v0"], f["v1"], f["v2"] = np.arange(0, 3 * n, 3), np.arange(1, 3 * n, 3), np.arange(2, 3 * n, 3)
    return scenes.SceneArrays("soup", v, f, scenes._materials([pt.default_material()]), pt.make_camera(width=8, height=8))


def _random(n, seed, size=0.3):
    rng = np.random.default_rng(seed)
    c = rng.uniform(-1, 1, (n, 1, 3))
    return (c + rng.uniform(-size, size, (n, 3, 3))).astype(np.float32)


def _scene(name):
    if name == "one":
        return _soup(_random(1, 1))
    if name == "one_leaf":
        return _soup(_random(3, 2))
    if name == "few":
        return _soup(_random(9, 3))
    if name == "flat":          # boxes without thickness, shared edges and planes
        g = np.linspace(-1, 1, 17, dtype=np.float32)
        x, z = np.meshgrid(g[:-1], g[:-1])
        x, z, h = x.ravel(), z.ravel(), g[1] - g[0]
        y = np.zeros_like(x)
        a, b = np.stack([x, y, z], 1), np.stack([x + h, y, z], 1)
        c, d = np.stack([x + h, y, z + h], 1), np.stack([x, y, z + h], 1)
        return _soup(np.concatenate([np.stack([a, b, c], 1), np.stack([a, c, d], 1)]))
    if name == "chain":         # sizes and distances in a geometric progression: a deep, lopsided tree
        k = 2.0 ** -np.arange(40)[:, None, None]
        return _soup(((_random(40, 4, 0.4) * 0.3 + 1.0) * k).astype(np.float32))
    if name == "far":           # coordinates large against the triangles
        return _soup(_random(400, 5) + np.float32(1e5))
    if name == "tiny":
        return _soup(_random(200, 6) * np.float32(1e-12))
    if name == "large":
        return _soup(_random(200, 7) * np.float32(1e12))
    if name == "beyond":        # beyond the four-wide tree's range: the binary walk
        return _soup(_random(50, 8) * np.float32(3e30))
    return scenes.icosphere_field(n_spheres=12, subdiv=2, width=8, height=8, env_size=None)


def _rays(sa, seed):
    p = sa.vertices["position"]
    lo, hi = p.min(0).astype(np.float64), p.max(0).astype(np.float64)
    ext = (hi - lo).max()
    rng = np.random.default_rng(seed)
    n = 30_000
    o = rng.uniform(lo - 0.5 * ext, hi + 0.5 * ext, (n, 3))
    d = rng.normal(size=(n, 3))
    # aimed at the triangles; along one axis or in one plane; from a box plane or a vertex
    q = p[rng.integers(0, len(p), n)]
    d[: n // 2] = (q - o)[: n // 2] + 0.05 * ext * rng.normal(size=(n // 2, 3))
    zero = rng.random((n, 3)) < np.where(np.arange(n) % 4 == 0, 0.5, 0.0)[:, None]
    d[zero] = 0.0
    d[(zero.all(1))] = (0.0, -1.0, 0.0)
    o[::7] = q[::7]
    o[1::7, rng.integers(0, 3)] = lo[rng.integers(0, 3)]
    nrm = np.linalg.norm(d, axis=1, keepdims=True)
    d = d / np.where(nrm > 0, nrm, 1)
    d = d.astype(np.float32)
    d[d == 0] *= np.where(rng.random((d == 0).sum()) < 0.5, -1, 1).astype(np.float32)    # -0 too
    # denormal, very short and very long directions
    d[3::50, rng.integers(0, 3)] = np.float32(1e-41)
    for start, k in ((5, 1e-25), (6, 1e-12), (8, 1e8), (9, 1e-18)):
        d[start::50] = (d[start::50] * np.float32(k)).astype(np.float32)
    tmax = (rng.uniform(0.05, 2.0, n) * ext).astype(np.float32)
    tmax[::3] = np.finfo(np.float32).max
    return o.astype(np.float32), d, tmax


@pytest.mark.parametrize("watertight", [False, True])
@pytest.mark.parametrize("name", ["one", "one_leaf", "few", "flat", "chain", "far", "tiny", "large", "beyond", "spheres"])
def test_wide_walks_equal_the_binary_walk(oracle, name, watertight):
    sa = _scene(name)
    s = sa.scene()
    s.build_accel()
    if watertight:
        s.update_settings(flags=pt.FLAG_WATERTIGHT)
    s.upload_to_device(0)
    prep = oracle.prepare(sa)
    o, d, tmax = _rays(sa, 17)
    rays = np.zeros((len(o), 8), np.float32)
    rays[:, :3], rays[:, 4:7], rays[:, 7] = o, d, tmax
    kw = {"watertight": True} if watertight else {}
    ref, _ = oracle.trace(prep.nodes, prep.vertices, prep.faces, rays, **kw)
    hits = pt.trace_closest(s, o, d)
    gpu = np.stack([hits["t"], hits["prim"].view(np.float32), hits["u"], hits["v"]], 1)
    assert np.array_equal(gpu.view(np.uint32), ref.view(np.uint32))
    ref_occ, _ = oracle.trace(prep.nodes, prep.vertices, prep.faces, rays, any_hit=True, **kw)
    assert np.array_equal(pt.trace_any(s, o, d, tmax), ref_occ)


def test_rays_that_are_not_numbers_hit_nothing():
    sa = _scene("few")
    s = sa.scene()
    s.build_accel()
    s.upload_to_device(0)
    o, d, tmax = _rays(sa, 3)
    o[0::3, 1] = np.nan
    d[1::3, 2] = np.nan
    o[2::3, 0] = np.inf
    assert (pt.trace_closest(s, o, d)["prim"] == -1).all()
    assert not pt.trace_any(s, o, d, tmax).any()


def test_reupload_rebuilds_the_wide_tree(oracle):
    """A rebuilt tree (GPU builder, same array sizes as far as they go) traces through its own wide tree."""
    sa = _scene("spheres")
    s = sa.scene()
    s.build_accel()
    s.upload_to_device(0)
    o, d, _ = _rays(sa, 4)
    a = pt.trace_closest(s, o, d)
    s.build_accel(builder="device")
    s.upload_to_device(0)
    b = pt.trace_closest(s, o, d)
    assert np.array_equal(a["t"], b["t"])

"""The four-wide tree's walks against the oracle's binary walk, bit for bit,
where its boxes have no thickness away from the coordinate 0, and on a tree that
needs the deep stack; and which scenes have a four-wide tree at all."""
import numpy as np
import pytest

import pathtracingtutorial_b200 as pt
from pathtracingtutorial_b200 import scenes

pytestmark = pytest.mark.gpu


def _soup(pos):
    """Triangles given as (n, 3, 3) positions."""
    n = len(pos)
    v = np.zeros(3 * n, pt.VERTEX_DTYPE)
    v["position"] = pos.reshape(-1, 3)
    v["normal"] = (0, 1, 0)
    f = np.zeros(n, pt.FACE_DTYPE)
    f["v0"], f["v1"], f["v2"] = np.arange(0, 3 * n, 3), np.arange(1, 3 * n, 3), np.arange(2, 3 * n, 3)
    return scenes.SceneArrays("soup", v, f, scenes._materials([pt.default_material()]), pt.make_camera(width=8, height=8))


def _grid(axis, at, cells=16):
    """A square of 2 cells^2 triangles in the plane where `axis` is `at`."""
    g = np.linspace(-1, 1, cells + 1, dtype=np.float32)
    a, b = np.meshgrid(g[:-1], g[:-1])
    a, b, h = a.ravel(), b.ravel(), g[1] - g[0]
    def at_(p, q):
        out = np.empty((len(p), 3), np.float32)
        out[:, axis], out[:, (axis + 1) % 3], out[:, (axis + 2) % 3] = at, p, q
        return out
    c = [at_(a, b), at_(a + h, b), at_(a + h, b + h), at_(a, b + h)]
    return np.concatenate([np.stack([c[0], c[1], c[2]], 1), np.stack([c[0], c[2], c[3]], 1)])


def _compare(oracle, sa, o, d, tmax, watertight):
    s = sa.scene()
    s.build_accel()
    if watertight:
        s.update_settings(flags=pt.FLAG_WATERTIGHT)
    s.upload_to_device(0)
    assert s.info()["walk_entries"] > 0
    prep = oracle.prepare(sa)
    rays = np.zeros((len(o), 8), np.float32)
    rays[:, :3], rays[:, 4:7], rays[:, 7] = o, d, tmax
    kw = {"watertight": True} if watertight else {}
    ref, _ = oracle.trace(prep.nodes, prep.vertices, prep.faces, rays, **kw)
    hits = pt.trace_closest(s, o, d)
    gpu = np.stack([hits["t"], hits["prim"].view(np.float32), hits["u"], hits["v"]], 1)
    assert np.array_equal(gpu.view(np.uint32), ref.view(np.uint32))
    ref_occ, _ = oracle.trace(prep.nodes, prep.vertices, prep.faces, rays, any_hit=True, **kw)
    assert np.array_equal(pt.trace_any(s, o, d, tmax), ref_occ)
    return s, hits


@pytest.mark.parametrize("watertight", [False, True])
@pytest.mark.parametrize("axis", [0, 1, 2])
@pytest.mark.parametrize("at", [1.0, -1.0, 1.5, 548.8, -1e-3])
def test_planes_away_from_zero(oracle, axis, at, watertight):
    sa = _soup(_grid(axis, np.float32(at)))
    rng = np.random.default_rng(int(axis + 10 * abs(at)))
    n = 12_000
    p = rng.uniform(-1.05, 1.05, (n, 3)).astype(np.float32)     # a point of the plane, or just beside the square
    p[:, axis] = np.float32(at)
    p[::5] = sa.vertices["position"][rng.integers(0, len(sa.vertices), len(p[::5]))]
    d = rng.normal(size=(n, 3)).astype(np.float32)
    d[1::4, axis] = 0.0                                          # along the plane
    d[2::4] = 0.0                                                # square to it
    d[2::4, axis] = np.where(rng.random(len(d[2::4])) < 0.5, -1, 1)
    dist = (10.0 ** rng.uniform(-3, 2, n)).astype(np.float32)
    o = p - d * dist[:, None]                                    # towards it
    o[3::8] = p[3::8]                                            # from it
    tmax = (dist * rng.choice([0.5, 2.0], n)).astype(np.float32)
    _, hits = _compare(oracle, sa, o, d, tmax, watertight)
    assert (hits["prim"] >= 0).mean() > 0.2


def _nested(levels=28, per=12, ratio=8.0, top=1e6):
    """Clusters of triangles in a geometric progression towards the origin: every
    level of the tree has one large child to split and the rest of the chain."""
    rng = np.random.default_rng(0)
    c = np.concatenate([(1 + rng.uniform(-0.4, 0.4, (per, 1, 3)) + rng.uniform(-0.08, 0.08, (per, 3, 3)))
                        * (top * ratio ** -k) for k in range(levels)])
    return c.astype(np.float32)


@pytest.mark.parametrize("watertight", [False, True])
def test_walks_that_need_more_than_64_entries(oracle, watertight):
    sa = _soup(_nested())
    sa.env = scenes.sky_env(64, 32)
    sa.camera = pt.make_camera(position=(2.2e6, 2.2e6, 2.2e6), look_at=(0, 0, 0), fov=40, width=48, height=40)
    rng = np.random.default_rng(2)
    p = sa.vertices["position"]
    n = 20_000
    o = rng.uniform(-2e6, 2e6, (n, 3)).astype(np.float32)
    o[::4] = p[rng.integers(0, len(p), len(o[::4]))]
    d = (p[rng.integers(0, len(p), n)] - o).astype(np.float32)
    d[1::4] = -1.0                                  # down the chain
    o[1::4] = rng.uniform(0.5, 2.0, (len(o[1::4]), 3)) * 1e6
    nrm = np.linalg.norm(d, axis=1, keepdims=True)
    d = (d / np.where(nrm > 0, nrm, 1)).astype(np.float32)
    d[(d == 0).all(1)] = (0, 1, 0)
    tmax = (10.0 ** rng.uniform(0, 7, n)).astype(np.float32)
    s, hits = _compare(oracle, sa, o, d, tmax, watertight)
    assert 64 < s.info()["walk_entries"] <= 192 and s.info()["bvh_max_depth"] < 64
    assert (hits["prim"] >= 0).mean() > 0.2
    # a render through the deep extension and shadow kernels, and through the binary ones
    flags = pt.FLAG_WATERTIGHT if watertight else 0
    img = pt.render(s, 8)
    s.update_settings(flags=flags | pt.FLAG_COUNT_TRAVERSAL)
    assert np.array_equal(pt.render(s, 8).view(np.uint32), img.view(np.uint32))
    for block in (64, 256):
        for depth in (32, 64):
            s.update_settings(flags=flags, trace_block=block, stack_depth=depth)
            assert np.array_equal(pt.render(s, 8).view(np.uint32), img.view(np.uint32))
    assert np.isfinite(img).all() and img[..., :3].std() > 0


def test_coordinates_out_of_range_keep_the_binary_tree():
    rng = np.random.default_rng(8)
    pos = (rng.uniform(-1, 1, (50, 1, 3)) + rng.uniform(-0.3, 0.3, (50, 3, 3))).astype(np.float32)
    for scale, wide in ((np.float32(1), True), (np.float32(3e30), False)):
        s = _soup(pos * scale).scene()
        s.build_accel()
        assert s.info()["walk_entries"] == 0
        s.upload_to_device(0)
        assert (s.info()["walk_entries"] > 0) == wide

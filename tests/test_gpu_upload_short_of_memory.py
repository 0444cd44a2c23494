"""A scene uploaded where the device has no room for all of its four-wide tree
keeps none of it, and walks the binary one."""
import numpy as np
import pytest

import pathtracingtutorial_b200 as pt
from pathtracingtutorial_b200 import scenes

pytestmark = pytest.mark.gpu

MB = 1 << 20


def test_no_part_of_the_tree_is_kept():
    import torch
    import bench
    sa = scenes.icosphere_field(n_spheres=200, subdiv=4, width=8, height=8, env_size=None)    # 1M triangles
    s = sa.scene()
    s.build_accel()
    base = bench.upload_bytes(s.info())
    nodes, records = 43 * s.info()["num_inner_nodes"], 64 * s.info()["num_faces"]
    assert records > 48 * MB
    rng = np.random.default_rng(1)
    o = rng.uniform(-5, 5, (2000, 3)).astype(np.float32)
    d = rng.normal(size=(2000, 3)).astype(np.float32)
    s.upload_to_device(0)
    assert s.info()["walk_entries"] > 0 and s.info()["device_bytes"] > base + records
    ref = pt.trace_closest(s, o, d)
    s.set_punctual_lights(np.zeros(0, pt.PUNCTUAL_DTYPE))                                     # frees the device scene
    torch.cuda.empty_cache()
    free, _ = torch.cuda.mem_get_info()
    # room for the copied arrays, the nodes and half of the records
    ballast = torch.empty(free - base - nodes - records // 2, dtype=torch.uint8, device="cuda")
    before = torch.cuda.mem_get_info()[0]
    s.upload_to_device(0)
    used = before - torch.cuda.mem_get_info()[0]
    del ballast
    torch.cuda.empty_cache()
    assert s.info()["walk_entries"] == 0 and s.info()["device_bytes"] == base
    assert used < base + nodes // 2 + 8 * MB
    assert np.array_equal(pt.trace_closest(s, o, d), ref)

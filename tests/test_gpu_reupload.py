"""Uploading a scene again in place (same device, same arrays): renders may be
in flight, so the four-wide tree that they read is not built anew."""
import numpy as np
import pytest

import pathtracingtutorial_b200 as pt
from pathtracingtutorial_b200 import scenes

pytestmark = pytest.mark.gpu


def test_reupload_in_place_launches_nothing_and_keeps_the_hits():
    import torch
    from torch.profiler import ProfilerActivity, profile

    sa = scenes.icosphere_field(n_spheres=12, subdiv=2, width=32, height=32, env_size=(64, 32))
    s = sa.scene()
    s.build_accel()

    def kernels(upload):
        torch.cuda.synchronize()
        with profile(activities=[ProfilerActivity.CUDA]) as prof:
            upload()
            torch.cuda.synchronize()
        return [e.name for e in prof.events() if "k_wide" in e.name]

    assert kernels(lambda: s.upload_to_device(0))          # the profiler sees the collapse of a first upload
    bytes_once = s.info()["device_bytes"]
    rng = np.random.default_rng(3)
    o = rng.uniform(-5, 5, (5000, 3)).astype(np.float32)
    d = rng.normal(size=(5000, 3)).astype(np.float32)
    tmax = np.full(5000, 4.0, np.float32)
    hits, occ, img = pt.trace_closest(s, o, d), pt.trace_any(s, o, d, tmax), pt.render(s, 4)
    assert kernels(lambda: s.upload_to_device(0)) == []
    assert s.info()["device_bytes"] == bytes_once
    assert np.array_equal(pt.trace_closest(s, o, d), hits)
    assert np.array_equal(pt.trace_any(s, o, d, tmax), occ)
    assert np.array_equal(pt.render(s, 4), img)

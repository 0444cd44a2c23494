"""The tuner's candidates are kernels that differ, timed without a graph capture,
and its choice is kept per way of walking the rays."""
import numpy as np
import pytest

import pathtracingtutorial_b200 as pt
from pathtracingtutorial_b200 import scenes

pytestmark = pytest.mark.gpu


def _scene(n_spheres=60, width=40, height=24, **kw):
    s = scenes.icosphere_field(n_spheres=n_spheres, subdiv=3, width=width, height=height, spp=4, env_size=(32, 16),
                               **kw).scene()
    s.build_accel()
    s.upload_to_device(0)
    return s


def test_calibration_renders_capture_no_graph():
    import torch
    from torch.profiler import ProfilerActivity, profile
    s = _scene(width=41)
    torch.cuda.synchronize()
    with profile(activities=[ProfilerActivity.CPU, ProfilerActivity.CUDA]) as prof:
        rep = s.autotune(calib_spp=4)
        torch.cuda.synchronize()
    names = {e.name for e in prof.events()}
    assert any("k_extend" in n for n in names) and not rep["cached"]
    assert not any("cudaGraph" in n for n in names)
    assert not s.settings().flags & pt.FLAG_NO_GRAPH


def test_no_candidate_runs_as_another():
    s = _scene(height=48)
    # a shallow tree whose four-wide walk still needs more than 32 entries
    assert s.info()["bvh_max_depth"] < 32 < s.info()["walk_entries"] <= 64
    rep = s.autotune(calib_spp=4)
    assert not rep["cached"] and {c["stack_depth"] for c in rep["candidates"]} == {64}
    t = scenes.cornell_box(width=40, height=24, spp=4, max_depth=4).scene()
    t.build_accel()
    t.upload_to_device(0)
    assert t.info()["walk_entries"] <= 32
    assert {c["stack_depth"] for c in t.autotune(calib_spp=4)["candidates"]} == {32, 64}


def test_the_choice_is_kept_per_walk():
    for flags in (0, pt.FLAG_WATERTIGHT, pt.FLAG_COUNT_TRAVERSAL):
        for cached in (False, True):
            s = _scene(width=320, height=24, seed=3 + cached)
            s.update_settings(flags=flags)
            ref = pt.render(s, 4)
            assert s.autotune(calib_spp=4)["cached"] == cached
            assert s.settings().flags == flags
            assert np.array_equal(pt.render(s, 4), ref)

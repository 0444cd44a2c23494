"""The traversal kernels that the render settings ask for are the ones that run:
block size and stack entries, on the four-wide tree, in watertight mode and with
traversal counters, with the same image from each."""
import re

import numpy as np
import pytest

import pathtracingtutorial_b200 as pt
from pathtracingtutorial_b200 import scenes

pytestmark = pytest.mark.gpu


def _shapes(run):
    """(kernel, block, entries, walk) of the traversal kernels that `run` launches."""
    import torch
    from torch.profiler import ProfilerActivity, profile
    torch.cuda.synchronize()
    with profile(activities=[ProfilerActivity.CUDA]) as prof:
        run()
        torch.cuda.synchronize()
    found = set()
    for e in prof.events():
        m = re.search(r"(k_extend|k_shadow)<(\d+), (\d+), (\d+)>", e.name)
        if m:
            found.add((m[1],) + tuple(int(x) for x in m.groups()[1:]))
    return found


@pytest.mark.parametrize("flags,walk", [(0, 1), (pt.FLAG_WATERTIGHT, 2), (pt.FLAG_COUNT_TRAVERSAL, 0)])
def test_the_settings_choose_the_kernel(flags, walk):
    s = scenes.cornell_box(width=24, height=16, spp=4, max_depth=4).scene()
    s.build_accel()
    s.upload_to_device(0)
    assert 0 < s.info()["walk_entries"] <= 32 and s.info()["bvh_max_depth"] < 32
    s.update_settings(flags=flags)
    ref = pt.render(s, 4)
    for block in (64, 128, 256):
        for entries in (32, 64):
            s.update_settings(trace_block=block, stack_depth=entries)
            imgs = []
            got = _shapes(lambda: imgs.append(pt.render(s, 4)))
            assert got == {("k_extend", block, entries, walk), ("k_shadow", block, entries, walk)}
            assert np.array_equal(imgs[0].view(np.uint32), ref.view(np.uint32))


@pytest.mark.parametrize("flags,walk", [(0, 1), (pt.FLAG_WATERTIGHT, 2)])
def test_a_walk_that_needs_more_gets_more(flags, walk):
    sa = scenes.icosphere_field(n_spheres=60, subdiv=3, width=24, height=16, env_size=(32, 16))
    s = sa.scene()
    s.build_accel()
    s.upload_to_device(0)
    need = s.info()["walk_entries"]
    assert 32 < need <= 64
    s.update_settings(flags=flags, trace_block=256, stack_depth=32)
    assert {k[1:] for k in _shapes(lambda: pt.render(s, 4))} == {(256, 64, walk)}

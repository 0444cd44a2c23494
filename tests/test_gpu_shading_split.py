"""Shading under an open sky takes hits and misses in separate batches: the
image does not depend on how a queue splits into them."""
import numpy as np
import pytest

import pathtracingtutorial_b200 as pt
from pathtracingtutorial_b200 import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("textured", [False, True])
@pytest.mark.parametrize("size", [(1, 1), (3, 5), (16, 16), (257, 1), (64, 47)])
def test_image_independent_of_queue_sizes(size, textured):
    w, h = size
    if textured:
        sa = scenes.textured_cornell(width=w, height=h, spp=12, max_depth=6)
        sa.env = scenes.sky_env(64, 32)
    else:
        sa = scenes.icosphere_field(n_spheres=5, subdiv=1, width=w, height=h, spp=12, max_depth=6, env_size=(64, 32))
    s = sa.scene()
    s.build_accel()
    s.upload_to_device(0)
    ref = pt.render(s, 12)
    assert np.isfinite(ref).all() and ref[..., :3].max() > 0
    for paths in (w * h, 3 * w * h, 5 * w * h):     # queues of other lengths, other batches
        s.update_settings(paths_in_flight=paths)
        assert np.array_equal(pt.render(s, 12), ref)

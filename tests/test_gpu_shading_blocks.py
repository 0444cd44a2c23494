"""Textured shading comes in blocks of 256 for short queues and of 1024 for long
ones: a long render's pixels do not depend on which, alone or with a guide."""
import numpy as np
import pytest

import pathtracingtutorial_b200 as pt
from pathtracingtutorial_b200 import scenes

pytestmark = pytest.mark.gpu

LONG = 6 * 1024 * 148       # path slots from which the textured kernels take blocks of 1024 (148 SMs)


@pytest.mark.parametrize("env", [False, True])
@pytest.mark.parametrize("spp", [1, 3])
def test_image_independent_of_the_shading_block(env, spp):
    # 1024 x 888 is exactly the first long queue, a row less the last short one
    for h in (887, 888):
        sa = scenes.textured_cornell(width=1024, height=h, spp=spp, max_depth=5)
        assert (1024 * h >= LONG) == (h == 888)
        sa.sample_per_frame = spp
        if env:
            sa.env = scenes.sky_env(64, 32)
        s = sa.scene()
        s.build_accel()
        s.upload_to_device(0)
        s.update_settings(paths_in_flight=1024 * h)           # one sample a pass
        one = pt.render(s, spp)
        s.update_settings(paths_in_flight=spp * 1024 * h)     # all at once
        assert np.array_equal(pt.render(s, spp).view(np.uint32), one.view(np.uint32))
        assert np.isfinite(one).all() and one[..., :3].max() > 0


def test_guided_textured_shading_on_both_sides():
    sa = scenes.textured_cornell(width=512, height=512, spp=4, max_depth=5)
    sa.sample_per_frame = 4
    s = sa.scene()
    s.build_accel()
    s.upload_to_device(0)
    r = pt.Renderer(s)
    g = pt.Guide(s, seed=2)
    g.attach(r.integrator, pt.Guide.TRAIN)
    r.render_frames(2)
    g.attach(r.integrator, pt.Guide.USE)
    imgs = []
    for paths in (512 * 512, 4 * 512 * 512):                  # 262k slots: blocks of 256; 1M: of 1024
        s.update_settings(paths_in_flight=paths)
        r.reset_accumulation()
        r.render_frames(1)
        imgs.append(r.download_current_image())
    assert np.array_equal(imgs[0].view(np.uint32), imgs[1].view(np.uint32))

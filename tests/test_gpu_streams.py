"""Renders on a caller's stream: what its owner may capture, and what is refused."""
import numpy as np
import pytest

import pathtracingtutorial_b200 as pt
from pathtracingtutorial_b200 import scenes

pytestmark = pytest.mark.gpu


def _renderer(stream, flags=0):
    sa = scenes.cornell_box(width=64, height=48, spp=4, max_depth=4)
    sa.sample_per_frame = 4
    s = sa.scene()
    s.update_settings(flags=flags)
    s.build_accel()
    s.upload_to_device(0)
    return pt.Renderer(s, stream=stream)


def _image(r):
    import torch
    torch.cuda.synchronize()
    return r.download_current_image()


def test_a_captured_frame_replays():
    """PT_FLAG_NO_GRAPH: the caller's graph holds the frame, its shadow rays on the second stream included."""
    import torch
    st = torch.cuda.Stream()
    r = _renderer(st.cuda_stream, pt.FLAG_NO_GRAPH)
    r.render_batch()
    ref = _image(r)
    r.reset_accumulation()
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=st, capture_error_mode="thread_local"):
        r.render_batch()
    g.replay()
    assert np.array_equal(_image(r), ref) and ref[..., :3].max() > 0


@pytest.mark.parametrize("launches", [0, 1, 2, 3])
def test_a_captured_stream_is_refused_and_its_capture_left_alone(launches):
    import torch
    st = torch.cuda.Stream()
    r = _renderer(None)
    r.render_batch()
    torch.cuda.synchronize()
    r.stream = st.cuda_stream
    for _ in range(launches):
        r.render_batch()
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with pytest.warns(UserWarning, match="empty"):          # nothing of the refused launch is in it
        with torch.cuda.graph(g, stream=st, capture_error_mode="thread_local"):
            with pytest.raises(pt.PTError, match="captured"):
                r.render_batch()
    r.reset_accumulation()
    r.render_batch()                                        # and the stream renders as before
    one = _image(r)
    own = _renderer(None)
    own.render_batch()
    assert np.array_equal(one, _image(own))


def test_the_legacy_stream_is_refused_from_the_first_launch():
    r = _renderer(1)                                        # cudaStreamLegacy
    for _ in range(3):
        with pytest.raises(pt.PTError, match="captur"):
            r.render_batch()
    r.scene.update_settings(flags=pt.FLAG_NO_GRAPH)
    r.render_batch()
    assert _image(r)[..., :3].max() > 0

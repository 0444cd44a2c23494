"""The host-to-device bytes of bench.py's end-to-end figure are those of the
arrays that an upload copies."""
import pytest

from pathtracingtutorial_b200 import scenes


@pytest.mark.parametrize("make", [
    lambda: scenes.icosphere_field(n_spheres=5, subdiv=2, width=8, height=8, env_size=(32, 16)),
    lambda: scenes.icosphere_field(n_spheres=5, subdiv=2, width=8, height=8, env_size=None),
    lambda: scenes.cornell_box(width=8, height=8)])
def test_upload_bytes_are_the_arrays(make):
    import bench
    s = make().scene()
    s.build_accel()
    info = s.info()
    inner, tris, _ = s.traversal_layout()
    arrays = [inner, tris, s.vertices(), s.faces(), s.materials(), s.punctual_lights(), *s.emissive_tables()]
    env = info["env_width"] * info["env_height"]
    if env:
        arrays += s.env_tables()
    assert bench.upload_bytes(info) == sum(a.nbytes for a in arrays) + 16 * env

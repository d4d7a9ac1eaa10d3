"""The algorithmic bytes that bench.py charges next-event rays: by the scene's lights, not by the
workload's name, and no more than each ray moves."""
import dataclasses

from conftest import ROOT  # noqa: F401  (puts the repository's root on the path)


def test_next_event_bytes_follow_the_lights():
    import bench
    from mcrt_gb300 import scenes
    area = scenes.cfg0_scene(sphere_level=1)
    env = scenes.cfg1_scene(level=1, env_size=(16, 8))
    assert bench.next_event_io_bytes(env) == 32
    assert bench.next_event_io_bytes(area) == 80
    assert bench.next_event_io_bytes(dataclasses.replace(area, envmap=env.envmap)) == 32

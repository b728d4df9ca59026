"""The list of a convex target's pairs whose shadow tests are walked in a pass of
their own: the same masks with room for all of them, for a few and for none, and
one list for all masks of a scene.
"""
import numpy as np
import pytest

from test_gpu_mask_classes import _load

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name,khz", [("sphere2", 6.0), ("sphere4", 9.0), ("box", 9.0), ("sliver", 14.0)])
def test_a_full_list_keeps_the_masks(api, scenes, name, khz):
    got = []
    try:
        _load(api, scenes, name, khz * 1e3)
        for cap in (1 << 22, 33, 1, 0):
            api.set_option("mask_walk_cap", cap)
            got.append([api.get_mask(1, 0, 0), api.get_mask(3, 0, 0)])
    finally:
        api.set_option("mask_walk_cap", 1 << 22)
        api.TearDownCuda()
    for other in got[1:]:
        for a, b in zip(got[0], other):
            assert np.array_equal(a, b)


def test_one_list_for_all_field_objects(api, scenes):
    """Six field surfaces, each with a mask of more than 1,024 blocks: the pool
    holds one walk list (32 MB) beside some 12 MB of masks each, not six."""
    f = 12e3
    api.TearDownCuda()
    api.set_option("memory_cache_mb", 0)
    api.set_option("release_memory", 1)
    try:
        base = api.stats()["pool_reserved_bytes"]
        api.set_initial_conditions(1480.0, f, 0.0)
        api.load_stl_mesh_to_cuda(scenes.icosphere(3, 0.5), api.TARGET, scenes.delta_for(f))
        plane = scenes.rotate(scenes.rectangle(2.0, 2.0), "y", 90.0)
        for k in range(6):
            api.load_stl_mesh_to_cuda(scenes.rotate(plane, "x", 15.0 * k), api.FIELD, 2.0 / 80)
        api.load_points_to_cuda(np.array([[0.0, 0.0, 4.0]], np.float32), isSource=True)
        api.render_cuda()
        api.project_source_points_to_objects(False)
        api.project_target_to_field_objects()
        held = api.stats()["pool_reserved_bytes"] - base
        P = [api.get_object_pressures(api.FIELD, k) for k in range(6)]
    finally:
        api.TearDownCuda()
        api.set_option("memory_cache_mb", 32768)
    print("held %.0f MB" % (held / 1e6))
    assert all(np.linalg.norm(p) > 0 for p in P)
    assert 33e6 < held < 180e6

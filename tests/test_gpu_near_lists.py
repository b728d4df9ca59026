"""The near lists and margins of convex targets away from the origin, where E =
2e-6 (1 + vmax + sc) decides: masks with the shortcuts equal those of the
general path (every pair's test walks the whole ray) bit for bit.
"""
import numpy as np
import pytest

from test_gpu_mask_classes import CP, _targets

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name,khz", [("sphere2", 6.0), ("sphere4", 8.0), ("box", 8.0), ("sliver", 11.0)])
@pytest.mark.parametrize("shift", [7.0, 60.0, 400.0])
def test_shortcuts_keep_the_masks(api, scenes, name, khz, shift):
    f, move = khz * 1e3, (shift, -0.5 * shift, 0.25 * shift)
    t = scenes.translate(_targets(scenes, name), move)
    rng = np.random.default_rng(8)
    d = rng.normal(size=(611, 3))
    # near points and, every fourth, points at the distance of the origin
    r = np.where(np.arange(611) % 4 == 0, shift, rng.uniform(0.9, 2.5, 611))[:, None]
    fp = d / np.linalg.norm(d, axis=1, keepdims=True) * r + move
    plane = scenes.translate(scenes.rotate(scenes.rectangle(2.2, 1.9), "y", 90.0), move)
    got = {}
    try:
        api.TearDownCuda()
        api.set_initial_conditions(CP, f, 0.0)
        api.load_stl_mesh_to_cuda(t, api.TARGET, scenes.delta_for(f))
        api.load_stl_mesh_to_cuda(plane, api.FIELD, 2.2 / 41)
        api.load_points_to_cuda(np.array([[0.2, 0.1, 5.0]]) + move, isSource=True)
        api.load_points_to_cuda(fp, isSource=False)
        api.render_cuda()
        for fast in (1, 0):
            api.set_option("mask_classify", fast)
            api.set_option("convex_masks", fast)
            got[fast] = [api.get_mask(hop, 0, 0) for hop in (0, 1, 3)]
    finally:
        api.set_option("mask_classify", 1)
        api.set_option("convex_masks", 1)
        api.TearDownCuda()
    for hop, a, b in zip((0, 1, 3), got[1], got[0]):
        print("hop %d: %d pairs, %d interact, %d differ" % (hop, a.size, int(b.sum()), int((a != b).sum())))
    for a, b in zip(got[1], got[0]):
        assert b.any()
        assert np.array_equal(a, b)

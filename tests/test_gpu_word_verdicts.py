"""Shadow verdicts per 32-source word: the masks of every hop equal those of the
pair kernel that tests each pair by itself (mask_classify 0), bit for bit, at the
origin and where coordinates are large against the scene.
"""
import numpy as np
import pytest

from test_gpu_mask_classes import CP, _targets

pytestmark = pytest.mark.gpu


def _room(scenes):
    """Three plates of which each shadows parts of the others, one at a small
    angle to the rays between the other two."""
    a = scenes.rectangle(0.8, 0.6)
    b = scenes.translate(scenes.rotate(scenes.rectangle(0.7, 0.6), "y", 90.0), (-0.5, 0.0, 0.45))
    c = scenes.translate(scenes.rotate(scenes.rectangle(0.3, 0.25), "y", 47.0), (-0.2, 0.05, 0.25))
    return np.concatenate([a, b, c, c[:, [0, 1, 2, 6, 7, 8, 3, 4, 5]] - np.float32(0.002)])


@pytest.mark.parametrize("name,khz", [("room", 7.0), ("room", 11.0), ("trihedral", 9.0), ("plates", 7.0), ("dented", 5.0)])
@pytest.mark.parametrize("shift", [0.0, 25.0])
def test_word_verdicts_keep_the_masks(api, scenes, name, khz, shift):
    f, move = khz * 1e3, (shift, -shift, 0.5 * shift)
    t = scenes.translate(_room(scenes) if name == "room" else _targets(scenes, name), move)
    rng = np.random.default_rng(5)
    d = rng.normal(size=(611, 3))
    fp = d / np.linalg.norm(d, axis=1, keepdims=True) * rng.uniform(0.9, 2.5, (611, 1)) + move
    plane = scenes.translate(scenes.rotate(scenes.rectangle(2.2, 1.9), "y", 90.0), move)
    src = np.array([[0.2, 0.1, 5.0], [1.5, -0.4, 2.0], [-3.0, 0.2, 0.4]]) + move
    got = {}
    try:
        api.TearDownCuda()
        api.set_initial_conditions(CP, f, 0.0)
        api.load_stl_mesh_to_cuda(t, api.TARGET, scenes.delta_for(f))
        api.load_stl_mesh_to_cuda(plane, api.FIELD, 2.2 / 41)
        api.load_points_to_cuda(src, isSource=True)
        api.load_points_to_cuda(fp, isSource=False)
        api.render_cuda()
        for fast in (1, 0):
            api.set_option("mask_classify", fast)
            got[fast] = [api.get_mask(hop, 0, 0) for hop in (0, 1, 2, 3)]
    finally:
        api.set_option("mask_classify", 1)
        api.TearDownCuda()
    for hop, (a, b) in enumerate(zip(got[1], got[0])):
        print("hop %d: %d pairs, %d interact" % (hop, a.size, int(a.sum())))
        assert np.array_equal(a, b)
    assert all(m.any() for m in got[1])

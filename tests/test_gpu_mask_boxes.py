"""Blocks of a one-gate mask settled from their boxes when the scene has at most
32 triangles, around that count and away from the origin.

The decisions equal those of the general path bit for bit.  The fields of the
two routes differ by FP32 rounding only: each is within 1e-5 of FP64 (the
parity bound), so they are within 2e-5 of each other.
"""
import numpy as np
import pytest

from conftest import rel_l2

pytestmark = pytest.mark.gpu


# ntri: on both sides of 32 (a corner reflector and parts of its halved form);
# shift: coordinates that are large against the scene
@pytest.mark.parametrize("ntri,shift", [(3, 0.0), (12, 0.0), (31, 0.0), (32, 0.0), (33, 0.0), (12, 25.0)])
def test_box_verdicts_keep_the_masks(api, scenes, ntri, shift):
    f, move = 20e3, (shift, -shift, 0.0)
    t = scenes.trihedral(0.8)
    while len(t) < ntri:
        t = scenes.halve_facets(t)
    t = t[:ntri]
    rng = np.random.default_rng(3)
    d = rng.normal(size=(9001, 3))
    fp = d / np.linalg.norm(d, axis=1, keepdims=True) * rng.uniform(0.9, 2.5, (9001, 1)) + move
    plane = scenes.translate(scenes.rotate(scenes.rectangle(2.2, 1.9), "y", 90.0), move)
    got = {}
    try:
        for fast in (1, 0):
            api.TearDownCuda()
            api.set_option("mask_classify", fast)
            api.set_initial_conditions(1480.0, f, 0.0)
            api.load_stl_mesh_to_cuda(scenes.translate(t, move), api.TARGET, scenes.delta_for(f))
            api.load_stl_mesh_to_cuda(plane, api.FIELD, 2.2 / 41)
            api.load_points_to_cuda((np.array([[0.2, 0.1, 5.0]]) + move).astype(np.float32), isSource=True)
            api.load_points_to_cuda(fp.astype(np.float32), isSource=False)
            api.render_cuda()
            api.project_source_points_to_objects(False)
            api.project_target_to_field_points()
            got[fast] = api.get_mask(1, 0, 0), api.get_mask(3, 0, 0), api.get_field_point_pressures(len(fp))
    finally:
        api.set_option("mask_classify", 1)
        api.TearDownCuda()
    for a, b in zip(got[1][:2], got[0][:2]):
        assert b.any() and not b.all()
        assert np.array_equal(a, b)
    lit = np.abs(got[0][2]) > 0.0  # only points that some fragment sees
    assert np.isfinite(got[0][2]).all() and lit.any() and not (lit & ~got[0][0].reshape(len(fp), -1).any(axis=1)).any()
    e = rel_l2(got[1][2], got[0][2])
    print(len(t), "triangles, shift", shift, "field", e)
    assert e < 2e-5

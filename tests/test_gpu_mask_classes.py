"""Masks of the readout and of target -> field object: block classification by
the gate's range, per-word shadow verdicts, near lists of convex targets.

Every shortcut must give the verdict of the general path: the masks with the
classification and the convex-target shortcuts equal those without them bit
for bit, and the oracle's outside grazing pairs.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CP = 1480.0


def _targets(scenes, name):
    if name.startswith("sphere"):
        return scenes.icosphere(int(name[6:]), 0.5)
    if name == "dented":  # 1,280 triangles, one vertex pushed in: not convex
        t = scenes.icosphere(3, 0.5).reshape(-1, 3)
        t[np.linalg.norm(t - t[100], axis=1) < 1e-4] *= 0.8
        return t.reshape(-1, 9)
    if name == "box":
        return scenes.rotate(scenes.rotate(scenes.box(0.7, 0.5, 0.4), "y", 17.0), "z", 31.0)
    if name == "sliver":  # a flat wedge: small dihedral angles, long thin faces
        return scenes.rotate(scenes.create_plate_triangle(1.2, 0.5, 0.02), "x", 12.0)
    if name == "trihedral":
        return scenes.trihedral(0.8)
    return np.concatenate([scenes.rectangle(0.8, 0.6), scenes.rectangle(0.5, 0.3, z=0.25, normal_up=False)])


def _load(api, scenes, name, f):
    t = _targets(scenes, name)
    plane = scenes.rotate(scenes.rectangle(2.2, 1.9), "y", 90.0)  # through the target
    rng = np.random.default_rng(5)
    d = rng.normal(size=(611, 3))
    fp = (d / np.linalg.norm(d, axis=1, keepdims=True) * rng.uniform(0.9, 2.5, (611, 1))).astype(np.float32)
    src = np.array([[0.2, 0.1, 5.0]], np.float32)
    api.TearDownCuda()
    api.set_initial_conditions(CP, f, 0.0)
    api.load_stl_mesh_to_cuda(t, api.TARGET, scenes.delta_for(f))
    api.load_stl_mesh_to_cuda(plane, api.FIELD, 2.2 / 41)
    api.load_points_to_cuda(src, isSource=True)
    api.load_points_to_cuda(fp, isSource=False)
    api.render_cuda()
    return t, plane, src, fp


@pytest.mark.parametrize("name,khz", [("sphere1", 9.0), ("sphere2", 6.0), ("sphere3", 9.0), ("sphere4", 9.0),
                                      ("dented", 7.0), ("box", 9.0),
                                      ("sliver", 14.0), ("trihedral", 9.0), ("plates", 7.0)])
def test_shortcuts_keep_the_masks(api, scenes, name, khz):
    _load(api, scenes, name, khz * 1e3)
    got = {}
    try:
        for fast in (1, 0):
            api.set_option("mask_classify", fast)
            api.set_option("convex_masks", fast)
            got[fast] = [api.get_mask(1, 0, 0), api.get_mask(3, 0, 0)]
    finally:
        api.set_option("mask_classify", 1)
        api.set_option("convex_masks", 1)
        api.TearDownCuda()
    for a, b in zip(got[1], got[0]):
        assert b.any() and not b.all()
        assert np.array_equal(a, b)


@pytest.mark.parametrize("name,khz", [("sphere2", 5.0), ("dented", 4.0), ("box", 6.0), ("trihedral", 6.0), ("plates", 6.0)])
def test_masks_match_oracle(api, oracle_mod, scenes, name, khz):
    f = khz * 1e3
    t, plane, src, fp = _load(api, scenes, name, f)
    o = oracle_mod.Oracle()
    o.set_initial_conditions(CP, f, 0.0)
    o.load_geometry(t, 0, scenes.delta_for(f))
    o.load_geometry(plane, 2, 2.2 / 41)
    o.load_source_points(src)
    o.load_field_points(fp)
    o.render()
    for hop, n in ((1, len(fp)), (2, o.nact(0, 0)), (3, o.nact(2, 0))):
        got = api.get_mask(hop, 0, 0).reshape(n, -1)
        _, ref = o.hop_subset(hop, 0, 0, np.arange(n), want_mask=True, nsrc=o.nact(0, 0))
        ref = np.asarray(ref).reshape(n, -1)
        bad = (got != (ref & 1)) & ((ref & 2) == 0)
        print(name, "hop", hop, "pairs", got.size, "interacting", int(got.sum()), "mismatch", int(bad.sum()))
        assert not bad.any()
    o.close()
    api.TearDownCuda()

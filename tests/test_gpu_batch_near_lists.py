"""The near lists of batch plans: at every range the visibility they give is that
of the plans without them, so that the outputs are the same bit for bit (one
tile shape, so the sums run in the same order).
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _grazing(tris, rng, n, radius):
    """n points at about radius, most of them within a degree of the plane of a
    random facet, above the triangle's own region or outside it."""
    t = tris[rng.integers(0, len(tris), n)].reshape(n, 3, 3).astype(np.float64)
    u, w = rng.uniform(size=(2, n, 1))
    base = t[:, 0] + u * (t[:, 1] - t[:, 0]) + (1 - u) * w * (t[:, 2] - t[:, 0])
    nrm = np.cross(t[:, 1] - t[:, 0], t[:, 2] - t[:, 0])
    nrm /= np.linalg.norm(nrm, axis=1, keepdims=True)
    side = np.cross(nrm, rng.normal(size=(n, 3)))
    side /= np.linalg.norm(side, axis=1, keepdims=True)
    c = np.exp(rng.uniform(np.log(1e-3), np.log(3e-2), (n, 1)))  # cosines on both sides of the lists' range
    return (base + radius * rng.uniform(0.8, 1.2, (n, 1)) * (side * np.sqrt(1 - c * c) + nrm * c)).astype(np.float32)


@pytest.mark.parametrize("radius", [0.5, 3.0, 30.0, 45.0, 300.0, 3000.0])
@pytest.mark.parametrize("shift", [0.0, 20.0])
def test_lists_keep_the_verdicts(api, scenes, radius, shift):
    from sonar_render_gb300 import batch
    rng = np.random.default_rng(int(radius) + int(shift))
    targets = [scenes.icosphere(2, 0.4), scenes.icosphere(4, 0.3), scenes.rotate(scenes.box(0.5, 0.4, 0.3), "y", 21.0),
               scenes.rotate(scenes.create_plate_triangle(0.6, 0.3, 0.01), "x", 12.0)]
    targets = [scenes.translate(t, (shift, -shift, 0.5 * shift)) for t in targets]
    src = np.concatenate([_grazing(t, rng, 16, radius) for t in targets])
    rx = np.concatenate([_grazing(t, rng, 16, radius) for t in targets])
    out = []
    try:
        for on in (1, 0):
            api.set_option("batch_near_lists", on)
            p = batch.Plan(targets, src, rx, np.array([30e3], np.float32))
            p.set_shape(32, 2)
            out.append(p.run())
            if on:
                assert p.stats()["convex_scenes"] == len(targets)
            p.close()
    finally:
        api.set_option("batch_near_lists", 1)
    assert np.linalg.norm(out[0]) > 0
    assert np.array_equal(out[0], out[1])

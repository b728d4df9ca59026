"""The batch's visibility words near the terminator: gates decided by a margin,
near triangles and walks, against the single-scene path (whose masks equal the
oracle's outside grazing pairs).  Tolerance: the batch's 1e-4 (split BF16)."""
import numpy as np
import pytest

from conftest import rel_l2
from test_gpu_batch import TOL, library_columns

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nsrc,nrx", [(1, 1), (31, 33), (64, 64)])
def test_points_near_the_facet_planes(api, scenes, nsrc, nrx):
    """Points close to convex targets, many of them almost in a facet's plane;
    the point counts sit at the edges of the 32-point words."""
    from sonar_render_gb300 import batch
    rng = np.random.default_rng(3)
    n = nsrc + nrx
    d = rng.normal(size=(n, 3))
    p = d / np.linalg.norm(d, axis=1, keepdims=True) * rng.uniform(0.3, 2.0, (n, 1))
    flat = rng.random(n) < 0.5  # just above the plane of the box's top face
    p[flat, 1] = 0.04 + rng.uniform(1e-4, 3e-3, int(flat.sum()))
    p[0] = p[-1] = (0.1, 0.2, 1.0)
    p = p.astype(np.float32)
    src, rx, f = p[:nsrc], p[nsrc:], np.array([30e3], np.float32)
    targets = [scenes.box(0.12, 0.08, 0.10), scenes.icosphere(1, 0.06), scenes.icosphere(3, 0.05)]
    got = batch.Plan(targets, src, rx, f).run()
    cols = slice(0, min(nsrc, 3))
    for s, t in enumerate(targets):
        ref = library_columns(api, t, src[cols], rx, f[0])
        assert np.linalg.norm(ref) > 0
        assert rel_l2(got[s, 0][:, cols], ref) < TOL

"""Host-only check of the field points' order (sonar_point_order): the Morton
order at 2^21 steps to a side of the bounding box, points of one step in the
caller's order, whatever part of the box the points fill.
"""
import numpy as np
import pytest


def _codes(p):
    p = p.astype(np.float64)
    lo, ext = p.min(0), p.max(0) - p.min(0)
    q = (p - lo) * np.where(ext > 0, 2097151.0 / np.where(ext > 0, ext, 1.0), 0.0)
    q = np.minimum(q, 2097151.0).astype(np.uint64)
    code = np.zeros(len(p), np.uint64)
    for b in range(21):
        for k in range(3):
            code |= ((q[:, k] >> np.uint64(b)) & np.uint64(1)) << np.uint64(3 * b + k)
    return code


def _hemisphere(n, seed):
    rng = np.random.default_rng(seed)
    d = rng.normal(size=(n, 3))
    d[:, 2] = np.abs(d[:, 2])
    return (2.0 * d / np.linalg.norm(d, axis=1, keepdims=True)).astype(np.float32)


def _sets():
    rng = np.random.default_rng(1)
    far = np.array([[2500.0, -1700.0, 900.0]], np.float32)
    yield "one", _hemisphere(1, 0)
    yield "two", _hemisphere(2, 0)
    yield "hemisphere", _hemisphere(20000, 0)
    # all but one point in one step of a 1,024 grid: more and fewer than 2,048
    yield "outlier", np.concatenate([_hemisphere(5000, 2), far])
    yield "small outlier", np.concatenate([_hemisphere(700, 3), far])
    # several clusters, coincident points, a line, one point many times
    c = np.concatenate([_hemisphere(3000, 4) * 0.01 + x for x in ((0, 0, 0), (50, 0, 0), (50, 50, 9))] + [far])
    yield "clusters", c.astype(np.float32)[rng.permutation(len(c))]
    yield "coincident", np.repeat(_hemisphere(900, 5), 4, 0)[rng.permutation(3600)]
    yield "line", np.outer(np.linspace(-1, 1, 4001)[rng.permutation(4001)], (1, 0, 0)).astype(np.float32)
    yield "equal", np.tile(_hemisphere(1, 6), (3000, 1))


@pytest.mark.parametrize("name,points", list(_sets()), ids=[n for n, _ in _sets()])
def test_order_is_the_morton_order(api, name, points):
    assert np.array_equal(api.point_order(points), np.argsort(_codes(points), kind="stable"))


def test_clustered_points_keep_compact_blocks(api):
    """256-point blocks of a hemisphere stay as compact beside a far receiver as
    without it (1,024 steps to a side would leave the caller's random order)."""
    p = _hemisphere(20000, 7)
    sizes = []
    for pts in (p, np.concatenate([p, np.array([[2500.0, -1700.0, 900.0]], np.float32)])):
        o = api.point_order(pts)
        o = o[o < len(p)]
        blocks = [p[o[i:i + 256]] for i in range(0, len(p) - 255, 256)]
        sizes.append(np.median([np.linalg.norm(b.max(0) - b.min(0)) for b in blocks]))
    assert sizes[1] < 1.5 * sizes[0]


def test_invalid_arguments(api):
    assert len(api.point_order(np.zeros((0, 3)))) == 0
    with pytest.raises(api.SonarError):
        api.point_order([[np.nan, 0, 0], [0, 0, 0]])

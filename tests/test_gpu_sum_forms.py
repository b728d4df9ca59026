"""The packed sums (readout, target -> field object, target -> target) over the
forms they choose from: one-facet and mixed tiles, partial last tiles and odd
source counts, blocks with bits, gates taken from the plane distance, pairs
below the regularisation radius, words split over several CTAs, attenuation.

Bound: the parity tests' 1e-5 against FP64 with the reference's FP32 distances
(FP32 terms, phase to 2^-24 turns, FP32 tile sums: about 1e-6).
"""
import numpy as np
import pytest

from conftest import rel_l2

pytestmark = pytest.mark.gpu

CP = 1480.0


def _points(n, seed):
    rng = np.random.default_rng(seed)
    d = rng.normal(size=(n, 3))
    d[:, 2] = np.abs(d[:, 2]) * rng.choice([1.0, 1.0, -1.0], n)  # a third behind the target
    return (d / np.linalg.norm(d, axis=1, keepdims=True) * rng.uniform(0.4, 6.0, (n, 1))).astype(np.float32)


# khz and cuts set fragments per facet (delta: lambda / 7.5): a tile or less
# (2 kHz), several facets to a tile (cuts), about 60 tiles (18 kHz)
@pytest.mark.parametrize("khz,cuts,npts,att", [(2.0, 0, 1, 0.0), (5.0, 0, 257, 0.2), (7.0, 2, 300, 0.0),
                                              (9.0, 3, 511, 0.1), (18.0, 0, 33, 0.0), (18.0, 1, 1000, 0.05)])
def test_readout_and_field_object(api, oracle_mod, scenes, khz, cuts, npts, att):
    f = khz * 1e3
    t = scenes.rotate(scenes.rectangle(1.1, 0.9), "x", 9.0)
    for _ in range(cuts):
        t = scenes.halve_facets(t)
    delta = scenes.delta_for(f)
    src, fp = np.array([[0.3, -0.2, 4.0]], np.float32), _points(npts, 11)
    # a field surface that stands on the target: some of its cells are closer than delta
    field = scenes.translate(scenes.rotate(scenes.rectangle(0.5, 0.6), "y", 90.0), (0.03, 0.0, 0.31))
    api.TearDownCuda()
    api.set_initial_conditions(CP, f, att)
    api.load_stl_mesh_to_cuda(t, api.TARGET, delta)
    api.load_stl_mesh_to_cuda(field, api.FIELD, 0.017)
    api.load_points_to_cuda(src, isSource=True)
    api.load_points_to_cuda(fp, isSource=False)
    api.render_cuda()
    api.project_source_points_to_objects(False)
    P = api.get_object_pressures(api.TARGET, 0)
    api.project_target_to_field_points()
    api.project_target_to_field_objects()
    got = api.get_field_point_pressures(npts), api.get_object_pressures(api.FIELD, 0)
    api.TearDownCuda()
    o = oracle_mod.Oracle()
    o.set_initial_conditions(CP, f, att)
    o.load_geometry(t, 0, delta)
    o.load_geometry(field, 2, 0.017)
    o.load_source_points(src)
    o.load_field_points(fp)
    o.render()
    o.set_pressures(0, 0, P)
    o.project_field_points()
    o.project_field_objects()
    e = rel_l2(got[0], o.field_points()), rel_l2(got[1], o.pressures(2, 0))
    o.close()
    print("%.0f kHz, %d cuts, %d points: readout %.2e, field object %.2e" % (khz, cuts, npts, *e))
    assert max(e) < 1e-5


@pytest.mark.parametrize("khz,cuts,att", [(3.0, 0, 0.0), (6.0, 2, 0.1), (9.0, 0, 0.0)])
def test_cross_objects(api, oracle_mod, scenes, khz, cuts, att):
    f = khz * 1e3
    a = scenes.rectangle(0.8, 0.6)
    b = scenes.translate(scenes.rotate(scenes.rectangle(0.7, 0.6), "y", 90.0), (-0.4, 0.0, 0.36))
    for _ in range(cuts):
        a, b = scenes.halve_facets(a), scenes.halve_facets(b)
    delta, src = scenes.delta_for(f), np.array([[4.0, 0.3, 5.0]], np.float32)
    api.TearDownCuda()
    api.set_option("cross_objects", 1)
    try:
        api.set_initial_conditions(CP, f, att)
        for m in (a, b):
            api.load_stl_mesh_to_cuda(m, api.TARGET, delta)
        api.load_points_to_cuda(src, isSource=True)
        api.render_cuda()
        api.project_source_points_to_objects(False)
        api.project_target_to_target_objects(2)
        P = [api.get_object_pressures(api.TARGET, i) for i in (0, 1)]
    finally:
        api.set_option("cross_objects", 0)
        api.TearDownCuda()
    o = oracle_mod.Oracle()
    o.set_initial_conditions(CP, f, att)
    for m in (a, b):
        o.load_geometry(m, 0, delta)
    o.load_source_points(src)
    o.render()
    o.project_sources(False)
    o.project_bounces(2, True)
    e = [rel_l2(P[i], o.pressures(0, i)) for i in (0, 1)]
    o.close()
    print("%.0f kHz, %d cuts: %.2e %.2e" % (khz, cuts, *e))
    assert max(e) < 1e-5


def test_non_finite_pressure_stays_with_its_pairs(api, scenes):
    """An infinite pressure on one facet reaches the points in front of that
    facet and no others (the pairs that do not interact are left out, not
    multiplied by zero)."""
    f = 9e3
    t = scenes.rotate(scenes.box(0.6, 0.5, 0.4), "z", 10.0)
    fp = np.array([[0.0, 0.0, 3.0], [0.0, 0.0, -3.0]], np.float32)
    api.TearDownCuda()
    api.set_initial_conditions(CP, f, 0.0)
    api.load_stl_mesh_to_cuda(t, api.TARGET, scenes.delta_for(f))
    # a source on the first cell of the top face: its pressure there is not finite
    frame = [api.fragment_triangle(x, scenes.delta_for(f)) for x in t]
    top = int(np.argmax([fr[1][2] for fr in frame]))
    (nx, _, neg), fr, _ = frame[top]
    d = np.float32(scenes.delta_for(f))
    xo = np.float32(d * np.float32(nx // 2 - neg)) + d / np.float32(2)
    p = (fr[3:6] + fr[6:9] * xo) + fr[9:12] * (d / np.float32(2))
    api.load_points_to_cuda(np.array([p, [0.0, 0.0, -4.0]], np.float32), isSource=True)
    api.load_points_to_cuda(fp, isSource=False)
    api.render_cuda()
    api.project_source_points_to_objects(False)
    P = api.get_object_pressures(api.TARGET, 0)
    api.project_target_to_field_points()
    got = api.get_field_point_pressures(2)
    api.TearDownCuda()
    if np.isfinite(P).all():
        pytest.skip("no cell coincides with the source")
    assert not np.isfinite(got[0])
    assert np.isfinite(got[1]) and abs(got[1]) > 0

"""The symmetric bounce sum's block forms: planar blocks (both factors of the
cosines taken out of the pair loop), general blocks (per-pair bits, gates,
tiles of several facets) and scalar ones (the diagonal, blocks at the
regularisation radius), over the work-list shapes that the problem size picks:
blocks cut into word ranges, one block to a chunk, several.

Bounds: FP32 terms with a phase reduced to 2^-24 turns and FP32 tile sums give
about 1e-6 of an FP64 evaluation with the same FP32 distances; the parity
tests' 1e-5 leaves a factor of ten.
"""
import numpy as np
import pytest

from conftest import rel_l2

pytestmark = pytest.mark.gpu

CP = 1480.0


def _bounce(api, tris, delta, f, att, n, sym=1):
    api.TearDownCuda()
    api.set_option("f2f_symmetric", sym)
    try:
        api.set_initial_conditions(CP, f, att)
        api.load_stl_mesh_to_cuda(tris, api.TARGET, delta)
        api.load_points_to_cuda(np.array([[4.0, 4.5, 3.5]], np.float32), isSource=True)
        api.render_cuda()
        api.project_source_points_to_objects(False)
        P0 = api.get_object_pressures(api.TARGET, 0)
        api.project_target_to_target_objects(n)
        P = api.get_object_pressures(api.TARGET, 0)
    finally:
        api.set_option("f2f_symmetric", 1)
        api.TearDownCuda()
    return P0, P


# frequency sets the fragment count (trihedral: 1.5 m^2 / delta^2): one tile,
# a few with a partial last one, 22 and 50 tiles; facets cut in four put
# several facets into a tile; coarse fragments (delta 6 cm) reach r_min often
@pytest.mark.parametrize("khz,cuts,att,per_wl", [(2.3, 0, 0.0, 7.5), (5.0, 0, 0.3, 7.5), (12.0, 0, 0.0, 7.5),
                                                (12.0, 2, 0.0, 7.5), (9.0, 3, 0.4, 7.5), (18.0, 0, 0.1, 7.5),
                                                (18.0, 1, 0.0, 7.5), (8.0, 0, 0.0, 3.0)])
def test_bounces_match_oracle(api, oracle_mod, scenes, khz, cuts, att, per_wl):
    f = khz * 1e3
    tris = scenes.trihedral(1.0)
    for _ in range(cuts):
        tris = scenes.halve_facets(tris)
    delta = scenes.delta_for(f, per_wavelength=per_wl)
    _, P = _bounce(api, tris, delta, f, att, 2)
    o = oracle_mod.Oracle()
    o.set_initial_conditions(CP, f, att)
    o.load_geometry(tris, 0, delta)
    o.load_source_points(np.array([[4.0, 4.5, 3.5]], np.float32))
    o.render()
    o.project_sources(False)
    o.project_bounces(2)
    err = rel_l2(P, o.pressures(0, 0))
    o.close()
    print("%.1f kHz, %d cuts, att %.1f: %.2e" % (khz, cuts, att, err))
    assert err < 1e-5


@pytest.mark.parametrize("khz,att", [(30.0, 0.0), (41.0, 0.05)])
def test_bounces_match_ordered_sum(api, scenes, khz, att):
    """Several blocks to a chunk (about 140 and 260 tiles), against the ordered
    sum, which evaluates every pair by itself."""
    f = khz * 1e3
    out = [_bounce(api, scenes.trihedral(1.0), scenes.delta_for(f), f, att, 2, sym) for sym in (1, 0)]
    err = rel_l2(out[0][1] - out[0][0], out[1][1] - out[1][0])
    print("%.0f kHz: symmetric against ordered %.2e" % (khz, err))
    assert err < 1e-5

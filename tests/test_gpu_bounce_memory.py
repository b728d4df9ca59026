"""The bounce sum's partial arrays: no larger than two blocks to a chunk need in
large problems, and the sum where that limit takes effect.
"""
import numpy as np
import pytest

from conftest import rel_l2

pytestmark = pytest.mark.gpu

CP = 1480.0


@pytest.mark.parametrize("f,khz", [(0.0, 41.0), (41e3, 41.0)])
def test_partials_and_result(api, scenes, f, khz):
    """About 260 tiles.  Without a wave number every block is a general one, one
    to a chunk: 22,000 chunks, more than the limit; with one most are planar.
    Bound: FP32 terms, the parity tests' 1e-5."""
    out = {}
    for sym in (1, 0):
        api.TearDownCuda()
        api.set_option("f2f_symmetric", sym)
        try:
            api.set_initial_conditions(CP, f, 0.0)
            api.load_stl_mesh_to_cuda(scenes.trihedral(1.0), api.TARGET, scenes.delta_for(khz * 1e3))
            api.load_points_to_cuda(np.array([[4.0, 4.5, 3.5]], np.float32), isSource=True)
            api.render_cuda()
            n = int((api.get_fragment_layout(api.TARGET, 0)[1] > 1e-6).sum())
            api.project_source_points_to_objects(False)
            P0 = api.get_object_pressures(api.TARGET, 0)
            api.project_target_to_target_objects(1)
            out[sym] = api.get_object_pressures(api.TARGET, 0) - P0
            if sym:
                nt = (n + 255) // 256
                used = api.stats()["bounce_partial_bytes"]
                chunks = max(sum((J + 1) // 2 + 1 for J in range(nt)), 1 << 14)
                assert nt > 250 and used <= 16 * 256 * (chunks + nt * (nt - 1) // 2)
        finally:
            api.set_option("f2f_symmetric", 1)
            api.TearDownCuda()
    err = rel_l2(out[1], out[0])
    print("%d tiles: symmetric against ordered %.2e" % (nt, err))
    assert np.abs(out[0]).max() > 0 and err < 1e-5

"""sonar_readout_noalloc against a plain FP64 sum with the reference's FP32
distances and gates, over the sizes and inputs that pick its forms: odd and
tiny counts, one word to many splits, wave numbers the packed form refuses,
points behind fragments, fragments without area or weight, coincident points
and pressures that are not finite.  Bound: the parity tests' 1e-5.
"""
import ctypes as C

import numpy as np
import pytest

from conftest import rel_l2

pytestmark = pytest.mark.gpu


def _entry(api):
    fn = api.lib().sonar_readout_noalloc
    fn.argtypes = [C.c_void_p, C.c_void_p, C.c_void_p, C.c_int, C.c_void_p, C.c_int, C.c_float, C.c_float, C.c_void_p,
                   C.c_void_p]
    fn.restype = C.c_int
    return fn


def _inputs(n, m, seed):
    rng = np.random.default_rng(seed)
    pos = np.concatenate([rng.uniform(-0.7, 0.7, (n, 3)), rng.uniform(1e-5, 4e-4, (n, 1))], 1).astype(np.float32)
    nrm = rng.normal(size=(n, 3))
    nrm = np.concatenate([nrm / np.linalg.norm(nrm, axis=1, keepdims=True), np.zeros((n, 1))], 1).astype(np.float32)
    pres = rng.normal(size=(n, 2))
    pos[rng.random(n) < 0.1, 3] = 1e-7  # below the area gate
    pres[rng.random(n) < 0.1] = 0.0
    pts = np.zeros((m, 4), np.float32)
    d = rng.normal(size=(m, 3))
    pts[:, :3] = d / np.linalg.norm(d, axis=1, keepdims=True) * rng.uniform(1.0, 6.0, (m, 1))
    return pos, nrm, pres, pts


def _reference(pos, nrm, pres, pts, kr, ki):
    f = np.float32
    out = np.zeros(len(pts), np.complex128)
    p = pres[:, 0] + 1j * pres[:, 1]
    on = (pos[:, 3] > f(1e-6)) & (p != 0)
    for j, q in enumerate(pts):
        with np.errstate(all="ignore"):
            v = q[None, :3] - pos[:, :3]
            r = np.sqrt((v[:, 0] * v[:, 0] + v[:, 1] * v[:, 1]) + v[:, 2] * v[:, 2])
            u = v * (f(1) / r)[:, None]
            c = (u[:, 0] * nrm[:, 0] + u[:, 1] * nrm[:, 1]) + u[:, 2] * nrm[:, 2]
            s = on & ~(c < f(1e-6))
            rd = r.astype(np.float64)[s]
            g = -np.exp((1j * kr - ki) * rd) / (4 * np.pi) * ((1j * kr - ki) / rd) + 1 / (rd * rd)
        out[j] = (pos[s, 3].astype(np.float64) * c[s].astype(np.float64) * p[s] * g).sum()
    return out


def _run(api, pos, nrm, pres, pts, kr, ki):
    import torch
    t = [torch.from_numpy(np.ascontiguousarray(x)).cuda() for x in (pos, nrm, pres, pts)]
    out = torch.full((len(pts), 2), 0.5, dtype=torch.float64, device="cuda")  # accumulated onto
    rc = _entry(api)(t[0].data_ptr(), t[1].data_ptr(), t[2].data_ptr(), len(pos), t[3].data_ptr(), len(pts), kr, ki,
                     out.data_ptr(), torch.cuda.current_stream().cuda_stream)
    assert rc == 0
    torch.cuda.synchronize()
    o = out.cpu().numpy() - 0.5
    return o[:, 0] + 1j * o[:, 1]


@pytest.mark.parametrize("n,m", [(1, 1), (2, 300), (31, 7), (33, 257), (257, 1), (1271, 181), (4099, 40), (70001, 3)])
@pytest.mark.parametrize("kr,ki", [(42.5, 0.0), (127.0, 0.3), (20.0, -0.05), (0.0, 0.1)])
def test_sizes_and_wave_numbers(api, n, m, kr, ki):
    x = _inputs(n, m, 100 * n + m)
    kr, ki = float(np.float32(kr)), float(np.float32(ki))
    got, ref = _run(api, *x, kr, ki), _reference(*x, kr, ki)
    assert rel_l2(got, ref) < 1e-5


def test_non_finite_and_coincident_inputs(api):
    pos, nrm, pres, pts = _inputs(300, 4, 5)
    pos[:, 2] = 0.0
    nrm[:] = (0, 0, 1, 0)
    pos[:, 3] = 1e-4
    pts[:, :3] = [(0.1, 0.2, 3.0), (0.3, -0.1, -2.0), (0.0, 0.1, 2.5), (0.0, 0.0, -4.0)]
    nrm[7] = (0, 0, -1, 0)
    pres[7] = np.nan  # faces down: reaches the points below only
    got = _run(api, pos, nrm, pres, pts, 30.0, 0.0)
    assert np.isfinite(got[[0, 2]]).all() and not np.isfinite(got[[1, 3]]).any()
    pos, nrm, pres, pts = _inputs(64, 2, 6)
    pres[3] = (1.0, 0.0)
    pos[3, 3] = 1e-4
    pts[1, :3] = pos[3, :3]  # r = 0: the reference's 0 / 0 passes its gate
    got = _run(api, pos, nrm, pres, pts, 30.0, 0.0)
    assert np.isfinite(got[0]) and not np.isfinite(got[1])
    pos[3, 3] = 1e-7  # the same fragment without area: skipped
    assert np.isfinite(_run(api, pos, nrm, pres, pts, 30.0, 0.0)).all()

"""sonar_readout_noalloc where sums leave FP32's range: an infinite pressure
gives an infinite sum of its term's sign (not NaN), and tile sums of 1e38 add up
in FP64.  Bound of the second: the parity tests' 1e-5.
"""
import numpy as np
import pytest

from test_gpu_noalloc_forms import _entry, _reference

pytestmark = pytest.mark.gpu


def _run(api, pos, nrm, pres, pts, kr, ki):
    import torch
    t = [torch.from_numpy(np.ascontiguousarray(x)).cuda() for x in (pos, nrm, pres, pts)]
    out = torch.zeros((len(pts), 2), dtype=torch.float64, device="cuda")
    rc = _entry(api)(t[0].data_ptr(), t[1].data_ptr(), t[2].data_ptr(), len(pos), t[3].data_ptr(), len(pts), kr, ki,
                     out.data_ptr(), torch.cuda.current_stream().cuda_stream)
    assert rc == 0
    torch.cuda.synchronize()
    return out.cpu().numpy().view(np.complex128).ravel()  # (1j times an infinite float has a NaN)


def _grid(n, m):
    """n fragments facing +z in a 10 cm square, m points 3 to 3.1 m above."""
    rng = np.random.default_rng(4)
    pos = np.concatenate([rng.uniform(-0.05, 0.05, (n, 2)), np.zeros((n, 1)), np.full((n, 1), 1e-4)], 1).astype(np.float32)
    nrm = np.tile(np.array([0, 0, 1, 0], np.float32), (n, 1))
    pts = np.concatenate([rng.uniform(-0.1, 0.1, (m, 2)), rng.uniform(3.0, 3.1, (m, 1)), np.zeros((m, 1))], 1)
    return pos, nrm, rng.normal(size=(n, 2)), pts.astype(np.float32)


@pytest.mark.parametrize("n,m,ki", [(1, 3, 0.0), (700, 300, 0.0), (700, 5, 0.2)])
def test_infinite_pressure(api, n, m, ki):
    pos, nrm, pres, pts = _grid(n, m)
    kr, ki = 40.0, float(np.float32(ki))
    v = pts[:, :3].astype(np.float64) - pos[n // 2, :3]
    r = np.linalg.norm(v, axis=1)
    g = -np.exp((1j * kr - ki) * r) / (4 * np.pi) * (1j * kr - ki) / r + 1 / (r * r)
    clear = (np.abs(g.real) > 1e-3 * np.abs(g)) & (np.abs(g.imag) > 1e-3 * np.abs(g))
    assert clear.any()
    for sign in (1.0, -1.0):
        pres[n // 2] = (sign * np.inf, 0.0)
        got = _run(api, pos, nrm, pres, pts, kr, ki)
        assert np.array_equal(got.real[clear], (sign * np.sign(g.real) * np.inf)[clear])
        assert np.array_equal(got.imag[clear], (sign * np.sign(g.imag) * np.inf)[clear])


def test_sum_beyond_fp32(api):
    """Thirteen splits (the scratch holds no more for so many points) of 2 or 3
    tiles whose sums are near 2e38."""
    pos, nrm, pres, pts = _grid(30 * 256, 40000)
    pres[:] = 0.0
    pres[:, 0] = 1.6e40
    kr = 15.0
    idx = np.arange(0, len(pts), 1999)
    got, ref = _run(api, pos, nrm, pres, pts, kr, 0.0)[idx], _reference(pos, nrm, pres, pts[idx], kr, 0.0)
    tiles = np.array([_reference(pos[i:i + 256], nrm[i:i + 256], pres[i:i + 256], pts[idx], kr, 0.0)
                      for i in range(0, len(pos), 256)])
    assert np.abs(tiles).max() < 2.5e38 and np.maximum(np.abs(ref.real), np.abs(ref.imag)).min() > 4e38
    assert np.isfinite(got).all()
    assert np.linalg.norm((got - ref) * 1e-39) < 1e-5 * np.linalg.norm(ref * 1e-39)


@pytest.mark.parametrize("kr,scale", [(1e-3, 1e37), (1e-6, 1e35), (30.0, 1e38)])
def test_terms_near_the_range(api, kr, scale):
    """Sums within FP32 that would leave it divided by k / (4 pi)."""
    pos, nrm, pres, pts = _grid(700, 40)
    kr = float(np.float32(kr))
    pres *= scale / 1e-4 / 700
    got, ref = _run(api, pos, nrm, pres, pts, kr, 0.0), _reference(pos, nrm, pres, pts, kr, 0.0)
    assert np.isfinite(got.real).all() and np.isfinite(got.imag).all()
    assert np.linalg.norm((got - ref) / scale) < 1e-5 * np.linalg.norm(ref / scale)

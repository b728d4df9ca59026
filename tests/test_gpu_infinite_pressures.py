"""Infinite pressures by value: a sum with one infinite term is infinite with
that term's sign, as in an FP64 accumulator, and not NaN.

One component of one cell's pressure gets infinite by a growing wave (negative
attenuation) from many sources in one place, whose finite terms add up beyond
FP32 there alone (the growth is chosen so that this component is 2 % over the
largest FP32 value and the next largest 2 % below it; rounding is below 0.1 %).
The hop under test runs without attenuation.  Its infinities then have the
signs of G's parts, checked where these and the cosines are clear of zero (1e-3,
FP32 rounding is below 1e-5), away from the few cells that are nearly infinite.
"""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CP, FMAX, NSRC = 1480.0, 3.4028e38, 64


def _k(f):
    return np.float64(np.float32(np.float32(2 * np.pi * f) / np.float32(CP)))


def _field_points(api, n):
    """GetFieldPointPressures, the real and imaginary parts as they are (1j times
    an infinite float is not)."""
    out = np.zeros((n, 2))
    api.lib().GetFieldPointPressures(out.ctypes.data_as(ctypes.POINTER(ctypes.c_double)), n)
    return out.view(np.complex128).ravel()


class Cells:
    """Normal, readout and source-hop centroid and area of every cell, in the
    pressures' order (centroids to about 1e-6 m)."""

    def __init__(self, api, tris, delta):
        n, c, s, a = [], [], [], []
        d = np.float64(np.float32(delta))
        for t in tris:
            (nx, ny, neg), fr, area = api.fragment_triangle(t, delta)
            fr = fr.astype(np.float64)
            y, x = np.mgrid[0:ny, 0:nx]
            x, y = x.ravel(), y.ravel()
            p = fr[3:6] + np.outer(d * (x - neg), fr[6:9]) + np.outer(d * y + d / 2, fr[9:12])
            c.append(p)
            s.append(p + fr[6:9] * d / 2)
            n.append(np.tile(fr[0:3], (nx * ny, 1)))
            a.append(area.ravel())
        self.n, self.c, self.s = np.concatenate(n), np.concatenate(c), np.concatenate(s)
        self.area = np.concatenate(a).astype(np.float64)
        self.on = self.area > 1e-6


def _growth(cells, src, f):
    """Attenuation (negative) that makes one component of one cell infinite, and
    that cell, or None."""
    v = src - cells.s
    r = np.linalg.norm(v, axis=1)
    q = np.where((v * cells.n).sum(1) > 0, NSRC * (v * cells.n).sum(1) / r**2, 0.0) * np.exp(1j * _k(f) * r)
    q = np.stack([np.abs(q.real), np.abs(q.imag)], 1)
    q[~cells.on] = 0.0
    a = 80.0 / r.max()
    for _ in range(60):  # the largest component 4 % over the largest FP32 value
        e = q * np.exp(a * r)[:, None]
        a += np.log(1.04 * FMAX / e.max()) / r[np.unravel_index(e.argmax(), e.shape)[0]]
    e = np.sort((q * np.exp(a * r)[:, None]).ravel())[::-1]
    bad = int(np.unravel_index((q * np.exp(a * r)[:, None]).argmax(), q.shape)[0])
    return (a, bad) if e[0] > 1.02 * FMAX and e[1] < 0.98 * FMAX and a * r[cells.on].max() < 88.6 else None


def _infinite_cell(api, f, cells, src):
    """Source hop after which one active cell's pressure has an infinite part."""
    a, bad = _growth(cells, src, f)
    api.set_initial_conditions(CP, f, -a)
    api.project_source_points_to_objects(False)
    api.set_initial_conditions(CP, f, 0.0)
    P = api.get_object_pressures(api.TARGET, 0)
    assert list(np.flatnonzero(~np.isfinite(P) & cells.on)) == [bad]
    assert np.isinf(P[bad].real) != np.isinf(P[bad].imag) and not np.isnan(P[bad])
    return bad, P[bad]


def _check(got, cells, bad, p, f, dst, rmin, dst_n=None):
    """Signs of the infinities that the cell's pressure p leaves at dst."""
    v = dst - cells.c[bad]
    r = np.linalg.norm(v, axis=1)
    g = -np.exp(1j * _k(f) * r) / (4 * np.pi) * 1j * _k(f) / r + 1 / (r * r)
    ok = ((v @ cells.n[bad]) / r > 1e-3) & (r > rmin)
    if dst_n is not None:
        ok &= -(v * dst_n).sum(1) / r > 1e-3
    ok &= (np.abs(g.real) > 1e-3 * np.abs(g)) & (np.abs(g.imag) > 1e-3 * np.abs(g))
    if np.isinf(p.real):
        re, im = np.sign(g.real * p.real), np.sign(g.imag * p.real)
    else:
        re, im = -np.sign(g.imag * p.imag), np.sign(g.real * p.imag)
    assert np.array_equal(got.real[ok], re[ok] * np.inf) and np.array_equal(got.imag[ok], im[ok] * np.inf)
    return int(ok.sum())


# a few tiles with their words split over CTAs, tiles of several facets, one tile to a split
READOUT = [(8.0, 0, (0.7, 0.45, 3.0)), (8.0, 2, (0.7, 0.45, 3.0)), (16.0, 0, (0.7, 0.45, 3.0))]


def _readout_mesh(scenes, cuts):
    t = scenes.rotate(scenes.rotate(scenes.rectangle(1.1, 0.9), "x", 7.0), "z", 13.0)
    for _ in range(cuts):
        t = scenes.halve_facets(t)
    return t


@pytest.mark.parametrize("khz,cuts,src", READOUT)
def test_readout_and_field_object(api, scenes, khz, cuts, src):
    f, src, t = khz * 1e3, np.array(src), _readout_mesh(scenes, cuts)
    fp = (np.random.default_rng(2).uniform(-1, 1, (300, 3)) * (1, 1, 0) + (0, 0, 1.5)).astype(np.float32)
    # facing the target, so that its active cells are the lit ones
    field = scenes.translate(scenes.rectangle(0.6, 0.5, normal_up=False), (0.1, 0.0, 0.9))
    delta = scenes.delta_for(f)
    cells, fcells = Cells(api, t, delta), Cells(api, field, 0.05)
    api.TearDownCuda()
    try:
        api.set_initial_conditions(CP, f, 0.0)
        api.load_stl_mesh_to_cuda(t, api.TARGET, delta)
        api.load_stl_mesh_to_cuda(field, api.FIELD, 0.05)
        api.load_points_to_cuda(np.tile(src, (NSRC, 1)), isSource=True)
        api.load_points_to_cuda(fp, isSource=False)
        api.render_cuda()
        bad, p = _infinite_cell(api, f, cells, src)
        api.project_target_to_field_points()
        api.project_target_to_field_objects()
        points, surface = _field_points(api, len(fp)), api.get_object_pressures(api.FIELD, 0)
    finally:
        api.TearDownCuda()
    assert _check(points, cells, bad, p, f, fp, 0.3) > 200
    assert _check(surface[fcells.on], cells, bad, p, f, fcells.c[fcells.on], 0.3) > 60


# blocks cut into words, one block to a chunk, several; tiles of several faces
BOUNCE = [(5.0, 0, (0.1, 1.2, 2.4)), (12.0, 0, (0.25, 0.74, 3.45)), (12.0, 2, (0.73, -0.07, 3.14)),
          (18.0, 1, (0.1, 1.2, 2.4))]


def _bounce_mesh(scenes, cuts):
    """A floor between two walls in the facets' order: the terms of the floor
    reach one wall forwards, the other by reciprocity."""
    t = np.concatenate([scenes.translate(scenes.rotate(scenes.rectangle(0.8, 0.7), "y", 90.0), (-0.5, 0.02, 0.45)),
                        scenes.rectangle(0.9, 0.7),
                        scenes.translate(scenes.rotate(scenes.rectangle(0.8, 0.6), "x", -90.0), (0.03, -0.4, 0.36))])
    for _ in range(cuts):
        t = scenes.halve_facets(t)
    return t


@pytest.mark.parametrize("khz,cuts,src", BOUNCE)
def test_bounce(api, scenes, khz, cuts, src):
    f, src, t = khz * 1e3, np.array(src), _bounce_mesh(scenes, cuts)
    delta = scenes.delta_for(f)
    cells = Cells(api, t, delta)
    api.TearDownCuda()
    try:
        api.set_initial_conditions(CP, f, 0.0)
        api.load_stl_mesh_to_cuda(t, api.TARGET, delta)
        api.load_points_to_cuda(np.tile(src, (NSRC, 1)), isSource=True)
        api.render_cuda()
        bad, p = _infinite_cell(api, f, cells, src)
        assert cells.n[bad][2] > 0.9
        api.project_target_to_target_objects(1)
        got = api.get_object_pressures(api.TARGET, 0)
    finally:
        api.TearDownCuda()
    on = cells.on & (np.abs(cells.n[:, 2]) < 0.5)
    assert _check(got[on], cells, bad, p, f, cells.c[on], 0.3, cells.n[on]) > 0.8 * on.sum()


def test_sum_beyond_fp32(api, scenes):
    """Tile sums within FP32 whose total is beyond it, in one split: FP64 holds
    the total.  Pressures of 2e38, nearly in phase (a far source), and a point so
    close that the 1 / r^2 term adds them up.  Bound: the parity tests' 1e-5."""
    f, src = 3e3, np.array([0.0, 0.0, 30.0])
    t, point = scenes.rectangle(1.1, 0.9), np.array([0.02, -0.03, 0.3])
    delta = scenes.delta_for(9e3)
    cells = Cells(api, t, delta)
    a = 88.6 / np.linalg.norm(cells.s - src, axis=1).max()
    api.TearDownCuda()
    api.set_option("split", 1)
    try:
        api.set_initial_conditions(CP, f, -a)
        api.load_stl_mesh_to_cuda(t, api.TARGET, delta)
        api.load_points_to_cuda(np.tile(src, (24, 1)), isSource=True)
        api.load_points_to_cuda(point[None], isSource=False)
        api.render_cuda()
        api.project_source_points_to_objects(False)
        api.set_initial_conditions(CP, f, 0.0)
        P = api.get_object_pressures(api.TARGET, 0)
        api.project_target_to_field_points()
        got = _field_points(api, 1)[0]
    finally:
        api.set_option("split", 0)
        api.TearDownCuda()
    assert np.isfinite(P[cells.on]).all()
    v = point - cells.c[cells.on]
    r = np.linalg.norm(v, axis=1)
    g = -np.exp(1j * _k(f) * r) / (4 * np.pi) * 1j * _k(f) / r + 1 / (r * r)
    term = cells.area[cells.on] * g * (v * cells.n[cells.on]).sum(1) / r * P[cells.on]
    ref = term.sum()
    print("sum %.3e, largest term %.1e" % (abs(ref), np.abs(term).max()))
    assert max(abs(ref.real), abs(ref.imag)) > 4e38 and np.abs(term).max() < 1e37
    assert np.isfinite(got.real) and np.isfinite(got.imag)
    assert abs(got - ref) < 1e-5 * abs(ref)


@pytest.mark.parametrize("f", [300.0, 3e3, 12e3])
def test_bounce_near_the_range(api, scenes, f):
    """Sums within FP32 whose terms would leave it without the factors k / (4 pi)
    and the plane distances: pressures of 2e38 against the FP64 sum over all
    pairs.  Bound: the parity tests' 1e-5."""
    src, t, delta = np.array([8.0, 9.0, 27.0]), _bounce_mesh(scenes, 0), scenes.delta_for(12e3)
    cells = Cells(api, t, delta)
    a = 88.6 / np.linalg.norm(cells.s - src, axis=1).max()
    api.TearDownCuda()
    try:
        api.set_initial_conditions(CP, f, -a)
        api.load_stl_mesh_to_cuda(t, api.TARGET, delta)
        api.load_points_to_cuda(np.tile(src, (24, 1)), isSource=True)
        api.render_cuda()
        api.project_source_points_to_objects(False)
        api.set_initial_conditions(CP, f, 0.0)
        P = api.get_object_pressures(api.TARGET, 0)
        api.project_target_to_target_objects(1)
        got = (api.get_object_pressures(api.TARGET, 0) - P)[cells.on]
    finally:
        api.TearDownCuda()
    c, n, w = cells.c[cells.on], cells.n[cells.on], 0.9 * cells.area[cells.on] * P[cells.on]
    ref = np.zeros(len(c), np.complex128)
    for j in range(len(c)):
        v = c[j] - c
        r = np.linalg.norm(v, axis=1) + (np.arange(len(c)) == j)
        cs, ci = (v * n).sum(1) / r, -(v @ n[j]) / r
        on = (cs > 1e-6) & (ci > 1e-6) & (n @ n[j] < 0.5)
        r = r[on]
        g = -np.exp(1j * _k(f) * r) / (4 * np.pi) * 1j * _k(f) / r + 1 / (r * r)
        ref[j] = (g * cs[on] * ci[on] * w[on]).sum()
    assert 1e37 < np.abs(ref).max() < 3e38
    assert np.isfinite(got.real).all() and np.isfinite(got.imag).all()
    err = np.linalg.norm((got - ref) * 1e-38) / np.linalg.norm(ref * 1e-38)
    print("%.0f Hz: largest %.1e, error %.1e" % (f, np.abs(ref).max(), err))
    assert err < 1e-5

"""The work this library is used for, as cases that can be measured.

A case is one of three kinds:

* ``scene``    one whole call sequence of the single-scene interface, from host
               arrays to host arrays: tear down, load, render, source hop,
               bounces, field objects, field points, read-back;
* ``batch``    one ping of a batch plan that a program keeps: new source and
               receiver positions, run, read-back;
* ``readout``  the allocation-free readout on device buffers the caller owns.

Sizes follow the benchmark workloads of ``scenes.py`` (plate, icosphere,
trihedral, batch) and the test scenes around them.  Pressures are kept in
single precision, as programs that store many of them do.
"""
import ctypes
import math

import numpy as np
import torch

import __graft_entry__

__graft_entry__.load_package()
from sonar_render_gb300 import api, batch, scenes  # noqa: E402

CP = 1480.0


def scene_case(shape, khz, sources=1, bounces=0, points=0, plane=0, tol=0.0, att=0.0):
    """points: field points per side; plane: cells per side of a field surface;
    tol: tolerance of compressed bounces (0: plain); att: Np/m."""
    return dict(kind="scene", shape=shape, khz=khz, sources=sources, bounces=bounces, points=points, plane=plane,
                tol=tol, att=att)


def batch_case(nscenes, nsrc, nrx, nfreq, n_lo, n_hi, relative=False, att=0.0):
    """n_lo, n_hi: fragments of a scene at the top frequency."""
    return dict(kind="batch", nscenes=nscenes, nsrc=nsrc, nrx=nrx, nfreq=nfreq, n_lo=n_lo, n_hi=n_hi,
                relative=relative, att=att)


def readout_case(fragments, points, khz, att=0.0):
    return dict(kind="readout", fragments=fragments, points=points, khz=khz, att=att)


def listed():
    return [
        # a real-time host that reads a small target back at one arc of hydrophones per ping
        dict(readout_case(1271, 181, 10.0), name="readout_small"),
        # the same host with a large target and a dense receiver surface, in an attenuating medium
        dict(readout_case(62003, 40001, 40.0, att=0.05), name="readout_large"),
        # the first thing a user runs: a plate, one source, a grid of field points
        dict(scene_case("plate", 10.0, points=64), name="plate_10khz"),
        # a target strength run: several source positions' sum over a box, attenuating medium
        dict(scene_case("box", 25.0, sources=5, points=101, att=0.02), name="box_25khz"),
        # two targets that scatter onto each other
        dict(scene_case("pair", 20.0, bounces=2, points=31), name="pair_20khz_2b"),
        # an ordinary corner reflector with two bounces and a coarse readout
        dict(scene_case("trihedral", 30.0, bounces=2, points=64), name="trihedral_30khz_2b"),
        # the fine corner reflector: three bounces and a 256 x 256 hemisphere
        dict(scene_case("trihedral", 40.0, bounces=3, points=256), name="trihedral_40khz_3b"),
        # the largest plain bounce problem
        dict(scene_case("trihedral", 60.0, bounces=2), name="trihedral_60khz_2b"),
        # the same with compressed bounces at the benchmark's tolerance
        dict(scene_case("trihedral", 60.0, bounces=2, tol=7e-4), name="trihedral_60khz_2b_compressed"),
        # a closed body onto a field surface through its centre, the shadowed projection
        dict(scene_case("sphere", 20.0, plane=512), name="sphere_20khz_plane512"),
        # a handful of scenes and positions, phases relative to the scenes' centres
        dict(batch_case(3, 13, 29, 3, 2000, 30000, relative=True), name="batch_small"),
        # the full bistatic survey
        dict(batch_case(16, 64, 64, 8, 2000, 200000), name="batch_full"),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    kind = rng.choice(["readout", "plate", "box", "pair", "trihedral", "trihedral", "compressed", "sphere", "batch"])
    att = rng.choice([0.0, 0.0, round(rng.uniform(0.005, 0.2), 3)])
    if kind == "readout":
        return readout_case(int(_log(rng, 300, 120000)), int(_log(rng, 1, 60000)), round(_log(rng, 5, 60), 2), att)
    if kind in ("plate", "box"):
        return scene_case(kind, round(_log(rng, 5, 40), 2), sources=rng.randint(1, 16),
                          points=int(_log(rng, 8, 200)), att=att)
    if kind == "pair":
        return scene_case(kind, round(_log(rng, 6, 30), 2), bounces=rng.randint(1, 3), points=int(_log(rng, 4, 90)),
                          att=att)
    if kind == "trihedral":
        return scene_case(kind, round(_log(rng, 9, 50), 2), bounces=rng.randint(1, 3),
                          points=rng.choice([0, int(_log(rng, 8, 200))]), att=att)
    if kind == "compressed":
        return scene_case("trihedral", round(_log(rng, 24, 60), 2), bounces=rng.randint(1, 3),
                          tol=rng.choice([1e-4, 3e-4, 5e-4, 7e-4]), att=att)
    if kind == "sphere":
        return scene_case(kind, round(_log(rng, 5, 18), 2), plane=int(_log(rng, 64, 450)), att=att)
    n_hi = int(_log(rng, 4000, 150000))
    return batch_case(rng.randint(1, 12), rng.randint(1, 64), rng.randint(1, 64), rng.randint(1, 8), 1000, n_hi,
                      relative=rng.random() < 0.5, att=att)


# ------------------------------------------------------------------ inputs
def _turned(tris, rng):
    """The mesh turned a little, as targets sit in a scene: not along the axes."""
    t = scenes.rotate(tris, "x", float(rng.uniform(-4.0, 4.0)))
    return scenes.rotate(t, "z", float(rng.uniform(-6.0, 6.0)))


def _scene_config(case, seed):
    """The arrays a program loads: targets, field surfaces, sources, points."""
    rng = np.random.default_rng(seed)
    f = case["khz"] * 1e3
    d = scenes.delta_for(f)
    n, shape = case["points"], case["shape"]
    jitter = rng.uniform(-0.3, 0.3, (case["sources"], 3))
    fields, points = [], None
    if shape == "plate":
        targets = [scenes.plate_1x05()]
        sources = np.array([0.0, 0.0, 5.0]) + jitter
        if n:
            points = scenes.grid_xy(n, 1.0, 3.0) + rng.uniform(-0.05, 0.05, 3)
    elif shape == "box":
        targets = [_turned(scenes.box(0.6, 0.4, 0.3), rng)]
        sources = np.array([0.5, -1.0, 6.0]) + 2.0 * jitter
        if n:
            points = scenes.hemisphere(n, n, 4.0, axis=(0.1, -0.2, 1.0)) + rng.uniform(-0.05, 0.05, 3)
    elif shape == "pair":
        # two plates that face each other at a right angle, a gap between them
        a = scenes.rectangle(0.8, 0.6)
        b = scenes.translate(scenes.rotate(scenes.rectangle(0.7, 0.6), "y", 90.0), (-0.5, 0.0, 0.45))
        targets = [a, b]
        sources = np.array([4.0, 0.3, 5.0]) + jitter
        if n:
            points = scenes.hemisphere(n, n, 3.0, axis=(1.0, 0.1, 1.0)) + rng.uniform(-0.05, 0.05, 3)
    elif shape == "trihedral":
        targets = [scenes.trihedral(1.0)]
        sources = (20.0 / math.sqrt(3.0)) * np.ones(3) + jitter
        if n:
            points = scenes.hemisphere(n, n, 2.0) + rng.uniform(0.0, 0.05, 3)
    else:
        targets = [scenes.icosphere(4, 1.0)]
        sources = np.array([0.0, 0.0, 10.0]) + jitter
        plane = np.array([[0, -2, -2, 0, 2, -2, 0, 2, 2], [0, -2, -2, 0, 2, 2, 0, -2, 2]], np.float32)
        fields = [(plane, 4.0 / case["plane"])]
    return dict(cp=CP, frequency=f, attenuation=case["att"], targets=[(t, d) for t in targets], fields=fields,
                sources=np.asarray(sources, np.float32),
                field_points=None if points is None else np.asarray(points, np.float32), bounces=case["bounces"])


def _batch_inputs(case, seed):
    cfg = scenes.batch_config(seed=seed, nscenes=case["nscenes"], npos=2, nfreq=case["nfreq"], n_lo=case["n_lo"],
                              n_hi=case["n_hi"])
    rng = np.random.default_rng(seed)
    src = scenes.arc_xz(30.0, np.linspace(-60.0, 60.0, case["nsrc"]) + rng.uniform(-0.5, 0.5))
    rx = scenes.arc_xz(30.0, np.linspace(-60.0, 60.0, case["nrx"]) + rng.uniform(-0.5, 0.5))
    moved = rng.uniform(-0.2, 0.2, (2, 3)).astype(np.float32)
    return cfg, (src, rx), (src + moved[0], rx + moved[1])


def _readout_inputs(case, seed):
    """Fragments of a shallow dish (an own normal per fragment), the pressures a
    distant source leaves on it, and points scattered over a half shell."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    n, m, f = case["fragments"], case["points"], case["khz"] * 1e3
    d = scenes.delta_for(f)
    side = d * math.sqrt(n)
    k = 2.0 * math.pi * f / CP
    u = (torch.rand((n, 2), generator=g, device="cuda", dtype=torch.float64) - 0.5) * side
    R = 1.5 * side
    z = (u * u).sum(1) / (2.0 * R)
    normal = torch.stack([-u[:, 0] / R, -u[:, 1] / R, torch.ones_like(z)], 1)
    normal = normal / normal.norm(dim=1, keepdim=True)
    area = d * d * (0.25 + 0.75 * torch.rand(n, generator=g, device="cuda", dtype=torch.float64))
    pos = torch.cat([u, z[:, None], area[:, None]], 1).float()
    source = torch.tensor([1.0, -2.0, 9.0], device="cuda", dtype=torch.float64)
    r = (pos[:, :3].double() - source).norm(dim=1)
    pres = torch.stack([torch.cos(k * r) / r, torch.sin(k * r) / r], 1)
    direction = torch.randn((m, 3), generator=g, device="cuda", dtype=torch.float64)
    direction[:, 2] = direction[:, 2].abs()
    direction = direction / direction.norm(dim=1, keepdim=True)
    pts = torch.zeros((m, 4), device="cuda")
    pts[:, :3] = (direction * (2.0 * side + 2.0)).float()
    nrm = torch.cat([normal, torch.zeros_like(z)[:, None]], 1).float()
    return pos.contiguous(), nrm.contiguous(), pres.contiguous(), pts, float(np.float32(k))


# ------------------------------------------------------------------ passes
def prepare(case, seed):
    if case["kind"] == "scene":
        return case, _scene_config(case, seed)
    if case["kind"] == "batch":
        cfg, (src, rx), moved = _batch_inputs(case, seed)
        plan = batch.Plan(cfg["scenes"], src, rx, cfg["freqs"], cp=CP, attenuation=case["att"])
        if case["relative"]:
            plan.set_relative(True)
        return case, plan, moved
    fn = api.lib().sonar_readout_noalloc
    p = ctypes.c_void_p
    fn.argtypes = [p, p, p, ctypes.c_int, p, ctypes.c_int, ctypes.c_float, ctypes.c_float, p, p]
    fn.restype = ctypes.c_int
    inputs = _readout_inputs(case, seed)
    return case, fn, inputs, torch.zeros((case["points"], 2), dtype=torch.float64, device="cuda")


def run(state):
    case = state[0]
    if case["kind"] == "scene":
        return _run_scene(case, state[1])
    if case["kind"] == "batch":
        _, plan, (src, rx) = state
        plan.set_points(src, rx)
        return plan.run().astype(np.complex64)
    _, fn, (pos, nrm, pres, pts, k), out = state
    out.zero_()
    status = fn(pos.data_ptr(), nrm.data_ptr(), pres.data_ptr(), pos.shape[0], pts.data_ptr(), pts.shape[0], k,
                case["att"], out.data_ptr(), torch.cuda.current_stream().cuda_stream)
    if status != 0:
        raise RuntimeError("sonar_readout_noalloc: %d" % status)
    return out.float()


def _run_scene(case, cfg):
    api.TearDownCuda()
    api.set_option("cross_objects", case["shape"] == "pair")
    api.set_option("compress", case["tol"] > 0)
    if case["tol"] > 0:
        api.set_option("compress_tol", case["tol"])
        api.set_option("compress_judge", 3 * case["tol"])
    api.run_scene(cfg)
    out = {"targets": [api.get_object_pressures(api.TARGET, i).astype(np.complex64)
                       for i in range(len(cfg["targets"]))]}
    if cfg["fields"]:
        out["fields"] = [api.get_object_pressures(api.FIELD, 0).astype(np.complex64)]
    if cfg["field_points"] is not None:
        out["points"] = api.get_field_point_pressures(len(cfg["field_points"])).astype(np.complex64)
    return out


# ------------------------------------------------------------------ work
_AREA = {"plate": 0.5, "box": 1.08, "pair": 0.9, "trihedral": 1.5, "sphere": 4.0 * math.pi}
_PAIR = 40.0   # operations of one ordered pair without its sine, cosine and square root
_BOTH = 24.0   # the same when one Green's function serves both directions


def work(case):
    if case["kind"] == "readout":
        n, m = case["fragments"], case["points"]
        return {"bytes": 48.0 * n + 32.0 * m, "flops": _PAIR * n * m}
    if case["kind"] == "batch":
        n = case["nscenes"] * 0.5 * (case["n_lo"] + case["n_hi"]) * sum(
            (f / 40e3) ** 2 for f in np.geomspace(5e3, 40e3, case["nfreq"]))
        s, r = case["nsrc"], case["nrx"]
        return {"bytes": 48.0 * n + 16.0 * case["nscenes"] * case["nfreq"] * s * r,
                "flops": n * (_PAIR * (s + r) + 8.0 * s * r)}
    d = CP / (case["khz"] * 1e3) / 7.5
    n = _AREA[case["shape"]] / (d * d)
    fp, fs = float(case["points"]) ** 2, float(case["plane"]) ** 2
    # shares of the ordered pairs that interact: two of a trihedral's three
    # facets, the lit half of a closed body
    inter = {"trihedral": 2.0 / 3.0, "pair": 0.5}.get(case["shape"], 0.0)
    lit = 0.5 if case["shape"] in ("box", "sphere") else 1.0
    flops = _PAIR * n * (case["sources"] * lit + fp * lit + fs * lit) + _BOTH * inter * n * n * case["bounces"]
    return {"bytes": 48.0 * n + 12.0 * case["sources"] + 28.0 * fp + 16.0 * fs, "flops": flops}


# ------------------------------------------------------------------ 64-bit values
def _frame(tri, delta):
    """Grid of one triangle: cell counts as single precision decides them, axes
    and origin in 64 bits.  The longest edge is the base."""
    def parts(dt):
        v = [np.asarray(tri[3 * i:3 * i + 3], dt) for i in range(3)]
        d = dt(delta)
        edge = [np.sqrt(((v[a] - v[b]) ** 2).sum(dtype=dt)) for a, b in ((0, 1), (0, 2), (1, 2))]
        return v, d, edge

    v, d32, edge = parts(np.float32)
    m = int(np.argmax(edge))
    o, e, a = [(0, 1, 2), (0, 2, 1), (1, 2, 0)][m]

    def axes(dt):
        v, d, edge = parts(dt)
        u = (v[e] - v[o]) / edge[m]
        base = v[o] + u * (u * (v[a] - v[o])).sum(dtype=dt)
        alt = v[a] - base
        h = np.sqrt((alt * alt).sum(dtype=dt))
        neg = np.sqrt(((v[o] - base) ** 2).sum(dtype=dt))
        pos = np.sqrt(((base - v[e]) ** 2).sum(dtype=dt))
        return v, d, u, base, alt / h, h, neg, pos

    _, d, _, _, _, h, neg, pos = axes(np.float32)
    nneg = int(np.ceil(neg / d))
    nx, ny = nneg + int(np.ceil(pos / d)), int(np.ceil(h / d))
    v, d, u, base, w, h, neg, pos = axes(np.float64)
    d = np.float64(np.float32(delta))
    normal = np.cross(v[1] - v[0], v[2] - v[0])
    return nx, ny, nneg, u, w, base, h, neg, pos, normal / np.linalg.norm(normal), d


def _cells(objects):
    """Cells of every object: centre (source hop), readout position, area,
    facet number over all objects, normal, delta; 64 bits, in the library's order."""
    out, facet = [], 0
    for tris, delta in objects:
        for tri in np.asarray(tris, np.float32).reshape(-1, 9):
            nx, ny, nneg, u, w, base, h, neg, pos, normal, d = _frame(tri, delta)
            x = (np.arange(nx) - nneg) * d
            y = np.arange(ny) * d
            slope = np.where(x >= 0, h / -pos, h / max(neg, 1e-300))

            def under(t):  # integral of min(max(t, 0), d)
                c = np.clip(t, 0.0, d)
                return 0.5 * c * c + d * (t - c) * (t > d)

            left = slope * x + h
            area = (under(left + slope * d - y[:, None]) - under(left - y[:, None])) / slope
            corner = base + x[None, :, None] * u + (y + d / 2)[:, None, None] * w
            n = nx * ny
            out.append((corner.reshape(n, 3) + u * (d / 2), corner.reshape(n, 3), area.reshape(n),
                        np.full(n, facet), np.broadcast_to(normal, (n, 3)), np.full(n, d)))
            facet += 1
    return [np.concatenate(p) for p in zip(*out)]


def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _t(x):
    return torch.as_tensor(np.ascontiguousarray(x), device=_device())


def _planes(objects):
    """Per target triangle: its plane and its three edge planes, inside positive."""
    got = []
    for tris, _ in objects:
        for t in np.asarray(tris, np.float64).reshape(-1, 3, 3):
            n = np.cross(t[1] - t[0], t[2] - t[0])
            n = n / np.linalg.norm(n)
            edges = []
            for a, b in ((0, 1), (1, 2), (2, 0)):
                m = np.cross(n, t[b] - t[a])
                m = m / np.linalg.norm(m)
                edges.append((m, float(m @ t[a])))
            got.append((n, float(n @ t[0]), edges))
    return got


def _occluded(planes, o, e):
    """Segments o -> e (broadcast against each other) that a triangle crosses
    before the last millimetre; a plane the origin lies on never occludes."""
    r = (e - o).norm(dim=-1)
    scale = 1.0 + torch.maximum(o.abs().amax(-1).expand(r.shape), e.abs().amax(-1).expand(r.shape))
    hit = torch.zeros(r.shape, dtype=torch.bool, device=r.device)
    for n, c, edges in planes:
        n = _t(n)
        d0, d1 = o @ n - c, e @ n - c
        s = d0.abs() / (d0.abs() + d1.abs())
        on = (d0 * d1 < 0) & (d0.abs() > 1e-4 * scale) & (r * s <= r - 1e-3)
        for m, cm in edges:
            m = _t(m)
            on &= (o @ m) * (1 - s) + (e @ m) * s >= cm
        hit |= on
    return hit


def _green(r, k, att):
    """-e^{ikr} / (4 pi) (ik / r) + 1 / r^2 with k + i att."""
    ik = torch.complex(torch.tensor(-att, dtype=torch.float64), torch.tensor(k, dtype=torch.float64)).to(r.device)
    return -torch.exp(ik * r) / (4 * math.pi) * (ik / r) + 1.0 / (r * r)


def _wave_number(f):
    """Re k as set_initial_conditions defines it: single precision."""
    return float(np.float32(2.0 * math.pi * f) / np.float32(CP))


def _blocks(n, others):
    step = max(1, min(n, (1 << 25) // max(1, others)))
    return [slice(a, min(n, a + step)) for a in range(0, n, step)]


def _hop(src, w, dst, k, att, planes, n_src=None, n_dst=None, green=True, facets=None, delta=None, dark=None):
    """sum over sources of w G (or e^{ikr} / r) with its cosines, gates and
    shadows.  facets: facet numbers (source, destination), pairs of one facet
    drop out and rays start at the lower one; dark: destinations that take
    nothing from higher facets; delta: regularisation radius per facet pair."""
    out = torch.zeros(dst.shape[0], dtype=torch.complex128, device=dst.device)
    ik = complex(-att, k)
    for b in _blocks(dst.shape[0], src.shape[0]):
        v = dst[b][:, None, :] - src[None, :, :]
        r = v.norm(dim=-1)
        on = torch.ones_like(r, dtype=torch.bool)
        weight = torch.ones_like(r)
        if n_src is not None:
            c = (v * n_src[None]).sum(-1) / r
            on &= c >= 1e-6
            weight = weight * c
        if n_dst is not None:
            c = -(v * n_dst[b][:, None, :]).sum(-1) / r
            on &= c >= 1e-6
            weight = weight * c
        o, e = src[None], dst[b][:, None, :]
        if facets is not None:
            fs, fd = facets[0][None, :], facets[1][b][:, None]
            on &= (fs != fd) & ~((fs > fd) & dark[b][:, None])
            swap = (fs > fd)[..., None]
            o, e = torch.where(swap, e.expand(v.shape), o.expand(v.shape)), torch.where(swap, o.expand(v.shape),
                                                                                       e.expand(v.shape))
        elif green and n_dst is None and planes:
            o, e = e, o  # the readout's rays start at the field point
        if planes:
            on &= ~_occluded(planes, o, e)
        del v, o, e
        if green:
            g = _green(r, k, att)
            if delta is not None:
                g = 0.9 * torch.where(r < delta, torch.full_like(g, ik / (4 * math.pi)), g)
        else:
            g = torch.exp(ik * r) / r
        out[b] = (torch.where(on, weight, torch.zeros_like(weight)) * g) @ w
    return out


def _exact_scene(case, seed):
    cfg = _scene_config(case, seed)
    n = _AREA[case["shape"]] / scenes.delta_for(cfg["frequency"]) ** 2
    pairs = n * (case["sources"] + case["points"] ** 2 + case["plane"] ** 2 + n * case["bounces"])
    if case["tol"] > 0 or pairs > 8e9:
        return None
    f, att = cfg["frequency"], float(np.float32(case["att"]))
    k = _wave_number(f)
    centre, pos, area, facet, normal, delta = [_t(x) for x in _cells(cfg["targets"])]
    # a closed convex body never shadows what its own cosines let through
    planes = [] if case["shape"] in ("plate", "box", "sphere") else _planes(cfg["targets"])
    sources = _t(cfg["sources"].astype(np.float64))
    one = torch.ones(len(sources), dtype=torch.complex128, device=sources.device)
    P = _hop(sources, one, centre, k, att, planes, n_dst=normal, green=False)
    act = (area > 1e-6).nonzero()[:, 0]
    p, a, nr, fa = pos[act], area[act], normal[act], facet[act]
    pin = P.clone()
    for _ in range(case["bounces"]):
        pout = torch.zeros_like(P)
        pout[act] = _hop(p, a * pin[act], p, k, att, planes, n_src=nr, n_dst=nr, facets=(fa, fa),
                         delta=float(delta[0]), dark=pin[act] == 0)
        P = P + pout
        pin = pout
    sizes = [sum(nx * ny for nx, ny in (_frame(t, d)[:2] for t in np.asarray(tris).reshape(-1, 9)))
             for tris, d in cfg["targets"]]
    out = {"targets": [x.cpu().numpy() for x in P.split(sizes)]}
    if cfg["fields"]:
        # field cells take pressure at their readout positions where they have area
        _, fpos, farea, _, _, _ = [_t(x) for x in _cells(cfg["fields"])]
        field = torch.zeros(len(fpos), dtype=torch.complex128, device=P.device)
        cells = (farea > 1e-6).nonzero()[:, 0]
        field[cells] = _hop(p, a * P[act], fpos[cells], k, att, planes, n_src=nr, delta=float(delta[0]))
        out["fields"] = [field.cpu().numpy()]
    if cfg["field_points"] is not None:
        pts = _t(cfg["field_points"].astype(np.float64))
        out["points"] = _hop(p, a * P[act], pts, k, att, planes, n_src=nr).cpu().numpy()
    return out


def _exact_batch(case, seed):
    cfg, _, (src, rx) = _batch_inputs(case, seed)
    att = float(np.float32(case["att"]))
    src, rx = _t(src.astype(np.float64)), _t(rx.astype(np.float64))
    if sum(len(t) for t in cfg["scenes"]) * case["nfreq"] > 40000:
        return None
    out = np.zeros((case["nscenes"], case["nfreq"], case["nrx"], case["nsrc"]), np.complex128)
    for s, tris in enumerate(cfg["scenes"]):
        for q, f in enumerate(cfg["freqs"]):
            f = float(f)
            k = _wave_number(f)
            # the fragment side as the plan forms it, in single precision
            d = np.float32(np.float32(np.float32(CP) / np.float32(f)) / np.float32(7.5))
            centre, pos, area, _, normal, _ = [_t(x) for x in _cells([(tris, d)])]
            act = area > 1e-6
            total = torch.zeros((case["nrx"], case["nsrc"]), dtype=torch.complex128, device=src.device)
            for b in _blocks(int(act.sum()), 64):
                c, p, a, n = centre[act][b], pos[act][b], area[act][b], normal[act][b]
                v = c[:, None, :] - src[None]
                r = v.norm(dim=-1)
                cos = -(v * n[:, None, :]).sum(-1) / r
                pin = torch.where(cos >= 1e-6, cos, 0.0 * cos) * torch.exp(complex(-att, k) * r) / r
                v = rx[:, None, :] - p[None]
                r = v.norm(dim=-1)
                cos = (v * n[None]).sum(-1) / r
                total += (torch.where(cos >= 1e-6, cos, 0.0 * cos) * a[None] * _green(r, k, att)) @ pin
            out[s, q] = total.cpu().numpy()
    return out


def exact(case, seed):
    if case["kind"] == "scene":
        return _exact_scene(case, seed)
    if case["kind"] == "batch":
        return _exact_batch(case, seed)
    pos, nrm, pres, pts, k = _readout_inputs(case, seed)
    w = pos[:, 3].double() * torch.complex(pres[:, 0], pres[:, 1])
    P = _hop(pos[:, :3].double(), w, pts[:, :3].double(), k, float(np.float32(case["att"])), [],
             n_src=nrm[:, :3].double())
    return torch.view_as_real(P)

"""The work a user of hussar_gb300 has it do, as cases that can be timed and checked.

A case is a dict of plain values with a "kind":

  run        one sensor, PathTracer.run + fetchFrame (the reference program's inner loop)
  sweep      many sensor poses over one scene in one simulate_batch call
  frame      a MIMO radar cube through simulate_frame
  far_field  an RCS sweep with plane-wave antennas through simulate_batch_ff
  graph      a batch over device buffers, captured once and replayed (batch_graph)
  serve      requests over resident scenes through the serving loop
  rays       closest-hit and occlusion queries (RT::intersect, RT::visible)
  build      a new scene: Backend(mesh) and the first ray queries against it
  refit      moved vertices: Backend.refit and the next frame

Scenes are the generators of hussar_gb300/scenes.py: the two-plate dihedral (4 triangles),
the thick evaluation plates (24), the icosphere over a ground quad, random boxes on a
ground quad and the urban canyon. Every input comes from the seed.
"""
import math

import numpy as np
import torch

import hussar_gb300 as hg
from hussar_gb300 import _lib, scenes
from hussar_gb300.serve import Server

REFERENCE, SPLIT = _lib.HSR_PHASE_REFERENCE_FP32, _lib.HSR_PHASE_SPLIT_FP64
DIRICHLET, SYNTH = _lib.HSR_SPLAT_DIRICHLET16, _lib.HSR_SPLAT_FINE_SYNTH


def listed():
    return [
        # the smallest call: one pose of the reference's dihedral example, first schedule step
        {"name": "run_dihedral", "kind": "run", "scene": "dihedral", "tris": 4, "log2_budget": 14, "bounces": 2,
         "bins": 256, "guided": False, "split": False},
        # the guided doubling schedule (PathTracer's default) on the same reflector
        {"name": "run_guided", "kind": "run", "scene": "plates", "tris": 24, "log2_budget": 18, "bounces": 10,
         "bins": 256, "guided": True, "split": True},
        # one long run of a curved target over ground: 2^22 samples, 512 ADC samples
        {"name": "run_sphere", "kind": "run", "scene": "sphere", "tris": 81922, "log2_budget": 22, "bounces": 3,
         "bins": 512, "guided": False, "split": False},
        # an azimuth sweep of the dihedral in one call, few samples per pose
        {"name": "sweep_dihedral", "kind": "sweep", "scene": "dihedral", "tris": 4, "poses": 91, "log2_lo": 12,
         "log2_hi": 12, "bounces": 2, "bins": 256, "split": False, "synth": False},
        # the batched workload: 1 M triangles, uneven budgets, exact-spectrum synthesis
        {"name": "sweep_boxes", "kind": "sweep", "scene": "boxes", "tris": 1000010, "poses": 96, "log2_lo": 14,
         "log2_hi": 19, "bounces": 4, "bins": 256, "split": True, "synth": True},
        # a data-set sweep: thousands of poses with short budgets, odd chirp length
        {"name": "sweep_many", "kind": "sweep", "scene": "boxes", "tris": 20006, "poses": 1999, "log2_lo": 8,
         "log2_hi": 12, "bounces": 3, "bins": 200, "split": True, "synth": True},
        # a captured batch replayed over device buffers, parity phase, ragged budgets
        {"name": "graph_boxes", "kind": "graph", "scene": "boxes", "tris": 100010, "poses": 33, "log2_lo": 13,
         "log2_hi": 18, "bounces": 4, "bins": 256, "split": False, "synth": False},
        # a 3 x 4 MIMO cube of a street scene, five bounces
        {"name": "frame_urban", "kind": "frame", "scene": "urban", "tris": 1000000, "log2_budget": 19, "bounces": 5,
         "bins": 256, "chirps": 128, "split": True},
        # an RCS sweep of the dihedral by plane waves
        {"name": "far_field", "kind": "far_field", "scene": "dihedral", "tris": 4, "poses": 27, "log2_budget": 14,
         "bounces": 2, "bins": 256},
        # a burst of requests over three resident scenes
        {"name": "serve_mix", "kind": "serve", "tris": 250000, "requests": 24, "log2_lo": 15, "log2_hi": 20,
         "bounces": 4},
        # a million ray queries against a dense scene
        {"name": "rays_boxes", "kind": "rays", "scene": "boxes", "tris": 1000010, "rays": 1 << 20},
        # a mesh becomes a resident scene and answers its first queries
        {"name": "build_boxes", "kind": "build", "scene": "boxes", "tris": 250010, "rays": 1 << 16},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["run", "sweep", "sweep", "frame", "far_field", "graph", "serve", "rays", "build", "refit"])
    scene = rng.choice(["dihedral", "plates", "sphere", "boxes", "urban"])
    dense = rng.choice(["sphere", "boxes", "urban"])
    c = {"kind": kind}
    if kind == "run":
        c |= {"scene": scene, "tris": _tris(rng, scene), "log2_budget": round(rng.uniform(12, 21), 3),
              "bounces": rng.choice([1, 2, 3, 5, 10]), "bins": rng.choice([128, 200, 255, 256, 512, 1000]),
              "guided": False, "split": rng.random() < 0.5}
    elif kind in ("sweep", "graph"):
        lo = rng.uniform(8, 14)
        c |= {"scene": scene, "tris": _tris(rng, scene), "poses": _log(rng, 2, 600), "log2_lo": round(lo, 3),
              "log2_hi": round(lo + rng.uniform(0, 2), 3), "bounces": rng.choice([1, 2, 3, 4, 6]),
              "bins": rng.choice([64, 128, 200, 256, 333, 512]), "split": rng.random() < 0.5,
              "synth": rng.random() < 0.5}
    elif kind == "frame":
        c |= {"scene": dense, "tris": _tris(rng, dense), "log2_budget": round(rng.uniform(14, 19), 3),
              "bounces": rng.choice([2, 4, 5]), "bins": rng.choice([128, 256, 300]), "chirps": rng.choice([1, 16, 128]),
              "split": rng.random() < 0.5}
    elif kind == "far_field":
        c |= {"scene": "dihedral", "tris": 4, "poses": _log(rng, 1, 90), "log2_budget": round(rng.uniform(10, 17), 3),
              "bounces": rng.choice([1, 2, 3]), "bins": rng.choice([128, 256, 500])}
    elif kind == "serve":
        c |= {"tris": _log(rng, 20000, 250000), "requests": _log(rng, 2, 40), "log2_lo": 13, "log2_hi": 18,
              "bounces": rng.choice([2, 4])}
    elif kind == "rays":
        c |= {"scene": dense, "tris": _tris(rng, dense), "rays": _log(rng, 100, 1 << 20)}
    elif kind == "build":
        c |= {"scene": dense, "tris": _log(rng, 500, 250000), "rays": _log(rng, 100, 1 << 16)}
    else:
        c |= {"scene": dense, "tris": _tris(rng, dense), "log2_budget": round(rng.uniform(12, 17), 3), "bounces": 3,
              "bins": 256}
    return c


def _tris(rng, scene):
    return {"dihedral": 4, "plates": 24}.get(scene) or _log(rng, 1000, 1000000 if scene != "sphere" else 80000)


# ---- scenes, sensors and chirps --------------------------------------------------------


def _mesh(scene, tris, rng):
    """(mesh, sensor positions generator, extent of the scene in metres)."""
    if scene == "dihedral":
        return scenes.dihedral_mesh(), _ring(rng, 1.0, 0.05), 0.1
    if scene == "plates":
        return scenes.evaluation_dihedral_workload(0.05, [0.0]).mesh, _ring(rng, 0.9, 0.03), 0.05
    if scene == "sphere":
        level = max(1, min(6, int(round(math.log(max(tris, 81) / 20.0, 4)))))
        m = hg.TriangleMesh()
        v, f = scenes.icosphere(level, 0.5, (0.0, 0.5 + 0.05 * rng.random(), 0.0))
        m.append(v, f)
        m.addQuad([-10, 0, -10], [20, 0, 0], [0, 0, 20])
        return m, _ring(rng, 9.5 + rng.random(), 0.5), 20.0
    if scene == "boxes":
        count = max(1, (tris - 2) // 12)
        extent = 100.0 * math.sqrt(max(count, 100) / 83334.0)
        m = scenes.boxes_mesh(int(rng.integers(1 << 31)), count, extent)
        return m, (lambda n: scenes.plane_poses(n, int(rng.integers(1 << 31)), extent)), extent
    m = scenes.urban_mesh(max(tris, 4000), int(rng.integers(1 << 31)))
    return m, (lambda n: scenes.street_poses(n, int(rng.integers(1 << 31)))), 500.0


def _ring(rng, distance, height):
    """Sensors around the y axis, in the quadrant that a corner at the origin opens to."""

    def poses(n):
        out = []
        for th in np.deg2rad(rng.uniform(3.0, 87.0, n)):
            d = distance * rng.uniform(0.95, 1.05)
            out.append(hg.NFAntenna(np.array([d * np.cos(th), height, d * np.sin(th)], np.float32), scenes.looking(th)))
        return out

    return poses


def _tracer(case):
    t = hg.PathTracer()
    t.doGuiding = bool(case.get("guided", False))
    t.maxDepth = int(case["bounces"])
    t.phaseMode = SPLIT if case.get("split") else REFERENCE
    return t


def _chirp(bins):
    return scenes.rf_77ghz(bins, 5e6 * bins / 256)[0]


def _budgets(case, rng):
    lo, hi = case["log2_lo"], case["log2_hi"]
    return np.round(2.0 ** rng.uniform(lo, hi, case["poses"]) if hi > lo else
                    np.full(case["poses"], 2.0 ** lo)).astype(np.int64)


def _offsets(rng, n):
    return rng.integers(0, 1 << 20, n).astype(np.int64)


def _queries(rng, n, extent):
    """Rays inside the scene: origins above the ground, directions over the sphere, and the
    segments between those origins and other points (occlusion)."""
    o = np.stack([rng.uniform(-extent / 2, extent / 2, n), rng.uniform(0.1, 6.0, n),
                  rng.uniform(-extent / 2, extent / 2, n)], 1)
    d = rng.standard_normal((n, 3))
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    return o.astype(np.float32), d.astype(np.float32), rng.uniform(0.5, 20.0, n).astype(np.float32)


def _inputs(case, seed):
    """Everything a case's pass reads, on the host, from the seed alone."""
    rng = np.random.default_rng([seed, 0x5EED])
    kind, s = case["kind"], {}
    if kind == "serve":
        s["scenes"] = [_mesh(k, t, rng) for k, t in
                       (("boxes", case["tris"] // 2), ("urban", case["tris"]), ("boxes", 2 * case["tris"]))]
        s["tracer"] = _tracer(case)
        s["requests"] = []
        for i in range(case["requests"]):
            k = int(rng.integers(3))
            a = s["scenes"][k][1](1)[0]
            bins = (128, 256, 512)[i % 3]
            s["requests"].append((k, scenes.rf_chirp(rng.uniform(1e9, 4e9), bins), bins, a, a,
                                  int(round(2.0 ** rng.uniform(case["log2_lo"], case["log2_hi"])))))
        return s
    s["mesh"], poses, extent = _mesh(case["scene"], case["tris"], rng)
    if kind in ("rays", "build"):
        s["queries"] = _queries(rng, case["rays"], min(extent, 100.0))
        return s
    s["tracer"], s["bins"] = _tracer(case), int(case["bins"])
    s["rf"] = _chirp(s["bins"])
    if kind in ("run", "refit"):
        a = poses(1)[0]
        s["scene"] = hg.Scene(s["rf"], a, a)
        s["budget"] = int(round(2.0 ** case["log2_budget"]))
        s["tracer"].configureFrame(hg.FrameConfig(1, s["bins"], 1))
        if kind == "refit":
            v = s["mesh"].vertexBuffer
            moved = v + (0.02 * np.sin(v[:, [1, 2, 0]] + rng.uniform(0, 6, 3))).astype(np.float32)
            s["moved"] = hg.TriangleMesh(moved, s["mesh"].indexBuffer)
    elif kind in ("sweep", "graph"):
        s["tx"] = poses(case["poses"])
        s["rx"] = list(s["tx"])
        s["budget"], s["offset"] = _budgets(case, rng), _offsets(rng, case["poses"])
        s["modes"] = (SPLIT if case["split"] else REFERENCE, SYNTH if case["synth"] else DIRICHLET)
    elif kind == "frame":
        a = poses(1)[0]
        s["tx"], s["rx"] = scenes.mimo_array(a.position(), rng.uniform(0, 2 * np.pi))
        s["frame"] = hg.FrameConfig(case["chirps"], s["bins"], len(s["tx"]) * len(s["rx"]))
        s["budget"] = int(round(2.0 ** case["log2_budget"]))
    else:
        c = np.full(3, 0.05, np.float32)
        s["tx"] = []
        for a in np.deg2rad(rng.uniform(5.0, 85.0, case["poses"])):
            d = np.array([np.cos(a), 0.0, np.sin(a)])
            s["tx"].append(hg.FFAntenna((d / np.linalg.norm(d)).astype(np.float32), [0, 1, 0], c, 0.1))
        s["rx"] = list(s["tx"])
        s["budget"] = np.full(case["poses"], int(round(2.0 ** case["log2_budget"])), np.int64)
        s["offset"] = _offsets(rng, case["poses"])
    return s


def prepare(case, seed):
    s = _inputs(case, seed)
    s["kind"] = kind = case["kind"]
    if kind == "build":
        return s
    if kind == "serve":
        backends = [hg.gb300.Backend(m, None) for m, _, _ in s["scenes"]]
        s["server"] = Server(s["tracer"], SPLIT, max_slots=64, max_samples_per_chirp=512)
        s["ids"] = [s["server"].add_scene(b) for b in backends]
        return s
    s["backend"] = hg.gb300.Backend(s["mesh"], s.get("tracer"))
    if kind == "graph":
        def dev(antennas):
            raw = (_lib.AntennaC * len(antennas))(*[a.to_c() for a in antennas])
            return torch.frombuffer(bytearray(bytes(raw)), dtype=torch.uint8).cuda()

        s["dev"] = [dev(s["tx"]), dev(s["rx"]), torch.from_numpy(s["budget"]).cuda(), torch.from_numpy(s["offset"]).cuda()]
        s["rows"] = torch.zeros((case["poses"], s["bins"], 2), dtype=torch.float32, device="cuda")
        torch.cuda.synchronize()
        s["graph"] = s["backend"].batch_graph(s["rf"], s["bins"], s["tracer"], case["poses"],
                                              *[t.data_ptr() for t in s["dev"]], s["rows"].data_ptr(), *s["modes"])
    return s


def run(s):
    kind = s["kind"]
    if kind == "run":
        s["tracer"].run(s["backend"], s["scene"], s["budget"])
        return s["tracer"].fetchFrame().data
    if kind == "sweep":
        return s["backend"].simulate_batch(s["rf"], s["bins"], s["tracer"], s["tx"], s["rx"], s["budget"], s["offset"],
                                           *s["modes"])
    if kind == "graph":
        s["graph"].launch(torch.cuda.current_stream().cuda_stream)
        return s["rows"]
    if kind == "frame":
        return s["backend"].simulate_frame(s["rf"], s["frame"], s["tracer"], s["tx"], s["rx"], s["budget"], 0,
                                           s["tracer"].phaseMode)
    if kind == "far_field":
        return s["backend"].simulate_batch_ff(s["rf"], s["bins"], s["tracer"], s["tx"], s["rx"], s["budget"],
                                              s["offset"])
    if kind == "serve":
        reqs = [s["server"].submit(s["ids"][r[0]], *r[1:]) for r in s["requests"]]
        return [r.result()[0] for r in reqs]
    if kind == "refit":
        s["backend"].refit(s["moved"])
        s["tracer"].run(s["backend"], s["scene"], s["budget"])
        return s["tracer"].fetchFrame().data
    backend = s["backend"] if kind == "rays" else hg.gb300.Backend(s["mesh"], None)
    o, d, far = s["queries"]
    return [*backend.intersect(o, d), backend.visible(o, d, far)]


def work(case):
    """Bytes: the mesh, sensors and outputs, each once. Flops: per ray one path down a binary
    tree (two boxes a level) and one triangle; per path its sampling; per bounce the field,
    the phase and the 33-bin kernel."""
    kind = case["kind"]
    tris = case["tris"] * (3.5 if kind == "serve" else 1)
    scene_bytes = 24.0 * tris
    per_ray = 2 * 30.0 * math.log2(tris + 1) + 60.0
    if kind in ("rays", "build"):
        n = case["rays"]
        return {"bytes": scene_bytes + n * (28 + 32 + 28 + 4.0), "flops": 2 * n * per_ray}
    if kind == "serve":
        poses, bins, samples = case["requests"], 256, case["requests"] * _mean(case["log2_lo"], case["log2_hi"])
    elif kind in ("sweep", "graph"):
        poses, bins, samples = case["poses"], case["bins"], case["poses"] * _mean(case["log2_lo"], case["log2_hi"])
    else:
        poses, bins = 12 if kind == "frame" else case.get("poses", 1), case["bins"]
        samples = poses * 2.0 ** case["log2_budget"]
    out = 8.0 * poses * bins * case.get("chirps", 1)
    # of the paths that leave the sensor about a third return to the scene at every bounce
    bounces = {"dihedral": 0.01, "plates": 0.01, "sphere": 0.6}.get(case.get("scene"), 0.5 * case["bounces"])
    if kind == "far_field":
        bounces = 0.6
    return {"bytes": scene_bytes + 96.0 * poses + out, "flops": samples * (150 + per_ray + bounces * (2 * per_ray + 800))}


def _mean(lo, hi):
    return 2.0 ** lo if hi <= lo else (2.0 ** hi - 2.0 ** lo) / (math.log(2.0) * (hi - lo))


# ---- the same estimates in 64 bits -----------------------------------------------------

C0, EPS = 299792458.0, 5e-5


def exact(case, seed):
    kind = case["kind"]
    if kind in ("rays", "build"):
        if float(case["tris"]) * case["rays"] > 4e9:
            return None
        s = _inputs(case, seed)
        return _exact_rays(s["mesh"], *s["queries"])
    if kind not in ("run", "sweep", "graph", "far_field") or case["tris"] > 24 or case.get("guided") or case.get("synth"):
        return None
    samples = 2.0 ** case.get("log2_budget", case.get("log2_hi", 0)) * case.get("poses", 1)
    if samples * case["tris"] > 6e7:
        return None
    s = _inputs(case, seed)
    if kind == "run":
        pairs, budget, offset = [(s["scene"].tx, s["scene"].rx)], [s["budget"]], [0]
    else:
        pairs, budget, offset = list(zip(s["tx"], s["rx"])), s["budget"], s["offset"]
    tri = s["mesh"].vertexBuffer.astype(np.float64)[s["mesh"].indexBuffer]
    rows = np.stack([_exact_row(tri, s["rf"], s["bins"], s["tracer"], tx, rx, int(b), int(o))
                     for (tx, rx), b, o in zip(pairs, budget, offset)])
    if kind == "run":
        return rows.reshape(1, -1, 1)
    return np.stack([rows.real, rows.imag], -1) if kind == "graph" else rows


def _halton(index, base):
    """The radical inverse of every index, digit by digit."""
    v, scale, out = index.copy(), 1.0, np.zeros(len(index))
    while v.any():
        scale /= base
        out += scale * (v % base)
        v //= base
    return np.minimum(out, 1.0 - 2.0 ** -24)


def _hit(tri, o, d, far):
    """Closest hit of every ray with a handful of triangles: (distance or inf, triangle)."""
    best, which = np.full(len(o), np.inf), np.full(len(o), -1)
    with np.errstate(divide="ignore", invalid="ignore"):
        for k, (a, b, c) in enumerate(tri):
            e1, e2 = b - a, c - a
            p = np.cross(d, e2)
            inv = 1.0 / (p @ e1)
            tv = o - a
            u = (tv * p).sum(1) * inv
            q = np.cross(tv, e1)
            v = (d * q).sum(1) * inv
            t = (q @ e2) * inv
            ok = np.isfinite(inv) & (u >= 0) & (u <= 1) & (v >= 0) & (u + v <= 1) & (t > EPS) & (t <= far) & (t < best)
            best[ok], which[ok] = t[ok], k
    return best, which


def _pattern(d):
    """The antenna's field for unit directions in its own frame."""
    ch, ce = np.sqrt(np.maximum(1 - d[:, 0] ** 2, 0)), np.sqrt(np.maximum(1 - d[:, 1] ** 2, 0))
    g = 2.622 / (ch - 1.8) ** 6 * 0.625 / (ce - 1.5) ** 4
    return np.stack([d[:, 2] * g, np.zeros(len(d)), -d[:, 0] * g], 1)


def _unit(v):
    return v / np.linalg.norm(v, axis=1, keepdims=True)


def _exact_row(tri, rf, bins, tracer, tx, rx, budget, offset):
    """One pose's row: `budget` Halton samples from `offset` traced through the triangles in
    geometrical-optics mode with the default filter, every quantity in 64 bits."""
    f0, slope, rate, ramp, delay = (float(np.float32(getattr(rf, n))) for n in
                                    ("startFreq", "freqSlope", "adcRate", "rampTime", "antennaDelay"))
    index = np.arange(offset, offset + budget, dtype=np.int64)
    freq = f0 + _halton(index, 2) * slope * ramp
    u, w = _halton(index, 5), _halton(index, 3)
    plane = isinstance(tx, hg.FFAntenna)
    if plane:
        def disk(a):
            k = a.direction.astype(np.float64)
            m = -k
            e0 = np.array([-m[2], 0, m[0]]) if abs(m[0]) > abs(m[1]) else np.array([0, m[2], -m[1]])
            e0 /= np.linalg.norm(e0)
            r = float(a.radius)
            return k, a.scene_center.astype(np.float64) + r * k, e0, np.cross(m, e0), r, a.polarization.astype(np.complex128)

        k, c, e0, e1, r0, pol = disk(tx)
        o = c + r0 * ((2 * u - 1)[:, None] * e0 + (2 * w - 1)[:, None] * e1)
        d = np.broadcast_to(-k, o.shape).copy()
        H = np.broadcast_to(pol * 4 * r0 * r0, o.shape).copy()
    else:
        y = 2 * w - 1
        r = np.sqrt(np.maximum(0, 1 - y * y))
        local = np.stack([-r * np.sin(2 * np.pi * u), y, -r * np.cos(2 * np.pi * u)], 1)
        R = tx.rotation().astype(np.float64)
        d = local @ R.T
        H = (_pattern(local) * 4 * np.pi) @ R.T + 0j
        o = np.broadcast_to(tx.position().astype(np.float64), d.shape).copy()
    row = np.zeros(bins, np.complex128)
    length = np.zeros(budget)
    for depth in range(1, tracer.maxDepth + 1):
        t, which = _hit(tri, o, d, np.inf)
        edge = np.cross(tri[:, 1] - tri[:, 0], tri[:, 2] - tri[:, 0])
        n = _unit(edge)[which]
        n = np.where(((n * d).sum(1) > 0)[:, None], -n, n)
        cos = np.abs((n * d).sum(1))
        keep = (which >= 0) & (cos >= 1e-3) & (length < rate / slope * C0)
        o, d, H, n, cos, t, freq, length = (x[keep] for x in (o, d, H, n, cos, t, freq, length))
        if not len(o):
            break
        o = o + t[:, None] * d
        length = length + t
        d_out = d - 2 * (n * d).sum(1)[:, None] * n
        # towards the receiver
        if plane:
            k, c, _, _, _, pol = disk(rx)
            lat = o - c
            lat = lat - (lat @ k)[:, None] * k
            seen = np.linalg.norm(lat, axis=1) <= 1
            dist = np.linalg.norm(lat + c - o, axis=1)
            nd = np.broadcast_to(k, o.shape)
            Hrx = pol[None, :] * (4 * np.pi * dist)[:, None]
        else:
            R = rx.rotation().astype(np.float64)
            to = rx.position().astype(np.float64) - o
            dist = np.linalg.norm(to, axis=1)
            nd = to / dist[:, None]
            Hrx = _pattern(-nd @ R) @ R.T
            seen = np.ones(len(o), bool)
        seen &= _hit(tri, o, nd, dist)[1] < 0
        back = np.where(((nd * n).sum(1) < 0)[:, None], 0, np.cross(nd, 2 * np.cross(n, H)))
        wave = C0 / freq
        green = (1 / np.maximum(dist, 1e-3) + 2j * np.pi / wave) / (4 * np.pi * dist)
        v = (np.conj(back * green[:, None]) * Hrx).sum(1) * (length / cos) / (4 * np.pi)
        rx_pos = o + dist[:, None] * nd
        along = np.maximum(0, (d_out * (rx_pos - o)).sum(1))
        off = np.linalg.norm(o + along[:, None] * d_out - rx_pos, axis=1) / wave
        over = off > tracer.filteringRadius
        v = np.where(over, v * np.maximum(1 - 0.2 * (off / tracer.filteringRadius - 1), 0), v)
        use = seen & (v != 0)
        dt = (length[use] + dist[use]) / C0 + delay
        x = dt * slope / rate
        pos = bins * (x - np.floor(x))
        cycles = (f0 - dt * slope / 2) * dt
        value = v[use] * np.exp(2j * np.pi * (cycles - np.floor(cycles)))
        centre = np.floor(pos + 0.5).astype(np.int64)
        shift = pos - centre
        for s in range(-16, 17):
            with np.errstate(divide="ignore", invalid="ignore"):
                g = np.where(np.abs(shift) < 1e-4, 1.0 * (s == 0),
                             np.exp(1j * np.pi * shift) * np.sin(np.pi * shift) / np.pi / (shift - s))
            np.add.at(row, (centre + s) % bins, g * value)
        H = 2 * n * (n * H).sum(1)[:, None] - H
        d = d_out
    return row / budget


def _exact_rays(mesh, o, d, far):
    """Closest hits by brute force in 64 bits: distances, points and normals (the triangle
    numbers and the occlusion flags are whole numbers, with no 64-bit value of their own)."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    tri = torch.from_numpy(mesh.vertexBuffer.astype(np.float64)[mesh.indexBuffer]).to(dev)
    a, e1, e2 = tri[:, 0], tri[:, 1] - tri[:, 0], tri[:, 2] - tri[:, 0]
    O, D = (torch.from_numpy(x.astype(np.float64)).to(dev) for x in (o, d))
    # u, v and t are ratios of triple products linear in (1, o, d, o x d): matrix products
    n = torch.linalg.cross(e1, e2)
    m2, m1 = torch.linalg.cross(a, e2), torch.linalg.cross(a, e1)
    k = (a * n).sum(1)
    t_all, which = [], []
    step = max(1, int(4e7 // max(1, len(tri))))
    for i in range(0, len(O), step):
        ro, rd = O[i:i + step], D[i:i + step]
        M = torch.linalg.cross(ro, rd)
        det = -(rd @ n.T)
        # tv.(d x e2) = e2.(tv x d) ; d.(tv x e1) = -e1.(tv x d)
        u = (M @ e2.T - rd @ torch.linalg.cross(e2, a).T) / det
        v = -(M @ e1.T - rd @ torch.linalg.cross(e1, a).T) / det
        t = (ro @ n.T - k) / det
        ok = (u >= 0) & (v >= 0) & (u + v <= 1) & (t > EPS)
        t = torch.where(ok, t, torch.full_like(t, math.inf))
        tt, w = t.min(1)
        t_all.append(tt)
        which.append(w)
    t, w = torch.cat(t_all), torch.cat(which)
    hit = torch.isfinite(t)
    unit = n / n.norm(dim=1, keepdim=True)
    N = unit[w]
    N = torch.where(((N * D).sum(1) > 0)[:, None], -N, N)
    zero = torch.zeros_like(N)
    P = torch.where(hit[:, None], O + torch.where(hit, t, torch.zeros_like(t))[:, None] * D, zero)
    return [t.cpu().numpy(), P.cpu().numpy(), torch.where(hit[:, None], N, zero).cpu().numpy(), None, None]

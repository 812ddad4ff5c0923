"""Performance cases of the framework: what its users run, through its public calls.

A case is a dict of plain values.  ``listed()`` gives the named ones, ``draw``
another of the same ranges, ``prepare`` what a program holds before the call,
``run`` one pass, ``work`` what one pass cannot do without and ``exact`` the
pass's results in 64 bits from plain torch and numpy.

Kinds of case:

* ``run``: a whole simulation of a voxelized room that is already set up (the
  fields cleared, every step run, receivers read back), over schemes, storage
  types, wall models and batched fields; returned are the receiver traces and
  both pressure fields;
* ``step``: the interactive loop, one step per call with the receivers read
  after each;
* ``captures``: a run that also captures pressure slices on the way;
* ``voxelize``: a triangle mesh to node bytes;
* ``render``: receiver traces to audio (low-pass, DC blocker, resampling).
"""
from __future__ import annotations

import ctypes
import math

import numpy as np
import torch

from parallelfdtd_gb300 import _lib as L
from parallelfdtd_gb300 import geometry, materials, postfilter
from parallelfdtd_gb300.domain import Domain, default_params

DEVICE = "cuda"
N_MATERIALS = 20
FIR_ORDER = 200

# Most field bytes x steps of a drawn run (a little below the largest listed).
MOST_WORK = 2.4e11
MOST_NODES = 52_000_000


# --------------------------------------------------------------------------
# The cases

def _run_case(name, x, y, z, steps, scheme="forward", precision="f32", fields=1, boxes=0,
              dif=False, sources=1, receivers=1, lam=0.0, kind="run", captures=0):
    """lam 0: the scheme's own default."""
    c = {"kind": kind, "x": x, "y": y, "z": z, "steps": steps, "scheme": scheme,
         "precision": precision, "fields": fields, "boxes": boxes, "dif": dif,
         "sources": sources, "receivers": receivers, "lam": lam, "captures": captures}
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # A viewer's loop over a small room: each call a step, latency is all.
        _run_case("step_48x40x36_f32", 48, 40, 36, 24, kind="step", receivers=2),
        # The shoebox of the first benchmark configuration: 500 short steps.
        _run_case("shoebox_64_f32", 64, 64, 64, 500),
        # A room as a mesh gives it, with odd sizes on every axis.
        _run_case("odd_203x155x119_f32", 203, 155, 119, 300, boxes=12, sources=2, receivers=4),
        # An ordinary room with the centred scheme.
        _run_case("centred_240x200x160_f32", 240, 200, 160, 200, scheme="centred", boxes=16,
                  receivers=4),
        # The headline configuration: 50 M nodes, 40 boxes, 8 receivers.
        _run_case("room_512x384x256_f32", 512, 384, 256, 300, boxes=40, receivers=8),
        # Double precision, for reference responses.
        _run_case("room_256x192x128_f64", 256, 192, 128, 150, precision="f64", boxes=16,
                  receivers=4),
        # 16-bit storage, for rooms that would not fit or finish otherwise.
        _run_case("room_384x320x256_f16", 384, 320, 256, 200, precision="f16", boxes=30,
                  receivers=4),
        # The 27-point scheme with third-order filters on every wall.
        _run_case("iwb_dif_512x384x256_f32", 512, 384, 256, 100, scheme="iwb", boxes=40, dif=True,
                  receivers=8),
        # Frequency-dependent walls, with slices captured for a film.
        _run_case("film_dif_240x180x120_f32", 240, 180, 120, 200, boxes=16, dif=True, receivers=4,
                  kind="captures", captures=10),
        # 16 source positions of one room at once.
        _run_case("batch16_384x320x256_f32", 384, 320, 256, 60, fields=16, boxes=30, sources=16,
                  receivers=64),
        # The mesh of a furnished room to voxels.
        {"name": "voxelize_512x384x256", "kind": "voxelize", "x": 512, "y": 384, "z": 256,
         "boxes": 40, "spheres": 2},
        # The receivers of a run to audio.
        {"name": "render_16x8000", "kind": "render", "channels": 16, "samples": 8000, "fs": 36000,
         "fs_out": 48000},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choices(["run", "step", "captures", "voxelize", "render"], [12, 1, 2, 1, 1])[0]
    if kind == "render":
        return {"kind": kind, "channels": _log_int(rng, 1, 64), "samples": _log_int(rng, 500, 16000),
                "fs": rng.choice([16000, 24000, 32000, 36000, 64000, 96000]), "fs_out": 48000}
    if kind == "voxelize":
        while True:
            x, y, z = (_log_int(rng, 40, 512) for _ in range(3))
            if x * y * z <= MOST_NODES:
                return {"kind": kind, "x": x, "y": y, "z": z, "boxes": rng.randint(0, 40),
                        "spheres": rng.randint(0, 2)}
    if kind == "step":
        x, y, z = (_log_int(rng, 24, 128) for _ in range(3))
        return _run_case("", x, y, z, rng.randint(10, 24), kind=kind,
                         precision=rng.choice(["f32", "f32", "f64"]),
                         scheme=rng.choice(["forward", "centred"]), receivers=rng.randint(1, 4))
    scheme = rng.choices(["forward", "centred", "iwb"], [4, 2, 2])[0]
    precision = rng.choices(["f32", "f64", "f16", "bf16"], [5, 1, 1, 1])[0]
    fields = 1
    if kind == "run" and scheme != "iwb":
        fields = rng.choices([1, 4, 8, 16], [8, 1, 1, 1])[0]
    size = {"f32": 4, "f64": 8, "f16": 2, "bf16": 2}[precision] * fields
    while True:
        x, y, z = (_log_int(rng, 32, 512) for _ in range(3))
        if rng.random() < 0.5:
            x = max(32, x // 16 * 16)
        n = x * y * z
        if n > MOST_NODES or n * size > 2.4e9:
            continue
        # 16-bit rounding travels far in many steps; keep the results telling
        steps = _log_int(rng, 40, 500 if size >= 4 * fields else 120)
        # FP64 runs at a tenth of the rate, the 27-point fallback at less
        per_node = (3 * size + 1) * (4 if precision == "f64" else 1) * (2 if scheme == "iwb" else 1)
        steps = max(10, min(steps, int(MOST_WORK / (n * per_node))))
        return _run_case("", x, y, z, steps, scheme=scheme, precision=precision, fields=fields,
                         boxes=rng.randint(0, 40) if min(x, y, z) >= 48 else rng.randint(0, 4),
                         dif=rng.random() < 0.3, sources=max(fields, rng.randint(1, 3)),
                         receivers=rng.randint(1, 4) * fields,
                         # the 27-point scheme in 16 bits needs lambda below its limit
                         lam=0.99 if scheme == "iwb" and size < 4 else 0.0,
                         kind=kind, captures=rng.randint(1, 12) if kind == "captures" else 0)


# --------------------------------------------------------------------------
# Rooms

# Voxelizer boundary id by the set of missing (solid) neighbours, bits
# -x 1, +x 2, -y 4, +y 8, -z 16, +z 32 (0 where both sides of an axis are).
_ID = np.zeros(64, np.uint8)
for _mask, _id in ((0, 27), (32, 21), (4, 22), (8, 23), (1, 24), (2, 25), (16, 26), (40, 9),
                   (36, 10), (34, 11), (33, 12), (24, 13), (20, 14), (18, 15), (17, 16), (10, 17),
                   (9, 18), (6, 19), (5, 20), (42, 1), (41, 2), (38, 3), (37, 4), (26, 5), (25, 6),
                   (22, 7), (21, 8)):
    _ID[_mask] = _id

_AXES = ((2, 1, 0), (2, -1, 0), (1, 1, 0), (1, -1, 0), (0, 1, 0), (0, -1, 0))


def _shifted(a, bit):
    """a's value at the neighbour of each node (order -x, +x, -y, +y, -z, +z)."""
    axis, by, _ = _AXES[bit]
    return torch.roll(a, by, axis)


class Room:
    """A shell one node thick with solid boxes inside, in the voxelizer's form:
    boundary ids and materials, x fastest."""

    def __init__(self, dims, n_boxes, seed):
        x, y, z = dims
        rng = np.random.default_rng(seed)
        solid = torch.zeros((z, y, x), dtype=torch.bool, device=DEVICE)
        smat = torch.zeros((z, y, x), dtype=torch.uint8, device=DEVICE)
        faces = ((2, 0), (2, x - 1), (1, 0), (1, y - 1), (0, 0), (0, z - 1))
        for m, (axis, at) in enumerate(faces):
            solid.select(axis, at).fill_(True)
            smat.select(axis, at).fill_(m)
        longest = [max(9, min(64, d // 3)) for d in (x, y, z)]
        for _ in range(n_boxes):
            e = [int(rng.integers(8, m)) for m in longest]
            a = [int(rng.integers(1, max(2, d - 1 - w))) for d, w in zip((x, y, z), e)]
            b = [min(s + w, d - 1) for s, w, d in zip(a, e, (x, y, z))]
            solid[a[2]:b[2], a[1]:b[1], a[0]:b[0]] = True
            smat[a[2]:b[2], a[1]:b[1], a[0]:b[0]] = int(rng.integers(0, N_MATERIALS))
        table = torch.from_numpy(_ID).to(DEVICE)
        while True:  # an air node with solid on both sides of an axis has no id: fill it
            missing = torch.zeros_like(smat)
            first = torch.zeros_like(smat)
            for bit in range(5, -1, -1):
                s = _shifted(solid, bit)
                missing |= s.to(torch.uint8) << bit
                first = torch.where(s, _shifted(smat, bit), first)
            ids = table[missing.to(torch.int32)]
            bad = (ids == 0) & ~solid
            if not bool(bad.any()):
                break
            smat = torch.where(bad, first, smat)
            solid = solid | bad
        ids[solid] = 0
        self.dims = dims
        self.solid = solid
        self.missing = torch.where(solid, torch.zeros_like(missing), missing)
        self.ids = ids
        self.mat = torch.where((ids > 0) & (ids < 27), first, torch.zeros_like(first))
        self.air = (ids == 27).reshape(-1).nonzero().reshape(-1)

    def places(self, n, rng):
        """n places (x, y, z) in the air."""
        x, y, _ = self.dims
        at = self.air[torch.from_numpy(rng.integers(0, self.air.numel(), n)).to(DEVICE)].cpu().numpy()
        return np.stack([at % x, at // x % y, at // (x * y)], axis=1)

    def near(self, centres, rng):
        """A place in the air not far from each of `centres`, so that a short
        run's sound arrives."""
        some = self.places(512 * len(centres), rng).reshape(len(centres), 512, 3)
        off = ((some - centres[:, None]) ** 2).sum(axis=2).argmin(axis=1)
        return some[np.arange(len(centres)), off]


def _pulses(rng, n, steps):
    """Short band-limited pulses, one a source."""
    t = np.arange(steps)[None, :]
    sigma = rng.uniform(2.0, 4.0, (n, 1))
    return rng.uniform(0.5, 1.5, (n, 1)) * np.exp(-0.5 * ((t - 4.0 * sigma) / sigma) ** 2)


def _inputs(case, seed):
    """Everything that describes the simulation: room, walls, sources, receivers."""
    rng = np.random.default_rng([seed, 1])
    room = Room((case["x"], case["y"], case["z"]), case["boxes"], [seed, 2])
    k = case["fields"]
    lam = case["lam"] or None
    n_src, n_rec = case["sources"], case["receivers"]
    src = room.places(n_src, rng)
    rec_field = np.arange(n_rec) % k
    q = {
        "room": room,
        "params": default_params(0, case["scheme"], lam),
        "admittance": rng.uniform(0.01, 0.9, N_MATERIALS),
        "filters": None,
        "src": src,
        "src_field": np.arange(n_src) % k,
        "pulses": _pulses(rng, n_src, case["steps"]),
        "rec": room.near(src[rec_field], rng),
        "rec_field": rec_field,
    }
    if case["dif"]:
        rows = materials.positive_real_filters(N_MATERIALS, 3, seed=int(rng.integers(1 << 30)))
        q["filters"] = materials.dif_table(rows, 3)
    if case["captures"]:
        # planes through the first source, one axis after the other
        every = max(1, case["steps"] // case["captures"])
        q["captures"] = [(min(case["steps"], (i + 1) * every), i % 3, int(src[0][2 - i % 3]))
                         for i in range(case["captures"])]
    return q


# --------------------------------------------------------------------------
# Meshes

def _sphere(centre, radius, material, around=24, rings=12):
    """A closed sphere of triangles."""
    phi = np.linspace(0, math.pi, rings + 1)[1:-1]
    theta = np.arange(around) * (2 * math.pi / around)
    ring = np.stack([np.outer(np.sin(phi), np.cos(theta)), np.outer(np.sin(phi), np.sin(theta)),
                     np.outer(np.cos(phi), np.ones(around))], axis=2).reshape(-1, 3)
    v = np.concatenate([ring, [[0, 0, 1], [0, 0, -1]]]) * radius + np.asarray(centre)
    top, bottom, t = len(ring), len(ring) + 1, []
    for i in range(around):
        j = (i + 1) % around
        t.append((top, i, j))
        last = (rings - 2) * around
        t.append((bottom, last + j, last + i))
        for r in range(rings - 2):
            a, b = r * around, (r + 1) * around
            t += [(a + i, b + i, b + j), (a + i, b + j, a + j)]
    t = np.array(t, np.uint32)
    return v.astype(np.float32), t, np.full(len(t), material, np.uint8)


def _mesh(case, seed):
    """A room's box with boxes and spheres in it, each in a cell of its own."""
    rng = np.random.default_rng([seed, 3])
    edge = 0.05
    size = np.array([case["x"], case["y"], case["z"]]) * edge - 2.3 * edge
    parts = [geometry.box_mesh((0, 0, 0), size, list(range(6)))]
    n = case["boxes"] + case["spheres"]
    side = max(1, math.ceil(n ** (1 / 3)))
    cells = rng.permutation(side ** 3)[:n]
    for i, c in enumerate(cells):
        lo = np.array([c % side, c // side % side, c // (side * side)]) * size / side
        cell = size / side
        m = int(rng.integers(0, N_MATERIALS))
        if i < case["spheres"]:
            parts.append(_sphere(lo + cell / 2, 0.35 * cell.min(), m))
        else:
            a = lo + cell * rng.uniform(0.1, 0.4, 3)
            b = lo + cell * rng.uniform(0.5, 0.9, 3)
            parts.append(geometry.box_mesh(a, b, [m] * 6))
    return geometry.merge(*parts) + (edge,)


# --------------------------------------------------------------------------
# Before the call, and the call

def prepare(case, seed):
    if case["kind"] == "render":
        rng = np.random.default_rng([seed, 4])
        x = rng.standard_normal((case["channels"], case["samples"]))
        decay = np.exp(-np.arange(case["samples"]) / (0.2 * case["samples"]))
        return {"case": case, "traces": x * decay}
    if case["kind"] == "voxelize":
        return {"case": case, "mesh": _mesh(case, seed)}
    q = _inputs(case, seed)
    room = q["room"]
    d = Domain(room.dims, case["precision"], fields=case["fields"])
    d.set_scheme(case["scheme"])
    d.set_voxels(room.ids.reshape(-1).cpu().numpy(), room.mat.reshape(-1).cpu().numpy(),
                 centred=case["scheme"] != "forward")
    d.set_materials(np.repeat(q["admittance"][:, None], 20, axis=1))
    d.set_params(q["params"])
    if q["filters"] is not None:
        d.set_dif_filters(np.ones(N_MATERIALS, np.int32), q["filters"])
    d.set_sources(q["src"], [L.SRC_SOFT] * len(q["src"]), q["pulses"], fields=q["src_field"])
    d.set_receivers(q["rec"], fields=q["rec_field"])
    return {"case": case, "domain": d, "captures": q.get("captures")}


_TYPES = {"f32": ("<f4", None), "f64": ("<f8", None), "f16": ("<f2", None),
          "bf16": ("<i2", torch.bfloat16)}


class _Field:
    """A domain's pressure field where it lies, for torch; keeps the domain."""

    def __init__(self, d, which, typestr):
        p = ctypes.c_void_p()
        L.call("pfdtd_get_field_ptr", d.handle, which, ctypes.byref(p))
        x, y, z = d.dims
        self.domain = d
        self.__cuda_array_interface__ = {
            "shape": (z * y * x, d.fields), "typestr": typestr, "data": (p.value, False),
            "version": 3}


def _field(d, which, precision):
    typestr, view = _TYPES[precision]
    t = torch.as_tensor(_Field(d, which, typestr), device=DEVICE)
    return t.view(view) if view is not None else t


def run(state):
    case = state["case"]
    if case["kind"] == "render":
        return {"audio": postfilter.render(state["traces"], case["fs"], fs_out=case["fs_out"])}
    if case["kind"] == "voxelize":
        v, t, m, edge = state["mesh"]
        ids, mat, _, _ = geometry.voxelize(v, t, m, edge)
        return {"ids": ids, "mat": mat}
    d, steps = state["domain"], case["steps"]
    d.reset_fields()
    out = {}
    if case["kind"] == "step":
        out["receivers"] = np.zeros((d.n_rec, steps), np.float64 if case["precision"] == "f64"
                                    else np.float32)
        for n in range(steps):
            d.step(n, 1, out["receivers"], steps)
    elif case["kind"] == "captures":
        out["receivers"], slices = d.run_captures(steps, state["captures"])
        out["slices"] = [p for p, _ in slices]
        out["nodes"] = [q for _, q in slices]
    else:
        out["receivers"], _, _ = d.run(steps)
    out["pressure"] = _field(d, L.FIELD_CURRENT, case["precision"])
    out["past"] = _field(d, L.FIELD_PAST, case["precision"])
    return out


# --------------------------------------------------------------------------
# What a pass cannot do without

def work(case):
    """Inputs read once, outputs written once, and the update's operations."""
    if case["kind"] == "render":
        n = case["channels"] * case["samples"]
        out = n * case["fs_out"] / case["fs"]
        return {"bytes": 8 * (n + out), "flops": 2 * n * (FIR_ORDER + 1) + 42 * out}
    if case["kind"] == "voxelize":
        return {"bytes": 2 * case["x"] * case["y"] * case["z"], "flops": 0}
    n = case["x"] * case["y"] * case["z"]
    size = {"f32": 4, "f64": 8, "f16": 2, "bf16": 2}[case["precision"]] * case["fields"]
    traces = case["receivers"] * case["steps"] * (8 if case["precision"] == "f64" else 4)
    per = 34 if case["scheme"] == "iwb" else 13 if case["scheme"] == "centred" else 11
    return {"bytes": n * (2 + 2 * size) + traces, "flops": per * n * case["fields"] * case["steps"]}


# --------------------------------------------------------------------------
# In 64 bits

def _low_pass(cutoff, n):
    k = np.arange(n) - (n - 1) / 2
    return cutoff * np.sinc(cutoff * k)


def _exact_render(case, seed):
    x = prepare(case, seed)["traces"]
    h = _low_pass(0.2, FIR_ORDER + 1) * np.hamming(FIR_ORDER + 1)
    h /= h.sum()
    y = np.stack([np.convolve(c, h)[:x.shape[1]] for c in x])
    fn = 10.0 / case["fs"]
    a = (math.sqrt(3) - 2 * math.sin(math.pi * fn)) / (
        math.sin(math.pi * fn) + math.sqrt(3) * math.cos(math.pi * fn))
    d = np.diff(y, axis=1, prepend=0.0)
    for n in range(1, d.shape[1]):
        d[:, n] += a * d[:, n - 1]
    g = math.gcd(case["fs_out"], case["fs"])
    up, down = case["fs_out"] // g, case["fs"] // g
    if up == down:
        return {"audio": d.T}
    top = max(up, down)
    h = _low_pass(1.0 / top, 20 * top + 1) * np.kaiser(20 * top + 1, 5.0)
    h *= up / h.sum()
    count = -(-d.shape[1] * up // down)
    out = []
    for c in d:
        wide = np.zeros(c.size * up)
        wide[::up] = c
        full = np.convolve(wide, h)[10 * top:]
        full = np.pad(full, (0, max(0, count * down - full.size)))
        out.append(full[::down][:count])
    return {"audio": np.stack(out, axis=1)}


class _Exact:
    """The update in 64 bits on flat arrays [nodes, fields] with a margin."""

    def __init__(self, case, q):
        room = q["room"]
        x, y, z = room.dims
        self.scheme, self.x, self.xy, self.n = case["scheme"], x, x * y, x * y * z
        self.pad = x + 8
        lam, l2 = float(q["params"][0]), float(q["params"][1])
        self.lam, self.l2 = lam, l2
        f8 = dict(dtype=torch.float64, device=DEVICE)
        inside = (~room.solid).reshape(-1)
        missing = room.missing.reshape(-1)
        side = [((missing >> b) & 1).to(torch.uint8) for b in range(6)]
        solid_sides = sum(side[1:], side[0])
        mat = room.mat.reshape(-1).to(torch.int64)
        self.p = [torch.zeros((self.n + 2 * self.pad, case["fields"]), **f8) for _ in range(2)]
        self.mirror = None
        if self.scheme == "iwb":
            closed = torch.zeros(self.n, dtype=torch.uint8, device=DEVICE)
            for dz in (-1, 0, 1):
                for dy in (-1, 0, 1):
                    for dx in (-1, 0, 1):
                        far = abs(dx) + abs(dy) + abs(dz)
                        if far:
                            s = torch.roll(room.solid, (-dz, -dy, -dx), (0, 1, 2)).reshape(-1)
                            closed += s.to(torch.uint8) * (8 >> far)
            self.own = (closed.double() / 16)[:, None]
            gain = lam * (closed.double() / 16) * (solid_sides > 0)
            self.b = 2 - 3.5 * l2
        elif self.scheme == "centred":
            gain = lam * solid_sides.double()
            self.b = -(2 - 6 * l2)
            self.mirror = side
        else:
            gain = 0.5 * lam * solid_sides.double()
            self.b = (2 - (6 - solid_sides.double()) * l2)[:, None]
        gain = gain * inside
        f = None
        if q["filters"] is not None:
            f = torch.from_numpy(q["filters"]).to(DEVICE)[mat]
            beta = gain * f[:, 0]
        else:
            beta = gain * torch.from_numpy(q["admittance"]).to(DEVICE)[mat]
        self.a = (inside / (1 + beta))[:, None]
        self.c = (1 - beta)[:, None]
        self.dif = None
        if f is not None:
            at = ((gain > 0) & inside).nonzero().reshape(-1)
            self.dif = at
            self.f = f[at][:, :, None]
            self.g2 = 2 * gain[at][:, None]
            self.s = torch.zeros((3, at.numel(), case["fields"]), **f8)

    def at(self, p, off):
        lo = self.pad + self.xy + off
        return p[lo:lo + self.n - 2 * self.xy]

    def step(self):
        p, pp = self.p
        mid = slice(self.xy, self.n - self.xy)
        at, x, xy = self.at, self.x, self.xy
        s = at(p, 1) + at(p, -1)
        s += at(p, x)
        s += at(p, -x)
        s += at(p, xy)
        s += at(p, -xy)
        own = at(p, 0)
        if self.scheme == "iwb":
            s *= 0.25
            for w, offs in ((0.125, [dy * x + dx for dy in (-1, 1) for dx in (-1, 1)]
                             + [dz * xy + d for dz in (-1, 1) for d in (-1, 1, -x, x)]),
                            (0.0625, [dz * xy + dy * x + dx for dz in (-1, 1) for dy in (-1, 1)
                                      for dx in (-1, 1)])):
                for o in offs:
                    s.add_(at(p, o), alpha=w)
            s.addcmul_(own, self.own[mid])
        elif self.mirror is not None:
            for b, o in enumerate((1, -1, x, -x, xy, -xy)):  # the neighbour across the node
                s.addcmul_(at(p, o), self.mirror[b][mid][:, None].double())
        s *= self.l2
        if isinstance(self.b, float):
            s.add_(own, alpha=self.b)
        else:
            s.addcmul_(own, self.b[mid])
        old = at(pp, 0)
        s.addcmul_(old, self.c[mid], value=-1)
        if self.dif is not None:
            k = self.dif - xy
            was = old[k]
            s[k] -= self.g2 * self.s[0]
        s *= self.a[mid]
        if self.dif is not None:
            v = 0.5 * (s[k] - was)
            f, st = self.f, self.s
            y = f[:, 0] * v + st[0]
            st[0] = f[:, 1] * v - f[:, 4] * y + st[1]
            st[1] = f[:, 2] * v - f[:, 5] * y + st[2]
            st[2] = f[:, 3] * v - f[:, 6] * y
        old.copy_(s)
        self.p = [pp, p]

    def whole(self, which):
        return self.p[which][self.pad:self.pad + self.n]


def _exact_run(case, seed):
    q = _inputs(case, seed)
    x, y, z = q["room"].dims
    e = _Exact(case, q)
    flat = lambda a: torch.from_numpy(a[:, 2] * x * y + a[:, 1] * x + a[:, 0]).to(DEVICE)  # noqa: E731
    src, rec = flat(q["src"]), flat(q["rec"])
    src_field = torch.from_numpy(q["src_field"]).to(DEVICE)
    rec_field = torch.from_numpy(q["rec_field"]).to(DEVICE)
    dtype = np.float64 if case["precision"] == "f64" else np.float32
    pulses = torch.from_numpy(q["pulses"].astype(dtype).astype(np.float64)).to(DEVICE)
    traces = torch.zeros((len(rec), case["steps"]), dtype=torch.float64, device=DEVICE)
    captures = q.get("captures") or []
    slices = [None] * len(captures)
    for n in range(case["steps"]):
        e.whole(0).index_put_((src, src_field), pulses[:, n], accumulate=True)
        e.step()
        traces[:, n] = e.whole(0)[rec, rec_field]
        for i, (at, orientation, place) in enumerate(captures):
            if at == n + 1:
                s = e.whole(0)[:, 0].reshape(z, y, x).select(orientation, place).clone()
                if orientation:
                    s[-1] = 0
                slices[i] = s
    out = {"receivers": traces, "pressure": e.whole(0), "past": e.whole(1)}
    if case["kind"] == "captures":
        out |= {"slices": slices, "nodes": None}
    return out


def exact(case, seed):
    if case["kind"] == "voxelize":
        return None  # bytes
    return _exact_render(case, seed) if case["kind"] == "render" else _exact_run(case, seed)

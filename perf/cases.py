"""The work whose time this repository watches, through its public entry points.

A case is one extraction (or one batch of extractions) as a program makes it:
the workspace and its CUDA graph are made once (``prepare``), and a pass
(``run``) replays the graph, reads the status, and takes the triangles in a
reproducible order.  Replays append polygons and triangles in an order that
varies, so a program that compares or stores results sorts them; ``_ordered``
does so on the GPU by a digest of each triangle's coordinates and labels, into
buffers that the program keeps (zeros past the triangles).

Kinds of scene (all seeded; see ``peel_b200.scenes``):
  icospheres   two nested noisy spheres, orthographic: the smallest meshes
  knot         a noisy tube swept along a torus knot, pinhole: a connected,
               depth-complex mesh (15 to 25 layers)
  stack        congruent triangles above one another, orthographic: as many
               layers as faces
  primitives   disjoint noisy spheres and tori, pinhole
  overlap      crossing spheres and tori, resolved into a mesh on the host
               first (deep: up to 70 layers)
  crossing     crossing spheres and tori, not resolved: DevicePeeler input
  batch        many small meshes and views in one graph replay
"""

import math
import sys
from dataclasses import replace
from pathlib import Path

import numpy as np
import torch

ROOT = Path(__file__).resolve().parents[1]
if str(ROOT / "exact-depth-peeling_b200") not in sys.path:
    sys.path.insert(0, str(ROOT / "exact-depth-peeling_b200"))

from peel_b200 import BatchPeeler, Capacities, DevicePeeler, scenes  # noqa: E402
from peel_b200.sizing import fit_event_capacities  # noqa: E402

DEVICE = "cuda:0"


def _case(name, kind, faces, peeler="event", predicates="filtered64", layers=0, count=0):
    """``faces``: about how many; ``layers``: 0 = all; ``count``: primitives,
    or scenes of a batch."""
    case = {"name": name, "kind": kind, "faces": faces, "peeler": peeler,
            "predicates": predicates, "layers": layers, "count": count}
    return {k: v for k, v in case.items() if not (k == "name" and name is None)}


def listed():
    return [
        # A small object per call, as an interactive tool peels it.
        _case("icospheres-640", "icospheres", 640),
        # The smallest benchmark mesh, at its own size.
        _case("icospheres-2560", "icospheres", 2560),
        # Only the nearest layers, as a renderer of transparency takes them.
        _case("knot-9702-layers4", "knot", 9702, layers=4),
        # The headline mesh.
        _case("knot-65536", "knot", 65536),
        # The plain binary64 predicates, on a ragged knot.
        _case("knot-63000-binary64", "knot", 63000, predicates="binary64"),
        # As many layers as faces: the deepest hit groups there are.
        _case("stack-65536", "stack", 65536),
        # A packed scene of middling size.
        _case("primitives-24001", "primitives", 24001, count=9),
        # The large benchmark mesh.
        _case("primitives-720000", "primitives", 720000, count=40),
        # A resolved crossing scene: deep, with many slivers along the crossings.
        _case("overlap-50000", "overlap", 50000, count=12),
        # Many small meshes and views in one replay.
        _case("batch-16", "batch", 4096, count=16),
        # Iterative clipping of a mesh that needs no resolving.
        _case("device-icospheres-2560", "icospheres", 2560, peeler="device"),
        # Iterative clipping of a scene whose surfaces cross.
        _case("device-crossing-1000", "crossing", 1000, peeler="device", count=6),
    ]


def draw(rng):
    def size(lo, hi):
        return int(math.exp(rng.uniform(math.log(lo), math.log(hi))))

    kind = rng.choice(("icospheres", "knot", "knot", "stack", "primitives", "primitives",
                       "overlap", "batch", "device", "device"))
    predicates = rng.choice(("filtered64", "filtered64", "binary64"))
    if kind == "icospheres":
        return _case(None, kind, size(200, 10000), predicates=predicates)
    if kind == "knot":
        return _case(None, kind, size(2000, 65536), predicates=predicates,
                     layers=rng.choice((0, 0, 3, 6)))
    if kind == "stack":
        return _case(None, kind, size(2000, 65536), predicates=predicates)
    if kind == "primitives":
        return _case(None, kind, size(4096, 400000), predicates=predicates,
                     count=rng.randint(4, 40))
    if kind == "overlap":
        return _case(None, kind, size(5000, 50000), predicates=predicates,
                     count=rng.randint(4, 12))
    if kind == "batch":
        return _case(None, kind, size(1024, 6000), predicates=predicates,
                     count=rng.randint(4, 16))
    return _case(None, *rng.choice((("icospheres", size(200, 2560)),
                                    ("crossing", size(200, 1000)))),
                 peeler="device", count=rng.randint(3, 6))


# ---------------------------------------------------------------- scenes
def _direction(rng):
    v = rng.normal(size=3)
    return v / np.linalg.norm(v)


def _uv_sphere(faces):
    """Unit sphere of about ``faces`` triangles (latitude rings)."""
    rings = max(3, int(round(math.sqrt(faces / 4.0))) + 1)
    segments = max(3, int(round(faces / (2.0 * (rings - 1)))))
    return scenes.uv_sphere(rings, segments, 1.0, 0.0, np.random.default_rng(0))


def _icospheres(faces, rng):
    """Two nested noisy spheres seen down -z: icospheres where the size is one
    of theirs (2 x 20 x 4^k faces), latitude spheres else."""
    level = round(math.log(max(faces, 40) / 40.0, 4))
    v, f = scenes.icosphere(level) if 40 * 4 ** level == faces else _uv_sphere(faces / 2)
    outer = v * (1 + rng.uniform(-0.15, 0.15, size=(len(v), 1)))
    inner = 0.5 * v * (1 + rng.uniform(-0.15, 0.15, size=(len(v), 1)))
    vertices = np.concatenate([outer, inner])
    lo, hi = vertices[:, :2].min(0), vertices[:, :2].max(0)
    pad = 0.05 * (hi - lo)
    return (vertices, np.concatenate([f, f + len(v)]).astype(np.int32),
            np.diag([1.0, 1.0, -1.0, 1.0]), np.array([*(lo - pad), *(hi + pad), 0.0, 0.01]))


def _knot(faces, seed):
    """rings x segments quads: 256 x 128 for 65,536 faces; otherwise about
    twice as many rings as segments, whatever the remainder."""
    segments = max(8, int(round(math.sqrt(faces / 4.0))))
    return scenes.knot_tube(max(24, faces // (2 * segments)), segments, seed=seed)


def _scene(kind, faces, count, seed):
    """Host arrays (vertices, faces, camera, settings) of one scene."""
    rng = np.random.default_rng(seed)
    if kind == "icospheres":
        return _icospheres(faces, rng)
    if kind == "knot":
        return _knot(faces, seed)
    if kind == "stack":
        vertices, f, camera, settings = scenes.stress_stack(faces, 0.0)
        # Another footprint for each seed, one for all triangles of a stack.
        vertices[:, :2] *= rng.uniform(0.7, 1.2)
        vertices[:, :2] += rng.uniform(-0.05, 0.05, size=2)
        return vertices, f, camera, settings
    if kind == "primitives":
        return scenes.packed_primitives(faces, count, seed=seed)
    if kind == "overlap":
        v, f, camera, settings = scenes.overlapping_primitives(faces, count, seed=seed)
        v, f, _, _ = scenes.resolve_mesh(v, f)
        return v, f, camera, settings
    return scenes.overlapping_primitives(faces, count, seed=seed)  # crossing


def _batch(faces, count, seed):
    """Half views of one knot on a turntable, half packed primitives of half to
    twice the faces."""
    rng = np.random.default_rng(seed)
    v, f, _, _ = _knot(faces, seed)
    views = [(v, f, c, s) for c, s in scenes.turntable_views(v, count // 2, seed=seed)]
    meshes = [scenes.packed_primitives(int(faces * 2 ** rng.uniform(-1, 1)), 3, seed=seed + k,
                                       direction=_direction(rng))
              for k in range(count - count // 2)]
    return views + meshes


# ---------------------------------------------------------------- passes
# Triangles per face: what the full extractions give on average at the listed
# sizes, and the room for them in the program's buffers.
_TRIANGLES = {"icospheres": (15.0, 64), "knot": (30.0, 56), "stack": (3.0, 3),
              "primitives": (20.0, 72), "overlap": (13.0, 40), "crossing": (6.0, 64),
              "batch": (10.0, 48)}


def _room(case):
    faces = case["faces"] * (2 * case["count"] if case["kind"] == "batch" else 1)
    if case["kind"] == "overlap":
        faces *= 2  # resolved faces
    return _TRIANGLES[case["kind"]][1] * faces


def _buffers(room, device=DEVICE):
    return {"uv": torch.zeros(room, 3, 2, dtype=torch.float64, device=device),
            "world": torch.zeros(room, 3, 3, dtype=torch.float64, device=device),
            "sources": torch.zeros(room, dtype=torch.int32, device=device),
            "layers": torch.zeros(room, dtype=torch.int32, device=device)}


def _mix(device=DEVICE):
    """Odd 64-bit multipliers of the digest, one per coordinate and label."""
    words = np.random.default_rng(20).integers(0, 1 << 63, size=8, dtype=np.int64) | 1
    return torch.from_numpy(words[:6].copy()).to(device), int(words[6]), int(words[7])


def prepare(case, seed):
    options = {"predicates": case["predicates"]}
    state = {}
    if case["peeler"] != "device":
        state = {"mesh": _buffers(_room(case)), "mix": _mix()}
    if case["kind"] == "batch":
        arrays = [scenes.to_device(s, DEVICE)
                  for s in _batch(case["faces"], case["count"], seed)]
        state["batch"] = BatchPeeler(arrays, fit=True, **options)
        state["batch"].capture()
        sizes = [p.n for p in state["batch"].peelers]
        state["firsts"] = [sum(sizes[:k]) for k in range(len(sizes))]
        return state
    for attempt in range(12):
        try:
            arrays = scenes.to_device(
                _scene(case["kind"], case["faces"], case["count"], seed + 7919 * attempt), DEVICE)
            state["peeler"] = _peeler(case, arrays, options)
            break
        except RuntimeError as error:
            # A few random scenes exceed the fixed per-edge noding capacity or
            # the pools: the next scene stands in.
            if attempt == 11 or "GPU extraction failed" not in str(error):
                raise
    if case["peeler"] == "device":
        state["coverage"] = torch.zeros(state["peeler"].cap.layers, 2 * case["faces"],
                                        dtype=torch.float64, device=DEVICE)
    state["peeler"].capture()
    return state


def _peeler(case, arrays, options):
    if case["peeler"] != "device":
        return fit_event_capacities(arrays, attempts=12, headroom=1.25, layers=case["layers"],
                                    **options)[0]
    n = arrays[1].shape[0]
    capacities = replace(Capacities.for_mesh(n), residual=16 * n, triangles=128 * n,
                         vertices=128 * n)
    peeler = DevicePeeler(*arrays, capacities=capacities, **options)
    peeler.run()
    peeler.read_status()
    return peeler


def _ordered(triangles, mesh, mix):
    """The triangles sorted by a 64-bit digest of their image coordinates,
    source and layer: one order for one set of triangles."""
    uv, _, sources, layers = triangles
    words, for_source, for_layer = mix
    key = (uv.view(torch.int64).reshape(-1, 6) * words).sum(1)
    key.add_(sources, alpha=for_source).add_(layers, alpha=for_layer)
    order = torch.sort(key)[1]
    for buffer, values in zip(mesh.values(), triangles):
        torch.index_select(values, 0, order, out=buffer[:len(order)])
    return mesh


def _coverage(triangles, coverage):
    """[layers, faces]: the image area of each face in each layer.  Iterative
    clipping cuts the same regions into pieces that depend on the order of its
    queues, so their areas are what one replay has in common with the next."""
    uv, _, sources, layers = triangles
    u, v = uv[:, 1] - uv[:, 0], uv[:, 2] - uv[:, 0]
    area = 0.5 * (u[:, 0] * v[:, 1] - u[:, 1] * v[:, 0])
    place = layers.long() * coverage.shape[1] + sources
    coverage.zero_()
    coverage.view(-1).index_add_(0, place, area)
    return coverage


def _triangles(p, count):
    return (p.triangles_uv[:count], p.triangles_world[:count], p.triangle_sources[:count],
            p.triangle_layers[:count])


def run(state):
    if "batch" in state:
        batch = state["batch"]
        batch.run()
        infos = batch.read_status()
        with torch.cuda.stream(batch.stream):
            parts = [_triangles(p, i["triangles"]) for p, i in zip(batch.peelers, infos)]
            parts = [(uv, world, sources + first, layers)  # faces numbered through the batch
                     for (uv, world, sources, layers), first in zip(parts, state["firsts"])]
            columns = [torch.cat(column) for column in zip(*parts)]
            mesh = _ordered(columns, state["mesh"], state["mix"])
        return {**mesh, "polygons": [i["polygons"] for i in infos],
                "depth": [i["layers"] for i in infos]}
    peeler = state["peeler"]
    peeler.run()
    info = peeler.read_status()
    if "coverage" in state:
        with torch.cuda.stream(peeler.stream):
            coverage = _coverage(_triangles(peeler, info["triangles"]), state["coverage"])
        return {"coverage": coverage, "depth": info["layers"]}
    with torch.cuda.stream(peeler.stream):
        mesh = _ordered(_triangles(peeler, info["triangles"]), state["mesh"], state["mix"])
    return {**mesh, "polygons": info["polygons"], "depth": info["layers"]}


def work(case):
    """Inputs read once (24 bytes a vertex, half as many vertices as faces;
    12 bytes a face) and outputs written once (128 bytes a triangle)."""
    faces = case["faces"] * (case["count"] if case["kind"] == "batch" else 1)
    triangles = _TRIANGLES[case["kind"]][0] * faces
    if case["layers"]:
        triangles *= 0.4
    return {"bytes": 24 * faces + 176 + 128 * triangles, "flops": 0}


def exact(case, seed):
    """The stack's layers are its faces in order of depth, each a fan of three
    triangles around its centroid.  The other kinds' arrangements have no short
    binary64 restatement: None."""
    if case["kind"] != "stack" or case["layers"]:
        return None
    vertices, faces, _, settings = _scene("stack", case["faces"], 0, seed)
    corners = vertices[faces].astype(np.float64)  # [n, 3, xyz], counter-clockwise
    lo, hi = settings[:2], settings[2:4]
    ring = (corners[:, :, :2] - lo) / (hi - lo)
    center = ring[:, 0] / 3.0 + ring[:, 1] / 3.0 + ring[:, 2] / 3.0
    n = len(faces)
    uv = np.empty((n, 3, 3, 2))
    for e in range(3):
        a, b = ring[:, e], ring[:, (e + 1) % 3]
        uv[:, e, 0], uv[:, e, 1], uv[:, e, 2] = center, a, a + (b - a)
    world = np.empty((n, 3, 3, 3))
    world[..., :2] = lo + uv * (hi - lo)
    world[..., 2] = corners[:, :1, 2][:, :, None]
    source = np.repeat(np.arange(n, dtype=np.int32), 3)
    # Depth is -z: the last triangle is the nearest.
    layer = np.repeat(np.arange(n - 1, -1, -1, dtype=np.int32), 3)
    triangles = [torch.from_numpy(a) for a in (uv.reshape(-1, 3, 2), world.reshape(-1, 3, 3),
                                               source, layer)]
    mesh = _ordered(triangles, _buffers(_room(case), "cpu"), _mix("cpu"))
    return {**mesh, "polygons": n, "depth": n}

"""The subdivision's candidate lists and lane groups where they end: convex
patches of up to 30 vertices (a group holds 8), lists longer than a warp's
buffer, and sources whose lists do not fit the pool and walk the hierarchy."""

import math
from dataclasses import replace

import numpy as np
import pytest
import parity

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

FORMS = ["filtered64", "filtered", "binary64"]


@pytest.fixture(scope="module", autouse=True)
def _device():
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")


def polygon_over_triangle(sides):
    """A triangulated regular polygon in front of one large triangle, whose
    middle patch takes the polygon's shape."""
    angles = 2.0 * math.pi * (np.arange(sides) + 0.25) / sides
    rim = np.stack([0.5 * np.cos(angles), 0.5 * np.sin(angles), np.ones(sides)], 1)
    v = np.concatenate([rim, [[0.01, 0.02, 1.0]], [[-3.0, -2.0, 2.0], [3.0, -2.0, 2.0],
                                                   [0.0, 4.0, 2.0]]])
    f = [(j, (j + 1) % sides, sides) for j in range(sides)] + [(sides + 1, sides + 2, sides + 3)]
    return (v, np.array(f, dtype=np.int32), np.eye(4),
            np.array([-1.0, -1.0, 1.0, 1.0, 0.0, 0.01]))


@pytest.mark.parametrize("form", FORMS)
@pytest.mark.parametrize("sides", [8, 9, 16, 30])
def test_many_sided_patches_against_the_oracle(sides, form):
    from peel_b200 import EventCapacities, EventPeeler, scenes

    arrays = polygon_over_triangle(sides)
    p = EventPeeler(*scenes.to_device(arrays), predicates=form,
                    capacities=replace(EventCapacities.for_mesh(256), layers=64))
    p.run()
    parity.check_against_oracle(p, parity.exact_scene_of(*arrays), range(sides + 1))
    assert max(len(v) for _, _, v in parity.polygons(p)) >= sides


def tiles_over_sheets(side, sheets):
    """side x side small disjoint triangles in front of ``sheets`` large
    triangles: every sheet's list holds every tile's edges."""
    i, j = np.meshgrid(np.arange(side), np.arange(side), indexing="ij")
    step = 1.0 / side
    # Uneven sizes, so that no two tile edges lie on one line.
    size = step * (0.3 + 0.2 * np.random.default_rng(1).uniform(size=(side, side, 3, 2)))
    corner = np.array([[0.0, 0.0], [1.0, 0.0], [0.0, 1.0]])
    xy = -0.5 + step * np.stack([i, j], -1)[:, :, None, :] + size + corner * (0.4 * step)
    tiles = np.concatenate([xy, np.ones((side, side, 3, 1))], -1).reshape(-1, 3)
    big = [[[-3.0, -2.0, 2.0 + k], [3.0, -2.0, 2.0 + k], [0.0, 4.0, 2.0 + k]]
           for k in range(sheets)]
    v = np.concatenate([tiles, np.array(big).reshape(-1, 3)])
    return (v, np.arange(len(v), dtype=np.int32).reshape(-1, 3), np.eye(4),
            np.array([-1.0, -1.0, 1.0, 1.0, 0.0, 0.01]))


# 3 side^2 segments per sheet against a pool of 24 (side^2 + sheets) + 4096:
# one sheet's list above the 192 buffered entries, and 40 sheets' lists above
# the pool.
@pytest.mark.parametrize("form", ["filtered64", "binary64"])
@pytest.mark.parametrize("side,sheets", [(10, 1), (20, 40)])
def test_long_lists_and_sources_without_one(side, sheets, form):
    from peel_b200 import EventCapacities, scenes
    from peel_b200.sizing import fit_event_capacities

    arrays = tiles_over_sheets(side, sheets)
    n = len(arrays[1])
    p, _ = fit_event_capacities(scenes.to_device(arrays), EventCapacities.for_mesh(16 * n),
                                attempts=12, predicates=form)
    info = p.read_status()
    assert info["layers"] == sheets + 1
    corners = arrays[0][arrays[1]][:, :, :2] * 0.5
    u, w = corners[:, 1] - corners[:, 0], corners[:, 2] - corners[:, 0]
    tiles = 0.5 * (u[:, 0] * w[:, 1] - u[:, 1] * w[:, 0])[: side * side]
    areas = parity.gpu_areas(parity.polygons(p), range(n))
    covered = float(tiles.sum())
    for s in range(side * side):
        assert abs(areas[(0, s)] - tiles[s]) <= 1e-9
    for k in range(sheets):  # the window shows a sheet's whole unit square
        s = side * side + k
        whole = areas[(k, s)] + areas[(k + 1, s)]
        assert abs(areas[(k + 1, s)] - covered) <= 1e-9
        assert abs(whole - areas[(0, n - sheets)] - areas[(1, n - sheets)]) <= 1e-9
        assert {key for key in areas if key[1] == s} == {(k, s), (k + 1, s)}


def clipped_area(subject, triangle):
    """Area of a convex polygon inside a counter-clockwise triangle."""
    for j in range(3):
        a, b = triangle[j], triangle[(j + 1) % 3]
        side = (b[0] - a[0]) * (subject[:, 1] - a[1]) - (b[1] - a[1]) * (subject[:, 0] - a[0])
        out = []
        for k in range(len(subject)):
            m = (k + 1) % len(subject)
            if side[k] >= 0.0:
                out.append(subject[k])
            if side[k] * side[m] < 0.0:
                t = side[k] / (side[k] - side[m])
                out.append(subject[k] + t * (subject[m] - subject[k]))
        if len(out) < 3:
            return 0.0
        subject = np.array(out)
    x, y = (subject - subject[0]).T
    return 0.5 * float(np.sum(x * np.roll(y, -1) - np.roll(x, -1) * y))


@pytest.mark.parametrize("form", ["filtered64", "binary64"])
def test_long_and_short_lists_past_the_pool(form):
    """Lists of very different lengths that together exceed the pool: no two
    sources share entries, so every region is the one the faces' order gives.
    Disjoint tiles in front of disjoint cards of a few tiles each, in front of
    sheets that fill the window."""
    from peel_b200 import EventCapacities, EventPeeler, scenes

    side, sheets, cards = 20, 24, 18
    v, f, camera, settings = tiles_over_sheets(side, sheets)
    rng = np.random.default_rng(2)
    i, j = np.meshgrid(np.arange(cards), np.arange(cards), indexing="ij")
    corner = np.array([[0.02, 0.05], [0.93, 0.11], [0.17, 0.95]])
    xy = -0.5 + (np.stack([i, j], -1)[:, :, None, :] + corner
                 + rng.uniform(-0.02, 0.02, size=(cards, cards, 3, 2))) / cards
    xy = xy.reshape(-1, 3, 2)
    front = np.concatenate([xy, np.full((len(xy), 3, 1), 1.5)], -1).reshape(-1, 3)
    v = np.concatenate([v, front])
    f = np.arange(len(v), dtype=np.int32).reshape(-1, 3)
    tiles = v.reshape(-1, 3, 3)[: side * side, :, :2] * 0.5
    short = xy * 0.5
    area = {}

    def doubled(t):
        return ((t[:, 1, 0] - t[:, 0, 0]) * (t[:, 2, 1] - t[:, 0, 1])
                - (t[:, 1, 1] - t[:, 0, 1]) * (t[:, 2, 0] - t[:, 0, 0]))

    tile_areas, card_areas = 0.5 * doubled(tiles), 0.5 * doubled(short)
    for s, a in enumerate(tile_areas):
        area[(0, s)] = a
    covered = 0.0
    for c, (t, a) in enumerate(zip(short, card_areas)):
        near = tiles[np.abs(tiles.mean(1) - t.mean(0)).max(1) < 1.5 / side]
        under = sum(clipped_area(x, t) for x in near)
        area[(0, side * side + sheets + c)] = a - under
        area[(1, side * side + sheets + c)] = under
        covered += under
    single = float(tile_areas.sum() + card_areas.sum()) - 2.0 * covered
    for k in range(sheets):
        s = side * side + k
        area[(k + 2, s)] = covered
        area[(k + 1, s)] = single
        area[(k, s)] = 1.0 - covered - single
    n = len(f)
    capacities = EventCapacities(400 * n, 800 * n, 8000 * n, 4000 * n, 4000 * n, layers=64)
    p = EventPeeler(*scenes.to_device((v, f, camera, settings)), predicates=form,
                    capacities=capacities)
    for _ in range(4):
        p.run()
        assert p.read_status()["layers"] == sheets + 2
        parity.assert_areas({key: a for key, a in parity.gpu_areas(parity.polygons(p),
                                                                   range(n)).items() if a},
                            {key: a for key, a in area.items() if a})


# 3 side^2 + 4 segments: hierarchies of 2^10, 2^12 and 2^14 leaves.
@pytest.mark.parametrize("form", ["filtered64", "filtered", "binary64"])
@pytest.mark.parametrize("side", [17, 30, 60])
def test_a_frontier_of_the_sources_suffices(side, form):
    """One sheet behind many tiles, whose patches search the hierarchy, cut
    into several times as many patches as there are faces, with a frontier that
    just holds the faces."""
    from peel_b200 import EventCapacities, EventPeeler, scenes

    arrays = tiles_over_sheets(side, 1)
    n = len(arrays[1])
    capacities = replace(EventCapacities.for_mesh(32 * n), frontier=n, layers=8)
    p = EventPeeler(*scenes.to_device(arrays), predicates=form, capacities=capacities)
    p.run()
    info = p.read_status()
    assert info["polygons"] > 5 * n and info["peak_residual_patches"] <= n
    areas = parity.gpu_areas(parity.polygons(p), range(n))
    covered = sum(areas[(0, s)] for s in range(n - 1))
    assert abs(areas[(1, n - 1)] - covered) <= 1e-9
    assert abs(areas[(0, n - 1)] + covered - 1.0) <= 1e-9


@pytest.mark.parametrize("form", ["filtered64", "binary64"])
@pytest.mark.parametrize("count", [127, 128, 129])
def test_lists_at_their_longest(count, form):
    """A sheet behind ``count`` tiles, three segments each, where a list holds
    384 of them."""
    from peel_b200 import EventCapacities, EventPeeler, scenes

    v, f, camera, settings = tiles_over_sheets(12, 1)
    v = np.concatenate([v[:3 * count], v[-3:]])
    f = np.arange(len(v), dtype=np.int32).reshape(-1, 3)
    p = EventPeeler(*scenes.to_device((v, f, camera, settings)), predicates=form,
                    capacities=replace(EventCapacities.for_mesh(32 * len(f)), layers=8))
    p.run()
    assert p.read_status()["unique_contours"] >= 3 * count
    areas = parity.gpu_areas(parity.polygons(p), range(len(f)))
    covered = sum(areas[(0, s)] for s in range(count))
    assert abs(areas[(1, count)] - covered) <= 1e-9
    assert abs(areas[(0, count)] + covered - 1.0) <= 1e-9


@pytest.mark.parametrize("form", ["filtered64", "binary64"])
@pytest.mark.parametrize("gap", [0.5, -0.5])
def test_many_candidates(gap, form):
    """A slanted sheet half a unit in front of (or behind) 1,600 tiles of its
    own slant: every tile's edges are candidates of the sheet, none (or all) of
    which cut it."""
    from peel_b200 import EventCapacities, EventPeeler, scenes

    side = 40
    v, f, camera, settings = tiles_over_sheets(side, 1)
    v[:, 2] = 10.0 + 4.0 * v[:, 0]
    v[:-3, 2] += gap
    n = len(f)
    p = EventPeeler(*scenes.to_device((v, f, camera, settings)), predicates=form,
                    capacities=replace(EventCapacities.for_mesh(32 * n), layers=8))
    p.run()
    assert p.read_status()["layers"] == 2
    areas = parity.gpu_areas(parity.polygons(p), range(n))
    tiles, sheet = (1, 0) if gap > 0.0 else (0, 1)
    covered = sum(areas[(tiles, s)] for s in range(n - 1))
    if gap > 0.0:
        assert len(areas) == n and abs(areas[(0, n - 1)] - 1.0) <= 1e-9
    else:
        assert abs(areas[(sheet, n - 1)] - covered) <= 1e-9
        assert abs(areas[(0, n - 1)] + covered - 1.0) <= 1e-9
    corners = v[f][:, :, :2] * 0.5
    u, w = corners[:, 1] - corners[:, 0], corners[:, 2] - corners[:, 0]
    whole = 0.5 * (u[:, 0] * w[:, 1] - u[:, 1] * w[:, 0])[:-1]
    assert abs(covered - whole.sum()) <= 1e-9

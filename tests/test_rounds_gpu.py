"""The rounds' capacity counts generations of right-hand parts, as the
reference's rounds do, however the loop hands the work on; and a workspace
sized by the usage that another one reports is large enough."""

from dataclasses import replace

import numpy as np
import pytest
import parity

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.fixture(scope="module", autouse=True)
def _device():
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")


def strips(count):
    """Thin slanted triangles across the view, one above the other, in front of
    a large one: one long chain of cuts whose other parts are final at once."""
    v = []
    for k in range(count):
        y, h = -0.9 + 1.8 * (k + 0.5) / count, 0.4 * 1.8 / count
        v += [[-0.95, y - h, 1.0], [0.95 - 0.001 * (k % 7), y, 1.0], [-0.95, y + h, 1.0]]
    v += [[-3.0, -2.0, 2.0], [3.0, -2.0, 2.0], [0.0, 4.0, 2.0]]
    v = np.array(v)
    return (v, np.arange(len(v), dtype=np.int32).reshape(-1, 3), np.eye(4),
            np.array([-1.0, -1.0, 1.0, 1.0, 0.0, 0.01]))


def assert_strips(p, arrays, count):
    corners = arrays[0][arrays[1]][:, :, :2] * 0.5
    u, w = corners[:, 1] - corners[:, 0], corners[:, 2] - corners[:, 0]
    area = 0.5 * (u[:, 0] * w[:, 1] - u[:, 1] * w[:, 0])[:count]
    expected = {(0, k): a for k, a in enumerate(area)}
    expected[(1, count)] = float(area.sum())
    expected[(0, count)] = 1.0 - float(area.sum())
    parity.assert_areas(parity.gpu_areas(parity.polygons(p), range(count + 1)), expected)


@pytest.mark.parametrize("form", ["filtered64", "binary64"])
@pytest.mark.parametrize("count", [20, 40])  # a patch edge holds 128 noded points
def test_a_long_chain_takes_no_rounds(count, form):
    from peel_b200 import EventCapacities, EventPeeler, scenes

    arrays = strips(count)
    device = scenes.to_device(arrays)
    capacities = replace(EventCapacities.for_mesh(64 * count), layers=8)
    p = EventPeeler(*device, capacities=capacities, predicates=form)
    p.run()
    info = p.read_status()
    assert_strips(p, arrays, count)
    # A right-hand part meets the strips past its cut: a few generations.
    assert info["rounds"] <= 8 < 3 * count < info["splits"]
    for rounds in (info["rounds"], info["rounds"] - 1):
        q = EventPeeler(*device, capacities=replace(capacities, rounds=rounds), predicates=form)
        q.run()
        if rounds == info["rounds"]:
            assert q.read_status()["rounds"] == rounds
            assert_strips(q, arrays, count)
        else:
            with pytest.raises(RuntimeError, match="subdivision round"):
                q.read_status()


@pytest.mark.parametrize("scene", ["strips", "icospheres", "knot"])
def test_pools_of_the_reported_usage_suffice(scene):
    from peel_b200 import EventCapacities, EventPeeler, scenes

    arrays = {"strips": lambda: strips(50), "knot": lambda: scenes.knot_tube(48, 24, seed=3),
              "icospheres": icospheres}[scene]()
    device = scenes.to_device(arrays)
    wide = EventCapacities.for_mesh(64 * len(arrays[1]))
    p = EventPeeler(*device, capacities=wide)
    p.run()
    info = p.read_status()
    tight = replace(wide, frontier=info["peak_residual_patches"], rounds=info["rounds"],
                    regions=info["polygons"])
    q = EventPeeler(*device, capacities=tight)
    for _ in range(2):
        q.run()
        again = q.read_status()
        assert {k: again[k] for k in ("polygons", "layers", "rounds", "splits")} == \
            {k: info[k] for k in ("polygons", "layers", "rounds", "splits")}


def icospheres():
    from peel_b200 import scenes

    v, f = scenes.icosphere(2)
    rng = np.random.default_rng(1)
    outer = v * (1 + rng.uniform(-0.15, 0.15, size=(len(v), 1)))
    inner = 0.5 * v * (1 + rng.uniform(-0.15, 0.15, size=(len(v), 1)))
    return (np.concatenate([outer, inner]),
            np.concatenate([f, f + len(v)]).astype(np.int32), np.diag([1.0, 1.0, -1.0, 1.0]),
            np.array([-1.3, -1.3, 1.3, 1.3, 0.0, 0.01]))


@pytest.mark.parametrize("form", ["filtered64", "binary64"])
def test_the_frontier_has_room_beside_a_generation(form):
    """The capacity is for a generation of right-hand parts; the patches that an
    iteration holds besides have room of their own."""
    from peel_b200 import EventCapacities, EventPeeler, scenes

    arrays = scenes.knot_tube(117, 60, seed=5)
    device = scenes.to_device(arrays)
    wide = EventCapacities.for_mesh(8 * len(arrays[1]))
    p = EventPeeler(*device, capacities=wide, predicates=form)
    p.run()
    info = p.read_status()
    frontier = max(len(arrays[1]), int(info["peak_residual_patches"] / 1.2))
    assert frontier < info["peak_residual_patches"]
    q = EventPeeler(*device, capacities=replace(wide, frontier=frontier), predicates=form)
    q.run()
    again = q.read_status()
    assert {k: again[k] for k in ("polygons", "layers", "rounds", "splits")} == \
        {k: info[k] for k in ("polygons", "layers", "rounds", "splits")}

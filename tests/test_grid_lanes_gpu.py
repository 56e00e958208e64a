"""The grids of the rays and the connection test, filled by a warp, eight lanes
or a thread per item: scenes of few large triangles, whose sources and segments
reach over up to all cells, against the exact oracle."""

import numpy as np
import pytest
import parity

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("form", ["filtered64", "binary64"])
@pytest.mark.parametrize("count", [1, 2, 9, 16])
def test_large_triangles_against_the_oracle(count, form):
    from peel_b200 import EventCapacities, EventPeeler, scenes

    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    rng = np.random.default_rng(count)
    v = rng.uniform(-1.2, 1.2, size=(count, 3, 3))
    v[:, :, 2] = np.arange(1, count + 1)[:, None]
    arrays = (v.reshape(-1, 3), np.arange(3 * count, dtype=np.int32).reshape(-1, 3), np.eye(4),
              np.array([-1.0, -1.0, 1.0, 1.0, 0.0, 0.01]))
    p = EventPeeler(*scenes.to_device(arrays), predicates=form,
                    capacities=EventCapacities.for_mesh(2000))
    for _ in range(2):  # the grids' counts are back at zero after a replay
        p.run()
        parity.check_against_oracle(p, parity.exact_scene_of(*arrays), range(count))


@pytest.mark.parametrize("side", [98, 260])  # eight lanes a source; a thread
def test_cards_of_many_cells(side):
    """Disjoint tiles in front of as many disjoint cards, half a step aside:
    each card lies under parts of up to four tiles, and the grid's cells are
    smaller than both."""
    from peel_b200 import EventCapacities, EventPeeler, scenes

    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    i, j = np.meshgrid(np.arange(side), np.arange(side), indexing="ij")
    corner = np.array([[0.03, 0.05], [0.93, 0.11], [0.17, 0.95]])
    xy = (-0.9 + 1.7 / side * (np.stack([i, j], -1)[:, :, None, :] + corner)).reshape(-1, 3, 2)
    layers = [np.concatenate([xy + k * 0.85 / side, np.full((len(xy), 3, 1), 1.0 + k)], -1)
              for k in range(2)]
    v = np.concatenate(layers).reshape(-1, 3)
    arrays = (v, np.arange(len(v), dtype=np.int32).reshape(-1, 3), np.eye(4),
              np.array([-1.0, -1.0, 1.0, 1.0, 0.0, 0.01]))
    n = len(arrays[1])
    p = EventPeeler(*scenes.to_device(arrays),
                    capacities=EventCapacities.for_mesh(2 * n))
    p.run()
    assert p.read_status()["layers"] == 2
    u, w = xy[:, 1] - xy[:, 0], xy[:, 2] - xy[:, 0]
    area = 0.125 * (u[:, 0] * w[:, 1] - u[:, 1] * w[:, 0])
    got = parity.gpu_areas(parity.polygons(p), range(n))
    hidden = 0.0
    for c in range(n // 2):
        assert abs(got[(0, c)] - area[c]) <= 1e-9
        front, back = got.get((0, n // 2 + c), 0.0), got.get((1, n // 2 + c), 0.0)
        assert abs(front + back - area[c]) <= 1e-9
        hidden += back
    assert 0.1 * area.sum() < hidden < 0.9 * area.sum()

"""The point and edge tables where a lane begins to look several entries up
together: a flat sheet of m x m cells, two triangles each, has 6 m^2 boundary
vertices and patch edges, of which the 3 m^2 - 2 m inner edges are matched in
pairs.  One lane per entry up to 148 x 16 x 128 = 303,104 of them (m = 224),
four to 8 times that (m = 635), eight above."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def sheet(m):
    c = np.linspace(-0.9, 0.9, m + 1)
    vertices = np.stack([*np.meshgrid(c, c), np.ones((m + 1, m + 1))], -1).reshape(-1, 3)
    i, j = np.meshgrid(np.arange(m), np.arange(m))
    a = (j * (m + 1) + i).ravel()
    faces = np.concatenate([np.stack([a, a + 1, a + m + 2], 1),
                            np.stack([a, a + m + 2, a + m + 1], 1)])
    return (vertices, faces.astype(np.int32), np.eye(4),
            np.array([-1.0, -1.0, 1.0, 1.0, 0.0, 0.01]))


@pytest.mark.parametrize("m", [1, 5, 224, 225, 635, 636])
def test_sheet(m):
    from peel_b200 import EventCapacities, EventPeeler, scenes

    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    n = 2 * m * m
    room = max(4 * n, 64)
    p = EventPeeler(*scenes.to_device(sheet(m)), capacities=EventCapacities(
        frontier=room, regions=room, hits=room, vertices=room, triangles=room,
        rounds=64, layers=8))
    for _ in range(2):
        p.run()
        info = p.read_status()
        assert info["polygons"] == n and info["layers"] == 1
        assert info["boundary_vertices"] == info["triangles"] == 3 * n
        assert info["matched_patch_edges"] == 3 * m * m - 2 * m
        uv = p.triangles_uv[: 3 * n].cpu().numpy()
        u, v = uv[:, 1] - uv[:, 0], uv[:, 2] - uv[:, 0]
        area = 0.5 * (u[:, 0] * v[:, 1] - u[:, 1] * v[:, 0])
        assert area.min() > 0.0 and abs(area.sum() - 0.81) < 1e-10

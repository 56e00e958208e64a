"""Noding by eight lanes per polygon where its buffers end, against the exact
oracle: a triangle with m - 1 T-junctions on every edge.  An edge's lane holds
8 split points, so m = 9 fills it and m = 10 sends the polygon to the warp
kernel; 3 m fan triangles and the neighbours' overflow the 32 triangles a warp
stages, so they are written directly."""

import numpy as np
import pytest
import parity

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def noded_triangle(m):
    """A large triangle (the last face) with m small ones on each edge."""
    corners = np.array([[-0.75, -0.75], [0.75, -0.75], [-0.75, 0.75]])
    apexes = np.array([[0.01, -0.95], [0.9, 0.8], [-0.95, 0.02]])
    points, faces = [], []
    for e in range(3):
        a, b = corners[e], corners[(e + 1) % 3]
        first = len(points)
        for k in range(m + 1):
            x = a + (b - a) * (k / m)
            if e == 1:
                x = np.array([x[0], -x[0]])  # on x + y = 0 exactly
            points.append([*x, 1.0])
        points.append([*apexes[e], 1.0])
        faces += [[first + k + 1, first + k, first + m + 1] for k in range(m)]
    k = len(points)
    points += [[*c, 1.0] for c in corners]
    faces.append([k, k + 1, k + 2])
    return (np.array(points), np.array(faces, dtype=np.int32), np.eye(4),
            np.array([-1.0, -1.0, 1.0, 1.0, 0.0, 0.01]))


@pytest.mark.parametrize("m", [2, 8, 9, 10])
def test_split_points_per_lane(m):
    from peel_b200 import EventPeeler, scenes

    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    arrays = noded_triangle(m)
    p = EventPeeler(*scenes.to_device(arrays))
    p.set_tuning(heavy_noding_work=1 << 30)
    p.run()
    info = p.read_status()
    assert (info["heavy_noded_polygons"] > 0) == (m > 9)
    parity.check_against_oracle(p, parity.exact_scene_of(*arrays), range(len(arrays[1])))
    sources = p.triangle_sources[: info["triangles"]].cpu().numpy()
    assert (sources == len(arrays[1]) - 1).sum() == 3 * m


@pytest.mark.parametrize("m", [2, 10, 11, 32])
def test_warp_kernel_fan(m):
    """Every polygon noded by a warp, whose lanes take 32 points and 32 pieces
    of edge at a time: 3 m pieces, of 3 (m - 1) points."""
    from peel_b200 import EventPeeler, scenes

    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    arrays = noded_triangle(m)
    p = EventPeeler(*scenes.to_device(arrays))
    p.set_tuning(heavy_noding_work=1)
    p.run()
    info = p.read_status()
    assert info["heavy_noded_polygons"] > 0
    parity.check_against_oracle(p, parity.exact_scene_of(*arrays), range(len(arrays[1])))
    sources = p.triangle_sources[: info["triangles"]].cpu().numpy()
    assert (sources == len(arrays[1]) - 1).sum() == 3 * m

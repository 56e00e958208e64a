"""One-launch scans and radix passes at the edges of their 2,048-element tiles
and over many tiles, replayed: a stack's n sources, n polygons and 3 n patch
edges go through every scan and sort of an extraction, and its ranks are the
faces' order."""

import numpy as np
import pytest
import parity

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("n", [1, 682, 683, 2047, 2048, 2049, 16385, 70001])
def test_stack_over_tile_edges(n):
    from peel_b200 import EventPeeler

    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    p = EventPeeler(*parity.stack_arrays(n))
    for _ in range(3):
        p.run()
        info = p.read_status()
        assert info["polygons"] == info["layers"] == n
        assert info["triangles"] == info["boundary_vertices"] == 3 * n
        layers = p.output_layers[:n].cpu().numpy()
        sources = p.output_sources[:n].cpu().numpy()
        np.testing.assert_array_equal(layers, sources)
        np.testing.assert_array_equal(np.sort(layers), np.arange(n))


@pytest.mark.parametrize("n", [1365, 1366, 4095, 4096, 4097])
def test_stack_over_scan_tile_edges(n):
    """A scan's tiles hold 4,096 elements (a radix pass's 2,048)."""
    test_stack_over_tile_edges(n)

"""Rays over the source grid, eight lanes each, where their buffers end: 8
candidates tested at a time, 57 to 64 hits held before they are written, and
sources clipped by the window, which have no binary32 edge functions."""

import numpy as np
import pytest
import parity

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("form", ["filtered64", "filtered", "binary64"])
@pytest.mark.parametrize("scale", [1.0, 1.9])  # 1.9: every footprint crosses the window's border
@pytest.mark.parametrize("n", [7, 8, 9, 56, 57, 64, 65, 129])
def test_stack_ranks(n, scale, form):
    from peel_b200 import EventPeeler

    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    vertices, faces, camera, settings = parity.stack_arrays(n)
    vertices[:, :2] *= scale
    p = EventPeeler(vertices, faces, camera, settings, predicates=form)
    p.run()
    info = p.read_status()
    assert info["polygons"] == info["layers"] == info["ray_hits"] == n
    assert info["ray_groups"] == 1
    np.testing.assert_array_equal(p.output_layers[:n].cpu().numpy(),
                                  p.output_sources[:n].cpu().numpy())

"""A boundary-vertex pool that overflows in one replay leaves nothing behind:
the workspace's next replay, of inputs that fit, equals a fresh workspace's."""

from dataclasses import replace

import numpy as np
import pytest
import parity

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def triangles(p):
    count = p.read_status()["triangles"]
    rows = np.concatenate([
        p.triangle_layers[:count, None].cpu().numpy(), p.triangle_sources[:count, None].cpu().numpy(),
        p.triangles_uv[:count].cpu().numpy().reshape(count, 6),
        p.triangles_world[:count].cpu().numpy().reshape(count, 9)], axis=1)
    return rows[np.lexsort(rows.T)]


@pytest.mark.parametrize("short", [1, 7, 6000])
def test_overflow_then_a_scene_that_fits(short):
    """A stack of n triangles has 3 n boundary vertices, ``short`` more than
    the pool; with its lower half moved out of the window it has half."""
    from peel_b200 import EventCapacities, EventPeeler

    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    n = 5000
    arrays = parity.stack_arrays(n)
    capacities = replace(EventCapacities.for_mesh(n), vertices=3 * n - short)
    whole = arrays[0].clone()
    half = whole.clone()
    half[3 * (n // 2):, 0] += 10.0
    torch.cuda.synchronize()
    p = EventPeeler(*arrays, capacities=capacities, propagate_ranks=False)
    p.run()
    for _ in range(2):
        with torch.cuda.stream(p.stream):
            arrays[0].copy_(whole)
        p.run()
        with pytest.raises(RuntimeError, match="boundary vertex"):
            p.read_status()
        with torch.cuda.stream(p.stream):
            arrays[0].copy_(half)
        p.run()
        got = triangles(p)
        assert len(got) == 3 * (n // 2)
        fresh = EventPeeler(*[a.clone() for a in arrays], propagate_ranks=False)
        torch.cuda.synchronize()
        fresh.run()
        np.testing.assert_array_equal(got, triangles(fresh))

"""Iterative clipping, a piece per warp, where its tiles end: convex pieces
with up to three edges per triangle above them (more uncovered parts than one
cut holds in shared memory, and residual candidates of many edges), against
the exact oracle."""

import math

import numpy as np
import pytest
import parity

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def rotated_stack(count):
    """``count`` concentric triangles, each turned a little against the one in
    front of it, over one large triangle: the part of the k-th that the ones
    in front hide has up to 3 k edges."""
    vertices = []
    for k in range(count):
        turn = 2.0 * math.pi / 3.0 * k / count
        vertices += [[0.5 * math.cos(turn + a), 0.5 * math.sin(turn + a), k + 1.0]
                     for a in (0.0, 2.0 * math.pi / 3.0, 4.0 * math.pi / 3.0)]
    vertices += [[-3.0, -2.0, count + 1.0], [3.0, -2.0, count + 1.0], [0.0, 4.0, count + 1.0]]
    v = np.array(vertices)
    f = np.arange(len(v), dtype=np.int32).reshape(-1, 3)
    return v, f, np.eye(4), np.array([-1.0, -1.0, 1.0, 1.0, 0.0, 0.01])


@pytest.mark.parametrize("budget", [1, 32])
@pytest.mark.parametrize("count", [1, 4, 5, 6])
def test_many_edged_pieces_against_the_oracle(count, budget):
    from peel_b200 import Capacities, DevicePeeler, scenes

    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    arrays = rotated_stack(count)
    p = DevicePeeler(*scenes.to_device(arrays), capacities=Capacities(1024, 1024, 8192, 8192))
    p.set_tuning(clip_budget=budget)
    p.run()
    parity.check_against_oracle(p, parity.exact_scene_of(*arrays), range(count + 1))


@pytest.mark.parametrize("count", [4, 6])
def test_tight_pools(count):
    """Pools that just hold the residual and the output: pieces queued past the
    pool's end spill to the next launch of the layer."""
    from dataclasses import replace

    from peel_b200 import Capacities, DevicePeeler, scenes

    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    arrays = rotated_stack(count)
    device = scenes.to_device(arrays)
    wide = Capacities(1024, 1024, 8192, 8192)
    p = DevicePeeler(*device, capacities=wide)
    p.run()
    info = p.read_status()
    tight = replace(wide, residual=info["peak_residual_patches"] + 8,
                    polygons=info["polygons"] + 8)
    p = DevicePeeler(*device, capacities=tight)
    for _ in range(2):
        p.run()
        parity.check_against_oracle(p, parity.exact_scene_of(*arrays), range(count + 1))

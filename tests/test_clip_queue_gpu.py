"""The clipping queue's end: pieces past it wait for another launch of their
layer, from the other of the two pools; when both are full the extraction ends
with the worker error.  And the queue holds as many pieces as there are, however
many turns their walks take."""

from dataclasses import replace

import pytest
import parity
from test_clip_gpu import rotated_stack

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.fixture(scope="module", autouse=True)
def _device():
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")


def peeler(arrays, slots, **options):
    from peel_b200 import Capacities, DevicePeeler, _lib, scenes

    p = DevicePeeler(*scenes.to_device(arrays), capacities=Capacities(1024, 1024, 8192, 8192),
                     **options)
    _lib.check(_lib.load().edp_set_clip_queue(p._ws.handle, slots), "clip queue")
    return p


@pytest.mark.parametrize("form", ["filtered64", "binary64"])
@pytest.mark.parametrize("count", [5, 6])
def test_pieces_past_the_queue(count, form):
    arrays = rotated_stack(count)
    expected = parity.exact_scene_of(*arrays)
    p = peeler(arrays, 0, predicates=form)
    p.run()
    info = p.read_status()
    # One launch per layer pass that has targets.
    assert 0 < int(p.status[11]) <= info["peeling_passes"]
    launches = []
    for slots in range(info["peak_residual_patches"], 1024):
        q = peeler(arrays, slots, predicates=form)
        q.run()
        try:
            again = q.read_status()
        except RuntimeError as error:  # twice the slots are too few
            assert "per-worker pieces" in str(error)
            launches.append(0)
            continue
        launches.append(int(q.status[11]))
        assert again["peeling_passes"] == info["peeling_passes"]
        parity.check_against_oracle(q, expected, range(count + 1))
        if launches[-1] == int(p.status[11]):  # all of them fit
            break
    assert launches[-1] == int(p.status[11])
    assert max(launches) > int(p.status[11]), launches  # some pieces spilled


def test_both_pools_full():
    """The error is clean: the workspace's next replay, of inputs that fit, is
    right."""
    arrays = rotated_stack(6)
    p = peeler(arrays, 8)
    whole = p.vertices.clone()
    apart = whole.clone()
    apart[:, 0] += 4.0 * torch.arange(len(whole), device="cuda").div(3, rounding_mode="floor")
    torch.cuda.synchronize()
    for _ in range(2):
        with torch.cuda.stream(p.stream):
            p.vertices.copy_(whole)
        p.run()
        with pytest.raises(RuntimeError, match="per-worker pieces"):
            p.read_status()
        with torch.cuda.stream(p.stream):
            p.vertices.copy_(apart)  # one triangle is left in the window
        p.run()
        info = p.read_status()
        assert info["polygons"] == info["layers"] == 1


def test_long_walks_take_no_slots():
    """One large triangle under 1,024 tiles: its walk takes many turns of eight
    steps, and the pools just hold the pieces."""
    from peel_b200 import Capacities, DevicePeeler, scenes
    from test_lists_gpu import tiles_over_sheets

    arrays = tiles_over_sheets(32, 1)
    device = scenes.to_device(arrays)
    wide = Capacities(8192, 16384, 200000, 200000, pieces_per_worker=16384, workers=64)
    p = DevicePeeler(*device, capacities=wide)
    p.run()
    info = p.read_status()
    tight = replace(wide, residual=info["peak_residual_patches"], polygons=info["polygons"])
    q = DevicePeeler(*device, capacities=tight)
    q.set_tuning(clip_budget=1)
    q.run()
    again = q.read_status()
    assert again["polygons"] == info["polygons"]
    areas = [parity.gpu_areas(parity.polygons(x), range(len(arrays[1]))) for x in (p, q)]
    parity.assert_areas(*areas)
    assert {layer for layer, _ in areas[1]} == {0, 1}

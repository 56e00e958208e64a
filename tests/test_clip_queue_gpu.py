"""The clipping queue holds as many pieces as there are, however many turns their
walks take."""

from dataclasses import replace

import pytest
import parity

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.fixture(scope="module", autouse=True)
def _device():
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")


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

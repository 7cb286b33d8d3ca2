"""The one-block pixel order at the edges of its range (films of up to 8192
pixels) and the two-launch form beyond."""
import pytest
import torch

import recursive_control_variates_gb300 as rcv

from test_gpu_volume import make_scene

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("res", [1, 5, 64, 90, 91, 128])
def test_orders_give_the_same_image(cuda, res):
    """Whatever the order (and after a call that left costs behind), every
    pixel is handed out once: the images are those of the row-major order."""
    scene, _, _ = make_scene(cuda, res=res)
    images = {}
    for order in ("row_major", "cost", "longest_first"):
        integ = rcv.load_dict({"type": "twostateprbvolpath", "max_depth": 6, "rr_depth": 6, "order": order})
        for _ in range(2):
            images[order] = integ.render_twostates(scene, 0, seed=3, spp=2)
    for order in ("cost", "longest_first"):
        for a, b in zip(images["row_major"], images[order]):
            assert torch.equal(a, b)

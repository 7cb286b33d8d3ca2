"""The pixel order of a first call, estimated from the medium (films below and
above the one-launch limit): every pixel is handed out once, so the images are
those of the row-major order bit for bit."""
import pytest
import torch

import recursive_control_variates_gb300 as rcv

from test_gpu_volume import make_scene

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("res", [1, 63, 90, 91, 160])
@pytest.mark.parametrize("scale", [1.0, 1e-3])
def test_first_call_gives_the_row_major_image(cuda, res, scale):
    scene, med, _ = make_scene(cuda, res=res)
    for state in (med.old, med.new):
        state.density.mul_(scale)
    med._dirty = True
    images = []
    for order in ("row_major", "cost"):
        integ = rcv.load_dict({"type": "twostateprbvolpath", "max_depth": 6, "rr_depth": 6, "order": order})
        images.append(integ.render_twostates(scene, 0, seed=3, spp=2))
    for a, b in zip(*images):
        assert torch.equal(a, b)

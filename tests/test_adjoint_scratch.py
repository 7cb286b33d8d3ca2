"""Scratch of the adjoints: no more than the call can use."""
import torch

import recursive_control_variates_gb300 as rcv
from recursive_control_variates_gb300 import _lib, scenes

W, SPP = 512, 2
PATHS = W * W * SPP


def volume_sensor():
    return rcv.load_dict(scenes.scene_dict(scenes.blob_density(4, 0), 0.8, res=W), device="cpu").sensors()[0]


def test_surface_adjoint_takes_what_it_uses(rcvlib):
    """Radiance (16 B), 16 tape slots (16 B) and the lost list (4 B) per path."""
    integ = rcv.load_dict({"type": "twostateprb"})
    integ.scratch("cpu", volume_sensor(), SPP, _lib.MODE_ADJOINT)
    assert integ._scratch[torch.device("cpu")].numel() <= 276 * PATHS + (1 << 20)

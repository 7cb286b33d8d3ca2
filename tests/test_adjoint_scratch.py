"""Scratch of the adjoints: no more than the call can use, and a smaller room
for the event tape where the large one does not fit the GPU."""
import numpy as np
import pytest
import torch

import recursive_control_variates_gb300 as rcv
from recursive_control_variates_gb300 import _lib, scenes
from recursive_control_variates_gb300.plugins import twostatevolpath

from test_gpu_volume import make_scene

W, SPP = 32, 512  # few pixels: what is zeroed stays below the size that torch splits over threads
PATHS = W * W * SPP


def small_room(pixels, paths):
    """16 tape slots and 2 checkpoints per path; the checkpoints' margin, the order and cost of the pixels, alignment."""
    return 480 * paths + 64 * 65536 + 8 * pixels + 8192


SMALL = small_room(W * W, PATHS)


def volume_sensor():
    return rcv.load_dict(scenes.scene_dict(scenes.blob_density(4, 0), 0.8, res=W), device="cpu").sensors()[0]


def scratch_bytes(props, spp=SPP):
    integ = rcv.load_dict({"type": "twostateprbvolpath", **props})
    integ.adjoint_scratch("cpu", volume_sensor(), spp)
    return integ._adj_scratch[torch.device("cpu")].numel()


def test_surface_adjoint_takes_what_it_uses(rcvlib):
    """Radiance (16 B), 16 tape slots (16 B) and the lost list (4 B) per path."""
    integ = rcv.load_dict({"type": "twostateprb"})
    integ.scratch("cpu", volume_sensor(), SPP, _lib.MODE_ADJOINT)
    assert integ._scratch[torch.device("cpu")].numel() <= 276 * PATHS + (1 << 20)


@pytest.mark.parametrize("props", [{"adjoint": "replay"}, {"tape_events_per_path": 16}, {"tape_events_per_path": 1}])
def test_no_room_for_a_tape_that_is_not_used(rcvlib, props):
    assert scratch_bytes(props) <= SMALL


def test_the_large_room_is_kept_where_it_fits(rcvlib):
    assert scratch_bytes({}) >= (64 * 20 + 8 * 64) * PATHS


def refuse_above(monkeypatch, limit):
    real, refused = twostatevolpath._new_scratch, []

    def limited(nbytes, film, device):
        if nbytes > limit:
            refused.append(nbytes)
            raise torch.cuda.OutOfMemoryError("no room")
        return real(nbytes, film, device)

    monkeypatch.setattr(twostatevolpath, "_new_scratch", limited)
    return refused


def test_smaller_room_on_a_full_gpu(rcvlib, monkeypatch):
    refused = refuse_above(monkeypatch, SMALL)
    sensor = volume_sensor()
    integ = rcv.load_dict({"type": "twostateprbvolpath"})
    integ.adjoint_scratch("cpu", sensor, SPP)
    assert integ._adj_scratch[torch.device("cpu")].numel() <= SMALL
    tries = len(refused)
    for _ in range(3):  # a step of the same size does not try again
        integ.adjoint_scratch("cpu", sensor, SPP)
    assert tries == 1 and len(refused) == 1
    with pytest.raises(torch.cuda.OutOfMemoryError):
        integ.adjoint_scratch("cpu", sensor, 4 * SPP)
    with pytest.raises(torch.cuda.OutOfMemoryError):
        rcv.load_dict({"type": "twostateprbvolpath", "adjoint": "replay"}).adjoint_scratch("cpu", sensor, 4 * SPP)


@pytest.mark.gpu
@pytest.mark.parametrize("integrator", ["alone", "cv"])
def test_gradient_in_the_smaller_room(cuda, monkeypatch, integrator):
    """Cameras close to the box, so that many paths do not fit the small room:
    a step with each room, radiance pass ahead (on the side stream, in the
    paired launch), gives the gradient of the replay; 2e-5, thousands of terms
    per voxel in another order."""
    width, spp = 96, 8
    d = scenes.scene_dict(scenes.blob_density(20, 3), scenes.albedo_grid(20, 3), res=width,
                          views=scenes.orbit_views(None, 2, distance=0.9))
    two = {"type": "twostateprbvolpath", "max_depth": 24, "rr_depth": 24}
    g = torch.from_numpy(np.random.default_rng(9).normal(0, 1, (width, 2 * width, 3)).astype(np.float32)).to(cuda)
    grads = {}
    for room in ("small", "full", "replay"):
        with monkeypatch.context() as mp:
            if room == "small":
                refuse_above(mp, small_room(2 * width * width, 2 * width * width * spp))
            scene = rcv.load_dict(d, device=cuda)
            params = rcv.traverse(scene)
            inner = rcv.load_dict({**two, **({"adjoint": "replay"} if room == "replay" else {})})
            integ = rcv.load_dict({"type": "cv", "integrator": inner}) if integrator == "cv" else inner
            opt = rcv.ad.Adam(lr=1e-3)
            for key in (scenes.DENSITY_KEY, scenes.ALBEDO_KEY):
                opt[key] = params[key].detach().clone()
            params.update(opt)
            for step in range(2):  # the second step finds the room that the first one took
                for key in (scenes.DENSITY_KEY, scenes.ALBEDO_KEY):
                    opt[key].grad = None
                rcv.render(scene, params, integrator=integ, seed=3, spp=spp).backward(g)
                assert inner.last_adjoint_call == "rcv_render_backward_replay"
                if integrator == "cv":
                    assert inner.last_primal_call == "rcv_render_twostates_volume_and_adjoint_radiance"
            grads[room] = [opt[k].grad.double() for k in (scenes.DENSITY_KEY, scenes.ALBEDO_KEY)]
    for room in ("small", "full"):
        for a, b in zip(grads[room], grads["replay"]):
            assert float((a - b).norm()) <= 2e-5 * float(b.norm())


@pytest.mark.gpu
def test_rooms_of_one_integrator(cuda):
    """Forward mode (no tape) between two backward calls of one integrator, in
    one scratch: each gives what it gives alone."""
    scene, _, _ = make_scene(cuda, res=24, albedo_grid=True)
    params = rcv.traverse(scene)
    g = torch.from_numpy(np.random.default_rng(2).normal(0, 1, (24, 24, 3)).astype(np.float32)).to(cuda)
    props = {"type": "twostateprbvolpath", "max_depth": 8, "rr_depth": 8}
    tangents = {scenes.DENSITY_KEY: torch.ones_like(params[scenes.DENSITY_KEY])}
    forward = rcv.load_dict(props).render_forward(scene, params, 0, seed=7, spp=4, tangents=tangents)
    want = rcv.load_dict(props).render_backward(scene, params, g, 0, seed=5, spp=4)
    for order in ("forward", "backward"):
        integ = rcv.load_dict(props)
        if order == "backward":
            integ.render_backward(scene, params, g, 0, seed=5, spp=4)
        f = integ.render_forward(scene, params, 0, seed=7, spp=4, tangents=tangents)
        b = integ.render_backward(scene, params, g, 0, seed=5, spp=4)
        # a pixel's tasks add up in any order: a few float additions
        assert float((f - forward).norm()) <= 1e-5 * float(forward.norm())
        for key in want:
            assert float((b[key] - want[key]).double().norm()) <= 1e-6 * float(want[key].double().norm())

"""The recorded volpathsimple adjoint (rcv_render_backward_volpathsimple_ws)
against the same adjoint with one thread per path: films in several passes,
paths whose shadow steps do not fit the tape, one-pixel films, and the
one-correction quotient of its free-flight step.

Both forms trace the same paths; the gradients differ by the order of float
additions and the rounding of the remaining radiance (a difference of sums
instead of a running difference), held to the 2e-5 relative L2 of the oracle
comparisons."""
import ctypes as C

import numpy as np
import pytest
import torch

import recursive_control_variates_gb300 as rcv
from recursive_control_variates_gb300 import _lib
from recursive_control_variates_gb300.utils import stream_handle

from test_gpu_volume import make_scene


def adjoint(scene, integ, gimg, spp, workspace_bytes, slots=0):
    med = scene.named_shapes()["object"].interior_medium()
    dev, sensor = med.device, scene.sensors()[0]
    st = stream_handle(dev)
    m, s, o, f = med.prepare(st), sensor.c_struct(), integ.options(scene), integ.flags()
    o.tape_events_per_path = slots
    dx, dy, dz = med.dims
    gd = torch.zeros((dz, dy, dx, 1), device=dev)
    ga = med.albedo_grad_buffer()
    ws = torch.full((workspace_bytes + 256,), 0xA5, dtype=torch.uint8, device=dev)
    _lib.check(_lib.load().rcv_render_backward_volpathsimple_ws(
        C.byref(m), C.byref(s), C.byref(o), C.byref(f), 31, spp, gimg.data_ptr(), gd.data_ptr(),
        ga.data_ptr() if ga is not None else None, ((ws.data_ptr() + 255) & ~255) if workspace_bytes else None,
        workspace_bytes, st), "vps adjoint")
    return [g.cpu().numpy().astype(np.float64) for g in (gd, ga) if g is not None]


def close(a, b):
    for x, y in zip(a, b):  # a one-path film may miss the medium: zero in both
        assert np.linalg.norm(x - y) <= 2e-5 * np.linalg.norm(y)


@pytest.mark.gpu
@pytest.mark.parametrize("flags", [{}, {"use_drt": False}, {"use_nee": False}, {"use_drt_mis": False}])
@pytest.mark.parametrize("res,spp,fit,slots,factor", [
    (128, 18, (128, 128, 4), 0, 0),  # 294 912 paths in passes of 65 536: the last one is half full
    (64, 5, (64, 64, 5), 1, 4),      # one shadow step per path fits: most paths are lost
    (1, 1, (1, 1, 1), 0, 0),
    (1, 3, (1, 1, 3), 0, 4),
])
def test_recorded_matches_one_thread_per_path(cuda, flags, res, spp, fit, slots, factor):
    scene, med, _ = make_scene(cuda, res=res, albedo_grid=True)
    med.set_majorant_resolution_factor(factor)
    integ = rcv.load_dict({"type": "volpathsimple", "max_depth": 12, "rr_depth": 4, **flags})
    gimg = torch.from_numpy(np.random.default_rng(3).normal(0, 1, (res, res, 3)).astype(np.float32)).to(cuda)
    need = int(_lib.load().rcv_volpathsimple_adjoint_workspace_bytes(*fit))
    close(adjoint(scene, integ, gimg, spp, need, slots), adjoint(scene, integ, gimg, spp, 0))


@pytest.mark.gpu
def test_workspace_too_small_for_a_pass(cuda):
    scene, _, _ = make_scene(cuda, res=32)
    integ = rcv.load_dict({"type": "volpathsimple", "max_depth": 6})
    gimg = torch.ones((32, 32, 3), device=cuda)
    close(adjoint(scene, integ, gimg, 2, 4096), adjoint(scene, integ, gimg, 2, 0))


def test_quotient_with_one_correction_rounds_correctly():
    """div_by (rcv_vps_trace.cuh): float32 steps restated in numpy, the fused
    ones by exact float64 products (24 + 24 bits) with one rounding to float64
    and one to float32, for st / majorant and sigma_n / majorant ratios."""
    rng = np.random.default_rng(0)
    b = np.exp(rng.uniform(np.log(1e-3), np.log(1e4), 400_000)).astype(np.float32)
    a = (b * rng.random(b.size, dtype=np.float32)).astype(np.float32)
    inv = (np.float32(1.0) / b).astype(np.float32)
    q = (a * inv).astype(np.float32)
    r = (a.astype(np.float64) - q.astype(np.float64) * b.astype(np.float64)).astype(np.float32)
    got = (q.astype(np.float64) + r.astype(np.float64) * inv.astype(np.float64)).astype(np.float32)
    want = (a / b).astype(np.float32)
    # the float64 sum can round before the float32 rounding: ties within 2^-53 of a midpoint only
    assert np.mean(got != want) == 0.0

"""The adjoint's radiance pass beside a single-state render: an integrator that
can pair the pass with a two-state render must still let it start right after
the packing where the step renders one state (``rcv.render`` with the two-state
integrator itself, ``meta`` with ``baseline`` or ``cv_pss``)."""
import numpy as np
import pytest
import torch

import recursive_control_variates_gb300 as rcv
from recursive_control_variates_gb300 import _lib, scenes

from test_gpu_volume import make_scene

pytestmark = pytest.mark.gpu

TWO = {"type": "twostateprbvolpath", "max_depth": 6, "rr_depth": 6}
INTEGRATORS = {
    "alone": TWO,
    "meta_baseline": {"type": "meta", "method": "baseline", "integrator": TWO},
    "meta_cv_pss": {"type": "meta", "method": "cv_pss", "integrator": TWO},
    "adjoint_of_another": {"type": "meta", "method": "cv_ps", "integrator": TWO, "adjoint_integrator": dict(TWO)},
}


@pytest.mark.parametrize("kind", list(INTEGRATORS))
def test_radiance_pass_waits_for_the_packing_only(cuda, monkeypatch, kind):
    """What the side stream waits for before the pass was recorded before the
    first primal launch, and the gradient is that of the backward call alone."""
    scene, _, _ = make_scene(cuda, res=24)
    params = rcv.traverse(scene)
    log = []

    class LoggedEvent(torch.cuda.Event):
        def record(self, stream=None):
            log.append(("record", id(self)))
            return super().record(stream) if stream is not None else super().record()

    lib = _lib.load()
    for name in ("rcv_render_volume", "rcv_render_twostates_volume", "rcv_render_adjoint_radiance"):
        real = getattr(lib, name)
        monkeypatch.setattr(lib, name, lambda *a, real=real, name=name: (log.append((name, 0)), real(*a))[1])
    wait = torch.cuda.Stream.wait_event
    monkeypatch.setattr(torch.cuda.Stream, "wait_event",
                        lambda self, e: (log.append(("wait", id(e))), wait(self, e))[1])
    monkeypatch.setattr(torch.cuda, "Event", LoggedEvent)

    integ = rcv.load_dict(INTEGRATORS[kind])
    key = scenes.DENSITY_KEY
    opt = rcv.ad.Adam(lr=1e-3)
    opt[key] = params[key].detach().clone()
    params.update(opt)
    img = rcv.render(scene, params, integrator=integ, seed=3, spp=4)
    steps = [e[0] for e in log]
    at = steps.index("rcv_render_adjoint_radiance")
    waited = [e[1] for e in log[:at] if e[0] == "wait"][-1]
    primal = min(steps.index(n) for n in ("rcv_render_volume", "rcv_render_twostates_volume") if n in steps)
    assert ("record", waited) in log[:primal]

    g = torch.from_numpy(np.random.default_rng(1).normal(0, 1, tuple(img.shape)).astype(np.float32)).to(cuda)
    img.backward(g)
    plain = rcv.load_dict({**TWO, "overlap_adjoint": False})
    want = plain.render_backward(scene, params, g, 0, seed=rcv.default_seed_grad(3), spp=4)[key].double()
    got = opt[key].grad.double()
    # the same events, added up in another order
    assert float((got - want).norm()) <= 1e-6 * float(want.norm())

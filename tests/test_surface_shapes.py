"""Surface kernels at the edges of their new pieces: texture records of one
texel, one row and ragged sizes (repeat wrap), films that never fill a warp's
shading threshold, a light between the spheres (shadow rays that reach its
plane), coloured light (quotients that share a divisor)."""
import numpy as np
import pytest
import torch

import recursive_control_variates_gb300 as rcv
from recursive_control_variates_gb300 import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tex_shape,res,spp", [((1, 1), 24, 4), ((1, 5), 24, 4), ((3, 2), 33, 3), ((5, 17), 48, 5),
                                               ((8, 8), 1, 1), ((8, 8), 1, 33), ((8, 8), 7, 2)])
@pytest.mark.parametrize("light_y,radiance", [(3.0, (15.0, 15.0, 15.0)), (0.45, (3.0, 0.5, 20.0))])
def test_surface_matches_oracle(cuda, oracle, tex_shape, res, spp, light_y, radiance):
    rng = np.random.default_rng(11)
    old, new = (rng.uniform(0.05, 0.95, (*tex_shape, 3)).astype(np.float32) for _ in range(2))
    d = scenes.surface_scene_dict(new, res=res, seed=1)
    d["light"] = {"type": "rectangle", "center": (0.0, light_y, 0.0), "half_size": (0.5, 0.5),
                  "emitter": {"type": "area", "radiance": radiance}}
    scene = rcv.load_dict(d, device=cuda)
    b = scene.named_shapes()["plane"].bsdf
    b.old.texture.data.copy_(torch.from_numpy(old))
    b._dirty = True
    cam = oracle.camera_basis(res, res, *scenes.SURFACE_CAMERA)
    osc = oracle.SurfaceScene(cam, old, new, scenes.surface_spheres(1), (0.0, light_y, 0.0), (0.5, 0.5), radiance,
                              plane_half=2.0, max_depth=7, rr_depth=3)
    integ = rcv.load_dict({"type": "twostateprb", "max_depth": 7, "rr_depth": 3})
    H, F = integ.render_twostates(scene, 0, seed=4, spp=spp)
    for a, o in zip((H, F), oracle.surface_render_twostates(osc, seed=4, spp=spp)):
        assert np.mean(np.all(a.cpu().numpy() == o, axis=-1)) >= 0.999
    gimg = rng.normal(0, 1, (res, res, 3)).astype(np.float32)
    want = oracle.surface_backward(osc, seed=9, spp=spp, grad_img=gimg)
    for adjoint in ("tape", "replay"):
        integ = rcv.load_dict({"type": "twostateprb", "max_depth": 7, "rr_depth": 3, "adjoint": adjoint})
        g = integ.render_backward(scene, rcv.traverse(scene), torch.from_numpy(gimg).to(cuda), 0, seed=9, spp=spp)
        got = g[scenes.TEXTURE_KEY].cpu().numpy().astype(np.float64)
        # float atomics in another order than the oracle's double sums
        assert np.linalg.norm(got - want) <= 2e-5 * np.linalg.norm(want)

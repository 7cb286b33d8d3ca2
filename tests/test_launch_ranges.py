"""Launches at the far ends of their dispatch rules: more than 64 paths per queue
fetch (single jobs of more than 15 M paths), and grids with an axis of 2^21
voxels or more, whose cells are located without the directed addition."""
import numpy as np
import pytest
import torch

import recursive_control_variates_gb300 as rcv
from recursive_control_variates_gb300 import scenes

from test_gpu_volume import frac_equal, make_scene, oracle_scene

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("spp", [65, 260])
def test_large_fetches_give_the_same_images(cuda, spp):
    """17 M and 68 M paths: fetches of 72 and 256 against the caller's 64."""
    scene, _, _ = make_scene(cuda, res=512)
    props = {"type": "twostateprbvolpath", "max_depth": 3, "rr_depth": 3}
    a = rcv.load_dict(props).render(scene, 0, seed=3, spp=spp)
    b = rcv.load_dict({**props, "batch": 64}).render(scene, 0, seed=3, spp=spp)
    assert torch.equal(a, b)


@pytest.mark.parametrize("n", [(1 << 21) - 1, 1 << 21, (1 << 21) + 5])
def test_long_axis_matches_oracle(cuda, oracle, n):
    """A column of n voxels along z of random density and albedo: images (99.9 %
    of the pixels bit-identical) and gradients (2e-5), the bounds of the other
    grids' tests."""
    rng = np.random.default_rng(n)
    old, new = (rng.uniform(1.0, 8.0, (n, 1, 1, 1)).astype(np.float32) for _ in range(2))
    ao, an = (rng.uniform(0.3, 0.95, (n, 1, 1, 3)).astype(np.float32) for _ in range(2))
    scene = rcv.load_dict(scenes.scene_dict(new, an, res=32, spp=4), device=cuda)
    med = scene.named_shapes()["object"].interior_medium()
    med.old.density.copy_(torch.from_numpy(old))
    med.old.albedo_grid.copy_(torch.from_numpy(ao))
    med._dirty = True
    osc = oracle_scene(oracle, scene, (old, new, ao, an), 8, True)
    integ = rcv.load_dict({"type": "twostateprbvolpath", "max_depth": 8, "rr_depth": 8})
    H, F = integ.render_twostates(scene, 0, seed=11, spp=4)
    Ho, Fo = oracle.render_twostates(osc, seed=11, spp=4)
    assert frac_equal(F.cpu().numpy(), Fo) >= 0.999 and frac_equal(H.cpu().numpy(), Ho) >= 0.999
    gimg = rng.normal(0, 1, (32, 32, 3)).astype(np.float32)
    g = integ.render_backward(scene, rcv.traverse(scene), torch.from_numpy(gimg).to(cuda), 0, seed=12, spp=4)
    od, oa = oracle.backward(osc, seed=12, spp=4, grad_img=gimg)
    for got, want in ((g[scenes.DENSITY_KEY].cpu().numpy()[..., 0], od), (g[scenes.ALBEDO_KEY].cpu().numpy(), oa)):
        assert np.linalg.norm(got.astype(np.float64) - want) <= 2e-5 * np.linalg.norm(want)

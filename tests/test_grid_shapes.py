"""Packing and gradient fold at the edges of their tiles: single-voxel axes,
rows of less than a warp, of a warp and one more, odd cell counts."""
import numpy as np
import pytest
import torch

import recursive_control_variates_gb300 as rcv
from recursive_control_variates_gb300 import scenes

from test_gpu_volume import frac_equal, oracle_scene

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(1, 1, 1), (2, 1, 3), (3, 2, 1), (31, 3, 2), (33, 2, 3), (64, 5, 3), (1, 4, 65)])
def test_grid_shapes_match_oracle(cuda, oracle, dims):
    """Images (>= 99.9 % of the pixels bit-identical) and gradients (2e-5) of
    a (dx, dy, dz) grid of random density and albedo, the bounds of the cubic
    grids' tests."""
    dx, dy, dz = dims
    rng = np.random.default_rng(dx * 100 + dy * 10 + dz)
    old, new = (rng.uniform(1.0, 8.0, (dz, dy, dx, 1)).astype(np.float32) for _ in range(2))
    ao, an = (rng.uniform(0.3, 0.95, (dz, dy, dx, 3)).astype(np.float32) for _ in range(2))
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
    gd = g[scenes.DENSITY_KEY].cpu().numpy()[..., 0].astype(np.float64)
    ga = g[scenes.ALBEDO_KEY].cpu().numpy().astype(np.float64)
    assert gd.shape == (dz, dy, dx) and ga.shape == (dz, dy, dx, 3)
    assert np.linalg.norm(gd - od) <= 2e-5 * np.linalg.norm(od)
    assert np.linalg.norm(ga - oa) <= 2e-5 * np.linalg.norm(oa)

"""Tracers whose warps have many paths each (one block per SM), so that lanes
walk several steps between two looks at the queue while others wait, against
the oracle with the tolerances of its other comparisons: images 99.9 % of the
pixels bit-identical, gradients 2e-5."""
import numpy as np
import pytest
import torch

import recursive_control_variates_gb300 as rcv
from recursive_control_variates_gb300 import scenes

from test_gpu_volume import frac_equal, make_scene, oracle_scene

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("albedo_grid,max_depth,factor", [(False, 6, 0), (True, 24, 0), (True, 8, 4)])
def test_many_paths_per_warp_match_oracle(cuda, oracle, albedo_grid, max_depth, factor):
    res, spp = 97, 16
    scene, med, grids = make_scene(cuda, albedo_grid=albedo_grid, res=res, max_depth=max_depth)
    med.set_majorant_resolution_factor(factor)
    osc = oracle_scene(oracle, scene, grids, max_depth, albedo_grid, majorant_factor=factor)
    integ = rcv.load_dict({"type": "twostateprbvolpath", "max_depth": max_depth, "rr_depth": max_depth,
                           "blocks_per_sm": 1})
    H, F = integ.render_twostates(scene, 0, seed=21, spp=spp)
    Ho, Fo = oracle.render_twostates(osc, seed=21, spp=spp)
    assert frac_equal(F.cpu().numpy(), Fo) >= 0.999 and frac_equal(H.cpu().numpy(), Ho) >= 0.999
    gimg = np.random.default_rng(5).normal(0, 1, (res, res, 3)).astype(np.float32)
    g = integ.render_backward(scene, rcv.traverse(scene), torch.from_numpy(gimg).to(cuda), 0, seed=22, spp=spp)
    want = oracle.backward(osc, seed=22, spp=spp, grad_img=gimg)
    for key, w in zip((scenes.DENSITY_KEY, scenes.ALBEDO_KEY)[: 1 + albedo_grid], want):
        got = g[key].cpu().numpy().astype(np.float64).reshape(w.shape)
        assert np.linalg.norm(got - w) <= 2e-5 * np.linalg.norm(w)

"""The flat gradient pass, whose lanes add their records pairwise, where pairs
are incomplete: a handful of paths, so that lanes without an event, odd event
counts and lone scattering events share a warp.  Same events as the replay,
another order of the additions: the 1e-6 of the larger films' comparison."""
import numpy as np
import pytest

from recursive_control_variates_gb300 import scenes

from test_gpu_volume import make_scene
from test_tape import grads_of

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("albedo_grid", [False, True])
@pytest.mark.parametrize("res,spp", [(1, 1), (1, 2), (1, 3), (2, 1), (5, 3)])
def test_few_paths_match_replay(cuda, res, spp, albedo_grid):
    scene, _, _ = make_scene(cuda, albedo_grid=albedo_grid, res=res)
    gimg = np.random.default_rng(res).normal(0, 1, (res, res, 3)).astype(np.float32)
    for seed in (1, 2, 3):
        tape = grads_of(cuda, scene, gimg, seed, spp, adjoint="tape")
        replay = grads_of(cuda, scene, gimg, seed, spp, adjoint="replay")
        for key in (scenes.DENSITY_KEY, scenes.ALBEDO_KEY)[: 1 + albedo_grid]:
            a, b = tape[key].astype(np.float64), replay[key].astype(np.float64)
            assert np.linalg.norm(a - b) <= 1e-6 * np.linalg.norm(b)

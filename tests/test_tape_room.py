"""Room of the adjoint's event tape: never smaller for more paths, and enough
for launches whose camera sees little else than the medium."""
import numpy as np
import pytest
import torch

import recursive_control_variates_gb300 as rcv
from recursive_control_variates_gb300 import _lib, scenes


def test_adjoint_scratch_grows_with_the_paths(rcvlib):
    """A workspace sized for a film serves every smaller one: across the path
    counts where the room per path changes (4.2 M, 16.8 M)."""
    paths = sorted({1, 2, 7, 255, 4096} | {(1 << 22) + k for k in (-2, -1, 0, 1, 2)} | {(1 << 24) + k for k in (-1, 0, 1)}
                   | {int(2 ** (k / 7)) for k in range(60, 180)})
    need = [rcvlib.rcv_render_workspace_bytes(1, 1, n, _lib.MODE_ADJOINT) for n in paths]
    assert all(a <= b for a, b in zip(need, need[1:]))
    # at least 16 slots of 20 bytes and 2 checkpoints of 64 per path, at most 10 GB beyond them
    for n, b in zip(paths, need):
        assert n * (16 * 20 + 2 * 64) <= b <= n * (16 * 20 + 2 * 64 + 28) + 10 * 10 ** 9


@pytest.mark.gpu
@pytest.mark.parametrize("width,spp,depth", [(29, 3, 8), (64, 16, 32)])
def test_full_view_tape_matches_replay(cuda, width, spp, depth):
    """Two cameras close to the box: nearly every path is long.  Same terms as
    the replay in another order of float additions (thousands per voxel):
    2e-5 relative L2."""
    d = scenes.scene_dict(scenes.blob_density(20, 3), scenes.albedo_grid(20, 3), res=width,
                          views=scenes.orbit_views(None, 2, distance=0.9))
    scene = rcv.load_dict(d, device=cuda)
    params = rcv.traverse(scene)
    g = torch.from_numpy(np.random.default_rng(9).normal(0, 1, (width, 2 * width, 3)).astype(np.float32)).to(cuda)
    got, want = (rcv.load_dict({"type": "twostateprbvolpath", "max_depth": depth, "rr_depth": depth, "adjoint": a})
                 .render_backward(scene, params, g, 0, seed=5, spp=spp) for a in ("tape", "replay"))
    for key in want:
        a, b = got[key].double(), want[key].double()
        assert float((a - b).norm()) <= 2e-5 * float(b.norm())

"""Room of the batched tape adjoint's event records: 2 per gradient path and the
margin, the list of paths that entered the medium kept elsewhere."""
import ctypes as C

import numpy as np
import pytest
import torch

import recursive_control_variates_gb300 as rcv
from recursive_control_variates_gb300 import _lib, batch, scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("graph", [False, True])
def test_records_fill_their_room(cuda, graph):
    """Thick constant media that fill the view: no null collisions, so a path
    makes about two tape events per scattering event and the records run out
    before the tape.  Every lost path asked for one record too many."""
    w, spp = 256, 4
    jobs = []
    for k in range(2):
        d = scenes.scene_dict(np.full((4, 4, 4, 1), 20.0 + k, np.float32), 0.9, res=w, two_state=False)
        d["sensor"]["to_world"] = rcv.core.look_at((0.5, 0.5, 1.4), (0.5, 0.5, 0.5), (0.0, 1.0, 0.0))
        scene = rcv.load_dict(d, device=cuda)
        target = torch.full((w, w, 3), 0.3, device=cuda)
        jobs.append(batch.CVJob(np.full((4, 4, 4, 1), 20.0 + k, np.float32), 0.9, target, scene.sensors()[0], spp=spp,
                                seed=3 + k, lr=1e-3, max_depth=7, rr_depth=7, device=cuda))
    others = [j.clone() for j in jobs]
    b = batch.BatchedCV(jobs, use_graph=graph)
    r = batch.BatchedCV(others, batch.LaunchOptions(adjoint="replay"), use_graph=graph)
    at = int(_lib.load().rcv_batch_counters(b._handle)) - b.workspace.data_ptr() - 256
    paths = 2 * w * w * spp
    b.step()
    torch.cuda.synchronize()
    q = b.workspace[at:at + 64].cpu().numpy().view(np.uint64).astype(np.int64)
    records, slots, lost, entered = q[3], q[4], q[5], q[6]
    assert entered == paths and slots <= 16 * paths and lost > 0
    assert records - lost == 2 * paths + 65536
    b.step()  # no longer constant: shadow walks go on, and the tape runs out too
    r.step(2)
    for a, o in zip(jobs, others):
        # gradients of two steps (moments): float atomics in another order, the second step's
        # parameters off by the first one's rounding
        d = (a.density_m.double() - o.density_m.double()).norm()
        assert float(d) <= 1e-3 * float(o.density_m.double().norm())
    b.close()
    r.close()

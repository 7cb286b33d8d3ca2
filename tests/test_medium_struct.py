"""The medium description of a call follows the medium's public attributes,
however they were changed."""
import numpy as np
import pytest

import recursive_control_variates_gb300 as rcv
from recursive_control_variates_gb300 import scenes


@pytest.mark.parametrize("kind", [list, np.array])
def test_constant_albedo_changed_in_place(rcvlib, kind):
    med = rcv.load_dict(scenes.scene_dict(scenes.blob_density(4, 0), 0.8, res=8, two_state=False),
                        device="cpu").named_shapes()["object"].interior_medium()
    med.albedo_value = kind([0.8, 0.8, 0.8])
    assert list(med.c_struct().albedo_value) == pytest.approx([0.8, 0.8, 0.8])
    med.albedo_value[1] = 0.25
    assert list(med.c_struct().albedo_value) == pytest.approx([0.8, 0.25, 0.8])
    med.albedo_value = kind([0.5, 0.25, 0.8])
    assert list(med.c_struct().albedo_value) == pytest.approx([0.5, 0.25, 0.8])

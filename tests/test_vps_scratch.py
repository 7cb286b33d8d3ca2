"""Scratch of the volpathsimple adjoint: only where paths are recorded."""
import pytest

import recursive_control_variates_gb300 as rcv

from test_adjoint_scratch import volume_sensor


@pytest.mark.parametrize("flags,uses", [({}, True), ({"use_drt": False}, True),
                                        ({"use_drt": False, "use_drt_subsampling": False}, True),
                                        ({"use_drt_subsampling": False}, False)])
def test_scratch_only_to_record(rcvlib, flags, uses):
    """DRT without subsampling runs one thread per path, without scratch."""
    integ = rcv.load_dict({"type": "volpathsimple", **flags})
    ws = integ._adjoint_scratch("cpu", volume_sensor(), 1)
    assert (ws is not None) == uses

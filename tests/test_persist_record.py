"""The closing record of a persistent solve lands where the solve before left its own: a copy or
a wait that failed, or a record that never landed, must not pass for a result (host logic, with
the CUDA codes given)."""
import os

import pytest

import semiconductor_devices_simulator_b200 as S

pytestmark = pytest.mark.skipif(not os.path.exists(S.LIB_PATH), reason="solver library not built")


@pytest.mark.parametrize("copy,wait,arrives,err,verdict", [
    (0, 0, 1, 0, 1),          # arrived, no barrier ran out
    (0, 0, 1, 1, -1),         # a barrier wait ran out
    (0, 0, 0, 0, -1),         # nothing arrived: the old record is still there
    (0, 719, 0, 0, -1),       # the launch failed (cudaErrorLaunchFailure seen by the wait)
    (0, 719, 1, 0, -1),
    (1, 0, 1, 0, -1),         # the copy was refused
])
def test_record_verdict(copy, wait, arrives, err, verdict):
    assert S.load().b200x_persist_record(copy, wait, arrives, err) == verdict

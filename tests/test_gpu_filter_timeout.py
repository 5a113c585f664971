"""The filter's last launch changes the state only from masks that settled: after a
wait of the resolution gave up (or its rounds ran out) a reported timeout leaves
the state as it was."""
import ctypes
import os

import pytest

pytestmark = pytest.mark.gpu

PROBE = os.path.join(os.path.dirname(os.path.abspath(__file__)), "_build", "libfilterprobe.so")


@pytest.mark.parametrize("settled,gave_up,changed", [(1, 0, 64), (0, 0, 0), (0, 1, 0), (1, 1, 0)])
def test_only_settled_masks_are_applied(pfd, settled, gave_up, changed):
    assert ctypes.CDLL(PROBE).filter_apply_probe(settled, gave_up) == changed

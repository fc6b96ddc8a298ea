"""What the kernels' sources have to hold that no run can show."""

import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "tensix-kernels_b200" / "csrc"


@pytest.mark.parametrize("name", ["tkd_stream_tc.cuh", "tkd_wide.cuh"])
def test_a_fence_after_every_wait_for_tensor_memory(name):
    """The barriers that tensor memory changes hands by (operand slots and accumulators, full and empty): behind a wait for one, and before
    the next wait, tcgen05.fence::after_thread_sync; without it the tensor memory's loads and stores may be ahead of the wait."""
    lines = (CSRC / name).read_text().splitlines()
    waits = [i for i, line in enumerate(lines) if re.search(r"mbar_wait(_parked)?\((a|acc)(full|empty)0", line)]
    assert len(waits) >= 4
    for i in waits:
        behind = lines[i + 1 : i + 20]
        fence = next((j for j, line in enumerate(behind) if "tc_fence_after();" in line), None)
        assert fence is not None, (name, i + 1, lines[i])
        assert not any("mbar_wait" in line and "xfull0" not in line for line in behind[:fence]), (name, i + 1, lines[i])

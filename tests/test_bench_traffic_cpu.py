"""The DRAM bytes that bench.py reports for a multi-step launch come from the
profile's record of a step."""
import pytest

import bench


@pytest.mark.parametrize("name", ["c2", "c3"])
def test_multi_step_launch_has_its_traffic(name):
    tr = bench.ncu_traffic(name)
    per_step = tr["step_dram_bytes_multi"]
    assert bench.multi_traffic(tr, 20, 3) == per_step * 20 // 3 > per_step
    assert bench.multi_traffic({}, 20, 3) is None

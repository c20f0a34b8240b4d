"""Multi-step launches beside other streams' work: a long run goes out as
launches of a bounded number of steps, and several handles stepped at the same
time share the GPU; results as alone."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _ready(dims, steps, amp=1.0):
    from maxwell_solver_gb300 import simFDTD

    P = simFDTD("CreateSimulation")
    simFDTD("SetParams", P, np.float64([5, 7, 3, 1, 0.08, 1, 0.8, 0]))
    simFDTD("SetConst", P, np.float32([20e9, 1e-3, 1.7e-12]), np.int32([steps, *dims, 0]))
    pulse = (np.sin(0.05 * np.arange(steps)) * amp).astype(np.float32)
    simFDTD("SetSource", P, pulse)
    simFDTD("ReadySimulation", P)
    simFDTD("SetIncidence", P, np.float64([0.9, -0.6, 1.2]))
    simFDTD("Init1D", P, np.float32(1), pulse)
    return P


@pytest.mark.parametrize("dims, most", [((26, 30, 24), 256), ((64, 64, 64), 256),
                                        ((200, 180, 160), 94)])
def test_long_runs_are_several_launches(dims, most):
    """256 steps or 2^29 cell-steps a launch."""
    from maxwell_solver_gb300 import launch_count, simFDTD

    steps = 5 * most
    P = _ready(dims, steps)
    before = launch_count()
    simFDTD("StepN", P, np.int32([0, steps, 5]))
    assert 5 <= launch_count() - before <= 6
    simFDTD("DeleteSimulation", P)

"""Checkpoints where no device memory is left for their scratch: the image is
the same, and a run resumed from it ends as the uninterrupted one.  The failing
allocation is injected on the host."""
import numpy as np
import pytest

from test_checkpoint_gpu import SC, _ready, _state, _steps

pytestmark = pytest.mark.gpu

FAULT_NONE, FAULT_DEVICE_ALLOC = 0, 1


@pytest.mark.parametrize("dims", [SC.dims, (53, 47, 50)])
def test_checkpoint_without_scratch(native_lib, dims):
    from maxwell_solver_gb300 import simFDTD

    sc = type(SC)(**{**SC.__dict__, "dims": dims})
    inp = sc.inputs()
    half = sc.steps // 2
    P = _ready(simFDTD, sc, inp)
    _steps(simFDTD, P, sc, 0, half)
    want_image = simFDTD("SaveCheckpoint", P)
    assert native_lib.fdtd_inject_fault(FAULT_DEVICE_ALLOC, 1) == 0
    image = simFDTD("SaveCheckpoint", P)  # takes the injected failure
    np.testing.assert_array_equal(image, want_image)
    Q = _ready(simFDTD, sc, inp)
    assert native_lib.fdtd_inject_fault(FAULT_DEVICE_ALLOC, 1) == 0
    simFDTD("LoadCheckpoint", Q, image)
    R = _ready(simFDTD, sc, inp)  # (its allocations succeed: the load took the failure)
    assert native_lib.fdtd_inject_fault(FAULT_NONE, 0) == 0
    simFDTD("DeleteSimulation", R)
    for X in (P, Q):
        _steps(simFDTD, X, sc, half, sc.steps - half)
    for a, b in zip(_state(simFDTD, P, sc)[0], _state(simFDTD, Q, sc)[0]):
        np.testing.assert_array_equal(a, b)
    simFDTD("DeleteSimulation", P)
    simFDTD("DeleteSimulation", Q)

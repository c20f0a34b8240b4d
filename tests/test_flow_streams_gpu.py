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


def _run_together(n, dims, steps, chunk, threads):
    """Fields of n handles stepped at the same time, and the seconds it took."""
    import threading
    import time

    from maxwell_solver_gb300 import _native, simFDTD

    lib = _native.load()
    Ps = [_ready(dims, steps, 1.0 + g) for g in range(n)]

    def go(mine):
        for first in range(0, steps, chunk):
            for P in mine:
                simFDTD("StepN", P, np.int32([first, chunk, 5]))
        for P in mine:
            assert lib.fdtd_synchronize(int(P[0])) == 0

    for P in Ps:
        assert lib.fdtd_synchronize(int(P[0])) == 0
    t = time.perf_counter()
    if threads:
        pool = [threading.Thread(target=go, args=([P],)) for P in Ps]
        for x in pool:
            x.start()
        for x in pool:
            x.join()
    else:
        go(Ps)
    t = time.perf_counter() - t
    out = [[simFDTD("OutputVis", P, np.uint32(np.prod(dims)), np.int32(f)) for f in range(1, 7)]
           for P in Ps]
    for P in Ps:
        simFDTD("DeleteSimulation", P)
    return out, t


@pytest.mark.parametrize("threads", [False, True])
def test_handles_at_the_same_time_share_the_gpu(threads):
    """Eight handles end as each does alone, in less time than one after the
    other (whole-GPU launches of a 40^3 grid in turn: eight times as long; as
    separate kernels 1.5 times)."""
    from maxwell_solver_gb300 import simFDTD

    dims, steps, chunk = (40, 41, 39), 600, 50
    _run_together(1, dims, steps, chunk, False)  # first use of the kernels
    together, t8 = _run_together(8, dims, steps, chunk, threads)
    t1 = min(_run_together(1, dims, steps, chunk, False)[1] for _ in range(3))
    for g in range(8):
        P = _ready(dims, steps, 1.0 + g)
        simFDTD("StepN", P, np.int32([0, steps, 5]))
        for f in range(6):
            np.testing.assert_array_equal(
                together[g][f], simFDTD("OutputVis", P, np.uint32(np.prod(dims)), np.int32(f + 1)))
        simFDTD("DeleteSimulation", P)
    assert t8 < 6 * t1, (t8, t1)

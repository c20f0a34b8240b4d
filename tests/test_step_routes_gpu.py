"""Whole steps on every route a StepN call may take, against the FP32 oracle,
bit for bit (every route does the same roundings): the item heights of mode 5,
and the separate half-step kernels where multi-step launches are not taken."""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

FIELDS = ("Ex", "Ey", "Ez", "Hx", "Hy", "Hz")


def _run_equal(dims, pml, inset, steps, mode, probes=None, calls=(1, 9)):
    """StepN in calls of 1, 9 and the remaining steps; returns the launches of
    the last call."""
    import oracle
    from maxwell_solver_gb300 import launch_count, simFDTD

    rng = np.random.default_rng(sum(dims))
    dx = 1e-3
    fr = np.float32([20e9, dx, 0.9 * dx / (math.sqrt(3) * 299792458.0)])
    td = np.int32([steps, *dims, 0 if probes is None else len(probes)])
    pulse = np.sin(0.4 * np.arange(steps) + 0.3).astype(np.float32)
    eps = (1 + rng.integers(0, 4, dims)).ravel(order="F").astype(np.float32)
    P = simFDTD("CreateSimulation")
    o = oracle.OracleSim("f32")
    simFDTD("SetParams", P, np.float64([pml, inset, 3, 1, 0.08, 1, 0.8, 0]))
    o.set_params(pml=pml, tfsf_width=inset)
    simFDTD("SetConst", P, fr, td)
    o.set_const(fr, td)
    if probes is not None:
        simFDTD("SetAntennaLocations", P, np.asfortranarray(np.int32(probes)))
        o.set_antenna_locations(np.asfortranarray(np.int32(probes)))
    simFDTD("UpdateMaterial", P, np.int32(5), eps)
    o.update_material(5, eps)
    simFDTD("ReadySimulation", P)
    o.ready_simulation()
    if mode == 5:
        simFDTD("SetIncidence", P, np.float64([0.9, -0.6, 1.2]))
        o.set_incidence(0.9, -0.6, 1.2)
    if mode:
        simFDTD("Init1D", P, np.float32(1), pulse)
        o.init_1d(1.0, pulse)
    at = 0
    for n in (*calls, steps - sum(calls)):
        before = launch_count()
        simFDTD("StepN", P, np.int32([at, n, mode]))
        at += n
    launches = launch_count() - before
    for n in range(steps):
        o.step(n, mode)
    for f, field in enumerate(FIELDS, 1):
        got = simFDTD("OutputVis", P, np.uint32(np.prod(dims)), np.int32(f))
        np.testing.assert_array_equal(got, o.field(field), err_msg=field)
    if probes is not None:
        rec = simFDTD("OutputProbes", P, np.uint32(steps * len(probes) * 6))
        np.testing.assert_array_equal(rec, o.array("probes"))
    if mode:
        assert max(np.abs(o.field(f)).max() for f in FIELDS) > 0
    simFDTD("DeleteSimulation", P)
    return launches


@pytest.mark.parametrize("dims, pml, steps", [
    ((45, 130, 79), 6, 40),     # one plane an item: few of them
    ((41, 301, 80), 6, 30),     # one plane: K <= 80
    ((95, 96, 97), 6, 40),      # two planes
    ((47, 99, 181), 6, 30),     # four planes
    ((40, 1003, 41), 6, 24),    # eight planes: many items
    ((65, 66, 313), 6, 24),     # eight planes: long
])
def test_item_heights_of_mode_5(dims, pml, steps):
    assert _run_equal(dims, pml, pml + 2, steps, 5) == 1


def test_long_grids_of_a_small_section_in_mode_5_take_the_separate_kernels():
    assert _run_equal((38, 41, 262), 6, 8, 60, 5) > 50


@pytest.mark.parametrize("to_end", [False, True])
def test_batch_of_24_in_mode_5(to_end):
    """Stepped together they run as separate kernels, to the end in one call as
    multi-step launches; each ends as alone."""
    from maxwell_solver_gb300 import launch_count, simFDTD
    from maxwell_solver_gb300.batch import Batch

    dims = [(26 + g % 7, 27 + g % 5, 26 + g % 9) for g in range(24)]
    steps = [60 + g % 4 for g in range(24)]

    def ready(d):
        P = simFDTD("CreateSimulation")
        simFDTD("SetParams", P, np.float64([5, 7, 3, 1, 0.08, 1, 0.8, 0]))
        simFDTD("SetConst", P, np.float32([20e9, 1e-3, 1.7e-12]), np.int32([70, *d, 0]))
        simFDTD("ReadySimulation", P)
        simFDTD("SetIncidence", P, np.float64([0.9, -0.6, 1.2]))
        simFDTD("Init1D", P, np.float32(1), np.sin(0.4 * np.arange(70)).astype(np.float32))
        return P

    Ps = [ready(d) for d in dims]
    with Batch() as b:
        for P, n in zip(Ps, steps):
            b.add(P, 0, n, 5)
        before = launch_count()
        if to_end:
            b.run()
            # one each, and 12 steps that measure the separate kernels' z-run
            assert launch_count() - before <= 24 + 12 * 6
        else:
            b.step(32)
            assert launch_count() - before > 24 + 12 * 6
            b.run()
    for P, d, n in zip(Ps, dims, steps):
        Q = ready(d)
        simFDTD("StepN", Q, np.int32([0, n, 5]))
        for f in range(1, 7):
            cells = np.uint32(np.prod(d))
            np.testing.assert_array_equal(simFDTD("OutputVis", P, cells, np.int32(f)),
                                          simFDTD("OutputVis", Q, cells, np.int32(f)))
        simFDTD("DeleteSimulation", P)
        simFDTD("DeleteSimulation", Q)


def _dense(dims, pml):
    """Probe positions (relative to the CPML) on an inner z-plane and on the
    last planes of the three axes, without the edge j = J-1, k = K-1."""
    I, J, K = (d - pml for d in dims)
    at = [(i, j, K // 2) for i in range(0, I, 2) for j in range(0, J)]
    at += [(I - 1, j, k) for j in range(0, J - 1, 3) for k in range(0, K, 2)]
    at += [(i, J - 1, k) for i in range(0, I, 5) for k in range(0, K - 1, 3)]
    at += [(i, j, K - 1) for i in range(0, I, 4) for j in range(0, J - 1, 5)]
    return at


@pytest.mark.parametrize("dims, pml, steps, mode", [
    ((45, 50, 41), 5, 24, 3),      # one plane an item
    ((97, 81, 67), 6, 16, 0),      # two planes
    ((331, 113, 109), 8, 12, 5),   # eight planes, tiles of 64 x 8
])
def test_dense_probes(dims, pml, steps, mode):
    assert _run_equal(dims, pml, pml + 2, steps, mode, _dense(dims, pml)) == 1


@pytest.mark.parametrize("tile", ["0", "1", "2"])
@pytest.mark.parametrize("mode", [0, 1, 3, 5])
def test_separate_kernels_with_a_probe_on_the_outer_edge(mode, tile, monkeypatch):
    """A probe at j = J-1, k = K-1: the steps run as separate half-step kernels
    in every tile geometry, 32 of them as a graph replay."""
    monkeypatch.setenv("FDTD_TILE", tile)
    dims, pml = (70, 53, 42), 5
    corner = [(20, dims[1] - 1 - pml, dims[2] - 1 - pml), (30, 20, 11)]
    assert _run_equal(dims, pml, pml + 2, 60, mode, corner) > 50


def test_separate_kernels_with_compacted_x():
    """The same with the compacted CPML X kernels (FDTD_XC=1, read once per
    process: in a child process)."""
    import os
    import subprocess
    import sys

    r = subprocess.run([sys.executable, "-m", "pytest", "-q", "-x", "-m", "gpu", "-k",
                        "probe_on_the_outer_edge", os.path.abspath(__file__)],
                       env=dict(os.environ, FDTD_XC="1"), capture_output=True, text=True,
                       timeout=300)
    assert r.returncode == 0, r.stdout[-3000:] + r.stderr[-2000:]


def test_a_source_on_a_face_in_mode_5_is_refused_at_its_step():
    """Per-op calls: the next step's first call reports it, not a later one."""
    from maxwell_solver_gb300 import SimFDTDError, simFDTD

    dims, pml, steps = (40, 36, 34), 5, 8
    P = simFDTD("CreateSimulation")
    simFDTD("SetParams", P, np.float64([pml, pml + 3, 3, 1, 0.08, 1, 0.8, 0]))
    simFDTD("SetConst", P, np.float32([20e9, 1e-3, 1.7e-12]), np.int32([steps, *dims, 0]))
    pulse = np.sin(0.4 * np.arange(steps)).astype(np.float32)
    simFDTD("SetSource", P, pulse)
    simFDTD("ReadySimulation", P)
    simFDTD("SetIncidence", P, np.float64([0.9, -0.6, 1.2]))
    simFDTD("Init1D", P, np.float32(1), pulse)
    tm = np.int32([0, 5])
    simFDTD("UpdateH_All", P)
    simFDTD("UpdateH_PlaneWave", P, tm)
    simFDTD("UpdateH_PML", P)
    simFDTD("UpdateE_All", P)
    simFDTD("UpdateE_PlaneWave", P, tm)
    simFDTD("UpdateE_PML", P)
    simFDTD("AddCurrents", P, np.int32([0, 1]), np.int32([pml + 3, pml + 3, 12, 14, 12, 14]))
    with pytest.raises(SimFDTDError):
        simFDTD("UpdateH_All", P)
    simFDTD("DeleteSimulation", P)

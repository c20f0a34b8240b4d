"""Steps as multi-step launches (fdtd_flow.cu) against the FP32 oracle, bit
for bit (every route does the same roundings, so the tolerance is zero): each
item height (1, 2, 4 and 8 planes, by grid size) and tile with partial tiles, partial
chunks and rows that are not a multiple of four cells, TF/SF modes, current
sources, coefficient arrays, per-cell H coefficients, and probes on the last
planes.  A run is split into several calls, so that launches go on from each
other's counters."""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

FIELDS = ("Ex", "Ey", "Ez", "Hx", "Hy", "Hz")
CASES = {
    # name: dims, pml, TF/SF inset, steps, mode, options
    "tiny": ((17, 18, 19), 3, 5, 40, 3, ""),
    "below_tile": ((33, 31, 20), 5, 7, 40, 1, "current"),
    "one_over_tile": ((65, 49, 34), 8, 10, 40, 2, ""),
    "x_slabs_apart": ((42, 34, 26), 7, 9, 40, 4, "arrays"),
    "magnetic": ((61, 46, 37), 6, 8, 40, 1, "magnetic"),
    "subnormal": ((50, 41, 33), 7, 9, 60, 4, "current 1e-36"),
    "huge": ((50, 41, 33), 7, 9, 60, 3, "current 1e24"),
    "plain_current": ((63, 47, 35), 8, 10, 40, 0, "current arrays"),
    "oblique": ((71, 38, 43), 6, 8, 60, 5, "arrays"),
    "oblique_small": ((33, 41, 35), 5, 7, 60, 5, "magnetic"),
    "oblique_over_tiles": ((65, 49, 34), 8, 10, 60, 5, ""),
    "oblique_two_planes": ((97, 73, 66), 9, 11, 60, 5, "magnetic"),
    "oblique_four_planes": ((130, 117, 109), 9, 11, 60, 5, ""),
    "two_planes": ((97, 81, 67), 10, 12, 48, 3, "current"),
    "four_planes": ((129, 95, 78), 9, 11, 48, 2, "magnetic"),
    "big": ((198, 155, 131), 10, 12, 48, 1, ""),
    "big_oblique": ((165, 173, 142), 9, 11, 64, 5, "magnetic"),
    "big_wide": ((331, 113, 109), 8, 10, 48, 3, "current arrays"),
}


@pytest.mark.parametrize("name", CASES)
def test_multi_step_launches_equal_oracle(name, monkeypatch):
    import oracle
    from maxwell_solver_gb300 import info, simFDTD

    dims, pml, inset, steps, mode, opts = CASES[name]
    rng = np.random.default_rng(len(name))
    if "arrays" in opts:
        monkeypatch.setenv("FDTD_COEF", "arrays")
    I, J, K = dims
    dx = 1e-3
    fr = np.float32([20e9, dx, 0.9 * dx / (math.sqrt(3) * 299792458.0)])
    probes = np.int32([rng.integers(1, d - 2 * pml, 4) for d in dims]).T
    last = np.int32(dims) - 1 - pml  # the last plane of an axis
    for a in range(3):
        probes[a, a] = last[a]
    probes[3] = inset - pml + 1  # where the wave enters
    probes = np.asfortranarray(probes)
    ids = rng.integers(0, 40, dims)
    vals = rng.random(40).astype(np.float32)
    mats = {f: (vals[ids] * (0.05 if f < 4 else 4) + (f > 3)).ravel(order="F").astype(np.float32)
            for f in range(1, 7)}
    mu = (1 + rng.random(dims)).astype(np.float32).ravel(order="F")
    size = float(opts.split()[-1]) if "1e" in opts else 1.0
    pulse = (np.sin(0.4 * np.arange(steps) + 0.3) * size).astype(np.float32)
    box = np.int32([I // 2 - 2, I // 2 + 3, J // 2, J // 2, pml + 1, K - pml - 2])
    cur = "current" in opts

    P = simFDTD("CreateSimulation")
    o = oracle.OracleSim("f32")
    simFDTD("SetParams", P, np.float64([pml, inset, 3, 1, 0.08, 1, 0.8, 0]))
    o.set_params(pml=pml, tfsf_width=inset)
    td = np.int32([steps, I, J, K, 4])
    simFDTD("SetConst", P, fr, td)
    o.set_const(fr, td)
    simFDTD("SetSource", P, pulse)
    o.set_source(pulse)
    simFDTD("SetAntennaLocations", P, probes)
    o.set_antenna_locations(probes)
    for f, v in mats.items():
        simFDTD("UpdateMaterial", P, np.int32(f), v)
        o.update_material(f, v)
    simFDTD("ReadySimulation", P)
    o.ready_simulation()
    if "magnetic" in opts:
        simFDTD("SetMagnetic", P, mu, mu, mu)
        o.set_magnetic([mu, mu, mu])
    if mode == 5:
        simFDTD("SetIncidence", P, np.float64([0.9, -0.6, 1.2]))
        o.set_incidence(0.9, -0.6, 1.2)
    if mode:
        simFDTD("Init1D", P, np.float32(1), pulse)
        o.init_1d(1.0, pulse)
    assert info(P)["coef_mode"] == (0 if "arrays" in opts else 1)

    at = 0
    for n in (1, steps // 2, steps - 1 - steps // 2):
        simFDTD("StepN", P, np.int32([at, n, mode]), *([np.int32([2, *box])] if cur else []))
        at += n
    for n in range(steps):
        o.step(n, mode)
        if cur:
            o.add_currents(n, 2, tuple(int(b) for b in box))
    for f, field in enumerate(FIELDS, 1):
        got = simFDTD("OutputVis", P, np.uint32(I * J * K), np.int32(f))
        np.testing.assert_array_equal(got, o.field(field), err_msg=field)
    rec = simFDTD("OutputProbes", P, np.uint32(steps * 4 * 6))
    np.testing.assert_array_equal(rec, o.array("probes"))
    assert max(np.abs(o.field(f)).max() for f in FIELDS) > 0
    simFDTD("DeleteSimulation", P)


def test_batch_changing_route_equals_alone():
    """42 members run as batched half-steps; as members finish, the 38 and fewer
    left go on as multi-step launches; a member added then starts there."""
    from maxwell_solver_gb300 import simFDTD
    from maxwell_solver_gb300.batch import Batch
    from scenarios import SCENARIOS, run_mex

    def ready(sc):
        return run_mex(simFDTD, type(sc)(**{**sc.__dict__, "steps": 0}), sc.inputs())

    def fields(P, sc):
        n = np.uint32(np.prod(sc.dims))
        return [simFDTD("OutputVis", P, n, np.int32(f)) for f in range(1, 7)]

    def current(sc):
        return (sc.cur_mode, sc.cur_box) if sc.cur_mode else None

    mix = [SCENARIOS[g % len(SCENARIOS)] for g in range(43)]
    steps = [10 + g for g in range(43)]
    members = [ready(sc) for sc in mix]
    with Batch() as b:
        for P, sc, n in zip(members[:42], mix, steps):
            b.add(P, 0, n, sc.mode, current(sc))
        for _ in range(8):  # past the change of route
            b.step(1 << 20)
        b.add(members[42], 0, steps[42], mix[42].mode, current(mix[42]))
        b.step(3)
        b.run()
        for P, sc, n in zip(members, mix, steps):
            Q = ready(sc)
            cur = [np.int32([sc.cur_mode, *sc.cur_box])] if sc.cur_mode else []
            simFDTD("StepN", Q, np.int32([0, n, sc.mode]), *cur)
            for a, w, f in zip(fields(P, sc), fields(Q, sc), FIELDS):
                np.testing.assert_array_equal(a, w, err_msg=f"{sc.name} {n} {f}")
            simFDTD("DeleteSimulation", Q)
            simFDTD("DeleteSimulation", P)

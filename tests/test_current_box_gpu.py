"""Current sources whose box reaches the grid's outer edge or past it, against
the FP32 oracle, bit for bit (every route does the same roundings).  Cells of
the box that lie outside the grid take nothing; a box wholly outside is no
source.  Grids that are whole tiles (32 x 16 cells) and that are not, through
StepN, the per-op calls and a batch."""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

FIELDS = ("Ex", "Ey", "Ez", "Hx", "Hy", "Hz")
PML, STEPS = 4, 24
PAST = {
    # name: dims, box; past the end of i, j, k, of all three, and outside
    "i": ((40, 36, 30), (37, 56, 17, 19, 12, 14)),
    "i_whole_tile": ((64, 48, 30), (60, 95, 20, 20, 9, 11)),
    "j": ((33, 31, 28), (15, 17, 28, 47, 13, 13)),
    "j_whole_tile": ((64, 48, 30), (31, 33, 45, 63, 14, 15)),
    "k": ((40, 36, 30), (18, 20, 17, 17, 27, 36)),
    "all": ((42, 31, 27), (0, 99, 0, 99, 0, 99)),
    "outside_i": ((42, 31, 27), (42, 60, 12, 14, 12, 14)),
    "outside_k": ((40, 36, 30), (18, 20, 17, 17, 30, 31)),
}


def _pulse():
    return np.sin(0.5 * np.arange(STEPS) + 0.4).astype(np.float32)


def _const(dims):
    dx = 1e-3
    fr = np.float32([20e9, dx, 0.9 * dx / (math.sqrt(3) * 299792458.0)])
    return fr, np.int32([STEPS, *dims, 0])


def _ready(dims):
    from maxwell_solver_gb300 import simFDTD

    P = simFDTD("CreateSimulation")
    simFDTD("SetParams", P, np.float64([PML, PML + 2, 3, 1, 0.08, 1, 0.8, 0]))
    simFDTD("SetConst", P, *_const(dims))
    simFDTD("SetSource", P, _pulse())
    simFDTD("UpdateMaterial", P, np.int32(4), _eps(dims))
    simFDTD("ReadySimulation", P)
    return P


def _eps(dims):
    rng = np.random.default_rng(sum(dims))
    return (1 + rng.integers(0, 4, dims)).ravel(order="F").astype(np.float32)


def _oracle(dims, mode, box):
    import oracle

    o = oracle.OracleSim("f32")
    o.set_params(pml=PML, tfsf_width=PML + 2)
    o.set_const(*_const(dims))
    o.set_source(_pulse())
    o.update_material(4, _eps(dims))
    o.ready_simulation()
    for n in range(STEPS):
        o.step(n, 0)
        o.add_currents(n, mode, box)
    return o


def _by_ops(P, mode, box):
    from maxwell_solver_gb300 import simFDTD

    for n in range(STEPS):
        for op in ("UpdateH_All", "UpdateH_PML", "UpdateE_All", "UpdateE_PML"):
            simFDTD(op, P)
        simFDTD("AddCurrents", P, np.int32([n, mode]), np.int32(box))


def _by_step_n(P, mode, box):
    from maxwell_solver_gb300 import simFDTD

    for first, n in ((0, 1), (1, STEPS - 1)):
        simFDTD("StepN", P, np.int32([first, n, 0]), np.int32([mode, *box]))


def _by_batch(P, mode, box):
    from maxwell_solver_gb300.batch import Batch

    with Batch() as b:
        b.add(P, 0, STEPS, 0, (mode, box))
        b.run()


def _assert_equal(P, o, dims):
    from maxwell_solver_gb300 import simFDTD

    for f, field in enumerate(FIELDS, 1):
        got = simFDTD("OutputVis", P, np.uint32(np.prod(dims)), np.int32(f))
        np.testing.assert_array_equal(got, o.field(field), err_msg=field)


@pytest.mark.parametrize("run", [_by_step_n, _by_ops, _by_batch])
@pytest.mark.parametrize("name", PAST)
def test_box_past_the_grid_is_clipped(name, run):
    from maxwell_solver_gb300 import simFDTD

    dims, box = PAST[name]
    mode = 1 + len(name) % 3
    P = _ready(dims)
    run(P, mode, box)
    o = _oracle(dims, mode, box)
    _assert_equal(P, o, dims)
    assert (max(np.abs(o.field(f)).max() for f in FIELDS) > 0) == ("outside" not in name)
    simFDTD("DeleteSimulation", P)


# The edge j = J-1, k = K-1 in items of its own: J-1 and K-1 multiples of the
# tile's height and of the item's planes (1, 2, 4 and 8 by grid size; tiles of
# 16 rows, of 8 for rows of 320 cells and more).  Only the source reaches it.
EDGE = {
    "one_plane": ((24, 33, 24), (8, 11, 30, 32, 20, 23)),
    "one_plane_64": ((64, 65, 64), (5, 40, 64, 64, 63, 63)),
    "two_planes": ((97, 81, 67), (0, 96, 79, 80, 64, 66)),
    "four_planes": ((129, 97, 93), (64, 66, 96, 96, 90, 92)),
    "eight_planes": ((198, 161, 129), (100, 140, 160, 160, 126, 128)),
    "wide": ((331, 113, 113), (300, 330, 110, 112, 112, 112)),
}


@pytest.mark.parametrize("name", EDGE)
def test_source_over_the_outer_edge(name):
    from maxwell_solver_gb300 import simFDTD

    dims, box = EDGE[name]
    P = _ready(dims)
    _by_step_n(P, 1, box)
    o = _oracle(dims, 1, box)
    assert np.abs(o.field("Ex").reshape(dims[::-1])[-1, -1]).max() > 0
    _assert_equal(P, o, dims)
    simFDTD("DeleteSimulation", P)

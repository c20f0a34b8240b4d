"""The recurrences' quotients away from millimetre cells: for every float
numerator, alone and beside a subnormal one, the GPU gives bit for bit what
its IEEE division a / dx gives, for cells from far below a nanometre to far
above a kilometre; and nanometre grids with metal reaching into the CPML,
where neighbouring cells differ by tens of orders of magnitude, equal the
FP32 oracle bit for bit."""
import ctypes
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dx", [2e-38, 1e-30, 1e-9, 2e-9, 3.6e-9, 3.8e-9, 1e-6, 1e3, 2e5, 1e25, 1e38])
def test_quotients_are_exact_on_gpu(native_lib, dx):
    bad = ctypes.c_uint64(123)
    assert native_lib.fdtd_check_division(ctypes.c_float(dx), ctypes.byref(bad)) == 0, \
        native_lib.fdtd_last_error()
    assert bad.value == 0


@pytest.mark.parametrize("amp", [1e-11, 1e-9])
@pytest.mark.parametrize("dims", [(40, 36, 34), (97, 81, 67)])
def test_nanometre_cells_with_metal_equal_oracle(dims, amp):
    import oracle
    from maxwell_solver_gb300 import simFDTD

    pml, steps, dx = 6, 40, 1e-9
    sig = np.zeros(dims, np.float32)
    sig[np.arange(dims[0]) % 12 >= 2] = 1e20  # sheets, two cells apart, across the CPML
    sig = sig.ravel(order="F")
    fr = np.float32([2e14, dx, 0.9 * dx / (math.sqrt(3) * 299792458.0)])
    td = np.int32([steps, *dims, 0])
    pulse = (np.sin(0.5 * np.arange(steps) + 0.4) * amp).astype(np.float32)
    box = np.int32([0, dims[0] - 1, 3, dims[1] // 2, 5, 8])
    prm = np.float64([pml, pml + 2, 3, 1, 0.08, 1, 0.8, 0])

    P = simFDTD("CreateSimulation")
    simFDTD("SetParams", P, prm)
    simFDTD("SetConst", P, fr, td)
    simFDTD("SetSource", P, pulse)
    for f in (1, 2, 3):
        simFDTD("UpdateMaterial", P, np.int32(f), sig)
    simFDTD("ReadySimulation", P)
    simFDTD("StepN", P, np.int32([0, steps, 0]), np.int32([3, *box]))

    o = oracle.OracleSim("f32")
    o.set_params(pml=pml, tfsf_width=pml + 2)
    o.set_const(fr, td)
    o.set_source(pulse)
    for f in (1, 2, 3):
        o.update_material(f, sig)
    o.ready_simulation()
    for n in range(steps):
        o.step(n, 0)
        o.add_currents(n, 3, box)
    for f, field in enumerate(("Ex", "Ey", "Ez", "Hx", "Hy", "Hz"), 1):
        got = simFDTD("OutputVis", P, np.uint32(np.prod(dims)), np.int32(f))
        assert np.isfinite(o.field(field)).all()
        np.testing.assert_array_equal(got, o.field(field), err_msg=field)
    simFDTD("DeleteSimulation", P)

"""The marching two-pass kernels of larger 3D grids (VTI and TTI with nz % 4 != 0): sizes beside the 32 x 16 tile's
edges, the fewest planes, several x-chunks with a shorter last one.
Strict build: bitwise against the restatement after 4 steps. Fast build: relative L2 1e-5, the bound of the step
kernels' own test."""
import ctypes

import pytest

from tests.harness import ABIRunner, OracleRunner, make_model, rel_l2, same

pytestmark = pytest.mark.gpu

# (nz, ny, nx); tests/test_host_fakecuda.py checks that each takes these kernels
SHAPES = [(127, 111, 80), (225, 226, 21), (95, 96, 120), (158, 159, 45), (289, 304, 12)]


@pytest.mark.parametrize("physics", ["VTI", "TTI"])
@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("fs", [True, False])
@pytest.mark.parametrize("linear", [False, True])
def test_marching_step(oracle, physics, shape, fs, linear):
    from wavefd_b200 import _lib
    if linear and physics != "VTI":
        pytest.skip("the linear step is VTI's")
    lib, name = _lib.library(), f"Prop3DAco{physics}DenQ_DEO2_FDTD"
    model = make_model(3, physics.lower(), shape, seed=3)
    orc = OracleRunner(oracle, name, shape, fs=fs)
    orc.load(model)
    for _ in range(4):
        orc.step(linear=linear)
    for strict in (1, 0):
        gpu = ABIRunner(lib, name, shape, fs=fs)
        lib.WFD_Prop_SetStrict(ctypes.c_void_p(gpu.p), strict)
        gpu.load(model)
        for _ in range(4):
            (gpu.abi.TimeStepLinear if linear else gpu.abi.TimeStep)(gpu.p)
        assert lib.WFD_Prop_Status(ctypes.c_void_p(gpu.p)) == 0
        for k in ("PCur", "POld", "PSpace", "MCur", "MOld", "MSpace"):
            a, b = gpu.arr(k), orc.arr(k)
            assert same(a, b) if strict else rel_l2(a, b) <= 1e-5, f"{name} {shape} strict={strict} {k}"
        gpu.close()


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("fs", [True, False])
def test_marching_step_iso_unfused(oracle, shape, fs):
    """3D Iso takes the two passes with the fused kernels off (WFD_Prop_SetFused)."""
    from wavefd_b200 import _lib
    lib, name = _lib.library(), "Prop3DAcoIsoDenQ_DEO2_FDTD"
    model = make_model(3, "iso", shape, seed=3)
    orc = OracleRunner(oracle, name, shape, fs=fs)
    orc.load(model)
    for _ in range(4):
        orc.step()
    for strict in (1, 0):
        gpu = ABIRunner(lib, name, shape, fs=fs)
        lib.WFD_Prop_SetStrict(ctypes.c_void_p(gpu.p), strict)
        lib.WFD_Prop_SetFused(ctypes.c_void_p(gpu.p), 0)
        gpu.load(model)
        for _ in range(4):
            gpu.abi.TimeStep(gpu.p)
        assert lib.WFD_Prop_Status(ctypes.c_void_p(gpu.p)) == 0 and lib.WFD_Prop_StepKernels(ctypes.c_void_p(gpu.p)) == 2
        for k in ("PCur", "POld", "PSpace"):
            a, b = gpu.arr(k), orc.arr(k)
            assert same(a, b) if strict else rel_l2(a, b) <= 1e-5, f"{shape} strict={strict} {k}"
        gpu.close()

"""3D steps on grids whose depth is not a multiple of 4 (rows that TMA cannot address): sizes beside the 32 x 16 tile's edges, every remainder, the smallest grid, several x-chunks.
Strict build: bitwise against the restatement after 4 steps. Fast build: relative L2 1e-5, the bound of the
aligned kernels' own test."""
import ctypes

import pytest

from tests.harness import ABIRunner, OracleRunner, make_model, rel_l2, same

pytestmark = pytest.mark.gpu

NAMES = ["Prop3DAcoIsoDenQ_DEO2_FDTD", "Prop3DAcoVTIDenQ_DEO2_FDTD", "Prop3DAcoTTIDenQ_DEO2_FDTD"]
SHAPES = [(9, 9, 9), (31, 15, 20), (33, 17, 40), (34, 16, 12), (35, 33, 17), (66, 18, 133),
          (101, 98, 107), (103, 33, 301)]  # (nz, ny, nx); the last two take the marching two-pass kernels in VTI and TTI


@pytest.fixture(scope="module")
def lib():
    from wavefd_b200 import _lib
    return _lib.library()


@pytest.fixture(scope="module")
def oracle():
    from oracle.oracle import Oracle
    return Oracle()


@pytest.mark.parametrize("name", NAMES)
@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("fs", [True, False])
@pytest.mark.parametrize("linear", [False, True])
def test_ragged_step(lib, oracle, name, shape, fs, linear):
    physics = {"I": "iso", "V": "vti", "T": "tti"}[name[9]]
    if linear and physics != "vti":
        pytest.skip("the linear step is VTI's")
    for strict in (1, 0):
        gpu, orc = ABIRunner(lib, name, shape, fs=fs), OracleRunner(oracle, name, shape, fs=fs)
        lib.WFD_Prop_SetStrict(ctypes.c_void_p(gpu.p), strict)
        model = make_model(3, physics, shape, seed=3)
        gpu.load(model)
        orc.load(model)
        for _ in range(4):
            (gpu.abi.TimeStepLinear if linear else gpu.abi.TimeStep)(gpu.p)
            orc.step(linear=linear)
        assert lib.WFD_Prop_Status(ctypes.c_void_p(gpu.p)) == 0
        if physics == "iso":
            assert lib.WFD_Prop_StepKernels(ctypes.c_void_p(gpu.p)) == 1
        fields = ["PCur", "POld", "PSpace"] + (["MCur", "MOld", "MSpace"] if physics != "iso" else [])
        for k in fields:
            a, b = gpu.arr(k), orc.arr(k)
            assert same(a, b) if strict else rel_l2(a, b) <= 1e-5, f"{name} {shape} strict={strict} {k}"
        gpu.close()

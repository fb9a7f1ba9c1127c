"""3D fused steps cut into short x-chunks: lengths 2 and 3 with a shorter last chunk, grids no longer than the x
stencil, windows of the chunk start that reach past both ends of the grid.
Strict build: bitwise against the restatement after 4 steps. Fast build: relative L2 1e-5, the bound of the step
kernels' own test."""
import ctypes

import pytest

from tests.harness import ABIRunner, OracleRunner, make_model, rel_l2, same

pytestmark = pytest.mark.gpu

SHAPES = [(12, 9, 9), (36, 17, 14), (32, 16, 131), (64, 48, 97)]  # (nz, ny, nx)


@pytest.fixture(scope="module")
def lib():
    from wavefd_b200 import _lib
    return _lib.library()


@pytest.fixture(scope="module")
def oracle():
    from oracle.oracle import Oracle
    return Oracle()


@pytest.mark.parametrize("physics", ["iso", "tti"])
@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("fs", [True, False])
def test_short_chunks(lib, oracle, physics, shape, fs):
    name = f"Prop3DAco{'Iso' if physics == 'iso' else physics.upper()}DenQ_DEO2_FDTD"
    for strict in (1, 0):
        gpu, orc = ABIRunner(lib, name, shape, fs=fs), OracleRunner(oracle, name, shape, fs=fs)
        lib.WFD_Prop_SetStrict(ctypes.c_void_p(gpu.p), strict)
        model = make_model(3, physics, shape, seed=5)
        gpu.load(model)
        orc.load(model)
        for _ in range(4):
            gpu.abi.TimeStep(gpu.p)
            orc.step()
        assert lib.WFD_Prop_Status(ctypes.c_void_p(gpu.p)) == 0
        for k in ["PCur", "POld", "PSpace"] + (["MCur", "MOld", "MSpace"] if physics != "iso" else []):
            a, b = gpu.arr(k), orc.arr(k)
            assert same(a, b) if strict else rel_l2(a, b) <= 1e-5, f"{name} {shape} strict={strict} {k}"
        gpu.close()

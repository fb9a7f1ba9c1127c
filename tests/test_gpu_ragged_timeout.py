"""A wait of the 3D Iso step that runs out where the tiles are staged by cp.async (nz % 4 != 0): the object reports
WFD_ERR_TIMEOUT, the kernel ends, and the context stays usable (a new object steps bitwise like the checker).
The wait is shortened to 1 ns, so that it gives up while its copies are in flight; no GPU fault."""
import ctypes

import numpy as np
import pytest

from tests.harness import ABIRunner, OracleRunner, make_model, mismatch_report

pytestmark = pytest.mark.gpu

NAME = "Prop3DAcoIsoDenQ_DEO2_FDTD"


@pytest.mark.parametrize("shape", [(65, 48, 96), (33, 17, 12), (9, 9, 9)])  # (nz, ny, nx): several, two, one chunk
@pytest.mark.parametrize("strict", [0, 1])
def test_ragged_wait_that_runs_out(oracle, shape, strict):
    from wavefd_b200 import _lib
    lib = _lib.library()
    gpu = ABIRunner(lib, NAME, shape)
    lib.WFD_Prop_SetStrict(ctypes.c_void_p(gpu.p), strict)
    gpu.load(make_model(3, "iso", shape, seed=1))
    try:
        assert lib.WFD_Debug_SetPipelineWait(1) == 0
        gpu.abi.TimeStep(gpu.p)
        status = lib.WFD_Prop_Status(ctypes.c_void_p(gpu.p))
    finally:
        assert lib.WFD_Debug_SetPipelineWait(0) == 0
    gpu.close()
    assert status == 5, status  # WFD_ERR_TIMEOUT
    gpu, orc = ABIRunner(lib, NAME, shape), OracleRunner(oracle, NAME, shape)
    lib.WFD_Prop_SetStrict(ctypes.c_void_p(gpu.p), 1)
    model = make_model(3, "iso", shape, seed=2)
    gpu.load(model)
    orc.load(model)
    for _ in range(3):
        gpu.abi.TimeStep(gpu.p)
        orc.step()
    assert lib.WFD_Prop_Status(ctypes.c_void_p(gpu.p)) == 0
    for k in ("PCur", "POld", "PSpace"):
        assert np.array_equal(gpu.arr(k), orc.arr(k)), f"{k}: {mismatch_report(gpu.arr(k), orc.arr(k))}"
    gpu.close()

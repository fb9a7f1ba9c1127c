"""A bounded wait that runs out is reported by the object (or batch) whose step it was, whichever synchronises
first. The waits are shortened to 1 ns (WFD_Debug_SetPipelineWait), so that they give up while their copies are
still in flight; no GPU fault."""
import ctypes

import pytest

from tests.harness import ABIRunner, make_model

pytestmark = pytest.mark.gpu

TIMEOUT = 5
NAMES = ["Prop3DAcoIsoDenQ_DEO2_FDTD", "Prop3DAcoVTIDenQ_DEO2_FDTD", "Prop3DAcoTTIDenQ_DEO2_FDTD"]


def _object(lib, name, shape=(64, 48, 96)):
    g = ABIRunner(lib, name, shape)
    g.load(make_model(3, {"I": "iso", "V": "vti", "T": "tti"}[name[9]], shape, seed=1))
    g.abi.TimeStep(g.p)
    assert lib.WFD_Prop_Status(ctypes.c_void_p(g.p)) == 0
    return g, ctypes.c_void_p(g.p)


def _batch(lib, props):
    lib.WFD_Batch_Create.restype = ctypes.c_void_p
    lib.WFD_Batch_Create.argtypes = [ctypes.POINTER(ctypes.c_void_p), ctypes.c_long]
    lib.WFD_Batch_Run.argtypes = [ctypes.c_void_p, ctypes.c_long, ctypes.c_long, ctypes.c_int]
    lib.WFD_Batch_Synchronize.argtypes = lib.WFD_Batch_Free.argtypes = [ctypes.c_void_p]
    b = lib.WFD_Batch_Create((ctypes.c_void_p * len(props))(*props), len(props))
    assert b
    return b


@pytest.fixture()
def lib():
    from wavefd_b200 import _lib
    lib = _lib.library()
    yield lib
    assert lib.WFD_Debug_SetPipelineWait(0) == 0


@pytest.mark.parametrize("name", NAMES)
def test_other_objects_and_batches_do_not_take_the_report(lib, name):
    a, pa = _object(lib, name)
    b, pb = _object(lib, name)
    c, pc = _object(lib, name)
    batch = _batch(lib, [pc])
    assert lib.WFD_Debug_SetPipelineWait(1) == 0
    assert lib.WFD_Prop_TimeStepAsync(pa, 1, 0) == 0
    assert lib.WFD_Debug_SetPipelineWait(0) == 0
    b.abi.TimeStep(b.p)
    assert lib.WFD_Prop_Status(pb) == 0
    assert lib.WFD_Batch_Run(batch, 2, 1, 0) == 0 and lib.WFD_Batch_Synchronize(batch) == 0
    assert lib.WFD_Prop_Synchronize(pc) == 0
    assert lib.WFD_Prop_Synchronize(pa) == TIMEOUT
    lib.WFD_Batch_Free(batch)
    for g in (a, b, c):
        g.close()


@pytest.mark.parametrize("name", NAMES)
@pytest.mark.parametrize("graph", [0, 1])
@pytest.mark.parametrize("batch_first", [True, False])
def test_a_batch_and_its_objects_report(lib, name, graph, batch_first):
    a, pa = _object(lib, name)
    b, pb = _object(lib, name)
    other, po = _object(lib, name)
    batch = _batch(lib, [pa, pb])
    assert lib.WFD_Debug_SetPipelineWait(1) == 0
    assert lib.WFD_Batch_Run(batch, 2, 1, graph) == 0
    assert lib.WFD_Debug_SetPipelineWait(0) == 0
    other.abi.TimeStep(other.p)
    assert lib.WFD_Prop_Status(po) == 0
    if batch_first:
        assert lib.WFD_Batch_Synchronize(batch) == TIMEOUT
    assert lib.WFD_Prop_Synchronize(pa) == TIMEOUT and lib.WFD_Prop_Synchronize(pb) == TIMEOUT
    assert lib.WFD_Batch_Synchronize(batch) == TIMEOUT
    lib.WFD_Batch_Free(batch)
    for g in (a, b, other):
        g.close()

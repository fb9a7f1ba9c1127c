"""Host side of the library on a stand-in CUDA runtime (fake_cudart.c): failures of single calls, and which kernels
a call takes. No GPU."""
import pytest

from tests.fakecuda import run

NAMES = ["Prop3DAcoIsoDenQ_DEO2_FDTD", "Prop2DAcoTTIDenQ_DEO2_FDTD"]

CREATE = r"""
name, dims = {name!r}, {dims!r}
free = getattr(lib, name + "_free")
free.argtypes = [ctypes.c_void_p]
"""


def _create(name):
    return CREATE.format(name=name, dims=(20, 18 if "3D" in name else 0, 16))


@pytest.mark.parametrize("name", NAMES)
def test_every_allocation_of_a_constructor_is_checked(name):
    """Each allocation in turn fails once: no object, WFD_ERR_ALLOC, nothing left behind; the next object of the
    process is whole and steps."""
    n = len(run(_create(name) + "a, p = create(name, *dims)\nfor l in log('alloc'): print(l)\n"))
    assert n >= 7
    for k in range(1, n + 1):
        out = run(_create(name) + r"""
a, p = create(name, *dims)
live = fake.fake_live()
print("NULL" if not p else "OBJECT", lib.WFD_LastError(), lib.WFD_LastErrorMessage().decode(), live)
a, p = create(name, *dims)
a.TimeStep(p)
print("OBJECT" if p else "NULL", lib.WFD_Prop_Status(ctypes.c_void_p(p)))
""", WAVEFD_B200_FAIL_ALLOC=str(k))
        assert out[0].startswith("NULL 2 ") and "injected" in out[0] and out[0].endswith(" 0"), (k, out)
        assert out[1] == "OBJECT 0", (k, out)


def test_objects_and_batches_give_their_memory_back():
    out = run(r"""
objs = [create("Prop3DAcoIsoDenQ_DEO2_FDTD", 20, 18, 16) for _ in range(2)]
lib.WFD_Batch_Create.restype = ctypes.c_void_p
lib.WFD_Batch_Create.argtypes = [ctypes.POINTER(ctypes.c_void_p), ctypes.c_long]
lib.WFD_Batch_Run.argtypes = [ctypes.c_void_p, ctypes.c_long, ctypes.c_long, ctypes.c_int]
lib.WFD_Batch_Free.argtypes = [ctypes.c_void_p]
b = lib.WFD_Batch_Create((ctypes.c_void_p * 2)(*[p for _, p in objs]), 2)
print(lib.WFD_Batch_Run(b, 3, 1, 1))
lib.WFD_Batch_Free(b)
for a, p in objs:
    a.free(p)
print(fake.fake_live())
""")
    assert out == ["0", "0"]


@pytest.mark.parametrize("strict", ["0", "1"])
@pytest.mark.parametrize("name,dims", [("Prop3DAcoIsoDenQ_DEO2_FDTD", (24, 20, 17)),
                                       ("Prop3DAcoIsoDenQ_DEO2_FDTD", (24, 20, 16)),
                                       ("Prop3DAcoVTIDenQ_DEO2_FDTD", (24, 20, 16)),
                                       ("Prop3DAcoTTIDenQ_DEO2_FDTD", (24, 20, 16)),
                                       ("Prop2DAcoVTIDenQ_DEO2_FDTD", (24, 0, 16)),
                                       ("Prop2DAcoTTIDenQ_DEO2_FDTD", (24, 0, 16))])
def test_a_second_device_steps_too(name, dims, strict):
    """Kernels with more than 48 KB of shared memory need it granted on each device that runs them."""
    out = run(f"""
for dev in (0, 1, 0):
    fake.cudaSetDevice(dev)
    a, p = create({name!r}, *{dims!r})
    fake.fake_reset()
    a.TimeStep(p)
    print(lib.WFD_Prop_Status(ctypes.c_void_p(p)), lib.WFD_Prop_Run(p, 3, 1, None, None, None, None, 3, 0))
    print(*launches())
""", WAVEFD_B200_STRICT=strict)
    assert out[::2] == ["0 0"] * 3, out
    assert out[1] == out[3] == out[5] != ""


def _two_pass(physics, sizes):
    """The kernels of a step, for (nx, ny, nz) with nz % 4 != 0."""
    return run(f"""
for size in {sizes!r}:
    a, p = create("Prop3DAco{physics}DenQ_DEO2_FDTD", *size)
    fake.fake_reset()
    a.TimeStep(p)
    print(*launches())
    a.free(p)
""")


@pytest.mark.parametrize("physics", ["VTI", "TTI"])
def test_two_pass_kernels_by_size(physics):
    """Marching kernels for a million cells and more in well filled tiles, one thread a cell elsewhere (thin grids
    took up to 3.9 times as long on the marching kernels)."""
    from tests.test_gpu_pass3d import SHAPES
    marching = [(nx, ny, nz) for nz, ny, nx in SHAPES] + [(203, 181, 251), (250, 90, 90), (16, 400, 301), (80, 112, 126)]
    cells = [(12000, 9, 10), (3000, 17, 33), (2000, 33, 17), (20, 20, 3001), (40, 33, 1001), (300, 18, 301), (300, 300, 33),
             (600, 33, 65), (300, 70, 70), (64, 60, 67)]
    for line in _two_pass(physics, marching):
        assert "k_pass1_3d" in line and "k_pass2_3d" in line, line
    for size, line in zip(cells, _two_pass(physics, cells)):
        assert "k_pass1I" in line and "k_pass2I" in line and "_3d" not in line, (size, line)


def test_two_pass_kernels_between_the_lines():
    """Where only one physics gains."""
    sizes = [(400, 180, 50), (101, 100, 101), (200, 97, 97), (9, 1000, 301)]
    assert all("_3d" not in line for line in _two_pass("VTI", sizes))
    assert all("k_pass1_3d" in line for line in _two_pass("TTI", sizes))


@pytest.mark.parametrize("call", ["injectdata", "extractdata"])
def test_host_points_copied_where_one_thread_reads_many(call):
    """Drop-in calls with host arrays: (groups, points a group) and whether the values go to the device by a copy."""
    want = {(1, 1): 0, (1, 64): 0, (1, 65): 1, (2, 512): 1, (40, 64): 0, (4096, 1): 0, (4097, 1): 1, (1, 5000): 1}
    out = run(f"""
import numpy as np
from wavefd_b200 import spacetime
for groups, per in {list(want)!r}:
    pts = np.zeros(groups * per, spacetime.SOURCEPOINT32)
    one, many = ("iu", "ir") if {call!r} == "injectdata" else ("ir", "iu")
    pts[one], pts[many], pts["c"] = np.repeat(np.arange(1, groups + 1), per), np.arange(groups * per) % 4000 + 1, 1.0
    field, data = np.zeros(8000, np.float32), np.zeros((8000, 2), np.float32)
    for again in range(2):  # the first call also uploads the points
        fake.fake_reset()
        if {call!r} == "injectdata": spacetime.injectdata(field, [pts], data, 1)
        else: spacetime.extractdata(data, field, 1, [pts])
    print(len(log("copy")), len(launches()))
""")
    assert out == [f"{n} 1" for n in want.values()], out


def test_run_allocates_scratch_only_for_steps_that_use_it():
    """Grid-sized allocations of WFD_Prop_Run: none where one kernel does the step."""
    want = {("Prop3DAcoIsoDenQ_DEO2_FDTD", 30, 20, 17): 0, ("Prop3DAcoIsoDenQ_DEO2_FDTD", 30, 20, 16): 0,
            ("Prop3DAcoTTIDenQ_DEO2_FDTD", 30, 20, 16): 0, ("Prop3DAcoVTIDenQ_DEO2_FDTD", 30, 20, 17): 6,
            ("Prop2DAcoIsoDenQ_DEO2_FDTD", 300, 0, 170): 3}
    out = run(f"""
for name, nx, ny, nz in {list(want)!r}:
    a, p = create(name, nx, ny, nz)
    fake.fake_reset()
    rc = lib.WFD_Prop_Run(p, 5, 1, None, None, None, None, 5, 1)
    print(rc, sum(int(n) >= 4 * nx * max(ny, 1) * nz for _, n in log("alloc")))
""")
    assert out == [f"0 {n}" for n in want.values()], out


def test_every_allocation_of_a_snapshot_file_is_checked(tmp_path):
    code = f"""
lib.WFD_Snap_Close.argtypes = [ctypes.c_void_p]
before = fake.fake_live()
f = lib.WFD_Snap_Open({str(tmp_path / "s")!r}.encode(), 3, 5000, 0)
print("FILE" if f else "NULL", lib.WFD_LastError(), fake.fake_live() - before if not f else len(log("alloc")))
if f: lib.WFD_Snap_Close(f)
"""
    kind, rc, n = run(code)[-1].split()
    assert kind == "FILE" and int(n) >= 2
    for k in range(1, int(n) + 1):
        assert run(code, WAVEFD_B200_FAIL_ALLOC=str(k))[-1] == "NULL 2 0", k

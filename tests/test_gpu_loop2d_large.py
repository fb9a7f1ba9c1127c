"""Whole 2D time loops on grids with more 64 x 16 tiles than any co-resident set of CTAs of 512 threads (four an
SM), which the fast build runs as two passes a step (k_loop2d)."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

NT = 13


def _run(physics, shape, fs, spts, rpts, loop=True):
    """Fields and traces after NT steps, by one WFD_Prop_Run or by the stepping calls."""
    import torch
    from tests.harness import ABIRunner, make_model
    from wavefd_b200 import _lib
    from wavefd_b200.abi import SourcePoint32
    lib = _lib.library()
    nx, nz = shape
    assert -(-nx // 16) * -(-nz // 64) > 4 * torch.cuda.get_device_properties(0).multi_processor_count
    g = ABIRunner(lib, f"Prop2DAco{physics}DenQ_DEO2_FDTD", (nz, 1, nx), fs=fs)
    g.load(make_model(2, physics.lower(), (nz, 1, nx), seed=8))
    wav = torch.from_numpy(np.random.default_rng(4).standard_normal((2, NT)).astype(np.float32)).cuda()
    tab = [lib.WFD_Points_Create((SourcePoint32 * len(p))(*[SourcePoint32(*q) for q in p]), len(p), k) if p else None
           for k, p in enumerate((spts, rpts))]
    trc = torch.zeros((nx, NT), device="cuda")
    torch.cuda.synchronize()
    vp = lambda t: ctypes.c_void_p(t.data_ptr())  # noqa: E731
    p = ctypes.c_void_p(g.p)
    if loop:
        assert lib.WFD_Prop_Run(p, NT, 1, tab[0], vp(wav), tab[1], vp(trc), NT, 1) == 0
        assert lib.WFD_Prop_RunLaunches(p) == 1
    else:
        s = ctypes.c_void_p(lib.WFD_Prop_Stream(p))
        for it in range(1, NT + 1):
            assert lib.WFD_Prop_TimeStepAsync(p, 1, 0) == 0
            pc = ctypes.c_void_p(ctypes.cast(g.abi.getPCur(g.p), ctypes.c_void_p).value)
            if tab[0]:
                assert lib.WFD_Inject(tab[0], pc, vp(wav), it, NT, s) == 0
            if tab[1]:
                assert lib.WFD_Extract(tab[1], vp(trc), pc, it, NT, s) == 0
    assert lib.WFD_Prop_Synchronize(p) == 0
    keys = ("PCur", "POld", "PSpace") + (() if physics == "Iso" else ("MCur", "MOld", "MSpace"))
    out = {k: g.arr(k).copy() for k in keys}
    out["traces"] = trc.cpu().numpy()
    for t in tab:
        if t:
            lib.WFD_Points_Free(t)
    g.close()
    return out


@pytest.mark.parametrize("physics", ["Iso", "VTI", "TTI"])
def test_source_points_beyond_the_grid_are_left_out(physics):
    """As in the loops of the smaller grids, whose tiles hold no such cell."""
    nx, nz = shape = (1211, 706)
    inside = [(5 * nz + 9, 1, 1.0)]
    rec = [(x * nz + 4, x + 1, 1.0) for x in range(nx)]
    want = _run(physics, shape, True, inside, rec)
    got = _run(physics, shape, True, inside + [(nx * nz + 1, 1, 3.0), ((nx + 200) * nz + 8, 2, 5.0)], rec)
    for k in want:
        assert np.array_equal(got[k], want[k]), k


# (nx, nz): tiles of 16 x 64 with 1, 11, 15 and 5 rows and 3, 2, 3, 9 and 63 columns over; row pairs that straddle the
# last computed row and the grid's end (odd nx)
SHAPES = [(5009, 67), (1211, 706), (4015, 131), (9509, 9), (1185, 575)]


@pytest.mark.parametrize("physics", ["Iso", "VTI", "TTI"])
@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("fs", [True, False])
@pytest.mark.parametrize("acquisition", [True, False])
def test_loop_is_the_stepping_calls_bit_for_bit(physics, shape, fs, acquisition):
    nx, nz = shape
    pt = lambda x, z, ir, c: (x * nz + z + 1, ir, c)  # noqa: E731
    spts = [pt(nx // 2, nz // 2, 1, 1.0), pt(nx // 2, nz // 2, 2, 0.5), pt(nx - 1, nz - 1, 2, 0.25), pt(4, 4, 1, 0.3),
            pt(nx - 5, nz - 5, 1, 0.7), pt(0, 0, 2, 0.1)]
    rpts = [pt(x, min(3, nz - 1), x + 1, 1.0) for x in range(nx)] + [pt(nx // 2, nz // 2, 2, 0.5)]
    if not acquisition:
        spts = rpts = []
    got, want = (_run(physics, shape, fs, spts, rpts, loop) for loop in (True, False))
    for k in want:
        assert np.isfinite(want[k]).all() and np.array_equal(got[k], want[k]), f"{physics} {shape} fs={fs} {k}"

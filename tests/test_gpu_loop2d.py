"""Whole 2D time loops in the fast build (two passes a step in one cooperative launch) against stepping call
by call, at sizes beside the 64 x 16 tiles, one tile, several rounds of tiles, no injection or extraction:
fields and traces to relative L2 1e-5 (the fast build's bound against the restatement after 40 steps)."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SHAPES = [(9, 9), (16, 64), (17, 65), (15, 63), (33, 130), (301, 257), (1210, 705)]  # (nx, nz)


@pytest.mark.parametrize("physics", ["Iso", "VTI", "TTI"])
@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("fs", [True, False])
@pytest.mark.parametrize("acquisition", [True, False])
def test_loop_against_steps(physics, shape, fs, acquisition):
    import torch
    from tests.harness import ABIRunner, make_model, rel_l2
    from wavefd_b200 import _lib
    from wavefd_b200.abi import SourcePoint32
    lib = _lib.library()
    nx, nz = shape
    name = f"Prop2DAco{physics}DenQ_DEO2_FDTD"
    nt = 13
    pt = lambda x, z, ir, c: SourcePoint32(x * nz + z + 1, ir, c)  # noqa: E731
    spts = [pt(nx // 2, nz // 2, 1, 1.0), pt(nx // 2, nz // 2, 2, 0.5), pt(nx - 1, nz - 1, 2, 0.25), pt(4, 4, 1, 0.3)]
    rpts = [pt(x, 3, x + 1, 1.0) for x in range(nx)] + [pt(nx // 2, nz // 2, 2, 0.5)]
    wav = torch.from_numpy(np.random.default_rng(4).standard_normal((2, nt)).astype(np.float32)).cuda()
    out = []
    for loop in (True, False):
        g = ABIRunner(lib, name, (nz, 1, nx), fs=fs)
        g.load(make_model(2, physics.lower(), (nz, 1, nx), seed=8))
        tab = [lib.WFD_Points_Create((SourcePoint32 * len(p))(*p), len(p), k) for k, p in enumerate((spts, rpts))]
        trc = torch.zeros((nx, nt), device="cuda")
        torch.cuda.synchronize()
        vp = lambda t: ctypes.c_void_p(t.data_ptr())  # noqa: E731
        p = ctypes.c_void_p(g.p)
        if loop:
            assert lib.WFD_Prop_Run(p, nt, 1, *((tab[0], vp(wav), tab[1], vp(trc)) if acquisition else (None,) * 4), nt,
                                    1) == 0
            assert lib.WFD_Prop_RunLaunches(p) == 1
        else:
            s = ctypes.c_void_p(lib.WFD_Prop_Stream(p))
            for it in range(1, nt + 1):
                assert lib.WFD_Prop_TimeStepAsync(p, 1, 0) == 0
                pc = ctypes.c_void_p(ctypes.cast(g.abi.getPCur(g.p), ctypes.c_void_p).value)
                if acquisition:
                    assert lib.WFD_Inject(tab[0], pc, vp(wav), it, nt, s) == 0
                    assert lib.WFD_Extract(tab[1], vp(trc), pc, it, nt, s) == 0
        assert lib.WFD_Prop_Synchronize(p) == 0
        keys = ("PCur", "POld", "PSpace") + (() if physics == "Iso" else ("MCur", "MOld", "MSpace"))
        out.append([g.arr(k).copy() for k in keys] + [trc.cpu().numpy()])
        for t in tab:
            lib.WFD_Points_Free(t)
        g.close()
    for a, b, k in zip(*out, keys + ("traces",)):
        assert np.isfinite(a).all() and rel_l2(a, b) <= 1e-5, f"{name} {shape} fs={fs} {k}: {rel_l2(a, b):.2e}"
